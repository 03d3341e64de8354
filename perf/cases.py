"""The work whose time matters, through the package's public entry points.

A case is a dict of plain values.  Its ``kind`` picks the entry points:

  solve     one ``Context.solve`` / ``Context.solve_raw`` call on a batch: pre-run, main run and
            (solve) stitching.  ``api`` = "couplings" decodes given bond patterns and ends with
            the logical-class log-probabilities
  prerun    ``wlg_prerun`` alone (what the pre-run program does)
  serve     requests submitted to a running ``Server`` and waited for
  setup     the set-up operators on the caller's device buffers: disorder, error chain, lattices,
            energies and the pre-run walk
  iterate   one outer iteration on the operators: sweep, flatness, averages, reset, finished
            check and both exchange passes, on the caller's device buffers
  plain     ``solve_plain``, the reference's program structure on the operators

Batches that would walk for minutes are capped at ``max_outer`` outer iterations and return every
window's log g as it stands (``solve_raw``).  The seed draws disorder and random streams; the lattice
sizes of an uneven batch follow from ``shapes``, so a case's outputs have one shape: log g curves
stand on the full energy range, windows one after another in a buffer of their largest total size.
"""
import ctypes as C
import math

import numpy as np
import torch

import qec_pf_wang_landau_gb300 as wlg

BASE = dict(kind="solve", api="solve", problems=1, x0=4, x1=4, square=True, boundary="periodic", classes="i", p0=0.04,
            p1=0.04, pre_walkers=128, pre_intervals=32, pre_iterations=0, pre_per_site=100, intervals=10, walkers=3,
            overlap=0.25, alpha=0.8, beta=1e-3, iterations=1000, exchange_every=20, max_outer=0, shapes=1)


def _case(name, **kw):
    unknown = set(kw) - set(BASE)
    if unknown:
        raise ValueError(f"unknown fields {unknown}")
    c = dict(BASE, **kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest run of the reference's README: one 4x4 sample, pre-run to log g
        _case("one_4x4", pre_walkers=32, pre_intervals=8, pre_iterations=1000),
        # one syndrome decoded: the four classes of a given 6x6 bond pattern
        _case("decode_6x6", api="couplings", problems=4, x0=6, x1=6, classes="ivhc", p0=0.08, p1=0.08,
              pre_iterations=4000),
        # a threshold study's unit of work: 100 disorder samples of 6x6, all four classes
        _case("batch_6x6", problems=400, x0=6, x1=6, classes="ivhc", pre_iterations=1000),
        # uneven lattices, rectangular, periodic and open, in one batch; windows scaled with the lattice
        _case("batch_mixed", api="raw", problems=240, x0=4, x1=12, square=False, boundary="both", classes="random",
              p0=0.02, p1=0.12, intervals=0, walkers=4, max_outer=150),
        # large lattices that fill the GPU: 64 windows x 8 walkers a problem
        _case("large_16x16", api="raw", problems=152, x0=16, x1=16, classes="ivhc", p0=0.10, p1=0.10,
              pre_intervals=128, intervals=64, walkers=8, overlap=0.3, beta=1e-8, exchange_every=10, max_outer=60),
        # the four classes of one larger sample: few problems, all of them long
        _case("few_24x24", api="raw", problems=4, x0=24, x1=24, classes="ivhc", p0=0.10, p1=0.10, pre_intervals=128,
              intervals=64, walkers=8, overlap=0.3, beta=1e-8, exchange_every=10, max_outer=60),
        # open boundaries, short sweeps between flatness checks, exchange after each
        _case("open_short_sweeps", api="raw", problems=96, x0=7, x1=11, square=False, boundary="open",
              classes="random", p0=0.05, p1=0.10, intervals=12, walkers=5, iterations=100, exchange_every=1,
              max_outer=400),
        # the pre-run program on its own over uneven lattices
        _case("prerun_mixed", kind="prerun", problems=120, x0=4, x1=16, square=False, boundary="both",
              classes="random", p0=0.02, p1=0.12),
        # decoding requests through the running server
        _case("serve", kind="serve", problems=24, x0=4, x1=9, p0=0.02, p1=0.12, pre_per_site=400, intervals=8,
              walkers=4, beta=2e-2),
        # set-up of a run on the operators: many samples, as a program written against them makes it
        _case("setup_ops", kind="setup", problems=64, x0=9, x1=9, classes="c", p0=0.08, p1=0.08, pre_iterations=1000),
        # one outer iteration of a program written against the operators
        _case("iterate_ops", kind="iterate", problems=16, x0=10, x1=10, p0=0.08, p1=0.08, pre_per_site=40,
              intervals=16, walkers=4, iterations=200),
        # the reference's program structure end to end
        _case("plain_6x6", kind="plain", problems=16, x0=6, x1=6, pre_iterations=1000, beta=0.3),
    ]


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    return dict(_draw(rng), shapes=rng.randint(2, 1 << 20))


def _draw(rng):
    def log_int(a, b):
        return min(b, max(a, int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))))

    p0 = rng.uniform(0.02, 0.10)
    p = dict(p0=round(p0, 4), p1=round(p0, 4))
    uneven = dict(p0=round(p0, 4), p1=round(p0 + 0.02, 4))
    bc = rng.choice(["periodic", "open", "both"])
    family = rng.choice(["one", "decode", "batch", "mixed", "large", "short", "prerun", "serve", "setup", "iterate",
                         "plain"])
    if family == "one":
        x = rng.randint(4, 6)
        return _case(None, x0=x, x1=x, boundary=rng.choice(["periodic", "open"]), pre_walkers=rng.choice([32, 64, 100]),
                     pre_intervals=8, pre_per_site=100, intervals=rng.randint(4, 10), walkers=rng.randint(2, 4),
                     beta=1e-2, **p)
    if family == "decode":
        x = rng.randint(4, 7)
        return _case(None, api="couplings", problems=4, x0=x, x1=x, classes="ivhc",
                     boundary=rng.choice(["periodic", "open"]), intervals=rng.randint(4, 10),
                     walkers=rng.randint(2, 4), beta=1e-2, **p)
    if family == "batch":
        x = rng.randint(5, 7)
        return _case(None, problems=log_int(20, 400), x0=x, x1=x, classes="ivhc", pre_per_site=60,
                     intervals=rng.randint(6, 10), walkers=rng.randint(2, 4), beta=1e-2, **p)
    if family == "mixed":
        return _case(None, api="raw", problems=log_int(12, 240), x0=4, x1=rng.randint(6, 12), square=False,
                     boundary=bc, classes="random", intervals=0, walkers=rng.randint(2, 5),
                     max_outer=log_int(10, 150), exchange_every=rng.randint(1, 25), **uneven)
    if family == "large":
        x = rng.randint(13, 24)
        return _case(None, api="raw", problems=log_int(1, 152 if x < 18 else 16), x0=x, x1=x, classes="ivhc",
                     pre_intervals=128, intervals=rng.choice([32, 48, 64]), walkers=rng.randint(4, 8), overlap=0.3,
                     beta=1e-8, exchange_every=10, max_outer=log_int(5, 40), **p)
    if family == "short":
        return _case(None, api="raw", problems=log_int(8, 96), x0=6, x1=rng.randint(8, 11), square=False, boundary=bc,
                     classes="random", intervals=rng.randint(6, 14), walkers=rng.randint(2, 6),
                     iterations=log_int(20, 400), exchange_every=rng.randint(1, 4), max_outer=log_int(40, 400),
                     **uneven)
    if family == "prerun":
        return _case(None, kind="prerun", problems=log_int(8, 120), x0=4, x1=rng.randint(6, 16), square=False,
                     boundary=bc, classes="random", pre_walkers=rng.choice([32, 100, 128, 192]),
                     pre_per_site=rng.randint(20, 100), **uneven)
    if family == "serve":
        return _case(None, kind="serve", problems=log_int(2, 24), x0=4, x1=rng.randint(5, 9), pre_per_site=400,
                     intervals=rng.randint(5, 8), walkers=rng.randint(2, 4), beta=2e-2, **uneven)
    if family == "setup":
        x = rng.randint(5, 12)
        return _case(None, kind="setup", problems=log_int(4, 64), x0=x, x1=x, classes=rng.choice("ivhc"),
                     boundary=rng.choice(["periodic", "open"]), pre_walkers=rng.choice([32, 100, 128]),
                     pre_iterations=log_int(100, 1000), **p)
    if family == "iterate":
        x = rng.randint(5, 12)
        return _case(None, kind="iterate", problems=log_int(2, 16), x0=x, x1=x, pre_per_site=40,
                     boundary=rng.choice(["periodic", "open"]), intervals=rng.randint(6, 12),
                     walkers=rng.randint(2, 5), iterations=log_int(20, 200), **p)
    x = rng.randint(4, 6)
    return _case(None, kind="plain", problems=log_int(1, 16), x0=x, x1=x, pre_per_site=40, intervals=rng.randint(4, 8),
                 walkers=rng.randint(2, 3), beta=0.3, **p)


# ------------------------------------------------------------------ inputs --

def _problems(case, seed):
    rng = np.random.default_rng(case["shapes"])
    out = []
    classes = case["classes"]
    run_seed = int(np.random.default_rng(seed).integers(1, 1 << 30))
    for k in range(case["problems"]):
        x = int(rng.integers(case["x0"], case["x1"] + 1))
        y = x if case["square"] else int(rng.integers(case["x0"], case["x1"] + 1))
        bc = {"periodic": 0, "open": 1, "both": int(rng.integers(0, 2))}[case["boundary"]]
        n = x * y
        p = float(rng.uniform(case["p0"], case["p1"])) if case["p1"] > case["p0"] else case["p0"]
        if classes == "random":
            cls, sample = "ivhc"[int(rng.integers(0, 4))], k
        else:
            cls, sample = classes[k % len(classes)], k // len(classes)
        out.append(wlg.problem(
            x, y, boundary=bc, prob=p, error_class=cls, seed=run_seed, sample=sample, pre_walkers=case["pre_walkers"],
            pre_intervals=case["pre_intervals"], pre_iterations=case["pre_iterations"] or case["pre_per_site"] * n,
            intervals=case["intervals"] or min(32, max(8, n // 8)), walkers_per_interval=case["walkers"],
            overlap=case["overlap"], alpha=case["alpha"], beta=case["beta"], iterations=case["iterations"],
            exchange_every=case["exchange_every"], max_outer=case["max_outer"]))
    return out


def _raw_size(p):
    """Most window values a problem can have: its windows of the full range, the last one longer."""
    full = 4 * p.X * p.Y + 1
    return p.intervals * int(full / (1 + p.overlap * (p.intervals - 1))) + full


def _pattern(case, seed):
    """The one bond pattern that a decoding case's four classes share."""
    x = case["x0"]
    return np.where(np.random.default_rng([seed, 1]).random(2 * x * x) < case["p0"], -1, 1).astype(np.int8)


def _prerun(ctx, probs):
    n = len(probs)
    arr = (wlg.Problem * n)(*probs)
    N = [p.X * p.Y for p in probs]
    B = [p.pre_intervals for p in probs]
    seen = np.zeros(sum(4 * v + 1 for v in N), np.uint8)
    J = np.zeros(sum(2 * v for v in N), np.int8)
    found = np.zeros(sum(B), np.int32)
    energy = np.zeros(sum(B), np.int32)
    lat = np.zeros(sum(b * v for b, v in zip(B, N)), np.int8)
    outs = [a.ctypes.data_as(C.c_void_p) for a in (seen, J, found, energy, lat)]
    ctx._check("wlg_prerun", wlg.lib().wlg_prerun(ctx._h, C.cast(arr, C.c_void_p), n, *outs))
    return seen, J, found, energy, lat


def _iterate_arrays(case, seed):
    """Host arrays of a run in progress on the operators' layout: windows and start lattices from a
    pre-run; log g near the Gaussian density of states with per-walker scatter, counts near their
    flatness threshold, every fourth window finished."""
    probs = _problems(case, seed)
    R, I, W = len(probs), case["intervals"], case["walkers"]
    X, Y = probs[0].X, probs[0].Y
    N = X * Y
    ctx = wlg.Context(0)
    pre = _prerun(ctx, probs)
    ctx.close()
    ho = wlg.handoff(probs, *pre)
    for h in ho:
        if h["status"] != 0:
            raise RuntimeError("the pre-run left a window without a start lattice")
    rng = np.random.default_rng([seed, 2])
    T = R * I * W
    spectrum, off_spec, at = [], [], 0
    for h in ho:
        off_spec.append(at)
        part = h["spectrum"][h["e_min"] + 2 * N:h["e_max"] + 2 * N + 1].astype(np.int8)
        spectrum.append(part)
        at += len(part)
    start = np.concatenate([h["start"] for h in ho]).astype(np.int32)
    end = np.concatenate([h["end"] for h in ho]).astype(np.int32)
    length = (end - start + 1).repeat(W)
    off_hist = (np.cumsum(length) - length).astype(np.int32)
    lat = np.concatenate([h["lattices"].repeat(W, axis=0).ravel() for h in ho])
    cond = np.zeros(R * I, np.int8)
    cond[3::4] = 1
    factor = np.where(cond == 1, math.exp(case["beta"] / 2), math.exp(2.0 ** -6)).repeat(W)
    size = W * sum(_raw_size(p) for p in probs)
    logG, H = np.zeros(size), np.zeros(size, np.int64)
    for t in range(T):
        b = t // W
        k = b // I
        e = np.arange(start[b], end[b] + 1)
        on = ho[k]["spectrum"][e + 2 * N] == 1
        s = slice(off_hist[t], off_hist[t] + length[t])
        logG[s] = np.where(on, N * math.log(2) - e * e / (4.0 * N) + 1 + 0.05 * rng.random(len(e)), 0.0)
        H[s] = np.where(on, rng.integers(300, 380, len(e)), 0)
    if cond.any():  # walkers of a finished window share its average
        for b in np.nonzero(cond)[0]:
            for w in range(1, W):
                n = length[b * W]
                logG[off_hist[b * W + w]:off_hist[b * W + w] + n] = logG[off_hist[b * W]:off_hist[b * W] + n]
    J = pre[1]
    return dict(X=X, Y=Y, N=N, R=R, I=I, W=W, T=T, seed=probs[0].seed, boundary=probs[0].boundary,
                lattice=lat.astype(np.int8), J=J, H=H, logG=logG, factor=factor,
                E=_energies(lat.reshape(T, N), J.reshape(R, 2 * N).repeat(I * W, axis=0), X, Y, probs[0].boundary),
                newE=np.zeros(T, np.int32), off_iter=np.zeros(T, np.int64), found=np.zeros(T, np.int32), start=start,
                end=end, off_hist=off_hist, off_lat=(np.arange(T) * N).astype(np.int32), cond=cond,
                spectrum=np.concatenate(spectrum), off_spec=np.array(off_spec, np.int32),
                cond_sample=np.zeros(R, np.int32), perm=(np.arange(T) % W).astype(np.int32))


_DEVICE = ["lattice", "J", "H", "logG", "factor", "E", "newE", "off_iter", "found", "start", "end", "off_hist",
           "off_lat", "cond", "spectrum", "off_spec", "cond_sample", "perm"]
_ITERATE_OUT = ["lattice", "H", "logG", "factor", "E", "off_iter", "found", "off_lat", "cond", "cond_sample", "perm"]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "iterate":
        host = _iterate_arrays(case, seed)
        st = {k: v for k, v in host.items() if k not in _DEVICE}
        st.update({k: torch.from_numpy(np.ascontiguousarray(host[k])).cuda() for k in _DEVICE})
        torch.cuda.synchronize()
        return dict(case=case, dev=st)
    probs = _problems(case, seed)
    if kind in ("solve", "prerun"):
        st = dict(case=case, probs=probs, ctx=wlg.Context(0))
        if case["api"] == "couplings":
            J = _pattern(case, seed)
            st["couplings"] = [J] * len(probs)
        return st
    if kind == "serve":
        return dict(case=case, probs=probs, server=wlg.Server(0))
    if kind == "plain":
        return dict(case=case, probs=probs)
    # setup: the caller's device buffers
    R, q = len(probs), probs[0]
    N, T, B = q.X * q.Y, len(probs) * q.pre_walkers, q.pre_intervals
    z = lambda n, dt: torch.zeros(n, dtype=dt, device="cuda")
    st = dict(case=case, q=q, R=R, N=N, T=T, B=B, J=z(R * 2 * N, torch.int8), lat=z(T * N, torch.int8),
              E=z(T, torch.int32), H=z(R * (4 * N + 1), torch.int64), off=z(T, torch.int64),
              found_lat=z(R * B * N, torch.int8), flag=z(R * B, torch.int32), found_E=z(R * B, torch.int32),
              off_lat=(torch.arange(T, device="cuda") * N).int(),
              off_found=(torch.arange(R * B, device="cuda") * N).int())
    torch.cuda.synchronize()
    return st


# --------------------------------------------------------------------- run --

def _p(t):
    return C.c_void_p(t.data_ptr())


def _results(out):
    res = [r for r, *_ in out]
    d = {f: np.array([getattr(r, f) for r in res], np.int64)
         for f in ("status", "new_energy", "outer_iterations", "flips", "pre_flips")}
    return d


def _dense(probs, curves):
    """(energies, log g) curves on the full range [-2N, 2N] of each problem, and which energies they have."""
    N = np.array([p.X * p.Y for p in probs])
    at = np.cumsum(4 * N + 1) - (4 * N + 1) + 2 * N
    where = np.repeat(at, [len(E) for E, _ in curves]) + np.concatenate([E for E, _ in curves])
    d = {"energies": np.zeros(int((4 * N + 1).sum()), np.uint8), "log_g": np.zeros(int((4 * N + 1).sum()))}
    d["energies"][where] = 1
    d["log_g"][where] = np.concatenate([G for _, G in curves])
    return d


def _run_solve(st):
    ctx, probs, api = st["ctx"], st["probs"], st["case"]["api"]
    if api == "raw":
        out = ctx.solve_raw(probs)
        d = _results(out)
        d["start"] = np.concatenate([o[1] for o in out])
        d["end"] = np.concatenate([o[2] for o in out])
        parts = np.concatenate([w for o in out for w in o[3]] or [np.zeros(0)])
        d["log_g"] = np.zeros(sum(_raw_size(p) for p in probs))
        d["log_g"][:len(parts)] = parts
        return d
    out = ctx.solve(probs, st.get("couplings"))
    d = dict(_results(out), **_dense(probs, [(E, G) for _, E, G in out]))
    if api == "couplings":
        ok = all(len(E) for _, E, _ in out)  # a class that met an energy its pre-run had missed has no curve
        d["log_z"], d["log_probs"] = (wlg.class_log_probs([(E, G) for _, E, G in out], probs[0].prob) if ok
                                      else (np.zeros(len(out)), np.zeros(len(out))))
    return d


def _run_serve(st):
    srv, probs = st["server"], st["probs"]
    ids = srv.submit(probs)
    got = srv.wait(ids, 120)
    ds = [got[i] for i in ids]
    return {"status": np.array([d.status for d in ds]), "readmissions": np.array([d.readmissions for d in ds]),
            "outer_iterations": np.array([list(d.outer_iterations) for d in ds]),
            "log_z": np.array([list(d.log_z) for d in ds]), "log_probs": np.array([list(d.log_probs) for d in ds])}


def _run_setup(st):
    q, R, N, T, B = st["q"], st["R"], st["N"], st["T"], st["B"]
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for k in ("H", "off", "found_lat", "flag"):
        st[k].zero_()
    wlg.call("wlg_init_interactions", _p(st["J"]), N, R, q.seed, q.prob, s)
    wlg.call("wlg_apply_error_class", _p(st["J"]), q.X, q.Y, R, q.error_class, s)
    wlg.call("wlg_init_lattice", _p(st["lat"]), q.X, q.Y, T, q.seed, q.pre_walkers, s)
    wlg.call("wlg_calc_energy", q.boundary, _p(st["E"]), _p(st["lat"]), _p(st["J"]), _p(st["off_lat"]), q.X, q.Y, T,
             q.pre_walkers, s)
    # coarse bins of [-2N, 2N] with overlap 1: the length every bin has
    wlg.call("wlg_wang_landau_pre_run", _p(st["E"]), _p(st["flag"]), _p(st["lat"]), _p(st["found_lat"]), _p(st["H"]),
             _p(st["off"]), _p(st["J"]), _p(st["off_lat"]), -2 * N, 2 * N, q.pre_iterations, q.X, q.Y, q.seed, B,
             int((4 * N + 1) / B), T, q.pre_walkers, q.boundary, s)
    wlg.call("wlg_calc_energy", q.boundary, _p(st["found_E"]), _p(st["found_lat"]), _p(st["J"]), _p(st["off_found"]),
             q.X, q.Y, R * B, B, s)
    return {k: st[k] for k in ("J", "lat", "E", "H", "off", "found_lat", "flag", "found_E")}


def _run_iterate(case, d):
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    X, Y, R, I, W, T, seed, bc = (d[k] for k in ("X", "Y", "R", "I", "W", "T", "seed", "boundary"))
    p = lambda *names: [_p(d[n]) for n in names]
    hist = p("off_hist", "end", "start", "spectrum", "off_spec", "cond_sample")
    wlg.call("wlg_wang_landau", *p("lattice", "J", "H", "logG", "factor", "E", "newE", "off_iter", "found", "start",
                                   "end", "off_hist", "off_lat", "cond", "spectrum", "off_spec", "cond_sample"),
             X, Y, case["iterations"], T, I, I * W, seed, bc, s)
    wlg.call("wlg_check_histogram", *p("H", "factor", "cond"), *hist, case["alpha"], T, I * W, I, s)
    wlg.call("wlg_average_log_g", *p("logG", "start", "end", "spectrum", "off_spec", "cond", "off_hist",
                                     "cond_sample"), R, W, I, s)
    wlg.call("wlg_reset_cond", *p("cond", "factor"), R * I, case["beta"], W, s)
    wlg.call("wlg_check_finished", *p("cond_sample", "cond"), I, R, s)
    for even in (1, 0):
        wlg.call("wlg_replica_exchange", *p("off_lat", "E", "perm", "off_iter", "start", "end", "off_hist",
                                            "cond_sample", "logG"), even, seed, I, I * W, R * I, 0, s)
    return {k: d[k] for k in _ITERATE_OUT}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        return _run_solve(state)
    if kind == "prerun":
        return dict(zip(("seen", "couplings", "found", "found_energy", "lattices"),
                        _prerun(state["ctx"], state["probs"])))
    if kind == "serve":
        return _run_serve(state)
    if kind == "setup":
        return _run_setup(state)
    if kind == "iterate":
        return _run_iterate(case, state["dev"])
    out, _ = wlg.solve_plain(state["probs"])
    return dict(_results(out), **_dense(state["probs"], [(E, G) for _, E, G in out]))


# -------------------------------------------------------------------- work --

# operations of one Monte Carlo move that no form can do without: two draws of Philox4x32-10 (half a
# block of ten rounds: 4 multiplies' halves and 4 xors each), site, energy change of four bonds,
# acceptance (log, difference, comparison), and the updates of histogram and log g
_OPS_PER_MOVE = 60


def work(case):
    n = ((case["x0"] + case["x1"]) / 2) ** 2
    R = case["problems"]
    pre = R * case["pre_walkers"] * (case["pre_iterations"] or case["pre_per_site"] * n)
    I = case["intervals"] or min(32, max(8, int(n) // 8))
    # a window's first iterations converge in a few tens of sweeps per halving of ln f
    outer = case["max_outer"] or 25 * math.log2(1 / case["beta"])
    main = R * I * case["walkers"] * case["iterations"] * outer
    kind = case["kind"]
    if kind == "prerun":
        moves, data = pre, R * (4 * n + 1 + 2 * n + case["pre_intervals"] * (n + 8))
    elif kind == "setup":
        moves, data = pre, R * (2 * n + case["pre_walkers"] * (n + 12) + 8 * (4 * n + 1) + case["pre_intervals"] * n)
    elif kind == "iterate":
        moves = R * I * case["walkers"] * case["iterations"]
        length = 4 * n / (1 + case["overlap"] * (I - 1))
        data = R * I * case["walkers"] * (2 * n + 2 * 16 * length + 40)
    elif kind == "serve":
        moves, data = 4 * (pre + main), 4 * R * 200
    else:
        moves, data = pre + main, R * (144 + 12 * 4 * n)
    return {"bytes": int(data), "flops": int(moves * _OPS_PER_MOVE)}


# ------------------------------------------------------------------- exact --

def _philox(key, sub, pos):
    """32-bit draws `pos` of subsequences `sub` under `key`: Philox4x32-10 (Salmon et al., SC'11)."""
    key, sub, pos = np.broadcast_arrays(*(np.asarray(a, np.uint64) for a in (key, sub, pos)))
    M, S = np.uint64(0xFFFFFFFF), np.uint64(32)
    blk = pos >> np.uint64(2)
    c0, c1, c2, c3 = blk & M, blk >> S, sub & M, sub >> S
    k0, k1 = key & M, key >> S
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c0, np.uint64(0xCD9E8D57) * c2
        c0, c1, c2, c3 = (b >> S) ^ c1 ^ k0, b & M, (a >> S) ^ c3 ^ k1, a & M
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & M, (k1 + np.uint64(0xBB67AE85)) & M
    w = pos & np.uint64(3)
    return np.where(w == 0, c0, np.where(w == 1, c1, np.where(w == 2, c2, c3)))


def _uniform(key, sub, pos):
    """The draw as a float in (0, 1], widened to double."""
    x = _philox(key, sub, pos).astype(np.float32)
    return (x * np.float32(2.0 ** -32) + np.float32(2.0 ** -33)).astype(np.float64)


def _chain(J, X, Y, cls):
    J = J.copy()
    N = X * Y
    if cls in "hc":
        J[N:N + Y] *= -1
    if cls in "vc":
        J[np.arange(X) * Y] *= -1
    return J


def _energies(lat, J, X, Y, boundary):
    """Energies of lattices [T, N] under couplings [T, 2N]."""
    T = len(lat)
    s = lat.reshape(T, X, Y).astype(np.int32)
    Jr, Jd = J[:, :X * Y].reshape(T, X, Y), J[:, X * Y:].reshape(T, X, Y)
    h, v = s * np.roll(s, -1, 2) * Jr, s * np.roll(s, -1, 1) * Jd
    if boundary:
        h, v = h[:, :, :-1], v[:, :-1]
    return (-(h.sum((1, 2)) + v.sum((1, 2)))).astype(np.int32)


def _log_dos(X, Y, boundary, J):
    """Energies and log of the number of states of every reachable energy, by adding one spin at a
    time to a front of Y spins, for each first row."""
    N = X * Y
    M = 1 << Y
    spin = 1 - 2 * ((np.arange(M)[:, None] >> np.arange(Y)) & 1)
    cnt = np.zeros((M, M, 4 * N + 1))  # [first row][front][E + 2N]
    last = Y - 1 if boundary else Y
    e0 = -sum(J[j] * spin[:, j] * spin[:, (j + 1) % Y] for j in range(last))
    cnt[np.arange(M), np.arange(M), e0 + 2 * N] = 1
    for i in range(1, X):
        wrap = i == X - 1 and not boundary
        for j in range(Y):
            new = np.zeros_like(cnt)
            for c in range(M):
                for s in (0, 1):
                    d = (c & ~(1 << j)) | (s << j)
                    v = 1 - 2 * s
                    e = -J[N + (i - 1) * Y + j] * v * spin[c, j]
                    if j > 0:
                        e -= J[i * Y + j - 1] * v * spin[d, j - 1]
                    if j == Y - 1 and not boundary:
                        e -= J[i * Y + j] * v * spin[d, 0]
                    if wrap:
                        for up in (0, 1):
                            rows = ((np.arange(M) >> j) & 1) == up
                            new[rows, d] += np.roll(cnt[rows, c], e - J[N + i * Y + j] * v * (1 - 2 * up), axis=1)
                    else:
                        new[:, d] += np.roll(cnt[:, c], e, axis=1)
            cnt = new
    total = cnt.sum((0, 1))
    e = np.nonzero(total)[0]
    return e - 2 * N, np.log(total[e])


def _exact_solve(case, seed):
    """The true density of states, which the walk estimates (same layout as run's)."""
    out = dict.fromkeys(["status", "new_energy", "outer_iterations", "flips", "pre_flips", "energies", "log_g"])
    probs = _problems(case, seed)
    if case["api"] == "raw" or len(probs) > 4 or max(min(p.X, p.Y) for p in probs) > 6 or probs[0].Y > 6:
        return None
    curves = []
    for p in probs:
        N = p.X * p.Y
        if case["api"] == "couplings":
            J = _pattern(case, seed)
        else:
            u = _uniform(p.seed + p.sample, 0, np.arange(2 * N))
            J = np.where(u < p.prob, -1, 1).astype(np.int8)
        curves.append(_log_dos(p.X, p.Y, p.boundary, _chain(J, p.X, p.Y, p.error_class.decode()).astype(np.int64)))
    out["log_g"] = _dense(probs, curves)["log_g"]
    if case["api"] == "couplings":
        b = 0.5 * math.log((1 - probs[0].prob) / probs[0].prob)
        z = np.array([np.logaddexp.reduce(g - b * e) for e, g in curves])
        out["log_z"], out["log_probs"] = z, z - np.logaddexp.reduce(z)
    return out


def _exact_iterate(case, seed):
    """One outer iteration replayed walker by walker with the same draws, log g in 64 bits."""
    a = _iterate_arrays(case, seed)
    X, Y, N, I, W, T, bc = (a[k] for k in ("X", "Y", "N", "I", "W", "T", "boundary"))
    if T * case["iterations"] > 2_000_000:
        return None
    t = np.arange(T)
    b, k = t // W, t // (I * W)
    key = np.uint64(a["seed"]) + k.astype(np.uint64)
    sub = (t % (I * W)).astype(np.uint64)
    s = a["lattice"].reshape(T, N).astype(np.int64).copy()
    J = a["J"].reshape(-1, 2 * N).astype(np.int64)
    lo, hi = a["start"][b], a["end"][b]
    e_first, e_last = a["start"].reshape(-1, I)[k, 0], a["end"].reshape(-1, I)[k, -1]
    H, G, E = a["H"].copy(), a["logG"].copy(), a["E"].astype(np.int64)
    pos, go = np.zeros(T, np.int64), np.ones(T, bool)
    found = np.zeros(T, np.int64)
    frozen, lnf, base = a["cond"][b] != 0, np.log(a["factor"]), a["off_hist"] - lo
    for _ in range(case["iterations"]):
        site = np.trunc(_uniform(key, sub, pos) * (N - 1 + 0.999999)).astype(np.int64)
        i, j = site // Y, site % Y
        im, ip, jm, jp = (i - 1) % X, (i + 1) % X, (j - 1) % Y, (j + 1) % Y
        up, left = s[t, im * Y + j] * J[k, N + im * Y + j], s[t, i * Y + jm] * J[k, i * Y + jm]
        down, right = s[t, ip * Y + j] * J[k, N + i * Y + j], s[t, i * Y + jp] * J[k, i * Y + j]
        if bc:
            up, down = np.where(i == 0, 0, up), np.where(i == X - 1, 0, down)
            left, right = np.where(j == 0, 0, left), np.where(j == Y - 1, 0, right)
        En = E + 2 * s[t, site] * (up + down + left + right)
        ranged = (En >= e_first) & (En <= e_last)
        seen = ranged & (a["spectrum"][a["off_spec"][k] + np.where(ranged, En - e_first, 0)] == 1)
        pos += go
        bad = go & ~seen
        found[bad] = t[bad] + 1
        go = go & seen
        inside = go & (En >= lo) & (En <= hi)
        with np.errstate(over="ignore"):
            prob = np.minimum(1.0, np.exp(G[base + E] - G[np.where(inside, base + En, 0)]))
        acc = inside & (_uniform(key, sub, pos) < prob)
        pos += inside
        s[t[acc], site[acc]] *= -1
        E = np.where(acc, En, E)
        upd = go & ~frozen
        H[(base + E)[upd]] += 1
        G[(base + E)[upd]] += lnf[upd]
    cond, factor = a["cond"].copy(), a["factor"].copy()
    on = lambda w: a["spectrum"][a["off_spec"][w // I] + a["start"][w] - a["start"][w // I * I] +
                                 np.arange(a["end"][w] - a["start"][w] + 1)] == 1
    for w in range(len(cond)):
        n = a["end"][w] - a["start"][w] + 1
        at = [slice(a["off_hist"][w * W + v], a["off_hist"][w * W + v] + n) for v in range(W)]
        m = on(w)
        if cond[w] == 0 and m.any() and all(H[q][m].min() >= case["alpha"] * (H[q][m].sum() / m.sum()) for q in at):
            for q in at:
                H[q] = 0
            factor[w * W:(w + 1) * W] = np.sqrt(factor[w * W:(w + 1) * W])
            cond[w] = 1
        if cond[w] == 1:
            avg = np.zeros(n)
            for q in at:
                avg = avg + G[q] / W
            for q in at:
                G[q] = np.where(m, avg, 0.0)
    out = dict.fromkeys(_ITERATE_OUT)
    out["logG"], out["factor"] = G, factor
    return out


def exact(case, seed):
    """Computed numbers in 64 bits without this repository's code: the true density of states of
    small solves, the operators' log g replayed.  Longer walks, and outputs that are whole numbers,
    have no such value within seconds."""
    if case["kind"] == "solve":
        return _exact_solve(case, seed)
    if case["kind"] == "iterate":
        return _exact_iterate(case, seed)
    return None
