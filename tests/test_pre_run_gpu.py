"""The pre-run walk against the oracle, array by array, at the edges of its
dispatch: rows of 16 and 17, 32 and 33 sites, one walker to 1024, a walk that
starts in the middle of a block of draws, on an odd draw, on a histogram of
large counts, with bins already found, out of its range, with a missing bond."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

#  X, Y, boundary, walkers, n_int, n_iter, option
WALKS = [
    (2, 2, 0, 33, 4, 101, ""), (2, 2, 1, 32, 17, 100, ""), (5, 2, 0, 64, 9, 200, ""), (2, 9, 1, 40, 9, 201, ""),
    (5, 16, 0, 128, 32, 400, ""), (16, 16, 1, 96, 64, 300, ""), (4, 17, 1, 128, 24, 401, ""), (17, 32, 0, 64, 40, 300, ""),
    (3, 33, 0, 64, 24, 200, ""), (6, 6, 0, 1, 8, 500, ""), (6, 6, 0, 1024, 32, 60, ""), (20, 20, 0, 300, 32, 80, ""),
    (6, 6, 1, 100, 145, 200, ""), (6, 6, 0, 64, 32, 150, "half"), (6, 6, 0, 64, 32, 151, "mixed"),
    (6, 6, 1, 64, 32, 150, "odd"), (6, 6, 0, 64, 32, 150, "counts"), (6, 6, 0, 64, 32, 150, "more"),
    (6, 6, 0, 64, 32, 300, "found"), (6, 6, 1, 64, 12, 300, "range"), (6, 20, 0, 64, 12, 300, "range"),
    (6, 6, 1, 64, 32, 150, "diluted"), (6, 6, 0, 64, 32, 0, ""),
]


@pytest.mark.parametrize("X,Y,boundary,walkers,n_int,n_iter,option", WALKS)
def test_pre_run_operator_edges(cuda, X, Y, boundary, walkers, n_int, n_iter, option):
    import ctypes as C
    import qec_pf_wang_landau_gb300 as wlg
    torch = cuda
    N, R, seed = X * Y, 2, 321
    T = R * walkers
    rng = np.random.default_rng(5)
    J = O.init_interactions(X, Y, R, seed, 0.2, "c").copy()
    if option == "diluted":
        J[::7] = 0
    lat = O.init_lattice(X, Y, T, seed, walkers).copy()
    off = (np.arange(T) * N).astype(np.int32)
    E = O.calc_energy(boundary, lat, J, off, X, Y, T, walkers).astype(np.int32).copy()
    e_min, e_max = -2 * N, 2 * N
    if option == "range":
        e_min, e_max = int(E.min()) - 12, int(E.max()) + 16
        E[::11] = e_max + 4  # these never start
    L = e_max - e_min + 1
    len_int = max(L // n_int, 1)
    H = np.zeros(R * L, np.uint64)
    if option == "counts":
        H[:] = rng.integers(0, 9, R * L).astype(np.uint64) + np.uint64((1 << 31) - 1 - 9 - n_iter * walkers)
    if option == "more":
        H[:] = rng.integers(0, 9, R * L).astype(np.uint64) + np.uint64(1 << 31)
    so = np.zeros(T, np.uint64)
    if option == "half":
        so[:] = 6
    if option == "mixed":
        so[:] = 2 * rng.integers(0, 9, T).astype(np.uint64)
    if option == "odd":
        so[:] = rng.integers(0, 9, T).astype(np.uint64)
    flags = np.zeros(R * n_int, np.int32)
    if option == "found":
        flags[::3] = 1
    found = np.zeros(R * n_int * N, np.int8)
    host = dict(E=E, flags=flags, lat=lat, found=found, H=H, so=so, J=J, off=off)
    dev = {k: torch.from_numpy(v.view(np.int64) if v.dtype == np.uint64 else v.copy()).clone().cuda()
           for k, v in host.items()}
    p = lambda k: C.c_void_p(dev[k].data_ptr())
    wlg.call("wlg_wang_landau_pre_run", p("E"), p("flags"), p("lat"), p("found"), p("H"), p("so"), p("J"), p("off"),
             e_min, e_max, n_iter, X, Y, seed, n_int, len_int, T, walkers, boundary, None)
    O.lib().orc_wang_landau_pre_run(*(O.ptr(host[k]) for k in ("E", "flags", "lat", "found", "H", "so", "J", "off")),
                                    e_min, e_max, n_iter, X, Y, seed, n_int, len_int, T, walkers, boundary)
    torch.cuda.synchronize()
    for k, v in host.items():
        got = dev[k].cpu().numpy()
        assert np.array_equal(got.view(np.uint64) if v.dtype == np.uint64 else got, v), k


@pytest.mark.parametrize("X,Y,boundary,walkers,n_int,n_iter",
                         [(16, 16, 0, 128, 64, 700), (5, 16, 1, 33, 32, 701), (4, 17, 0, 128, 32, 700),
                          (9, 32, 1, 64, 32, 701), (3, 33, 0, 64, 32, 300), (6, 6, 0, 1024, 32, 50),
                          (2, 2, 1, 32, 8, 41), (20, 20, 0, 400, 64, 60), (6, 6, 1, 1, 72, 900)])
def test_batched_pre_run_edges(cuda, X, Y, boundary, walkers, n_int, n_iter):
    import ctypes as C
    import qec_pf_wang_landau_gb300 as wlg
    N, R = X * Y, 2
    out = []
    for f in (0, 1):
        a = dict(seen=np.zeros(R * (4 * N + 1), np.uint8), J=np.zeros(R * 2 * N, np.int8),
                 flag=np.zeros(R * n_int, np.int32), E=np.zeros(R * n_int, np.int32),
                 lat=np.zeros(R * n_int * N, np.int8))
        out.append(a)
    probs = [wlg.problem(X, Y, boundary=boundary, prob=0.15, error_class="c", seed=77, sample=k, pre_walkers=walkers,
                         pre_intervals=n_int, pre_iterations=n_iter) for k in range(R)]
    arr = (wlg.Problem * R)(*probs)
    ctx = wlg.Context(0)
    wlg.call("wlg_prerun", ctx._h, C.cast(arr, C.c_void_p), R,
             *(out[0][k].ctypes.data_as(C.c_void_p) for k in ("seen", "J", "flag", "E", "lat")))
    O.lib().orc_prerun(X, Y, boundary, C.c_float(0.15), b"c", 77, R, walkers, n_int, n_iter,
                       *(O.ptr(out[1][k]) for k in ("seen", "J", "lat", "flag", "E")))
    for k, want in out[1].items():
        if k == "E":
            want = np.where(out[1]["flag"] != 0, want, out[0]["E"] * 0)
        assert np.array_equal(out[0][k], want), k
