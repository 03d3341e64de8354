"""The main run's tight layout (no guard bins, the draw ring in local memory), bit for
bit against the oracle, in every lattice storage that has it.

A single problem of many walkers is spread over a cluster, whose teams are too small
for the layout; batches with more problems than SMs, windows of more walkers than a
cluster's CTA takes, and resumable runs keep a problem on one CTA.  The layout that
the dispatch chooses for the windows at hand is asserted."""
import ctypes as C

import numpy as np
import pytest

from tests.test_dispatch import build_check, dispatch
from tests.test_engine_gpu import big_problems, oracle_run
from tests.test_main_run_clusters_gpu import assert_equals_oracle

pytestmark = pytest.mark.gpu

#  copies, store, (X, Y, boundary, prob, cls, seed, R, pre_w, pre_i, pre_n, I, W, overlap, alpha, beta, n_iter, xc, xmode, gpar, outer)
CASES = {
    "rows": (160, "rows", (16, 16, 0, 0.10, "c", 4242, 1, 128, 128, 25600, 64, 12, 0.3, 0.8, 1e-8, 130, 1, 1, 0, 2)),
    "rows_17": (160, "rows", (4, 17, 1, 0.10, "c", 19, 1, 128, 64, 13600, 32, 32, 0.15, 0.8, 1e-3, 70, 1, 1, 0, 2)),
    "table": (160, "table", (8, 8, 1, 0.10, "v", 16, 1, 128, 64, 12800, 32, 32, 0.28, 0.8, 1e-3, 130, 1, 1, 0, 2)),
    "linear": (160, "linear", (2, 40, 0, 0.10, "v", 17, 1, 128, 64, 16000, 32, 32, 0.15, 0.8, 1e-3, 130, 1, 1, 0, 2)),
    "reg": (160, "reg", (2, 30, 1, 0.10, "v", 20, 1, 128, 64, 12000, 28, 36, 0.3, 0.8, 1e-3, 70, 1, 1, 0, 3)),
    # one problem of a single window, and of two with 512 walkers each
    "table_1": (1, "table", (3, 3, 1, 0.20, "i", 5, 1, 64, 8, 3600, 1, 1024, 0.25, 0.8, 1e-3, 200, 1, 1, 0, 6)),
    "reg_2": (1, "reg", (2, 7, 1, 0.20, "i", 6, 1, 64, 12, 4800, 2, 512, 0.4, 0.8, 1e-3, 200, 1, 1, 0, 6)),
}


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    return build_check(tmp_path_factory.mktemp("dispatch"))


def chosen(check, cfg, s, e, copies, resumable=False):
    """The dispatch of a problem whose windows are s..e."""
    X, Y, boundary, I, W = cfg[0], cfg[1], cfg[2], cfg[10], cfg[11]
    lg = 2 if boundary == 0 else 1
    L = max((int(b) - int(a)) // (1 << lg) + 1 for a, b in zip(s, e))
    # the first bin of a window may lie after its edge: both lengths must agree
    got = {dispatch(check, X, Y, boundary, lg, I, W, n, copies, resumable=resumable) for n in (L - 1, L)}
    return got.pop() if len(got) == 1 else (None,) * 5


@pytest.mark.parametrize("name", CASES)
def test_tight_layout_bit_exact(cuda, check, name):
    import qec_pf_wang_landau_gb300 as wlg
    copies, store, case = CASES[name]
    cfg, outer = case[:-1], case[-1]
    ref = oracle_run(*cfg, max_outer=outer)
    out = wlg.Context(0).solve_raw(big_problems(cfg, max_outer=outer) * copies)
    assert chosen(check, cfg, out[0][1], out[0][2], copies) == (store, True, True, 1, (cfg[10] * cfg[11] + 31) // 32 * 32)
    for q in out:
        assert_equals_oracle([q], ref, cfg[10], cfg[11])


@pytest.mark.parametrize("name", ["rows", "table", "linear"])
def test_resumable_tight_layout(cuda, check, name):
    """Under a time limit, against the same problem spread over a cluster."""
    import qec_pf_wang_landau_gb300 as wlg
    case = CASES[name][2]
    cfg, outer = case[:-1], 9  # three launches
    p, = big_problems(cfg, max_outer=outer)
    N, B = p.X * p.Y, p.pre_intervals
    ctx = wlg.Context(0)
    (res, E, G), = ctx.solve([p])
    (_, s, e, _), = ctx.solve_raw([p])
    assert chosen(check, cfg, s, e, 1)[3] > 1
    assert chosen(check, cfg, s, e, 1, resumable=True)[:4] == (CASES[name][1], True, True, 1)
    arr = (wlg.Problem * 1)(p)
    a = [np.zeros(4 * N + 1, np.uint8), np.zeros(2 * N, np.int8), np.zeros(B, np.int32), np.zeros(B, np.int32),
         np.zeros(B * N, np.int8)]
    ptr = [x.ctypes.data_as(C.c_void_p) for x in a]
    wlg.call("wlg_prerun", ctx._h, C.cast(arr, C.c_void_p), 1, *ptr)
    r2, E2, G2 = (wlg.Result * 1)(), np.zeros(4 * N + 1, np.int32), np.zeros(4 * N + 1)
    wlg.call("wlg_mainrun", ctx._h, C.cast(arr, C.c_void_p), 1, *ptr, 600.0, C.cast(r2, C.c_void_p),
             E2.ctypes.data_as(C.c_void_p), G2.ctypes.data_as(C.c_void_p), len(E2))
    n = r2[0].n_energies
    assert (r2[0].status, r2[0].outer_iterations, r2[0].flips) == (res.status, res.outer_iterations, res.flips)
    assert np.array_equal(E2[:n], E) and np.array_equal(G2[:n], G)
