"""The persistent main run against the oracle, bit for bit, at the edges of its
dispatch: lattice storages at their first and last row lengths, the tight layout
of each storage, sweeps shorter than a chunk of steps and longer than a part, and
factors down to where an addition of ln f is a few units in log g's last place."""
import numpy as np
import pytest

from tests.test_engine_gpu import big_problems, oracle_run

pytestmark = pytest.mark.gpu

#  X, Y, boundary, prob, cls, seed, R, pre_w, pre_i, pre_n, I, W, overlap, alpha, beta, n_iter, xc, xmode, gpar, outer
CASES = {
    # 65-site and longer lattices: rows of 2, 16 (bonds), 17, 32 (two-word bonds) and 33 sites (linear words)
    "bonds_40x2": (40, 2, 0, 0.10, "v", 11, 1, 64, 32, 8000, 6, 3, 0.25, 0.8, 1e-3, 300, 2, 1, 0, 6),
    "bonds_40x2_open": (40, 2, 1, 0.10, "h", 11, 1, 64, 32, 8000, 6, 3, 0.25, 0.8, 1e-3, 300, 2, 1, 0, 6),
    "bonds_5x16_open": (5, 16, 1, 0.10, "c", 12, 1, 64, 32, 8000, 6, 4, 0.25, 0.8, 1e-3, 300, 1, 1, 0, 6),
    "rows_5x17": (5, 17, 0, 0.10, "c", 13, 1, 64, 32, 8500, 6, 4, 0.25, 0.8, 1e-3, 300, 1, 1, 0, 6),
    "rows_5x17_open": (5, 17, 1, 0.10, "i", 13, 1, 64, 32, 8500, 6, 4, 0.25, 0.8, 1e-3, 300, 1, 1, 0, 6),
    "rows_3x32": (3, 32, 0, 0.10, "v", 14, 1, 64, 32, 9600, 6, 4, 0.25, 0.8, 1e-3, 300, 1, 1, 0, 6),
    "rows_24x24": (24, 24, 0, 0.10, "c", 28, 1, 128, 64, 57600, 64, 8, 0.3, 0.8, 1e-8, 60, 1, 1, 0, 2),
    "linear_3x33": (3, 33, 0, 0.10, "v", 15, 1, 64, 32, 9900, 6, 4, 0.25, 0.8, 1e-3, 300, 1, 1, 0, 6),
    # states whose guard bins and draw ring do not fit: 1024 walkers
    "tight_rows": (16, 16, 0, 0.10, "c", 4242, 1, 128, 128, 25600, 64, 12, 0.3, 0.8, 1e-8, 130, 1, 1, 0, 2),
    "tight_table": (8, 8, 1, 0.10, "v", 16, 1, 128, 64, 12800, 32, 32, 0.28, 0.8, 1e-3, 130, 1, 1, 0, 2),
    "tight_linear": (2, 40, 0, 0.10, "v", 17, 1, 128, 64, 16000, 32, 32, 0.15, 0.8, 1e-3, 130, 1, 1, 0, 2),
    # windows spread over clusters of 2, 4 and 8 CTAs, evenly and not, in every lattice storage;
    # exchange crosses CTAs, its draws come from the ring or (W = 16) not
    "cluster_table": (8, 8, 0, 0.10, "v", 21, 1, 128, 64, 6400, 11, 30, 0.28, 0.8, 1e-3, 200, 1, 1, 0, 8),
    "cluster_reg": (2, 30, 1, 0.10, "v", 22, 1, 128, 32, 9000, 10, 26, 0.28, 0.8, 1e-3, 200, 1, 1, 1, 8),
    "cluster_bonds": (12, 12, 1, 0.10, "c", 23, 1, 128, 64, 14400, 32, 16, 0.3, 0.8, 1e-3, 150, 1, 1, 0, 6),
    "cluster_rows": (20, 20, 0, 0.10, "h", 24, 1, 128, 128, 40000, 43, 12, 0.3, 0.8, 1e-3, 120, 2, 1, 0, 4),
    "cluster_linear": (3, 40, 0, 0.10, "i", 25, 1, 128, 64, 12000, 13, 20, 0.28, 0.8, 1e-3, 150, 1, 1, 0, 6),
    "cluster_8": (10, 10, 0, 0.10, "v", 26, 1, 128, 64, 10000, 30, 34, 0.28, 0.8, 1e-3, 100, 1, 1, 0, 4),
    "cluster_global": (20, 20, 0, 0.10, "v", 27, 1, 128, 64, 40000, 16, 16, 0.28, 0.8, 1e-3, 100, 1, 1, 0, 3),
    # one step, less than a chunk, a chunk and one step; more than a part
    "steps_1": (6, 6, 0, 0.04, "i", 18, 1, 128, 32, 2000, 4, 3, 0.25, 0.8, 1e-3, 1, 3, 1, 0, 200),
    "steps_7": (6, 6, 1, 0.04, "i", 18, 1, 128, 32, 2000, 4, 3, 0.25, 0.8, 1e-3, 7, 3, 1, 0, 60),
    "steps_9": (9, 9, 1, 0.04, "i", 18, 1, 128, 32, 8100, 4, 3, 0.25, 0.8, 1e-3, 9, 3, 1, 0, 60),
    "steps_70001": (4, 4, 0, 0.04, "i", 12345, 1, 32, 8, 2000, 4, 2, 0.25, 0.8, 1e-3, 70001, 1, 1, 0, 3),
    # ln f from 1 to 1e-9 within few steps: log g gains additions of every relative size
    "small_ln_f": (4, 4, 0, 0.10, "c", 7, 1, 32, 8, 2000, 4, 3, 0.25, 0.05, 1e-9, 200, 2, 1, 0, 400),
    "small_ln_f_open": (5, 4, 1, 0.10, "v", 9, 1, 64, 12, 2000, 4, 2, 0.25, 0.05, 1e-9, 300, 1, 1, 0, 400),
}


@pytest.mark.parametrize("name", CASES)
def test_main_run_edges_bit_exact(cuda, name):
    import qec_pf_wang_landau_gb300 as wlg
    cfg, outer = CASES[name][:-1], CASES[name][-1]
    I, W = cfg[10], cfg[11]
    ref = oracle_run(*cfg, max_outer=outer)
    (res, s, e, wins), = wlg.Context(0).solve_raw(big_problems(cfg, max_outer=outer))
    assert res.status in (wlg.WLG_OK, wlg.WLG_ERR_TIMEOUT) and res.outer_iterations == ref["outer"]
    assert res.flips == ref["flips"]
    assert np.array_equal(s, ref["start"][:I]) and np.array_equal(e, ref["end"][:I])
    for b in range(I):
        o = ref["off_hist"][b * W]
        want = ref["logG"][o:o + (e[b] - s[b] + 1)]
        assert np.array_equal(wins[b], want), f"window {b}: max |d| {np.abs(wins[b] - want).max()}"


@pytest.mark.parametrize("X,Y,boundary", [(5, 17, 0), (5, 17, 1), (4, 32, 0), (9, 9, 1), (3, 33, 0)])
def test_resumable_main_run_equals_the_uninterrupted_one(cuda, X, Y, boundary):
    """Under a time limit the main run saves its state every few iterations, and
    lattices stay in the saved form's storage: the same curves as without."""
    import ctypes as C
    import qec_pf_wang_landau_gb300 as wlg
    N = X * Y
    p = wlg.problem(X, Y, boundary=boundary, prob=0.08, error_class="v", seed=31, pre_walkers=64, pre_intervals=24,
                    pre_iterations=100 * N, intervals=6, walkers_per_interval=3, beta=0.3, iterations=400,
                    exchange_every=1)
    ctx = wlg.Context(0)
    (res, E, G), = ctx.solve([p])
    arr = (wlg.Problem * 1)(p)
    a = [np.zeros(4 * N + 1, np.uint8), np.zeros(2 * N, np.int8), np.zeros(24, np.int32), np.zeros(24, np.int32),
         np.zeros(24 * N, np.int8)]
    ptr = [x.ctypes.data_as(C.c_void_p) for x in a]
    wlg.call("wlg_prerun", ctx._h, C.cast(arr, C.c_void_p), 1, *ptr)
    r2, E2, G2 = (wlg.Result * 1)(), np.zeros(4 * N + 1, np.int32), np.zeros(4 * N + 1)
    wlg.call("wlg_mainrun", ctx._h, C.cast(arr, C.c_void_p), 1, *ptr, 600.0, C.cast(r2, C.c_void_p),
             E2.ctypes.data_as(C.c_void_p), G2.ctypes.data_as(C.c_void_p), len(E2))
    assert res.status == 0 and r2[0].status == 0 and r2[0].outer_iterations == res.outer_iterations
    n = r2[0].n_energies
    assert np.array_equal(E2[:n], E) and np.array_equal(G2[:n], G)
