"""wlg_solve_raw_noalloc on a batch of many launch groups that each keep log g in global
memory: what the arena admits by the problems' parameters runs, however many groups it
makes.  Collected among the last on purpose (file name)."""
import pytest

from tests.test_zz_no_alloc import _compare

pytestmark = pytest.mark.gpu

# X, Y, boundary: (windows, walkers of each, overlap) whose log g and histogram leave shared
# memory, each of another team size or lattice storage; 58 teams of 100 to 200 KB
GROUPS = {
    (8, 8, 1): [(1, 128, 0.25), (2, 96, 0.3), (2, 112, 0.5), (5, 57, 0.25), (4, 80, 0.4), (6, 58, 0.3),
                 (5, 83, 0.5), (9, 49, 0.3), (7, 68, 0.4), (6, 85, 0.5), (11, 49, 0.3), (8, 80, 0.5),
                 (11, 61, 0.5), (10, 73, 0.5), (13, 59, 0.5), (13, 61, 0.5)],
    (8, 8, 0): [(2, 192, 0.4), (4, 144, 0.4), (7, 100, 0.3), (6, 138, 0.5), (9, 96, 0.4), (9, 99, 0.4),
                 (7, 132, 0.5), (7, 137, 0.5), (7, 141, 0.5), (7, 146, 0.5)],
    (2, 32, 1): [(1, 160, 0.25), (2, 96, 0.25), (2, 128, 0.5), (5, 64, 0.25), (5, 70, 0.3), (4, 104, 0.5),
                 (9, 49, 0.25), (5, 96, 0.5), (9, 56, 0.3), (6, 90, 0.5), (10, 57, 0.3), (12, 50, 0.25),
                 (8, 84, 0.5), (9, 78, 0.5), (11, 66, 0.4), (12, 64, 0.4), (12, 66, 0.4), (10, 86, 0.5),
                 (10, 89, 0.5), (15, 59, 0.4), (14, 68, 0.5), (15, 66, 0.4), (15, 68, 0.4)],
    (2, 30, 1): [(2, 112, 0.25), (3, 96, 0.3), (4, 96, 0.4), (8, 80, 0.4), (12, 69, 0.4), (15, 57, 0.4),
                 (14, 66, 0.5), (15, 61, 0.4), (15, 64, 0.4)],
}


def test_noalloc_many_groups_with_log_g_in_global_memory(cuda):
    import qec_pf_wang_landau_gb300 as wlg
    probs = [wlg.problem(X, Y, boundary=boundary, prob=0.1, error_class="i", seed=5, pre_walkers=128, pre_intervals=64,
                         pre_iterations=100 * X * Y, intervals=I, walkers_per_interval=W, overlap=overlap,
                         iterations=40, exchange_every=1, max_outer=2)
             for (X, Y, boundary), shapes in GROUPS.items() for I, W, overlap in shapes]
    # one-warp problems, whose stored lattices take 41 KB each: none of the others is spread over a cluster
    probs += [wlg.problem(12, 12, prob=0.04, seed=12345, sample=k, pre_intervals=288, pre_iterations=2000, iterations=100,
                          max_outer=2) for k in range(100)]
    ctx = wlg.Context(0)
    ctx.solve_raw(probs)
    assert ctx.stats()["main_forms"] == 1 << 0 | 1 << 3 and ctx.stats()["kernel_launches"] >= 55
    _compare(wlg, probs)
    _compare(wlg, probs)
