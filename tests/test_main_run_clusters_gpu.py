"""Problems whose windows could be spread over a cluster, against the oracle, bit for
bit: teams that the cluster kernel has no threads for, several clusters side by side,
and clusters that take one problem after another."""
import numpy as np
import pytest

from tests.test_engine_gpu import big_problems, oracle_run

pytestmark = pytest.mark.gpu


def assert_equals_oracle(out, ref, I, W):
    for k, (res, s, e, wins) in enumerate(out):
        assert res.status in (0, 7), (k, res.status)
        w = slice(k * I, (k + 1) * I)
        assert np.array_equal(s, ref["start"][w]) and np.array_equal(e, ref["end"][w])
        for b in range(I):
            o = ref["off_hist"][(k * I + b) * W]
            assert np.array_equal(wins[b], ref["logG"][o:o + (e[b] - s[b] + 1)]), (k, b)


#  X, Y, boundary, prob, cls, seed, R, pre_w, pre_i, pre_n, I, W, overlap, alpha, beta, n_iter, xc, xmode, gpar, outer
CASES = {
    # two or four ranks would hold more than 256 walkers each
    "wide_2": (4, 4, 0, 0.10, "c", 41, 1, 64, 16, 3200, 2, 512, 0.5, 0.8, 1e-3, 60, 1, 1, 0, 4),
    "wide_3": (6, 6, 0, 0.04, "v", 42, 1, 128, 32, 4000, 3, 130, 0.5, 0.8, 1e-3, 100, 1, 1, 0, 4),
    "wide_5": (6, 6, 0, 0.04, "v", 42, 1, 128, 32, 4000, 5, 130, 0.28, 0.8, 1e-3, 100, 1, 1, 0, 4),
    "wide_10": (6, 6, 0, 0.04, "h", 43, 1, 128, 32, 4000, 10, 90, 0.28, 0.8, 1e-3, 100, 1, 1, 0, 4),
    # 40 problems of 768 walkers: two ranks of 384 fit the SMs, four of 192 do not
    "forty_768": (16, 16, 0, 0.10, "c", 4242, 40, 128, 128, 12800, 64, 12, 0.3, 0.8, 1e-8, 40, 1, 1, 0, 2),
    # 30 clusters of four side by side
    "thirty_512": (12, 12, 0, 0.10, "i", 44, 30, 128, 64, 7200, 32, 16, 0.3, 0.8, 1e-3, 60, 1, 1, 0, 3),
}


@pytest.mark.parametrize("name", CASES)
def test_wide_teams_and_many_clusters(cuda, name):
    import qec_pf_wang_landau_gb300 as wlg
    cfg, outer = CASES[name][:-1], CASES[name][-1]
    ref = oracle_run(*cfg, max_outer=outer)
    assert_equals_oracle(wlg.Context(0).solve_raw(big_problems(cfg, max_outer=outer)), ref, cfg[10], cfg[11])


def test_clusters_take_one_problem_after_another(cuda):
    """log g in global memory, and a memory budget that holds it for ever fewer of the
    ten clusters that could run side by side."""
    import qec_pf_wang_landau_gb300 as wlg
    cfg = (12, 12, 1, 0.10, "v", 27, 10, 128, 64, 8640, 4, 64, 0.45, 0.8, 1e-3, 60, 1, 1, 0)
    ref = oracle_run(*cfg, max_outer=3)
    probs = big_problems(cfg, max_outer=3)
    budget, queued = 64 << 20, 0
    while True:
        ctx = wlg.Context(0, budget)
        try:
            out = ctx.solve_raw(probs)
        except wlg.WlgError as e:
            assert "budget" in str(e) and queued > 0
            break
        assert ctx.stats()["main_forms"] == 1 << 3
        assert_equals_oracle(out, ref, 4, 64)
        start, end = ctx.main_times()
        queued = int((start >= end.min()).sum())  # problems that began when another had ended
        budget = budget * 9 // 10
    assert queued >= 8  # the last budget held one or two clusters' log g
