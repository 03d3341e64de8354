"""Contexts with a device memory budget: a batch whose pool of log g takes what the
budget leaves does not keep it from the next batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def equal(a, b):
    return len(a) == len(b) and all(
        r.status == q.status and r.outer_iterations == q.outer_iterations and len(w) == len(v)
        and all(np.array_equal(x, y) for x, y in zip(w, v)) for (r, _, _, w), (q, _, _, v) in zip(a, b))


def test_pool_of_one_solve_leaves_room_for_the_next(cuda):
    import qec_pf_wang_landau_gb300 as wlg
    # 160 teams whose log g lies in global memory: 147 KB each, of 8 bytes a bin and walker
    wide = [wlg.problem(16, 16, prob=0.04, seed=12345, sample=k, pre_iterations=2000, intervals=1,
                        walkers_per_interval=96, iterations=50, max_outer=2) for k in range(160)]
    many = [wlg.problem(6, 6, prob=0.04, error_class=c, seed=3, sample=k, iterations=50, max_outer=2)
            for k in range(400) for c in "ivhc"]
    free = wlg.Context(0)
    want = free.solve_raw(wide), free.solve_raw(many)
    ctx = wlg.Context(0, 32 << 20)
    for _ in range(2):
        assert equal(ctx.solve_raw(wide), want[0])
        assert ctx.stats()["main_forms"] == 1 << 3
        assert equal(ctx.solve_raw(many), want[1])
