"""What the autotuner times is the launch that its entry names: a team of all windows on
one CTA, also where a solve of the same problem would spread them over a cluster."""
import pytest

pytestmark = pytest.mark.gpu


def test_autotune_times_the_unspread_team(cuda):
    import qec_pf_wang_landau_gb300 as wlg
    # four CTAs of 192 walkers in a solve, one of 768 in the entry: three to four times the time
    p = wlg.problem(16, 16, prob=0.10, error_class="c", seed=4242, pre_walkers=128, pre_intervals=128,
                    pre_iterations=25600, intervals=64, walkers_per_interval=12, overlap=0.3, beta=1e-8,
                    iterations=400, exchange_every=20, max_outer=4)
    ctx = wlg.Context(0)
    ctx.solve_raw([p])
    ctx.solve_raw([p])
    spread_ms = ctx.stats()["main_ms"]
    ctx.autotune([p], max_outer=4)
    t, = ctx.autotune([p], max_outer=4)
    assert (t["form"], t["team"], t["per_cta"], t["candidates"]) == (3, 768, 1, 1)
    assert t["main_ms"] > 1.5 * spread_ms
    ctx.solve_raw([p])  # solves stay spread
    assert ctx.stats()["main_ms"] < 1.3 * spread_ms
