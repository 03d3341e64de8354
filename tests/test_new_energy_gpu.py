"""The energy that a problem reports when its walkers meet ones that the pre-run never
saw: the last one found, by step, and of several in one step the lowest walker's."""
import numpy as np
import pytest

from tests.helpers import mainrun_state, o_wang_landau, prerun_outputs

pytestmark = pytest.mark.gpu

#  X, Y, boundary, seed, pre_n, I, W, n_iter: short pre-runs that miss energies
RUNS = [(3 + k % 6, 3 + k // 6 % 6, k // 36 % 2, 900 + k, (40, 80, 160)[k % 3], 1 + k % 4, (2, 4, 8)[k // 4 % 3],
         (1, 2, 3, 8)[k // 12 % 4]) for k in range(288)]


def found_first(st, n_iter, seed):
    """(step, energy) at which each walker stops."""
    seen = {}
    for step in range(n_iter):
        st["found"][:] = 0
        o_wang_landau(st, 1, seed)
        for t in np.nonzero(st["found"])[0]:
            seen.setdefault(int(t), (step, int(st["newE"][t])))
    return seen


@pytest.mark.parametrize("copies", [1, 4])
def test_reported_new_energy(cuda, copies):
    import qec_pf_wang_landau_gb300 as wlg
    probs, want, ties = [], [], 0
    for X, Y, boundary, seed, pre_n, I, W, n_iter in RUNS:
        try:
            st = mainrun_state(prerun_outputs(X, Y, boundary, 0.1, "i", seed, 1, 4, 16, pre_n), I, W, 0.25)
        except (StopIteration, ValueError, IndexError, RuntimeError):
            continue  # no start lattice in a window
        seen = found_first(st, n_iter, seed)
        if not seen:
            continue
        last = max(s for s, _ in seen.values())
        energies = [e for t, (s, e) in sorted(seen.items()) if s == last]
        ties += len(set(energies)) > 1
        want.append(energies[0])
        probs.append(wlg.problem(X, Y, boundary=boundary, prob=0.1, error_class="i", seed=seed, pre_walkers=4,
                                 pre_intervals=16, pre_iterations=pre_n, intervals=I, walkers_per_interval=W,
                                 overlap=0.25, iterations=n_iter, exchange_every=1, max_outer=1))
    assert len(want) > 40 and ties >= 5
    out = wlg.Context(0).solve_raw(probs * copies)
    assert [r.status for r, *_ in out] == [wlg.WLG_ERR_NEW_ENERGY] * len(out)
    assert [r.new_energy for r, *_ in out] == want * copies
