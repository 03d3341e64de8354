"""The flatness operator against the oracle at every number of lanes that a walker can
get (1 to 32, by walkers of a window and number of windows), with windows that are
flat, that fail in their first, last or only one walker, and finished ones."""
import numpy as np
import pytest

from tests.helpers import Dev, assert_state_equal, copy_state, mainrun_state, o_check_histogram, prerun_outputs

pytestmark = pytest.mark.gpu

#  R, I, W, overlap: 32 lanes; 8, 4, 2 and 1 by the block; two and three rounds of a block; 16, 8, 4, 2 and 1 by the windows
SIZES = [(2, 3, 3, 0.25), (1, 2, 16, 0.25), (1, 2, 33, 0.25), (1, 2, 100, 0.5), (1, 2, 250, 0.25), (1, 1, 300, 0.25),
         (1, 1, 513, 0.25), (1, 1, 1024, 0.25), (200, 4, 3, 0.25), (200, 4, 9, 0.25), (150, 4, 17, 0.4),
         (170, 4, 40, 0.25), (600, 4, 31, 0.25), (900, 3, 1, 0.25)]


@pytest.mark.parametrize("R,I,W,overlap", SIZES)
@pytest.mark.parametrize("boundary", [0, 1])
def test_flatness_lanes(cuda, R, I, W, overlap, boundary):
    st = mainrun_state(prerun_outputs(4, 4, boundary, 0.08, "i", 5, R, 32, 16, 600), I, W, overlap)
    rng = np.random.default_rng(R * I * W)
    st["H"][:] = rng.integers(900, 1000, len(st["H"])).astype(np.uint64)
    st["factor"][:] = np.exp(rng.random(len(st["factor"])))
    n = R * I
    for b in range(n):
        kind = b % 5 if n > 1 else 0
        walkers = {1: [0], 2: [W - 1], 3: [int(rng.integers(W))]}.get(kind, [])
        for w in walkers:
            o = st["off_hist"][b * W + w]
            on = np.nonzero(st["spectrum"][st["off_spec"][b // I] + st["start"][b] - st["start"][b // I * I]:][
                :st["end"][b] - st["start"][b] + 1] == 1)[0]
            st["H"][o + int(on[int(rng.integers(len(on)))])] = 300
        if kind == 4:
            st["cond"][b] = 1
    dev = Dev(cuda, copy_state(st))
    o_check_histogram(st, 0.8)
    dev.check_histogram(0.8)
    assert_state_equal(dev.snapshot(), st, "first")
    assert (st["cond"] == 1).sum() >= (n + 4) // 5
    o_check_histogram(st, 0.8)  # the windows left, and those reset
    dev.check_histogram(0.8)
    assert_state_equal(dev.snapshot(), st, "second")
