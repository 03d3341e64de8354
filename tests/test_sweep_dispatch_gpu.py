"""The sweep operator over sweeps of 1 to 144 steps on the same arrays, against the
oracle: short ones walk on global memory, longer ones on packed walkers, with 8, 4 and
1 warps a block and with columns that leave room for one block on an SM."""
import pytest

from tests.helpers import Dev, assert_state_equal, copy_state, mainrun_state, o_wang_landau, prerun_outputs

pytestmark = pytest.mark.gpu

#  X, Y, boundary, R, I, W, overlap, bins stored by the pre-run
SHAPES = [(4, 4, 0, 1, 2, 3, 0.25, 16), (6, 6, 1, 3, 8, 4, 0.25, 36), (16, 16, 0, 2, 12, 6, 0.25, 64),
          (24, 24, 0, 1, 16, 4, 0.25, 96), (4, 17, 1, 2, 6, 6, 0.25, 48), (4, 4, 0, 320, 2, 17, 0.25, 16),
          (4, 4, 1, 640, 2, 16, 0.25, 16), (16, 16, 1, 60, 2, 81, 0.25, 32)]


@pytest.mark.parametrize("X,Y,boundary,R,I,W,overlap,bins", SHAPES)
def test_sweeps_short_and_long(cuda, X, Y, boundary, R, I, W, overlap, bins):
    seed = 991
    pre = prerun_outputs(X, Y, boundary, 0.06, "v", seed, R, 64, bins, (40 if R > 10 else 80) * X * Y)
    st = mainrun_state(pre, I, W, overlap)
    dev = Dev(cuda, copy_state(st))
    for n in (1, 2, 3, 5, 8, 13, 21, 34, 55, 89, 144):
        o_wang_landau(st, n, seed)
        dev.wang_landau(n, seed)
        assert_state_equal(dev.snapshot(), st, f"{n} steps")
