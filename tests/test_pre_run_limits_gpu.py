"""The batched pre-run where its state just fits a CTA's shared memory, and where the
walk on bond words no longer does and the walk on int8 lattices takes over."""
import ctypes as C

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


# 64 x 2 with 28 warps of walkers: bond words of 232 384 to 232 864 bytes, beside 112 of the int8 walk's table
@pytest.mark.parametrize("n_int", [1, 2, 3, 4, 7, 8, 12, 13, 20, 64])
def test_bond_words_at_the_shared_memory_limit(cuda, n_int):
    import qec_pf_wang_landau_gb300 as wlg
    X, Y, walkers, n_iter = 64, 2, 896, 60
    N = X * Y
    p = wlg.problem(X, Y, prob=0.1, error_class="v", seed=8, pre_walkers=walkers, pre_intervals=n_int,
                    pre_iterations=n_iter)
    a, b = (dict(seen=np.zeros(4 * N + 1, np.uint8), J=np.zeros(2 * N, np.int8), flag=np.zeros(n_int, np.int32),
                 E=np.zeros(n_int, np.int32), lat=np.zeros(n_int * N, np.int8)) for _ in range(2))
    ctx = wlg.Context(0)
    wlg.call("wlg_prerun", ctx._h, C.byref(p), 1, *(a[k].ctypes.data_as(C.c_void_p) for k in ("seen", "J", "flag", "E", "lat")))
    O.lib().orc_prerun(X, Y, 0, C.c_float(0.1), b"v", 8, 1, walkers, n_int, n_iter,
                       *(O.ptr(b[k]) for k in ("seen", "J", "lat", "flag", "E")))
    b["E"] = np.where(b["flag"] != 0, b["E"], 0)
    for k, want in b.items():
        assert np.array_equal(a[k], want), k
