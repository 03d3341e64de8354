"""The pre-run operator over calls of 1 to 400 rounds on the same arrays, against the
oracle: short ones walk on the caller's int8 lattices, longer ones on bond words.  And
arrays that bond words cannot take, in one lattice of many."""
import ctypes as C

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

NAMES = ("E", "flags", "lat", "found", "H", "so", "J", "off")


def arrays(X, Y, boundary, R, walkers, n_int, L, seed):
    N, T = X * Y, R * walkers
    J = O.init_interactions(X, Y, R, seed, 0.12, "h").copy()
    lat = O.init_lattice(X, Y, T, seed, walkers).copy()
    off = (np.arange(T) * N).astype(np.int32)
    E = O.calc_energy(boundary, lat, J, off, X, Y, T, walkers).astype(np.int32).copy()
    return dict(E=E, flags=np.zeros(R * n_int, np.int32), lat=lat, found=np.zeros(R * n_int * N, np.int8),
                H=np.zeros(R * L, np.uint64), so=np.zeros(T, np.uint64), J=J, off=off)


def compare(cuda, host, calls, e_min, e_max, X, Y, seed, n_int, len_int, walkers, boundary):
    import qec_pf_wang_landau_gb300 as wlg
    T = len(host["E"])
    dev = {k: cuda.from_numpy(v.view(np.int64) if v.dtype == np.uint64 else v.copy()).clone().cuda()
           for k, v in host.items()}
    for n_iter in calls:
        wlg.call("wlg_wang_landau_pre_run", *(C.c_void_p(dev[k].data_ptr()) for k in NAMES), e_min, e_max, n_iter, X, Y,
                 seed, n_int, len_int, T, walkers, boundary, None)
        O.lib().orc_wang_landau_pre_run(*(O.ptr(host[k]) for k in NAMES), e_min, e_max, n_iter, X, Y, seed, n_int,
                                        len_int, T, walkers, boundary)
        cuda.cuda.synchronize()
        for k, v in host.items():
            got = dev[k].cpu().numpy()
            assert np.array_equal(got.view(np.uint64) if v.dtype == np.uint64 else got, v), (n_iter, k)


@pytest.mark.parametrize("X,Y,boundary,R,walkers,calls", [
    (4, 4, 0, 2, 1, (1, 3, 4, 5, 6, 40)), (5, 7, 0, 3, 64, (2, 5, 10, 20, 80)), (9, 9, 1, 2, 128, (1, 10, 13, 14, 30, 120)),
    (16, 16, 0, 2, 128, (5, 30, 36, 40, 200)), (4, 17, 1, 2, 300, (1, 3, 9, 30, 100)), (6, 6, 0, 1, 1024, (1, 7, 9, 50)),
    (6, 6, 0, 400, 32, (2, 8, 30)), (24, 24, 0, 1, 600, (20, 90, 120, 300)),
])
def test_short_and_long_walks(cuda, X, Y, boundary, R, walkers, calls):
    N, n_int, seed = X * Y, 16, 77
    L = 4 * N + 1
    host = arrays(X, Y, boundary, R, walkers, n_int, L, seed)
    compare(cuda, host, calls, -2 * N, 2 * N, X, Y, seed, n_int, max(L // n_int, 1), walkers, boundary)


@pytest.mark.parametrize("walkers", [40, 290])
@pytest.mark.parametrize("where", [(0, 0), (33, 31), (-1, -1), (7, 32)])
def test_one_spin_that_is_not_one(cuda, walkers, where):
    """A spin of 3 in one walker's lattice sends its sample to int8 lattices."""
    X, Y, boundary, R, n_int, seed = 7, 9, 0, 2, 16, 78
    N = X * Y
    e_max = 2 * N + 24
    L = 2 * e_max + 1
    host = arrays(X, Y, boundary, R, walkers, n_int, L, seed)
    host["lat"].reshape(R, walkers, N)[1, where[0], where[1]] *= 3
    host["E"][:] = O.calc_energy(boundary, host["lat"], host["J"], host["off"], X, Y, R * walkers, walkers)
    compare(cuda, host, (60, 61), -e_max, e_max, X, Y, seed, n_int, L // n_int, walkers, boundary)
