"""The pre-run operator on a caller's histogram, against the oracle, array by array:
a walk that starts on counts, and one walk made in two calls.

The walk on bond words keeps two copies of the histogram, one entry per energy the
sample's lattices can have.  Where the sample's energies begin above E_min (an odd
number of -1 bonds on an odd lattice, or a range whose edge lies between them), the
range holds one energy fewer than the entries laid out for it; the sizes here are
those where that crosses a multiple of four entries, and neighbours where it does not."""
import ctypes as C

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

NAMES = ("E", "flags", "lat", "found", "H", "so", "J", "off")


def entries(first, last, e, step):
    """Entries laid out for the range, and those of energies that lie `step` apart through e."""
    bin0 = (e - first) % step
    return (last - first) // step + 1, (last - first - bin0) // step + 1


def padded(n):
    return (n + 4) // 4 * 4


#  X, Y, boundary, range (energies cut off the full one: below, above), crossing
RANGES = [
    (3, 5, 0, (0, 0), True), (5, 7, 0, (0, 0), True), (7, 9, 0, (0, 0), True), (9, 11, 0, (0, 0), True),
    (3, 21, 0, (0, 0), True), (5, 5, 0, (0, 0), False), (6, 6, 0, (0, 0), False), (6, 6, 0, (37, 47), True),
    (5, 17, 0, (80, 136), True), (6, 6, 1, (41, 41), True), (7, 5, 1, (39, 39), True), (4, 17, 1, (46, 108), True),
]


def sample(X, Y, boundary, cut, walkers, n_int, seed=4711, R=4):
    """Samples with even and odd numbers of -1 bonds, counts of every size, some bins found."""
    N = X * Y
    rng = np.random.default_rng([X, Y, boundary])
    J = np.where(rng.random((R, 2 * N)) < 0.2, -1, 1).astype(np.int8)
    for k in range(R):
        if (J[k] < 0).sum() % 2 != k % 2:
            J[k, 0] *= -1
    J = J.ravel().copy()
    T = R * walkers
    lat = O.init_lattice(X, Y, T, seed, walkers).copy()
    off = (np.arange(T) * N).astype(np.int32)
    E = O.calc_energy(boundary, lat, J, off, X, Y, T, walkers).astype(np.int32).copy()
    e_min, e_max = -2 * N + cut[0], 2 * N - cut[1]
    L = e_max - e_min + 1
    H = rng.integers(0, 40, R * L).astype(np.uint64)
    flags = (rng.random(R * n_int) < 0.2).astype(np.int32)
    return (dict(E=E, flags=flags, lat=lat, found=np.zeros(R * n_int * N, np.int8), H=H, so=np.zeros(T, np.uint64), J=J,
                 off=off), e_min, e_max, max(L // n_int, 1), T, seed)


@pytest.mark.parametrize("X,Y,boundary,cut,crossing", RANGES)
@pytest.mark.parametrize("calls", [(120,), (1, 2, 61)])
def test_pre_run_operator_continues_on_counts(cuda, X, Y, boundary, cut, crossing, calls):
    import qec_pf_wang_landau_gb300 as wlg
    walkers, n_int = 64, 12
    host, e_min, e_max, len_int, T, seed = sample(X, Y, boundary, cut, walkers, n_int)
    step = 4 if boundary == 0 else 2
    pairs = [entries(e_min, e_max, int(e), step) for e in host["E"][::walkers]]
    assert any(padded(a) != padded(b) for a, b in pairs) == crossing
    dev = {k: cuda.from_numpy(v.view(np.int64) if v.dtype == np.uint64 else v.copy()).clone().cuda()
           for k, v in host.items()}
    for n_iter in calls:
        wlg.call("wlg_wang_landau_pre_run", *(C.c_void_p(dev[k].data_ptr()) for k in NAMES), e_min, e_max, n_iter, X, Y,
                 seed, n_int, len_int, T, walkers, boundary, None)
    # the walk's draws do not depend on how it is divided into calls
    for n_iter in calls:
        O.lib().orc_wang_landau_pre_run(*(O.ptr(host[k]) for k in NAMES), e_min, e_max, n_iter, X, Y, seed, n_int,
                                        len_int, T, walkers, boundary)
    cuda.cuda.synchronize()
    for k, v in host.items():
        got = dev[k].cpu().numpy()
        assert np.array_equal(got.view(np.uint64) if v.dtype == np.uint64 else got, v), k
