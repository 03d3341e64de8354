"""The sweep operator against the oracle, array by array, at the edges of its
dispatch: warps with 1 to 32 walkers, rows of 16, 17 and 33 sites, one step, a
sweep longer than a part, log g from zero and far along, finished windows, and
arrays that only the walk on global memory takes."""
import numpy as np
import pytest

from tests.helpers import (Dev, assert_state_equal, copy_state, mainrun_state, o_check_histogram, o_exchange,
                           o_wang_landau, prerun_outputs)

pytestmark = pytest.mark.gpu

#  X, Y, boundary, R, I, W, overlap, prob, n_iter, sweeps, option
SWEEPS = [
    (4, 4, 0, 1, 1, 1, 0.25, 0.04, 300, 3, ""), (6, 6, 0, 2, 11, 3, 0.25, 0.08, 200, 3, ""),
    (6, 6, 1, 2, 8, 4, 0.25, 0.08, 1, 5, ""), (5, 16, 0, 2, 5, 7, 0.25, 0.10, 333, 3, ""),
    (5, 17, 1, 2, 5, 7, 0.25, 0.10, 333, 3, ""), (3, 32, 0, 1, 6, 6, 0.25, 0.10, 200, 3, ""),
    (3, 33, 0, 1, 6, 6, 0.25, 0.10, 200, 2, ""), (9, 9, 0, 1, 16, 8, 0.25, 0.10, 500, 3, "far"),
    (9, 9, 1, 2, 12, 5, 0.25, 0.10, 500, 3, "far"), (2, 2, 1, 1, 1, 40, 0.25, 0.0, 100, 3, ""),
    (6, 6, 0, 1, 40, 2, 0.05, 0.08, 200, 2, "narrow overlap"), (4, 4, 0, 1, 2, 2, 0.25, 0.04, 70001, 1, ""),
    (6, 6, 0, 1, 8, 4, 0.25, 0.08, 200, 2, "negative"), (6, 6, 0, 1, 8, 4, 0.25, 0.08, 200, 2, "factor"),
    (6, 6, 1, 2, 8, 5, 0.25, 0.08, 200, 2, "diluted"), (6, 6, 0, 2, 8, 5, 0.25, 0.08, 300, 2, "missed"),
]


@pytest.mark.parametrize("X,Y,boundary,R,I,W,overlap,prob,n_iter,sweeps,option", SWEEPS)
def test_sweep_operator_edges(cuda, X, Y, boundary, R, I, W, overlap, prob, n_iter, sweeps, option):
    seed = 12345
    pre = prerun_outputs(X, Y, boundary, prob, "i", seed, R, 128, min(48, X * Y), 100 * X * Y)
    st = mainrun_state(pre, I, W, overlap)
    rng = np.random.default_rng(3)
    T = R * I * W
    if option == "far":  # a run in progress: log g in the hundreds, small factors, every third window finished
        st["logG"][:] = 300.0 + 40.0 * rng.random(len(st["logG"]))
        st["H"][:] = rng.integers(0, 1 << 40, len(st["H"])).astype(np.uint64)
        st["factor"][:] = np.exp(2.0 ** -np.repeat(rng.integers(1, 40, R * I), W).astype(np.float64))
        st["cond"][::3] = 1
    if option == "negative":
        st["logG"][:] = -5.0 * rng.random(len(st["logG"]))
    if option == "factor":
        st["factor"][::7] = 0.9
    if option == "diluted":
        st["J"][::5] = 0
        st["spectrum"][:] = 1
    if option == "missed":  # energies taken out of the spectrum: walkers stop there
        on = np.nonzero(st["spectrum"])[0]
        st["spectrum"][on[len(on) // 3::len(on) // 3]] = 0
    dev = Dev(cuda, copy_state(st))
    for it in range(sweeps):
        o_wang_landau(st, n_iter, seed)
        dev.wang_landau(n_iter, seed)
        assert_state_equal(dev.snapshot(), st, f"sweep {it}")


# blocks of 8, 4 and 1 warps: up to 304, up to 608 and more blocks of 32 walkers
HELPERS = [(4, 4, 0, 61, 2, 80), (4, 4, 1, 61, 2, 74), (4, 4, 0, 122, 2, 80), (3, 4, 1, 122, 2, 77), (40, 3, 0, 3, 6, 9)]


@pytest.mark.parametrize("X,Y,boundary,R,I,W", HELPERS)
def test_sweep_operator_helpers(cuda, X, Y, boundary, R, I, W):
    seed = 777
    st = mainrun_state(prerun_outputs(X, Y, boundary, 0.06, "i", seed, R, 64, min(16, X * Y), 60 * X * Y), I, W, 0.25)
    dev = Dev(cuda, copy_state(st))
    for it in range(3):
        o_wang_landau(st, 40, seed)
        dev.wang_landau(40, seed)
        assert_state_equal(dev.snapshot(), st, f"sweep {it}")


@pytest.mark.parametrize("X,I,W", [(4, 3, 1), (6, 2, 16), (6, 4, 17), (4, 3, 33), (6, 1, 5), (4, 2, 1024)])
def test_flatness_and_exchange_edges(cuda, X, I, W):
    """One warp per walker up to 16, windows longer than a warp; permutations of 1 to 1024."""
    st = mainrun_state(prerun_outputs(X, X, 0, 0.08, "i", 5, 2, 64, 16, 60 * X * X), I, W, 0.6)
    rng = np.random.default_rng(I * W)
    st["H"][:] = rng.integers(900, 1000, len(st["H"])).astype(np.uint64)
    st["H"][len(st["H"]) // 2] = 100  # one window is not flat
    st["logG"][:] = 3.0 * rng.random(len(st["logG"]))
    dev = Dev(cuda, copy_state(st))
    o_check_histogram(st, 0.8)
    dev.check_histogram(0.8)
    assert_state_equal(dev.snapshot(), st, "flatness")
    assert st["cond"].any()
    for it in range(3):
        for even in (1, 0):
            o_exchange(st, even, 5)
            dev.exchange(even, 5)
            assert_state_equal(dev.snapshot(), st, f"exchange {it}")


# a thread or a warp per lattice; Philox blocks that end inside a lattice
@pytest.mark.parametrize("X,Y,nl,wpi", [(6, 8, 8192, 64), (6, 8, 8196, 4), (7, 7, 33, 3), (5, 9, 40, 8), (8, 16, 8200, 8),
                                        (1, 3, 7, 7), (3, 1, 5, 5), (1, 128, 3, 1), (64, 2, 129, 3)])
@pytest.mark.parametrize("boundary", [0, 1])
def test_set_up_operators_edges(cuda, X, Y, nl, wpi, boundary):
    import ctypes as C

    import qec_pf_wang_landau_gb300 as wlg
    import oracle as O
    R, N = (nl + wpi - 1) // wpi, X * Y
    p = lambda t: C.c_void_p(t.data_ptr())
    J = cuda.zeros(R * 2 * N, dtype=cuda.int8, device="cuda")
    lat = cuda.zeros(nl * N, dtype=cuda.int8, device="cuda")
    E = cuda.zeros(nl, dtype=cuda.int32, device="cuda")
    off = (np.arange(nl) * N).astype(np.int32)
    wlg.call("wlg_init_interactions", p(J), N, R, 11, C.c_float(0.2), None)
    wlg.call("wlg_init_lattice", p(lat), X, Y, nl, 11, wpi, None)
    wlg.call("wlg_calc_energy", boundary, p(E), p(lat), p(J), p(cuda.from_numpy(off).cuda()), X, Y, nl, wpi, None)
    h_J, h_lat = O.init_interactions(X, Y, R, 11, 0.2, "i"), O.init_lattice(X, Y, nl, 11, wpi)
    assert np.array_equal(J.cpu().numpy(), h_J)
    assert np.array_equal(lat.cpu().numpy(), h_lat)
    assert np.array_equal(E.cpu().numpy(), O.calc_energy(boundary, h_lat, h_J, off, X, Y, nl, wpi))
