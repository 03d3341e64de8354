"""CPU test of the main run's dispatch (csrc/wlg_batch.h): which kernel a problem
gets, and how many CTAs of a cluster share its windows."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
STORES = ["linear", "reg", "table", "rows", "bonds", "bonds2", "bonds_open", "bonds2_open"]


def build_check(folder):
    """The dispatch as a program (tests/csrc/dispatch_check.cpp)."""
    cxx, nvcc = shutil.which("g++"), shutil.which("nvcc")
    home = os.path.dirname(os.path.dirname(os.path.realpath(nvcc))) if nvcc else "/usr/local/cuda"
    if cxx is None or not os.path.exists(os.path.join(home, "include", "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    exe = os.path.join(str(folder), "dispatch_check")
    subprocess.run([cxx, "-std=c++20", "-O2", "-pthread", "-I" + os.path.join(ROOT, "qec_pf_wang_landau_gb300", "csrc"),
                    "-I" + os.path.join(home, "include"), os.path.join(ROOT, "tests", "csrc", "dispatch_check.cpp"),
                    "-o", exe], check=True)
    return exe


def dispatch(exe, X, Y, boundary, lg, I, W, L, problems=1, sms=152, resumable=False):
    """(store, log g in global memory, tight, ranks, team) of a batch of such problems."""
    args = [X, Y, boundary, lg, I, W, L, problems, sms, int(resumable)]
    out = subprocess.run([exe] + [str(int(a)) for a in args], capture_output=True, text=True, check=True).stdout.split()
    return STORES[int(out[0])], out[1] == "1", out[2] == "1", int(out[3]), int(out[4])


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    return build_check(tmp_path_factory.mktemp("dispatch"))


def test_every_team_fits_its_kernel(check):
    out = subprocess.run([check], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr


@pytest.mark.parametrize("I,W,problems,ranks", [
    (2, 512, 1, 1), (3, 150, 1, 1), (5, 130, 1, 1), (10, 90, 1, 1),  # a rank's windows take more threads
    (64, 12, 40, 1), (64, 16, 40, 1), (64, 9, 60, 1),                 # two ranks would, four would not fit the SMs
    (64, 12, 1, 4), (64, 8, 38, 4), (64, 8, 39, 2), (64, 8, 77, 1), (30, 34, 1, 8), (11, 30, 1, 2),
])
def test_spread_of_windows_over_a_cluster(check, I, W, problems, ranks):
    _, _, _, got, team = dispatch(check, 16, 16, 0, 2, I, W, 6, problems)
    assert got == ranks and team >= I // ranks * W
