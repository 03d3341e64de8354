"""Entry points called by several host threads at once, with launches of different
amounts of shared memory: every call succeeds and gives what it gives alone."""
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_operators_from_several_threads(cuda, tmp_path):
    """Threads of a C++ program (tests/csrc/threads_check.cpp), as Python's take turns."""
    import qec_pf_wang_landau_gb300 as wlg
    nvcc = shutil.which("nvcc")
    if nvcc is None:
        pytest.skip("no compiler")
    wlg.lib()
    package = os.path.join(ROOT, "qec_pf_wang_landau_gb300")
    exe = str(tmp_path / "threads_check")
    subprocess.run([nvcc, "-std=c++20", "-O2", "-I" + os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "csrc", "threads_check.cpp"), "-o", exe, "-L" + package, "-lwlg",
                    "-lpthread", "-Xlinker", "-rpath," + package], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr


def test_solves_from_several_threads(cuda):
    """One context a thread, problems whose teams and pre-runs differ in shared memory."""
    import qec_pf_wang_landau_gb300 as wlg
    batches = [[wlg.problem(X, X, prob=0.08, error_class="v", seed=3, sample=k, pre_walkers=w, pre_iterations=60 * X * X,
                            intervals=I, walkers_per_interval=4, iterations=100, exchange_every=2, max_outer=3)
                for k in range(2)] for X, w, I in [(6, 128, 6), (12, 128, 12), (20, 256, 16), (16, 64, 24)]]
    want = [wlg.Context(0).solve_raw(b) for b in batches]
    contexts = [wlg.Context(0) for _ in batches]
    out, errors = [None] * len(batches), []
    gate = threading.Barrier(len(batches))

    def solves(i):
        try:
            gate.wait(60)
            for _ in range(40):
                out[i] = contexts[i].solve_raw(batches[i])
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=solves, args=(i,)) for i in range(len(batches))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors[0]
    for got, ref in zip(out, want):
        for (r, s, e, wins), (r0, s0, e0, wins0) in zip(got, ref):
            assert r.status == r0.status and np.array_equal(s, s0) and np.array_equal(e, e0)
            assert len(wins) == len(wins0) and all(np.array_equal(a, b) for a, b in zip(wins, wins0))
