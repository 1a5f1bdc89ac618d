"""The copy threads that large transfers and fields of 1 to 64 MB share
(csrc/copy_pool.h, csrc/transfer.cu): callers in several threads, each with a
handle of its own, get their own bytes."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ is not available")
    exe = str(tmp_path_factory.mktemp("pool") / "copy_pool_host_check")
    subprocess.run([gxx, "-std=c++17", "-O2", "-pthread", "-ldl", "-I" + os.path.join(ROOT, "lambrex_gb300", "csrc"),
                    os.path.join(HERE, "copy_pool_host_check.cpp"), "-o", exe], check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("threads", [1, 2, 12])
def test_two_callers_at_once(harness, threads):
    out = subprocess.run([harness, str(threads), "60"], check=True, capture_output=True, text=True, timeout=300)
    assert out.stdout.split() == ["0", "0"]


@pytest.mark.parametrize("given", [0, 1, 5])
def test_fewer_threads_than_asked_for(harness, given):
    """The pool goes on with the threads that the system gives."""
    out = subprocess.run([harness, "12", "20", str(given)], check=True, capture_output=True, text=True, timeout=300)
    assert out.stdout.split() == ["0", "0"]


READERS = """
import mmap, sys, threading
import numpy as np
from lambrex_gb300 import lbx
lbx.lambrexInit()
wrong = []
def read(n, rounds):
    rng = np.random.default_rng(n)
    rho = rng.uniform(0.9, 1.1, (n, n, n))
    s = lbx.AmrSim(n, n, n, 0, [1, 1, 1], 0.8, 0.8, precision="f32s")
    s.SetInitialDensity(rho.ravel())
    s.SetInitialVelocity(0.0)
    s.InitFromScratch(0.0)
    s.CalcHydroVars(0)
    for _ in range(rounds):
        new = mmap.mmap(-1, 8 * n ** 3)  # pages still to be made: staged
        got = s.density_field(0, out=np.frombuffer(new, dtype=np.float64).reshape(n, n, n))
        # FAB order is the C order's transpose; the FP32 store holds 1e-7 of a fluctuation
        if not np.allclose(got.reshape(n, n, n), rho.transpose(2, 1, 0), rtol=0, atol=1e-6):
            wrong.append(n)
t = [threading.Thread(target=read, args=a) for a in ((208, 30), (80, 400), (100, 200))]
for x in t: x.start()
for x in t: x.join()
sys.exit(len(wrong))
"""


@pytest.mark.gpu
def test_fields_read_in_several_threads(gpu_lib):
    """Fields of 72, 4.1 and 8 MB, the first by the copy-engine path whatever
    the host's page tables offer."""
    env = dict(os.environ, LBX_HOST_ACCESS="copy", PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", READERS], env=env, cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
