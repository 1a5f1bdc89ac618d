"""Fields of 1 to 64 MB pass through page-locked buffers that the library keeps
(csrc/transfer.cu); they go with the context that holds them.  A program that
resets the device and starts over reads its fields all the same."""
import glob
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes, mmap, sys
import numpy as np
from lambrex_gb300 import lbx
def once(rho):
    lbx.lambrexInit()
    s = lbx.AmrSim(128, 128, 128, 0, [1, 1, 1], 0.8, 0.8)
    s.SetInitialDensity(rho)
    s.SetInitialVelocity(0.0)
    s.InitFromScratch(0.0)
    s.Iterate(3)
    s.CalcHydroVars(0)
    # 16 MB into pages still to be made: staged
    d = s.density_field(0, out=np.frombuffer(mmap.mmap(-1, 128 ** 3 * 8), dtype=np.float64).reshape(128, 128, 128))
    s.close()
    lbx.lambrexFinalise()
    assert abs(d - rho).max() <= 1e-12
once(1.25)
assert ctypes.CDLL(sys.argv[1]).cudaDeviceReset() == 0
once(1.5)
once(0.75)
"""


@pytest.mark.gpu
def test_fields_after_a_device_reset(gpu_lib):
    cudart = sorted(glob.glob("/usr/local/cuda/lib64/libcudart.so*"))
    if not cudart:
        pytest.skip("no shared CUDA runtime to reset the device with")
    r = subprocess.run([sys.executable, "-c", PROGRAM, cudart[0]], env=dict(os.environ, PYTHONPATH=ROOT),
                       cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
