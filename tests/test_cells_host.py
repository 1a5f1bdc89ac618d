"""The box kernels' thread number -> cell map (csrc/kernels.cuh): against the
quotients, for boxes below 2^31 cells (32-bit numbers) and from there on, which
the steps, the equilibrium and the fields on device pointers take (64-bit)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA_INCLUDE = "/usr/local/cuda/include"


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are not available")
    exe = str(tmp_path_factory.mktemp("cells") / "cells_host_check")
    subprocess.run([gxx, "-std=c++17", "-O2", "-I" + CUDA_INCLUDE,
                    "-I" + os.path.join(ROOT, "lambrex_gb300", "csrc"),
                    os.path.join(HERE, "cells_host_check.cpp"), "-o", exe], check=True, capture_output=True)
    return exe


DIMS = [(1, 1, 1), (10, 10, 50), (7, 1, 3), (512, 512, 512), (251, 190, 133), (2147483647, 1, 1),
        (1, 2147483647, 1), (1, 1, 2147483647), (1289, 1290, 1291), (1449, 1449, 1022),  # below 2^31 cells
        (1449, 1449, 1030), (2048, 1024, 1024), (65536, 65536, 2), (2147483647, 2, 1),
        (1 << 20, 1 << 20, 1), (3, 2147483647, 5), (1625, 1624, 1626)]


@pytest.mark.parametrize("dims", DIMS)
def test_cell_of_a_thread(harness, dims):
    nx, ny, nz = dims
    n = nx * ny * nz
    rng = np.random.default_rng(5)
    cells = sorted({0, n - 1, n // 2, max(n - nx, 0), max(n - nx * ny, 0), max(n - nx * ny - 1, 0)}
                   | {int(v) for v in rng.integers(0, n, 300)} | {c for c in (2 ** 31 - 1, 2 ** 31, 2 ** 32) if c < n})
    cells += range(n, -(-n // 32) * 32)  # threads of the last block without a cell
    out = subprocess.run([harness], input="".join("%d %d %d %d\n" % (nx, ny, nz, c) for c in cells),
                         check=True, capture_output=True, text=True).stdout.split("\n")
    for c, line in zip(cells, out):
        *got, threads = line.split()
        assert got == ([str(c % nx), str(c // nx % ny), str(c // (nx * ny))] if c < n else ["beyond"]), c
        # past 2^31 - 1 blocks the grid is one that a launch refuses
        assert n <= int(threads) < n + 128 if n <= 128 * (2 ** 31 - 1) else int(threads) >= 128 * 2 ** 31
