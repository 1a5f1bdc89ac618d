"""Fluid at rest on the levels of refined FP64 runs (csrc/fx64.cuh): cells that
are exactly uniform take a short form of the FP64 collision, which has the
general form's bits; without a density both are NaN."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_fx64 import CUDA_INCLUDE, HERE, ROOT

RATES = [(1.25, 0.9), (0.625, 0.45), (1.9, 1.6), (0.02, 1.98), (1.0, 1.0)]


def uniform(r, a, d):
    return np.array([r] + [a] * 6 + [d] * 8)


def rest_cells():
    """(cell, whether the short form takes it)"""
    rng = np.random.default_rng(4)
    w = uniform(2 / 9, 1 / 9, 1 / 72)
    out = [(w, True), (1.1 * w, True), (uniform(0.25, 0.125, 0.015625), True)]
    for _ in range(40):
        out.append((rng.uniform(0.5, 2) * uniform(*(np.array([2 / 9, 1 / 9, 1 / 72]) * rng.uniform(0.9, 1.1, 3))), True))
    for s in (2.0 ** -940, 1e-200, 1e-30, 1e30, 1e200, 2.0 ** 990):
        out.append((s * 1.07 * w, True))
    out += [(uniform(0.0, 0.0, 0.0), False), (-w, False), (uniform(0.2, -0.1, 0.01), False),
            (uniform(-0.0, 0.0, 0.0), False), (uniform(0.0, 0.1, 0.01), True), (uniform(1e-310, 1e-310, 0.0), False),
            (uniform(np.nan, 0.1, 0.1), False), (uniform(np.inf, 0.1, 0.1), False)]
    return out


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are not available")
    exe = str(tmp_path_factory.mktemp("quiet") / "quiet_host_check")
    subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I" + CUDA_INCLUDE,
                    "-I" + os.path.join(ROOT, "lambrex_gb300", "csrc"),
                    os.path.join(HERE, "quiet_host_check.cpp"), "-o", exe], check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("om_s,om_b", RATES)
def test_uniform_cells_on_the_host(harness, tmp_path, om_s, om_b):
    inp, out = str(tmp_path / "in.bin"), str(tmp_path / "out.bin")
    cells = rest_cells()
    np.stack([c for c, _ in cells]).tofile(inp)
    subprocess.run([harness, inp, out, repr(om_s), repr(om_b)], check=True)
    for (c, short), g in zip(cells, np.fromfile(out).reshape(-1, 31)):
        assert bool(g[30]) == short, c
        a, b = g[:15], g[15:30]
        assert np.array_equal(np.isnan(a), np.isnan(b)), c
        # one and the same formula, rounded in other places here than on the GPU:
        # a dozen operations on values of at most the density
        ok = np.isfinite(b)
        assert np.all(np.abs(a - b)[ok] <= 16 * 2.0 ** -53 * np.sum(np.abs(c))), c


def one_step_of_a_refined_run(gpu_lib, cell, tau):
    """Level 0's cells away from the patch after a step from a uniform state."""
    s = gpu_lib.AmrSim(12, 12, 12, 1, [1, 1, 1], tau[0], tau[1], precision="f64", amr_mode="conservative")
    s.SetInitialDensity(1.0)
    s.SetInitialVelocity(0.0)
    s.InitFromScratch(0.0)
    s.SetStaticRefinement(0, (4, 4, 4), (7, 7, 7))
    for lev in (0, 1):
        n = s.copy_f(lev).shape
        s.set_f(lev, np.broadcast_to(cell[:, None, None, None], n))
    s.Iterate(1)
    return s.copy_f(0)[:, 0, 0, 0]


def general_form(gpu_lib, cell, tau):
    """collide<double> of a cell through the device-pointer step, which takes
    cells with a sign bit to it: minus the collision of minus the cell (rounding
    to nearest knows no sign)."""
    import torch

    f = torch.from_numpy(np.ascontiguousarray(np.broadcast_to(-cell[:, None], (15, 8)))).cuda()
    g = torch.empty_like(f)
    L = gpu_lib.lib()
    assert L.lbx_step_periodic_f64(ctypes.c_void_p(f.data_ptr()), ctypes.c_void_p(g.data_ptr()), 2, 2, 2,
                                   ctypes.c_double(tau[0]), ctypes.c_double(tau[1]),
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    return -g.cpu().numpy()[:, 0]


@pytest.mark.gpu
@pytest.mark.parametrize("om_s,om_b", RATES)
def test_uniform_cells_have_the_general_forms_bits(gpu_lib, om_s, om_b):
    tau = (1.0 / om_s - 0.5, 1.0 / om_b - 0.5)
    for cell, short in rest_cells():
        if short:
            assert np.array_equal(one_step_of_a_refined_run(gpu_lib, cell, tau), general_form(gpu_lib, cell, tau)), cell


@pytest.mark.gpu
def test_no_density_is_nan(gpu_lib):
    assert np.all(np.isnan(one_step_of_a_refined_run(gpu_lib, np.zeros(15), (0.9, 0.8))))
