"""The paired-FP32 collision on the GPU (csrc/df32.cuh): the levels of refined
f64p runs, and single levels and the device-pointer step at rates that the fixed
point cannot hold, against the oracle's reference-order collision.

The bound is the one of the host form's test, 1e-13 of a population at rates up
to 1.9 (28 units of the pairs' 2^-48), times |omega - 1| / 0.9 beyond.  The
fixed point that other f64p runs take is two orders of magnitude closer, which
tells the two apart."""
import ctypes

import numpy as np
import pytest

from test_fx64 import C, equilibrium

pytestmark = pytest.mark.gpu
BOUND = 1e-13
N = 12


def state(seed):
    """Populations near equilibrium in FAB order, and their collision to be filled in."""
    rng = np.random.default_rng(seed)
    f = np.empty((15, N, N, N))
    for k in np.ndindex(N, N, N):
        f[(slice(None),) + k] = equilibrium(rng.uniform(0.95, 1.05), rng.uniform(-0.05, 0.05, 3))
    return f * (1 + 1e-3 * rng.uniform(-1, 1, f.shape))


def one_step(oracle, f, om_s, om_b, xs):
    """The step's result at the planes x in xs."""
    out = np.empty_like(f)
    for k in np.ndindex(N, N, N):
        if any((k[2] - x) % N in (0, 1, N - 1) for x in xs):
            out[(slice(None),) + k] = oracle.collide_cell(f[(slice(None),) + k], om_s, om_b)
    return np.stack([np.roll(out[q], C[q][::-1], axis=(0, 1, 2)) for q in range(15)])[..., xs]


def worst(got, ref):
    return float(np.max(np.abs(got - ref) / np.abs(ref)))


@pytest.mark.parametrize("mode", ["conservative", "rescaled"])
@pytest.mark.parametrize("om_s,om_b", [(1.25, 0.9), (1.9, 1.6)])
def test_refined_levels_collide_in_pairs(gpu_lib, oracle, mode, om_s, om_b):
    s = gpu_lib.AmrSim(N, N, N, 1, [1, 1, 1], 1 / om_s - 0.5, 1 / om_b - 0.5, precision="f64p", amr_mode=mode)
    s.SetInitialDensity(1.0)
    s.SetInitialVelocity(0.0)
    s.InitFromScratch(0.0)
    s.SetStaticRefinement(0, (4, 4, 4), (7, 7, 7))
    f = state(3)
    s.set_f(0, f)
    s.Iterate(1)
    xs = [0, 1, N - 1]  # two cells and more from the patch
    err = worst(s.copy_f(0)[..., xs], one_step(oracle, f, om_s, om_b, xs))
    assert 2e-15 < err <= BOUND


@pytest.mark.parametrize("om_s,om_b", [(3.2, 1.0), (1.0, -1.2)])
def test_pairs_at_rates_outside_the_fixed_point(gpu_lib, oracle, om_s, om_b):
    import torch

    f = state(4)
    bound = BOUND * max(abs(om_s - 1), abs(om_b - 1)) / 0.9
    tau = (1 / om_s - 0.5, 1 / om_b - 0.5)
    xs = list(range(N))
    ref = one_step(oracle, f, om_s, om_b, xs)
    fin = torch.from_numpy(f).cuda()
    fout = torch.empty_like(fin)
    assert gpu_lib.lib().lbx_step_periodic_f64p(
        ctypes.c_void_p(fin.data_ptr()), ctypes.c_void_p(fout.data_ptr()), N, N, N, ctypes.c_double(tau[0]),
        ctypes.c_double(tau[1]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    push = fout.cpu().numpy()
    assert 2e-15 < worst(push, ref) <= bound
    s = gpu_lib.AmrSim(N, N, N, 0, [1, 1, 1], tau[0], tau[1], precision="f64p")
    s.SetInitialDensity(1.0)
    s.SetInitialVelocity(0.0)
    s.InitFromScratch(0.0)
    s.set_f(0, f)
    s.Iterate(1)
    pull = s.copy_f(0)
    assert np.array_equal(pull, push)  # pull and push collide the same values in the same form
