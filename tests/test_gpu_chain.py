"""Runs replayed in long and short graphs of chained launches (csrc/launch.cuh)
give the bits, times and launch counts of single steps, whatever the lengths
of the calls and whatever is read between them."""
import numpy as np
import pytest

from golden_util import smooth_random

pytestmark = pytest.mark.gpu
CASES = [("f32s", "conservative", 0), ("f64", "conservative", 0), ("f64p", "rescaled", 1),
         ("f32s", "conservative", 1), ("f64", "rescaled", 2), ("f64", "faithful", 1)]


@pytest.mark.parametrize("precision,mode,levels", CASES)
@pytest.mark.parametrize("lengths", [(64, 3, 70), (33, 100, 5, 2), (4, 63, 65, 1)])
def test_long_graphs_equal_single_steps(gpu_lib, precision, mode, levels, lengths):
    dims = (12, 16, 12)
    rho_c, u_c = smooth_random(*dims, seed=7)

    def make():
        s = gpu_lib.AmrSim(*dims, levels, [1, 1, 1], 0.9, 0.8, precision=precision, amr_mode=mode)
        s.SetInitialDensity(rho_c)
        s.SetInitialVelocity(u_c)
        s.InitFromScratch(0.0)
        if levels >= 1:
            s.SetStaticRefinement(0, (3, 4, 3), (8, 11, 8))
        if levels >= 2:
            s.SetStaticRefinement(1, (8, 10, 8), (13, 19, 13))
        return s

    a, b = make(), make()
    if mode == "faithful":
        lengths = lengths[:1]  # it grows without bound on longer runs
    for n in lengths:
        for _ in range(n):
            a.Iterate(1)
        b.Iterate(n)
        for s in (a, b):  # a readout between the calls: the store roles swap
            s.CalcHydroVars(0)
        for lev in range(levels + 1):
            assert np.array_equal(a.copy_f(lev), b.copy_f(lev), equal_nan=True), (n, lev)
            assert a.GetTime(lev) == b.GetTime(lev) and a.GetTimeStep(lev) == b.GetTimeStep(lev)
        assert a.launch_count() == b.launch_count()


@pytest.mark.parametrize("precision,levels,warm,steps", [("f64", 0, 2, 6), ("f32s", 0, 34, 64),
                                                         ("f32s", 0, 14, 64), ("f64", 1, 2, 8)])
def test_steps_captured_by_the_caller(gpu_lib, precision, levels, warm, steps):
    """Steps inside a capture of the handle's own stream, with and without a
    graph at hand from earlier calls, replay to the bits of direct ones."""
    import ctypes

    import torch

    dims = (12, 16, 12)
    rho_c, u_c = smooth_random(*dims, seed=7)

    def make():
        s = gpu_lib.AmrSim(*dims, levels, [1, 1, 1], 0.9, 0.8, precision=precision)
        s.SetInitialDensity(rho_c)
        s.SetInitialVelocity(u_c)
        s.InitFromScratch(0.0)
        if levels:
            s.SetStaticRefinement(0, (3, 4, 3), (8, 11, 8))
        s.Iterate(warm)
        return s

    a, b = make(), make()
    a.Iterate(steps)
    b.copy_f(0)  # waits for the queued steps
    p = ctypes.c_void_p()
    assert b._L.lbx_get_stream(b._h, ctypes.byref(p)) == 0
    stream = torch.cuda.ExternalStream(p.value)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream, capture_error_mode="thread_local"):
        b.Iterate(steps)
    with torch.cuda.stream(stream):
        g.replay()  # once: a second run would want the stores back in their roles
    stream.synchronize()
    for lev in range(levels + 1):
        assert np.array_equal(a.copy_f(lev), b.copy_f(lev))
    del g
