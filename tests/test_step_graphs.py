"""The graphs in which lbx_iterate replays steps (csrc/step_graphs.h): each
brings every level's buffers back into their roles, and a program that calls
Iterate with the same number again and again finds its graphs again."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from golden_util import smooth_random

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
SLOTS, MIN_STEPS = 4, 4  # graphs a handle keeps; shorter runs launch directly


@pytest.fixture(scope="module")
def choose(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ is not available")
    exe = str(tmp_path_factory.mktemp("graphs") / "step_graphs_host_check")
    subprocess.run([gxx, "-std=c++17", "-O2", "-I" + os.path.join(ROOT, "lambrex_gb300", "csrc"),
                    os.path.join(HERE, "step_graphs_host_check.cpp"), "-o", exe], check=True, capture_output=True)

    def run(finest, faithful):
        """for left = 0 .. 1000: (role period, steps, whether a first run is direct)"""
        out = subprocess.run([exe], input="".join("%d %d %d\n" % (finest, faithful, n) for n in range(1001)),
                             check=True, capture_output=True, text=True).stdout.split("\n")[:1001]
        return [tuple(int(v) for v in line.split()) for line in out]

    return run


def step(roles, finest, faithful):
    """The buffers' roles (now, next, tmp) of each level after a step."""
    def swap(lev, a, b):
        r = roles[lev]
        r[a], r[b] = r[b], r[a]

    def advance(lev):
        if not faithful or finest == 0:
            swap(lev, 0, 1)
            if lev < finest:
                advance(lev + 1)
                advance(lev + 1)
            return
        if lev + 1 == finest:  # two collide-stream sub-steps, one update
            swap(finest, 1, 2)
            swap(finest, 1, 2)
            swap(finest, 0, 1)
        else:
            advance(lev + 1)
            advance(lev + 1)
        swap(lev, 1, 2)
        swap(lev, 0, 1)

    advance(0)


@pytest.mark.parametrize("finest,faithful", [(f, m) for f in range(5) for m in (0, 1)])
def test_graphs_return_the_roles(choose, finest, faithful):
    first, roles, period = [[0, 1, 2] for _ in range(finest + 1)], [[0, 1, 2] for _ in range(finest + 1)], 0
    while period == 0 or roles != first:
        step(roles, finest, faithful)
        period += 1
    for left, (p, steps, _) in enumerate(choose(finest, faithful)):
        assert p % period == 0 and p <= 6
        assert steps % p == 0 and 0 <= steps <= left


# one level deep the faithful cycle's roles return after six steps; odd lengths
# start from more roles than a handle keeps graphs
@pytest.mark.parametrize("finest,faithful,n", [(f, 0, n) for f in (0, 1, 2) for n in (4, 5, 8, 9, 20, 45, 100)]
                         + [(1, 1, n) for n in (6, 8, 9, 12, 18, 20, 21, 40, 100)]
                         + [(2, 1, n) for n in (3, 4, 8, 9, 10, 20, 100)])
def test_repeated_calls_capture_nothing(choose, finest, faithful, n):
    table = choose(finest, faithful)
    period = table[0][0]
    at, kept, captures = 0, [], []  # kept: (roles, steps), the last used one last
    for _ in range(30):
        left, captured = n, 0
        while left >= MIN_STEPS and table[left][1]:
            have = max((k[1] for k in kept if k[0] == at % period and k[1] <= left), default=0)
            if have < table[left][1]:  # (a handle's first direct runs are over)
                captured += 1
                have = table[left][1]
                kept.append((at % period, have))
                del kept[:-SLOTS]
                left -= have  # a capture runs its steps once
            else:
                kept.append(kept.pop(kept.index((at % period, have))))
                left %= have
            # whole periods: `at` keeps its roles
        at += n
        captures.append(captured)
    assert not any(captures[6:])


@pytest.mark.gpu
@pytest.mark.parametrize("finest,n,calls", [(1, 9, 3), (1, 8, 3), (1, 20, 1), (2, 8, 2)])
def test_faithful_runs_equal_single_steps(gpu_lib, finest, n, calls):
    dims = (12, 16, 12)
    rho_c, u_c = smooth_random(*dims, seed=7)

    def make():
        s = gpu_lib.AmrSim(*dims, finest, [1, 1, 1], 0.9, 0.8, precision="f64", amr_mode="faithful")
        s.SetInitialDensity(rho_c)
        s.SetInitialVelocity(u_c)
        s.InitFromScratch(0.0)
        s.SetStaticRefinement(0, (3, 4, 3), (8, 11, 8))
        if finest > 1:
            s.SetStaticRefinement(1, (8, 10, 8), (13, 19, 13))
        return s

    a, b = make(), make()
    for _ in range(calls):
        for _ in range(n):
            a.Iterate(1)
        b.Iterate(n)
        for lev in range(finest + 1):
            assert np.array_equal(a.copy_f(lev), b.copy_f(lev), equal_nan=True)
            assert a.GetTime(lev) == b.GetTime(lev) and a.GetTimeStep(lev) == b.GetTimeStep(lev)
        assert a.launch_count() == b.launch_count()


def make(gpu_lib, precision, mode, levels, dims=(12, 16, 12)):
    rho_c, u_c = smooth_random(*dims, seed=7)
    s = gpu_lib.AmrSim(*dims, levels, [1, 1, 1], 0.9, 0.8, precision=precision, amr_mode=mode)
    s.SetInitialDensity(rho_c)
    s.SetInitialVelocity(u_c)
    s.InitFromScratch(0.0)
    if levels >= 1:
        s.SetStaticRefinement(0, (3, 4, 3), (8, 11, 8))
    if levels >= 2:
        s.SetStaticRefinement(1, (8, 10, 8), (13, 19, 13))
    s.synchronize()
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("precision,mode,levels", [("f32s", "conservative", 0), ("f64", "rescaled", 1)])
@pytest.mark.parametrize("steps", [3, 9, 64])
def test_steps_captured_with_graphs_at_hand(gpu_lib, precision, mode, levels, steps):
    """Steps captured by the caller where the handle has graphs for them (a
    capture takes no launch of a graph, so they are not used there)."""
    import ctypes

    import torch

    a, b = make(gpu_lib, precision, mode, levels), make(gpu_lib, precision, mode, levels)
    for s in (a, b):
        for n in (1, 300, 40):  # an even number from the first: the roles are those of the graphs
            s.Iterate(n)
        s.synchronize()
    a.Iterate(steps)
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


@pytest.mark.gpu
@pytest.mark.parametrize("precision,mode,levels", [("f64", "conservative", 0), ("f32s", "conservative", 0),
                                                   ("f64", "rescaled", 1), ("f32s", "conservative", 2)])
@pytest.mark.parametrize("lengths", [(300, 40, 9), (130, 70, 33, 64), (100, 29, 8, 45)])
def test_direct_runs_and_graphs_equal_single_steps(gpu_lib, precision, mode, levels, lengths):
    """A long first run in graphs; first runs launched directly, later ones in graphs."""
    a, b = make(gpu_lib, precision, mode, levels), make(gpu_lib, precision, mode, levels)
    for n in lengths:
        for _ in range(n):
            a.Iterate(1)
        b.Iterate(n)
        for s in (a, b):  # a readout between the calls: the store roles swap
            s.CalcHydroVars(0)
        for lev in range(levels + 1):
            assert np.array_equal(a.copy_f(lev), b.copy_f(lev)), (n, lev)
            assert a.GetTime(lev) == b.GetTime(lev) and a.GetTimeStep(lev) == b.GetTimeStep(lev)
        assert a.launch_count() == b.launch_count()


@pytest.mark.gpu
def test_a_first_run_costs_no_more_than_its_steps(gpu_lib):
    """Nine steps of a new handle, against the same in runs too short for a
    graph: making a graph of eight launches took as long as twenty of them."""
    import statistics
    import time

    def first(lengths):
        t = []
        for _ in range(25):
            s = make(gpu_lib, "f32s", "conservative", 0)
            t0 = time.perf_counter()
            for n in lengths:
                s.Iterate(n)
            s.synchronize()
            t.append(time.perf_counter() - t0)
            s.close()
        return statistics.median(t)

    first([9])
    assert first([9]) < 1.5 * first([3, 3, 3])
