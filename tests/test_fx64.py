"""The FP64 collision in block fixed point (csrc/fx64.cuh) at the edges of its
range, on the host and on the GPU, against the same collision in exact
rational arithmetic (src/AmrSim.cpp:25-107).

The bound is derived, not measured.  A unit is 2^-57 of the power of two below
the largest population.  Each product is off by at most 0.75 unit and u_a by
one, each converted population by less than one; carried through the
relaxation at rates in (0, 2) that is at most 40 units of an axis or rest
population and 16 of a diagonal one, and the result is rounded once, by half
an ulp.  Cells outside the range take the FP64 instructions: 64 ulp of the
density there, as 15 terms of at most rho pass through four roundings each."""
import ctypes
import os
import shutil
import subprocess
from fractions import Fraction as Fr

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA_INCLUDE = "/usr/local/cuda/include"
C = np.array([[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1],
              [1, 1, 1], [1, 1, -1], [1, -1, 1], [1, -1, -1],
              [-1, 1, 1], [-1, 1, -1], [-1, -1, 1], [-1, -1, -1]])
W = [Fr(2, 9)] + [Fr(1, 9)] * 6 + [Fr(1, 72)] * 8
RATES = [(1.25, 0.9), (1.9, 1.6), (0.02, 1.98), (2.0, 1.0), (-0.3, -0.7), (3.5, 1.0)]


def equilibrium(rho, u):
    w = np.array([float(x) for x in W])
    cu = C @ u
    return w * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * u @ u)


def cells():
    """(name, populations, whether the fixed point takes it at rates in (-1, 3))"""
    rng = np.random.default_rng(3)
    out = []

    def add(name, f, fx):
        out.append((name, np.asarray(f, dtype=np.float64), fx))

    rest = equilibrium(1.0, np.zeros(3))
    add("rest", rest, True)
    for k in range(24):  # ordinary states
        u = rng.uniform(-0.1, 0.1, 3)
        add("near %d" % k, equilibrium(rng.uniform(0.9, 1.1), u)
            + 1e-2 * rng.uniform(-1, 1, 15) * rest, True)
    for s in (2.0 ** -940, 1e-200, 1e-30, 1e30, 1e200, 2.0 ** 990):  # scales within the range
        add("scale %g" % s, s * equilibrium(1.07, np.array([0.03, -0.02, 0.05])), True)
    for s in (2.0 ** -1000, 2.0 ** 1005):  # and beyond it
        add("scale %g" % s, s * equilibrium(1.07, np.array([0.03, -0.02, 0.05])), False)
    for q in (0, 1, 6, 7, 14):  # an empty population, a tiny one, a negative one
        f = rest.copy()
        f[q] = 0.0  # without the rest population the density is seven times the largest
        add("empty %d" % q, f, q > 0)
        f = rest.copy()
        f[q] = 1e-25
        add("tiny %d" % q, f, q > 0)
        f = rest.copy()
        f[q] = -1e-3
        add("negative %d" % q, f, False)
    add("below 1/4", equilibrium(1.0, np.array([0.24, 0.0, 0.0])), True)
    add("above 1/4", equilibrium(1.0, np.array([0.26, 0.0, 0.0])), False)
    add("even", np.full(15, 1.0), False)  # density out of proportion to the largest
    add("single", np.array([1.0] + [0.0] * 14), False)
    add("all bits", np.nextafter(np.array([0.25] + [0.125] * 6 + [0.015625] * 8), 0), True)
    add("powers", np.array([0.25] + [0.125] * 6 + [0.015625] * 8), True)
    return out


def exact(f, om_s, om_b):
    f = [Fr(float(x)) for x in f]
    ws, wb = Fr(om_s), Fr(om_b)
    rho = sum(f)
    j = [sum(int(C[q][a]) * f[q] for q in range(15)) for a in range(3)]
    P = [[sum(int(C[q][a] * C[q][b]) * f[q] for q in range(15)) - (rho / 3 if a == b else 0)
          for b in range(3)] for a in range(3)]
    T = sum(P[a][a] for a in range(3))
    ruu = sum(x * x for x in j) / rho
    Tn = T + wb * (ruu - T)
    m = [[P[a][b] + ws * (j[a] * j[b] / rho - P[a][b]) for b in range(3)] for a in range(3)]
    for a in range(3):
        d = P[a][a] - T / 3
        m[a][a] = d + ws * (j[a] * j[a] / rho - ruu / 15 - d) + Tn / 3
    tr = sum(m[a][a] for a in range(3))
    out = []
    for q in range(15):
        c = [int(v) for v in C[q]]
        s = rho - Fr(3, 2) * tr + 3 * sum(c[a] * j[a] for a in range(3))
        s += Fr(9, 2) * sum(c[a] * c[b] * m[a][b] for a in range(3) for b in range(3))
        out.append(W[q] * s)
    return out


def check(name, f, got, om_s, om_b, fx):
    ref = exact(f, om_s, om_b)
    top = max(abs(x) for x in f)
    unit = Fr(2) ** (int(np.frexp(top)[1]) - 1 - 57)
    rho = sum(Fr(abs(float(x))) for x in f)
    for q in range(15):
        if fx:
            bound = Fr(float(np.spacing(abs(got[q])))) / 2 + (40 if q < 7 else 16) * unit
        else:
            bound = 64 * rho / 2 ** 52
        err = abs(Fr(float(got[q])) - ref[q])
        assert err <= bound, (name, q, float(err / bound), (om_s, om_b))


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are not available")
    exe = str(tmp_path_factory.mktemp("fx") / "fx_host_check")
    subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I" + CUDA_INCLUDE,
                    "-I" + os.path.join(ROOT, "lambrex_gb300", "csrc"),
                    os.path.join(HERE, "fx_host_check.cpp"), "-o", exe], check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("om_s,om_b", RATES)
def test_fixed_point_collision_on_the_host(harness, tmp_path, om_s, om_b):
    inp, out = str(tmp_path / "in.bin"), str(tmp_path / "out.bin")
    all_cells = cells()
    np.stack([c[1] for c in all_cells]).tofile(inp)
    subprocess.run([harness, inp, out, repr(om_s), repr(om_b)], check=True)
    got = np.fromfile(out).reshape(-1, 16)
    assert len(got) == len(all_cells)
    for (name, f, fx), g in zip(all_cells, got):
        fx = fx and -1 < om_s < 3
        assert bool(g[15]) == fx, (name, om_s)
        check(name, f, g[:15], om_s, om_b, fx)


@pytest.mark.gpu
@pytest.mark.parametrize("om_s,om_b", [r for r in RATES if r[0] > 0])
def test_fixed_point_collision_on_the_gpu(om_s, om_b):
    """The same cells as a row along x through lbx_step_periodic_f64: a step
    moves each result by c_x, which is undone here."""
    import torch

    from lambrex_gb300 import lbx
    all_cells = cells()
    n = len(all_cells)
    f = np.ascontiguousarray(np.stack([c[1] for c in all_cells]).T)
    fin = torch.from_numpy(f).cuda()
    fout = torch.empty_like(fin)
    L = lbx.lib()
    tau = [ctypes.c_double(1.0 / om - 0.5) for om in (om_s, om_b)]
    rc = L.lbx_step_periodic_f64(ctypes.c_void_p(fin.data_ptr()), ctypes.c_void_p(fout.data_ptr()),
                                 n, 1, 1, tau[0], tau[1],
                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    got = fout.cpu().numpy()
    got = np.stack([np.roll(got[q], -C[q][0]) for q in range(15)])
    # the rates as the library forms them from tau
    ws, wb = (1.0 / (t.value + 0.5) for t in tau)
    for k, (name, fc, fx) in enumerate(all_cells):
        check(name, fc, got[:, k], ws, wb, fx and ws < 2.99)
