"""The FP64 equilibrium, hydrodynamic fields and mass and momentum sums in
fixed point (csrc/fx64.cuh, csrc/sums.cuh) at the edges of their ranges,
against exact rational arithmetic.

The bounds are derived.  Fields: every population is cut by less than one unit
(2^-57 of the power of two below the largest), the density and the momenta are
rounded once, the inverse is within 2^-56 and the product rounded.
Equilibrium: 32 units of 2^-60 in the velocity polynomial, 3/4 of a unit of
2^-55.8 in its product with the density, and the rounding.  Sums: 15 units of
2^-57 per cell at the largest scale met, and one rounding."""
import ctypes
import math
import os
import shutil
import subprocess
from fractions import Fraction as Fr

import numpy as np
import pytest

from test_fx64 import C, CUDA_INCLUDE, HERE, ROOT, W, cells, equilibrium


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are not available")
    exe = str(tmp_path_factory.mktemp("fxf") / "fx_fields")
    subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I" + CUDA_INCLUDE,
                    "-I" + os.path.join(ROOT, "lambrex_gb300", "csrc"),
                    os.path.join(HERE, "fx_fields_host_check.cpp"), "-o", exe], check=True, capture_output=True)

    def run(what, rows, width, tmp_path):
        inp, out = str(tmp_path / "in.bin"), str(tmp_path / "out.bin")
        np.asarray(rows, dtype=np.float64).tofile(inp)
        subprocess.run([exe, what, inp, out], check=True)
        return np.fromfile(out).reshape(-1, width)

    return run


def states():
    """(rho, ux, uy, uz), whether the fixed point takes it"""
    rng = np.random.default_rng(8)
    out = [((1.0, 0, 0, 0), True), ((1.0, -0.0, 0, 0), True), ((2.0 ** -900, 0.1, 0.2, -0.1), True),
           ((1e200, 1e-300, -1e-17, 0.24), True), ((1.0, 0.25, 0, 0), False), ((1.0, 0, 0, -0.3), False),
           ((0.0, 0, 0, 0), False), ((-1.0, 0.1, 0, 0), False), ((1.0, np.nan, 0, 0), False),
           ((np.inf, 0, 0, 0), False), ((2.0 ** -1000, 0, 0, 0), False),
           ((1.0,) + (float(np.nextafter(0.25, 0)),) * 3, True),
           ((float(np.nextafter(2, 0)),) + (-float(np.nextafter(0.25, 0)),) * 3, True)]
    for _ in range(200):
        out.append(((rng.uniform(0.3, 3), *rng.uniform(-0.249, 0.249, 3)), True))
    return out


def test_equilibrium_in_fixed_point(harness, tmp_path):
    got = harness("eq", [s for s, _ in states()], 16, tmp_path)
    for (s, fx), g in zip(states(), got):
        assert bool(g[15]) == fx, s
        if not fx:
            continue
        rho, u = Fr(s[0]), [Fr(float(v)) for v in s[1:]]
        uu = sum(v * v for v in u)
        for q in range(15):
            cu = sum(int(C[q][a]) * u[a] for a in range(3))
            ref = W[q] * rho * (1 + 3 * cu + Fr(9, 2) * cu * cu - Fr(3, 2) * uu)
            bound = Fr(float(np.spacing(g[q]))) / 2 + W[q] * rho * (Fr(32, 2 ** 60) + Fr(1, 2 ** 55))
            assert abs(Fr(float(g[q])) - ref) <= bound, (s, q)


def test_fields_in_fixed_point(harness, tmp_path):
    all_cells = cells()
    got = harness("hydro", [f for _, f, _ in all_cells], 5, tmp_path)
    taken = 0
    for (name, f, _), g in zip(all_cells, got):
        if not g[4]:
            continue
        taken += 1
        fr = [Fr(float(x)) for x in f]
        rho = sum(fr)
        unit = Fr(2) ** (int(np.frexp(max(f))[1]) - 1 - 57)
        assert abs(Fr(float(g[0])) - rho) <= Fr(float(np.spacing(g[0]))) / 2 + 15 * unit, name
        for a in range(3):
            u = sum(int(C[q][a]) * fr[q] for q in range(15)) / rho
            assert abs(Fr(float(g[1 + a])) - u) <= 4 * abs(u) / 2 ** 53 + 30 * unit / rho, name
    # ordinary states, scales in range, and cells the collision leaves alone for their velocity
    assert taken >= 24 + 6 + 2
    assert not any(g[4] for (name, _, _), g in zip(all_cells, got) if name.startswith("negative"))


def sums_of(f):
    return [math.fsum(f.ravel())] + [math.fsum((C[:, a][:, None] * f).ravel()) for a in range(3)]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 255, 257, 152 * 3 * 256 - 1, 152 * 3 * 256 * 2 + 5])
@pytest.mark.parametrize("what", ["ordinary", "scales", "odd", "none positive"])
def test_sums_on_the_gpu(n, what):
    """Ordinary cells; blocks whose cells are a factor of four and 1e6 apart;
    negative, empty and out-of-proportion populations; all cells negative."""
    import torch

    from lambrex_gb300 import lbx
    rng = np.random.default_rng(n)
    w = np.array([float(x) for x in W])
    f = w[:, None] * (1.0 + 0.2 * rng.uniform(-1, 1, (15, n)))
    if what == "scales":
        f *= np.where(rng.uniform(size=n) < 0.3, 4.0 ** rng.integers(-10, 11, n), 1.0)
    elif what == "odd":
        f[rng.integers(0, 15, n), np.arange(n)] *= rng.choice([1.0, 0.0, -1.0, 1e-30], n)
    elif what == "none positive":
        f *= -1e-3
    fin = torch.from_numpy(np.ascontiguousarray(f)).cuda()
    out = torch.empty(4, dtype=torch.float64, device="cuda")
    rc = lbx.lib().lbx_reduce_mass_momentum_f64(
        ctypes.c_void_p(fin.data_ptr()), ctypes.c_size_t(n), ctypes.c_void_p(out.data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    got, scale = out.cpu().numpy(), math.fsum(np.abs(f).ravel())
    for g, r in zip(got, sums_of(f)):
        # a cell's FP64 sum (where the integers do not hold it) rounds 15 times
        assert abs(g - r) <= abs(r) * 2 ** -53 + scale * 15 * (2.0 ** -53 if what != "ordinary" else 2.0 ** -57)


@pytest.mark.gpu
def test_sums_of_infinite_and_nan_cells_are_nan():
    import torch

    from lambrex_gb300 import lbx
    for bad in (np.inf, -np.inf, np.nan):
        f = torch.full((15, 700), 0.1, dtype=torch.float64, device="cuda")
        f[3, 600] = bad
        out = torch.empty(4, dtype=torch.float64, device="cuda")
        assert lbx.lib().lbx_reduce_mass_momentum_f64(
            ctypes.c_void_p(f.data_ptr()), ctypes.c_size_t(700), ctypes.c_void_p(out.data_ptr()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        assert math.isnan(out.cpu().numpy()[0])


@pytest.mark.gpu
def test_equilibrium_and_fields_on_the_gpu():
    """The device entry points on the same states: the host's values, whose
    approximate reciprocal differs in bits that the series removes."""
    import torch

    from lambrex_gb300 import lbx
    st = [s for s, fx in states() if fx]
    n = len(st)
    a = torch.tensor(np.array(st).T.copy(), device="cuda")
    f = torch.empty((15, n), dtype=torch.float64, device="cuda")
    r, u = torch.empty(n, dtype=torch.float64, device="cuda"), torch.empty((3, n), dtype=torch.float64, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    v = a[1:].contiguous()
    assert lbx.lib().lbx_equilibrium_f64(p(a), p(v), p(f), n, 1, 1, s) == 0
    assert lbx.lib().lbx_hydro_f64(p(f), p(r), p(u), n, 1, 1, s) == 0
    fh, rh, uh = f.cpu().numpy(), r.cpu().numpy(), u.cpu().numpy()
    for k, t in enumerate(st):
        ref = equilibrium(1.0, np.array(t[1:]))
        assert np.all(np.abs(fh[:, k] / t[0] - ref) <= 16 * 2.0 ** -53 * ref), t
        # the populations' roundings: 15 of half an ulp of at most half the density
        assert abs(rh[k] / t[0] - 1) <= 8 * 2.0 ** -53, t
        assert np.all(np.abs(uh[:, k] - t[1:]) <= 16 * 2.0 ** -53), t
