"""The restriction's means of eight and the interpolation in time of refined FP64
runs (csrc/fx64.cuh), against exact rational arithmetic.

Means: populations far apart are cut by less than one unit of 2^-57 of the power
of two below the largest (eight of them at most, where half an ulp of the sum is
16 units or more) and rounded once; where FP64 additions are kept, seven of
them round.  Halves: one rounding, whatever the size of the sum."""
import os
import shutil
import subprocess
from fractions import Fraction as Fr

import numpy as np
import pytest

from test_fx64 import CUDA_INCLUDE, HERE, ROOT


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are not available")
    exe = str(tmp_path_factory.mktemp("means") / "means_host_check")
    subprocess.run([gxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I" + CUDA_INCLUDE,
                    "-I" + os.path.join(ROOT, "lambrex_gb300", "csrc"),
                    os.path.join(HERE, "means_host_check.cpp"), "-o", exe], check=True, capture_output=True)

    def run(what, rows, tmp_path):
        inp, out = str(tmp_path / "in.bin"), str(tmp_path / "out.bin")
        np.asarray(rows, dtype=np.float64).tofile(inp)
        subprocess.run([exe, what, inp, out], check=True)
        return np.fromfile(out)

    return run


def ulp(x):
    return Fr(2) ** (max(int(np.frexp(abs(x))[1]), -1021) - 53)


def eights():
    """(children, whether they are summed as integers)"""
    rng = np.random.default_rng(6)
    out = []
    for _ in range(60):
        out.append((rng.uniform(0.05, 0.3, 8), True))
    for _ in range(20):
        out.append((0.1 * 10.0 ** rng.uniform(-12, 0, 8), True))
    for s in (2.0 ** -940, 1e-100, 1e100, 2.0 ** 990):
        out.append((s * rng.uniform(0.5, 1, 8), True))
    for k in range(8):  # an empty child, a tiny one, a negative one
        for v, fx in ((0.0, True), (1e-40, True), (5e-324, True), (-0.01, False), (-0.0, False)):
            e = rng.uniform(0.1, 0.2, 8)
            e[k] = v
            out.append((e, fx))
    x = 1 / 9.0
    out.append((np.full(8, x), False))
    for ulps in (1, 100, 511, 512, 600, 5000):  # near equal: either way
        e = np.full(8, x)
        e[5] += ulps * np.spacing(x)
        out.append((e, ulps >= 600))
    out += [(np.zeros(8), False), (np.full(8, -0.3), False), (np.array([0.5] * 7 + [1.0]), True),
            (np.full(8, 2.0 ** -1000) * np.arange(1, 9), False), (2.0 ** 1005 * np.arange(1, 9), False)]
    return out


def test_means_of_eight(harness, tmp_path):
    got = harness("mean", [e for e, _ in eights()], tmp_path)
    for (e, integers), g in zip(eights(), got):
        ref = sum(Fr(float(v)) for v in e) / 8
        bound = ulp(g) / 2
        if integers:
            bound += Fr(2) ** (int(np.frexp(np.max(e))[1]) - 1 - 57)  # eight units, an eighth of them
        elif len(set(e)) > 1:
            bound = 7 * sum(Fr(abs(float(v))) for v in e) / 8 / 2 ** 53
        assert abs(Fr(float(g)) - ref) <= bound, e


def test_means_that_are_no_numbers(harness, tmp_path):
    rows = [[0.1] * 7 + [v] for v in (np.nan, np.inf, -np.inf)] + [[np.inf, -np.inf] + [0.1] * 6]
    got = harness("mean", rows, tmp_path)
    assert np.isnan(got[0]) and got[1] == np.inf and got[2] == -np.inf and np.isnan(got[3])


def test_interpolation_in_time(harness, tmp_path):
    rng = np.random.default_rng(7)
    big, tiny = float(np.finfo(np.float64).max), 5e-324
    ab = [tuple(rng.uniform(-0.3, 0.3, 2)) for _ in range(200)]
    ab += [(0.1, 0.1), (0.1, -0.1), (0.0, 0.0), (1e300, -1e300), (2.0 ** -1000, 2.0 ** -1020),
           (2.0 ** -1022, 2.0 ** -1022), (2.0 ** -1022, 2.0 ** -1023), (2.0 ** -1021, 0.0),
           (1e308, 1.5e308), (-1.7e308, -1.7e308), (big, big), (big, -big), (big, tiny), (tiny, tiny)]
    halves = harness("weighted", [(0.5, a, 0.5, b) for a, b in ab], tmp_path)
    for (a, b), g in zip(ab, halves):
        ref = (Fr(float(a)) + Fr(float(b))) / 2
        # half an ulp; among the subnormals the two products round as well
        bound = ulp(g) / 2 if abs(g) >= 2.0 ** -1021 else Fr(tiny)
        assert np.isfinite(g) and abs(Fr(float(g)) - ref) <= bound, (a, b)
    others = harness("weighted", [(1.0, a, 0.0, b) for a, b in ab], tmp_path)
    assert np.array_equal(others, np.array([a for a, _ in ab]))
    assert np.isnan(harness("weighted", [(0.5, np.nan, 0.5, 0.1)], tmp_path)[0])
    assert harness("weighted", [(0.5, np.inf, 0.5, 0.1)], tmp_path)[0] == np.inf
