"""The fields where the density is barely twice the power of two below the
largest population, the end of the fixed point's range (csrc/fx64.cuh): there
the inverse's FP32 start reaches 2^31."""
import ctypes
from fractions import Fraction as Fr

import numpy as np
import pytest

from test_fx64 import C
from test_fx64_fields import harness  # noqa: F401


def boundary_cells():
    """Populations whose sum is 2 (1 + x) for small x >= 0, the largest in [1, 2)."""
    out = []
    for x in [0.0] + [2.0 ** -k for k in range(2, 52)]:
        for a, b in ((1, 3), (3, 14), (6, 8), (2, 5)):
            f = np.zeros(15)
            f[a], f[b], f[0] = 1.0, 0.75 + x, 0.25 + x
            out.append(f)
    return out


def check(f, rho, u):
    fr = [Fr(float(v)) for v in f]
    ref = sum(fr)
    unit = Fr(1, 2 ** 57)  # the bounds of test_fx64_fields
    assert abs(Fr(float(rho)) - ref) <= Fr(float(np.spacing(rho))) / 2 + 15 * unit, f
    for a in range(3):
        v = sum(int(C[q][a]) * fr[q] for q in range(15)) / ref
        assert abs(Fr(float(u[a])) - v) <= 4 * abs(v) / 2 ** 53 + 30 * unit / ref, f


def test_fields_on_the_host(harness, tmp_path):  # noqa: F811
    cells = boundary_cells()
    got = harness("hydro", cells, 5, tmp_path)
    assert np.all(got[:, 4] == 1)
    for f, g in zip(cells, got):
        check(f, g[0], g[1:4])


@pytest.mark.gpu
def test_fields_on_the_gpu():
    import torch

    from lambrex_gb300 import lbx
    cells = boundary_cells()
    n = len(cells)
    f = torch.from_numpy(np.ascontiguousarray(np.stack(cells).T)).cuda()
    r, u = torch.empty(n, dtype=torch.float64, device="cuda"), torch.empty((3, n), dtype=torch.float64, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert lbx.lib().lbx_hydro_f64(p(f), p(r), p(u), n, 1, 1,
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    r, u = r.cpu().numpy(), u.cpu().numpy()
    for k, c in enumerate(cells):
        check(c, r[k], u[:, k])
