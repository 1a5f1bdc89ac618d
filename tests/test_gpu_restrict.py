"""The rescaled restriction's two forms (one thread a covered cell, four warps
for 32 of them; csrc/kernels_amr.cu) on both sides of the line between them,
2^16 covered cells in FP64 and 2^17 in FP32, and with a few cells left over."""
import numpy as np
import pytest

from golden_util import smooth_random
from test_gpu_amr import RTOL, pair, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "f64p", "f32s"])
@pytest.mark.parametrize("covered", [(3, 5, 7), (32, 64, 31), (32, 64, 32), (32, 64, 63), (32, 64, 64)])
def test_rescaled_restriction_forms(gpu_lib, oracle, precision, covered):
    if (covered[2] > 32) != (precision == "f32s") and covered[0] > 3:
        pytest.skip("the line of the other store")
    dims = tuple(n + 6 for n in covered)
    rho_c, u_c = smooth_random(*dims, seed=11)
    lo, hi = (3, 3, 3), tuple(n + 2 for n in covered)
    sim, o = pair(gpu_lib, oracle, dims, 0.8, "rescaled", lo, hi, rho_c, u_c, precision=precision)
    sim.Iterate(1)
    o.iterate(1)
    for lev in (0, 1):
        f, g = sim.copy_f(lev), o.f(lev)
        if precision == "f32s":  # of order one; some thirty roundings of 2^-24 a step
            assert np.max(np.abs(f - g)) <= 1e-5
        else:
            assert rel(f, g) <= RTOL
