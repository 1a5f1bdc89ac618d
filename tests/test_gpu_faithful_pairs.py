"""The faithful cycle's paired collision gives a block whole rows in small boxes
with rows longer than a warp (csrc/kernels_amr.cu): rows shorter and longer than a
warp and a block, row counts that leave a block part empty, a level on either side
of the line, against the oracle."""
import numpy as np
import pytest

from golden_util import smooth_random

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,lo,hi", [((4, 5, 4), (1, 1, 1), (2, 3, 2)), ((33, 7, 6), (8, 2, 2), (20, 4, 3)),
                                        ((64, 5, 9), (10, 1, 2), (40, 3, 6)), ((130, 6, 5), (20, 1, 1), (100, 4, 3)),
                                        ((44, 42, 40), (10, 10, 10), (30, 28, 26))])
def test_rows_of_the_paired_collision(gpu_lib, oracle, dims, lo, hi):
    rho_c, u_c = smooth_random(*dims, seed=5)
    s = gpu_lib.AmrSim(*dims, 1, [1, 1, 1], 0.9, 0.8, precision="f64p", amr_mode="faithful")
    s.SetInitialDensity(rho_c)
    s.SetInitialVelocity(u_c)
    s.InitFromScratch(0.0)
    s.SetStaticRefinement(0, lo, hi)
    o = oracle.AmrOracle(*dims, 1, 0.9, 0.8, 0)
    o.init(rho_c, u_c)
    o.refine(0, lo, hi)
    s.Iterate(2)
    o.iterate(2)
    for lev in (0, 1):
        ref = np.asarray(o.f(lev))
        got = s.copy_f(lev).reshape(ref.shape)
        assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))
