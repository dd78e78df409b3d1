"""FP64 dust growth by lane groups against the oracle at the species counts where its layout changes:
one bin, one slot of eight, one past it, sixteen, one past it and the most; grids whose cells do not
fill the last block.  The sub-cycle follows the oracle's operations, so the tolerance is the FP64
parity tolerance, after the first step: later ones amplify the last bits of exp, log and pow."""
import numpy as np
import pytest

from shark_gb300 import config as K, setups
from tests.test_gpu_parity import FP64_TOL, rel_l1, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ndust", [(5, 1), (9, 2), (7, 8), (11, 9), (5, 16), (9, 17), (7, 32)])
@pytest.mark.parametrize("kernel,sticking", [(0, 1.0), (0, 0.3), (2, 1e4)])   # the additive kernel's rates are small here
def test_growth_lane_groups(n, ndust, kernel, sticking):
    cfg, u0 = setups.dusty_turb(n=n, ndust=ndust, nH=1e10, smin=1e-5, smax=1e-2, growth=True)
    cfg.grw_kernel, cfg.grw_sticking = kernel, sticking
    dto, dtg, uo, ug, st = run_pair(cfg, u0, 1)
    assert st & ~K.STATUS_GROWTH == 0
    np.testing.assert_allclose(dtg, dto, rtol=1e-13, atol=0)
    assert rel_l1(cfg, ug, uo).max() <= FP64_TOL
