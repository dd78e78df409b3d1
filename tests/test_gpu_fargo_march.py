"""The FARGO remap's march against the oracle at the edges of its split (32 columns a warp, 32 rows a
thread in batches of 8, 256 rows a block): rings shorter than a batch, one off a thread's and a
block's rows, one column past a warp, with whole-cell shifts, every limiter and both precisions.  The
tolerances are the parity tolerances of the paths."""
import numpy as np
import pytest

from shark_gb300 import config as K, setups
from tests.test_gpu_parity import FP64_TOL, MIXED_TOL, rel_l1, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nphi", [(5, 6), (31, 33), (33, 255), (32, 256), (65, 257), (36, 40)])
@pytest.mark.parametrize("slope", [0, 1, 2, 3])
@pytest.mark.parametrize("precision", [K.PREC_FP64, K.PREC_MIXED])
def test_ring_sizes(nr, nphi, slope, precision):
    cfg, u0 = setups.disk_polar(nr=nr, nphi=nphi, ndust=2, noise=1e-2, seed=3, fargo=True, cfl=2.6 if nphi < 200 else 0.8,
                                slope_type=slope, precision=precision)
    dto, dtg, uo, ug, st = run_pair(cfg, u0, 3)
    np.testing.assert_allclose(dtg, dto, rtol=1e-13 if precision == K.PREC_FP64 else 1e-5, atol=0)
    assert rel_l1(cfg, ug, uo).max() <= (FP64_TOL if precision == K.PREC_FP64 else MIXED_TOL)
