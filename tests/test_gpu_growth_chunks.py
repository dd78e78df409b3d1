"""Mixed-precision dust growth (chunks of 4 cells, two at a time, one warp per cell) at the sizes where
its layout changes: grids narrower than a chunk, odd numbers of cells, one bin, sixteen bins and
one more (5 and 17 pairs a lane), the most.  Against the FP64 path on the same state after one
step; the mixed growth tolerance, and the dust mass to 1e-5."""
import numpy as np
import pytest

from shark_gb300 import config as K, setups
from shark_gb300.solver import Shark
from tests.test_gpu_growth import GROWTH_MIXED_TOL
from tests.test_gpu_parity import active, rel_l1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ndust", [(4, 1), (5, 2), (7, 16), (13, 17), (6, 32), (33, 9)])
def test_growth_mixed_chunks(n, ndust):
    out = {}
    for precision in (K.PREC_FP64, K.PREC_MIXED):
        cfg, u0 = setups.dusty_turb(n=n, ndust=ndust, nH=1e10, smin=1e-5, smax=1e-2, growth=True, precision=precision)
        with Shark(cfg) as g:
            g.upload(u0)
            g.solve()
            out[precision] = g.download()
            assert g.sync() == 0
    a, b = out[K.PREC_MIXED], out[K.PREC_FP64]
    assert rel_l1(cfg, a, b).max() <= GROWTH_MIXED_TOL
    A, B = active(cfg, a)[5:5 + ndust], active(cfg, b)[5:5 + ndust]
    assert abs(A.sum() / B.sum() - 1.0) <= 1e-5
    assert np.isfinite(a).all()
