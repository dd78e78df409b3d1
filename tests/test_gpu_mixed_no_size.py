"""A dust species without a size (a configuration that left it out): its stopping time is zero, and the
step's status says so in either precision."""
import pytest

from shark_gb300 import config as K, setups
from shark_gb300.solver import Shark

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [K.PREC_FP64, K.PREC_MIXED])
@pytest.mark.parametrize("ndust", [1, 3])
def test_grains_without_a_size(precision, ndust):
    cfg, u0 = setups.sod(nx=40, ndust=ndust, precision=precision)
    cfg.dust_size[ndust - 1] = 0.0
    with Shark(cfg) as g:
        g.upload(u0)
        g.run_steps(2)
        assert g.sync() & K.STATUS_NAN
