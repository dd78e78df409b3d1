"""Mixed-precision K2 with a run-time species count: its passes take four species at a time.  Counts
around whole chunks, with each kind of drag coefficient (one set a step, per cell) against the oracle,
at the mixed path's tolerance on the same setups."""
import numpy as np
import pytest

from shark_gb300 import config as K, setups
from tests.test_gpu_parity import MIXED_TOL, rel_l1, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndust", [3, 5, 7, 12, 13])
@pytest.mark.parametrize("setup", ["si", "turb", "disk"])
def test_species_counts(setup, ndust):
    if setup == "si":
        cfg, u0 = setups.si(n=20, ndust=ndust, precision=K.PREC_MIXED)
    elif setup == "turb":
        cfg, u0 = setups.dusty_turb(n=20, ndust=ndust, forcing=True, precision=K.PREC_MIXED)
    else:
        cfg, u0 = setups.disk_polar(nr=20, nphi=24, ndust=ndust, noise=1e-2, seed=4, precision=K.PREC_MIXED)
    dto, dtg, uo, ug, st = run_pair(cfg, u0, 4)
    assert st == 0
    np.testing.assert_allclose(dtg, dto, rtol=1e-4)
    assert rel_l1(cfg, ug, uo).max() <= 10 * MIXED_TOL
