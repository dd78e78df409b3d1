"""Mixed-precision column march against the oracle where its strips are shortest and where they do not
divide the box: two-row gas strips, four-row dust strips with shorter gas strips beside them, a column
past a strip's 28.  The tolerances are those of the mixed path on the same setups."""
import numpy as np
import pytest

from shark_gb300 import config as K, setups
from tests.test_gpu_parity import MIXED_TOL, rel_l1, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 29, 57, 151])
@pytest.mark.parametrize("slope,solver", [(1, 2), (2, 1), (3, 0)])
def test_gas_alone(n, slope, solver):
    cfg, u0 = setups.sedov(n=n, slope_type=slope, precision=K.PREC_MIXED)
    cfg.solver = solver
    dto, dtg, uo, ug, st = run_pair(cfg, u0, 3)
    assert st == 0
    np.testing.assert_allclose(dtg, dto, rtol=1e-4)
    assert rel_l1(cfg, ug, uo).max() <= 10 * MIXED_TOL


@pytest.mark.parametrize("nr,nphi,ndust", [(5, 6, 1), (29, 35, 3), (56, 133, 2), (300, 9, 5)])
@pytest.mark.parametrize("slope", [1, 3])
def test_dust_and_gas(nr, nphi, ndust, slope):
    cfg, u0 = setups.disk_polar(nr=nr, nphi=nphi, ndust=ndust, noise=1e-2, seed=6, slope_type=slope, precision=K.PREC_MIXED)
    dto, dtg, uo, ug, st = run_pair(cfg, u0, 3)
    np.testing.assert_allclose(dtg, dto, rtol=1e-5)
    assert rel_l1(cfg, ug, uo).max() <= MIXED_TOL
