"""Drag and drag heating of an adiabatic gas in mixed precision against the oracle for every form of
the species loop: fewer species than a chunk of loads, whole chunks, run-time counts.  The tolerance is
that of the mixed path on the same setup."""
import numpy as np
import pytest

from shark_gb300 import config as K, setups
from tests.test_gpu_parity import MIXED_TOL, rel_l1, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndust", [1, 2, 3, 4, 8, 9, 16])
def test_species_counts(ndust):
    kw = dict(setups.KH_NML, scut=setups.KH_NML["smax"]) if ndust == 1 else setups.KH_NML
    cfg, u0 = setups.kh(n=33, ny=18, ndust=ndust, precision=K.PREC_MIXED, **kw)
    dto, dtg, uo, ug, st = run_pair(cfg, u0, 6)
    assert st == 0
    np.testing.assert_allclose(dtg, dto, rtol=1e-4)
    assert rel_l1(cfg, ug, uo).max() <= 10 * MIXED_TOL
