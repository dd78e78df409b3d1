"""FP64 column-march flux kernels against the oracle at the edges of their split: one and two rows,
rows and columns one off the strip sizes (28 columns; heights chosen per grid), every limiter and
solver form of the FP64 path.  The path follows the oracle's operations, so the tolerance is the
FP64 parity tolerance."""
import numpy as np
import pytest

from shark_gb300 import config as K, setups
from tests.test_gpu_parity import FP64_TOL, rel_l1, run_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,ndust", [(4, 4, 1), (28, 5, 2), (29, 31, 3), (57, 67, 1), (300, 4, 0), (31, 200, 2)])
@pytest.mark.parametrize("slope,solver,solverdust", [(1, 2, 0), (2, 1, 1), (3, 0, 2), (3, 2, 0)])
def test_adiabatic_box(nx, ny, ndust, slope, solver, solverdust):
    cfg, u0 = setups.kh(n=nx, ny=ny, ndust=ndust, **dict(setups.KH_NML, scut=setups.KH_NML["smax"], slope_type=slope))
    cfg.solver, cfg.solverdust = solver, solverdust
    dto, dtg, uo, ug, st = run_pair(cfg, u0, 4)
    assert st == 0
    np.testing.assert_allclose(dtg, dto, rtol=1e-14, atol=0)
    assert rel_l1(cfg, ug, uo).max() <= FP64_TOL


@pytest.mark.parametrize("n,ndust", [(5, 1), (27, 9), (61, 2)])
@pytest.mark.parametrize("slope,solver,solverdust", [(1, 1, 3), (2, 2, 0), (3, 0, 1)])
def test_isothermal_forced_box(n, ndust, slope, solver, solverdust):
    cfg, u0 = setups.si(n=n, ndust=ndust, slope_type=slope)
    cfg.solver, cfg.solverdust = solver, solverdust
    dto, dtg, uo, ug, st = run_pair(cfg, u0, 4)
    assert st == 0
    np.testing.assert_allclose(dtg, dto, rtol=1e-14, atol=0)
    assert rel_l1(cfg, ug, uo).max() <= FP64_TOL


@pytest.mark.parametrize("n,ndust", [(9, 1), (31, 3)])
@pytest.mark.parametrize("slope,solver,solverdust", [(1, 2, 0), (2, 1, 2), (3, 0, 1), (1, 0, 2), (3, 2, 0)])
def test_not_a_number_spreads_as_in_the_oracle(n, ndust, slope, solver, solverdust):
    # an odd box has the star's softened offsets 0/0 in its middle cell; what is not a number takes
    # the cells of its stencil that the operations take it to, and no others (one step: the cells that
    # are not numbers count differently in the two time steps)
    cfg, u0 = setups.disk_cart(n=n, ndust=ndust, slope_type=slope)
    cfg.solver, cfg.solverdust = solver, solverdust
    assert not np.isfinite(u0).all()
    dto, dtg, uo, ug, st = run_pair(cfg, u0, 1)
    assert st != 0
    np.testing.assert_array_equal(np.isfinite(ug), np.isfinite(uo))
