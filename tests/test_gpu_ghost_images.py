"""Ghost images written by the step's last kernel, a block's threads sharing the ends of its row: row
lengths at which the edge columns fall into one block of 128 columns, straddle two, or leave a block
with a single column, for each kind of boundary and both precisions, against the oracle over enough
steps that every ghost is used.  The tolerances are the parity tolerances."""
import numpy as np
import pytest

from shark_gb300 import config as K, setups
from tests.test_gpu_parity import FP64_TOL, MIXED_TOL, rel_l1, run_pair

pytestmark = pytest.mark.gpu


def _setup(name, nx, precision):
    if name == "si":
        return setups.si(n=nx, ndust=3, precision=precision)
    if name == "kh":
        return setups.kh(n=nx, ny=10, ndust=2, precision=precision, **dict(setups.KH_NML, scut=setups.KH_NML["smax"]))
    if name == "polar":
        return setups.disk_polar(nr=nx, nphi=10, ndust=2, noise=1e-2, seed=5, precision=precision)
    if name == "cart":
        cfg, _ = setups.disk_cart(n=nx, ndust=2, precision=precision)
        cfg.ny = 10
        return cfg, setups.disk_cart_ic(cfg)
    return setups.sod(nx=nx, ndust=2, precision=precision)


@pytest.mark.parametrize("nx", [126, 127, 128, 129, 130, 257])
@pytest.mark.parametrize("name", ["si", "kh", "polar", "cart", "sod"])
@pytest.mark.parametrize("precision", [K.PREC_FP64, K.PREC_MIXED])
def test_row_lengths(name, nx, precision):
    cfg, u0 = _setup(name, nx, precision)
    dto, dtg, uo, ug, st = run_pair(cfg, u0, 3)
    fp64 = precision == K.PREC_FP64
    np.testing.assert_allclose(dtg, dto, rtol=1e-13 if fp64 else 1e-4)
    assert rel_l1(cfg, ug, uo).max() <= (FP64_TOL if fp64 else 10 * MIXED_TOL)
