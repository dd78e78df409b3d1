"""Charging where the column shields the ions: the inner rings of a massive polar disk, whose ionisation
falls by exp(-Sigma / 96 g cm-2).  The charge balance then has its root at psi -> -0."""
import numpy as np
import pytest

from shark_gb300 import config as K, setups
from shark_gb300.solver import Shark
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mass", [2, 3, 5, 8])
def test_fp64_converges_where_the_oracle_does(mass):
    """The residual is proportional to psi there, so that two psi that meet |f| < 1e-6 lie within 2e-6 of
    each other."""
    cfg, u0 = setups.disk_polar_au(nr=96, nphi=8, ndust=6)
    u0 = mass * u0
    o = Oracle(cfg)
    o.set_u(u0)
    o.apply_boundaries()
    conv = o.charge() < cfg.chg_nitermax
    co = o.get_charge()
    with Shark(cfg) as g:
        g.upload(u0)
        g.charge()
        cg = g.download_charge()
    np.testing.assert_array_equal(cg["iters"] < cfg.chg_nitermax, conv)
    np.testing.assert_allclose(cg["psi"][conv], co["psi"][conv], rtol=2e-6, atol=0)


def test_mixed_converges_where_fp64_does():
    """A cold and a warm call, the second at a tenth more mass; the mixed charging's tolerance.  (The
    smooth disk: beside it some cells lie where the FP32 sums no longer resolve the root.)"""
    out = {}
    for precision in (K.PREC_FP64, K.PREC_MIXED):
        cfg, u0 = setups.disk_polar_au(nr=96, nphi=8, ndust=6, noise=0.0, precision=precision)
        with Shark(cfg) as g:
            for mass in (3.5, 3.85):
                g.upload(mass * u0)
                g.charge()
            out[precision] = g.download_charge()
    a, b = out[K.PREC_MIXED], out[K.PREC_FP64]
    conv = b["iters"] < cfg.chg_nitermax
    np.testing.assert_allclose(a["psi"][conv], b["psi"][conv], rtol=1e-4, atol=0)
    assert (a["iters"][conv] < cfg.chg_nitermax).all()
