"""The FP64 forms of shark_gb300/csrc/fp64.cuh (quotients from a reciprocal, compares and conversions on
the bit patterns) and the FP64 limiters against the plain operations on the host, and a run that
takes the quotients below the normal range.

Quotients: bit for bit on operands well inside the range.  Elsewhere, where a first product or a
residual that underflows leaves the last correction out, the product stands: the reciprocal's
error (an ulp) and its own rounding put it within two units in the last place, and zeros, infinities
and not-a-numbers are those of the division."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from shark_gb300 import build as B, config as K, setups
from oracle.oracle import Oracle
from tests.test_gpu_parity import active, run_pair

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
OPS = ("div", "rcp", "min", "max", "less", "minmod", "van_leer", "mc", "narrow", "widen")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fp64") / "fp64_check.so")
    subprocess.run([B.nvcc(), *B.ARCH, *B.COMMON, "--fmad=false", "-I" + B.CSRC, "-shared", "-o", so,
                    os.path.join(HERE, "fp64_check.cu")], check=True)
    fn = ctypes.CDLL(so).fp64_check
    P = ctypes.POINTER(ctypes.c_double)

    def run(a, b):
        a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
        out = np.empty((len(OPS), a.size))
        rc = fn(ctypes.c_int(a.size), a.ctypes.data_as(P), b.ctypes.data_as(P), out.ctypes.data_as(P))
        assert rc == 0
        return dict(zip(OPS, out))
    return run


def _random(rng, n, lo, hi):
    """Random sign and mantissa, exponents in [lo, hi)."""
    return rng.choice([-1.0, 1.0], n) * np.ldexp(1.0 + rng.random(n), rng.integers(lo, hi, n))


def _same(x, y):
    """Bit for bit, every not-a-number alike."""
    nan = np.isnan(x) & np.isnan(y)
    return nan | (x.view(np.int64) == y.view(np.int64))


def _key(x):
    b = x.view(np.int64)
    return np.where(b < 0, np.int64(-2**63) - b, b)


SPECIAL = np.array([0.0, 5e-324, 3e-310, 2.2250738585072009e-308, 2.2250738585072014e-308, 3e-308, 4e-300, 1e-200, 1e-30,
                    0.3, 1.0, 1.5, 7.0, 1e30, 1e200, 1e300, 4.4e307, 4.5e307, 1.7e308, 1.7976931348623157e308, np.inf])
SPECIAL = np.concatenate([SPECIAL, -SPECIAL, [np.nan]])


def test_quotients_inside_the_range(check):
    rng = np.random.default_rng(1)
    a, b = _random(rng, 1 << 20, -480, 480), _random(rng, 1 << 20, -480, 480)
    got = check(a, b)
    assert _same(got["div"], a / b).all()
    assert np.abs(_key(got["rcp"]) - _key(1.0 / b)).max() <= 1


def test_quotients_at_the_ends_of_the_range(check):
    a, b = (x.ravel() for x in np.meshgrid(SPECIAL, SPECIAL))
    rng = np.random.default_rng(2)
    wide = [_random(rng, 1 << 16, -1074, 1024) for _ in range(2)]
    a, b = np.concatenate([a, wide[0]]), np.concatenate([b, wide[1]])
    with np.errstate(all="ignore"):
        want, inv = a / b, 1.0 / b
    got = check(a, b)
    for x, y, ulps in ((got["div"], want, 2), (got["rcp"], inv, 1)):
        np.testing.assert_array_equal(np.isnan(x), np.isnan(y))
        ok = ~np.isnan(y)
        np.testing.assert_array_equal(np.signbit(x[ok]), np.signbit(y[ok]))
        assert np.abs(_key(x[ok]) - _key(y[ok])).max() <= ulps


def test_compares(check):
    a, b = (x.ravel() for x in np.meshgrid(SPECIAL, SPECIAL))
    got = check(a, b)
    differ = ~((a == 0.0) & (b == 0.0))        # -0 orders below +0
    assert np.array_equal(got["less"][differ] != 0.0, (a < b)[differ])
    assert _same(got["min"], np.where(a < b, a, b))[differ].all()
    assert _same(got["max"], np.where(a > b, a, b))[differ].all()


def test_limiters(check):
    """slope_limiters.f90's operations, for slopes whose product does not underflow."""
    rng = np.random.default_rng(3)
    ordinary = np.concatenate([SPECIAL[(np.abs(SPECIAL) > 1e-100) & (np.abs(SPECIAL) < 1e100) | (SPECIAL == 0.0)], [np.inf, -np.inf, np.nan]])
    a, b = (x.ravel() for x in np.meshgrid(ordinary, ordinary))
    a = np.concatenate([a, _random(rng, 1 << 18, -60, 60), _random(rng, 1 << 18, 0, 1)])
    b = np.concatenate([b, _random(rng, 1 << 18, -60, 60), _random(rng, 1 << 18, 0, 1)])
    got = check(a, b)
    with np.errstate(all="ignore"):
        minmod = np.where(a * b < 0.0, 0.0, np.where(np.abs(b) < np.abs(a), b, a))
        van_leer = np.where(a * b <= 0.0, 0.0, 2.0 * a * b / (a + b))
        c = 0.5 * (a + b)
        l, r = 1.5 * np.abs(a), 1.5 * np.abs(b)
        lim = np.where(a * b <= 0.0, 0.0, np.where(l < r, l, r))
        mc = np.where(np.signbit(c), -1.0, 1.0) * np.where(lim < np.abs(c), lim, np.abs(c))
    for name, want in (("minmod", minmod), ("van_leer", van_leer), ("mc", mc)):
        same = _same(got[name], want) | ((got[name] == 0.0) & (want == 0.0))   # zeros of either sign
        assert same.all(), (name, a[~same][:5], b[~same][:5], got[name][~same][:5], want[~same][:5])


def test_conversions(check):
    rng = np.random.default_rng(4)
    f = rng.integers(0, 1 << 32, 1 << 18, dtype=np.uint64).astype(np.uint32).view(np.float32)
    f = np.concatenate([f, np.array([0x00000001, 0x007fffff, 0x00800000, 0x7f7fffff, 0x7f800000], np.uint32).view(np.float32)])
    with np.errstate(all="ignore"):
        x = f.astype(np.float64)
        up = np.nextafter(f, np.float32(np.inf)).astype(np.float64)
        tie = np.where(np.isfinite(up) & np.isfinite(x), 0.5 * (x + up), x)
        d = np.concatenate([x, tie, np.nextafter(tie, np.inf), np.nextafter(tie, -np.inf), SPECIAL,
                            [np.finfo(np.float32).max * (1.0 + 2.0**-25), np.finfo(np.float32).max * (1.0 + 2.0**-24)]])
        want = d.astype(np.float32).astype(np.float64)
    got = check(d, d)
    assert _same(got["narrow"], want).all()
    assert _same(got["widen"], want).all()


# ---------------------------------------------------------------------------------------------
# dust at rest but for velocities below the normal range: what a drag without back reaction leaves
# of them in a gas at rest after some hundred stopping times
# ---------------------------------------------------------------------------------------------
def _slow_dust(cfg, u0, v):
    """The gas at rest and uniform, dust velocities of random sign and a modulus up to v."""
    rng = np.random.default_rng(5)
    u = u0.reshape(cfg.nvar, -1)
    N = cfg.ndust
    u[1:4] = 0.0
    u[0], u[4] = u[0].max(), u[4].max()
    for k in range(N):
        u[5 + k] = 0.1 * u[0] * (1.0 + 0.2 * rng.random(u.shape[1]))
        for c in (1, 2, 3):
            u[5 + c * N + k] = u[5 + k] * (v * (2.0 * rng.random(u.shape[1]) - 1.0))
    return u.reshape(-1)


@pytest.mark.parametrize("solverdust", [0, 1, 2])
@pytest.mark.parametrize("drag", [False, True])
@pytest.mark.parametrize("ny", [1, 24])
def test_dust_velocities_below_the_normal_range(ny, drag, solverdust):
    if ny == 1:
        cfg, u0 = setups.sod(nx=80, ndust=2, rho_r=1.0, P_r=1.0, slope_type=0)
    else:
        cfg, u0 = setups.kh(n=31, ny=ny, ndust=2, **dict(setups.KH_NML, scut=setups.KH_NML["smax"], slope_type=0))
    cfg.solverdust = solverdust
    cfg.flags = K.FLAG_DRAG if drag else 0
    v = 1e-309
    u0 = _slow_dust(cfg, u0, v)
    rho_max = u0.reshape(cfg.nvar, -1)[5:7].max()
    dto, dtg, uo, ug, st = run_pair(cfg, u0, 3)
    assert st == 0
    np.testing.assert_allclose(dtg, dto, rtol=1e-14, atol=0)
    a, b = active(cfg, ug), active(cfg, uo)
    assert np.isfinite(a).all() and np.isfinite(b).all()
    np.testing.assert_allclose(a[:7], b[:7], rtol=1e-14, atol=0)
    # the momenta stay of the order of rho v on both sides
    np.testing.assert_allclose(a[7:], b[7:], rtol=0, atol=1e2 * rho_max * v)


@pytest.mark.parametrize("solverdust", [0, 1])
def test_dust_density_below_the_normal_range(solverdust):
    """Without drag nothing floors a dust density; a cell's velocity stays that of its momentum."""
    cfg, u0 = setups.sod(nx=80, ndust=1, rho_r=1.0, P_r=1.0, slope_type=0)
    cfg.solverdust, cfg.flags = solverdust, 0
    u0 = _slow_dust(cfg, u0, 0.1)
    u = u0.reshape(cfg.nvar, -1)
    f = np.where(np.arange(u.shape[1]) // 8 % 2 == 0, 1e-309 / 0.1, 1.0)
    u[5:] *= f
    dto, dtg, uo, ug, st = run_pair(cfg, u0, 1)
    assert st == 0
    np.testing.assert_allclose(dtg, dto, rtol=1e-14, atol=0)
    a, b = active(cfg, ug), active(cfg, uo)
    assert np.isfinite(a).all()
    np.testing.assert_allclose(a, b, rtol=1e-12, atol=1e-305)


@pytest.mark.parametrize("setup", ["sod", "si"])
def test_stopping_times_below_the_normal_range(setup):
    """dt/t_k near the largest number: 1 + dt/t_k has a reciprocal below the normal range, the drag's
    weight is 1 and the dust moves with the gas."""
    if setup == "sod":
        cfg, u0 = setups.sod(nx=64, ndust=2, rho_r=1.0, P_r=1.0)
    else:
        cfg, u0 = setups.si(n=16, ndust=2)
    u = u0.reshape(cfg.nvar, -1)
    u[7:9] += 0.01 * u[5:7]          # the dust's x velocities
    o = Oracle(cfg)
    o.set_u(u0)
    ts = o.solve() / 8e307
    for k in range(2):
        if setup == "si":
            cfg.dust_tstop[k] = ts
        else:                         # t = sqrt(pi gamma / 8) rhograin s / (rho c_s) with rho = P = 1
            cfg.dust_size[k] = ts * np.sqrt(cfg.gamma) / (np.sqrt(np.pi * cfg.gamma / 8.0) * cfg.rhograin)
    dto, dtg, uo, ug, st = run_pair(cfg, u0, 1)
    assert st == 0
    np.testing.assert_allclose(dtg, dto, rtol=1e-14, atol=0)
    assert np.isfinite(uo).all()
    np.testing.assert_allclose(active(cfg, ug), active(cfg, uo), rtol=1e-12, atol=1e-15)
