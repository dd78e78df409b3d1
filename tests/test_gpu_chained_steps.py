"""Steps whose kernels come in while their predecessors drain against the same steps with an event
between every two kernels (kernel_times), which run one after the other: the same operations on the
same data, so the same bits."""
import numpy as np
import pytest

from shark_gb300 import config as K, setups
from shark_gb300.solver import Shark

pytestmark = pytest.mark.gpu


def _setup(name, n, precision):
    if name == "sod":
        return setups.sod(nx=n, ndust=2, precision=precision)
    if name == "si":
        return setups.si(n=n, ndust=3, precision=precision)
    if name == "sedov":
        return setups.sedov(n=n, precision=precision)
    return setups.kh(n=n, ny=n // 2 + 3, ndust=2, precision=precision, **dict(setups.KH_NML, scut=setups.KH_NML["smax"]))


@pytest.mark.parametrize("name", ["sod", "si", "sedov", "kh"])
@pytest.mark.parametrize("n", [16, 131, 600])
@pytest.mark.parametrize("precision", [K.PREC_FP64, K.PREC_MIXED])
def test_same_state_as_one_kernel_at_a_time(name, n, precision):
    cfg, u0 = _setup(name, n, precision)
    steps = 12
    with Shark(cfg) as g:
        g.upload(u0)
        g.kernel_times(steps)
        apart = g.download()
        for _ in range(2):
            g.upload(u0)
            g.run_steps(steps)
            np.testing.assert_array_equal(g.download(), apart)
