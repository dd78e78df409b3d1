"""Phase times of the last step (shark_gpu_last_step_ms) beside calls that are no step."""
import pytest

from shark_gb300 import config as K, setups
from shark_gb300.solver import Shark

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, K.CHARGE_ANALYTICAL])
def test_charging_outside_a_step_leaves_them(mode):
    cfg, u0 = setups.dusty_turb(n=8, ndust=2, charging=True)
    cfg.chg_mode |= mode
    with Shark(cfg) as g:
        g.upload(u0)
        g.solve()
        ms = g.last_step_ms()
        g.charge()
        assert g.last_step_ms() == ms
    assert all(t >= 0.0 for t in ms) and ms[0] > 0.0


def test_forcing_update_precedes_the_flux_phase():
    """The flux phase begins when the forcing's update has ended: it takes what the flux kernel takes
    between two events (which bracket the launch too), the least of five steps."""
    cfg, u0 = setups.dusty_turb(n=128, ndust=4, forcing=True, precision=K.PREC_MIXED)
    with Shark(cfg) as g:
        g.upload(u0)
        g.run_steps(3)
        flux = []
        for _ in range(5):
            g.solve()
            flux.append(g.last_step_ms()[1])
        kernel = g.kernel_times(5)[1]
    assert min(flux) <= 1.2 * kernel
