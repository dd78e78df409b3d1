"""The dt and status a step posts to the host, and the device-clock phase times."""
import numpy as np
import pytest

from shark_gb300 import config as K, setups
from shark_gb300.solver import Shark

pytestmark = pytest.mark.gpu


def test_posts_after_a_new_upload_and_between_contexts():
    """Steps of two contexts in turn, a timed run in between and the same state uploaded again: every
    step returns its own dt (a post of an earlier step or run is never taken for it)."""
    cfg, u0 = setups.sod(nx=64, ndust=1)
    with Shark(cfg) as a, Shark(cfg) as b:
        a.upload(u0)
        first = [a.solve() for _ in range(6)]
        assert len(set(first)) > 1
        b.upload(u0)
        a.upload(u0)
        for dt in first[:3]:
            assert a.solve() == dt
            assert b.solve() == dt
        a.timed_run(2)
        b.run_steps(2)
        assert a.solve() == b.solve() == first[5]
        a.upload(u0)
        assert a.solve() == first[0]


@pytest.mark.parametrize("precision", [K.PREC_FP64, K.PREC_MIXED])
def test_phase_times(precision):
    cfg, u0 = setups.si(n=256, ndust=4, precision=precision)
    with Shark(cfg) as g:
        g.upload(u0)
        g.run_steps(3)
        ms = g.last_step_ms()
        whole = g.kernel_times(3)[3]
    assert all(t >= 0.0 for t in ms) and ms[1] > 0.0 and ms[2] > 0.0
    assert sum(ms) <= 3.0 * whole      # the clock's phases lie within the step
