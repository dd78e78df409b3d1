"""Mixed dust growth of two contexts of different species counts (and so of different shared memory a
block) stepped by two threads at once: as each steps alone."""
import threading

import numpy as np
import pytest

from shark_gb300 import config as K, setups
from shark_gb300.solver import Shark

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(17, 32), (2, 16)])
def test_two_threads(counts):
    steps = 4000

    def run(ndust, out):
        try:
            cfg, u0 = setups.dusty_turb(n=8, ndust=ndust, nH=1e3, growth=True, precision=K.PREC_MIXED)
            with Shark(cfg) as g:
                g.upload(u0)
                g.run_steps(steps)
                out.append(g.download())
        except Exception as e:      # handed to the test's thread
            out.append(e)

    alone, together = [[] for _ in counts], [[] for _ in counts]
    for n, out in zip(counts, alone):
        run(n, out)
    threads = [threading.Thread(target=run, args=(n, out)) for n, out in zip(counts, together)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for (a,), (b,) in zip(alone, together):
        assert not isinstance(a, Exception), a
        assert not isinstance(b, Exception), b
        np.testing.assert_array_equal(a, b)
