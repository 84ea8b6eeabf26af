"""The first queued steps of a context cost what later ones do: they allocate
nothing and prepare nothing (as they did: 300 us for two steps of 4x4 blocks,
89 from then on)."""
import statistics
import time

import pytest

from walicxe2d_b200.params import sedov

pytestmark = pytest.mark.gpu


def test_first_queue_of_a_context():
    from walicxe2d_b200.api import Simulation
    first, later = [], []
    for _ in range(15):
        s = Simulation(*sedov(nbroot=4, nlevs=1))
        s.ctx.set_graphs(True)
        s.run(1)
        for out in (first, later, later):
            t0 = time.perf_counter()
            s.run(2)
            out.append(time.perf_counter() - t0)
        s.close()
    assert statistics.median(first) < 2.0 * statistics.median(later)
