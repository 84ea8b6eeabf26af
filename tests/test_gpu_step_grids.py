"""The step kernels at leaf counts around their persistent grids (3 or 4 CTAs
per SM by the number of equations) against the oracle, bit for bit."""
import numpy as np
import pytest

from helpers import compare_blocks, noncorner_mask
from walicxe2d_b200.params import sedov

pytestmark = pytest.mark.gpu


# the smallest pool; under, at (148 x 3 = 444 = 12 x 37, 148 x 4 = 592 = 16 x 37) and over a wave
@pytest.mark.parametrize("neq", [4, 5, 6])
@pytest.mark.parametrize("bx,by", [(2, 2), (17, 26), (12, 37), (5, 89), (16, 37), (593, 1)])
def test_leaf_counts_around_a_wave(neq, bx, by, oracle_lib):
    from walicxe2d_b200.api import Simulation
    p, ic = sedov(nbroot=1, nlevs=1, nblocks=bx * by, neq=neq, npas=neq - 4)
    p.nbroot_x, p.nbroot_y = bx, by
    p.xmax, p.ymax = 1.0, by / bx
    ic.xc, ic.yc, ic.rb = 0.5 * p.xmax, 0.5 * p.ymax, 0.2 * min(p.xmax, p.ymax)
    o = oracle_lib.Oracle(p, ic, threads=8)
    o.startup()
    s = Simulation(p, ic)
    s.ctx.set_graphs(True)
    for _ in range(2):
        dt = o.run(2, amr=False)
        s.run(2)
        assert s.status()["dt"] == dt
    ids = o.leaves()
    dmax, _, n = compare_blocks(s.ctx.get_blocks(ids), o.u[ids], noncorner_mask())
    assert dmax == 0.0 and n == 0, (dmax, n)
