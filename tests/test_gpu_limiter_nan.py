"""A velocity that is not a number reaches through the minmod slopes exactly as
far as src/limiter.f90:38-43 lets it: cells whose right-hand differences hold
it, whatever the sign of their left-hand ones, become NaN with it."""
import numpy as np
import pytest

from walicxe2d_b200.params import HLL, config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1])
def test_nan_through_minmod(oracle_lib, axis):
    from walicxe2d_b200.api import Simulation
    p, ic = config("sedov64")
    p.solver, p.limiter = HLL, 1           # (HLL has no stop on NaN)
    o = oracle_lib.Oracle(p, ic, threads=4)
    o.startup()
    s = Simulation(p, ic)
    s.run(1)                               # (plans are in place)
    ids = o.leaves()
    rng = np.random.default_rng(3)
    sh = (ids.size, 20, 20)
    rho, pr = 1.0 + rng.uniform(0, 1, sh), 1.0 + rng.uniform(0, 1, sh)
    v = rng.normal(0, 0.1, (2,) + sh)      # slopes of both signs in every component
    u = np.zeros((ids.size, 4, 20, 20))
    u[:, 0], u[:, 1], u[:, 2] = rho, rho * v[0], rho * v[1]
    u[:, 3] = 1.5 * pr + 0.5 * rho * (v[0] ** 2 + v[1] ** 2)
    at = (slice(None), 1 + axis) + ((slice(None), 12) if axis == 0 else (12, slice(None)))
    u[at] = np.nan
    o.u[ids] = u
    o.boundaryI()
    o.calcprim()
    u = o.u[ids].copy()
    s.ctx.put_blocks(ids, u)
    o.tstep(0.0, 1e-4)
    s.ctx.tstep(0.0, 1e-4)
    # Cells 6..12 (tile index) before the NaN; those behind it take the sign of a
    # NaN into their slopes (as the left-hand difference), which no standard fixes.
    a, b = (x[:, :, 2:18, 6:12] if axis == 0 else x[:, :, 6:12, 2:18] for x in (s.ctx.get_blocks(ids), o.u[ids]))
    np.testing.assert_array_equal(a, b)
    # the half step carries it one cell, the slopes two
    line = np.isnan(b).any(axis=(0, 1, 2 if axis == 0 else 3))
    np.testing.assert_array_equal(line, [False, False, False, True, True, True])
