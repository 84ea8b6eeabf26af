"""coolingh at the edges of its branches against the CPU routine, cell by cell:
the 1000 K floor of ALOSS, the window where the line cooling gives way to the
equilibrium curve, the collision strength's fits, exponents beyond the FP64
range and very short and long steps."""
import numpy as np
import pytest

from walicxe2d_b200.params import snr

pytestmark = pytest.mark.gpu

EDGES = [1.0, 1.5, 10.0, 150.0, 169.0, 225.0, 226.0, 999.0, 1000.0, 1001.0, 1.0e4, 44769.0, 44770.0, 44771.0, 49770.0,
         54769.0, 54770.0, 54771.0, 55000.0, 55001.0, 71999.0, 72000.0, 72001.0, 5.5e6, 5.6e6, 5.8e6, 1.0e8, 1.0e9]


@pytest.mark.parametrize("dt", [1.0, 1.0e6, 1.0e9, 1.0e13])
def test_coolingh_at_branch_edges(dt, oracle_lib):
    from oracle.oracle import atomic
    from walicxe2d_b200.api import Simulation
    p, ic = snr(nbroot=2, nlevs=1, nblocks=4)
    s = Simulation(p, ic)
    s.run(1)                                   # (plans are in place)
    ids = s.leaf_ids()
    rng = np.random.default_rng(17)
    sh = (ids.size, 20, 20)
    T = rng.choice(EDGES, sh) * (1.0 + 1e-4 * rng.choice([-1.0, 0.0, 1.0], sh))
    T = np.maximum(T, 1.0)
    rho = 10.0 ** rng.uniform(-2, 3, sh)
    y = rng.choice([1e-4, 1e-2, 0.5, 0.999, 1.0], sh)
    v = rng.normal(0, 1, (2,) + sh)
    u = np.zeros((ids.size, 6, 20, 20))
    u[:, 0], u[:, 1], u[:, 2], u[:, 4], u[:, 5] = rho, rho * v[0], rho * v[1], rho * y, rho
    u[:, 3] = 1.5 * (rho * (2 - y) * T / p.tempsc) + 0.5 * rho * (v[0] ** 2 + v[1] ** 2)
    s.ctx.put_blocks(ids, u)
    s.ctx.coolingh(dt)
    got = s.ctx.get_blocks(ids)

    c = u[:, :, 2:18, 2:18].transpose(0, 2, 3, 1).reshape(-1, 6)
    g = got[:, :, 2:18, 2:18].transpose(0, 2, 3, 1).reshape(-1, 6)
    want = np.array([atomic(p, dt, c[k].copy()) for k in range(c.shape[0])])
    # Rounding of the neutral fraction: its closed form subtracts terms of size
    # |b| / (2 a y1) of the result (y1 >= 1e-4) and divides by 1 - g0 e, which is
    # about d n dt on short steps; a few dozen roundings of 2^-53 enter each.
    r = c[:, 0]
    t = np.maximum(1.0, (c[:, 3] - 0.5 * r * ((c[:, 1] / r) ** 2 + (c[:, 2] / r) ** 2)) / 1.5 /
                   (2 * r - c[:, 4]) * p.tempsc)
    col = 5.83e-11 * np.sqrt(t) * np.exp(-157828.0 / t)
    rec = 2.55e-13 * (1e4 / t) ** 0.79
    a, b = rec + col, (2 + 1e-4) * rec + (1 + 1e-4) * col
    d = np.sqrt(np.maximum(b * b - 4 * a * (1 + 1e-4) * rec, 1e-300))
    cond = (b + d) / (2 * a) * (1.0 + 1.0 / np.minimum(1.0, d * r * dt)) * (1.0 + b / d)
    eps = 64 * 2.0 ** -53
    y1 = want[:, 4] / r
    dy = np.minimum(eps * cond, 1.0)
    ok = np.abs(g[:, 4] / r - y1) <= dy + 4 * eps * y1
    assert ok.all(), (dt, t[~ok][:5], (g[:, 4] / r - y1)[~ok][:5], dy[~ok][:5])
    # The temperature: T exp(-ce dt) moves by at most 0.37 of the rate's relative
    # error (the neutral density's, plus the exponents' products, below 1e-12);
    # the kinetic energy subtracts from the total once, and the thermal energy
    # carries 2 - y1.
    etot, rel = want[:, 3], 1e-12 + 2.0 * dy / np.maximum(y1, 1e-4)
    ok = np.abs(g[:, 3] - etot) <= np.minimum(rel, 1.0) * c[:, 3] + 1e-12 * np.abs(etot)
    assert ok.all(), (dt, t[~ok][:5], ((g[:, 3] - etot) / etot)[~ok][:5])
    for k in (0, 1, 2, 5):
        np.testing.assert_array_equal(g[:, k], c[:, k])
