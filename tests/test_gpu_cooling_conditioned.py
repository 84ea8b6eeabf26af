"""coolingh at the edges of its branches on cells where both results are well
conditioned, each held to a tight bound: the neutral fraction over about one
ionisation or recombination time, the energy over about one cooling time and
for the neutral fraction that came back."""
import numpy as np
import pytest

from test_gpu_cooling_edges import EDGES
from walicxe2d_b200.params import snr

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def rates(t):
    """a, b, d of the neutral fraction's closed form (src/coolingh.f90:190-200)."""
    col, rec = 5.83e-11 * np.sqrt(t) * np.exp(-157828.0 / t), 2.55e-13 * (1e4 / t) ** 0.79
    a, b = rec + col, (2 + 1e-4) * rec + (1 + 1e-4) * col
    return a, b, np.sqrt(b * b - 4 * a * (1 + 1e-4) * rec)


def cooling_rate(oracle, t, y0, r, dh0):
    """ce of src/coolingh.f90:232: t1 = 10 + (t - 10) exp(-ce dt)."""
    al = oracle.aloss(y0, 0.0, 0.0, r, dh0, t) / (r * r)
    return (2.0 * r * al) / (3.0 * 1.3807e-16 * t)


def cells(p, edge, n, rng):
    """n blocks at rest near temperature `edge`."""
    sh = (n, 20, 20)
    t = np.maximum(edge * (1.0 + 1e-4 * rng.choice([-1.0, 0.0, 1.0], sh)), 1.0)
    rho = 10.0 ** rng.uniform(-0.5, 0.5, sh)
    y = rng.choice([1e-4, 1e-2, 0.5, 0.999, 1.0], sh)
    u = np.zeros((n, 6, 20, 20))
    u[:, 0], u[:, 4], u[:, 5] = rho, rho * y, rho
    u[:, 3] = p.cv * (rho * (2 - y) * t / p.tempsc)
    return u


def interior(u):
    return u[:, :, 2:18, 2:18].transpose(0, 2, 3, 1).reshape(-1, 6)


def temperature(p, c):
    """uprim's, in its operation order (src/uprim.f90:30-40)."""
    dent = 2.0 * c[:, 0] - c[:, 4]
    return np.maximum(1.0, np.maximum(c[:, 3] / p.cv, 1e-15) / dent * p.tempsc)


def fraction_bound(t, r, dt):
    """Rounding of the neutral fraction: its closed form subtracts terms of size
    (b + d) / 2a and divides by 1 - g0 e, which is about d r dt on short steps
    and itself the difference of terms b / d larger; a few dozen roundings."""
    a, b, d = rates(t)
    return 64 * EPS * (b + d) / (2 * a) * (1.0 + 1.0 / np.minimum(1.0, d * r * dt)) * (1.0 + b / d)


def energy(oracle, p, c, g, dt):
    """The energy that belongs to the neutral densities g[:, 4]."""
    t = temperature(p, c)
    ce = np.array([cooling_rate(oracle, t[k], c[k, 4] / c[k, 0], c[k, 0], g[k, 4]) for k in range(t.size)])
    t1 = 10.0 + (t - 10.0) * np.exp(-ce * dt)
    t1 = np.maximum(np.minimum(np.maximum(t1, 0.1 * t), 10.0 * t), 10.0)
    return t, t1, p.cv * (2.0 * c[:, 0] - g[:, 4]) * t1 / p.tempsc


def steps(oracle, edge):
    """One time of the neutral fraction and one of the temperature."""
    return 1.0 / rates(max(edge, 1.0))[0], 1.0 / cooling_rate(oracle, max(edge, 1.0), 0.5, 1.0, 0.5)


@pytest.mark.parametrize("edge", EDGES)
def test_coolingh_where_it_is_well_conditioned(edge, oracle_lib):
    from oracle import oracle
    from walicxe2d_b200.api import Simulation
    p, ic = snr(nbroot=2, nlevs=1, nblocks=4)
    s = Simulation(p, ic)
    s.run(1)                                   # (plans are in place)
    ids = s.leaf_ids()
    rng = np.random.default_rng(int(edge))
    u = cells(p, edge, ids.size, rng)
    c, moved = interior(u), []
    for k, dt in enumerate(steps(oracle, edge)):
        s.ctx.put_blocks(ids, u)
        s.ctx.coolingh(dt)
        g = interior(s.ctx.get_blocks(ids))
        t, t1, e = energy(oracle, p, c, g, dt)
        # exponents of up to 160, each rounded, and a handful of products: below
        # 1e-13 of the rate, times ce dt, of which exp(-ce dt) leaves at most 0.4
        np.testing.assert_allclose(g[:, 3], e, rtol=1e-12, atol=0.0)
        if k == 0:
            y = np.array([oracle.atomic(p, dt, x.copy())[4] for x in c]) / c[:, 0]
            dy = fraction_bound(t, c[:, 0], dt)
            assert dy.max() < 1e-5             # (every cell is held to that)
            assert (np.abs(g[:, 4] / c[:, 0] - y) <= dy + 4 * EPS * y).all()
        moved.append(np.mean((np.abs(t1 / t - 1.0) > 1e-3) & (t1 > 0.1001 * t)))
    assert edge <= 20.0 or max(moved) > 0.15   # (many temperatures move, and not to their clamps)
