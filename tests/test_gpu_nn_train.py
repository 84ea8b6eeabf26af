"""Training steps on batches of several tiles against the CPU restatement of
the network: the loss of the first batch, the direction of Adam's first step,
and that the same training repeats bit for bit."""
import os

import numpy as np
import pytest

from oracle import nn_oracle as nno
from walicxe2d_b200.params import jet

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


def _mix(x):
    with np.errstate(over="ignore"):
        x = x + np.uint64(0x9E3779B97F4A7C15)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return x ^ (x >> np.uint64(31))


def _samples(n, seed, tab, p):
    """The coolingdmc training set: n, T log-uniform from the counter hash, the
    rate from the table (src/coolingdmc.f90:30-40, src/dmc_module.f90:14-32)."""
    k = _mix(np.uint64(seed) ^ _mix(np.arange(n, dtype=np.uint64)))
    with np.errstate(over="ignore"):
        u = [(_mix(k + np.uint64(q)) >> np.uint64(11)).astype(np.float64) / 2.0 ** 53 for q in (1, 2)]
    dens, T = 10.0 ** (-2 + 6 * u[0]), 10.0 ** (4.0 + 4.0 * u[1])
    t, lam = 10.0 ** tab[:, 0], 10.0 ** (-tab[:, 1])
    i = np.clip((np.log10(T) * 10).astype(int) - 39, 1, 40)
    c = (lam[i] - lam[i - 1]) * (T - t[i - 1]) / (t[i] - t[i - 1]) + lam[i - 1]
    ce = c * dens ** 2 / (p.cv * (dens * T / p.tempsc) * p.psc)
    X = np.zeros((n, 4))
    X[:, 0], X[:, 1] = (np.log10(dens) - 1) / 3, (np.log10(T) - 5) / 3
    Y = np.zeros((n, 2))
    Y[:, 1] = (np.log10(ce / dens) + 12.5) / 3.5
    return X.astype(np.float32).astype(np.float64), Y.astype(np.float32).astype(np.float64)


# two tiles, an odd count, the usual batch, and more tiles than SMs
@pytest.mark.parametrize("batch", [256, 640, 8192, 149 * 128])
def test_first_step_of_a_batch_of_tiles(batch):
    from walicxe2d_b200.api import Surrogate
    tab = np.loadtxt(os.path.join(GOLDEN, "coolingDMC.tab"))
    p, _ = jet(nlevs=1, nblocks=256)
    out = []
    for _ in range(2):
        nn = Surrogate(11)
        w0 = nn.params()
        nn.samples_dmc(batch, tab[:, 0], tab[:, 1], p, seed=99)
        loss = nn.train(1, batch=batch, lr=1e-3, lr_end=1e-3)
        out.append((loss, nn.params()))
    assert out[0][0] == out[1][0]
    np.testing.assert_array_equal(out[0][1], out[1][1])
    X, Y = _samples(batch, 99, tab, p)
    want, g = nno.loss_grad(w0, X, Y, bf=True)
    # (the bounds of the single gradient's test: BF16 rounding points agree, FP32
    # sums differ; a step is lr g / |g| wherever g is not small)
    assert abs(out[0][0] - want) <= 1e-3 * abs(want)
    step = (w0.astype(np.float64) - out[0][1]) / 1e-3
    big = np.abs(g) > 0.05 * np.abs(g).max()
    assert big.sum() > 20
    np.testing.assert_allclose(step[big], np.sign(g[big]), atol=1e-2)
