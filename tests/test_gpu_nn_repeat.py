"""Training on one tile at a time gives the same network again, whatever else
the process has on the GPU."""
import numpy as np
import pytest

from walicxe2d_b200.params import ensemble_members

pytestmark = pytest.mark.gpu


def test_one_tile_training_repeats():
    from walicxe2d_b200.api import Ensemble, Surrogate
    weights = []
    for k in range(8):
        e = Ensemble(ensemble_members(count=4 + 4 * (k % 3), precision=32)) if k else None
        nn = Surrogate(20261203)
        nn.samples(1 << 14, seed=20261203)
        nn.train(2, batch=128, lr=2e-3, lr_end=2e-5)
        weights.append(nn.params())
        if e:
            e.run(3)
    for w in weights[1:]:
        np.testing.assert_array_equal(w, weights[0])
