"""A failed step ends the queue of an ensemble, with its step graphs and
without: the state and the clocks are those of steps taken one at a time."""
import numpy as np
import pytest

from walicxe2d_b200 import _lib
from walicxe2d_b200.params import ensemble_members

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("bad_run", [0, 2])
@pytest.mark.parametrize("graphs", [False, True])
def test_a_failed_step_ends_the_queue_of_an_ensemble(graphs, bad_run, precision):
    from walicxe2d_b200.api import Ensemble
    mem = ensemble_members(count=3, precision=precision)
    for p, _ in mem:
        p.nblocks = min(p.nblocks, 2000)
    got, ens = [], []
    for at_once in (True, False):
        e = Ensemble(mem, threads=2)
        e.ctx.set_graphs(graphs)
        e.run(3)
        e.set_amr(False)
        e.run(2)
        ids = (e.leaves(bad_run) + e.slots(bad_run)[0]).astype(np.int32)
        u = e.ctx.get_blocks(ids)
        u[ids.size // 2, 3, 9, 9] = np.inf     # a NaN contact speed
        e.ctx.put_blocks(ids, u)
        with pytest.raises(_lib.W2dException) as err:
            for _ in range(1 if at_once else 5):
                e.run(5 if at_once else 1)
        got.append((err.value.code, [e.status(r) for r in range(3)], e.status()["steps"],
                    np.concatenate([e.blocks(r)[1] for r in range(3)])))
        ens.append(e)
    assert got[0][:3] == got[1][:3]
    np.testing.assert_array_equal(got[0][3], got[1][3])
    for e in ens:                              # a sound state runs on
        for r in range(3):
            ids = (e.leaves(r) + e.slots(r)[0]).astype(np.int32)
            u = e.ctx.get_blocks(ids)
            u[:] = 0.0
            u[:, 0], u[:, 3], u[:, 4], u[:, 5] = 1.0, 1.0, 0.9, 1.0
            e.ctx.put_blocks(ids, u)
        e.run(3)
    for r in range(3):
        assert ens[0].status(r) == ens[1].status(r)
        np.testing.assert_array_equal(ens[0].blocks(r)[1], ens[1].blocks(r)[1])
