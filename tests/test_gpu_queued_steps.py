"""Steps queued without a wait between them (a mesh that stays, dt on the
device) against the same steps taken one call at a time: bit for bit, and the
same after a step that fails."""
import numpy as np
import pytest

from walicxe2d_b200 import _lib
from walicxe2d_b200.params import config, ensemble_members, sedov, snr

pytestmark = pytest.mark.gpu


def _runs(cfg):
    """Two equal runs; cfg "frozen" stops admesh after 30 steps."""
    from walicxe2d_b200.api import Simulation
    p, ic = {"fixed": lambda: sedov(nbroot=3, nlevs=1), "frozen": lambda: config("sedov_amr_small"),
             "cooling": lambda: snr(nbroot=3, nlevs=1, nblocks=9, size_pc=10.0)}[cfg]()
    out = []
    for _ in range(2):
        s = Simulation(p, ic)
        s.ctx.set_graphs(True)
        if cfg == "frozen":
            s.set_tree_mode("host")
            s.run(30)
            s.set_amr(False)
        out.append(s)
    return out


# 1: no queue; 2: the smallest; 129: one more than a batch holds
@pytest.mark.parametrize("cfg,n", [("fixed", 1), ("fixed", 2), ("fixed", 129), ("frozen", 7), ("cooling", 5)])
def test_queued_steps_equal_single_steps(cfg, n):
    a, b = _runs(cfg)
    a.run(n)
    for _ in range(n):
        b.run(1)
    assert a.status() == b.status()
    np.testing.assert_array_equal(a.blocks()[1], b.blocks()[1])
    a.run(1)      # and on from there
    b.run(1)
    assert a.status() == b.status()


@pytest.mark.parametrize("graphs", [False, True])
def test_queued_ensemble_equals_single_steps(graphs):
    from walicxe2d_b200.api import Ensemble
    mem = ensemble_members(count=3, precision=32)
    for p, _ in mem:
        p.nblocks = min(p.nblocks, 2000)
    ens = []
    for _ in range(2):
        e = Ensemble(mem, threads=2)
        e.ctx.set_graphs(graphs)
        e.run(5)
        e.set_amr(False)
        ens.append(e)
    a, b = ens
    a.run(6)
    for _ in range(6):
        b.run(1)
    for r in range(3):
        assert a.status(r) == b.status(r)
        np.testing.assert_array_equal(a.blocks(r)[1], b.blocks(r)[1])
    assert a.status()["steps"] == b.status()["steps"] == 11


@pytest.mark.parametrize("after", [0, 3])
def test_a_failed_step_ends_the_queue(after):
    """An infinite energy gives the solver a NaN contact speed: the call fails
    with the reference's stop, and the run stands where single steps leave it."""
    a, b = _runs("fixed")
    got = []
    for s, one in ((a, False), (b, True)):
        s.run(after)
        ids, u = s.blocks()
        u[4, 3, 9, 9] = np.inf
        s.ctx.put_blocks(ids, u)
        with pytest.raises(_lib.W2dException) as e:
            for _ in range(4 if one else 1):
                s.run(1 if one else 4)
        got.append((e.value.code, s.status(), s.blocks()[1]))
    assert got[0][0] == got[1][0]
    assert got[0][1] == got[1][1]
    np.testing.assert_array_equal(got[0][2], got[1][2])
    # a sound state runs on (the leaf count is back)
    for s in (a, b):
        ids, u = s.blocks()
        u[:] = u[0]
        u[:, 0], u[:, 1:3], u[:, 3] = 1.0, 0.0, 1.0
        s.ctx.put_blocks(ids, u)
        s.run(3)
    assert a.status() == b.status()
    np.testing.assert_array_equal(a.blocks()[1], b.blocks()[1])
