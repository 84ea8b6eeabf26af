"""What a captured step holds and a run changes between two queued runs.  Steps
that replay a captured one must do what steps without graphs do, bit for bit."""
import numpy as np
import pytest

from walicxe2d_b200.params import ensemble_members, snr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nets():
    """Two networks whose served cells differ."""
    from walicxe2d_b200.api import Surrogate
    out = []
    for seed in (20261203, 5):
        nn = Surrogate(seed)
        nn.samples(1 << 14, seed=seed)
        nn.train(2, batch=128, lr=2e-3, lr_end=2e-5)
        out.append(nn)
    return out


def _sim(graphs, nlevs=1):
    from walicxe2d_b200.api import Simulation
    p, ic = snr(nbroot=4, nlevs=nlevs, nblocks=4000 if nlevs > 1 else 16, size_pc=10.0, precision=32)
    s = Simulation(p, ic)
    s.set_tree_mode("host")
    s.ctx.set_graphs(graphs)
    return s


def _ens(graphs):
    from walicxe2d_b200.api import Ensemble
    mem = ensemble_members(count=3, precision=32)
    for p, _ in mem:
        p.nblocks = min(p.nblocks, 2000)
    e = Ensemble(mem, threads=2)
    e.ctx.set_graphs(graphs)
    return e


def _state(kind, s):
    if kind == "single":
        return s.status(), s.blocks()[1]
    return [s.status(r) for r in range(3)], np.concatenate([s.blocks(r)[1] for r in range(3)])


def _same(kind, a, b):
    sa, sb = _state(kind, a), _state(kind, b)
    assert sa[0] == sb[0]
    np.testing.assert_array_equal(sa[1], sb[1])
    assert a.ctx.surrogate_counts() == b.ctx.surrogate_counts()


def _pair(kind):
    """The run that queues replays of a captured step, and one that launches
    every step's kernels."""
    a, b = (_sim(g) if kind == "single" else _ens(g) for g in (True, False))
    for s in (a, b):
        s.set_amr(False)
    return a, b


def _grow(s):
    """admesh on until the mesh has outgrown the fallback list of the leaves
    it had (one and a half times them and 4,096 cells)."""
    most = 1.5 * s.leaf_ids().size + 4096 / 320
    s.set_amr(True)
    for _ in range(60):
        s.run(10)
        if s.leaf_ids().size > most:
            break
    assert s.leaf_ids().size > most
    s.set_amr(False)


@pytest.mark.parametrize("profiled", [False, True])
@pytest.mark.parametrize("single_steps", [False, True])
def test_fallback_list_moves_between_queued_runs(single_steps, profiled, nets):
    """The list of cells left to the exact routine is freed and made anew on a
    grown mesh, by captured single steps or by launches beside them
    (profiling): no captured step may keep the old one."""
    a, b = (_sim(g, nlevs=4) for g in (True, False))
    for s in (a, b):
        s.ctx.set_surrogate(nets[0])
        s.set_amr(False)
        for _ in range(4 if single_steps else 1):
            s.run(1 if single_steps else 4)
        s.ctx.profile(profiled)
        _grow(s)
        s.ctx.profile(False)
        for _ in range(4 if single_steps else 1):
            s.run(1 if single_steps else 4)
    _same("single", a, b)


@pytest.mark.parametrize("kind", ["single", "ensemble"])
def test_tolerance_between_queued_runs(kind, nets):
    a, b = _pair(kind)
    for s in (a, b):
        s.ctx.set_surrogate(nets[0])
        s.ctx.set_surrogate_tol(0.05)
        s.run(4)
        before = s.ctx.surrogate_counts()
        s.ctx.set_surrogate_tol(1e-6)
        s.run(4)
        after = s.ctx.surrogate_counts()
    _same(kind, a, b)
    # (the two tolerances serve different shares, so an old one would show)
    assert before[0] > after[0] - before[0]


@pytest.mark.parametrize("single_steps", [False, True])
@pytest.mark.parametrize("kind", ["single", "ensemble"])
def test_surrogate_attached_replaced_and_taken_off(kind, single_steps, nets):
    a, b = _pair(kind)
    for s in (a, b):
        for nn in (None, nets[0], nets[1], None):
            s.ctx.set_surrogate(nn)
            if single_steps:
                s.run(1)
                s.run(1)
            else:
                s.run(2)
    _same(kind, a, b)
    assert a.ctx.surrogate_counts()[0] > 0
