"""The work that users of this framework have it do, as timed cases.

A case is a dict of plain values; its "kind" says which program it stands for:

  mesh      a fixed uniform mesh: the program puts its own initial state,
            advances it and takes the result back (Simulation, step graphs)
  run       a whole AMR run from its initial conditions to its first output
  amr       an AMR blast at a developed state between mesh changes: state in,
            steps, state out
  remnant   the same for the supernova remnant with coolingh
  jet       the same for the reference's shipped cylindrical jet or the planar
            jet, with coolingdmc from its table
  host      the drop-in use: a host program that owns the block tree calls
            timestep, tstep, criteria, refine and coarse through the context,
            handing over its tree and innerbounds after every mesh change
  ensemble  independent runs of uneven size advanced together, with the exact
            cooling routine or the learned one
  train     a cooling network trained from its initial weights on samples at hand
  dt        the CFL time step of blocks that the caller holds on the device

The seed sets the densities and energies (or the modes of the initial fields)
that a pass starts from.  State and results travel through page-locked host
arrays, as in bench.py.  FP32 runs hand their results back in FP32.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import random

import numpy as np
import torch

from walicxe2d_b200 import _lib
from walicxe2d_b200.api import Context, Ensemble, Simulation, Surrogate
from walicxe2d_b200.params import (BC_REFLECTIVE, COMPAT_HLLC_STAR, COMPAT_OUTFYB, COOLINGDMC,
                                   GEOM_CYLINDRICAL, HLL, HLL_HLLC, HLLC, IC_SEDOV, W2dInit, base_params,
                                   ensemble_members, jet, jet_cyl, sedov, snr)

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NX, W = 16, 20


def listed():
    return [
        # configuration 1: 64x64 zones, no AMR; 16 blocks, so launches and latency are the cost
        dict(name="mesh_64x64", kind="mesh", bx=4, by=4, solver=HLLC, limiter=1, precision=64, steps=20),
        # time step of 20,011 blocks a host holds itself (256 MB, beyond L2)
        dict(name="dt_of_caller_blocks", kind="dt", blocks=20011, neq=4),
        # the network's training (the batch size bench.py and the runner use)
        dict(name="train_network", kind="train", samples=262144, epochs=2, batch=8192),
        # the reference's main loop in a host program (about 1,000 leaves, the mesh changes in most steps)
        dict(name="host_main_loop", kind="host", nbroot=8, nlevs=5, grow=120, steps=12),
        # configuration 2 from its initial conditions: set-up, 200 steps with admesh after each, the output
        dict(name="blast_whole_run", kind="run", nbroot=8, nlevs=5, steps=200),
        # the shipped set-up: cylindrical jet, van Leer limiter, coolingdmc (about 550 leaves)
        dict(name="jet_coolingdmc", kind="jet", cyl=True, nlevs=6, grow=1800, steps=16),
        # configuration 3: remnant with coolingh, FP64, about 2,000 leaves
        dict(name="remnant_coolingh", kind="remnant", nbroot=10, nlevs=6, grow=1300, steps=16),
        # configuration 2 developed (the bench's workload, about 3,400 leaves)
        dict(name="blast_developed", kind="amr", nbroot=8, nlevs=5, grow=250, solver=HLLC, limiter=1, cyl=False,
             steps=24),
        # configuration 5: ensembles in FP32 (6,600 leaves) with the exact routine and with the network
        dict(name="ensemble_fp32", kind="ensemble", runs=24, nn=False, precision=32, steps=20),
        dict(name="ensemble_fp32_nn", kind="ensemble", runs=24, nn=True, precision=32, steps=20),
        # a fixed mesh of 1520 x 1488 zones (95 x 93 blocks): the largest working set, beyond L2
        dict(name="mesh_95x93_blocks", kind="mesh", bx=95, by=93, solver=HLLC, limiter=1, precision=64, steps=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mesh", "mesh", "run", "amr", "amr", "host", "remnant", "jet", "ensemble", "ensemble", "train",
                       "dt"])
    if kind == "mesh":
        bx = _log(rng, 2, 90)
        by = min(90, max(1, _log(rng, max(1, bx // 3), 3 * bx)))
        return dict(kind=kind, bx=bx, by=by, solver=rng.choice([HLLC, HLLC, HLLC, HLL, HLL_HLLC]),
                    limiter=rng.choice([1, 1, 2, 0, 3, 4, 5, 6]), precision=rng.choice([64, 64, 32]),
                    steps=rng.randint(8, 20))
    if kind == "run":
        return dict(kind=kind, nbroot=rng.randint(3, 9), nlevs=rng.randint(3, 5), steps=rng.randint(40, 200))
    if kind == "amr":
        return dict(kind=kind, nbroot=rng.randint(3, 10), nlevs=rng.randint(3, 5), grow=_log(rng, 40, 320),
                    solver=rng.choice([HLLC, HLLC, HLL_HLLC]), limiter=rng.choice([1, 1, 2, 4]),
                    cyl=rng.random() < 0.25, steps=rng.randint(8, 24))
    if kind == "host":
        return dict(kind=kind, nbroot=rng.randint(3, 9), nlevs=rng.randint(3, 5), grow=_log(rng, 20, 160),
                    steps=rng.randint(4, 12))
    if kind == "remnant":
        return dict(kind=kind, nbroot=rng.randint(4, 12), nlevs=rng.randint(4, 6), grow=_log(rng, 150, 1500),
                    steps=rng.randint(6, 18))
    if kind == "jet":
        return dict(kind=kind, cyl=rng.random() < 0.5, nlevs=rng.randint(5, 6), grow=_log(rng, 200, 2000),
                    steps=rng.randint(6, 18))
    if kind == "ensemble":
        return dict(kind=kind, runs=_log(rng, 3, 40), nn=rng.random() < 0.4, precision=32, steps=rng.randint(6, 20))
    if kind == "train":
        batch = rng.choice([1024, 4096, 8192, 16384])
        return dict(kind=kind, samples=_log(rng, 40000, 400000), epochs=rng.randint(1, 2), batch=batch)
    return dict(kind=kind, blocks=_log(rng, 100, 60000), neq=rng.choice([4, 5, 6]))


# ---- inputs ----------------------------------------------------------------


def _pinned(n, neq, dtype=torch.float64):
    return torch.empty((n, neq, W, W), dtype=dtype, pin_memory=True)


def _cooltab():
    rows = np.loadtxt(os.path.join(ROOT, "tests", "golden", "coolingDMC.tab"))
    return rows[:, 0], rows[:, 1]


def _mesh_params(case):
    bx, by = case["bx"], case["by"]
    p = base_params(nlevs=1, nbroot_x=bx, nbroot_y=by, nblocks=bx * by, solver=case["solver"],
                    limiter=case["limiter"], precision=case["precision"])
    p.xmax, p.ymax = 1.0, by / bx
    ic = W2dInit()
    ic.kind, ic.init_levels, ic.startup_admesh = IC_SEDOV, 1, 0
    ic.rho0, ic.p0, ic.e_dep = 1.0, 1.0, 1.0
    return p, ic


def _mesh_blocks(case, seed, device):
    """u of every block, block-major: smooth waves of density and velocity
    with a hot, dense disc, as conserved variables; ghosts hold the
    neighbours' cells (the edge cell at the box)."""
    bx, by = case["bx"], case["by"]
    r = random.Random(1000003 * seed + 7)
    nx, ny = NX * bx, NX * by
    x = ((torch.arange(nx, dtype=torch.float64, device=device) + 0.5) / nx)[None, :]
    y = ((torch.arange(ny, dtype=torch.float64, device=device) + 0.5) / nx)[:, None]

    def waves(amp):
        f = torch.zeros((ny, nx), dtype=torch.float64, device=device)
        for _ in range(4):
            kx, ky, ph = 2 * math.pi * r.randint(1, 5), 2 * math.pi * r.randint(1, 5), r.uniform(0, 2 * math.pi)
            f += r.uniform(0.3, 1.0) * amp * torch.sin(kx * x + ky * y + ph)
        return f

    rho = 1.0 + 0.15 * torch.tanh(waves(1.0))
    vx, vy = waves(0.3), waves(0.3)
    p = 0.6 + 0.2 * torch.tanh(waves(1.0))
    disc = ((x - r.uniform(0.3, 0.7)) ** 2 + (y - r.uniform(0.3, 0.7) * by / bx) ** 2) < r.uniform(0.08, 0.16) ** 2
    rho = torch.where(disc, 2.0 * rho, rho)
    p = torch.where(disc, 8.0 * p, p)
    g = torch.stack([rho, rho * vx, rho * vy, 0.5 * rho * (vx * vx + vy * vy) + 1.5 * p])
    g = torch.nn.functional.pad(g[None], (2, 2, 2, 2), mode="replicate")[0]
    return g.unfold(1, W, NX).unfold(2, W, NX).permute(1, 2, 0, 3, 4).reshape(bx * by, 4, W, W).contiguous()


def _blast(case, seed=None):
    """A blast at the box's centre.  The seed scales density and pressure by
    a power of two, under which the flow is the same to the last bit: every
    seed's mesh is the same, so the results of all seeds have one shape."""
    a = 1.0 if seed is None else 2.0 ** (37 * seed % 61 - 20)
    p, ic = sedov(nbroot=case["nbroot"], nlevs=case["nlevs"], tol=0.1,
                  nblocks=4000 if case["kind"] == "run" else 9000, rho0=a, p0=1e-5 * a, e0=a)
    if case["kind"] == "amr":
        p.solver, p.limiter = case["solver"], case["limiter"]
        if case["cyl"]:
            p.geometry, p.bc_bottom = GEOM_CYLINDRICAL, BC_REFLECTIVE
    return p, ic


def _remnant(case):
    return snr(nbroot=case["nbroot"], nlevs=case["nlevs"], nblocks=20000)


def _jet(case):
    return (jet_cyl(nlevs=case["nlevs"], nblocks=16000) if case["cyl"] else
            jet(nlevs=case["nlevs"], rj_cm=2.0e15, nblocks=16000))


def _developed(p, ic, grow, denser=1.0):
    """A run advanced `grow` steps and the leaves of its mesh, which then
    stays; the state the passes start from is `denser` times it (the same
    velocities and temperatures)."""
    sim = Simulation(p, ic)
    if p.cooling == COOLINGDMC:
        sim.set_cooltab(*_cooltab())
    sim.ctx.set_graphs(True)
    sim.run(grow)
    sim.set_amr(False)
    ids, u = sim.blocks()
    u0 = _pinned(ids.size, p.neq)
    u0.copy_(torch.from_numpy(u * denser))
    return dict(sim=sim, ctx=sim.ctx, ids=ids, u0=u0.numpy(), out=_pinned(ids.size, p.neq).numpy())


def _admesh_ops(lp0, leaf0, lp1, leaf1):
    """Refines and coarsenings between two trees, in admesh's order: (parent
    or dad, its four sons)."""
    gone = np.nonzero((leaf0 != 0) & (leaf1 == 0))[0]
    came = np.nonzero((leaf1 != 0) & (leaf0 == 0))[0]
    refines, coarsens, sons = [], [], set()

    def family(lp, nb):
        s1 = int(lp[nb, 2])
        s3 = int(lp[s1, 7])
        return (int(nb), s1, int(lp[s1, 5]), s3, int(lp[s3, 5]))

    for nb in gone:
        q = family(lp1, nb) if lp1[nb, 2] else None
        if q and all(leaf1[s] for s in q[1:]):
            refines.append((int(lp1[nb, 0]), int(nb), q))
            sons.update(q[1:])
    for nb in came:
        if int(nb) not in sons:
            coarsens.append((-int(lp1[nb, 0]), int(nb), family(lp0, nb)))
    refines.sort()
    coarsens.sort()
    return ([q[2] for q in refines], [q[2] for q in coarsens])


def _host_program(case, seed):
    """What a host program has at some step of its run: its tree, innerbounds
    and mesh changes for the steps to come, and its blocks."""
    p, ic = _blast(case, seed)
    sim = Simulation(p, ic)
    sim.set_tree_mode("host")
    sim.run(case["grow"])
    ids, u = sim.blocks()
    u0 = _pinned(ids.size, p.neq)
    u0.copy_(torch.from_numpy(u))
    time, plan = sim.status()["time"], []
    lp, leaf, icoord, ib = sim.tree()
    for _ in range(case["steps"]):
        nbmax = sim.status()["nbmax"]
        now = dict(lp=lp[1:nbmax + 1].copy(), leaf=leaf[1:nbmax + 1].copy(), icoord=icoord[1:nbmax + 1].copy(),
                   nbmax=nbmax, bounds=ib)
        sim.run(1)
        lp1, leaf1, icoord, ib = sim.tree()
        now["refine"], now["coarse"] = (np.array(q, np.int32) for q in _admesh_ops(lp, leaf, lp1, leaf1))
        now["changed"] = bool(len(now["refine"]) or len(now["coarse"]))
        lp, leaf = lp1, leaf1
        plan.append(now)
    last = sim.leaf_ids()
    dx = np.array([p.xmax / p.nx / 2.0 ** k / p.nbroot_x for k in range(p.nlevs)])
    dy = np.array([p.ymax / p.ny / 2.0 ** k / p.nbroot_y for k in range(p.nlevs)])
    sim.close()
    return dict(ctx=Context(p), ids=ids, u0=u0.numpy(), plan=plan, last=last, dx=dx, dy=dy, time=time,
                out=_pinned(last.size, p.neq).numpy())


def _network():
    """A network as a user's program has it in hand: trained before the run
    (one tile a batch: the sums' order, and so the network, repeats)."""
    nn = Surrogate(20261203)
    nn.samples(1 << 14, seed=20261203)
    nn.train(2, batch=128, lr=2e-3, lr_end=2e-5)
    return nn


def _ensemble(case, seed):
    members = ensemble_members(count=case["runs"], precision=case["precision"])
    for p, _ in members:
        p.nblocks = min(p.nblocks, 3000)
    ens = Ensemble(members)
    ctx = ens.ctx
    nn = None
    if case["nn"]:
        nn = _network()
        ctx.set_surrogate(nn)
    ctx.set_graphs(True)
    ens.run(30)
    ens.set_amr(False)
    slots = [ens.leaves(r) + ens.slots(r)[0] for r in range(ens.n)]
    ids = np.concatenate(slots).astype(np.int32)
    neq = members[0][0].neq
    u0 = _pinned(ids.size, neq)
    ctx.get_blocks(ids, u0.numpy())
    rnd, at = random.Random(1000003 * seed + 19), 0
    for one in slots:      # every run its own density
        u0[at:at + one.size] *= rnd.uniform(0.9, 1.1)
        at += one.size
    out = _pinned(ids.size, neq)
    return dict(ens=ens, nn=nn, ctx=ctx, ids=ids, u0=u0.numpy(), out=out.numpy(), out64=out,
                out32=_pinned(ids.size, neq, torch.float32))


def _dt_blocks(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, neq = case["blocks"], case["neq"]
    rnd = lambda: torch.rand((n, W, W), generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    rho, vx, vy, pr = 0.2 + rnd(), 4.0 * rnd() - 2.0, 4.0 * rnd() - 2.0, 0.05 + rnd()
    u = torch.empty((n, neq, W, W), device="cuda", dtype=torch.float64)
    u[:, 0], u[:, 1], u[:, 2] = rho, rho * vx, rho * vy
    u[:, 3] = 0.5 * rho * (vx * vx + vy * vy) + 1.5 * pr
    for k in range(4, neq):
        u[:, k] = rho * rnd()
    lev = torch.randint(1, 6, (n,), generator=g, device="cuda", dtype=torch.int32)
    p = base_params(neq=neq, npas=neq - 4, nlevs=5, nbroot_x=8, nbroot_y=8)
    d = np.array([p.xmax / p.nx / 2.0 ** k / 8 for k in range(5)])
    return p, u, lev, d


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mesh":
        p, ic = _mesh_params(case)
        sim = Simulation(p, ic)
        sim.ctx.set_graphs(True)
        n = p.nblocks
        u0, out = _pinned(n, 4), _pinned(n, 4)
        u0.copy_(_mesh_blocks(case, seed, "cuda"))
        s = dict(sim=sim, ctx=sim.ctx, ids=np.arange(1, n + 1, dtype=np.int32), u0=u0.numpy(), out=out.numpy())
        if p.precision == 32:
            s.update(out64=out, out32=_pinned(n, 4, torch.float32))
    elif kind == "run":
        s = dict(zip(("p", "ic"), _blast(case, seed)))
    elif kind == "amr":
        s = _developed(*_blast(case), case["grow"], random.Random(1000003 * seed + 23).uniform(0.9, 1.1))
    elif kind == "remnant":
        s = _developed(*_remnant(case), case["grow"], random.Random(1000003 * seed + 13).uniform(0.9, 1.1))
    elif kind == "jet":
        s = _developed(*_jet(case), case["grow"], random.Random(1000003 * seed + 17).uniform(0.9, 1.1))
    elif kind == "host":
        s = _host_program(case, seed)
    elif kind == "ensemble":
        s = _ensemble(case, seed)
    elif kind == "train":
        nn = Surrogate(seed % 1000 + 1)
        nn.samples(case["samples"], seed=seed)
        s = dict(nn=nn, weights=nn.params())
    else:
        p, u, lev, d = _dt_blocks(case, seed)
        s = dict(p=p, u=u, lev=lev, d=d, lib=_lib.load())
    s.update(kind=kind, case=dict(case))
    return s


# ---- one pass --------------------------------------------------------------


def _host_loop(s):
    """src/main.f90:87-98 with the host's own tree."""
    ctx, t, grads = s["ctx"], s["time"], None
    first = s["plan"][0]
    ctx.set_topology(first["lp"], first["leaf"], first["icoord"], first["nbmax"], s["dx"], s["dy"])
    ctx.put_blocks(s["ids"], s["u0"])
    fresh, dts = True, []
    for k, now in enumerate(s["plan"]):
        dt = ctx.timestep()
        t += dt
        dts.append(dt)
        if fresh:
            if k:
                ctx.set_topology(now["lp"], now["leaf"], now["icoord"], now["nbmax"], s["dx"], s["dy"])
            ctx.set_bounds(now["bounds"])
        ctx.tstep(t, dt)
        grads = ctx.criteria(now["nbmax"])
        if len(now["refine"]):
            ctx.refine(now["refine"])
        if len(now["coarse"]):
            ctx.coarse(now["coarse"])
        fresh = now["changed"]
    return dict(u=ctx.get_blocks(s["last"], s["out"]), dt=np.array(dts), criteria=grads)


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "host":
        return _host_loop(s)
    if kind == "run":
        sim = Simulation(s["p"], s["ic"])
        sim.ctx.set_graphs(True)
        sim.run(case["steps"])
        ids, u = sim.blocks()
        st = sim.status()
        sim.close()
        return dict(ids=ids, u=u, time=st["time"])
    if kind == "train":
        nn = s["nn"]
        nn.set_params(s["weights"])
        loss = nn.train(case["epochs"], batch=case["batch"])
        return dict(params=nn.params(), loss=loss)
    if kind == "dt":
        dt, pd = C.c_double(), C.POINTER(C.c_double)
        d = s["d"].ctypes.data_as(pd)
        rc = s["lib"].w2d_timestep_noalloc(C.byref(s["p"]), C.c_void_p(s["u"].data_ptr()),
                                           C.c_void_p(s["lev"].data_ptr()), s["u"].shape[0], d, d, C.byref(dt))
        if rc:
            raise RuntimeError(f"w2d_timestep_noalloc: status {rc}")
        return dt.value
    s["ctx"].put_blocks(s["ids"], s["u0"])
    (s["ens"] if kind == "ensemble" else s["sim"]).run(case["steps"])
    u = s["ctx"].get_blocks(s["ids"], s["out"])
    if "out32" in s:
        s["out32"].copy_(s["out64"])
        return s["out32"]
    if kind == "jet":   # the run's clock goes on from pass to pass, the jet's speed with it
        return dict(u=u, time=s["sim"].status()["time"])
    return u


# ---- what a pass cannot do without -----------------------------------------


def _about_leaves(case):
    """Leaf count at the timed state (measured growth of the default runs)."""
    kind = case["kind"]
    if kind == "mesh":
        return case["bx"] * case["by"]
    if kind in ("amr", "host", "run"):
        g = case.get("grow", 0.6 * case["steps"])
        most = case["nbroot"] ** 2 * 4 ** (case["nlevs"] - 1)
        return int(min(most, case["nbroot"] ** 2 + 140 + 790 * (g / 100.0) ** 1.5))
    if kind == "remnant":
        return int(min(case["nbroot"] ** 2 * 4 ** (case["nlevs"] - 1), 4 * case["nbroot"] ** 2 + 1.3 * case["grow"]))
    if kind == "jet":
        return int((40 + 0.27 * case["grow"]) if case["cyl"] else (330 + 0.37 * case["grow"]))
    return 280 * case["runs"]


def work(case):
    kind = case["kind"]
    if kind == "train":   # features and targets read once per epoch; the MLP's products, forward and backward
        n = case["samples"]
        macs = 4 * 64 + 64 * 64 + 64 * 2
        return {"bytes": 24.0 * n * case["epochs"], "flops": 6.0 * macs * n * case["epochs"]}
    if kind == "dt":      # interior cells of the four hydro variables
        return {"bytes": case["blocks"] * 256 * 4 * 8.0, "flops": case["blocks"] * 256 * 25.0}
    # per step and zone: two passes over the state with its halo (20x20 of 16x16 cells) and two writes;
    # the flux arithmetic of both half steps
    neq = 4 if kind in ("mesh", "amr", "host", "run") else 6
    size = 4 if case.get("precision", 64) == 32 else 8
    leaves, zones = _about_leaves(case), 256 * _about_leaves(case)
    ends = (1 if kind == "run" else 2) * leaves * neq * W * W * 8.0
    return {"bytes": zones * case["steps"] * 5.125 * neq * size + ends,
            "flops": zones * case["steps"] * (130.0 + 80.0 * neq)}


# ---- the same in 64 bits with plain torch ----------------------------------


def _slope(lim, a, b):
    """average(a, b) of LIMITER -1..6 (src/limiter.f90:24-86)."""
    one = torch.ones((), dtype=a.dtype, device=a.device)
    zero = 0.0 * one
    s = torch.copysign(one, a)
    if lim == 0:
        return 0.5 * (a + b)
    if lim == 1:
        return s * torch.maximum(zero, torch.minimum(a.abs(), s * b))
    if lim == 2:
        return torch.where(a * b <= 0, zero, a * b * (a + b) / torch.where(a * b <= 0, one, a * a + b * b))
    if lim == 3:
        d = 1e-7
        return (a * (b * b + d) + b * (a * a + d)) / (a * a + b * b + d)
    if lim == 4:
        m = torch.minimum(torch.minimum(2 * a.abs(), 2 * s * b), s * (0.25 * a + 0.75 * b))
        return s * torch.maximum(zero, torch.minimum(m, s * (0.75 * a + 0.25 * b)))
    if lim == 5:
        return s * torch.maximum(zero, torch.minimum(torch.minimum(2 * a.abs(), 2 * s * b), s * 0.5 * (a + b)))
    s = torch.copysign(one, b)
    return s * torch.maximum(torch.maximum(zero, torch.minimum(2 * b.abs(), s * a)), torch.minimum(b.abs(), 2 * s * a))


def _flux(q):
    e = 0.5 * q[0] * (q[1] ** 2 + q[2] ** 2) + 1.5 * q[3]
    return torch.stack([q[0] * q[1], q[0] * q[1] ** 2 + q[3], q[0] * q[1] * q[2], q[1] * (e + q[3])])


def _cons(q):
    return torch.stack([q[0], q[0] * q[1], q[0] * q[2], 0.5 * q[0] * (q[1] ** 2 + q[2] ** 2) + 1.5 * q[3]])


def _prim(u):
    r = u[0].clamp(min=1e-15)
    vx, vy = u[1] / r, u[2] / r
    return torch.stack([r, vx, vy, ((u[3] - 0.5 * r * (vx ** 2 + vy ** 2)) / 1.5).clamp(min=1e-15)])


def _riemann(p, l, r):
    """Flux between the states l and r ([4, ...], normal velocity in row 1)."""
    cl, cr = (p.gamma * l[3] / l[0]).sqrt(), (p.gamma * r[3] / r[0]).sqrt()
    sr, sl = torch.maximum(l[1] + cl, r[1] + cr), torch.minimum(l[1] - cl, r[1] - cr)
    fl, fr = _flux(l), _flux(r)
    hll = (sr * fl - sl * fr + sl * sr * (_cons(r) - _cons(l))) / (sr - sl)
    if p.solver == HLL:
        f = hll
    else:
        ml, mr = sl - l[1], sr - r[1]
        st = (mr * r[0] * r[1] - ml * l[0] * l[1] - r[3] + l[3]) / (mr * r[0] - ml * l[0])
        left = st >= 0
        den = torch.where(left, l[0], r[3] if p.compat & COMPAT_HLLC_STAR else r[0])   # src/hllcfluxes.f90:157
        q, s, m = torch.where(left, l, r), torch.where(left, sl, sr), torch.where(left, ml, mr)
        e = 0.5 * q[0] * (q[1] ** 2 + q[2] ** 2) + 1.5 * q[3]
        rs = q[0] * m / (s - st)
        us = torch.stack([rs, rs * st, rs * q[2], rs * (e / q[0] + (st - q[1]) * (st + q[3] / (den * m)))])
        f = torch.where(left, fl, fr) + s * (us - _cons(q))
        if p.solver == HLL_HLLC:
            d1, d2 = r[1] - l[1], r[2] - l[2]
            mag = (d1 ** 2 + d2 ** 2).sqrt()
            b1 = torch.where(mag <= 1e-6, torch.ones_like(mag), (d1.abs() / mag.clamp(min=1e-300)).sqrt())
            f = b1 * f + (1.0 - b1) * hll
    return torch.where(sl > 0, fl, torch.where(sr < 0, fr, f))


def _exact_mesh(case, seed):
    p, _ = _mesh_params(case)
    bx, by = case["bx"], case["by"]
    u = _mesh_blocks(case, seed, "cuda" if torch.cuda.is_available() else "cpu").transpose(0, 1).contiguous()
    if case["precision"] == 32:
        u = u.float().double()
    dx, dy = p.xmax / NX / bx, p.ymax / NX / by
    g = u.view(4, by, bx, W, W)
    lo, hi, mid = slice(0, 2), slice(18, 20), slice(2, 18)

    def fill(v, layers):
        """The ghost layers next to the interior from the neighbours, outflow at the box."""
        for k in range(layers):
            v[:, :, 1:, mid, 1 - k] = v[:, :, :-1, mid, 17 - k]
            v[:, :, :-1, mid, 18 + k] = v[:, :, 1:, mid, 2 + k]
            v[:, 1:, :, 1 - k, mid] = v[:, :-1, :, 17 - k, mid]
            v[:, :-1, :, 18 + k, mid] = v[:, 1:, :, 2 + k, mid]
            v[:, :, 0, mid, 1 - k] = v[:, :, 0, mid, 2 + k]
            v[:, :, -1, mid, 18 + k] = v[:, :, -1, mid, 17 - k]
            v[:, -1, :, 18 + k, mid] = v[:, -1, :, 17 - k, mid]

    # innerbounds: per block its walls and the faces toward higher IDs, in the order left, right, bottom, top;
    # the bottom outflow of boundaryI goes to the block whose ID is the entry's position (src/boundaryI.f90:87)
    pos, top_at, bottom_at = 0, {}, {}
    for nb in range(bx * by):
        ix, iy = nb % bx, nb // bx
        pos += (1 if ix == 0 else 0) + 1
        if iy == 0:
            pos += 1
            bottom_at[pos] = nb
        pos += 1
        top_at[nb] = pos
    stray = [e - 1 for e in bottom_at
             if e <= bx * by and (e - 1 < bx or e > top_at[e - 1 - bx])] if p.compat & COMPAT_OUTFYB else range(bx)

    def fluxes(q, order):
        out = []
        for ax in (0, 1):
            v = q if ax == 0 else q[[0, 2, 1, 3]].transpose(-1, -2)
            v = v[..., mid, :]
            if order == 1:
                a, b = v[..., 1:18], v[..., 2:19]
            else:
                w = v.double()
                d = w[..., 1:] - w[..., :-1]
                s = 0.5 * _slope(p.limiter, d[..., :-1], d[..., 1:])      # cells 1..18 of 0..19
                a, b = w[..., 1:18] + s[..., 0:17], w[..., 2:19] - s[..., 1:18]
            f = _riemann(p, a, b)
            out.append(f if ax == 0 else f[[0, 2, 1, 3]].transpose(-1, -2))
        return out

    def update(uo, f, dt):
        return (uo - dt / dx * (f[0][..., 1:] - f[0][..., :-1]) - dt / dy * (f[1][..., 1:, :] - f[1][..., :-1, :]))

    for _ in range(case["steps"]):
        q = _prim(g)
        cs = (p.gamma * q[3] / q[0]).sqrt()[..., mid, mid]
        dt = p.cfl * float(torch.minimum(dx / (q[1][..., mid, mid].abs() + cs), dy / (q[2][..., mid, mid].abs() + cs)).min())
        up = g.clone()
        up[..., mid, mid] = update(g[..., mid, mid], fluxes(q, 1), 0.5 * dt)
        fill(up, 2)
        for k in range(2):
            up[:, 0, :, 1 - k, mid] = up[:, 0, :, 2 + k, mid]
        new = update(g[..., mid, mid], fluxes(_prim(up), 2), dt)
        new = new + p.eta * (g[..., mid, 3:19] + g[..., mid, 1:17] + g[..., 3:19, mid] + g[..., 1:17, mid]
                             - 4.0 * g[..., mid, mid])
        for s in (lo, hi):
            g[..., mid, s] = up[..., mid, s]
            g[..., s, mid] = up[..., s, mid]
        g[..., mid, mid] = new
        fill(g, 1)
        for b in stray:
            g[:, b // bx, b % bx, 1, mid] = g[:, b // bx, b % bx, 2, mid]
    out = g.view(4, bx * by, W, W).transpose(0, 1).contiguous().cpu()
    return out


def exact(case, seed):
    if case["kind"] == "mesh":
        return _exact_mesh(case, seed)
    if case["kind"] == "dt":
        p, u, lev, d = _dt_blocks(case, seed)
        q = _prim(u[:, :4, 2:18, 2:18].transpose(0, 1))
        cs = (p.gamma * q[3] / q[0]).sqrt()
        dl = torch.from_numpy(d).cuda()[lev.long() - 1][:, None, None]
        return p.cfl * float((dl / (torch.maximum(q[1].abs(), q[2].abs()) + cs)).min())
    return None
