"""The allocation-free time step on values its FP32 bounds cannot rank: it
must give the CFL minimum of plain FP64 arithmetic whatever the cells hold."""
import ctypes as C

import numpy as np
import pytest

from walicxe2d_b200.params import ADIABATIC, COOLINGH, base_params

pytestmark = pytest.mark.gpu


def _call(p, u, lev, dx, shift=0):
    import torch

    from walicxe2d_b200 import _lib
    L = _lib.load()
    flat = torch.empty(u.size + shift, dtype=torch.float64, device="cuda")
    flat[shift:] = torch.from_numpy(u.reshape(-1)).cuda()
    ld = torch.from_numpy(lev).cuda()
    torch.cuda.synchronize()
    dt, pd = C.c_double(-1.0), C.POINTER(C.c_double)
    d = dx.ctypes.data_as(pd)
    rc = L.w2d_timestep_noalloc(C.byref(p), C.c_void_p(flat.data_ptr() + 8 * shift), C.c_void_p(ld.data_ptr()),
                                u.shape[0], d, d, C.byref(dt))
    return rc, dt.value


def _exact(p, u, lev, dx):
    """src/timestep.f90:21-48 with uprim's floors, in the reference's operation order."""
    c = u[:, :, 2:18, 2:18]
    with np.errstate(all="ignore"):
        r = np.where(c[:, 0] > 1e-15, c[:, 0], 1e-15)
        vx, vy = c[:, 1] / r, c[:, 2] / r
        pr = (c[:, 3] - 0.5 * r * (vx * vx + vy * vy)) / p.cv
        pr = np.where(pr > 1e-15, pr, 1e-15)
        if p.cooling == COOLINGH:
            dent = 2.0 * r - (c[:, 4] if p.neq > 4 else r)
            dent = np.where(dent > 1e-15, dent, 1e-15)
            t = (pr / dent) * p.tempsc
            pr = dent * np.where(t < 1.0, 1.0, t) / p.tempsc
        cs = np.sqrt(p.gamma * pr / r)
        dl = dx[lev - 1][:, None, None]
        m = np.fmin.reduce(np.fmin(dl / (np.abs(vx) + cs), dl / (np.abs(vy) + cs)), axis=None)
    return p.cfl * min(1e30, m)


def _state(kind, n, neq, rng):
    rho = 10.0 ** rng.uniform(-3, 3, (n, 20, 20))
    vx, vy = rng.normal(0, 1, (2, n, 20, 20))
    pr = 10.0 ** rng.uniform(-3, 2, (n, 20, 20))
    if kind == "hypersonic":          # the pressure is lost in FP32's energy
        vx, vy, pr = 1e4 * vx, 1e4 * vy, 1e-3 * pr
    if kind == "uniform":             # every cell holds the maximum
        rho[:], vx[:], vy[:], pr[:] = 1.3, 0.7, -0.7, 0.9
    if kind == "ties":                # cells an ulp apart
        rho[:], vx[:], vy[:], pr[:] = 1.0, 0.5, 0.25, 1.0
        vx += rng.integers(-3, 4, vx.shape) * 2.0 ** -53
    u = np.zeros((n, neq, 20, 20))
    u[:, 0], u[:, 1], u[:, 2] = rho, rho * vx, rho * vy
    u[:, 3] = 0.5 * rho * (vx * vx + vy * vy) + 1.5 * pr
    for k in range(4, neq):
        u[:, k] = rho * rng.uniform(0, 1, rho.shape)
    if kind == "extreme":             # beyond FP32's range, floors, NaN
        at = rng.integers(0, u.size, 40 * n)
        u.reshape(-1)[at] = rng.choice([0.0, -1.0, 1e-300, -1e-40, 1e39, -1e39, 1e60, np.nan], at.size)
    return u


@pytest.mark.parametrize("kind", ["plain", "hypersonic", "uniform", "ties", "extreme"])
@pytest.mark.parametrize("neq,cooling,n", [(4, ADIABATIC, 1), (4, COOLINGH, 9), (5, ADIABATIC, 130),
                                           (6, COOLINGH, 301), (4, ADIABATIC, 2500)])
def test_noalloc_is_the_fp64_minimum(kind, neq, cooling, n):
    rng = np.random.default_rng([n, neq, len(kind)])
    p = base_params(neq=neq, npas=neq - 4, nlevs=4, cooling=cooling)
    dx = np.array([0.1, 0.05, 0.025, 0.0125])
    u = _state(kind, n, neq, rng)
    lev = rng.integers(1, 5, n).astype(np.int32)
    want = _exact(p, u, lev, dx)
    for shift in (0, 1):              # on and off the 16-byte boundary
        rc, dt = _call(p, u, lev, dx, shift)
        assert rc == 0 and dt == want, (shift, dt, want)


def test_noalloc_refuses_and_recovers():
    p = base_params(nlevs=4)
    dx = np.array([0.1, 0.05, 0.025, 0.0125])
    rng = np.random.default_rng(4)
    u, lev = _state("plain", 77, 4, rng), np.full(77, 2, np.int32)
    for bad in (0, 5):
        lev[40] = bad
        assert _call(p, u, lev, dx) == (5, -1.0)       # W2D_ERR_TOPOLOGY, dt untouched
    lev[40] = 2
    assert _call(p, u, lev, -dx)[0] == 5
    assert _call(p, u, lev, dx) == (0, _exact(p, u, lev, dx))


@pytest.mark.parametrize("kind", ["plain", "extreme"])
@pytest.mark.parametrize("past", [0, 1, 9])
def test_noalloc_around_one_block_per_cta(kind, past):
    import torch
    n = 4 * torch.cuda.get_device_properties(0).multi_processor_count + past
    rng = np.random.default_rng([n, len(kind)])
    p = base_params(neq=5, npas=1, nlevs=4, cooling=COOLINGH)
    dx = np.array([0.1, 0.05, 0.025, 0.0125])
    u = _state(kind, n, 5, rng)
    lev = rng.integers(1, 5, n).astype(np.int32)
    want = _exact(p, u, lev, dx)
    assert _call(p, u, lev, dx) == (0, want)
    keep = lev[n - 1]
    lev[n - 1] = 5                    # W2D_ERR_TOPOLOGY, dt untouched
    assert _call(p, u, lev, dx) == (5, -1.0)
    lev[n - 1] = keep
    assert _call(p, u, lev, dx) == (0, want)
