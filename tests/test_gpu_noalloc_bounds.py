"""The allocation-free time step on more blocks than fit one per CTA, where FP32
bounds pick the cells computed in FP64: every number of equations and cooling,
on and off the 16-byte boundary, on values the bounds cannot rank."""
import numpy as np
import pytest

from test_gpu_noalloc_ranges import _call, _exact, _state
from walicxe2d_b200.params import ADIABATIC, COOLINGH, base_params

pytestmark = pytest.mark.gpu

DX = np.array([0.1, 0.05, 0.025, 0.0125])


def _blocks():
    import torch
    return 4 * torch.cuda.get_device_properties(0).multi_processor_count + 37


@pytest.mark.parametrize("eps", [1e-8, 1e-7, 1e-6, 1e-5, 1e-3, 0.1])
@pytest.mark.parametrize("neq", [5, 6])
def test_coolingh_floor_with_neutral_density_near_twice_the_density(neq, eps):
    """The pressure of a cold cell is (2 rho - u5) / tempsc there, a difference
    that FP32 loses."""
    n = _blocks()
    rng = np.random.default_rng([neq, int(-np.log10(eps))])
    p = base_params(neq=neq, npas=neq - 4, nlevs=4, cooling=COOLINGH)
    p.tempsc = 100.0
    rho = rng.uniform(0.5, 2.0, (n, 20, 20))
    u = np.zeros((n, neq, 20, 20))
    u[:, 0], u[:, 3] = rho, 1e-11
    u[:, 4] = 2.0 * rho * (1.0 - eps * rng.uniform(0.9, 1.0, rho.shape))
    lev = np.ones(n, np.int32)
    want = _exact(p, u, lev, DX)
    for shift in (0, 1):
        assert _call(p, u, lev, DX, shift) == (0, want)


@pytest.mark.parametrize("kind", ["plain", "hypersonic", "uniform", "ties", "extreme"])
@pytest.mark.parametrize("cooling", [ADIABATIC, COOLINGH])
@pytest.mark.parametrize("neq", [4, 5, 6])
def test_noalloc_is_the_fp64_minimum_on_many_blocks(neq, cooling, kind):
    n = _blocks()
    rng = np.random.default_rng([neq, cooling, len(kind)])
    p = base_params(neq=neq, npas=neq - 4, nlevs=4, cooling=cooling)
    u = _state(kind, n, neq, rng)
    lev = rng.integers(1, 5, n).astype(np.int32)
    want = _exact(p, u, lev, DX)
    for shift in (0, 1):
        assert _call(p, u, lev, DX, shift) == (0, want)
