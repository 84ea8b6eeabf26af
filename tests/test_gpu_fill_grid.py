"""Fill I's persistent grid is whole waves of the CTAs an SM holds: four in FP32,
two waves of three in FP64."""
import pytest

from walicxe2d_b200.params import sedov

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,per_sm", [(32, 4), (64, 6)])
def test_fill_grid(precision, per_sm):
    from walicxe2d_b200.api import Simulation
    p, ic = sedov(nbroot=2, nlevs=1, nblocks=4)
    p.precision = precision
    s = Simulation(p, ic)
    s.ctx.set_graphs(True)
    assert s.ctx.tuning()["fill_I"]["ctas_per_sm"] == per_sm
