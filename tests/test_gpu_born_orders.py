"""The Born operators at every Taylor order that a plan takes, on the same problem in
metres and Hz and scaled down to millimetres and MHz: the filter (|k| / w)^2n is a ratio
that does not depend on the units, while k^2n and w^2n leave the range of a float."""
import numpy as np
import pytest

from oracle import wem
from tests.gpu_helpers import make_case, make_plan, rel, to_dev, to_host, wavefield

pytestmark = pytest.mark.gpu

TOL = 1e-5  # as in test_gpu_ops


# columns of a compile-time plan by TMA and by plain loads, of run-time ones (two and three
# stages), and of a length with neither
@pytest.mark.parametrize("nx,ny", [(64, 256), (50, 64), (42, 45), (48, 147), (30, 15)])
@pytest.mark.parametrize("scale", [1.0, 2.0e3, 2.0e5])
@pytest.mark.parametrize("taylor", [3, 4])
def test_orders_in_any_unit(nx, ny, scale, taylor):
    g, rng, sref, labels, slow, den = make_case(nx=nx, ny=ny, nw=3, nz=1, nref=1, taylor=taylor)
    g.dx, g.dy, g.dz = g.dx / scale, g.dy / scale, g.dz / scale
    g.ow, g.dw = g.ow * scale, g.dw * scale  # 3 - 8 Hz on a 10 m grid, 0.6 - 1.6 MHz on 50 um
    p = make_plan(g, 1, sref, labels, slow, den)
    x = wavefield(rng, 1, g)
    y = to_host(p.scatter(0, to_dev(x), to_dev(np.zeros_like(x))))
    assert rel(y, wem.scatter_forward(g, slow[0], x)) < TOL
    y = to_host(p.scatter(0, to_dev(x), to_dev(np.zeros_like(x)), adjoint=True))
    assert rel(y, wem.scatter_adjoint(g, slow[0], x)) < TOL
