"""Results that an operator writes in full do not depend on what the output held, and
an output that is the input's own memory behaves as before (a sum onto zeros)."""
import numpy as np
import pytest
import torch

from tests.gpu_helpers import make_case, rel, to_dev, to_host, wavefield

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["PSPI", "NSPS"])
def test_step_overwrites_its_output(name):
    from pyfwix_b200 import CudaWEM
    g, rng, _, _, slow, _ = make_case(nx=30, ny=21, nw=3, nz=2, nref=2)
    par = dict(nref=2, dx=g.dx, dy=g.dy, dz=g.dz, ow=g.ow, dw=g.dw, taperx=3, tapery=2)
    x = to_dev(wavefield(rng, 1, g))
    op = getattr(CudaWEM, name)(x, x, to_dev(slow), par)
    for run in (lambda out: op.forward(False, x, out), lambda out: op.adjoint(False, out, x)):
        want, got = torch.zeros_like(x), torch.full_like(x, float("nan"))
        run(want)
        run(got)
        assert rel(to_host(got), to_host(want)) == 0 and np.linalg.norm(to_host(want)) > 0
        host = np.full(tuple(x.shape), np.nan, dtype=np.complex64)
        run(host)
        assert np.array_equal(host, want.cpu().numpy())
        same = x.clone()  # in and out one tensor: the output is zeroed first
        op.forward(False, same, same)
        assert not same.any()


def test_labels_keep_their_range_check():
    from pyfwix_b200.plan import Plan
    p = Plan(16, 16, 2, 1, 1, nref=1)
    sref = torch.ones((1, 1, 2), dtype=torch.complex64)
    with pytest.raises(ValueError):
        p.set_refs(sref, torch.full((1, 1, 16, 16), 256, dtype=torch.int32))
    with pytest.raises(ValueError):
        p.set_refs(sref, torch.full((1, 1, 16, 16), -1, dtype=torch.int64))
    p.set_refs(sref, torch.zeros((1, 1, 16, 16), dtype=torch.uint8))
