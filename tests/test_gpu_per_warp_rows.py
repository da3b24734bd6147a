"""The lengths without a register-resident plan (1 to 12, 15, 25, 125, 625, 875) in every kind
of pass, as rows and as columns, against the FP64 oracle; and the smooth steps' slowness
derivative at lengths of every kind of plan, padded ones among them.  Tolerances as in
test_gpu_ops and test_gpu_fwi: 1e-5 per operator."""
import numpy as np
import pytest
import torch

from oracle import wem
from pyfwix_b200 import _lib as L
from pyfwix_b200.plan import Plan
from tests.gpu_helpers import make_case, make_plan, oracle_labels, rel, to_dev, to_host, wavefield

pytestmark = pytest.mark.gpu

TOL = 1e-5
NEITHER = [  # nx, ny, padx, pady
    (15, 20, 0, 0), (10, 25, 2, 0), (25, 24, 0, 4), (100, 12, 25, 3), (20, 110, 5, 15), (625, 5, 0, 0), (6, 800, 0, 75),
]


@pytest.mark.parametrize("nx,ny,padx,pady", NEITHER)
@pytest.mark.parametrize("eps,nref", [(0.0, 4), (0.01, 3)])
def test_steps(nx, ny, padx, pady, eps, nref):
    g, rng, sref, labels, _, _ = make_case(nx=nx, ny=ny, padx=padx, pady=pady, nw=2, nz=2, nref=nref, eps=eps,
                                           complex_refs=eps > 0, labels_per_w=eps > 0)
    lab = oracle_labels(labels, g)
    x, d0 = wavefield(rng, 2, g), wavefield(rng, 2, g)
    for kind, fwd, adj in (("pspi", wem.pspi_forward, wem.pspi_adjoint), ("nsps", wem.nsps_forward, wem.nsps_adjoint)):
        p = make_plan(g, 2, sref, labels, step=kind)
        for cache in (True, False):
            if not cache:
                p.disable_phase_cache()
            y = to_host(p.step(1, to_dev(x), to_dev(d0), direction=0, add=True))
            assert rel(y, fwd(g, sref[1], lab[1], x, d0)) < TOL
            y = to_host(p.step(1, to_dev(x), to_dev(d0), direction=1, add=True))
            assert rel(y, adj(g, sref[1], lab[1], x, d0)) < TOL


@pytest.mark.parametrize("nx,ny", [(64, 1), (50, 1), (1, 64), (1, 48), (1, 1)])
def test_one_row_or_column(nx, ny):
    g, rng, sref, labels, _, _ = make_case(nx=nx, ny=ny, nw=2, nz=1, nref=3, taperx=0, tapery=0)
    lab, x = oracle_labels(labels, g), wavefield(rng, 1, g)
    p = make_plan(g, 1, sref, labels)
    for kind, fwd, adj in (("pspi", wem.pspi_forward, wem.pspi_adjoint), ("nsps", wem.nsps_forward, wem.nsps_adjoint)):
        y = torch.empty(p.wshape, dtype=torch.complex64, device="cuda")
        assert rel(to_host(p.step(0, to_dev(x), y, kind=kind)), fwd(g, sref[0], lab[0], x)) < TOL
        assert rel(to_host(p.step(0, to_dev(x), y, kind=kind, direction=1)), adj(g, sref[0], lab[0], x)) < TOL


@pytest.mark.parametrize("nx,ny,padx,pady", NEITHER)
@pytest.mark.parametrize("taylor,shared", [(0, True), (1, True), (4, False)])
def test_scatter(nx, ny, padx, pady, taylor, shared):
    g, rng, sref, labels, slow, den = make_case(nx=nx, ny=ny, padx=padx, pady=pady, nw=2, nz=1, nref=1, taylor=taylor)
    if shared:
        slow, den = slow[:, :1], den[:, :1]
    p = make_plan(g, 1, sref, labels, slow, den)
    x, d0 = wavefield(rng, 1, g), wavefield(rng, 1, g)
    full = np.repeat(slow[0], g.nw, axis=0) if shared else slow[0]
    y = to_host(p.scatter(0, to_dev(x), to_dev(d0), add=True))
    assert rel(y, wem.scatter_forward(g, full, x, d0)) < TOL
    y = to_host(p.scatter(0, to_dev(x), to_dev(d0), adjoint=True, add=True))
    assert rel(y, wem.scatter_adjoint(g, full, x, d0)) < TOL


# and rows of the compile-time plan, of two and of three run-time stages
@pytest.mark.parametrize("nx,ny,padx,pady", NEITHER + [(250, 18, 6, 2), (45, 40, 5, 8), (140, 20, 7, 1), (64, 64, 0, 0)])
@pytest.mark.parametrize("nref", [1, 3])
def test_smooth_steps_and_derivative(nx, ny, padx, pady, nref):
    """References far apart and deep steps: w dz (s_{j+1} - s_j) of 0.26 radian and more, so
    that the derivative's difference of neighbouring terms keeps its digits."""
    g, rng, _, _, _, _ = make_case(nx=nx, ny=ny, padx=padx, pady=pady, nw=2, nz=1, nref=nref)
    g.dz, g.ow, g.dw = 25.0, 10.0, 10.0
    s = rng.uniform(1 / 3000.0, 1 / 1500.0, (1, ny, nx))
    refs = wem.smooth_refs(s, nref).astype(np.float32)
    s = s.astype(np.float32)
    s[0, 0, : nx // 2] = np.float32(0.95) * refs[0, 0]
    s[0, -1, nx // 2:] = np.float32(1.05) * refs[0, -1]
    sp = wem.pad_edge(g, s.astype(np.float64))
    p = Plan(nx=nx, ny=ny, nw=g.nw, ns=2, nz=1, dx=g.dx, dy=g.dy, dz=g.dz, ow=g.ow, dw=g.dw, padx=padx, pady=pady,
             nref=nref, taperx=g.taperx, tapery=g.tapery)
    p.set_smooth(sp.astype(np.float32), refs)
    r64 = refs[0].astype(np.float64)
    x, d0, d1 = (wavefield(rng, 2, g) for _ in range(3))
    fwd, der = wem.smooth_forward(g, r64, sp[0], x), wem.smooth_deriv(g, r64, sp[0], x)
    assert rel(to_host(p.smooth_step(0, to_dev(x), to_dev(d0), add=True)), d0 + fwd) < TOL
    assert rel(to_host(p.smooth_step(0, to_dev(x), to_dev(d0), mode=L.SMOOTH_ADJ, add=True)),
               d0 + wem.smooth_adjoint(g, r64, sp[0], x)) < TOL
    empty = torch.empty(p.wshape, dtype=torch.complex64, device="cuda")
    assert rel(to_host(p.smooth_step(0, to_dev(x), empty, mode=L.SMOOTH_DERIV)), der) < TOL
    out, d = to_dev(d0), torch.empty_like(empty)
    p.smooth_step_pair(0, to_dev(x), out, d)
    assert rel(to_host(out), fwd) < TOL and rel(to_host(d), der) < TOL
    scale = np.linalg.norm(der) / np.linalg.norm(d1)  # the derivative's own size
    out, d = to_dev(d0), to_dev(scale * d1)
    p.smooth_step_pair(0, to_dev(x), out, d, add=True)
    assert rel(to_host(out), d0 + fwd) < TOL and rel(to_host(d), scale * d1 + der) < TOL
