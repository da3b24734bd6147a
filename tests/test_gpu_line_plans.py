"""The run-time-length row and column passes (flex.cuh) against the FP64 oracle, at the
lengths where they can go wrong: every 7-smooth length once as rows and once as
columns, then every kind of pass on two- and three-stage lines, kernels of a
length's own and shared ones, odd pitches, pads, and grids that mix them with the
compile-time plans.  Tolerances as in test_gpu_ops: 1e-5 per operator; 2e-6 for a
plain transform (20 rounded radix-2 levels of 6e-8 each at 1024 x 1024)."""
import numpy as np
import pytest
import torch

from oracle import wem
from tests.conftest import crandn
from tests.gpu_helpers import make_case, make_plan, oracle_labels, rel, to_dev, to_host, wavefield

pytestmark = pytest.mark.gpu

TOL = 1e-5
FFT_TOL = 2e-6


def _seven_smooth(n):
    for f in (2, 3, 5, 7):
        while n % f == 0:
            n //= f
    return n == 1


@pytest.mark.parametrize("first,last", [(1, 64), (65, 256), (257, 512), (513, 1024)])
def test_every_length(first, last):
    for n in filter(_seven_smooth, range(first, last + 1)):
        for NX, NY in ((n, 3), (5, n)):
            g, rng, sref, labels, _, _ = make_case(nx=NX, ny=NY, nw=2, nz=1, nref=1)
            p = make_plan(g, 1, sref, labels)
            x = wavefield(rng, 1, g)
            y = torch.empty(p.wshape, dtype=torch.complex64, device="cuda")
            assert rel(to_host(p.fft2d(to_dev(x), y)), wem.fft2(x)) < FFT_TOL, (NX, NY)
            assert rel(to_host(p.fft2d(to_dev(x), y, inverse=True)), wem.ifft2(x)) < FFT_TOL, (NX, NY)


SIZES = [  # nx, ny, padx, pady
    (14, 16, 0, 0),      # the smallest plans, run-time radices
    (147, 49, 0, 0),     # three stages at run time, odd pitch
    (330, 100, 13, 5),   # 343 = 7 7 7 and 105 = 7 15, padded
    (200, 168, 0, 0),    # radix 20, radix 14
    (270, 216, 0, 0),    # radix 18
    (500, 27, 0, 0),     # three stages, kernels of its own; run-time columns
    (18, 1024, 0, 0),    # the longest column
    (1000, 15, 8, 0),    # the longest three-stage row; a column with neither plan
    (256, 150, 0, 0),    # compile-time rows, run-time columns
    (135, 64, 0, 0),     # and the other way round
]


@pytest.mark.parametrize("nx,ny,padx,pady", SIZES)
@pytest.mark.parametrize("eps,nref", [(0.0, 4), (0.01, 3)])
def test_steps(nx, ny, padx, pady, eps, nref):
    g, rng, sref, labels, _, _ = make_case(nx=nx, ny=ny, padx=padx, pady=pady, nw=2, nz=2, nref=nref, eps=eps,
                                           complex_refs=eps > 0, labels_per_w=eps > 0)
    # rows whose cells take one reference only: the passes skip the others
    labels[:, :, : g.NY // 2] = labels[:, :, :1, :1]
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


@pytest.mark.parametrize("nx,ny,padx,pady", SIZES)
@pytest.mark.parametrize("taylor,shared", [(1, True), (2, False), (0, True)])
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
    buf = to_dev(x)
    assert rel(to_host(p.scatter(0, buf, buf, adjoint=True)), wem.scatter_adjoint(g, full, x)) < TOL


@pytest.mark.parametrize("nx,ny,padx,pady", SIZES)
@pytest.mark.parametrize("nref", [1, 4])
def test_smooth_steps(nx, ny, padx, pady, nref):
    g, rng, _, labels, _, _ = make_case(nx=nx, ny=ny, padx=padx, pady=pady, nw=2, nz=1, nref=nref)
    s = 1.0 / 1800.0 * (1 + 0.2 * rng.random((1, ny, nx)))
    refs = wem.smooth_refs(s, nref).astype(np.float32)
    s = s.astype(np.float32)
    # cells outside the references (clamped) and exactly on them
    s[0, 0, :] = np.float32(0.9) * refs[0, 0]
    s[0, -1, :] = np.float32(1.1) * refs[0, -1]
    s[0, ny // 2, : nref] = refs[0, : min(nref, nx)]
    sp = wem.pad_edge(g, s.astype(np.float64))
    from pyfwix_b200 import _lib as L
    from pyfwix_b200.plan import Plan
    p = Plan(nx=nx, ny=ny, nw=g.nw, ns=1, nz=1, dx=g.dx, dy=g.dy, dz=g.dz, ow=g.ow, dw=g.dw, padx=padx, pady=pady,
             nref=nref, taperx=g.taperx, tapery=g.tapery)
    p.set_smooth(sp.astype(np.float32), refs)
    r64 = refs[0].astype(np.float64)
    x, d0, d1 = (wavefield(rng, 1, g) for _ in range(3))
    y = to_host(p.smooth_step(0, to_dev(x), to_dev(d0), add=True))
    assert rel(y, d0 + wem.smooth_forward(g, r64, sp[0], x)) < TOL
    y = to_host(p.smooth_step(0, to_dev(x), to_dev(d0), mode=L.SMOOTH_ADJ, add=True))
    assert rel(y, d0 + wem.smooth_adjoint(g, r64, sp[0], x)) < TOL
    # (the derivative's values are checked in test_gpu_fwi, on references far enough
    # apart that its difference of neighbouring terms is well conditioned)
    out, der = to_dev(d0), to_dev(d1)
    p.smooth_step_pair(0, to_dev(x), out, der, add=True)
    assert rel(to_host(out), d0 + wem.smooth_forward(g, r64, sp[0], x)) < TOL


@pytest.mark.parametrize("nx,ny,pad", [(50, 45, 0), (42, 57, 6), (64, 63, 0), (98, 64, 0)])
@pytest.mark.parametrize("step", ["pspi", "nsps"])
def test_born_shared_model(nx, ny, pad, step):
    """Born forward and adjoint on a model shared by every frequency, where the
    reflections ride in the row passes."""
    ns = 2
    g, rng, sref, labels, slow, den = make_case(nx=nx, ny=ny, padx=pad, pady=pad, nw=3, nz=4, nref=3, taperx=0,
                                                tapery=0)
    slow, den = slow[:, :1], den[:, :1]
    lab = oracle_labels(labels, g)
    p = make_plan(g, ns, sref, labels, slow, den, step=step)
    slow_w, den_w = (np.repeat(v, g.nw, axis=1) for v in (slow, den))
    geom = dict(sx=[nx * 4.0, nx * 6.0], sy=[ny * 5.0, ny * 7.0], sz=[0.0, 0.0], s_ids=[0, 1],
                rx=rng.uniform(0, (nx - 1) * g.dx, 24), ry=rng.uniform(0, (ny - 1) * g.dy, 24),
                rz=np.zeros(24), r_ids=np.arange(24) % 2)
    acq = wem.make_acquisition(g, geom)
    st = wem.Stepper(g, sref, lab, kind=step)
    wav = crandn(rng, (2, g.nw))
    _, bd, bu = wem.propagate(g, st, acq, slow_w, den_w, wav)
    ds = 0.1 * slow * (1 + crandn(rng, slow.shape).real)
    dr = 0.1 * crandn(rng, den.shape).real
    want = wem.born_forward(g, st, acq, slow_w, den_w, bd, bu, np.repeat(ds, g.nw, axis=1), np.repeat(dr, g.nw, axis=1))
    rec = p.traces(geom["rx"], geom["ry"], geom["rz"], geom["r_ids"])
    D, U = to_dev(np.stack(bd)), to_dev(np.stack(bu))
    data = torch.zeros((24, g.nw), dtype=torch.complex64, device="cuda")
    p.born(rec, D, U, to_dev(ds), to_dev(dr), data)
    assert rel(to_host(data), want) < 1e-4
    d = crandn(rng, (24, g.nw))
    gs, gr = wem.born_adjoint(g, st, acq, slow_w, den_w, bd, bu, d)
    ms, mr = (torch.zeros((g.nz, 1, ny, nx), dtype=torch.complex64, device="cuda") for _ in range(2))
    p.born(rec, D, U, ms, mr, to_dev(d), adjoint=True)
    assert rel(to_host(ms)[:, 0], gs.sum(axis=1)) < 1e-4
    assert rel(to_host(mr)[:, 0], gr.sum(axis=1)) < 1e-4
