"""Chained launches keep stream order in the per-cell operators too: injection,
recording, imaging, linearised reflection, reflection, taper and correlation queued back
to back give what separately synchronised calls give, bit for bit, and whole sweeps
(chained) what the same sweeps on several streams (not chained) give."""
import numpy as np
import pytest
import torch

from pyfwix_b200 import _lib as L
from pyfwix_b200.plan import sweep
from tests.conftest import crandn
from tests.gpu_helpers import make_case, make_plan, rel, to_dev, to_host, wavefield

pytestmark = pytest.mark.gpu

SIZES = [(42, 30, 4), (64, 64, 8), (256, 150, 24), (128, 256, 96)]  # below and above one wave


def _traces(p, rng, g, ns, n=40):
    return p.traces(rng.uniform(0, (g.nx - 1) * g.dx, n), rng.uniform(0, (g.ny - 1) * g.dy, n), np.zeros(n),
                    np.arange(n) % ns)


@pytest.mark.parametrize("nx,ny,nw", SIZES)
@pytest.mark.parametrize("ns", [1, 2])
def test_operators_in_stream_order(nx, ny, nw, ns):
    g, rng, sref, labels, slow, den = make_case(nx=nx, ny=ny, nw=nw, nz=2, nref=2)
    p = make_plan(g, ns, sref, labels, slow, den)
    tr = _traces(p, rng, g, ns)
    x, bg = to_dev(wavefield(rng, ns, g)), to_dev(wavefield(rng, ns, g))
    t0 = to_dev(crandn(rng, (40, nw)))
    dm0 = to_dev(crandn(rng, (4, nw, ny, nx)))

    def walk(sync):
        w, u, t = x.clone(), torch.empty_like(x), t0.clone()
        dr, im, dm = dm0[0].clone(), torch.empty_like(dm0[0]), dm0.clone()
        img = torch.empty((g.NY, g.NX), dtype=torch.float32, device="cuda")
        out = []
        for k in range(4):
            for op in (lambda: p.inject(tr, 0, t, w), lambda: p.step(k % 2, w, u), lambda: p.imaging(u, dr, w, add=True),
                       lambda: p.inject(tr, 0, t, w, adjoint=True), lambda: p.reflect(0, w, u, add=True),
                       lambda: p.imaging(u, im, w, adjoint=True), lambda: p.lin_reflect(0, dm, im, adjoint=True),
                       lambda: p.lin_reflect(0, dm, dr), lambda: p.taper(u, w), lambda: p.correlate(w, u, img),
                       lambda: w.mul_(img.abs().mean().rsqrt()), lambda: t.mul_(t.abs().mean().reciprocal()),
                       lambda: dr.mul_(dr.abs().mean().reciprocal()), lambda: dm.mul_(dm.abs().mean().reciprocal())):
                op()
                if sync:
                    torch.cuda.synchronize()
            out += [v.clone() for v in (w, u, t, dr, im, dm, img)]
        return out

    want = walk(True)
    assert all(torch.isfinite(torch.view_as_real(v) if v.is_complex() else v).all() for v in want)
    for _ in range(3):
        assert all(torch.equal(a, b) for a, b in zip(walk(False), want))


@pytest.mark.parametrize("nx,ny,nw", SIZES)
@pytest.mark.parametrize("shared", [True, False])
def test_sweeps_chained_and_not(nx, ny, nw, shared):
    g, rng, sref, labels, slow, den = make_case(nx=nx, ny=ny, nw=nw, nz=3, nref=2)
    if shared:
        slow, den = slow[:, :1], den[:, :1]
    wav, ds = to_dev(crandn(rng, (1, nw))), to_dev(0.1 * slow)
    inst = []
    for k in range(2):
        p = make_plan(g, 1, sref, labels, slow, den)
        rec = _traces(p, np.random.default_rng(k), g, 1)
        src = p.traces([nx * 3.0 + 20 * k], [ny * 4.0], [0.0], [0])
        inst.append(dict(plan=p, src=src, rec=rec))
    streams = [torch.cuda.Stream() for _ in range(2)]

    def run(lanes):
        out = []
        for q in inst:
            q.update(wavelet=wav, data=torch.zeros((40, nw), dtype=torch.complex64, device="cuda"),
                     image=torch.zeros((3, ny, nx), device="cuda"),
                     bg_down=torch.empty((3,) + q["plan"].wshape, dtype=torch.complex64, device="cuda"),
                     bg_up=torch.empty((3,) + q["plan"].wshape, dtype=torch.complex64, device="cuda"))
        sweep(L.SWEEP_MODEL, inst, lanes)
        out += [q["data"].clone() for q in inst]
        sweep(L.SWEEP_IMAGE, inst, lanes)
        img = [q["image"].clone() for q in inst]
        born = [dict(q, dslow=ds.clone(), dden=ds.clone(), data=torch.zeros_like(q["data"])) for q in inst]
        sweep(L.SWEEP_BORN_FWD, born, lanes)
        out += [q["data"].clone() for q in born]
        born = [dict(q, dslow=torch.zeros_like(ds), dden=torch.zeros_like(ds), adjoint=1) for q in inst]
        sweep(L.SWEEP_BORN_ADJ, born, lanes)
        out += [q[k] for q in born for k in ("dslow", "dden")]
        torch.cuda.synchronize()
        return out, img

    want, wimg = run(streams)
    for _ in range(2):
        got, gimg = run([])
        assert all(torch.equal(a, b) and a.abs().max() > 0 for a, b in zip(got, want))
        # the image may be summed by atomics: nw terms per cell, 6e-8 each in any order
        assert all(rel(to_host(a), to_host(b)) < 6e-8 * nw for a, b in zip(gimg, wimg))
