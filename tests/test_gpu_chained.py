"""Chained launches (a kernel's prologue under the kernel before it) keep stream order:
steps queued back to back, captured into a graph, or interleaved with other work on
the same buffers and with another stream, give what separately synchronised steps
give, bit for bit."""
import pytest
import torch

from tests.gpu_helpers import make_case, make_plan, to_dev, wavefield

pytestmark = pytest.mark.gpu

# less than a wave and more than one, compile-time and run-time lengths
SIZES = [(42, 30, 4), (64, 64, 8), (256, 150, 24), (128, 256, 96)]


def _case(nx, ny, nw, step):
    g, rng, sref, labels, slow, den = make_case(nx=nx, ny=ny, nw=nw, nz=3, nref=3)
    p = make_plan(g, 1, sref, labels, slow, den, step=step)
    return p, to_dev(wavefield(rng, 1, g))


def _walk(p, x, sync):
    """Steps, scatterings and reflections in place and out of place, ping-pong over two
    buffers, each reading what the one before has just written."""
    a, b = x.clone(), torch.empty_like(x)
    out = []
    for k in range(6):
        iz = k % 3
        for op in (lambda: p.step(iz, a, b, direction=k % 3), lambda: p.scatter(iz, b, a, adjoint=bool(k % 2)),
                   lambda: p.step(iz, a, a), lambda: p.reflect(iz, a, b, add=True), lambda: p.taper(b, a),
                   lambda: a.mul_(2.0 ** (k % 5)), lambda: p.step(iz, a, b, add=True)):
            op()
            if sync:
                torch.cuda.synchronize()
        n = torch.linalg.vector_norm(b)
        a.copy_(b / n)
        out.append(a.clone())
    return out


@pytest.mark.parametrize("nx,ny,nw", SIZES)
@pytest.mark.parametrize("step", ["pspi", "nsps"])
def test_stream_order(nx, ny, nw, step):
    p, x = _case(nx, ny, nw, step)
    want = _walk(p, x, sync=True)
    for _ in range(3):
        got = _walk(p, x, sync=False)
        assert all(torch.equal(u, v) for u, v in zip(got, want))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        got = _walk(p, x, sync=False)
    torch.cuda.current_stream().wait_stream(side)
    assert all(torch.equal(u, v) for u, v in zip(got, want))


@pytest.mark.parametrize("nx,ny,nw", SIZES)
def test_capture(nx, ny, nw):
    p, x = _case(nx, ny, nw, "pspi")
    a, b = x.clone(), torch.empty_like(x)

    def work():
        for k in range(3):
            p.step(k, a, b)
            p.step(k, b, a, direction=1)

    work()
    want = a.clone()
    a.copy_(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        work()
    for _ in range(2):
        a.copy_(x)
        graph.replay()
        assert torch.equal(a, want)
