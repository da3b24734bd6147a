"""Hat weights and split-step phases of the smooth steps, apart from the transforms.

A depth whose slowness is reference r everywhere gives T_r, the transform pair of that
reference as the device computes it; a depth of varying slowness is then the sum over r of
w_r exp(-i w (s - s_r) dz) T_r, formed here in 64 bits, and only the weights' and
phases' own rounding is left.  With u = 2^-24 (rms of a rounding 0.4 u): two factors from
sines and their products with the sample in T_r, the same and the weighted sum in the
result, 1.8 u = 1.05e-7 together; the bound is twice that."""
import numpy as np
import pytest
import torch

from pyfwix_b200 import _lib as L
from pyfwix_b200.plan import Plan
from tests.conftest import crandn
from tests.gpu_helpers import rel, to_dev, to_host

pytestmark = pytest.mark.gpu

TOL = 2.1e-7
# rows of the compile-time plan, of two and three run-time stages, of neither
SIZES = [(256, 20), (50, 45), (147, 24), (15, 30)]


def _case(nx, ny, n, dz, fmax, clamped=True):
    rng = np.random.default_rng(n + nx)
    lo, hi = 1.0 / 2200.0, 1.0 / 1500.0
    refs = np.linspace(lo, hi, n).astype(np.float32) if n > 1 else np.array([lo], np.float32)
    s = rng.uniform(lo, hi, (ny, nx)).astype(np.float32)
    # clamped cells; cells on a reference and one step below and above it
    if clamped:
        s.flat[0::7] = rng.choice([0.9 * lo, 1.1 * hi], s.flat[0::7].size).astype(np.float32)
    s.flat[1::7] = rng.choice(refs, s.flat[1::7].size)
    s.flat[2::7] = np.nextafter(rng.choice(refs, s.flat[2::7].size), np.float32(0))
    s.flat[3::7] = np.nextafter(rng.choice(refs, s.flat[3::7].size), np.float32(1))
    p = Plan(nx=nx, ny=ny, nw=3, ns=1, nz=n + 1, dx=25.0, dy=25.0, dz=dz, ow=0.4 * fmax, dw=0.3 * fmax, nref=n)
    p.set_smooth(np.stack([np.full_like(s, r) for r in refs] + [s]), np.repeat(refs[None], n + 1, axis=0))
    w = 2 * np.pi * (0.4 + 0.3 * np.arange(3)) * fmax
    x = crandn(rng, (1, 3, ny, nx))
    return p, refs.astype(np.float64), s.astype(np.float64), w, x


def _hat(refs, s):
    """Weights [n][ny][nx] and their derivatives, clamped outside the references."""
    n = len(refs)
    wt, dw = np.zeros((n,) + s.shape), np.zeros((n,) + s.shape)
    if n == 1:
        wt[0] = 1
        return wt, dw
    wt[0][s <= refs[0]] = 1
    wt[-1][s >= refs[-1]] = 1
    j = np.clip(np.searchsorted(refs, s, side="right") - 1, 0, n - 2)
    inside = (s > refs[0]) & (s < refs[-1])
    span = refs[j + 1] - refs[j]
    u = (s - refs[j]) / span
    iy, ix = np.nonzero(inside)
    wt[j[inside], iy, ix], wt[j[inside] + 1, iy, ix] = 1 - u[inside], u[inside]
    dw[j[inside], iy, ix], dw[j[inside] + 1, iy, ix] = -1 / span[inside], 1 / span[inside]
    return wt, dw


def _run(p, iz, x, mode):
    return to_host(p.smooth_step(iz, to_dev(x), torch.empty(p.wshape, dtype=torch.complex64, device="cuda"), mode=mode))


CASES = [(1, 10.0, 40.0), (4, 10.0, 40.0), (4, 50.0, 100.0), (32, 10.0, 40.0), (40, 50.0, 100.0), (128, 10.0, 40.0),
         (200, 10.0, 40.0)]


def _forward_and_derivative(case, n, dz):
    p, refs, s, w, x = case
    wt, dw = _hat(refs, s)
    wdz = (w * dz)[None, :, None, None]
    want, wder, mag = 0, 0, 0
    for r in range(n):
        T = _run(p, r, x, L.SMOOTH_FWD)
        ss = np.exp(-1j * wdz * (s - refs[r])) * T
        want = want + wt[r] * ss
        wder = wder + (dw[r] - 1j * wdz * wt[r]) * ss
        mag = mag + (np.abs(dw[r]) + wdz * wt[r]) * np.abs(T)
    assert rel(_run(p, n, x, L.SMOOTH_FWD), want) < TOL
    # the derivative is a difference of neighbouring terms: its error is relative to them
    assert np.linalg.norm(_run(p, n, x, L.SMOOTH_DERIV) - wder) < TOL * np.linalg.norm(mag)
    out, der = (torch.empty(p.wshape, dtype=torch.complex64, device="cuda") for _ in range(2))
    p.smooth_step_pair(n, to_dev(x), out, der)
    assert rel(to_host(out), want) < TOL
    assert np.linalg.norm(to_host(der) - wder) < TOL * np.linalg.norm(mag)


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("n,dz,fmax", CASES)
def test_forward_and_derivative(nx, ny, n, dz, fmax):
    _forward_and_derivative(_case(nx, ny, n, dz, fmax), n, dz)


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("n", [128, 255])
def test_every_bit_of_the_weights(nx, ny, n):
    """Many references on steps of 2 km, so that neighbouring ones give transforms a radian or
    two apart and a weight's error is not cancelled by its neighbour's.  (Beside the
    roundings above only that of the frequency, 0.6 u of a bracket's 2 radians at most:
    the same bound.  No cells beyond the references: those are 60 radians away.)"""
    _forward_and_derivative(_case(nx, ny, n, 2000.0, 100.0, clamped=False), n, 2000.0)


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("n,dz,fmax", CASES)
def test_adjoint(nx, ny, n, dz, fmax):
    """The adjoint's weights come before the transforms: the terms here round them to
    float on their way through the device, and both sides carry the rounding of a
    transform pair of up to 25 levels (0.8 u each in rms), 3.4e-7 together; bound 6e-7."""
    p, refs, s, w, x = _case(nx, ny, n, dz, fmax)
    wt, _ = _hat(refs, s)
    wdz = (w * dz)[None, :, None, None]
    want = 0
    for r in range(n):
        want = want + _run(p, r, wt[r] * np.exp(1j * wdz * (s - refs[r])) * x, L.SMOOTH_ADJ)
    assert rel(_run(p, n, x, L.SMOOTH_ADJ), want) < 6e-7
