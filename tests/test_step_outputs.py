"""The output of a single depth step is written without a zero fill before it; what the
fill refused, recorded or separated stays so."""
import numpy as np
import pytest
import torch
from torch.autograd import forward_ad

from pyfwix_b200.CudaWEM import _out

CPU = torch.device("cpu")


def _field(n=8):
    return torch.randn(n, dtype=torch.complex64)


def test_plain_operand_is_itself():
    src, t = _field(), _field()
    want = t.clone()
    out = _out(t, CPU, src)
    assert out is t and torch.equal(t, want)


def test_other_sizes_and_types_are_zeroed():
    src = _field()
    t = _field(12)
    assert _out(t, CPU, src) is t and not t.any()
    assert not _out(np.ones(8, np.complex64), CPU, src).any()
    t = torch.ones(8, dtype=torch.complex128)
    assert not _out(t, CPU, src).any()


def test_leaf_that_requires_grad_is_refused():
    t = _field().requires_grad_()
    with pytest.raises(RuntimeError):
        _out(t, CPU, _field())
    with torch.no_grad():
        assert _out(t, CPU, _field()) is t


def test_saved_tensor_is_seen_to_change():
    a, t = _field().requires_grad_(), _field()
    y = (a * t).abs().sum()
    _out(t, CPU, _field())
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward()


def test_forward_mode_tangent_does_not_survive():
    with forward_ad.dual_level():
        t = forward_ad.make_dual(_field(), _field())
        _out(t, CPU, _field())
        tangent = forward_ad.unpack_dual(t).tangent
        assert tangent is None or not tangent.any()


def test_inference_tensors_stay_as_they_were():
    with torch.inference_mode():
        t = _field()
        assert _out(t, CPU, _field()) is t
    with pytest.raises(RuntimeError):
        _out(t, CPU, _field())


@pytest.mark.parametrize("shift", [-7, -1, 0, 1, 7])
def test_overlap_across_storages_is_zeroed_first(shift):
    buf = np.ones(32, np.complex64)
    src = torch.from_numpy(buf[8:16])
    t = torch.from_numpy(buf[8 + shift:16 + shift])
    _out(t, CPU, src)
    assert not t.any() and int(src.abs().sum()) == abs(shift)
    beside = torch.from_numpy(buf[16:24])
    beside[:] = 1
    assert _out(beside, CPU, src).all()
