"""swap_storage: what an in-place exchange has to keep -- object identity, views of the old
buffers, offsets into a larger buffer, version counters, gradients flags, inference mode."""
import pytest

torch = pytest.importorskip("torch")

from thermal_inflation_phase_transition_b200._common import dims_of, swap_storage  # noqa: E402


def _pair(shape, offset):
    n = 1
    for x in shape:
        n *= x
    buf = torch.arange(float(2 * n + offset))
    return buf[offset:offset + n].view(shape), torch.arange(-float(n), 0.0).view(shape)


@pytest.mark.parametrize("shape", [(1, 1, 3), (2, 5, 7), (2, 3, 4, 5)])
@pytest.mark.parametrize("offset", [0, 3])
def test_exchange(shape, offset):
    a, b = _pair(shape, offset)
    wa, wb, pa, pb = a.clone(), b.clone(), a.data_ptr(), b.data_ptr()
    va, vb = a.view(-1), b[..., 0]
    ia, ib = a, b
    na, nb = a._version, b._version
    swap_storage(a, b)
    assert a is ia and b is ib
    assert a.data_ptr() == pb and b.data_ptr() == pa
    assert torch.equal(a, wb) and torch.equal(b, wa)
    assert torch.equal(va, wa.view(-1)) and torch.equal(vb, wb[..., 0])
    assert a.is_contiguous() and b.is_contiguous() and a.shape == torch.Size(shape)
    assert a._version > na and b._version > nb
    a.fill_(1.0)
    assert torch.equal(vb, torch.ones_like(vb)) and torch.equal(b, wa)
    assert dims_of(a) == tuple(shape[-3:]) and all(type(x) is int for x in dims_of(a))
    swap_storage(a, b)
    assert a.data_ptr() == pa and b.data_ptr() == pb


def test_saved_tensors_are_still_checked():
    a, b = torch.ones(2, 3, 4), torch.zeros(2, 3, 4)
    w = torch.ones(2, 3, 4, requires_grad=True)
    y = (a * w).sum()                # saves a
    swap_storage(a, b)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward()


def test_leaf_and_inference_mode():
    a, b = torch.ones(2, 3, 4, requires_grad=True), torch.zeros(2, 3, 4)
    swap_storage(a, b)
    assert a.requires_grad and not b.requires_grad and a.is_leaf
    assert float(a.detach().sum()) == 0.0 and float(b.sum()) == 24.0
    with torch.inference_mode():
        c, d = torch.ones(2, 3, 4), torch.zeros(2, 3, 4)
        swap_storage(c, d)
        assert float(c.sum()) == 0.0 and float(d.sum()) == 24.0
    with pytest.raises(RuntimeError):
        swap_storage(c, d)
    assert float(c.sum()) == 0.0
