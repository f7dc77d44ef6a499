"""What the Python layer answers for empty batches and for shapes with more or
fewer dimensions than a call speaks of."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def zeros(*shape, **kw):
    return torch.zeros(shape, device="cuda", **kw)


@pytest.mark.parametrize("shape", [(0, 4, 3, 3), (4, 0, 3, 3), (0, 0), (0, 4)])
def test_bias_gradient_of_an_empty_batch_is_an_error(shape):
    from singa_b200 import singa_wrap as sw
    with pytest.raises(ZeroDivisionError):
        sw.GpuConvBackwardb(zeros(*shape), None)


def test_bias_gradient_of_other_shapes():
    from singa_b200 import singa_wrap as sw
    with pytest.raises(IndexError):
        sw.GpuConvBackwardb(zeros(4), None)
    assert torch.equal(sw.GpuConvBackwardb(zeros(3, 5, 0, 2), None), zeros(5))       # empty planes: sums of nothing
    dy = torch.arange(30.0, device="cuda").view(2, 3, 5)
    assert torch.equal(sw.GpuConvBackwardb(dy, None), dy.sum((0, 2)))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
def test_cross_entropy_of_an_empty_batch_is_an_error(dtype):
    from singa_b200 import singa_wrap as sw
    p, t = zeros(0, 10, dtype=dtype), zeros(0, dtype=torch.int32)
    for call in (sw.CrossEntropyFwd, sw.SoftmaxCrossEntropyBwd):
        with pytest.raises(ZeroDivisionError):
            call(p, t)


def test_row_maximum_takes_the_first_two_sizes():
    from singa_b200 import singa_wrap as sw
    m = torch.randn(6, 7, device="cuda")
    assert torch.equal(sw.RowMax(m), m.max(1).values)
    assert torch.equal(sw.RowMax(m.view(6, 7, 1)), m.max(1).values)
    with pytest.raises(IndexError):
        sw.RowMax(m.view(-1))
