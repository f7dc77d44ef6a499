"""The row softmax where there are more rows than the SMs hold with four vectors a
thread: both sides of each line in rows and in columns.  Tolerance: exp is within 2
units in the last place, the sum of up to 32768 terms (trees over 32 per thread) within
600 * 2^-24, the division within one: 4e-5 relative.  The fused head has the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [2048, 2049, 4096, 4097, 5001, 8192, 8193, 16384, 16385])
@pytest.mark.parametrize("per_sm", [1, 2, 4])
@pytest.mark.parametrize("more", [0, 1])
def test_lines(cols, per_sm, more):
    from singa_b200 import singa_wrap as sw
    rows = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    g = torch.Generator(device="cuda").manual_seed(cols)
    x = torch.randn(rows, cols, device="cuda", generator=g) * 3
    x[0, :] = -float("inf")
    x[0, cols - 1] = 1.0
    t = torch.randint(0, cols, (rows,), device="cuda", generator=g, dtype=torch.int32)
    p = sw.SoftMax(x)
    want = torch.softmax(x.double(), 1)
    assert bool(((p.double() - want).abs() <= 4e-5 * want + 1e-37).all())
    fp, fl, fg = sw.SoftMaxCrossEntropyFused(x, t, 0.5)
    assert torch.equal(fp, p) and torch.equal(fl, sw.CrossEntropyFwd(p, t))
    assert torch.equal(fg, sw.SoftmaxCrossEntropyBwd(p, t) * 0.5)
