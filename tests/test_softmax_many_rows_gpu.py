"""The row softmax where there are more rows than SMs: both sides of each line in rows and
in columns, and a row has the same bits whatever the number of rows.

Tolerance, in units of u = 2^-24 relative to the result: the sum is a chain of at most 32
terms in a thread and two trees of five steps, 42 roundings; exp is within 2 units in the
last place (4 u) in the term and in the sum; x - max is rounded, which exp turns into
|x - max| u, in the sum by the mean over the row with the probabilities as weights; one
division.  The fused head has the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu

COLS = [2048, 2049, 4096, 4097, 5001, 8192, 8193, 12384, 16381, 16384, 16385]


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def draw(rows, cols):
    g = torch.Generator(device="cuda").manual_seed(cols)
    x = torch.randn(rows, cols, device="cuda", generator=g) * 3
    x[0, :] = -float("inf")
    x[0, cols - 1] = 1.0
    return x, torch.randint(0, cols, (rows,), device="cuda", generator=g, dtype=torch.int32)


@pytest.mark.parametrize("cols", COLS)
@pytest.mark.parametrize("per_sm", [1, 2, 4])
@pytest.mark.parametrize("more", [0, 1])
def test_lines(cols, per_sm, more):
    from singa_b200 import singa_wrap as sw
    x, t = draw(per_sm * sms() + more, cols)
    p = sw.SoftMax(x)
    want = torch.softmax(x.double(), 1)
    below = torch.where(want > 0, x.amax(1, keepdim=True).double() - x.double(), 0.0)
    units = 42 + 4 + 4 + 1 + below + (want * below).sum(1, keepdim=True)
    assert bool(((p.double() - want).abs() <= units * 2.0 ** -24 * want + 1e-37).all())
    fp, fl, fg = sw.SoftMaxCrossEntropyFused(x, t, 0.5)
    assert torch.equal(fp, p) and torch.equal(fl, sw.CrossEntropyFwd(p, t))
    assert torch.equal(fg, sw.SoftmaxCrossEntropyBwd(p, t) * 0.5)


@pytest.mark.parametrize("cols", COLS)
def test_a_row_does_not_depend_on_the_others(cols):
    from singa_b200 import singa_wrap as sw
    many, few = sms() + 1, 7
    x, t = draw(many, cols)
    together, alone = sw.SoftMax(x), torch.cat([sw.SoftMax(x[i:i + few]) for i in range(0, many, few)])
    assert torch.equal(together, alone)
    heads = [sw.SoftMaxCrossEntropyFused(x[i:i + few].contiguous(), t[i:i + few].contiguous(), 0.5) for i in range(0, many, few)]
    for whole, parts in zip(sw.SoftMaxCrossEntropyFused(x, t, 0.5), zip(*heads)):
        assert torch.equal(whole, torch.cat(parts))
