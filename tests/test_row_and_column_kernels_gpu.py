"""Column sums, channel sums and the row softmax where their plans change: one
CTA, a full cluster, more slices than a cluster; rows held by a warp, by CTAs of
each size, and rows too long for registers; odd lengths and misaligned rows.

Tolerances.  A sum of n fp32 terms in any order is off by at most
(n - 1) * 2^-24 * sum |x|; the sums here have at most 2^17 terms per chain but
are formed by trees and short chains (< 600 additions deep), so
600 * 2^-24 * sum |x| is a bound.  Softmax: exp is within 2 ulp, the sum within
600 * 2^-24 and the division within 1 ulp of it: 4e-5 relative.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEPTH = 600 * 2.0 ** -24


def gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


@pytest.mark.parametrize("shape", [(1, 1), (2, 3), (7, 16), (64, 17), (257, 31), (256, 10), (31, 33), (600, 1000),
                                   (256, 4096), (3, 4100), (5000, 10), (100000, 7), (70000, 130), (4096, 4099)])
def test_column_sums(shape):
    from singa_b200 import singa_wrap as sw
    for offset in (0, 1):                 # 1: rows start off a 16-byte boundary
        flat = torch.randn(shape[0] * shape[1] + offset, device="cuda", generator=gen(shape[0]))
        M = flat[offset:].view(shape)
        got = sw.SumRows(M).double()
        assert bool(((got - M.double().sum(0)).abs() <= DEPTH * M.double().abs().sum(0) + 1e-30).all())
        assert torch.equal(sw.SumRows(M), sw.SumRows(M))


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (3, 5, 7, 7), (64, 32, 24, 24), (64, 32, 8, 8), (2, 300, 3, 5),
                                   (64, 2, 112, 112), (257, 3, 33, 31)])
def test_channel_sums(shape):
    from singa_b200 import singa_wrap as sw
    dy = torch.randn(shape, device="cuda", generator=gen(shape[1]))
    got = sw.GpuConvBackwardb(dy).double()
    want, size = dy.double().sum((0, 2, 3)), dy.double().abs().sum((0, 2, 3))
    assert bool(((got - want).abs() <= DEPTH * size).all())


@pytest.mark.parametrize("cols", [1, 10, 127, 128, 129, 512, 513, 1000, 1025, 2048, 4097, 8192, 16385, 32768, 32769])
@pytest.mark.parametrize("rows", [1, 5])
def test_softmax_and_loss_head(cols, rows):
    from singa_b200 import singa_wrap as sw
    x = torch.randn(rows, cols, device="cuda", generator=gen(cols)) * 3
    t = torch.randint(0, cols, (rows,), device="cuda", generator=gen(cols), dtype=torch.int32)
    want = torch.softmax(x.double(), 1)
    p = sw.SoftMax(x)
    assert bool(((p.double() - want).abs() <= 4e-5 * want + 1e-37).all())
    loss, g = sw.CrossEntropyFwd(p, t), sw.SoftmaxCrossEntropyBwd(p, t)
    hot = torch.zeros_like(p).scatter_(1, t.long().view(-1, 1), 1.0)
    assert torch.equal(g, p - hot)
    fp, fl, fg = sw.SoftMaxCrossEntropyFused(x, t, 0.25)
    assert torch.equal(fp, p) and torch.equal(fl, loss) and torch.equal(fg, g * 0.25)
    h = x.half()
    ph = sw.SoftMax(h)
    wh = torch.softmax(h.double(), 1)
    # one rounding to fp16 (half an ulp; 2^-25 where the result is subnormal)
    assert bool(((ph.double() - wh).abs() <= (2.0 ** -11 + 4e-5) * wh + 2.0 ** -25).all())
    gh = sw.SoftmaxCrossEntropyBwd(ph, t)
    assert torch.equal(gh, ph - hot.half())
