"""Both sides of the lines from which a batch norm visits its data twice: against fp64,
and a fused call has the bits of its parts.  Tolerances as in test_bn_two_visits_gpu.py."""
import pytest
import torch
from test_bn_two_visits_gpu import Backward, close, no_faults, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 488, 6148, 1), (1, 489, 6144, 1), (2, 487, 3076, 1),     # whole vectors: 6144 a channel, 3e6
                                   (16, 686, 401, 1), (16, 685, 401, 1), (17, 650, 399, 1)])    # odd planes of 400, 4.4e6
def test_backward(shape):
    b = Backward(shape, 7)
    outs = [b.run(mask) for mask in (0, 1, 2)]
    for mask in (0, 1, 2):
        assert close(outs[mask], b.want(mask), b), (shape, mask)
    assert all(torch.equal(p, q) for p, q in zip(outs[1], outs[2])), "float mask != bit record"
    b.dy = torch.where(b.r > 0, b.dy, 0.0)
    assert all(torch.equal(p, q) for p, q in zip(outs[1], b.run(0))), "fused call != its parts"
    assert no_faults()


@pytest.mark.parametrize("shape", [(36, 62, 901, 1), (36, 61, 901, 1), (36, 64, 899, 1), (35, 66, 901, 1)])
def test_forward(shape):
    from singa_b200 import singa_wrap as sw
    g = torch.Generator(device="cuda").manual_seed(8)
    x = torch.randn(shape, device="cuda", generator=g) * 1.5 + 3.0
    c = shape[1]
    scale, bias = torch.rand(c, device="cuda", generator=g) + 0.5, torch.randn(c, device="cuda", generator=g)
    y, mean, inv = sw.GpuBatchNormForwardTraining(sw.CudnnBatchNormHandle(0.1, x), x, scale, bias, torch.zeros(c, device="cuda"),
                                                  torch.ones(c, device="cuda"), 1e-5)
    X, col = x.double(), (1, -1, 1, 1)
    mu, var = X.mean((0, 2, 3)), X.var((0, 2, 3), unbiased=False)
    want = (var + 1e-5).rsqrt()
    assert rel(mean, mu) <= 2e-6 and rel(inv, want) <= 4e-6
    assert rel(y, (X - mu.view(col)) * (scale.double() * want).view(col) + bias.double().view(col)) <= 4e-6
    assert no_faults()
