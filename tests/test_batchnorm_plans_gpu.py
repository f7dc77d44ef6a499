"""Batch norm, forward and backward, where the choice of kernel changes: channels
held by a warp, by CTAs of each size, by clusters, by none; planes that are a
multiple of four floats, odd ones (channel groups, aligned vectors with masked
ends), tiny ones; tensors off a 16-byte boundary.  Reference: the formulas in
fp64.

Tolerance: a sum of M terms by trees over chains of at most 2^10 additions is
off by at most 2^10 * 2^-24 = 6e-5 of the sum of magnitudes in the worst case;
rounding errors of that many additions are independent, so their root mean
square (what `rel` measures) stays below sqrt(2^10) * 2^-24 = 2e-6."""
import pytest
import torch

pytestmark = pytest.mark.gpu

#         n, c, h, w
SHAPES = [(1, 1, 1, 1), (1, 5, 4, 32), (1, 5, 4, 33), (4, 7, 8, 8), (4, 7, 8, 16), (4, 6, 16, 16), (4, 6, 16, 36),
          (8, 5, 32, 32), (1, 9, 64, 96), (1, 9, 64, 97), (4, 3, 46, 46), (33, 8, 7, 7), (33, 6, 7, 7), (9, 5, 2, 3),
          (16, 10, 27, 27), (17, 48, 35, 29), (40, 3, 57, 57), (65, 2, 111, 113), (64, 2, 112, 112), (2, 300, 13, 13),
          (32, 75, 56, 56), (7, 300, 44, 44), (11, 299, 28, 28)]


def rel(got, want):
    return float((got.double() - want).norm() / (want.norm() + 1e-300))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("offset", [0, 1])
def test_against_fp64(shape, offset):
    from singa_b200 import _lib, singa_wrap as sw
    n, c, h, w = shape
    m = n * h * w
    g = torch.Generator(device="cuda").manual_seed(m + c)

    def make(std=1.0, mean=0.0):
        flat = torch.empty(m * c + offset, device="cuda")[offset:]
        return flat.copy_(torch.randn(m * c, device="cuda", generator=g) * std + mean).view(shape)

    x, dy, relu_in = make(1.5, 3.0), make(1e-2), make()
    scale, bias = torch.rand(c, device="cuda", generator=g) + 0.5, torch.randn(c, device="cuda", generator=g)
    handle = sw.CudnnBatchNormHandle(0.1, x)
    rm, rv = torch.zeros(c, device="cuda"), torch.ones(c, device="cuda")
    y, mean, invstd = sw.GpuBatchNormForwardTraining(handle, x, scale, bias, rm, rv, 1e-5)
    X, col = x.double(), (1, c, 1, 1)
    mu = X.mean((0, 2, 3))
    var = (X - mu.view(col)).square().mean((0, 2, 3))
    inv = (var + 1e-5).rsqrt()
    assert rel(mean, mu) <= 2e-6 and rel(invstd, inv) <= (4e-6 if m > 1 else 1.0)
    assert rel(rm, 0.1 * mu) <= 2e-6 and rel(rv, 0.9 + 0.1 * var * m / max(m - 1, 1)) <= 4e-6
    if m > 1:
        assert rel(y, (X - mu.view(col)) * (scale * inv).view(col) + bias.view(col)) <= 4e-6
    record = torch.zeros(_lib.lib().sgb_relu_mask_bytes(m * c), dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    _lib.call("sgb_relu_forward_mask_f32", relu_in.data_ptr(), torch.empty_like(relu_in).data_ptr(), record.data_ptr(),
              m * c, stream)
    mu, inv = mean.double(), invstd.double()
    for masked in (False, True):
        G = torch.where(relu_in > 0, dy, 0.0).double() if masked else dy.double()
        xc = X - mu.view(col)
        db, ds = G.sum((0, 2, 3)), (G * xc).sum((0, 2, 3)) * inv
        want = (scale * inv).view(col) * (G - db.view(col) / m - xc * (ds * inv).view(col) / m)
        outs = [sw.GpuBatchNormReLUBackward(handle, dy, relu_in, x, scale, mean, invstd) if masked
                else sw.GpuBatchNormBackward(handle, dy, x, scale, mean, invstd)]
        if masked:
            dx, a, b = torch.empty_like(dy), torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
            ws = torch.empty(64 * c * 8, dtype=torch.uint8, device="cuda")
            _lib.call("sgb_bn_relu_backward_mask_f32", x.data_ptr(), dy.data_ptr(), record.data_ptr(), scale.data_ptr(),
                      mean.data_ptr(), invstd.data_ptr(), dx.data_ptr(), a.data_ptr(), b.data_ptr(), n, c, h * w,
                      ws.data_ptr(), ws.numel(), stream)
            outs.append((dx, a, b))
        for dx, dscale, dbias in outs:
            bound = 6e-5 * G.abs().sum((0, 2, 3))
            assert bool(((dbias.double() - db).abs() <= bound + 1e-30).all())
            assert bool(((dscale.double() - ds).abs() <= 6e-5 * (G * xc).abs().sum((0, 2, 3)) * inv + 1e-30).all())
            if m > 4:
                assert rel(dx, want) <= 4e-6


def test_a_large_mean_does_not_cost_the_variance_its_digits():
    """Standard deviation 1 around a mean of 1000 (values carry 6e-5 absolute
    rounding): the variance is right to the input's own rounding."""
    from singa_b200 import singa_wrap as sw
    for shape in ((2, 3, 20, 20), (16, 4, 56, 56), (65, 2, 112, 112), (64, 2, 111, 113)):
        x = torch.randn(shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)) + 1000.0
        one, zero = torch.ones(shape[1], device="cuda"), torch.zeros(shape[1], device="cuda")
        _, _, inv = sw.GpuBatchNormForwardTraining(sw.CudnnBatchNormHandle(0.1, x), x, one, zero, zero.clone(),
                                                   one.clone(), 1e-5)
        X = x.double()
        want = (X.var((0, 2, 3), unbiased=False) + 1e-5).rsqrt()
        assert rel(inv, want) <= 1e-6, shape
