"""Batch-norm backward of planes that no 16-byte vector divides, in groups of adjacent
channels: a plane within one vector of the next, groups of two and of four, both sides of
the lines where the groups take over, the most units a thread holds; plain, masked by the
ReLU's input and by its record.

Tolerance: a sum is a tree over chains of at most 2^10 additions, whose independent
rounding errors have a root mean square below sqrt(2^10) * 2^-24 = 2e-6 of the terms'."""
import pytest
import torch

pytestmark = pytest.mark.gpu

#         n, c, h, w
SHAPES = [(11, 20000, 3, 3), (17, 21000, 1, 6), (400, 2600, 1, 2), (350, 2048, 1, 3),          # tiny planes
          (32, 1300, 7, 7), (32, 1276, 7, 7),                                                  # 2e6 elements, both sides
          (9, 3000, 9, 9), (16, 3000, 7, 7), (6, 2200, 13, 13), (50, 1600, 5, 5), (33, 1300, 7, 7), (23, 3500, 9, 9),
          (25, 1024, 9, 9), (33, 1024, 9, 9), (65, 640, 7, 7), (128, 512, 5, 5), (14, 700, 15, 15), (42, 340, 10, 15)]
# both sides of each line in elements of a channel (512, 640, 768, 960, 1024, 1680, 1920, 2048)
# and in all (2e6, 3.5e6, 4e6, 6e6); groups of two: 1024
SHAPES += [(10, 4200, 3, 17), (9, 4000, 3, 19), (128, 3300, 1, 5), (129, 3200, 1, 5), (129, 6300, 1, 5), (256, 5300, 1, 3),
           (257, 5300, 1, 3), (64, 6400, 3, 5), (64, 6200, 3, 5), (65, 6400, 3, 5), (341, 2000, 1, 3), (205, 2000, 1, 5),
           (336, 1200, 1, 5), (561, 1200, 1, 3), (384, 1840, 1, 5), (384, 1800, 1, 5), (641, 1840, 1, 3), (641, 3124, 1, 3),
           (683, 1000, 1, 3), (102, 2000, 1, 10), (103, 2000, 1, 10)]


def rel(got, want):
    return float((got.double() - want).norm() / (want.norm() + 1e-300))


@pytest.mark.parametrize("shape", SHAPES)
def test_against_fp64(shape):
    from singa_b200 import _lib
    n, c, h, w = shape
    m, col = n * h * w, (1, c, 1, 1)
    g = torch.Generator(device="cuda").manual_seed(m + c)
    x, dy, relu_in = [torch.randn(shape, device="cuda", generator=g) for _ in range(3)]
    scale, mean, invstd = [torch.rand(c, device="cuda", generator=g) + 0.5 for _ in range(3)]
    record = torch.zeros(_lib.lib().sgb_relu_mask_bytes(m * c), dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    _lib.call("sgb_relu_forward_mask_f32", relu_in.data_ptr(), torch.empty_like(relu_in).data_ptr(), record.data_ptr(), m * c, stream)
    ws = torch.empty(_lib.lib().sgb_bn_backward_workspace_bytes(n, c, h * w), dtype=torch.uint8, device="cuda")
    results = []
    for masked, mask in ((False, None), (True, relu_in), (True, record)):
        dx, ds, db = torch.empty_like(x), torch.empty_like(scale), torch.empty_like(scale)
        name = "sgb_bn_backward_f32" if mask is None else "sgb_bn_relu_backward%s_f32" % ("_mask" if mask is record else "")
        tensors = [x, dy] + ([mask] if masked else []) + [scale, mean, invstd, dx, ds, db]
        _lib.call(name, *[t.data_ptr() for t in tensors], n, c, h * w, ws.data_ptr(), ws.numel(), stream)
        G = torch.where(relu_in > 0, dy, 0.0).double() if masked else dy.double()
        mu, inv = mean.double(), invstd.double()
        xc = x.double() - mu.view(col)
        sb, ss = G.sum((0, 2, 3)), (G * xc).sum((0, 2, 3)) * inv
        want = (scale.double() * inv).view(col) * (G - sb.view(col) / m - xc * (ss * inv).view(col) / m)
        assert rel(dx, want) <= 2e-6
        terms = G.square().sum((0, 2, 3)).sqrt()
        assert float(((db.double() - sb) / (terms * m ** 0.5)).abs().max()) <= 2e-6
        assert float(((ds.double() - ss) / ((G * xc).abs().sum((0, 2, 3)) * inv)).abs().max()) <= 2e-6
        results.append((dx, ds, db))
    assert all(torch.equal(a, b) for a, b in zip(*results[1:]))
