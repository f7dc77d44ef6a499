"""Kernels that do the work of two neighbouring calls: the same bits as the two
calls, for sizes around the vector width, the slices and the clusters of the
sums, the planes of the joined batch norm, and tensors off a 16-byte boundary."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def call(name, *args):
    from singa_b200 import _lib
    _lib.call(name, *[a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args],
              torch.cuda.current_stream().cuda_stream)


def tensors(n, count, offset):
    gen = torch.Generator(device="cuda").manual_seed(n)
    return [torch.randn(n + offset, device="cuda", generator=gen)[offset:] for _ in range(count)]


@pytest.mark.parametrize("shape", [(1, 1), (3, 4), (7, 33), (64, 500), (65, 4096), (255, 4100), (1000, 12), (9000, 40)])
@pytest.mark.parametrize("offset", [0, 1])
def test_relu_and_column_sums(shape, offset):
    r, c = shape
    dy, x, d1, d2 = tensors(r * c, 4, offset)
    ws = torch.empty(8 << 20, dtype=torch.uint8, device="cuda")
    v1, v2 = torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
    call("sgb_relu_backward_f32", dy, x, d1, r * c)
    call("sgb_sum_rows_f32", d1, v1, r, c, ws, ws.numel())
    call("sgb_relu_backward_sum_rows_f32", dy, x, d2, v2, r, c, ws, ws.numel())
    assert torch.equal(d1, torch.where(x > 0, dy, 0.0)) and torch.equal(d1, d2) and torch.equal(v1, v2)


@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (3, 5, 3, 3), (4, 8, 8, 8), (33, 7, 9, 9), (64, 32, 24, 24), (70, 3, 64, 64)])
@pytest.mark.parametrize("offset", [0, 1])
def test_relu_and_channel_sums(shape, offset):
    n, c, h, w = shape
    m = n * c * h * w
    dy, x, d1, d2 = tensors(m, 4, offset)
    ws = torch.empty(8 << 20, dtype=torch.uint8, device="cuda")
    v1, v2 = torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
    call("sgb_relu_backward_f32", dy, x, d1, m)
    call("sgb_conv_bias_backward_f32", d1, v1, n, c, h * w, ws, ws.numel())
    call("sgb_relu_backward_conv_bias_f32", dy, x, d2, v2, n, c, h * w, ws, ws.numel())
    assert torch.equal(d1, torch.where(x > 0, dy, 0.0)) and torch.equal(d1, d2) and torch.equal(v1, v2)


@pytest.mark.parametrize("shape", [(2, 5, 1, 1), (1, 6, 1, 3), (3, 2048, 5, 5), (3, 6, 15, 17), (24, 9, 8, 8), (3, 7, 40, 40),
                                   (20, 2048, 7, 7)])
@pytest.mark.parametrize("offset", [0, 1])
def test_join_and_batch_norm(shape, offset):
    n, c, h, w = shape
    m = n * c * h * w
    x, a, b, r, j1, j2, d1, d2 = tensors(m, 8, offset)
    ws = torch.empty(8 << 20, dtype=torch.uint8, device="cuda")
    scale, mean, inv, s1, b1, s2, b2 = [t.abs() + 0.5 for t in tensors(c, 7, 0)]
    call("sgb_add_relu_backward_f32", a, b, r, j1, m)
    call("sgb_bn_backward_f32", x, j1, scale, mean, inv, d1, s1, b1, n, c, h * w, ws, ws.numel())
    call("sgb_bn_add_relu_backward_f32", x, a, b, r, scale, mean, inv, j2, d2, s2, b2, n, c, h * w, ws, ws.numel())
    for got, want in ((j2, j1), (d2, d1), (s2, s1), (b2, b1)):
        assert torch.equal(got, want)


@pytest.mark.parametrize("shape", [(1, 1, 2, 2), (3, 5, 3, 3), (2, 4, 7, 5), (4, 8, 8, 8), (5, 3, 2, 6), (64, 32, 24, 24), (9, 7, 9, 4),
                                   (200, 6, 33, 31), (3, 2, 5, 64)])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("window", [2, 3])
def test_pooling_relu_and_channel_sums(shape, offset, window):
    n, c, h, w = shape
    if min(h, w) < window:
        pytest.skip("no window")
    m, geom = n * c * h * w, (n, c, h, w, window, window, 0, 0, 2, 2)
    px, rx, p1, p2, d1, d2 = tensors(m, 6, offset)
    px.mul_(2).round_()                                # ties
    px[::97] = float("nan")
    px[1::89] = -float("inf")
    dy = tensors(n * c * ((h - window) // 2 + 1) * ((w - window) // 2 + 1), 1, offset)[0]
    ws = torch.empty(8 << 20, dtype=torch.uint8, device="cuda")
    v1, v2 = torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
    call("sgb_maxpool_backward_f32", px, px, dy, p1, *geom)
    call("sgb_relu_backward_conv_bias_f32", p1, rx, d1, v1, n, c, h * w, ws, ws.numel())
    call("sgb_maxpool_relu_backward_conv_bias_f32", px, px, dy, p2, *geom, rx, d2, v2, ws, ws.numel())
    for got, want in ((p2, p1), (d2, d1), (v2, v1)):
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("shape", [(1, 1), (4, 10), (64, 10), (256, 10), (33, 7), (1024, 16), (1025, 10), (5, 512), (31, 500), (9, 513),
                                   (40, 129), (300, 54), (32, 1000), (5000, 3)])
@pytest.mark.parametrize("offset", [0, 1])
def test_loss_head(shape, offset):
    r, c = shape
    x, p1, p2, g1, g2 = tensors(r * c, 5, offset)
    t = torch.randint(0, c, (r,), device="cuda", dtype=torch.int32)
    if r > 4:
        t[3] = c                                       # out of range: that sample's loss is NaN
    l1, l2, v1, v2 = (torch.zeros(k, device="cuda") for k in (r, r, c, c))
    s1, s2 = torch.zeros(1, device="cuda"), torch.zeros(1, device="cuda")
    ws = torch.empty(8 << 20, dtype=torch.uint8, device="cuda")
    call("sgb_softmax_cross_entropy_fused_f32", x, t, r, c, 1.0 / r, p1, l1, g1)
    call("sgb_sum_all_f32", l1, s1, r, ws, ws.numel())
    call("sgb_sum_rows_f32", g1, v1, r, c, ws, ws.numel())
    call("sgb_loss_head_f32", x, t, r, c, 1.0 / r, p2, l2, g2, s2, v2, ws, ws.numel())
    for got, want in ((p2, p1), (l2, l1), (g2, g1), (s2, s1), (v2, v1)):
        assert torch.equal(got.view(torch.int32), want.view(torch.int32))
