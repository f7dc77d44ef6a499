"""The register-strip pooling kernels at the edges of their layout: rows that end
inside a lane's four columns, several planes side by side in a warp, planes of
exactly one warp (128 columns) and cut into segments, one-row planes, bands that
end at the last row, rows off a 16-byte boundary, NaNs.  Bitwise against the
oracle (selection, and raster-order sums of the same products)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
WIDTHS = [1, 2, 3, 4, 5, 7, 31, 64, 113, 124, 127, 128, 129, 131, 242]


@pytest.mark.parametrize("k, s, p", [(3, 2, 1), (3, 1, 1), (2, 2, 0)])
@pytest.mark.parametrize("h", [2, 5, 30])
def test_strips_match_the_oracle(oracle, k, s, p, h):
    from singa_b200 import singa_wrap as sw
    rng = np.random.default_rng(100 * k + 10 * s + h)
    for w in WIDTHS:
        if w + 2 * p < k:
            continue
        shape = (2, 5, h, w)
        for kind in ("plain", "ties", "shifted"):
            x = rng.standard_normal(shape).astype(np.float32)
            if kind == "ties":
                x = np.round(x)
            def dev(a, shift=int(kind == "shifted")):
                t = torch.empty(a.size + shift, device="cuda")[shift:].view(a.shape)
                return t.copy_(torch.from_numpy(a))
            handle = sw.CudnnPoolingHandle(dev(x), (k, k), (s, s), (p, p), True)
            dy = rng.standard_normal((2, 5, handle.pooled_height, handle.pooled_width)).astype(np.float32)
            dx_, ddy = dev(x), dev(dy)
            y, arg = sw.GpuPoolingForwardArgmax(handle, dx_)
            want_y, want = oracle.maxpool_forward(x, (k, k), (s, s), (p, p)), \
                oracle.maxpool_backward(dy, x, (k, k), (s, s), (p, p))
            where = (k, s, p, shape, kind)
            assert np.array_equal(y.cpu().numpy(), want_y), where
            assert np.array_equal(sw.GpuPoolingForward(handle, dx_).cpu().numpy(), want_y), where
            for got in (sw.GpuPoolingBackward(handle, ddy, dx_, y), sw.GpuPoolingBackwardArgmax(handle, ddy, arg)):
                assert np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32)), where
            if s == 2:
                avg = sw.CudnnPoolingHandle(dx_, (k, k), (s, s), (p, p), False)
                got = sw.GpuPoolingBackward(avg, ddy, dx_, y).cpu().numpy()
                want = oracle.avgpool_backward(dy, shape, (k, k), (s, s), (p, p))
                assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), where
                # nine fp32 additions and a division: 9 * 2^-24 relative to the sum of magnitudes
                got = sw.GpuPoolingForward(avg, dx_).cpu().numpy()
                want = oracle.avgpool_forward(x, (k, k), (s, s), (p, p))
                mag = oracle.avgpool_forward(np.abs(x), (k, k), (s, s), (p, p))
                assert np.all(np.abs(got - want) <= 10 * 2.0 ** -24 * mag), where


@pytest.mark.parametrize("k, s, p", [(3, 2, 1), (3, 1, 1), (2, 2, 0)])
def test_a_nan_wins_its_windows_and_sticks(k, s, p):
    from singa_b200 import singa_wrap as sw
    x = torch.randn(1, 3, 12, 20, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    x[0, :, 4:6, 7:9] = float("nan")
    x[0, :, 8, 3] = float("inf")
    x[0, :, 9, 3] = float("-inf")
    handle = sw.CudnnPoolingHandle(x, (k, k), (s, s), (p, p), True)
    y, arg = sw.GpuPoolingForwardArgmax(handle, x)
    want = torch.nn.functional.max_pool2d(x, k, s, p)          # propagates NaN
    assert torch.equal(y.isnan(), want.isnan())
    assert torch.equal(torch.nan_to_num(y, nan=3.0), torch.nan_to_num(want, nan=3.0))
    dy = torch.ones_like(y)
    dx = sw.GpuPoolingBackward(handle, dy, x, y)
    assert torch.equal(dx, sw.GpuPoolingBackwardArgmax(handle, dy, arg))
    assert float(dx.sum()) == dy.numel()                       # every window credits exactly one cell
