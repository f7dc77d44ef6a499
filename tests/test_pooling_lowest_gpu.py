"""Max pooling of cells at the ends of the number line: windows that hold nothing above
the lowest finite value, infinities of both signs (whose warps take the other
comparisons), zeros of both signs.  Bitwise against the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
LOWEST = -float(np.finfo(np.float32).max)


@pytest.mark.parametrize("k, s, p", [(3, 2, 1), (3, 1, 1), (2, 2, 0)])
@pytest.mark.parametrize("w", [4, 29, 128, 131])
@pytest.mark.parametrize("cells", [[-np.inf, LOWEST], [LOWEST, -1.0, 1.0], [-np.inf, np.inf, 0.0, -0.0, 2.0], [0.0, -0.0]])
def test_windows_of_extreme_cells(oracle, k, s, p, w, cells):
    from singa_b200 import singa_wrap as sw
    rng = np.random.default_rng(w)
    x = rng.choice(np.array(cells, np.float32), size=(2, 3, 17, w))
    x[:, :, 9:] = np.where(rng.random(x[:, :, 9:].shape) < 0.5, x[:, :, 9:], rng.standard_normal(x[:, :, 9:].shape)).astype(np.float32)
    dev = torch.from_numpy(x).cuda()
    handle = sw.CudnnPoolingHandle(dev, (k, k), (s, s), (p, p), True)
    dy = rng.standard_normal((2, 3, handle.pooled_height, handle.pooled_width)).astype(np.float32)
    y, arg = sw.GpuPoolingForwardArgmax(handle, dev)
    bits = lambda a: np.ascontiguousarray(a).view(np.uint32)   # noqa: E731
    assert np.array_equal(bits(y.cpu().numpy()), bits(oracle.maxpool_forward(x, (k, k), (s, s), (p, p))))
    assert np.array_equal(bits(sw.GpuPoolingForward(handle, dev).cpu().numpy()), bits(y.cpu().numpy()))
    want = oracle.maxpool_backward(dy, x, (k, k), (s, s), (p, p))
    ddy = torch.from_numpy(dy).cuda()
    for got in (sw.GpuPoolingBackward(handle, ddy, dev, y), sw.GpuPoolingBackwardArgmax(handle, ddy, arg)):
        assert np.array_equal(bits(got.cpu().numpy()), bits(want))
