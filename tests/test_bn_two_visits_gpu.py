"""Batch norm that visits its data twice (large calls): items that end inside a
plane, last items that are short, ragged planes with masked ends, channels of many
items; a workspace full of anything, reused and replayed; one too small for it.

Tolerance: as in test_batchnorm_plans_gpu.py (root mean square error of sums over
chains of at most 2^10 additions, and the normalisation's few roundings)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

#         n, c, h, w
SHAPES = [(5, 25, 200, 160),      # 40000 units a channel: items of 896, the last of them short
          (1, 1, 2000, 2004),     # one channel, 1002000 units: more entries than a batch of lanes
          (257, 999, 4, 4),       # planes of four units
          (2, 1000, 2, 1002),     # 1002 units a channel: two items
          (33, 2, 251, 243),      # ragged, few channels
          (9, 240, 53, 53),       # ragged, 53 * 53 % 4 == 1
          (10, 241, 50, 51)]      # ragged, planes of two leads


def rel(got, want):
    return float((got.double() - want).norm() / (want.norm() + 1e-300))


def reference(x, dy, keep, scale, mean, invstd):
    col, m = (1, -1, 1, 1), x.numel() // x.shape[1]
    g = dy.double() if keep is None else torch.where(keep, dy, 0.0).double()
    xc, inv = x.double() - mean.double().view(col), invstd.double()
    db, ds = g.sum((0, 2, 3)), (g * xc).sum((0, 2, 3)) * inv
    return (scale.double() * inv).view(col) * (g - db.view(col) / m - xc * (ds * inv).view(col) / m), ds, db


def make(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = lambda std, mean=0.0: torch.randn(shape, device="cuda", generator=g) * std + mean   # noqa: E731
    c = shape[1]
    return (t(1.5, 3.0), t(1e-2), t(1.0), torch.rand(c, device="cuda", generator=g) + 0.5,
            torch.randn(c, device="cuda", generator=g) + 3.0, torch.rand(c, device="cuda", generator=g) + 0.5)


class Backward(object):
    """One set of buffers and the three calls."""

    def __init__(self, shape, seed, ws_bytes=None):
        from singa_b200 import _lib
        self.call, lib = _lib.call, _lib.lib()
        n, c, h, w = shape
        self.x, self.dy, self.r, self.scale, self.mean, self.invstd = make(shape, seed)
        self.record = torch.zeros(lib.sgb_relu_mask_bytes(self.x.numel()), dtype=torch.uint8, device="cuda")
        self.call("sgb_relu_forward_mask_f32", self.r.data_ptr(), torch.empty_like(self.r).data_ptr(),
                  self.record.data_ptr(), self.x.numel(), torch.cuda.current_stream().cuda_stream)
        self.dx, self.ds, self.db = torch.empty_like(self.x), torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
        need = lib.sgb_bn_backward_workspace_bytes(n, c, h * w)
        self.ws = torch.randint(0, 256, (ws_bytes or need,), dtype=torch.uint8, device="cuda")
        self.tail = (n, c, h * w, self.ws.data_ptr(), self.ws.numel())

    def run(self, mask, dx=None):
        p = [t.data_ptr() for t in (self.x, self.dy)]
        p += [[], [self.r.data_ptr()], [self.record.data_ptr()]][mask]
        p += [t.data_ptr() for t in (self.scale, self.mean, self.invstd, self.dx if dx is None else dx, self.ds, self.db)]
        self.call(("sgb_bn_backward_f32", "sgb_bn_relu_backward_f32", "sgb_bn_relu_backward_mask_f32")[mask], *p, *self.tail,
                  torch.cuda.current_stream().cuda_stream)
        return [t.clone() for t in (self.dx if dx is None else dx, self.ds, self.db)]

    def want(self, mask):
        return reference(self.x, self.dy, self.r > 0 if mask else None, self.scale, self.mean, self.invstd)


def no_faults():
    from singa_b200 import _lib
    flags = ctypes.c_uint(1)
    _lib.call("sgb_bn_backward_faults", ctypes.byref(flags))
    return flags.value == 0


def close(got, want, b):
    return rel(got[0], want[0]) <= 4e-6 and all(
        bool(((g.double() - w).abs() <= 6e-5 * scale + 1e-30).all())
        for g, w, scale in zip(got[1:], want[1:], ((b.dy * (b.x - b.mean.view(1, -1, 1, 1))).abs().sum((0, 2, 3)).double() *
                                                   b.invstd, b.dy.abs().sum((0, 2, 3)).double())))


@pytest.mark.parametrize("shape", SHAPES)
def test_backward_against_fp64(shape):
    b = Backward(shape, 1)
    outs = [b.run(mask) for mask in (0, 1, 2)]
    for mask in (0, 1, 2):
        assert close(outs[mask], b.want(mask), b), (shape, mask)
        assert all(torch.equal(p, q) for p, q in zip(outs[mask], b.run(mask))), "not repeatable"
    assert all(torch.equal(p, q) for p, q in zip(outs[1], outs[2])), "float mask != bit record"
    b.dy = torch.where(b.r > 0, b.dy, 0.0)
    assert all(torch.equal(p, q) for p, q in zip(outs[1], b.run(0))), "fused call != its parts"
    want = [t.clone() for t in outs[1]]
    assert all(torch.equal(p, q) for p, q in zip(b.run(0, dx=b.dy), want)), "in place"
    assert no_faults()


@pytest.mark.parametrize("shape", [SHAPES[0], SHAPES[5]])
def test_replays_and_a_shared_workspace(shape):
    a, b = Backward(shape, 2), Backward((3,) + shape[1:], 3)
    b.ws, b.tail = a.ws, b.tail[:3] + a.tail[3:]
    want = [[t.clone() for t in m.run(mask)] for m in (a, b) for mask in (0, 1)]
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        with torch.cuda.graph(g, stream=s):
            got = [m.run(mask) for m in (a, b) for mask in (0, 1)]
    for replay in range(4):
        if replay == 2:                                # other data, the same launches
            for m in (a, b):
                m.dy.mul_(2.0)
                m.scale.mul_(0.5)
            want = [[dx, 2 * ds, 2 * db] for dx, ds, db in want]       # exact: powers of two
        if replay % 2:
            a.ws.random_(0, 256)
        g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(p, q) for x, y in zip(got, want) for p, q in zip(x, y)), replay
    assert no_faults()


def test_a_workspace_of_partial_sums_only():
    shape = SHAPES[0]
    b = Backward(shape, 4, ws_bytes=64 * shape[1] * 8)
    for mask in (0, 1, 2):
        assert close(b.run(mask), b.want(mask), b), mask


@pytest.mark.parametrize("shape", SHAPES)
def test_forward_against_fp64(shape):
    from singa_b200 import singa_wrap as sw
    x, _, _, scale, bias, _ = make(shape, 5)
    c = shape[1]
    handle = sw.CudnnBatchNormHandle(0.1, x)
    runs = []
    for _ in range(2):
        rm, rv = torch.zeros(c, device="cuda"), torch.ones(c, device="cuda")
        runs.append(list(sw.GpuBatchNormForwardTraining(handle, x, scale, bias, rm, rv, 1e-5)) + [rm, rv])
    assert all(torch.equal(p, q) for p, q in zip(*runs)), "not repeatable"
    y, mean, invstd, rm, rv = runs[0]
    col, m, X = (1, -1, 1, 1), x.numel() // c, x.double()
    mu = X.mean((0, 2, 3))
    var = (X - mu.view(col)).square().mean((0, 2, 3))
    inv = (var + 1e-5).rsqrt()
    assert rel(mean, mu) <= 2e-6 and rel(invstd, inv) <= 4e-6
    assert rel(rm, 0.1 * mu) <= 2e-6 and rel(rv, 0.9 + 0.1 * var * m / (m - 1)) <= 4e-6
    assert rel(y, (X - mu.view(col)) * (scale.double() * inv).view(col) + bias.double().view(col)) <= 4e-6
    assert no_faults()
