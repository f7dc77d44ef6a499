"""Batch norm in two visits counts the readers of a channel from whatever its workspace
holds: the same bits when the counters are 0, wrap around, or are another call's."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 25, 200, 160), (1, 1, 2000, 2004), (9, 240, 53, 53)])
@pytest.mark.parametrize("fill", [0x00, 0xff, 0x7f])
def test_counters_of_any_value(shape, fill):
    from singa_b200 import _lib
    n, c, h, w = shape
    g = torch.Generator(device="cuda").manual_seed(c)
    x, dy = (torch.randn(n * c * h * w, device="cuda", generator=g) for _ in range(2))
    scale, mean, inv = (torch.rand(c, device="cuda", generator=g) + 0.5 for _ in range(3))
    out, stats = torch.empty_like(x), [torch.zeros(c, device="cuda") for _ in range(4)]
    ws = torch.full((_lib.lib().sgb_bn_backward_workspace_bytes(n, c, h * w),), fill, dtype=torch.uint8, device="cuda")

    def run(forward):
        p = lambda *t: [v.data_ptr() for v in t]   # noqa: E731
        tail = (n, c, h * w, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
        if forward:
            _lib.call("sgb_bn_forward_training_f32", *p(x, scale, mean, *stats[:2]), 0.1, 1e-5, *p(out, *stats[2:]), *tail)
        else:
            _lib.call("sgb_bn_backward_f32", *p(x, dy, scale, mean, inv, out, *stats[2:]), *tail)
        return [out.clone()] + [s.clone() for s in stats[2:]]
    for forward in (False, True):
        runs = []
        for k in range(3):
            if k == 2:
                ws.random_(0, 256, generator=g)
            runs.append(run(forward))
        assert all(torch.equal(a, b) for r in runs[1:] for a, b in zip(r, runs[0])), forward
