"""Tensors of any length back to back, so that few of them start on a 16-byte boundary:
update, rounding, pack and unpack give the same bits as on aligned copies."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def table(ts):
    n = len(ts)
    return ((ctypes.c_void_p * n)(*[t.data_ptr() for t in ts]), (ctypes.c_size_t * n)(*[t.numel() for t in ts]), n)


def at(t, offset):
    """A copy that starts `offset` elements behind a boundary."""
    room = torch.empty(t.numel() + offset + 4, device="cuda", dtype=t.dtype)
    return room[offset:offset + t.numel()].copy_(t)


def call(name, *args):
    from singa_b200 import _lib
    _lib.call(name, *args, torch.cuda.current_stream().cuda_stream)


SIZES = [1, 3, 4, 5, 7, 1023, 1024, 1025, 4099, 2051]


@pytest.mark.parametrize("offsets", [(0, 0, 0), (0, 2, 0), (1, 1, 1), (0, 3, 2), (2, 0, 1), (3, 1, 0)])
@pytest.mark.parametrize("momentum", [0.0, 0.9])
def test_update(offsets, momentum):
    from singa_b200.communicator import Communicator, NcclIdHolder
    g = torch.Generator(device="cuda").manual_seed(1)
    base = [[torch.randn(n, device="cuda", generator=g) for n in SIZES] for _ in range(3)]
    comm = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=1 << 16)
    outs = []
    for offs in ((0, 0, 0), offsets):
        for half in (False, True):
            p, d, m = ([at(t, o) for t in ts] for ts, o in zip(base, offs))
            (pp, sizes, n), (gp, _, _), (mp, _, _) = table(p), table(d), table(m)
            if half:
                call("sgb_comm_update_half", comm._h, pp, gp, mp, sizes, n, max(SIZES), 0.1, momentum, 0.0, 1e-3, 0, 0.5)
            else:
                call("sgb_sgd_update_multi_f32", pp, gp, mp, sizes, n, 0.1, momentum, 0.0, 1e-3, 0, 0.5)
            outs.append(torch.cat(p + d + m))
    torch.cuda.synchronize()
    comm.close()
    assert torch.equal(outs[0], outs[2]) and torch.equal(outs[1], outs[3])
    assert not torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("start", [0, 1, 2])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_pack_and_unpack(start, offset):
    g = torch.Generator(device="cuda").manual_seed(2)
    base = [torch.randn(n, device="cuda", generator=g) for n in SIZES]
    ts = [at(t, offset) for t in base]
    ptrs, sizes, n = table(ts)
    want = torch.cat(base)
    flat = torch.zeros(start + want.numel() + 8, device="cuda")
    call("sgb_pack_f32", ptrs, sizes, n, flat.data_ptr(), start)
    assert torch.equal(flat[start:start + want.numel()], want)
    for t in ts:
        t.zero_()
    call("sgb_unpack_f32", flat.data_ptr(), start, ptrs, sizes, n, 0.5)
    assert torch.equal(torch.cat(ts), want * 0.5)
    assert float(flat[:start].abs().sum()) == 0 and float(flat[start + want.numel():].abs().sum()) == 0
