"""Lists of more buckets, pieces or elements than one top-K launch takes, and of tensors
that begin inside a vector: the same bits as a call per bucket."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def at(t, offset):
    """A copy that starts `offset` elements behind a boundary."""
    room = torch.empty(t.numel() + offset + 4, device="cuda", dtype=t.dtype)
    return room[offset:offset + t.numel()].copy_(t)


# more than 32 buckets; more than 256 pieces; tensors that begin inside a vector; 2^25 elements and more
LISTS = [([40000] * 40, 20000, 0), ([30001] * 75, 25000, 0), ([4097] * 300, 60000, 1), ([17, 299999, 3, 250001, 1, 600000], 200000, 0),
         ([1 << 21] * 17 + [5], 1 << 20, 0)]


# whole tiles and their ends, on and off a vector's boundary; one tensor by threshold, of any size that one selection takes
ONE = [(4096, 0), (4097, 0), (8191, 1), (4000001, 0), (5000003, 2), (1 << 25, 0)]


@pytest.mark.parametrize("size, offset", ONE)
@pytest.mark.parametrize("topk, spars", [(False, 2.0), (True, 0.03)])
def test_one_tensor(size, offset, topk, spars):
    compare([size], 1 << 22, offset, "magnitude", topk, spars, 1 << 25)


@pytest.mark.parametrize("sizes, threshold, offset", LISTS)
@pytest.mark.parametrize("mode", ["magnitude", "compat"])
def test_topk_of_long_lists(sizes, threshold, offset, mode):
    compare(sizes, threshold, offset, mode, True, 0.02, 1 << 22)


def compare(sizes, threshold, offset, mode, topk, spars, room):
    """A list, which goes through the joint launches, against a generator, a call per bucket."""
    from singa_b200 import _lib
    from singa_b200.communicator import Communicator, NcclIdHolder
    from singa_b200.opt import SGD, DistOpt
    comm = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=room)
    comm.set_topk_mode(mode)
    sides = []
    for as_list in (True, False):
        g = torch.Generator(device="cuda").manual_seed(3)
        opt = DistOpt(SGD(lr=0.05, momentum=0.9), communicator=comm)
        params = [at(torch.zeros(n, device="cuda"), offset) for n in sizes]
        for _ in range(2):
            grads = [at(torch.randn(n, device="cuda", generator=g), offset) for n in sizes]
            triples = [("p%d" % i, p, d) for i, (p, d) in enumerate(zip(params, grads))]
            assert comm.takesSparseUpdate(triples, threshold, topk)
            opt.backward_and_sparse_update(triples if as_list else (t for t in triples), threshold=threshold, spars=spars,
                                           topK=topk)
        sides.append(grads + params + [opt.opt.moments["p%d" % i] for i in range(len(sizes))] + opt.gradAccumulation)
    torch.cuda.synchronize()
    assert all(torch.equal(a.view(torch.int32), b.view(torch.int32)) for a, b in zip(*sides))
    faults = ctypes.c_uint(1)
    _lib.call("sgb_sparse_faults", ctypes.byref(faults))
    assert faults.value == 0
    comm.close()
