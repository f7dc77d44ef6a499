"""The exchange of a whole list of gradients in half precision on one rank: a
list that exists is rounded in one go, a generator bucket by bucket, and with
profiling on per bucket as well.  The same roundings either way: bitwise equal."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,threshold", [([5], 10), ([11], 10), ([10], 10), ([3, 4, 100001, 7, 64, 1], 50),
                                             ([1, 2, 3] * 200, 40), ([4097] * 3, 1 << 20)])
@pytest.mark.parametrize("offset", [0, 1])
def test_list_generator_and_profiled_agree(sizes, threshold, offset):
    from singa_b200.communicator import Communicator, NcclIdHolder
    comm = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=100001)
    try:
        gen = torch.Generator(device="cuda").manual_seed(len(sizes))
        grads = [torch.randn(n + offset, device="cuda", generator=gen)[offset:] * 1e-3 for n in sizes]
        want = [g.half().float() for g in grads]

        def run(form, kind=list):
            ts = [torch.empty(g.numel() + offset, device="cuda")[offset:].copy_(g) for g in grads]
            triples = kind((str(i), None, t) for i, t in enumerate(ts))
            names, params, out = comm.syncDense(form(triples), threshold, True)
            comm.wait()
            assert names == [str(i) for i in range(len(ts))] and params == [None] * len(ts)
            assert all(a is b for a, b in zip(out, ts))
            for t, w in zip(ts, want):
                assert torch.equal(t, w)

        run(iter)
        run(lambda x: x)
        run(iter, tuple)
        run(lambda x: (t for t in x))
        comm.profile_begin()
        run(iter)
        assert len(comm.profile_end()) >= 1
    finally:
        torch.cuda.synchronize()
        comm.close()


def test_a_bucket_above_the_capacity_is_still_refused():
    from singa_b200 import _lib
    from singa_b200.communicator import Communicator, NcclIdHolder
    comm = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=100)
    try:
        with pytest.raises(_lib.SgbError):
            comm.syncDense([("a", None, torch.ones(101, device="cuda"))], 10, True)
        with pytest.raises(AssertionError):
            comm.syncDense([("a", None, torch.ones(8, device="cuda").half())], 10, True)
    finally:
        torch.cuda.synchronize()
        comm.close()


@pytest.mark.parametrize("sizes,threshold", [([5], 10), ([11, 12], 10), ([3, 4, 100001, 7, 64, 1, 512], 50),
                                             ([1, 2, 3] * 200, 40), ([513, 511, 512, 2049] * 40, 3000),
                                             ([2097151, 1, 2, 2097152, 5, 1 << 21, 77, 1 << 21, 4096] * 4, 1 << 21)])
@pytest.mark.parametrize("spars", [1e-3, 0.0, 1.0])
def test_buckets_selected_together_equal_bucket_by_bucket(sizes, threshold, spars):
    """More than 32 buckets, 2^25 elements and 256 tensors cut the list; ends of
    buckets inside a tile; nothing and everything selected.  Bitwise equal."""
    from singa_b200.communicator import Communicator, NcclIdHolder
    from singa_b200.opt import SGD, DistOpt
    comm = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=1 << 22)
    try:
        gen = torch.Generator(device="cuda").manual_seed(len(sizes))
        steps = [[torch.randn(n, device="cuda", generator=gen) * 1e-3 for n in sizes] for _ in range(2)]
        base = [torch.randn(n, device="cuda", generator=gen) for n in sizes]
        results = []
        for form in (list, lambda x: (t for t in x)):
            opt = DistOpt(SGD(lr=0.1), communicator=comm)
            params = [t.clone() for t in base]
            seen = []
            for grads in steps:
                gs = [g.clone() for g in grads]
                opt.backward_and_sparse_update(form([(str(i), p, g) for i, (p, g) in enumerate(zip(params, gs))]),
                                               threshold=threshold, spars=spars)
                seen += gs
            results.append(params + seen + list(opt.gradAccumulation))
        for a, b in zip(*results):
            assert torch.equal(a, b)
    finally:
        torch.cuda.synchronize()
        comm.close()
