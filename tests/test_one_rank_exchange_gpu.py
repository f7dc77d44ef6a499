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
