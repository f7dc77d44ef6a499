"""Joint top-K passes over lists with buckets that nothing is selected from (tensors without
elements, a share of 0): the same bits as a call per bucket, on a communicator whose buffers
are as small as these lists make them, and between lists that select from all."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def run(lists, as_list):
    from singa_b200.communicator import Communicator, NcclIdHolder
    from singa_b200.opt import SGD, DistOpt
    comm = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=1 << 16)
    comm.set_topk_mode("magnitude")
    out = []
    g = torch.Generator(device="cuda").manual_seed(5)
    for sizes, threshold, spars in lists:
        opt = DistOpt(SGD(lr=0.05, momentum=0.9), communicator=comm)
        params = [torch.randn(n, device="cuda", generator=g) for n in sizes]
        for _ in range(2):
            grads = [torch.randn(n, device="cuda", generator=g) for n in sizes]
            triples = [("p%d" % i, p, d) for i, (p, d) in enumerate(zip(params, grads))]
            opt.backward_and_sparse_update(triples if as_list else (t for t in triples), threshold=threshold, spars=spars,
                                           topK=True)
            out += grads
        out += params + opt.gradAccumulation
    torch.cuda.synchronize()
    comm.close()
    return out


@pytest.mark.parametrize("lists", [
    [([4000] * 16, 3000, 0.0)], [([12000] * 32, 3000, 0.0)], [([1000, 1000], 900, 0.0)],
    [([100, 1000, 0], 50, 0.05)], [([0, 100, 1000, 0], 0, 0.05)],
    [([12000] * 32, 3000, 0.0), ([12000] * 32, 3000, 0.02), ([100, 1000, 0], 50, 0.05), ([12000] * 32, 3000, 0.02),
     ([5], 9, 0.0), ([1000, 1000], 900, -1.0), ([12000] * 32, 3000, 0.02)]])
def test_as_a_call_per_bucket(lists):
    assert all(torch.equal(a.view(torch.int32), b.view(torch.int32)) for a, b in zip(run(lists, True), run(lists, False)))
