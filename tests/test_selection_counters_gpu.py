"""One-rank exchanges of all kinds, one behind the other on one communicator: a selection
finds its counters as it needs them whatever ran before it (lists of few and many
buckets, one tensor, by size and by threshold, calls per bucket, a replayed graph)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

KINDS = {"many": ([3000] * 40, 10000, True), "few": ([70000, 12, 4097, 30000], 20000, True), "one": ([300001], 1 << 20, True),
         "threshold": ([3000] * 6, 5000, False), "one threshold": ([3000001], 1 << 20, False), "wide": ([2100000, 1 << 19, 5], 1 << 18, True)}


def run(order, in_lists):
    from singa_b200.communicator import Communicator, NcclIdHolder
    from singa_b200.opt import SGD, DistOpt
    comm = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=1 << 22)
    comm.set_topk_mode("magnitude")
    out, opts = [], {}
    g = torch.Generator(device="cuda").manual_seed(9)
    for kind, as_list in order:
        sizes, threshold, topk = KINDS[kind]
        if kind not in opts:
            opts[kind] = DistOpt(SGD(lr=0.05, momentum=0.9), communicator=comm), [torch.zeros(n, device="cuda") for n in sizes]
        opt, params = opts[kind]
        grads = [torch.randn(n, device="cuda", generator=g) for n in sizes]
        triples = [("p%d" % i, p, d) for i, (p, d) in enumerate(zip(params, grads))]
        opt.backward_and_sparse_update(triples if as_list and in_lists else (t for t in triples), threshold=threshold,
                                       spars=0.03 if topk else 2.0, topK=topk)
        out += grads
    out += [p for opt, params in opts.values() for p in params] + [r for opt, _ in opts.values() for r in opt.gradAccumulation]
    torch.cuda.synchronize()
    comm.close()
    return out


@pytest.mark.parametrize("seed", range(4))
def test_any_order(seed):
    g = torch.Generator().manual_seed(seed)
    kinds = sorted(KINDS)
    order = [(kinds[int(torch.randint(len(kinds), (1,), generator=g))], bool(torch.randint(4, (1,), generator=g))) for _ in range(24)]
    assert all(torch.equal(a.view(torch.int32), b.view(torch.int32)) for a, b in zip(run(order, True), run(order, False)))


def test_replays_between_calls():
    from singa_b200.communicator import Communicator, NcclIdHolder
    from singa_b200.opt import SGD, DistOpt
    comm = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=1 << 22)
    comm.set_topk_mode("magnitude")

    def make(kind):
        sizes, threshold, topk = KINDS[kind]
        opt = DistOpt(SGD(lr=0.05, momentum=0.9), communicator=comm)
        g = torch.Generator(device="cuda").manual_seed(4)
        params, grads = [[torch.randn(n, device="cuda", generator=g) for n in sizes] for _ in range(2)]
        pristine = [d.clone() for d in grads]

        def step():
            for d, v in zip(grads, pristine):
                d.copy_(v)
            opt.backward_and_sparse_update([("p%d" % i, p, d) for i, (p, d) in enumerate(zip(params, grads))], threshold=threshold,
                                           spars=0.03 if topk else 2.0, topK=topk)
        return step, lambda: params + grads + opt.gradAccumulation
    (a, state_a), (ref, state_ref) = make("few"), make("few")
    others = [make(k)[0] for k in ("many", "threshold", "one", "wide")]
    for f in [a, ref] + others:                # buffers grow outside captures
        f()
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
            a()
    torch.cuda.current_stream().wait_stream(s)
    for k in range(8):
        graph.replay()
        others[k % len(others)]()
        if k % 3 == 0:
            others[(k + 1) % len(others)]()
        ref()
    torch.cuda.synchronize()
    assert all(torch.equal(x.view(torch.int32), y.view(torch.int32)) for x, y in zip(state_a(), state_ref()))
    del graph
    comm.close()
