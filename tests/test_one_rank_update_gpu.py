"""On one rank, gradients that all exist are exchanged and their parameters updated
in one pass (half precision), or in the kernel that writes the dense gradients
(sparse): the same bits in gradients, parameters, momentum and residuals as the
call-by-call path, which a generator takes; and that path wherever an optimizer
or a call of its own is to be used."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

# (sizes, threshold): buckets that end inside a tile, on one, gaps, large tensors between, many small ones
LISTS = [([5], 100), ([40000, 33], 50000), ([3000] * 120, 5000), ([1, 511, 513, 4096, 3], 2000), ([70000, 12, 4097, 30000, 8191, 1], 20000),
         ([64] * 300, 1000), ([300001, 4, 4, 4, 1 << 20], 1 << 19), ([0, 7, 0, 9], 4)]
OPTIONS = [dict(lr=0.05, momentum=0.9, weight_decay=1e-4), dict(lr=0.1), dict(lr=0.1, momentum=0.8, nesterov=True)]


@pytest.fixture(scope="module")
def comm():
    from singa_b200.communicator import Communicator, NcclIdHolder
    c = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=1 << 22)
    c.set_topk_mode("magnitude")
    yield c
    torch.cuda.synchronize()
    c.close()


def run(comm, sizes, threshold, options, method, as_list, offset, steps=3, opt_type=None, **kw):
    from singa_b200.opt import SGD, DistOpt
    opt = DistOpt((opt_type or SGD)(**options), communicator=comm)
    g = torch.Generator(device="cuda").manual_seed(1)
    make = lambda n: torch.randn(n + offset, device="cuda", generator=g)[offset:]   # noqa: E731
    params, out = [make(n) for n in sizes], []
    for _ in range(steps):
        grads = [make(n) for n in sizes]
        triples = [("p%d" % i, p, d) for i, (p, d) in enumerate(zip(params, grads))]
        getattr(opt, method)(triples if as_list else (t for t in triples), threshold=threshold, **kw)
        out += [d.clone() for d in grads]
    torch.cuda.synchronize()
    assert opt.opt.step_counter == steps
    return out + params + [opt.opt.moments[k] for k in sorted(opt.opt.moments)] + getattr(opt, "gradAccumulation", [])


def same(a, b):
    return len(a) == len(b) and all(torch.equal(x.view(torch.int32), y.view(torch.int32)) for x, y in zip(a, b))


@pytest.mark.parametrize("sizes,threshold", LISTS)
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("options", OPTIONS)
def test_half(comm, sizes, threshold, offset, options):
    args = (comm, sizes, threshold, options, "backward_and_update_half")
    assert same(run(*args, True, offset), run(*args, False, offset))


@pytest.mark.parametrize("sizes,threshold", LISTS[:-1])
@pytest.mark.parametrize("topk,spars", [(False, 1.5), (False, 0.0), (True, 0.01), (True, 0.6)])
@pytest.mark.parametrize("options", OPTIONS[:2])
def test_sparse(comm, sizes, threshold, topk, spars, options):
    args = (comm, sizes, threshold, options, "backward_and_sparse_update")
    for offset in (0, 1):
        kw = dict(spars=spars, topK=topk)
        assert same(run(*args, True, offset, **kw), run(*args, False, offset, **kw)), offset


def test_an_optimizer_of_its_own_is_called(comm):
    from singa_b200.opt import SGD

    class Counting(SGD):
        calls = 0

        def apply_many(self, *a):
            Counting.calls += 1
            super().apply_many(*a)
    for method, kw in (("backward_and_update_half", {}), ("backward_and_sparse_update", dict(spars=1.0))):
        Counting.calls = 0
        got = run(comm, [700, 30, 9], 500, OPTIONS[0], method, True, 0, opt_type=Counting, **kw)
        assert Counting.calls == 3 and same(got, run(comm, [700, 30, 9], 500, OPTIONS[0], method, True, 0, **kw))


def test_a_captured_update(comm):
    from singa_b200.opt import SGD, DistOpt
    opt = DistOpt(SGD(**OPTIONS[0]), communicator=comm)
    p, g = [torch.randn(n, device="cuda") for n in (5000, 300)], [torch.randn(n, device="cuda") for n in (5000, 300)]
    triples = [("p%d" % i, a, b) for i, (a, b) in enumerate(zip(p, g))]
    for method, kw in (("backward_and_update_half", {}), ("backward_and_sparse_update", dict(spars=1.0)),
                       ("backward_and_sparse_update", dict(spars=0.05, topK=True))):
        step = lambda: getattr(opt, method)(list(triples), threshold=1000, **kw)   # noqa: E731
        step()
        state = [t.clone() for t in p + g + list(opt.opt.moments.values()) + getattr(opt, "gradAccumulation", [])]
        live = p + g + list(opt.opt.moments.values()) + getattr(opt, "gradAccumulation", [])
        step()
        want = [t.clone() for t in live]
        graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
                step()
        for t, v in zip(live, state):
            t.copy_(v)
        graph.replay()
        torch.cuda.synchronize()
        assert same(live, want), (method, kw)
        del graph


# Larger lists: chunks drawn from a part's ticket (6e6 elements in all), runs of four
# tiles and the sampled bound (from 9.7e6), one bucket a fifth of the others.
WIDE = [([190003, 1900001, 333] * 3, 500000), ([2100000, 57000, 1] * 11, 1 << 21), ([4100000, 4100000, 500000, 400000, 4100000], 1 << 19)]


def bucket_sizes(sizes, threshold):
    out, held = [], 0
    for n in sizes:
        if n > threshold:
            out.append(n)
            continue
        held += n
        if held > threshold:
            out.append(held)
            held = 0
    return out + [held] * (held > 0)


def gradients(values, sizes, threshold, g):
    n, dev = sum(sizes), torch.device("cuda")
    flat = torch.randn(n, device=dev, generator=g)
    if values == "small":                        # every integer-truncated key is 0
        flat.mul_(1e-2)
    if values == "ties":                         # a crowded bin
        flat.round_()
    out = list(flat.split(sizes))
    if values == "misleading":
        # large where the sample looks (128 elements at the start of each warp's share of the bucket) and
        # nowhere else: fewer than k lie above the bound that it gives
        ctas, total = 4 * torch.cuda.get_device_properties(0).multi_processor_count, sum(sizes)
        for i, size in enumerate(sizes):
            if size > threshold:
                share = max(1, (ctas - len(bucket_sizes(sizes, threshold))) * size // total)
                at = torch.arange(size, device=dev) % (size // (8 * share)) < 128
                out[i] = torch.where(at, out[i] * 100, out[i] * 0.01)
    return [t.clone() for t in out]


@pytest.mark.parametrize("sizes,threshold", WIDE)
@pytest.mark.parametrize("spars", [0.003, 0.04, 0.2])           # the sample is for shares up to a twelfth
@pytest.mark.parametrize("mode", ["magnitude", "compat"])
@pytest.mark.parametrize("values", ["normal", "small", "ties", "misleading"])
def test_joint_selection_of_large_lists(comm, sizes, threshold, spars, mode, values):
    from singa_b200 import _lib
    from singa_b200.opt import SGD, DistOpt
    comm.set_topk_mode(mode)
    try:
        sides = []
        for as_list in (True, False):
            g = torch.Generator(device="cuda").manual_seed(3)
            opt = DistOpt(SGD(**OPTIONS[0]), communicator=comm)
            params, grads = [torch.zeros(n, device="cuda") for n in sizes], []
            for _ in range(2):
                grads = gradients(values, sizes, threshold, g)
                triples = [("p%d" % i, p, d) for i, (p, d) in enumerate(zip(params, grads))]
                assert comm.takesSparseUpdate(triples, threshold, True)
                opt.backward_and_sparse_update(triples if as_list else (t for t in triples), threshold=threshold,
                                               spars=spars, topK=True)
            sides.append(grads + params + [opt.opt.moments["p%d" % i] for i in range(len(sizes))] + opt.gradAccumulation)
        torch.cuda.synchronize()
        assert same(*sides)
        faults = ctypes.c_uint(1)
        _lib.call("sgb_sparse_faults", ctypes.byref(faults))
        assert faults.value == 0
    finally:
        comm.set_topk_mode("magnitude")


def test_what_is_taken_is_known_ahead(comm):
    """By size: 2 to 32 buckets of at most 256 pieces, or one of 16 tensors.  By threshold: at most 8 tensors and 4 million elements."""
    for sizes, threshold, topk, want in (([300] * 33, 100, True, False), ([300] * 32, 100, True, True),
                                         ([500000] * 8, 1 << 21, False, True), ([400000] * 9, 1 << 21, False, False),
                                         ([1 << 20] * 4, 1 << 21, False, False), ([50] * 16, 1000, True, True), ([50] * 17, 1000, True, False),
                                         ([1 << 22], 1 << 21, True, True), ([8] * 600, 1000, True, True)):
        flat = torch.zeros(sum(sizes), device="cuda")      # back to back: one piece a bucket
        grads = list(flat.split(sizes))
        assert comm.takesSparseUpdate([("p", g, g) for g in grads], threshold, topk) is want, (len(sizes), topk)
    apart = [torch.zeros(8, device="cuda") for _ in range(257)]
    assert not comm.takesSparseUpdate([("p", g, g) for g in apart], 1000, True)
    assert comm.takesSparseUpdate([("p", g, g) for g in apart[:-1]], 1000, True)
