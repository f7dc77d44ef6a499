"""The Python layer's scratch: calls that overlap (two streams, a replay beside eager
calls, two host threads) exchange their sums through buffers of their own, so each
gives the bits that it gives alone; and a graph's buffer goes when the graph does."""
import ctypes
import threading

import pytest
import torch

from singa_b200 import _lib, singa_wrap as sw

pytestmark = pytest.mark.gpu

SHAPES = [(32, 64, 112, 112), (12, 96, 112, 112), (32, 128, 57, 57)]     # sums of many CTAs, of different numbers


def layer(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(shape, device="cuda", generator=g) + 1.0
    dy = torch.randn(shape, device="cuda", generator=g) * 1e-2
    c, h = shape[1], sw.CudnnBatchNormHandle(0.1, x)
    scale, bias = torch.rand(c, device="cuda", generator=g) + 0.5, torch.zeros(c, device="cuda")

    def step():
        rm, rv = torch.zeros(c, device="cuda"), torch.ones(c, device="cuda")
        y, mean, inv = sw.GpuBatchNormForwardTraining(h, x, scale, bias, rm, rv, 1e-5)
        return [y, mean, inv, rm, rv] + list(sw.GpuBatchNormReLUBackward(h, dy, y, x, scale, mean, inv)) + \
            list(sw.GpuBatchNormBackward(h, dy, x, scale, mean, inv))
    return step


def same(a, b):
    return all(torch.equal(p, q) for p, q in zip(a, b))


def no_faults():
    flags = ctypes.c_uint(1)
    _lib.call("sgb_bn_backward_faults", ctypes.byref(flags))
    return flags.value == 0


def test_two_streams_at_once():
    steps = [layer(s, i) for i, s in enumerate(SHAPES)]
    want = [f() for f in steps]
    streams = [torch.cuda.Stream() for _ in steps]
    torch.cuda.synchronize()
    got = [[] for _ in steps]
    for _ in range(6):
        for f, s, out in zip(steps, streams, got):
            with torch.cuda.stream(s):
                out.append(f())
    torch.cuda.synchronize()
    assert no_faults()
    for outs, w in zip(got, want):
        assert all(same(o, w) for o in outs)


def test_a_replay_beside_calls_on_the_stream_of_its_capture():
    a, b = layer(SHAPES[0], 1), layer(SHAPES[1], 2)
    want_a, want_b = a(), b()
    s, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s), torch.cuda.graph(graph, stream=s):
        held = a()
    for _ in range(6):
        with torch.cuda.stream(other):
            graph.replay()
        with torch.cuda.stream(s):
            got = b()
    torch.cuda.synchronize()
    assert same(held, want_a) and same(got, want_b) and no_faults()


def test_whose_buffer_it_is():
    t, s = torch.zeros(1, device="cuda"), torch.cuda.Stream()
    address = lambda: sw._workspace(t, 1000).data_ptr()   # noqa: E731
    mine, others = address(), []
    assert address() == mine
    with torch.cuda.stream(s):
        others.append(address())
        assert address() == others[0]
    worker = threading.Thread(target=lambda: others.append(address()))
    worker.start()
    worker.join()
    assert mine not in others and address() == mine


def test_a_graph_takes_its_buffer_along():
    t, big = torch.zeros(1, device="cuda"), 32 << 20
    sw._workspace(t, 1000)
    before = torch.cuda.memory_allocated()
    for _ in range(4):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            a, b = sw._workspace(t, big).data_ptr(), sw._workspace(t, 1000).data_ptr()
            t.add_(1)
        assert a == b and a != sw._workspace(t, 1000).data_ptr()
        graph.replay()
        torch.cuda.synchronize()
        graph.reset()
        assert torch.cuda.memory_allocated() - before <= 2 * big
