"""DistOpt hands an exchange and the update behind it to a one-rank communicator
that does both, only where nothing in between has been replaced; and the ordering
of the sparse form, which runs on one stream (host logic)."""
import ctypes as C

import pytest
import torch

from singa_b200 import _lib
from singa_b200.opt import SGD, DistOpt


class Comm(object):
    world_size, local_rank, global_rank = 1, 0, 0
    takes = True

    def __init__(self):
        self.seen = []

    def synch(self, t): pass                                                 # noqa: E704
    fusedSynch = synchHalf = fusedSynchHalf = sparsification = fusedSparsification = synch

    def syncDense(self, stream, threshold, half=False):
        triples = list(stream)
        self.seen.append("dense")
        return [[t[i] for t in triples] for i in range(3)]

    def beginSparsification(self, ts, acc, spars, topK):
        self.seen.append("begin")

    def endSparsification(self):
        self.seen.append("end")

    def updateHalf(self, params, grads, moments, threshold, hyper):
        self.seen.append(("half", len(params), moments and len(moments), hyper))
        return self.takes

    def sparseUpdate(self, buckets, residuals, params, moments, spars, topK, hyper):
        self.seen.append(("sparse", [[g.numel() for g in b] for b in buckets], [p.numel() for p in params], topK))
        return self.takes

    def wait(self):
        self.seen.append("wait")


class Other(Comm):
    def syncDense(self, stream, threshold, half=False):
        return super().syncDense(stream, threshold, half)

    def beginSparsification(self, ts, acc, spars, topK):
        super().beginSparsification(ts, acc, spars, topK)


class OwnUpdate(DistOpt):
    def _update_all(self, plist):
        self.communicator.seen.append("mine")


class OwnSGD(SGD):
    def apply_many(self, *a):
        pass


def triples():
    return [("p%d" % i, torch.zeros(n), torch.ones(n)) for i, n in enumerate([30, 4, 50, 5])]


def run(opt, method, stream=None, **kw):
    opt.communicator.seen.clear()
    opt.opt.apply_many = lambda *a: opt.communicator.seen.append("apply") if type(opt.opt) is not SGD else None
    if type(opt.opt) is SGD:
        del opt.opt.apply_many
    getattr(opt, method)(triples() if stream is None else stream, threshold=20, **kw)
    return list(opt.communicator.seen)


def test_both_at_once():
    opt = DistOpt(SGD(lr=0.5, momentum=0.9), communicator=Comm())
    assert run(opt, "backward_and_update_half") == [("half", 4, 4, (0.5, 0.9, 0, 0, False, 1.0))]
    for topk in (False, True):
        # large tensors are buckets of their own, in front of the bucket that is still open
        assert run(opt, "backward_and_sparse_update", spars=0.1, topK=topk) == \
            [("sparse", [[30], [50], [4, 5]], [30, 50, 4, 5], topk), "wait"]
    assert opt.opt.step_counter == 3 and sorted(opt.opt.moments) == ["p0", "p1", "p2", "p3"]


@pytest.mark.parametrize("what", ["generator", "subclass of the optimizer", "communicator", "driver", "instance", "ranks"])
def test_one_after_the_other(what):
    comm = Other() if what == "communicator" else Comm()
    if what == "ranks":
        comm.world_size = 2
    opt = (OwnUpdate if what == "driver" else DistOpt)(OwnSGD() if what == "subclass of the optimizer" else
                                                       SGD(lr=0.0), communicator=comm)
    if what == "instance":
        comm.wait = lambda: comm.seen.append("own wait")
    stream = (lambda: (t for t in triples())) if what == "generator" else triples
    opt._update_all = opt._update_all if what == "driver" else lambda plist: None     # CPU tensors: not applied
    seen = run(opt, "backward_and_update_half", stream())
    assert seen[0] == "dense" and not any(isinstance(s, tuple) for s in seen)
    seen = run(opt, "backward_and_sparse_update", stream(), spars=0.1, topK=True)
    assert seen[0] == "begin" and not any(isinstance(s, tuple) for s in seen)


def test_a_communicator_that_declines():
    comm = Comm()
    comm.takes = False
    opt = DistOpt(SGD(lr=0.0), communicator=comm)
    with pytest.raises(ValueError):                    # the separate update: no CPU path
        run(opt, "backward_and_update_half")
    assert comm.seen[0][0] == "half" and comm.seen[1] == "dense"


def test_the_sparse_form_waits_for_the_reader_of_its_slot():
    lib, select, local, update = _lib.lib(), 16, 18, 20
    state, edges, stream = (C.c_ubyte * 4)(), (C.c_uint * 4)(), C.c_int()

    def plan(call):
        assert lib.sgb_comm_order_plan(state, call, edges, C.byref(stream)) == 0
        return list(edges)
    assert plan(update) == [1, 0, 0, 0] and stream.value == 1         # compute -> c1, and nothing else
    slots = state[3] >> 1 & 3
    assert slots in (0, 3)                                            # both halves' slots have moved on together
    for _ in range(2):
        plan(select), plan(local)                                     # both payloads are being read on c2
    assert plan(update)[0] == 1 | 1 << 14
    plan(7)
    assert list(state) == [0, 0, 0, 0] and plan(update)[0] == 1


def test_a_communicator_without_attributes_of_its_own():
    class Slots(object):
        __slots__ = ("world_size", "local_rank", "global_rank", "synchHalf", "fusedSynchHalf")

        def syncDense(self, stream, threshold, half=False):
            raise AssertionError("updateHalf is there")

        def updateHalf(self, params, grads, moments, threshold, hyper):
            return True

        def wait(self):
            pass
    comm = Slots()
    comm.world_size, comm.local_rank, comm.global_rank = 1, 0, 0
    opt = DistOpt(SGD(lr=0.5), communicator=comm)
    opt.backward_and_update_half(triples(), threshold=20)
    assert opt.opt.step_counter == 1


@pytest.mark.parametrize("owner, name", [(SGD, "apply_many"), (DistOpt, "_update_all"), (DistOpt, "wait")])
def test_a_function_put_into_the_class_is_called(owner, name, monkeypatch):
    opt, called = DistOpt(SGD(lr=0.5), communicator=Comm()), []
    for method, kw in (("backward_and_update_half", {}), ("backward_and_sparse_update", dict(spars=0.1))):
        both = run(opt, method, **kw)
        assert isinstance(both[0], tuple)
        with monkeypatch.context() as m:
            m.setattr(SGD, "apply_many", lambda self, *a: None)          # CPU tensors: not applied
            m.setattr(owner, name, lambda self, *a: called.append(name))
            seen = run(opt, method, **kw)
        assert called and not any(isinstance(s, tuple) for s in seen)
        called.clear()
        assert run(opt, method, **kw) == both


def test_a_communicator_that_declines_by_sizes():
    class Asked(Comm):
        """Asked first, before anything is prepared for the call."""
        answer = False

        def takesSparseUpdate(self, triples, threshold, topK):
            self.seen.append(("asked", [g.numel() for _, _, g in triples], threshold))
            return self.answer
    opt = DistOpt(SGD(lr=0.0), communicator=Asked())
    opt.opt._moments_of = lambda *a: opt.communicator.seen.append("prepared")
    with pytest.raises(ValueError):                      # the separate update: no CPU path
        run(opt, "backward_and_sparse_update", iter(triples()), spars=0.1, topK=True)
    assert opt.communicator.seen == [("asked", [30, 4, 50, 5], 20), "begin", "begin", "end", "begin", "end", "end",
                                     "wait", "prepared"]
    opt.communicator.answer = True
    assert [s[0] for s in run(opt, "backward_and_sparse_update", iter(triples()), spars=0.1, topK=True)][:3] == \
        ["asked", "p", "sparse"]


def test_no_communicator_takes_nothing():
    assert _lib.lib().sgb_comm_sparse_update_takes(None, None, None, None, 0, 0) == 0
    assert _lib.native.comm_sparse_update_takes(None, [("p", 1, 2)], 20, True) is False
