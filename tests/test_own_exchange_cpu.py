"""DistOpt hands a whole exchange to a communicator that offers it in one call,
but a subclass's or an instance's own version of one of the calls that it stands
for is still the one that is called (host logic)."""
import pytest
import torch

from singa_b200.opt import DistOpt


class Comm(object):
    world_size, local_rank, global_rank = 1, 0, 0

    def __init__(self):
        self.seen = []

    def synch(self, t):
        self.seen.append(("synch", t.numel()))

    def fusedSynch(self, ts, send=True):
        self.seen.append(("fusedSynch", sum(t.numel() for t in ts), send))

    def synchHalf(self, t):
        self.seen.append(("synchHalf", t.numel()))

    def fusedSynchHalf(self, ts, send=True):
        self.seen.append(("fusedSynchHalf", sum(t.numel() for t in ts), send))

    def sparsification(self, t, acc, spars, topK):
        self.seen.append(("sparsification", t.numel()))

    def fusedSparsification(self, ts, acc, spars, topK):
        self.seen.append(("fusedSparsification", sum(t.numel() for t in ts)))

    def syncDense(self, stream, threshold, half=False):
        triples = list(stream)
        self.seen.append(("syncDense", half))
        return [[t[i] for t in triples] for i in range(3)]

    def beginSparsification(self, ts, acc, spars, topK):
        self.seen.append(("begin", sum(t.numel() for t in ts)))

    def endSparsification(self):
        self.seen.append(("end",))

    def sparsifyBuckets(self, buckets, residuals, threshold):
        self.seen.append(("joint", len(buckets)))
        return True

    def wait(self):
        pass


class OwnSynch(Comm):
    def synch(self, t):
        super().synch(t)


class OwnSparse(Comm):
    def fusedSparsification(self, ts, acc, spars, topK):
        super().fusedSparsification(ts, acc, spars, topK)


class OwnForwards(DistOpt):
    def all_reduce(self, t):
        self.communicator.seen.append(("mine",))

    def fused_sparsification(self, ts, acc, spars, topK):
        self.communicator.seen.append(("mine sparse",))


class Opt(object):
    def apply_many(self, *args):
        pass

    def step(self):
        pass


SIZES = [30, 4, 5]
DENSE = [("synch", 30), ("fusedSynch", 4, False), ("fusedSynch", 5, False), ("fusedSynch", 9, True)]


def triples():
    return [("p%d" % i, torch.zeros(n), torch.ones(n)) for i, n in enumerate(SIZES)]


def run(opt, method, **kw):
    opt.communicator.seen.clear()
    getattr(opt, method)(iter(triples()), threshold=20, **kw)
    return list(opt.communicator.seen)


def test_nobodys_own_version():
    opt = DistOpt(Opt(), communicator=Comm())
    assert run(opt, "backward_and_update") == [("syncDense", False)]
    assert run(opt, "backward_and_update_half") == [("syncDense", True)]
    assert run(opt, "backward_and_sparse_update", spars=0.1) == [("joint", 2)]
    assert run(opt, "backward_and_sparse_update", spars=0.1, topK=True) == [("begin", 30), ("begin", 9), ("end",), ("end",)]


def test_a_communicator_with_its_own_call():
    opt = DistOpt(Opt(), communicator=OwnSynch())
    assert run(opt, "backward_and_update") == DENSE
    assert run(opt, "backward_and_update_half") == [("syncDense", True)]
    opt = DistOpt(Opt(), communicator=OwnSparse())
    want = [("sparsification", 30), ("fusedSparsification", 9)]
    assert run(opt, "backward_and_sparse_update", spars=0.1) == want
    assert run(opt, "backward_and_sparse_update", spars=0.1, topK=True) == want
    assert run(opt, "backward_and_update") == [("syncDense", False)]


def test_an_instance_with_its_own_call():
    opt = DistOpt(Opt(), communicator=Comm())
    counted = []
    opt.communicator.fusedSynchHalf = lambda ts, send=True: counted.append(send)
    assert run(opt, "backward_and_update_half") == [("synchHalf", 30)] and counted == [False, False, True]
    assert run(opt, "backward_and_update") == [("syncDense", False)]


@pytest.mark.parametrize("topK", [False, True])
def test_an_optimizer_with_its_own_forward(topK):
    opt = OwnForwards(Opt(), communicator=Comm())
    assert run(opt, "backward_and_update") == [("mine",)] + DENSE[1:]
    assert run(opt, "backward_and_sparse_update", spars=0.1, topK=topK) == [("sparsification", 30), ("mine sparse",)]


def test_a_communicator_without_whole_calls():
    class Plain(object):
        world_size, local_rank, global_rank = 1, 0, 0
        seen = []
        synch, fusedSynch, wait = Comm.synch, Comm.fusedSynch, Comm.wait
    assert run(DistOpt(Opt(), communicator=Plain()), "backward_and_update") == DENSE


@pytest.mark.parametrize("where", ["communicator", "driver"])
def test_a_call_put_into_the_class_is_called(where, monkeypatch):
    """Also after the same classes have been looked at without it, and no longer than it is there."""
    class Traced(Comm):
        pass
    Traced.synch = Comm.synch
    Traced.syncDense = Comm.syncDense
    Traced._defined = dict(vars(Traced))
    opt = DistOpt(Opt(), communicator=Traced())
    stream = lambda: [("p%d" % i, torch.zeros(n), torch.ones(n)) for i, n in enumerate(SIZES)]   # noqa: E731

    def seen():
        opt.communicator.seen.clear()
        opt.backward_and_update(stream(), threshold=20)
        return list(opt.communicator.seen)
    whole = [("syncDense", False)]
    assert seen() == whole
    with monkeypatch.context() as m:
        if where == "communicator":
            m.setattr(Traced, "synch", lambda self, t: self.seen.append(("traced",)))
        else:
            m.setattr(DistOpt, "all_reduce", lambda self, t: self.communicator.seen.append(("traced",)))
        assert seen() == [("traced",)] + DENSE[1:]
    assert seen() == whole
