"""A gradient stream or an exchange that fails in the middle of a sparse update
leaves the communicator usable and the residuals in step (host logic, with a
communicator that keeps the rules of the real one: at most two exchanges open,
ended in order, none open at wait())."""
import pytest
import torch

from singa_b200.opt import DistOpt


class Comm(object):
    world_size, local_rank, global_rank = 2, 0, 0

    def __init__(self, capacity=100):
        self.capacity, self.open, self.ended, self.waits = capacity, [], [], 0

    def beginSparsification(self, ts, accumulation, spars, topK):
        n = sum(t.numel() for t in ts)
        if n > self.capacity:
            raise RuntimeError("capacity")
        assert len(self.open) < 2 and (accumulation is None or accumulation.numel() == n)
        self.open.append(n)

    def endSparsification(self):
        self.ended.append(self.open.pop(0))

    def wait(self):
        assert not self.open
        self.waits += 1


class Opt(object):
    def __init__(self):
        self.updates = []

    def apply_many(self, names, params, grads, scale):
        self.updates.append(list(names))

    def step(self):
        pass


def triples(sizes, fail_at=None):
    for i, n in enumerate(sizes):
        if i == fail_at:
            raise ValueError("backward")
        yield "p%d" % i, torch.zeros(n), torch.ones(n)


SIZES = [30, 7, 8, 40, 50]                     # above 20: direct; 7 + 8 wait for the end of the list


@pytest.mark.parametrize("fail_at", range(len(SIZES)))
@pytest.mark.parametrize("corr", [True, False])
def test_a_stream_that_raises(fail_at, corr):
    comm, inner = Comm(), Opt()
    opt = DistOpt(inner, communicator=comm)
    for done in (1, 2):                        # once before the residuals exist, once again
        with pytest.raises(ValueError, match="backward"):
            opt.backward_and_sparse_update(triples(SIZES, fail_at), threshold=20, spars=0.1, corr=corr)
        assert inner.updates == [] and comm.waits == done
    comm.ended.clear()
    opt.backward_and_sparse_update(triples(SIZES), threshold=20, spars=0.1, corr=corr)
    assert comm.ended == [30, 40, 50, 15] and len(inner.updates) == 1
    if corr:
        assert [r.numel() for r in opt.gradAccumulation] == [30, 40, 50, 15]
    with pytest.raises(ValueError, match="backward"):
        opt.backward_and_sparse_update(triples(SIZES, fail_at), threshold=20, spars=0.1, corr=corr)
    opt.backward_and_sparse_update(triples(SIZES), threshold=20, spars=0.1, corr=corr)
    if corr:
        assert len(opt.gradAccumulation) == 4


def test_an_exchange_that_is_refused():
    comm, inner = Comm(capacity=45), Opt()
    opt = DistOpt(inner, communicator=comm)
    with pytest.raises(RuntimeError, match="capacity"):
        opt.backward_and_sparse_update(triples(SIZES), threshold=20, spars=0.1)
    assert comm.ended == [30, 40] and comm.waits == 1
    opt.backward_and_sparse_update(triples(SIZES[:4]), threshold=20, spars=0.1)
    assert len(inner.updates) == 1
