"""A step that is recorded once and replayed still follows what its owner sets
between two runs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def comm():
    import gc
    from singa_b200.communicator import Communicator, NcclIdHolder
    c = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=1 << 20)
    yield c
    gc.collect()
    torch.cuda.synchronize()
    c.close()


def small_step(comm=None, **kw):
    from singa_b200.hot_path import HotPathGPU
    from singa_b200.resnet50_path import build_mlp_plan
    return HotPathGPU(build_mlp_plan(batch=8, dims=(12, 16, 16, 10)), communicator=comm, seed=3, threshold=200, **kw)


@pytest.mark.parametrize("dist_option", ["plain", "half"])
def test_phases_are_timed_when_a_step_has_been_replayed(comm, dist_option):
    hp = small_step(comm, dist_option=dist_option)
    for _ in range(6):
        hp.run_step()
    for rounds in (1, 5):                       # also past the run at which a step is captured
        comm.profile_begin()
        for _ in range(rounds):
            hp.run_step()
        rows = comm.profile_end()
        names = [n for n, _, _ in rows]
        assert names.count("sgd_update_bucket") == rounds * len(hp.events), names
        assert sum(n.startswith("Dist_") for n in names) >= rounds * len(hp.events)
        assert all(t1 >= t0 >= 0 for _, t0, t1 in rows)
        for _ in range(4):
            hp.run_step()


def parameters(hp):
    torch.cuda.synchronize()
    return [hp.t[p].clone() for p in hp.plan["params"]]


@pytest.mark.parametrize("every, most", [(0, 1), (1, 0), (2, 0), (3, 2), (4, 2), (50, 2)])
def test_captures_are_few_when_the_rate_keeps_changing(every, most):
    """A rate that changes every few runs makes one short-lived capture, and the
    next one only after 40 runs, and then 160; 48 replays pay for a capture."""
    from singa_b200 import _lib
    hp, one_by_one = small_step(), small_step()
    one_by_one.profile = True                   # never captured
    for i in range(100):
        if every and i % every == 0:
            hp.lr = one_by_one.lr = 0.1 / (i + 1)
        hp.run_step()
        one_by_one.run_step()
    assert _lib.native.program_captures(hp._program) <= most
    assert _lib.native.program_captures(one_by_one._program) == 0
    for a, b in zip(parameters(hp), parameters(one_by_one)):
        assert torch.equal(a, b)
    if every:                                   # settings that last are captured in the end
        before = _lib.native.program_captures(hp._program)
        for _ in range(170):
            hp.run_step()
        assert _lib.native.program_captures(hp._program) == before + (every not in (50,))


def test_a_step_captured_by_its_owner_while_phases_are_timed(comm):
    hp = small_step(comm)
    hp.run_step()
    torch.cuda.synchronize()
    comm.profile_begin()
    g = hp.capture()                            # no timing event goes into the graph
    g.replay()
    hp.run_step()
    rows = comm.profile_end()
    assert sum(n == "sgd_update_bucket" for n, _, _ in rows) == len(hp.events)
    hp.release_graph()
    del g


def test_world_size_and_exchange_may_change_between_runs(comm):
    a, b = small_step(), small_step(world=4)
    for _ in range(4):                          # `a` has been captured by now
        a.run_step()
    a.world = 4
    for hp in (a, b):
        for p in hp.plan["params"]:
            hp.t[p].fill_(0.5)
            hp.moments[p].zero_()
        hp.grad_arena.fill_(0.25)
    assert a.run_step() == b.run_step()
    for x, y in zip(parameters(a), parameters(b)):
        assert torch.equal(x, y)
    alone, at_the_end = small_step(comm), small_step(comm, update_on_arrival=False)
    alone.run_step()
    alone.update_on_arrival = False             # from here on one update behind the last exchange
    at_the_end.run_step()
    assert alone.run_step() == at_the_end.run_step()
    for x, y in zip(parameters(alone), parameters(at_the_end)):
        assert torch.equal(x, y)
    top = small_step(comm, dist_option="sparseTopK", spars=0.5)
    top.run_step()
    top.spars = 0.01
    top.run_step()
    torch.cuda.synchronize()
    largest_bucket = max(r.numel() for r in top.residuals.values())
    kept = sum(int((r != 0).sum()) for r in top.residuals.values())
    assert kept > 0.9 * largest_bucket          # nearly everything stays behind


def test_a_closed_communicator_is_an_error():
    from singa_b200 import _lib
    from singa_b200.communicator import Communicator, NcclIdHolder
    c = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=1 << 20)
    hp = small_step(c)
    for _ in range(4):
        hp.run_step()
    torch.cuda.synchronize()
    c.close()
    with pytest.raises(_lib.SgbError, match="closed"):
        hp.run_step()
    hp.comm = None                              # without an exchange the step still runs
    hp.update_on_arrival = False
    assert hp.run_step() > 0
    torch.cuda.synchronize()


def test_a_step_with_layers_that_visit_their_data_twice_is_captured():
    from singa_b200 import _lib
    from singa_b200.hot_path import HotPathGPU
    from singa_b200.resnet50_path import build_plan
    steps = [HotPathGPU(build_plan(batch=9, image=224, fused=True), seed=3) for _ in range(2)]
    steps[1].profile = True                     # never captured
    for _ in range(5):
        for hp in steps:
            hp.run_step()
    assert [_lib.native.program_captures(hp._program) for hp in steps] == [1, 0]
    for a, b in zip(*map(parameters, steps)):
        assert torch.equal(a, b)
