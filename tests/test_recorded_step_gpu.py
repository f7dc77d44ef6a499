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
