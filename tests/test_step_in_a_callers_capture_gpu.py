"""A captured step of one rank, which exchanges nothing itself, beside exchanges that the
caller has queued on the same communicator: those of the same capture are joined, those
from before it are left for the caller's wait()."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def make(sync, threshold):
    from singa_b200.communicator import Communicator, NcclIdHolder
    from singa_b200.hot_path import HotPathGPU
    from singa_b200.resnet50_path import add_wgrad_refresh, build_mlp_plan, fuse_plan
    comm = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=1 << 20)
    plan = add_wgrad_refresh(fuse_plan(build_mlp_plan(batch=9, dims=(23, 130, 57, 10))))
    return comm, HotPathGPU(plan, communicator=comm, seed=5, threshold=threshold, dist_option=sync)


def bits(hp):
    torch.cuda.synchronize()
    return [hp.t[p].clone() for p in hp.plan["params"]] + [hp.moments[p].clone() for p in hp.plan["params"]] + [hp.grad_arena.clone()]


@pytest.mark.parametrize("sync", ["plain", "half"])
@pytest.mark.parametrize("threshold", [1, 3000, 1 << 20])
@pytest.mark.parametrize("queued", ["inside", "before"])
def test_with_an_exchange_of_the_callers(sync, threshold, queued):
    comm, hp = make(sync, threshold)
    alone_comm, alone = make(sync, threshold)
    x = torch.linspace(-3, 3, 70001, device="cuda")
    want = x.half().float()
    comm.synchHalf(torch.ones(70001, device="cuda"))          # its buffers are made outside captures
    comm.wait()
    for _ in range(2):
        hp.run_step()
        alone.run_step()
    torch.cuda.synchronize()
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    if queued == "before":
        comm.synchHalf(x)
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
            if queued == "inside":
                comm.synchHalf(x)
            hp.run_step()
    torch.cuda.current_stream().wait_stream(s)
    comm.wait()                                   # nothing is left over that this cannot join
    for _ in range(3):
        graph.replay()
        alone.run_step()
    assert torch.equal(x, want)
    assert all(torch.equal(a, b) for a, b in zip(bits(hp), bits(alone)))
    del graph
    comm.close()
    alone_comm.close()
