"""The joint selection of a list of buckets and captured graphs: its buffers do
not grow inside a capture, and a graph that holds them stays valid when a wider
list makes them grow afterwards."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def make(sizes, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    grads = [[torch.randn(n, device="cuda", generator=gen) * 1e-3 for n in b] for b in sizes]
    return grads, [torch.zeros(sum(b), device="cuda") for b in sizes]


def expected(grads, residuals, threshold):
    out, left = [], []
    for bucket, r in zip(grads, residuals):
        s = torch.cat(bucket) + r
        kept = torch.where(s.abs() >= threshold, s, 0.0)
        out += list(kept.split([g.numel() for g in bucket]))
        left.append(s - kept)
    return out, left


def check(grads, residuals, want):
    torch.cuda.synchronize()
    for got, ref in zip(sum(grads, []) + residuals, want[0] + want[1]):
        assert torch.equal(got, ref)


@pytest.fixture
def comm():
    import gc
    from singa_b200.communicator import Communicator, NcclIdHolder
    c = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=1 << 22)
    yield c
    gc.collect()
    torch.cuda.synchronize()
    c.close()


SMALL, WIDE = [[700, 3], [513]], [[1 << 20, 5], [1 << 21], [4097]]
T = torch.tensor(1e-3).item()


def captured(body):
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        result = body()
    return g, result


def test_first_use_inside_a_capture_goes_bucket_by_bucket(comm):
    grads, residuals = make(SMALL, 1)
    comm.fusedSparsification([grads[1][0].clone()], residuals[1].clone(), T, False)   # the per-bucket buffers exist
    comm.wait()
    fresh = [[g.clone() for g in b] for b in grads]
    want = expected(fresh, residuals, T)

    def body():
        done = comm.sparsifyBuckets(grads, residuals, T)
        if not done:
            for b, r in zip(grads, residuals):
                comm.fusedSparsification(b, r, T, False)
        comm.wait()
        return done

    g, done = captured(body)
    assert done is False
    g.replay()
    check(grads, residuals, want)
    assert comm.sparsifyBuckets(*make(SMALL, 2), T) is True            # outside the capture it may allocate
    comm.wait()


def test_a_captured_selection_survives_growth(comm):
    grads, residuals = make(SMALL, 3)
    assert comm.sparsifyBuckets(*make(SMALL, 4), T) is True            # sized for the small list
    comm.wait()

    def body():
        done = comm.sparsifyBuckets(grads, residuals, T)
        comm.wait()
        return done

    g, done = captured(body)
    assert done is True
    wide, wide_residuals = make(WIDE, 5)
    want_wide = expected([[t.clone() for t in b] for b in wide], wide_residuals, T)
    assert comm.sparsifyBuckets(wide, wide_residuals, T) is True       # grows
    comm.wait()
    check(wide, wide_residuals, want_wide)
    for seed in (6, 7):
        fresh, _ = make(SMALL, seed)
        for a, b in zip(sum(grads, []), sum(fresh, [])):
            a.copy_(b)
        want = expected(fresh, [r.clone() for r in residuals], T)
        g.replay()
        check(grads, residuals, want)
    check(wide, wide_residuals, want_wide)                             # and nothing else was written
    del g
