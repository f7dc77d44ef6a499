"""The one-kernel selectors where their plan changes: one tile, the last size of
one-tile runs and the first of four-tile runs, chunks drawn from the counter,
runs whose list overflows, every key alike - and the two-halves exchange.  Sums
are single fp32 additions and selections are exact, so equality is bitwise."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TURN = 4 * 8 * 4 * 148 * 512            # elements up to which a warp's run is one tile on 148 SMs


def largest(s, k, mode):
    key = s.abs() if mode == "magnitude" else s.double().trunc().abs()
    return torch.sort(key, descending=True, stable=True).indices[:k].sort().values


@pytest.mark.parametrize("n", [511, 512, 513, TURN // 2 + 5, TURN, TURN + 1, 2 * TURN + 4099])
@pytest.mark.parametrize("shape", ["gaussian", "clustered", "alike"])
def test_selection_where_the_plan_changes(n, shape):
    from singa_b200 import singa_wrap as sw
    gen = torch.Generator(device="cuda").manual_seed(n)
    g = torch.randn(n, device="cuda", generator=gen) * 1e-3
    if shape == "clustered":             # one range in which everything is selected: its lists overflow
        g[n // 3:n // 3 + n // 20 + 1] *= 100
    elif shape == "alike":
        g.fill_(0.25)
    acc = torch.randn(n, device="cuda", generator=gen) * 1e-3 if shape != "alike" else torch.zeros(n, device="cuda")
    s = g + acc
    want = torch.nonzero(s.abs() >= torch.tensor(2e-3, device="cuda")).flatten()
    got_acc = acc.clone()
    idx, val = sw.sparse_threshold(g, got_acc, 2e-3)
    assert torch.equal(idx.long() - 1, want) and torch.equal(val, s[want])
    left = s.clone()
    left[want] = 0
    assert torch.equal(got_acc, left)
    k = max(1, n // 25)
    for mode in ("magnitude", "compat"):
        scaled = g * 1e6 if mode == "compat" and shape != "alike" else g   # keys with a middle digit
        s = scaled + acc
        got_acc = acc.clone()
        idx, val = sw.sparse_topk(scaled, got_acc, k, mode)
        want = largest(s, k, mode)
        assert torch.equal(idx.long() - 1, want) and torch.equal(val, s[want])
        left = s.clone()
        left[want] = 0
        assert torch.equal(got_acc, left)


@pytest.mark.parametrize("n", [2 * TURN + 1, 2 * TURN + 4099])
@pytest.mark.parametrize("shape", ["gaussian", "heavy", "planted", "alike"])
def test_top_k_with_a_sampled_bound(n, shape):
    """`planted`: one sampled warp in twelve sees large keys that are nowhere
    else, so the bound is too high and the full count has to take over."""
    from singa_b200 import singa_wrap as sw
    gen = torch.Generator(device="cuda").manual_seed(n)
    g = torch.randn(n, device="cuda", generator=gen)
    if shape == "heavy":
        g = g ** 7
    elif shape == "planted":
        warps = 148 * 4 * 8
        starts = torch.arange(0, warps, 12, device="cuda") * (n // warps)
        g[(starts[:, None] + torch.arange(128, device="cuda")).flatten()] = 1000.0
    elif shape == "alike":
        g.fill_(0.25)
        g[n // 2:n // 2 + 500] = 0.5
    for k in (1, 499, 501, n // 100, n // 12, n // 12 + 1):
        acc = torch.zeros(n, device="cuda")
        idx, val = sw.sparse_topk(g, acc, k, "magnitude")
        want = largest(g, k, "magnitude")
        assert torch.equal(idx.long() - 1, want) and torch.equal(val, g[want])
        left = g.clone()
        left[want] = 0
        assert torch.equal(acc, left)


def test_two_halves_equal_one_call_and_keep_their_order():
    from singa_b200 import _lib
    from singa_b200.communicator import Communicator, NcclIdHolder
    comm = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=300000)
    try:
        gen = torch.Generator(device="cuda").manual_seed(3)
        buckets = [[torch.randn(m, device="cuda", generator=gen) * 1e-3 for m in sizes]
                   for sizes in ((70000, 3, 4097), (250001,), (8, 8, 8))]
        for topk, spars in ((False, 1e-3), (True, 0.05)):
            one = [[t.clone() for t in b] for b in buckets]
            two = [[t.clone() for t in b] for b in buckets]
            acc1 = [torch.zeros(sum(t.numel() for t in b), device="cuda") for b in buckets]
            acc2 = [a.clone() for a in acc1]
            for b, a in zip(one, acc1):
                comm.fusedSparsification(b, a, spars, topk)
            comm.wait()
            comm.beginSparsification(two[0], acc2[0], spars, topk)
            comm.beginSparsification(two[1], acc2[1], spars, topk)
            with pytest.raises(_lib.SgbError):                     # two are open already
                comm.beginSparsification(two[2], acc2[2], spars, topk)
            with pytest.raises(_lib.SgbError):
                comm.wait()
            comm.endSparsification()
            comm.beginSparsification(two[2], acc2[2], spars, topk)
            comm.endSparsification()
            comm.endSparsification()
            with pytest.raises(_lib.SgbError):
                comm.endSparsification()
            comm.wait()
            for x, y in zip(sum(one, []) + acc1, sum(two, []) + acc2):
                assert torch.equal(x, y)
    finally:
        torch.cuda.synchronize()
        comm.close()
