"""A captured step without other ranks updates its buckets on a branch beside the
backward pass: the same bits as the calls one by one, captured by the library or by
the caller, for one bucket and for many, and whatever the exchange."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def step(sync, threshold, comm, **kw):
    from singa_b200.hot_path import HotPathGPU
    from singa_b200.resnet50_path import add_wgrad_refresh, build_mlp_plan, fuse_plan
    plan = fuse_plan(build_mlp_plan(batch=9, dims=(23, 130, 57, 10)))
    if sync != "none":
        plan = add_wgrad_refresh(plan)
    return HotPathGPU(plan, communicator=comm if sync != "none" else None, seed=5, threshold=threshold,
                      dist_option=sync if sync != "none" else "plain", **kw)


def state(hp):
    torch.cuda.synchronize()
    return [hp.t[p] for p in hp.plan["params"]] + [hp.moments[p] for p in hp.plan["params"]] + [hp.grad_arena, hp.t["loss"]]


@pytest.mark.parametrize("sync", ["none", "plain", "half"])
@pytest.mark.parametrize("threshold", [1, 200, 3000, 1 << 20])          # a bucket a tensor ... one bucket
@pytest.mark.parametrize("on_arrival", [True, False])
def test_captured_steps_equal_single_calls(sync, threshold, on_arrival):
    from singa_b200.communicator import Communicator, NcclIdHolder
    comm = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=1 << 20)
    make = lambda: step(sync, threshold, comm, update_on_arrival=on_arrival)   # noqa: E731
    single, library, caller = make(), make(), make()
    single.profile = True                        # one by one
    caller.run_step()
    torch.cuda.synchronize()
    graph = caller.capture()
    for k in range(6):
        single.run_step()
        library.run_step()
        if k:
            graph.replay()
    for other in (library, caller):
        assert all(torch.equal(a, b) for a, b in zip(state(single), state(other))), (sync, threshold)
    caller.release_graph()
    del graph
    comm.close()


def replayed(hp, runs=3):
    hp.run_step()
    torch.cuda.synchronize()
    graph = hp.capture()
    for _ in range(runs - 1):
        graph.replay()
    out = [t.clone() for t in state(hp)]
    hp.release_graph()
    return out


def branches(hp):
    """What the recorded step does on a branch of its own."""
    return hp._forked_update()[0]


def test_the_branch_can_be_turned_off():
    on, off, built_off = step("none", 200, None), step("none", 200, None), step("none", 200, None, update_on_arrival=False)
    assert branches(on) and not branches(built_off)
    off.update_on_arrival = False
    assert not branches(off)
    assert all(torch.equal(a, b) for a, b in zip(replayed(on), replayed(off)))


@pytest.mark.parametrize("change", ["no communicator", "sparse"])
def test_what_arrives_follows_what_is_set(change):
    """Captured steps and single ones do the same after the exchange has been changed."""
    from singa_b200.communicator import Communicator, NcclIdHolder
    comm = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=1 << 20)
    single, captured = step("plain", 200, comm), step("plain", 200, comm)
    reference = step("plain", 200, comm)
    reference.update_on_arrival = False
    for hp in (single, captured, reference):
        if change == "sparse":
            hp.dist_option, hp.spars = "sparseTopK", 0.4
            hp.residuals = {i: torch.zeros(sum(hp.grads[k].numel() for k in ev[1]), device="cuda") for i, ev in hp.flush_after.items()}
        else:
            hp.comm = None
    assert not (change == "sparse" and branches(captured))
    for _ in range(3):
        single.run_step()
        reference.run_step()
    want = state(reference)
    assert all(torch.equal(a, b) for a, b in zip(state(single), want))
    assert any(bool(m.any()) for m in single.moments.values())
    if change != "sparse":                       # (a captured sparse step is not replayed here: the host takes part)
        assert all(torch.equal(a, b) for a, b in zip(replayed(captured), want))
    comm.close()


@pytest.mark.parametrize("kind", ["no update", "a gradient changed behind its report"])
def test_plans_of_other_forms(kind):
    from singa_b200.hot_path import HotPathGPU
    from singa_b200.resnet50_path import Op, build_mlp_plan, fuse_plan
    plan = fuse_plan(build_mlp_plan(batch=9, dims=(23, 130, 57, 10)))
    if kind == "no update":
        ops = [op for op in plan["ops"] if op.kind != "sync_and_update"]
    else:
        ops = plan["ops"][:-1] + [Op("scale", dict(x="d:" + plan["grad_order"][0], c=0.5))] + plan["ops"][-1:]
    single, captured = [HotPathGPU(dict(plan, ops=ops), seed=5, threshold=200) for _ in range(2)]
    assert not branches(captured)
    single.profile = True                        # one by one
    for _ in range(3):
        single.run_step()
    assert all(torch.equal(a, b) for a, b in zip(replayed(captured), state(single)))


@pytest.mark.parametrize("count", [2, 11])      # more than there are side streams
@pytest.mark.parametrize("mode", ["thread_local", "global"])
def test_several_steps_in_one_capture(count, mode):
    single, together = [[step("none", 200, None) for _ in range(count)] for _ in range(2)]
    for hp in single:
        hp.profile = True                        # one by one
    for hp in together:
        hp.run_step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode=mode):
        for hp in together:
            hp.run_step()
    for _ in range(3):
        graph.replay()
    for a, b in zip(single, together):
        for _ in range(4):
            a.run_step()
        assert all(torch.equal(x, y) for x, y in zip(state(a), state(b)))


def test_what_does_not_fit_the_communicator_is_still_refused():
    from singa_b200 import _lib
    from singa_b200.communicator import Communicator, NcclIdHolder
    comm = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=64)
    for sync in ("plain", "half"):
        hp = step(sync, 1 << 20, comm)
        for _ in range(4):
            with pytest.raises(_lib.SgbError):
                hp.run_step()
    torch.cuda.synchronize()


@pytest.mark.parametrize("sizes", [[1, 5, 1023, 1024, 1025], [700001, 3], [7] * 100])    # one walk of the tiles, several; a long table
@pytest.mark.parametrize("offset", [0, 1, 2])
@pytest.mark.parametrize("round_f16", [0, 1])
def test_the_narrow_update_has_the_bits_of_the_wide_one(sizes, offset, round_f16):
    import ctypes
    from singa_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(6)
    make = lambda: [torch.randn(n + 4, device="cuda", generator=g)[offset:offset + n] for n in sizes]   # noqa: E731
    p, d, m = make(), make(), make()
    copies = [[t.clone() for t in ts] for ts in (p, d, m)]
    n, stream = len(sizes), torch.cuda.current_stream().cuda_stream
    table = lambda ts: (ctypes.c_void_p * n)(*[t.data_ptr() for t in ts])   # noqa: E731
    counts = (ctypes.c_size_t * n)(*sizes)
    rates = (0.1, 0.9, 0.0, 1e-3, 0, 0.5)
    _lib.call("sgb_sgd_update_beside_f32", table(p), table(d), table(m), counts, n, *rates, round_f16, stream)
    cp, cd, cm = copies
    if round_f16:
        for t in cd:
            t.copy_(t.half().float())
    _lib.call("sgb_sgd_update_multi_f32", table(cp), table(cd), table(cm), counts, n, *rates, stream)
    assert all(torch.equal(a, b) for x, y in ((p, cp), (d, cd), (m, cm)) for a, b in zip(x, y))
