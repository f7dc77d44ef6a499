"""Which batch-norm backward calls take the streaming kernel (host arithmetic):
a recorded step asks, because a captured streaming launch would keep its
counter table.  A channel streams when the x and dy of its N planes do not fit
the shared memory of eight CTAs, 100 KB each, and its planes can be cut."""
import ctypes
import itertools

import pytest

from singa_b200 import _lib


def expected(N, C, HW, mask):
    if HW % 4:
        return 0
    units = N * HW // 4
    if -(-units // 8) * 32 <= 100 * 1024:
        return 0
    return _lib.lib().sgb_bn_backward_stream_plan(N, C, HW, mask, (ctypes.c_int * 6)())


def test_the_query_follows_the_capacity_of_a_cluster():
    lib = _lib.lib()
    shapes = [(32, 64, 112 * 112), (32, 256, 56 * 56), (33, 256, 56 * 56), (1, 3, 102400), (1, 3, 102404), (1, 3, 102432),
              (16, 8, 80 * 80), (17, 8, 80 * 80), (32, 64, 111 * 111), (32, 5000, 12544), (2, 4, 1)]
    shapes += itertools.product((1, 7, 32, 65), (1, 64, 2048), (49, 196, 784, 3136, 12544, 50176))
    for N, C, HW in shapes:
        for mask in (0, 1, 2):
            assert lib.sgb_bn_backward_streams(N, C, HW, mask) == expected(N, C, HW, mask), (N, C, HW, mask)
    assert lib.sgb_bn_backward_streams(32, 64, 112 * 112, 0) == 1
    assert lib.sgb_bn_backward_streams(32, 256, 56 * 56, 0) == 0


@pytest.mark.parametrize("args", [(0, 4, 16, 0), (4, 0, 16, 0), (4, 4, 0, 0), (32, 64, 12544, 3), (32, 64, 12544, -1)])
def test_no_call_no_stream(args):
    assert _lib.lib().sgb_bn_backward_streams(*args) == 0


@pytest.mark.parametrize("shape", [(32, 64, 12544), (9, 64, 12544), (64, 8, 3136), (16, 8, 6400), (65, 64, 3136), (32, 256, 3136)])
def test_a_call_that_visits_its_data_twice_draws_no_table(shape):
    """From 4 million elements on, given the workspace for it; below, the streaming form is what it was."""
    lib = _lib.lib()
    for mask in (0, 1, 2):
        streams = lib.sgb_bn_backward_streams(*shape, mask)
        whole, sums = lib.sgb_bn_backward_workspace_bytes(*shape), 64 * shape[1] * 8
        twice = shape[0] * shape[1] * shape[2] >= 4000000
        assert lib.sgb_bn_backward_draws_table(*shape, mask, min(sums, whole - 1) if twice else sums) == streams
        assert lib.sgb_bn_backward_draws_table(*shape, mask, whole) == (0 if twice else streams)


def test_a_recorded_step_has_room_for_its_largest_call():
    from singa_b200.hot_path import workspace_bytes
    from singa_b200.resnet50_path import build_plan
    plan = build_plan(batch=2, image=64, fused=False)
    assert workspace_bytes(plan) == 8 << 20
    op = next(op for op in plan["ops"] if op.kind == "bn_bwd")
    plan["tensors"][op.args["x"]] = plan["tensors"][op.args["x"]]._replace(shape=(300, 1300, 57, 57))
    need = _lib.lib().sgb_bn_backward_workspace_bytes(300, 1300, 57 * 57)      # 1.27e9 elements of odd planes
    assert workspace_bytes(plan) == need > 8 << 20


@pytest.mark.parametrize("shape, backward, forward", [
    ((79, 20, 50176), True, True), ((80, 20, 50176), False, False), ((1, 4, 4000000), True, True), ((2, 2, 4000000), True, True),
    ((4, 1, 1 << 24), False, False), ((1, 1, 1 << 24), True, True), ((20, 8, 49729), True, True), ((21, 8, 49729), False, True),
    ((53, 8, 49729), False, False), ((1, 8, 1000001), False, True)])
def test_very_large_channels_are_not_visited_twice(shape, backward, forward):
    """Seen in the workspace that is asked for: an entry for each item of 3584 (odd planes: 2304) elements or,
    where only the forward visits twice, of 6144 (3072)."""
    n, c, hw = shape
    whole = _lib.lib().sgb_bn_backward_workspace_bytes(n, c, hw)
    items = lambda vec, odd: 16 * n * c * hw / (odd if hw % 4 else vec)   # noqa: E731
    least = items(3584, 2304) if backward else items(6144, 3072) if forward else 64 * 8 * c
    assert least * 0.99 <= whole <= least * 1.1, (whole, least)
