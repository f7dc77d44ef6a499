"""Which joins a batch-norm backward takes into itself: both sides of each line
of the rule, and that a recorded step follows it."""
import pytest

from singa_b200.hot_path import join_pays, merge_calls


@pytest.mark.parametrize("shape, pays", [
    ((1, 2048, 4), True), ((2, 256, 3136), True), ((8, 64, 4096), True), ((8, 64, 4100), False),      # 2^21
    ((5, 8, 64), True), ((5, 8, 68), False), ((32, 8, 16), False), ((33, 8, 16), True),               # 320, 512
    ((64, 256, 64), True), ((1, 256, 4100), False), ((1, 255, 4100), True), ((1, 256, 6144), False),  # 4096 at 2^20
    ((1, 256, 6148), True),                                                                           # 6144
    ((2, 1337, 49), True), ((2, 1338, 49), True), ((2, 2674, 49), True), ((2, 2675, 49), False),      # 2^17, 2^18
    ((1, 1015, 129), True), ((1, 1017, 129), False), ((3, 2048, 25), True), ((4, 512, 625), False)])
def test_lines(shape, pays):
    assert join_pays(*shape) is pays
    n, c, hw = shape
    calls = [("sgb_add_relu_backward_f32", (1, 2, 3, 4, n * c * hw, "STREAM")),
             ("sgb_bn_backward_f32", (10, 4, 11, 12, 13, 14, 15, 16, n, c, hw, 17, 18, "STREAM"))]
    assert (len(merge_calls(calls)) == 1) is pays
