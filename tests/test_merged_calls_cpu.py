"""Which neighbours of a bound call list are merged (host logic only)."""
from singa_b200.hot_path import merge_calls


def test_pairs_merge_only_when_one_feeds_the_other():
    S = "STREAM"
    relu = ("sgb_relu_backward_f32", (1, 2, 3, 12, S))
    rows = ("sgb_sum_rows_f32", (3, 4, 3, 4, 5, 6, S))
    chan = ("sgb_conv_bias_backward_f32", (3, 4, 2, 3, 2, 5, 6, S))
    assert merge_calls([relu, rows]) == [("sgb_relu_backward_sum_rows_f32", (1, 2, 3, 4, 3, 4, 5, 6, S))]
    assert merge_calls([relu, chan]) == [("sgb_relu_backward_conv_bias_f32", (1, 2, 3, 4, 2, 3, 2, 5, 6, S))]
    for other in ([("sgb_relu_backward_f32", (1, 2, 9, 12, S)), rows], [relu, ("grad_ready", "w"), rows],
                  [relu, ("sgb_sum_rows_f32", (3, 4, 3, 3, 5, 6, S))]):
        assert merge_calls(other) == other
    join = ("sgb_add_relu_backward_f32", (1, 2, 3, 4, 24, S))
    bn = ("sgb_bn_backward_f32", (10, 4, 11, 12, 13, 14, 15, 16, 2, 3, 4, 17, 18, S))
    assert merge_calls([join, bn]) == [
        ("sgb_bn_add_relu_backward_f32", (10, 1, 2, 3, 11, 12, 13, 4, 14, 15, 16, 2, 3, 4, 17, 18, S))]
    wide = [("sgb_add_relu_backward_f32", (1, 2, 3, 4, 1 << 24, S)),
            ("sgb_bn_backward_f32", (10, 4, 11, 12, 13, 14, 15, 16, 1 << 10, 1 << 10, 16, 17, 18, S))]
    assert merge_calls(wide) == wide


def test_the_loss_head_becomes_one_call():
    S = "STREAM"
    head = [("sgb_softmax_rows_f32", (1, 2, 8, 10, S)), ("sgb_cross_entropy_f32", (1, 8, 10, 2, 3, 4, S)),
            ("sgb_sum_all_f32", (4, 5, 8, 6, 7, S)), ("sgb_softmax_cross_entropy_bwd_f32", (1, 8, 10, 2, 3, 9, S)),
            ("sgb_scalar_f32", (1, 9, 0.125, 9, 80, S))]
    assert merge_calls(head) == [("sgb_softmax_cross_entropy_fused_f32", (1, 3, 8, 10, 0.125, 2, 4, 9, S)), head[2]]
    other = list(head)
    other[3] = ("sgb_softmax_cross_entropy_bwd_f32", (1, 8, 10, 12, 3, 9, S))    # another tensor's probabilities
    assert merge_calls(other)[:3] == other[:3]


def test_three_calls_become_one():
    S = "STREAM"
    pool = ("sgb_maxpool_backward_f32", (20, 21, 22, 1, 2, 3, 4, 6, 2, 2, 0, 0, 2, 2, S))
    relu = ("sgb_relu_backward_f32", (1, 2, 3, 144, S))
    bias = ("sgb_conv_bias_backward_f32", (3, 4, 2, 3, 24, 5, 6, S))
    assert merge_calls([pool, relu, bias]) == [
        ("sgb_maxpool_relu_backward_conv_bias_f32", (20, 21, 22, 1, 2, 3, 4, 6, 2, 2, 0, 0, 2, 2, 2, 3, 4, 5, 6, S))]
    other = ("sgb_maxpool_backward_f32", (20, 21, 22, 9, 2, 3, 4, 6, 2, 2, 0, 0, 2, 2, S))       # not what the ReLU reads
    assert merge_calls([other, relu, bias])[0] == other
    fused = ("sgb_softmax_cross_entropy_fused_f32", (1, 3, 8, 10, 0.125, 2, 4, 9, S))
    total, rows = ("sgb_sum_all_f32", (4, 5, 8, 6, 7, S)), ("sgb_sum_rows_f32", (9, 11, 8, 10, 6, 7, S))
    assert merge_calls([fused, total, rows]) == [("sgb_loss_head_f32", (1, 3, 8, 10, 0.125, 2, 4, 9, 5, 11, 6, 7, S))]
    for apart in (("sgb_sum_rows_f32", (12, 11, 8, 10, 6, 7, S)), ("sgb_sum_rows_f32", (9, 11, 10, 8, 6, 7, S))):
        assert merge_calls([fused, total, apart]) == [fused, total, apart]


def test_results_over_earlier_operands_stay_apart():
    S = "STREAM"
    pool = lambda x, dy: ("sgb_maxpool_backward_f32", (x, 21, dy, 1, 2, 3, 4, 6, 2, 2, 0, 0, 2, 2, S))   # noqa: E731
    relu, bias = ("sgb_relu_backward_f32", (1, 2, 3, 144, S)), ("sgb_conv_bias_backward_f32", (3, 4, 2, 3, 24, 5, 6, S))
    for first in (pool(3, 22), pool(20, 3), pool(4, 22), pool(20, 4)):     # the ReLU's result, then the sums
        assert merge_calls([first, relu, bias])[0] == first
    over = ("sgb_relu_backward_f32", (1, 2, 1, 144, S)), ("sgb_conv_bias_backward_f32", (1, 4, 2, 3, 24, 5, 6, S))
    assert len(merge_calls([pool(20, 22), *over])) == 1                    # over the pooling's result: element by element
    for over in (1, 2):                                                    # the sums over what the ReLU has read
        for sums in (("sgb_conv_bias_backward_f32", (3, over, 2, 3, 24, 5, 6, S)), ("sgb_sum_rows_f32", (3, over, 6, 24, 5, 6, S))):
            assert merge_calls([relu, sums]) == [relu, sums]
    fused = ("sgb_softmax_cross_entropy_fused_f32", (1, 3, 8, 10, 0.125, 2, 4, 9, S))
    total, rows = ("sgb_sum_all_f32", (4, 5, 8, 6, 7, S)), ("sgb_sum_rows_f32", (9, 11, 8, 10, 6, 7, S))
    for apart in ([fused, total, ("sgb_sum_rows_f32", (9, 4, 8, 10, 6, 7, S))],        # the sums over the losses
                  [fused, ("sgb_sum_all_f32", (4, 4, 8, 6, 7, S)), rows]):             # the total over them
        assert merge_calls(apart) == apart
