"""Which plans may update a parameter before the backward pass is over: those of the
models, and none that touches a gradient or a parameter again, reports it twice, in
another order or behind the update, or updates other parameters or not at all."""
import pytest

from singa_b200.hot_path import leaves_what_is_ready
from singa_b200.resnet50_path import Op, add_wgrad_refresh, build_cnn_plan, build_mlp_plan, build_plan, fuse_plan, mask_plan

MODELS = {"mlp": lambda: build_mlp_plan(batch=9, dims=(23, 130, 57, 10)), "cnn": lambda: build_cnn_plan(4, 8),
          "resnet50": lambda: build_plan(batch=2, image=64)}


@pytest.mark.parametrize("model", sorted(MODELS))
@pytest.mark.parametrize("refresh", [None, "start", "each"])
def test_plans_of_the_models(model, refresh):
    for form in (lambda p: p, fuse_plan, lambda p: mask_plan(fuse_plan(p))):
        plan = form(MODELS[model]())
        assert leaves_what_is_ready(add_wgrad_refresh(plan, refresh) if refresh else plan)


def test_other_plans():
    plan = MODELS["mlp"]()
    ops, order = plan["ops"], plan["grad_order"]
    end = next(k for k, op in enumerate(ops) if op.kind == "sync_and_update")
    first = next(k for k, op in enumerate(ops) if op.kind == "grad_ready")
    p = ops[first].args["param"]

    def with_ops(new, **other):
        return leaves_what_is_ready(dict(plan, ops=new, **other))
    assert with_ops(list(ops))
    assert not with_ops(ops[:end] + ops[end + 1:])                                            # no update
    assert not with_ops(ops[:end + 1] + [ops[end]])                                           # two
    assert not with_ops(ops[:first] + ops[first + 1:end + 1] + [ops[first]] + ops[end + 1:])  # ready behind it
    assert not with_ops(ops[:first] + ops[first + 1:])                                        # never ready
    assert not with_ops(ops[:end] + [ops[first]] + ops[end:])                                 # twice
    assert not with_ops([op for op in ops if op.kind != "grad_ready"])
    for kind, args in (("fill", dict(x="d:" + p, value=0.0)), ("scale", dict(x=p, c=2.0)),
                       ("wgrad_refresh", dict(params=(order[-1], p)))):                       # touched again
        assert not with_ops(ops[:end] + [Op(kind, args)] + ops[end:])
        assert with_ops(ops[:first] + [Op(kind, args)] + ops[first:])
    assert not with_ops(list(ops), params=plan["params"][:-1])                                # others are updated
    assert not with_ops(list(ops), grad_order=order[::-1])
