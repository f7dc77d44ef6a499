"""What to time before and after a change of this framework: the calls that its users make.

Seven kinds of work, each through public entry points only:

  step    a whole backward + (synchronisation) + update step of one of the three models of this
          repository's benchmark (MLP, small CNN, ResNet-50), run by ``HotPathGPU``, either call by
          call (``run_step``) or as a captured graph
  bn      a convolution layer's BatchNorm + ReLU in training, forward and backward
  pool    max / average pooling, forward and backward
  head    the loss head: softmax, cross entropy, its gradient and the bias gradient
  join    the end of a residual block: add + ReLU forward, ReLU + gradient join backward
  opt     the optimizer over a model's parameter tensors, alone or with the dense gradient exchange
  sparse  the sparsified gradient exchange with residuals, and the update behind it

``listed`` holds the sizes of the repository's own configurations and some ragged ones; ``draw``
spreads the same kinds over their ranges.  Inputs are made on the GPU from the seed.
"""
import math

import torch

from singa_b200 import singa_wrap as sw
from singa_b200.communicator import Communicator, NcclIdHolder
from singa_b200.hot_path import HotPathGPU
from singa_b200.opt import SGD, DistOpt, plan_buckets
from singa_b200.resnet50_path import (add_wgrad_refresh, algorithmic_bytes, build_cnn_plan, build_mlp_plan,
                                      build_plan, fuse_plan, numel)

F32, F16 = torch.float32, torch.float16
HALF = {"f32": F32, "f16": F16}


def listed():
    return [
        # MLP 784-4096-4096-10 at batch 256, call by call: few kernels, the host has to keep up
        dict(name="mlp_step", kind="step", model="mlp", batch=256, size=4096, fused=True, graph=False, sync="none"),
        # small CNN at batch 64 in the reference's call order: the smallest kernels of all
        dict(name="cnn_step", kind="step", model="cnn", batch=64, size=32, fused=False, graph=False, sync="none"),
        # ResNet-50, batch 32 a GPU, 224 x 224, data parallel, replayed as one graph: the headline workload
        dict(name="resnet50_step_graph", kind="step", model="resnet50", batch=32, size=224, fused=True, graph=True,
             sync="plain"),
        # ResNet-50 on a ragged small batch of smaller images, call by call (planes of 80, 40, 20, 10, 5)
        dict(name="resnet50_step_ragged", kind="step", model="resnet50", batch=3, size=160, fused=True, graph=False,
             sync="none"),
        # the largest BatchNorm layers of ResNet-50
        dict(name="bn_256x56x56", kind="bn", n=32, c=256, h=56, w=56, fused=True),
        # a layer whose planes have an odd size, each call on its own
        dict(name="bn_odd", kind="bn", n=17, c=48, h=35, w=29, fused=False),
        # the max pool of ResNet-50's stem
        dict(name="maxpool_stem", kind="pool", n=32, c=64, h=112, w=112, k=3, s=2, p=1, max=True, record=False),
        # a classifier's loss head: 256 samples of 1000 classes, six small calls
        dict(name="loss_head", kind="head", batch=256, classes=1000, dtype="f32", fused=False),
        # half-precision activations at a residual join
        dict(name="join_f16", kind="join", n=32, c=512, h=28, w=28, dtype="f16"),
        # 161 parameter tensors, gradients exchanged in half precision, SGD with momentum
        dict(name="opt_half_resnet50", kind="opt", model="resnet50", size=64, mode="half", threshold=2097152),
        # the sparse exchange's benchmark: a flat gradient of 1e8 elements, the largest 1 % of it
        dict(name="sparse_topk_1e8", kind="sparse", model="flat", size=100_000_000, topk=True, spars=0.01,
             key="magnitude", threshold=2097152),
        # the same exchange by threshold over ResNet-50's gradients, bucket by bucket
        dict(name="sparse_threshold_resnet50", kind="sparse", model="resnet50", size=64, topk=False, spars=2e-3,
             key="compat", threshold=2097152),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "bn", "bn", "pool", "head", "join", "opt", "sparse", "sparse"])
    if kind == "step":
        model = rng.choice(["mlp", "cnn", "resnet50"])
        case = dict(kind=kind, model=model, fused=rng.random() < 0.7, graph=rng.random() < 0.4,
                    sync=rng.choice(["none", "none", "plain", "half"]))
        if model == "mlp":
            case.update(batch=_log(rng, 1, 1024), size=_log(rng, 128, 4096))
        elif model == "cnn":
            case.update(batch=_log(rng, 4, 512), size=rng.randint(8, 64))
        else:
            case.update(batch=_log(rng, 1, 24), size=rng.randint(64, 224))
        return case
    if kind == "bn":
        h = _log(rng, 4, 112)
        w = h if rng.random() < 0.6 else _log(rng, 4, 112)
        n, c = _log(rng, 2, 64), _log(rng, 8, 2048)
        while n * c * h * w > 26_000_000:
            n, c = (n + 1) // 2, (c + 1) // 2
        return dict(kind=kind, n=n, c=c, h=h, w=w, fused=rng.random() < 0.5)
    if kind == "pool":
        k, s, p, mx = rng.choice([(3, 2, 1, True), (3, 2, 1, True), (2, 2, 0, True), (3, 1, 1, True),
                                  (2, 2, 0, False), (3, 2, 1, False), (0, 1, 0, False)])   # 0: the whole plane
        h = _log(rng, 6, 112)
        w = h if rng.random() < 0.6 else _log(rng, 6, 112)
        n, c = _log(rng, 2, 64), _log(rng, 8, 512)
        while n * c * h * w > 26_000_000:
            n, c = (n + 1) // 2, (c + 1) // 2
        return dict(kind=kind, n=n, c=c, h=h, w=w, k=k, s=s, p=p, max=mx, record=mx and rng.random() < 0.3)
    if kind == "head":
        batch, classes = _log(rng, 4, 4096), _log(rng, 10, 32000)
        while batch * classes > 16_000_000:
            batch //= 2
        dtype = "f32" if rng.random() < 0.7 else "f16"
        return dict(kind=kind, batch=batch, classes=classes, dtype=dtype,
                    fused=dtype == "f32" and rng.random() < 0.4)
    if kind == "join":
        n, c, h, w = _log(rng, 1, 64), _log(rng, 16, 1024), _log(rng, 4, 112), _log(rng, 4, 112)
        while n * c * h * w > 26_000_000:
            n, c = (n + 1) // 2, (c + 1) // 2
        return dict(kind=kind, n=n, c=c, h=h, w=w, dtype=rng.choice(["f32", "f16"]))
    if kind == "opt":
        model = rng.choice(["mlp", "cnn", "resnet50"])
        size = {"mlp": _log(rng, 128, 4096), "cnn": rng.randint(8, 64), "resnet50": 64}[model]
        return dict(kind=kind, model=model, size=size, mode=rng.choice(["sgd", "plain", "half"]),
                    threshold=_log(rng, 100_000, 2_097_152))
    model = rng.choice(["flat", "flat", "resnet50", "mlp"])
    size = {"flat": _log(rng, 100_000, 100_000_000), "resnet50": 64, "mlp": _log(rng, 128, 4096)}[model]
    topk = rng.random() < 0.5
    return dict(kind=kind, model=model, size=size, topk=topk,
                spars=math.exp(rng.uniform(math.log(1e-3), math.log(5e-2))) if topk else rng.uniform(1.5e-3, 4e-3),
                key=rng.choice(["compat", "magnitude"]), threshold=_log(rng, 200_000, 2_097_152))


# ------------------------------------------------------------------------------ preparation
_COMMS = {}


def _communicator(elems):
    """A program creates its communicator once; it is sized for the largest bucket it will see."""
    size = 1 << 23 if elems <= 1 << 23 else 1 << 25 if elems <= 1 << 25 else 1 << 27
    if size not in _COMMS:
        _COMMS[size] = Communicator(torch.cuda.current_device(), 1, NcclIdHolder(), buffSize=size)
    return _COMMS[size]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, *shape, std=1.0, mean=0.0, dtype=F32):
    t = torch.randn(shape, generator=g, device="cuda").mul_(std)
    if mean:
        t.add_(mean)
    return t if dtype == F32 else t.to(dtype)


def _plan(model, batch, size, fused):
    if model == "mlp":
        plan = build_mlp_plan(batch=batch, dims=(784, size, size, 10))
    elif model == "cnn":
        plan = build_cnn_plan(batch=batch, channels=size)
    else:
        plan = build_plan(batch=batch, image=size, fused=False)
    return fuse_plan(plan) if fused else plan


def _grad_sizes(case):
    """Sizes of a model's gradients in the order in which backward produces them."""
    if case["model"] == "flat":
        return [case["size"]]
    plan = _plan(case["model"], 1, case["size"], False)
    return [numel(plan["tensors"][p].shape) for p in plan["grad_order"]]


def _step_plan(case):
    plan = _plan(case["model"], case["batch"], case["size"], case["fused"])
    # in data-parallel runs every weight gradient is written anew in each step, as its contraction would do
    return add_wgrad_refresh(plan) if case["sync"] != "none" else plan


def _prepare_step(case, seed):
    comm = _communicator(max(1, *_grad_sizes(case))) if case["sync"] != "none" else None
    hp = HotPathGPU(_step_plan(case), communicator=comm, world=1, seed=seed, lr=0.005, momentum=0.9,
                    weight_decay=1e-5, dist_option=case["sync"] if comm is not None else "plain")
    if case["graph"]:
        hp.run_step()
        torch.cuda.synchronize()
        hp.capture()
    t = hp.t
    if case["model"] == "resnet50":      # parameters: the 54 weight matrices (the 107 vectors' gradients are in the arena)
        outs = [t[p] for p in hp.plan["params"] if t[p].dim() > 1] + [t["maxpool.dx"], t["bn1.dx"]]
    else:
        outs = [t[p] for p in hp.plan["params"]] + [t[n] for n, s in hp.plan["tensors"].items() if s.kind == "grad"]
    return dict(hp=hp, outs=[hp.grad_arena, t["loss"], t["prob"]] + outs)


def _run_step(s):
    if s["hp"].graph is not None:
        s["hp"].graph.replay()
    else:
        s["hp"].run_step()
    return s["outs"]


def _prepare_bn(case, seed):
    g, c = _gen(seed), case["c"]
    shape = (case["n"], c, case["h"], case["w"])
    x = _randn(g, *shape, std=1.5, mean=0.2)
    return dict(x=x, dy=_randn(g, *shape, std=1e-2), handle=sw.CudnnBatchNormHandle(0.1, x), fused=case["fused"],
                scale=torch.rand(c, generator=g, device="cuda") + 0.5, bias=_randn(g, c, std=0.1),
                rm=torch.zeros(c, device="cuda"), rv=torch.ones(c, device="cuda"))


def _run_bn(s):
    h, x, dy = s["handle"], s["x"], s["dy"]
    y, mean, invstd = sw.GpuBatchNormForwardTraining(h, x, s["scale"], s["bias"], s["rm"], s["rv"], 1e-5)
    r = sw.ReLU(y)
    if s["fused"]:
        dx, ds, db = sw.GpuBatchNormReLUBackward(h, dy, y, x, s["scale"], mean, invstd)
    else:
        dx, ds, db = sw.GpuBatchNormBackward(h, sw.ReLUBackward(dy, y), x, s["scale"], mean, invstd)
    return [r, mean, invstd, s["rm"], s["rv"], dx, ds, db]


def _pool_geometry(case):
    k = (case["k"], case["k"]) if case["k"] else (case["h"], case["w"])
    return k, (case["s"], case["s"]), (case["p"], case["p"])


def _prepare_pool(case, seed):
    g = _gen(seed)
    x = _randn(g, case["n"], case["c"], case["h"], case["w"]).relu_()       # pooling follows a ReLU
    handle = sw.CudnnPoolingHandle(x, *_pool_geometry(case), is_max=case["max"])
    dy = _randn(g, case["n"], case["c"], handle.pooled_height, handle.pooled_width, std=1e-2)
    return dict(x=x, dy=dy, handle=handle, record=case["record"])


def _run_pool(s):
    h, x, dy = s["handle"], s["x"], s["dy"]
    if s["record"]:
        y, arg = sw.GpuPoolingForwardArgmax(h, x)
        return [y, arg, sw.GpuPoolingBackwardArgmax(h, dy, arg)]
    y = sw.GpuPoolingForward(h, x)
    return [y, sw.GpuPoolingBackward(h, dy, x, y)]


def _prepare_head(case, seed):
    g, dt = _gen(seed), HALF[case["dtype"]]
    return dict(x=_randn(g, case["batch"], case["classes"], dtype=dt), fused=case["fused"],
                t=torch.randint(0, case["classes"], (case["batch"],), generator=g, device="cuda", dtype=torch.int32))


def _run_head(s):
    x, t = s["x"], s["t"]
    batch = x.shape[0]
    if s["fused"]:
        p, loss, g = sw.SoftMaxCrossEntropyFused(x, t, 1.0 / batch)
        return [p, loss, sw.SumAll(loss), g, sw.SumRows(g)]
    p = sw.SoftMax(x)
    loss = sw.CrossEntropyFwd(p, t)
    g = sw.SoftmaxCrossEntropyBwd(p, t)
    sw.DivFloatWithRet(g, batch, g)
    if x.dtype == F16:
        return [p, loss, g]
    return [p, loss, sw.SumAll(loss), g, sw.SumRows(g)]


def _prepare_join(case, seed):
    g, dt = _gen(seed), HALF[case["dtype"]]
    shape = (case["n"], case["c"], case["h"], case["w"])
    return dict(a=_randn(g, *shape, dtype=dt), b=_randn(g, *shape, dtype=dt), dy=_randn(g, *shape, std=1e-2, dtype=dt),
                other=_randn(g, *shape, std=1e-2, dtype=dt))


def _run_join(s):
    t = sw.binary("add", s["a"], s["b"])
    y = sw.ReLU(t)
    dx = sw.ReLUBackward(s["dy"], t)
    return [t, y, dx, sw.binary("add", dx, s["other"])]


class _Pool(object):
    """Tensors as an allocator hands them out: 512-byte blocks of one buffer, forward order."""

    def __init__(self, g, sizes, std):
        starts, off = [], 0
        for n in sizes:
            starts.append(off)
            off += -(-n // 128) * 128
        self.flat = _randn(g, off, std=std) if std else torch.zeros(off, device="cuda")
        self.tensors = [self.flat[o:o + n] for o, n in zip(starts, sizes)]


def _optimizer(case, seed):
    """(name, param, grad) triples in backward order, and the SGD object with the momentum of earlier steps."""
    g, sizes = _gen(seed), _grad_sizes(case)
    params, grads, moments = (_Pool(g, sizes[::-1], std) for std in (0.05, 1e-3, 1e-3))
    names = ["p%d" % i for i in range(len(sizes))]
    opt = SGD(lr=0.005, momentum=0.9, weight_decay=1e-5)
    for n, m in zip(names, moments.tensors[::-1]):
        opt.moments[n] = m
    triples = list(zip(names, params.tensors[::-1], grads.tensors[::-1]))
    return opt, triples, [params.flat, grads.flat, moments.flat]


def _prepare_opt(case, seed):
    opt, triples, outs = _optimizer(case, seed)
    if case["mode"] != "sgd":
        opt = DistOpt(opt, communicator=_communicator(max(n.numel() for _, n, _ in triples)))
    return dict(opt=opt, triples=triples, outs=outs, mode=case["mode"], threshold=case["threshold"])


def _run_opt(s):
    opt, triples = s["opt"], s["triples"]
    if s["mode"] == "sgd":
        opt.apply_many(*zip(*triples))
        opt.step()
    elif s["mode"] == "plain":
        opt.backward_and_update(iter(triples), threshold=s["threshold"])
    else:
        opt.backward_and_update_half(iter(triples), threshold=s["threshold"])
    return s["outs"]


def _prepare_sparse(case, seed):
    opt, triples, outs = _optimizer(case, seed)
    comm = _communicator(max(n.numel() for _, n, _ in triples))
    comm.set_topk_mode(case["key"])
    return dict(opt=DistOpt(opt, communicator=comm), triples=triples, outs=outs, case=case)


def _run_sparse(s):
    opt, case = s["opt"], s["case"]
    opt.backward_and_sparse_update(iter(s["triples"]), threshold=case["threshold"], spars=case["spars"],
                                   topK=case["topk"])
    return s["outs"] + opt.gradAccumulation


_PREPARE = dict(step=_prepare_step, bn=_prepare_bn, pool=_prepare_pool, head=_prepare_head, join=_prepare_join,
                opt=_prepare_opt, sparse=_prepare_sparse)
_RUN = dict(step=_run_step, bn=_run_bn, pool=_run_pool, head=_run_head, join=_run_join, opt=_run_opt,
            sparse=_run_sparse)


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    state["run"] = _RUN[case["kind"]]
    return state


def run(state):
    return state["run"](state)


# --------------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes and operations of one pass: every call of it reads its inputs once and writes its outputs once."""
    kind = case["kind"]
    if kind == "step":
        plan = _step_plan(case)
        by_family, nparam = algorithmic_bytes(plan)
        return dict(bytes=sum(by_family.values()), flops=6 * nparam)
    if kind in ("bn", "join"):
        n = case["n"] * case["c"] * case["h"] * case["w"]
        if kind == "join":           # add 3, ReLU 2, ReLU backward 3, join 3 elements
            return dict(bytes=11 * n * (4 if case["dtype"] == "f32" else 2), flops=4 * n)
        # forward 2, ReLU 2, backward 4 (fused) or 3 + 3 elements
        return dict(bytes=4 * n * (8 if case["fused"] else 10) + 60 * case["c"], flops=20 * n)
    if kind == "pool":
        (kh, kw), (sh, sw_), (ph, pw) = _pool_geometry(case)
        x = case["n"] * case["c"] * case["h"] * case["w"]
        y = case["n"] * case["c"] * ((case["h"] + 2 * ph - kh) // sh + 1) * ((case["w"] + 2 * pw - kw) // sw_ + 1)
        if case["record"]:           # x -> y, record; dy, record -> dx
            return dict(bytes=4 * (2 * x + 2 * y) + 2 * y, flops=2 * y * kh * kw)
        # x -> y; x, dy -> dx (the average needs no x)
        return dict(bytes=4 * ((3 if case["max"] else 2) * x + 2 * y), flops=2 * y * kh * kw)
    if kind == "head":
        n, e = case["batch"] * case["classes"], 4 if case["dtype"] == "f32" else 2
        if case["fused"]:            # logits -> probabilities, gradient; column sums
            return dict(bytes=4 * n * e + 16 * case["batch"], flops=8 * n)
        # softmax 2, gradient 2, division 2, column sums 1
        return dict(bytes=(7 if e == 4 else 6) * n * e + 16 * case["batch"], flops=8 * n)
    sizes = _grad_sizes(case)
    n = sum(sizes)
    if kind == "opt":                # update 5 elements; exchange: read and write each gradient once
        return dict(bytes=4 * n * (5 if case["mode"] == "sgd" else 7), flops=6 * n)
    # gradient and residual in, residual and dense result out, then the update
    return dict(bytes=4 * n * (4 + 5), flops=8 * n)


def tolerance(case):
    kind = case["kind"]
    if kind == "join":
        return "exact"               # one correctly rounded operation an element
    if kind in ("sparse", "opt"):
        return {"rel": 5e-4, "max": 2e-3} if case.get("mode") == "half" else {"rel": 1e-6}
    if kind == "pool":
        return {"rel": 1e-6 if case["max"] else 1e-5, "differ": 0.0}
    if kind == "head" and case["dtype"] == "f16":
        return {"rel": 1e-3, "max": 4e-3}
    if kind == "step" and case["sync"] == "half":
        return {"rel": 5e-4, "max": 2e-3}
    return {"rel": 1e-5}
