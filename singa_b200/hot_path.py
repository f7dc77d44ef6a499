"""GPU executor of a hot-path plan (see ``resnet50_path.build_plan``).

Owns the device tensors (torch is the allocator), turns every op into one
pre-bound C-ABI call, replays DistOpt's bucket policy on the communicator as
gradients become ready, and finishes with the fused multi-tensor SGD update.
The calls of a step are recorded once as a native program; ``run_step`` is one
call that issues them in order (2 us a call instead of 5: the arguments are
already converted, and no interpreter runs between two launches), or, for steps
of small kernels repeated with the same hyper-parameters, launches them as one
graph that it has captured itself.
The whole step can be captured once into a CUDA graph and replayed, which is
this implementation's counterpart of the reference's buffered-operation graph
(``Device::EnableGraph`` / ``RunGraph``).
"""
import ctypes as C

import numpy as np
import torch

from . import _lib
from .opt import plan_buckets
from .resnet50_path import numel


def _table(tensors):
    n = len(tensors)
    return ((C.c_void_p * n)(*[t.data_ptr() for t in tensors]),
            (C.c_size_t * n)(*[t.numel() for t in tensors]), n)


def join_pays(n, c, hw):
    """Whether a batch-norm backward takes the join in front of it into itself:
    where both are short, one launch and one latency less is worth more than
    what the streaming join does better.  The lines follow whole ResNet-50 steps
    (us with all such joins apart -> merged, three captures of each):

      up to 2^21 elements, as a rule: 1x224^2 285.7 -> 275, 4x224^2 400.5 -> 395.3,
        2x256x56x56 alone 355.4 -> 347.6; beyond, where a cluster shares a
        channel: 8x512x28x28 585.8 -> 597.8, 16x512x20x20 595.7 -> 606.0;
      not where a warp holds a channel in nearly all of its four vectors
        (32x1024x4x4 386.2 -> 390.7, 24x1024x4x4 342.3 -> 344.2) nor, above 2^20,
        where a thread holds more than four (24x256x16x16 344 -> 350,
        8x256x24x24 317.5 -> 321.6, 3x256x40x40 317.3 -> 322.5);
      planes that are no multiple of four, one float an access: up to 2^17
        elements, or 2^18 where a channel has no more than 128 (3x2048x5x5
        319.6 -> 317.9, 1x2048x7x7 285.7 -> 283.3; but 4x512x25x25 423 -> 451,
        10x1024x13x13 649 -> 669, 3x1024x7x7 271.1 -> 273.1)."""
    channel, elements = n * hw, n * c * hw
    if hw % 4:
        return elements <= 1 << 17 or (elements <= 1 << 18 and channel <= 128)
    if 320 < channel <= 512 or (4096 < channel <= 6144 and elements > 1 << 20):
        return False
    return elements <= 1 << 21


def merge_calls(calls):
    """The bound calls with neighbours merged that one kernel does together.
    Every tensor that the separate calls write is written, with the same bits.  Calls
    stay apart where one writes over what an earlier one has read (its operands are
    not needed any more by then, but one kernel still reads them):

      add_relu_backward(-> t) ; bn_backward(dy=t)       =>  bn_add_relu_backward
      relu_backward(-> t) ; sum_rows(t)                 =>  relu_backward_sum_rows
      relu_backward(-> t) ; conv_bias_backward(t)       =>  relu_backward_conv_bias
      cross_entropy_bwd(-> g) ; g *= c                  =>  cross_entropy_grad
      maxpool_backward(-> s) ; relu_backward(s -> t) ; conv_bias_backward(t)
                                                        =>  maxpool_relu_backward_conv_bias
      softmax(-> p) ; cross_entropy(p -> l) ; sum of l ; cross_entropy_grad(p)
                                                        =>  softmax_cross_entropy_fused ; sum of l
      softmax_cross_entropy_fused(-> l, g) ; sum of l ; sum_rows(g)
                                                        =>  loss_head
    """
    out = []
    for name, a in calls:
        last, b = out[-1] if out else ("", None)
        if name == "sgb_bn_backward_f32" and last == "sgb_add_relu_backward_f32" and a[1] == b[3] and \
                b[4] == a[8] * a[9] * a[10] and join_pays(*a[8:11]):
            out[-1] = ("sgb_bn_add_relu_backward_f32", (a[0],) + b[:3] + a[2:5] + (a[1],) + a[5:])
        elif name == "sgb_sum_rows_f32" and last == "sgb_relu_backward_f32" and a[0] == b[2] and \
                b[3] == a[2] * a[3] and a[1] not in b[:2]:
            out[-1] = ("sgb_relu_backward_sum_rows_f32", b[:3] + a[1:])
        elif name == "sgb_conv_bias_backward_f32" and last == "sgb_relu_backward_f32" and a[0] == b[2] and \
                b[3] == a[2] * a[3] * a[4] and a[1] not in b[:2]:
            out[-1] = ("sgb_relu_backward_conv_bias_f32", b[:3] + a[1:])
            before, p = out[-2] if len(out) > 1 else ("", None)
            # (pooling: x, y, dy, dx, n, c, h, w, windows, S; the pair: dy, x, dx, db, n, c, hw, ws, ws bytes, S)
            if before == "sgb_maxpool_backward_f32" and p[3] == b[0] and p[4:6] == a[2:4] and p[6] * p[7] == a[4] and \
                    not {b[2], a[1]} & {p[0], p[2]}:
                out[-2:] = [("sgb_maxpool_relu_backward_conv_bias_f32", p[:-1] + b[1:3] + a[1:2] + a[5:])]
        elif name == "sgb_scalar_f32" and last == "sgb_softmax_cross_entropy_bwd_f32" and a[0] == 1 and \
                a[1] == a[3] == b[5] and a[4] == b[1] * b[2]:
            out[-1] = ("sgb_softmax_cross_entropy_grad_f32", b[:5] + (a[2],) + b[5:])
        else:
            out.append((name, a))
        # (softmax: x, p, rows, columns; forward: 1, rows, columns, p, t, l; sum: l, ...; gradient: 1, rows, columns, p, t, c, g)
        if [n for n, _ in out[-4:]] == ["sgb_softmax_rows_f32", "sgb_cross_entropy_f32", "sgb_sum_all_f32",
                                        "sgb_softmax_cross_entropy_grad_f32"]:
            (_, sm), (_, fwd), total, (_, grd) = out[-4:]
            if fwd[:5] == grd[:5] == (1,) + sm[2:4] + (sm[1], fwd[4]) and total[1][0] == fwd[5] and grd[6] != sm[0]:
                out[-4:] = [("sgb_softmax_cross_entropy_fused_f32",
                             (sm[0], fwd[4]) + sm[2:4] + (grd[5], sm[1], fwd[5], grd[6]) + sm[4:]), total]
        # (fused: x, t, rows, columns, scale, p, l, g, S; sum: l, out, n, ws, ws bytes, S; rows: g, v, rows, columns, ...)
        if [n for n, _ in out[-3:]] == ["sgb_softmax_cross_entropy_fused_f32", "sgb_sum_all_f32", "sgb_sum_rows_f32"]:
            (_, f), (_, total), (_, rows) = out[-3:]
            if total[0] == f[6] and total[2] == f[2] and rows[0] == f[7] and rows[2:4] == f[2:4] and \
                    total[3:5] == rows[4:6] and total[1] not in (f[6], f[7]) and rows[1] not in (f[6], f[7]):
                out[-3:] = [("sgb_loss_head_f32", f[:8] + total[1:2] + rows[1:2] + rows[4:])]
    return out


def workspace_bytes(plan):
    """What the plan's calls need of workspace, each for itself; 8 MiB serve all sums
    and batch norms of up to 10^9 elements."""
    need = [8 << 20]
    for op in plan["ops"]:
        if op.kind in ("bn_bwd", "bn_relu_bwd", "bn_relu_mask_bwd", "bn_add_relu_bwd"):
            n, c, h, w = plan["tensors"][op.args["x"]].shape
            need.append(_lib.lib().sgb_bn_backward_workspace_bytes(n, c, h * w))
    return max(need)


def leaves_what_is_ready(plan):
    """Whether the parameters can be updated before the pass is over, with the results of
    one update at its end: each gradient is reported ready once, in the order of the
    buckets, no op behind that touches it or its parameter, and the one update comes
    behind all of them and is of them all."""
    order, done = list(plan["grad_order"]), set()
    ready = [op.args["param"] for op in plan["ops"] if op.kind == "grad_ready"]
    if ready != order or sorted(order) != sorted(plan["params"]) or \
            sum(op.kind == "sync_and_update" for op in plan["ops"]) != 1:
        return False
    for op in plan["ops"]:
        if op.kind == "sync_and_update":
            break
        if op.kind == "grad_ready":
            done |= {op.args["param"], "d:" + op.args["param"]}
            continue
        for value in op.args.values():
            names = value if isinstance(value, (tuple, list)) else (value,)
            if any(isinstance(name, str) and name in done for name in names):
                return False
    return len(done) == 2 * len(order)


def _recorded(name, *with_it):
    """An attribute that the recorded program of a step holds (the communicator by
    its address): setting it has the program recorded anew at the next run.  Setting it
    sets those `with_it` to the same truth value."""
    def read(self):
        return getattr(self, "_" + name)

    def write(self, value):
        setattr(self, "_" + name, value)
        for other in with_it:
            setattr(self, other, bool(value))
        self._program = None
    return property(read, write)


# When a recorded call is issued: in every run, in timed ones, in runs into a capture, in
# those that are not.
_ALWAYS, _PROFILED, _CAPTURED, _SINGLE = range(4)


class HotPathGPU(object):
    comm, world, dist_option = _recorded("comm"), _recorded("world"), _recorded("dist_option")
    # _branch: without a communicator nothing arrives, but a captured step may update its
    # buckets before the pass is over, unless it was asked not to.
    spars, update_on_arrival = _recorded("spars"), _recorded("update_on_arrival", "_branch")

    def __init__(self, plan, communicator=None, world=1, seed=0, lr=0.1, momentum=0.9,
                 weight_decay=1e-5, threshold=2097152, dist_option="plain", spars=0.05,
                 device=None, update_on_arrival=True, pool_argmax=False):
        self.plan, self.comm, self.world = plan, communicator, world
        self.lr, self.momentum, self.weight_decay = lr, momentum, weight_decay
        self.threshold, self.dist_option, self.spars = threshold, dist_option, spars
        # With a communicator, every bucket's parameters are updated on the
        # communicator's side stream as soon as that bucket's reduced gradients
        # have landed, overlapped with the rest of the backward pass (same
        # results as updating everything after the final wait).
        self.update_on_arrival = bool(update_on_arrival) and communicator is not None \
            and dist_option in ("plain", "half")
        self._branch = bool(update_on_arrival)
        # pool_argmax: max-pool backward consumes the arg-max record of the forward
        # partner (produced once at set-up: the forward pass is outside this path)
        # instead of recomputing the winners from x and y.  Same dx bit for bit.
        self.pool_argmax = bool(pool_argmax)
        self.device = torch.device("cuda", torch.cuda.current_device()) if device is None else device
        self.lib = _lib.lib()
        self.t = {}
        self._alloc(seed)
        self._bind()
        self.graph = None
        self.launches_per_step = None
        self.profile = False      # True: mark "bucket_ready" on the compute stream (communicator timing on)

    # ------------------------------------------------------------------ tensors
    def _alloc(self, seed):
        gen = torch.Generator(device=self.device)
        gen.manual_seed(seed)
        T, dev = self.plan["tensors"], self.device

        def randn(shape, std=1.0, mean=0.0):
            return torch.randn(shape, generator=gen, device=dev) * std + mean

        # Parameter gradients live back to back, in the order they are produced,
        # in one arena: every bucket of the synchronisation policy is then a
        # contiguous slice and is all-reduced in place (no pack / unpack pass).
        names = self.plan["grad_order"]
        sizes = [numel(T["d:" + n].shape) for n in names]
        order = [names[i] for _, idx in plan_buckets(sizes, self.threshold) for i in idx]   # bucket by bucket
        total = sum(sizes)
        self.grad_arena = torch.empty(total, device=dev)
        arena_view, off = {}, 0
        for n in order:
            cnt = numel(T["d:" + n].shape)
            arena_view["d:" + n] = self.grad_arena[off:off + cnt].view(T["d:" + n].shape)
            off += cnt
        self.t["grad_arena"] = self.grad_arena
        # pristine stand-ins of the contractions' weight gradients, back to back in
        # refresh order (one flat buffer: a refresh is one multi-tensor copy)
        wsyn = [n for n, spec in T.items() if spec.kind == "wsyn"]
        self.wsyn_flat = torch.empty(sum(numel(T[n].shape) for n in wsyn), device=dev)
        self.wsyn_off, off = {}, 0
        for n in wsyn:
            cnt = numel(T[n].shape)
            self.wsyn_off[n] = off
            self.t[n] = self.wsyn_flat[off:off + cnt].view(T[n].shape)
            self.t[n].copy_(randn(T[n].shape, 1e-3))
            off += cnt
        for name, spec in T.items():
            k = spec.kind
            if k in ("wsyn", "mask"):
                continue
            if k == "pgrad" and name in arena_view:
                self.t[name] = arena_view[name]
                self.t[name].copy_(randn(spec.shape, 1e-3))
                continue
            if k == "label":
                self.t[name] = torch.randint(0, T["logits"].shape[1], spec.shape, generator=gen,
                                             device=dev, dtype=torch.int32)
            elif k == "act":
                self.t[name] = randn(spec.shape, 1.5, 0.2) if name.endswith(".x") and ".bn" in name or name == "bn1.x" \
                    else randn(spec.shape)
            elif k == "syn":
                self.t[name] = randn(spec.shape, 1e-2)
            elif k == "param":
                if name.endswith(".scale"):
                    self.t[name] = torch.ones(spec.shape, device=dev)
                elif name.endswith(".bias") or name == "fc.b":
                    self.t[name] = torch.zeros(spec.shape, device=dev)
                else:
                    self.t[name] = randn(spec.shape, 0.05)
            elif k == "pgrad":
                self.t[name] = randn(spec.shape, 1e-3)
            else:
                self.t[name] = torch.zeros(spec.shape, device=dev)
        # forward-consistent statistics and ReLU inputs (set-up only, not timed)
        for name in list(T):
            if name.endswith(".mean"):
                base = name[:-5]
                x = self.t[base + ".x"]
                var, mean = torch.var_mean(x, dim=(0, 2, 3), unbiased=False)
                self.t[base + ".mean"].copy_(mean)
                self.t[base + ".invstd"].copy_(torch.rsqrt(var))
                relu_name = {"bn1": "relu.x"}.get(base, base.replace(".bn", ".relu") + ".x")
                if relu_name in self.t and ".down" not in base and not base.endswith("bn3"):
                    s = self.t[base + ".scale"].view(1, -1, 1, 1)
                    b = self.t[base + ".bias"].view(1, -1, 1, 1)
                    self.t[relu_name].copy_((x - mean.view(1, -1, 1, 1)) * torch.rsqrt(var).view(1, -1, 1, 1) * s + b)
        if "maxpool.x" in self.t:
            self.t["maxpool.x"].copy_(torch.relu(self.t["relu.x"]))
            self.t["maxpool.y"].copy_(torch.nn.functional.max_pool2d(self.t["maxpool.x"], 3, 2, 1))
        for op in self.plan["ops"]:        # other max-pool layers: post-ReLU input, consistent output
            if op.kind == "maxpool_bwd" and op.args["x"] != "maxpool.x":
                a = op.args
                self.t[a["x"]].copy_(torch.relu(self.t[a["x"]]))
                self.t[a["y"]].copy_(torch.nn.functional.max_pool2d(self.t[a["x"]], a["kernel"], a["stride"], a["pad"]))
        # bit records of the ReLU forward partner (produced once at set-up: the
        # forward pass is outside this path), from the stored ReLU inputs
        for name, spec in T.items():
            if spec.kind != "mask":
                continue
            src = self.t[name[len("mask:"):]]
            n = src.numel()
            rec = torch.zeros(self.lib.sgb_relu_mask_bytes(n), dtype=torch.uint8, device=dev)
            y = torch.empty_like(src)
            _lib.call("sgb_relu_forward_mask_f32", src.data_ptr(), y.data_ptr(), rec.data_ptr(), n,
                      torch.cuda.current_stream().cuda_stream)
            self.t[name] = rec
        self.moments = {p: torch.zeros_like(self.t[p]) for p in self.plan["params"]}
        self.ws = torch.empty(workspace_bytes(self.plan), dtype=torch.uint8, device=dev)
        torch.cuda.synchronize()

    def host_copy(self):
        """numpy copies of every tensor + moments (inputs for the oracle)."""
        out = {k: v.detach().cpu().numpy().copy() for k, v in self.t.items() if k != "grad_arena"}
        out.update({"m:" + k: v.detach().cpu().numpy().copy() for k, v in self.moments.items()})
        return out

    # -------------------------------------------------------------------- bind
    def _bind(self):
        """One (function name, argument tuple) per op; ``None`` stream slots are
        filled at run time with the current stream."""
        t, ws, L = self.t, self.ws, self.lib
        self.calls = []
        S = "STREAM"

        def p(name):
            return t[name].data_ptr()

        def geom(x, kernel, stride, pad):
            n, c, h, w = t[x].shape
            return (n, c, h, w, kernel[0], kernel[1], pad[0], pad[1], stride[0], stride[1])

        for op in self.plan["ops"]:
            a, k = op.args, op.kind
            if k == "relu_bwd":
                self.calls.append(("sgb_relu_backward_f32", (p(a["dy"]), p(a["x"]), p(a["dx"]), t[a["x"]].numel(), S)))
            elif k == "relu_mask_bwd":
                self.calls.append(("sgb_relu_backward_mask_f32", (p(a["dy"]), p(a["x"]), p(a["dx"]), t[a["dx"]].numel(), S)))
            elif k == "add_relu_mask_bwd":
                self.calls.append(("sgb_add_relu_backward_mask_f32",
                                   (p(a["dy_a"]), p(a["dy_b"]), p(a["x"]), p(a["dx"]), t[a["dx"]].numel(), S)))
            elif k == "add_relu_bwd":
                self.calls.append(("sgb_add_relu_backward_f32",
                                   (p(a["dy_a"]), p(a["dy_b"]), p(a["x"]), p(a["dx"]), t[a["x"]].numel(), S)))
            elif k == "add_out":
                self.calls.append(("sgb_binary_f32", (0, p(a["a"]), p(a["b"]), p(a["out"]), t[a["out"]].numel(), S)))
            elif k in ("bn_bwd", "bn_relu_bwd", "bn_relu_mask_bwd"):
                n, c, h, w = t[a["x"]].shape
                if k == "bn_bwd":
                    self.calls.append(("sgb_bn_backward_f32",
                                       (p(a["x"]), p(a["dy"]), p(a["scale"]), p(a["mean"]), p(a["invstd"]), p(a["dx"]),
                                        p(a["dscale"]), p(a["dbias"]), n, c, h * w, ws.data_ptr(), ws.numel(), S)))
                else:
                    self.calls.append(("sgb_bn_relu_backward_mask_f32" if k == "bn_relu_mask_bwd" else "sgb_bn_relu_backward_f32",
                                       (p(a["x"]), p(a["dy"]), p(a["relu_x"]), p(a["scale"]), p(a["mean"]),
                                        p(a["invstd"]), p(a["dx"]), p(a["dscale"]), p(a["dbias"]), n, c, h * w,
                                        ws.data_ptr(), ws.numel(), S)))
            elif k == "bn_add_relu_bwd":
                n, c, h, w = t[a["x"]].shape
                self.calls.append(("sgb_bn_add_relu_backward_f32",
                                   (p(a["x"]), p(a["dy_a"]), p(a["dy_b"]), p(a["relu_x"]), p(a["scale"]),
                                    p(a["mean"]), p(a["invstd"]), p(a["joined"]), p(a["dx"]), p(a["dscale"]),
                                    p(a["dbias"]), n, c, h * w, ws.data_ptr(), ws.numel(), S)))
            elif k == "maxpool_bwd" and self.pool_argmax:
                y_scratch = torch.empty_like(t[a["y"]])
                record = torch.empty(t[a["y"]].shape, dtype=torch.uint8, device=self.device)
                _lib.call("sgb_maxpool_forward_argmax_f32", p(a["x"]), y_scratch.data_ptr(), record.data_ptr(),
                          *geom(a["x"], a["kernel"], a["stride"], a["pad"]), torch.cuda.current_stream().cuda_stream)
                torch.cuda.synchronize()
                t[a["dx"] + ".argmax"] = record
                self.calls.append(("sgb_maxpool_backward_argmax_f32",
                                   (p(a["dy"]), record.data_ptr(), p(a["dx"])) + geom(a["x"], a["kernel"], a["stride"], a["pad"]) + (S,)))
            elif k == "maxpool_bwd":
                self.calls.append(("sgb_maxpool_backward_f32",
                                   (p(a["x"]), p(a["y"]), p(a["dy"]), p(a["dx"])) + geom(a["x"], a["kernel"], a["stride"], a["pad"]) + (S,)))
            elif k == "avgpool_bwd":
                self.calls.append(("sgb_avgpool_backward_f32",
                                   (p(a["dy"]), p(a["dx"])) + geom(a["dx"], a["kernel"], a["stride"], a["pad"]) + (S,)))
            elif k == "softmax":
                r, c = t[a["x"]].shape
                self.calls.append(("sgb_softmax_rows_f32", (p(a["x"]), p(a["y"]), r, c, S)))
            elif k == "softmax_ce":
                r, c = t[a["x"]].shape
                self.calls.append(("sgb_softmax_cross_entropy_fused_f32",
                                   (p(a["x"]), p(a["t"]), r, c, float(np.float32(a["scale"])), p(a["y"]),
                                    p(a["loss"]), p(a["grad"]), S)))
            elif k == "ce_fwd":
                r, c = t[a["p"]].shape
                self.calls.append(("sgb_cross_entropy_f32", (1, r, c, p(a["p"]), p(a["t"]), p(a["loss"]), S)))
            elif k == "sum_all":
                self.calls.append(("sgb_sum_all_f32", (p(a["x"]), p(a["out"]), t[a["x"]].numel(), ws.data_ptr(), ws.numel(), S)))
            elif k == "ce_bwd":
                r, c = t[a["p"]].shape
                self.calls.append(("sgb_softmax_cross_entropy_bwd_f32", (1, r, c, p(a["p"]), p(a["t"]), p(a["grad"]), S)))
            elif k == "ce_grad":
                r, c = t[a["p"]].shape
                self.calls.append(("sgb_softmax_cross_entropy_grad_f32",
                                   (1, r, c, p(a["p"]), p(a["t"]), float(np.float32(a["scale"])), p(a["grad"]), S)))
            elif k == "scale":
                self.calls.append(("sgb_scalar_f32", (1, p(a["x"]), float(np.float32(a["c"])), p(a["x"]), t[a["x"]].numel(), S)))
            elif k == "sum_rows":
                r, c = t[a["M"]].shape
                self.calls.append(("sgb_sum_rows_f32", (p(a["M"]), p(a["v"]), r, c, ws.data_ptr(), ws.numel(), S)))
            elif k == "conv_bias_bwd":
                n, c = t[a["dy"]].shape[:2]
                hw = t[a["dy"]].numel() // (n * c)
                assert L.sgb_conv_bias_backward_workspace_bytes(n, c, hw) <= ws.numel()
                self.calls.append(("sgb_conv_bias_backward_f32",
                                   (p(a["dy"]), p(a["db"]), n, c, hw, ws.data_ptr(), ws.numel(), S)))
            elif k == "wgrad_refresh":
                # consecutive stand-ins are one run of the flat buffer
                names = ["wsyn:" + q for q in a["params"]]
                for i in range(1, len(names)):
                    assert self.wsyn_off[names[i]] == self.wsyn_off[names[i - 1]] + t[names[i - 1]].numel()
                ptrs, sizes, n = _table([t["d:" + q] for q in a["params"]])
                self._keep = getattr(self, "_keep", []) + [ptrs, sizes]
                self.calls.append(("sgb_unpack_f32", (self.wsyn_flat.data_ptr(), self.wsyn_off[names[0]], ptrs, sizes,
                                                      n, 1.0, S)))
            elif k == "fill":
                x = t[a["x"]]
                self.calls.append(("sgb_set_f32", (float(a["value"]), x.data_ptr(), x.numel(), S)))
            elif k == "grad_ready":
                self.calls.append(("grad_ready", a["param"]))
            elif k == "sync_and_update":
                self.calls.append(("sync_and_update", None))
            else:
                raise ValueError(k)
        # DistOpt policy over the gradient production order
        order = self.plan["grad_order"]
        self.grads = [t["d:" + n] for n in order]
        sizes = [g.numel() for g in self.grads]
        self.events = plan_buckets(sizes, self.threshold)
        self.flush_after = {ev[1][-1]: ev for ev in self.events}
        self.fused_tables = {ev[1][-1]: _table([self.grads[i] for i in ev[1]]) for ev in self.events if ev[0] == "fused"}
        self.single_tables = {i: _table([self.grads[i]]) for i in range(len(order))}
        names = self.plan["grad_order"]
        self.bucket_sgd = {}
        for ev in self.events:
            ps = [names[i] for i in ev[1]]
            self.bucket_sgd[ev[1][-1]] = (_table([t[n] for n in ps])[0], _table([t["d:" + n] for n in ps])[0],
                                          _table([self.moments[n] for n in ps])[0],
                                          _table([t[n] for n in ps])[1], len(ps))
        plist = self.plan["params"]
        self.sgd_tables = (_table([t[n] for n in plist])[0], _table([t["d:" + n] for n in plist])[0],
                           _table([self.moments[n] for n in plist])[0], _table([t[n] for n in plist])[1], len(plist))
        if self.dist_option.startswith("sparse") and self.comm is not None:
            self.residuals = {}
            for ev in self.events:
                tot = sum(sizes[i] for i in ev[1])
                self.residuals[ev[1][-1]] = torch.zeros(tot, device=self.device)

        self._record_program()

    # ----------------------------------------------------------------- program
    def _record_program(self):
        """The whole step as one native program: the compute calls, the exchange
        and the update of every bucket at the place where its last gradient is
        ready (opt.py:846-862 plain, :885-912 half, :1030-1090 sparse)."""
        prog, self.calls_per_step = [], 0
        self.launched = merge_calls(self.calls)
        order_index = {n: i for i, n in enumerate(self.plan["grad_order"])}
        beside, behind, self._late_tables = self._forked_update()
        forks = behind is not None
        if forks and self.comm is not None:
            # the captured step exchanges nothing itself: behind what the caller has in the capture
            prog.append(("sgb_comm_wait_captured", (self.comm._h.value, "STREAM"), _CAPTURED))
        for name, args in self.launched:
            if name == "grad_ready":
                idx = order_index[args]
                self.calls_per_step += self._record_exchange(prog, idx, _SINGLE if forks else _ALWAYS)
                if idx in beside:
                    prog += [("fork", (), _CAPTURED), beside[idx]]
            elif name == "sync_and_update":
                when = _SINGLE if forks else _ALWAYS
                if self.comm is not None:
                    prog.append(("sgb_comm_wait", (self.comm._h.value, "STREAM"), when))
                prog += behind or []
                if beside:
                    prog.append(("join", (), _CAPTURED))
                if self._arrives():
                    continue                  # every bucket was updated as it arrived
                prog.append(self._sgd_call(self.sgd_tables, "STREAM", when))
                self.calls_per_step += 1
            else:
                prog.append((name, tuple(C.addressof(a) if isinstance(a, C.Array) else a for a in args), _ALWAYS))
                self.calls_per_step += 1
        # The library may capture the program by itself unless the launches have to be
        # made one by one: collectives (a graph that holds them keeps the communicator
        # from closing), the sparse exchange (more ranks wait for counts on the host)
        # and the streaming batch-norm form (each launch draws one of eight counter
        # tables, a captured one would keep its own), where a call takes it.
        single = self.comm is not None and (self.comm.world_size > 1 or self.dist_option not in ("plain", "half"))
        masks = {"bn_bwd": 0, "bn_add_relu_bwd": 0, "bn_relu_bwd": 1, "bn_relu_mask_bwd": 2}
        for op in self.plan["ops"]:
            if op.kind in masks:
                n, c, h, w = self.t[op.args["x"]].shape
                single = single or \
                    self.lib.sgb_bn_backward_draws_table(n, c, h * w, masks[op.kind], self.ws.numel()) != 0
        self._program = _lib.native.program(prog, None if self.comm is None else self.comm._h.value, not single)

    def _arrives(self):
        """Whether buckets are updated where their reduced gradients land."""
        return self.update_on_arrival and self.comm is not None and self.dist_option in ("plain", "half")

    def _forked_update(self):
        """The update in a captured step without other ranks: what goes on a branch of
        its own beside the rest of the backward pass, as {gradient that completes a
        bucket: call}, the calls behind the pass, and the tables that these read.  ({}, None,
        None) where the update stays as it is: several ranks, the sparse exchanges, one
        update behind the whole pass was asked for, or `leaves_what_is_ready` does not hold.

        A step of small layers leaves most of the memory's rate unused, and the update
        is nothing but memory traffic.  A bucket goes on the branch if that gets done
        while the pass lasts; what does not is updated behind it, by all of the GPU at
        once.  Launched one by one (the first runs of a program and those after its rates
        have changed) the step stays as it is.  All figures here are of one B200 and of
        graphs, as are the rates below, from which it follows which buckets go where.

        Without -> with it, us a step: ResNet-50, batch 3 at 160^2 277 -> 249, 2 at 159^2
        241 -> 211, 9 at 97^2 321 -> 302; on one rank, where the communicator's streams had
        the update, plain 10 at 85^2 314 -> 300 and in half precision 2 at 190^2 313 -> 304;
        the MLP of 2035 at batch 5, plain, 41 -> 31, of 748 at batch 177 in half precision
        35 -> 19, the CNN of 53 channels at batch 49 35 -> 23.  All of the 4096 MLP's update
        on the branch: 76 -> 111, so its rate matters."""
        half = self.comm is not None and self.dist_option == "half"
        if not leaves_what_is_ready(self.plan):
            return {}, None, None

        def largest(kinds):
            return max((sum(self.grads[i].numel() for i in ev[1]) for ev in self.events if ev[0] in kinds), default=0)

        if self.comm is None:
            if not self._branch:
                return {}, None, None
        # one rank: the sum over the ranks is the gradient (rounded, in half precision);
        # what does not fit the communicator's buffers is refused by its own calls
        elif self.comm.world_size != 1 or not self._arrives() or \
                largest(("direct", "fused") if half else ("fused",)) > getattr(self.comm, "buffSize", 0):
            return {}, None, None
        rates = ("LR", "MOMENTUM", 0.0, "DECAY", 0, float(np.float32(1.0) / np.float32(self.world)))

        def addresses(tables):
            pp, gp, mp, sizes, n = tables
            return C.addressof(pp), C.addressof(gp), C.addressof(mp), C.addressof(sizes), n

        # when each gradient is ready, in us: a call takes 2.5, or what its tensors (three of
        # the result's size, about) take at 6 TB/s
        now, ready, order = 0.0, {}, {n: i for i, n in enumerate(self.plan["grad_order"])}
        for op in self.plan["ops"]:
            if op.kind == "grad_ready":
                ready[order[op.args["param"]]] = now
            elif op.kind != "sync_and_update":
                result = self.t.get(op.args.get("dx"))
                now += 2.5 if result is None else max(2.5, 2e-6 * result.numel())
        beside, late, free = {}, [], 0.0
        for idx in sorted(self.flush_after):
            bucket = self.flush_after[idx][1]
            # the branch moves 2.4 TB/s
            done = max(free, ready[idx]) + sum(self.grads[i].numel() for i in bucket) * (24e-6 if half else 20e-6) / 2.4
            if done <= now:
                free = done
                beside[idx] = ("sgb_sgd_update_beside_f32",
                               addresses(self.bucket_sgd[idx]) + rates + (int(half), "SIDE_STREAM"), _CAPTURED)
            else:
                late += bucket
        if not late:
            return beside, [], None
        names = [self.plan["grad_order"][i] for i in late]
        ps, gs, ms = ([t[n] for n in names] for t in (self.t, {n: self.t["d:" + n] for n in names}, self.moments))
        keep = (_table(ps)[0], _table(gs)[0], _table(ms)[0], _table(ps)[1], len(names))
        tables = addresses(keep)
        if half:
            return beside, [("sgb_comm_update_half", (self.comm._h.value,) + tables + (max(p.numel() for p in ps),) + rates +
                             ("STREAM",), _CAPTURED)], keep
        return beside, [("sgb_sgd_update_multi_f32", tables + rates + ("STREAM",), _CAPTURED)], keep

    def _sgd_call(self, tables, stream, when=_ALWAYS):
        pp, gp, mp, sizes, n = tables
        scale = float(np.float32(1.0) / np.float32(self.world))
        return ("sgb_sgd_update_multi_f32", (C.addressof(pp), C.addressof(gp), C.addressof(mp), C.addressof(sizes), n,
                                             "LR", "MOMENTUM", 0.0, "DECAY", 0, scale, stream), when)

    def _record_exchange(self, prog, idx, when=_ALWAYS):
        """Appends what happens when gradient `idx` is ready; returns how many
        calls that counts for."""
        if self.comm is None:
            return 0
        h = self.comm._h.value
        ev = self.flush_after.get(idx)
        opt = self.dist_option
        is_direct = ev is not None and ev[0] == "direct"

        def addresses(tables):
            ptrs, sizes, n = tables
            return C.addressof(ptrs), C.addressof(sizes), n

        if ev is not None:
            prog.append(("sgb_comm_profile_mark", (h, b"bucket_ready", "STREAM"), _PROFILED))
        if opt not in ("plain", "half"):
            # sparse options: nothing is staged, the whole bucket is handed over at flush time
            if ev is None:
                return 0
            prog.append(("sgb_comm_sparsification",
                         (h,) + addresses(self.single_tables[idx] if is_direct else self.fused_tables[idx]) +
                         (self.residuals[idx].data_ptr(), float(self.spars), int(opt == "sparseTopK"), "STREAM"), when))
            return 1
        half = opt == "half"
        if is_direct:
            g = self.grads[idx]
            prog.append(("sgb_comm_synch_half", (h, g.data_ptr(), g.numel(), "STREAM"), when) if half else
                        ("sgb_comm_synch", (h, g.data_ptr(), g.numel(), 0, "STREAM"), when))
            self._record_bucket_update(prog, idx, when)
            return 1

        def fused(tables, send):
            mode = (send, "STREAM") if half else (0, send, "STREAM")
            prog.append(("sgb_comm_fused_synch_half" if half else "sgb_comm_fused_synch",
                         (h,) + addresses(tables) + mode, when))

        fused(self.single_tables[idx], 0)
        if ev is None:
            return 1
        fused(self.fused_tables[idx], 1)
        self._record_bucket_update(prog, idx, when)
        return 3

    def _record_bucket_update(self, prog, idx, when):
        """The bucket's parameters are updated on the side stream on which its
        reduced gradients land (never on the NCCL stream: the next bucket's
        all-reduce does not wait for this update)."""
        if not self._arrives():
            return
        h = self.comm._h.value
        prog.append(("sgb_comm_profile_range", (h, b"sgd_update_bucket", "RESULT_INDEX", 1), when))
        prog.append(self._sgd_call(self.bucket_sgd[idx], "RESULT_STREAM", when))
        prog.append(("sgb_comm_profile_range", (h, b"sgd_update_bucket", "RESULT_INDEX", 0), when))

    # --------------------------------------------------------------------- run
    def run_step(self):
        """Enqueues one full step on the current stream (+ the communicator's
        side streams).  Returns the number of C-ABI calls issued."""
        comm = self._comm
        if comm is not None and comm._h is None:
            raise _lib.SgbError("sgb_comm", -1, "the communicator is closed")
        if self._program is None:
            self._record_program()
        _lib.native.run_program(self._program, self.lr, self.momentum, self.weight_decay, self.profile)
        return self.calls_per_step

    def capture(self):
        """Captures one step into a CUDA graph (after a warm-up step has run)."""
        g = torch.cuda.CUDAGraph()
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
                self.run_step()
        torch.cuda.current_stream().wait_stream(s)
        self.graph = g
        return g

    def release_graph(self):
        """Drops the captured step.  Must be called before the communicator is
        closed: NCCL keeps a communicator alive (its destroy call waits) for as
        long as a CUDA graph that captured its collectives exists."""
        self.graph = None

    def loss(self):
        return self.t["loss"]
