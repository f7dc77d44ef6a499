"""SGD and DistOpt drivers with the reference's structure (python/singa/opt.py),
written against ``singa_b200.singa_wrap`` / ``singa_b200.communicator``.

The reference builds gradients with its autograd generator; this module takes
any iterable of ``(param, grad)`` pairs in the order gradients are produced
(what ``autograd.backward(loss)`` yields, python/singa/autograd.py:128-224).
"""
import functools
import operator

import numpy as np

from . import singa_wrap as sw


def plan_buckets(sizes, threshold=2097152):
    """Bucket policy of DistOpt.backward_and_update (opt.py:846-862): a tensor
    larger than ``threshold`` is reduced directly; smaller ones are staged and
    the bucket is flushed as soon as it holds more than ``threshold``
    elements.  Returns [("direct" | "fused", [indices])] in issue order."""
    events, glist, acc = [], [], 0
    for i, n in enumerate(sizes):
        if n > threshold:
            events.append(("direct", [i]))
            continue
        glist.append(i)
        acc += n
        if acc > threshold:
            events.append(("fused", glist))
            glist, acc = [], 0
    if glist:
        events.append(("fused", glist))
    return events


class SGD(object):
    """SGD with momentum / dampening / weight decay / Nesterov (opt.py:161-333).

    ``apply`` is one fused kernel pass per call; ``apply_many`` updates a whole
    parameter list in one launch group.  Hyper-parameters are python floats
    (the reference keeps them in one-element device tensors)."""

    def __init__(self, lr=0.1, momentum=0, dampening=0, weight_decay=0, nesterov=False):
        if momentum < 0.0:
            raise ValueError("Invalid momentum value: {}".format(momentum))
        if weight_decay < 0.0:
            raise ValueError("Invalid weight_decay value: {}".format(weight_decay))
        if nesterov and (momentum <= 0 or dampening != 0):
            raise ValueError("Nesterov momentum requires a momentum and zero dampening")
        self.lr, self.momentum, self.dampening = lr, momentum, dampening
        self.weight_decay, self.nesterov = weight_decay, nesterov
        self.moments = dict()
        self.step_counter = 0

    def _moment(self, name, like):
        import torch
        if name not in self.moments:
            self.moments[name] = torch.zeros_like(like)
        return self.moments[name]

    def apply(self, param_name, param_value, param_grad, grad_scale=1.0):
        assert param_value.shape == param_grad.shape, ("shape mismatch", param_value.shape,
                                                       param_grad.shape)
        self.apply_many([param_name], [param_value], [param_grad], grad_scale)

    def _moments_of(self, names, params):
        if self.momentum == 0:
            return None
        have = self.moments
        try:
            return [have[n] for n in names]
        except KeyError:                                  # first step of a parameter
            return [self._moment(n, p) for n, p in zip(names, params)]

    def apply_many(self, names, params, grads, grad_scale=1.0):
        moments = self._moments_of(names, params)
        sw.sgd_update_multi(params, grads, moments, self.lr, self.momentum, self.dampening,
                            self.weight_decay, self.nesterov, grad_scale)

    def step(self):
        self.step_counter += 1


# exchange: (the communicator's method for all of it, DistOpt's forwards and the
# communicator's calls that it stands for)
_WHOLE = {
    "plain": ("syncDense", ("all_reduce", "fused_all_reduce"), ("synch", "fusedSynch")),
    "half": ("syncDense", ("all_reduce_half", "fused_all_reduce_half"), ("synchHalf", "fusedSynchHalf")),
    "sparse": ("beginSparsification", ("sparsification", "fused_sparsification"),
               ("sparsification", "fusedSparsification")),
    "joint": ("sparsifyBuckets", ("sparsification", "fused_sparsification"), ("sparsification", "fusedSparsification")),
}


# the communicator's method that does an exchange and the update behind it
# (and what else of the communicator it stands for)
_WITH_UPDATE = {"half": ("updateHalf", ("syncDense", "wait")),
                "sparse": ("sparseUpdate", ("beginSparsification", "endSparsification", "sparsifyBuckets", "wait"))}
_AROUND = ("wait", "_update_all", "_sync_dense")     # of DistOpt: what lies between the two
_LISTS = (list, tuple, type(iter([])), type(iter(())))


@functools.lru_cache(maxsize=64)
def _inverse(world_size):
    """1 / world_size as fp32 forms it."""
    return float(np.float32(1.0) / np.float32(world_size))


def _as_defined(cls, names):
    """Whether the class still has the functions that it was defined with (classes
    that keep those in ``_defined``; others are taken as they are)."""
    defined = vars(cls).get("_defined", {})
    return all(vars(cls).get(f) is defined[f] for f in names if f in defined)


def _reader(names):
    """Function of a class: what it has under these names, None where it has nothing."""
    read = operator.attrgetter(*names)

    def functions(cls):
        try:
            return read(cls)
        except AttributeError:
            return tuple(getattr(cls, f, None) for f in names)
    return functions


# By exchange: the names that must not be an instance's own (of DistOpt, of the
# communicator), and what reads the classes' functions.
_OF_WHOLE = {x: (f + c, operator.attrgetter(*f), operator.attrgetter(name, *c)) for x, (name, f, c) in _WHOLE.items()}
_OF_UPDATE = {x: (frozenset(_WHOLE[x][1] + _AROUND), frozenset((name,) + c + _WHOLE[x][2]),
                  _reader(_WHOLE[x][1] + _AROUND), _reader((name, _WHOLE[x][0]) + c + _WHOLE[x][2]))
              for x, (name, c) in _WITH_UPDATE.items()}


# The last arguments of these two: what the classes have in place of the functions that
# the answer is about, so that a remembered answer is not given for others.
@functools.lru_cache(maxsize=64)
def _stands(own, kind, exchange, *functions):
    """Whether the method of communicators of class `kind` does what `own` (DistOpt
    or a subclass) would do call by call: nobody below the class that defines it
    has a version of its own of a call, and nobody has put one into that class."""
    name, forwards, calls = _WHOLE[exchange]
    owner = next((k for k in kind.__mro__ if name in vars(k)), None)
    return owner is not None and all(getattr(own, f) is getattr(DistOpt, f) for f in forwards) and \
        all(getattr(kind, f, None) is getattr(owner, f, None) for f in calls) and \
        _as_defined(DistOpt, forwards) and _as_defined(owner, calls)


@functools.lru_cache(maxsize=64)
def _stands_with_update(own, kind, exchange, *functions):
    """Whether the method of communicators of class `kind` that also updates does what
    the exchange, wait() and the update of `own` would do one after the other."""
    def owner(name):
        return next((k for k in kind.__mro__ if name in vars(k)), None)
    name, calls = _WITH_UPDATE[exchange]
    return owner(name) is not None and all(owner(x) in (None, owner(name)) for x in calls) and \
        all(getattr(own, f) is getattr(DistOpt, f) for f in _AROUND) and \
        _as_defined(DistOpt, _AROUND) and _as_defined(owner(name), calls) and _as_defined(SGD, ("apply_many",)) and \
        _stands.__wrapped__(own, kind, exchange)


class DistOpt(object):
    """Data-parallel wrapper of an optimizer (opt.py:686-1094).

    ``nccl_id`` is a ``communicator.NcclIdHolder`` shared by all ranks.  The
    1/world scaling of ``DistOpt.update`` (opt.py:738-746) and the optimizer
    step run as ONE multi-tensor launch group at the end of each
    ``backward_and_*`` call (``grad_scale`` of the fused SGD kernel)."""

    def __init__(self, opt, nccl_id=None, local_rank=0, world_size=1, buffSize=4194304,
                 communicator=None):
        self.opt = opt
        if communicator is None:
            from .communicator import Communicator
            communicator = Communicator(local_rank, world_size, nccl_id, buffSize)
        # any object with the reference Communicator's methods and rank fields
        self.communicator = communicator
        self.world_size = self.communicator.world_size
        self.local_rank = self.communicator.local_rank
        self.global_rank = self.communicator.global_rank

    # thin forwards, names as in the reference
    def all_reduce(self, tensor):
        self.communicator.synch(tensor)

    def fused_all_reduce(self, tensors, send=True):
        self.communicator.fusedSynch(tensors, send)

    def all_reduce_half(self, tensor):
        self.communicator.synchHalf(tensor)

    def fused_all_reduce_half(self, tensors, send=True):
        self.communicator.fusedSynchHalf(tensors, send)

    def sparsification(self, tensor, accumulation, spars, topK):
        self.communicator.sparsification(tensor, accumulation, spars, topK)

    def fused_sparsification(self, tensors, accumulation, spars, topK):
        self.communicator.fusedSparsification(tensors, accumulation, spars, topK)

    def wait(self):
        self.communicator.wait()

    def update(self, param, grad, name=None):
        """grad /= world_size, then the wrapped optimizer's update."""
        scale = _inverse(self.world_size)
        self.opt.apply(name if name is not None else id(param), param, grad, grad_scale=scale)

    def _whole(self, exchange):
        """The communicator's method that does the whole `exchange` (_WHOLE): None
        where it has none, or where a subclass or an instance has its own version
        of one of the calls that it stands for, which then has to be called."""
        c = self.communicator
        (f, g, x, y), of_mine, of_theirs = _OF_WHOLE[exchange]
        mine, theirs, own, kind = self.__dict__, getattr(c, "__dict__", ()), type(self), type(c)
        try:
            if f in mine or g in mine or x in theirs or y in theirs or \
                    not _stands(own, kind, exchange, of_mine(own), of_theirs(kind)):
                return None
        except AttributeError:                            # a communicator without one of the calls
            if not _stands.__wrapped__(own, kind, exchange):
                return None
        return getattr(c, _WHOLE[exchange][0])

    def _with_update(self, exchange, grad_stream):
        """The communicator's method that does the whole `exchange` of gradients that
        exist already and the update behind it (_WITH_UPDATE), on one rank.  None
        where it has none, or where something that it stands for has been replaced."""
        c, opt = self.communicator, self.opt
        if self.world_size != 1 or type(grad_stream) not in _LISTS or type(opt) is not SGD:
            return None
        mine, theirs, of_mine, of_theirs = _OF_UPDATE[exchange]
        own, kind = type(self), type(c)
        if "apply_many" in opt.__dict__ or not (
                mine.isdisjoint(self.__dict__) and theirs.isdisjoint(getattr(c, "__dict__", ())) and
                _stands_with_update(own, kind, exchange, SGD.apply_many, of_mine(own), of_theirs(kind))):
            return None
        return getattr(c, _WITH_UPDATE[exchange][0])

    def _hyper(self):
        o = self.opt
        return o.lr, o.momentum, o.dampening, o.weight_decay, o.nesterov, _inverse(self.world_size)

    def _update_all(self, plist):
        scale = _inverse(self.world_size)
        names, params, grads = plist
        if names:
            self.opt.apply_many(names, params, grads, scale)
        self.opt.step()

    def _sync_dense(self, grad_stream, threshold, direct, fused, half=False):
        """Names, parameters and (reduced) gradients of the stream."""
        whole = self._whole("half" if half else "plain")
        if whole is not None:
            plist = whole(grad_stream, threshold, half)
            self.wait()
            return plist
        names, params, grads, glist, acc = [], [], [], [], 0
        for name, p, g in grad_stream:
            n = g.numel()
            if n > threshold:
                direct(g)
            else:
                glist.append(g)
                fused([g], False)
                acc += n
                if acc > threshold:
                    fused(glist, True)
                    acc, glist = 0, []
            names.append(name)
            params.append(p)
            grads.append(g)
        if glist:
            fused(glist, True)
        self.wait()
        return names, params, grads

    def backward_and_update(self, grad_stream, threshold=2097152):
        """opt.py:826-865 over (name, param, grad) triples."""
        self._update_all(self._sync_dense(grad_stream, threshold, self.all_reduce,
                                          self.fused_all_reduce))

    def backward_and_update_half(self, grad_stream, threshold=2097152, clipping=False,
                                 clip_Value=100):
        """opt.py:867-920: fp16 transport of fp32 gradients."""
        update = None if clipping else self._with_update("half", grad_stream)
        if update is not None:
            grad_stream = list(grad_stream)
            if grad_stream and all(len(t) == 3 for t in grad_stream):
                names, params, grads = map(list, zip(*grad_stream))
                if update(params, grads, self.opt._moments_of(names, params), threshold, self._hyper()):
                    self.opt.step()
                    return

        def clipped(stream):
            for name, p, g in stream:
                sw.Clamp(g, -clip_Value, clip_Value, out=g)
                yield name, p, g
        self._update_all(self._sync_dense(clipped(grad_stream) if clipping else grad_stream, threshold,
                                          self.all_reduce_half, self.fused_all_reduce_half, half=True))

    def _divide_by_world(self, t):
        sw.DivFloatWithRet(t, self.world_size, t)

    def backward_and_partial_update(self, grad_stream, threshold=2097152):
        """opt.py:922-992 (asynchronous variant): every parameter is updated with
        its LOCAL gradient first; then ONE partition of the PARAMETERS - the
        ``self.partial``-th bucket in production order, cycling - is all-reduced
        and averaged.  A partition is a tensor above ``threshold`` or a bucket of
        smaller ones, exactly as in ``backward_and_update``."""
        self.partial = getattr(self, "partial", 0) + 1
        names, params, grads = [], [], []
        k, acc, bucket, reduced = 0, 0, [], []
        picked = []                                   # (kind, tensors) of the partition to exchange
        for name, p, g in grad_stream:
            names.append(name)
            params.append(p)
            grads.append(g)
            if p.numel() > threshold:
                k += 1
                if k == self.partial:
                    picked.append(("direct", [p]))
            else:
                bucket.append(p)
                acc += p.numel()
                if acc > threshold:
                    k += 1
                    if k == self.partial:
                        picked.append(("fused", bucket))
                    acc, bucket = 0, []
        if bucket:
            k += 1
            if k == self.partial:
                picked.append(("fused", bucket))
        # local update of everything (grad_scale 1: no averaging of gradients in this mode)
        self.opt.apply_many(names, params, grads, 1.0)
        for kind, tensors in picked:
            if kind == "direct":
                self.all_reduce(tensors[0])
            else:
                self.fused_all_reduce(tensors, send=False)
                self.fused_all_reduce(tensors)
            reduced = tensors
        self.wait()
        for r in reduced:
            self._divide_by_world(r)                   # "r /= world_size" on the exchanged parameters
        if k == self.partial:
            self.partial = 0
        self.opt.step()

    def backward_and_sparse_update(self, grad_stream, threshold=2097152, spars=0.05, topK=False,
                                   corr=True):
        """opt.py:994-1094: sparsified synchronisation with local residuals."""
        import torch
        if corr and not getattr(self, "sparsInit", False):
            # also when an earlier first pass was cut short: a part of the list would
            # hand each bucket another bucket's residual
            self.gradAccumulation = []
            self.sparsInit = False
        names, params, grads, k = [], [], [], -1

        def buckets():
            glist, acc = [], 0
            for name, p, g in grad_stream:
                names.append(name)
                params.append(p)
                grads.append(g)
                n = g.numel()
                if n > threshold:
                    yield [g], n, True
                    continue
                glist.append(g)
                acc += n
                if acc > threshold:
                    yield glist, acc, False
                    acc, glist = 0, []
            if glist:
                yield glist, acc, False

        def residual(n, like):
            if corr and not self.sparsInit:
                self.gradAccumulation.append(torch.zeros(n, dtype=like.dtype, device=like.device))
            return self.gradAccumulation[k] if corr else None

        # A communicator that offers the exchange in two halves has bucket k's
        # selection issued before the host waits for the counts of bucket k-1.
        begin = None
        opened = 0

        def exchange(tensors, res, single):
            nonlocal opened
            if begin is not None:
                begin(tensors, res, spars, topK)
                opened += 1
                if opened == 2:
                    opened = 1
                    self.communicator.endSparsification()
            elif single:
                self.sparsification(tensors[0], res, spars, topK)
            else:
                self.fused_sparsification(tensors, res, spars, topK)

        # On one rank, gradients that all exist already go through one selection,
        # and are updated as they are written.
        joint = update = None
        if corr and self.world_size == 1 and type(grad_stream) in _LISTS:
            takes = getattr(self.communicator, "takesSparseUpdate", None)
            if takes is not None and type(self.opt) is SGD:
                grad_stream = list(grad_stream)
                takes = takes(grad_stream, threshold, topK)
            if takes is None or takes:
                update = self._with_update("sparse", grad_stream)
            if not topK and update is None:
                joint = self._whole("joint")
        updated = False
        try:
            if joint is not None or update is not None:
                ready = []
                for tensors, n, single in buckets():
                    k += 1
                    ready.append((tensors, residual(n, tensors[0]), single))
                lists, residuals = [b[0] for b in ready], [b[1] for b in ready]
                if update is not None and ready:
                    # in bucket order: a large tensor's bucket may come before an open one's
                    place = {id(g): i for i, g in enumerate(grads)}
                    order = [place[id(g)] for b in lists for g in b]
                    moments = self.opt._moments_of(names, params)
                    updated = len(place) == len(grads) and update(
                        lists, residuals, [params[i] for i in order],
                        None if moments is None else [moments[i] for i in order], spars, topK, self._hyper())
                if not updated and update is not None and not topK:
                    joint = self._whole("joint")
                if not updated and (joint is None or not ready or not joint(lists, residuals, spars)):
                    begin = self._whole("sparse")
                    for b in ready:
                        exchange(*b)
            else:
                begin = self._whole("sparse")
                for tensors, n, single in buckets():
                    k += 1
                    exchange(tensors, residual(n, tensors[0]), single)
        finally:
            # Whatever the stream or an exchange raised: one left open would refuse every
            # later call, and without wait() the side streams could still be reading
            # tensors that the unwinding frees.
            if opened:
                self.communicator.endSparsification()
            self.wait()
        self.sparsInit = True
        if updated:
            self.opt.step()
        else:
            self._update_all((names, params, grads))


SGD._defined, DistOpt._defined = dict(vars(SGD)), dict(vars(DistOpt))
