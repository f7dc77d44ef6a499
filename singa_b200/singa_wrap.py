"""Host-side mirror of the reference's ``singa_wrap`` names for the backward path.

The reference exposes its C++ tensor functions and operation handles to
Python through SWIG (src/api/core_tensor.i, src/api/model_operation.i).  This
module offers the same names, argument order and return conventions for the
functions on the backward path, over CUDA ``torch.Tensor`` storage (torch is
only the owner of device memory and streams here).  Every function calls the
C ABI in ``libsgb.so``, most of them through the native module that checks
the tensors, allocates the result and launches in one call; nothing is
computed by torch and there is no CPU path: a CPU tensor raises ``ValueError``.

Tensors must be contiguous, as ``singa::Tensor`` blocks are on this path.
"""
import numpy as np
import torch

from . import _lib

_n = _lib.native
_F32, _F16, _I32 = torch.float32, torch.float16, torch.int32


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _chk(*ts):
    for t in ts:
        if not t.is_cuda:
            raise ValueError("singa_b200 has no CPU path: tensor is on %s" % t.device)
        if not t.is_contiguous():
            raise ValueError("tensor must be contiguous")


def _p(t):
    return t.data_ptr()


def _suffix(t):
    if t.dtype == _F32:
        return "f32"
    if t.dtype == _F16:
        return "f16"
    raise TypeError("unsupported dtype %s" % t.dtype)


# ------------------------------------------------------------------ ReLU path
def ReLU(t):
    """core_tensor.i:203 ``Tensor ReLU(const Tensor&)``."""
    return _n.relu(t)


def ReLUBackward(in1, in2):
    """core_tensor.i:221 ``Tensor ReLUBackward(in1 = dy, in2 = x)``."""
    return _n.relu_backward(in1, in2)


def AddReLUBackward(dy_a, dy_b, x):
    """Fused ``(dy_a + dy_b)`` join followed by ReLUBackward (no reference
    counterpart as one call; equals ReLUBackward(dy_a + dy_b, x) bit for bit)."""
    return _n.add_relu_backward(dy_a, dy_b, x)


# ---------------------------------------------------------- elementwise family
BINARY = {"add": 0, "sub": 1, "mul": 2, "div": 3, "pow": 4,
          "gt": 5, "ge": 6, "eq": 7, "lt": 8, "le": 9}
SCALAR = {"add": 0, "mul": 1, "rdiv": 2, "pow": 3, "gt": 4, "ge": 5, "eq": 6,
          "lt": 7, "le": 8, "threshold": 9}
UNARY = {n: i for i, n in enumerate(
    ["abs", "sign", "exp", "erf", "ceil", "floor", "round", "rounde", "log",
     "sqrt", "square", "cos", "cosh", "acos", "acosh", "sin", "sinh", "asin",
     "asinh", "tan", "tanh", "atan", "atanh", "sigmoid", "softplus", "softsign"])}


def binary(op, a, b, out=None):
    """Tensor (op) tensor; ``out`` may alias an input (``a += b`` joins)."""
    return _n.binary(BINARY[op], a, b, out)


def scalar(op, t, x, out=None):
    return _n.scalar(SCALAR[op], t, x, out)


def unary(op, t, out=None):
    return _n.unary(UNARY[op], t, out)


def iAdd(t, other):
    """core_tensor.i:151 ``operator+=`` (the gradient join)."""
    return binary("add", t, other, out=t)


def EltwiseMultFloatWithRet(t, x, ret):
    """core_tensor.i:321-322."""
    return scalar("mul", t, x, out=ret)


def DivFloatWithRet(t, x, ret):
    """core_tensor.i:325-326: Div(t, x) is EltwiseMult(t, 1/x)
    (src/core/tensor/tensor_math.h:149-153)."""
    return _n.scalar(SCALAR["mul"], t, np.float32(1.0) / np.float32(x), ret)


def Clamp(t, low, high, out=None):
    return _n.clamp(t, low, high, out)


def SetValue(t, v):
    return _n.set_value(t, v)


_CASTS = {(_F32, _F16): 0, (_F16, _F32): 1, (_F32, _I32): 2, (_I32, _F32): 3}


def AsType(t, dtype):
    """core_tensor.i:129 ``Tensor::AsType`` for f32<->f16 and f32<->int."""
    _chk(t)
    kind = _CASTS.get((t.dtype, dtype))
    if kind is None:
        raise TypeError("unsupported cast %s -> %s" % (t.dtype, dtype))
    return _n.cast(t, kind)


def Axpy(alpha, inp, out):
    """core_tensor.i:345-347: ``out += alpha * in``; alpha is a python float
    or a one-element device tensor."""
    if isinstance(alpha, torch.Tensor) and alpha.dtype != _F32:
        alpha = alpha.float()                         # AsType(kFloat32), tensor_math_cuda.h:1056
    return _n.axpy(alpha, inp, out)


def Transform(t_storage, shape, stride):
    """Materialises a strided / broadcast view (element strides, 0 = broadcast)
    as a contiguous tensor: Transform<float, lang::Cuda>
    (src/core/tensor/tensor_math_cuda.h:238-298)."""
    import ctypes as C
    _chk(t_storage)
    n = 1
    for s in shape:
        n *= s
    out = torch.empty(tuple(shape), dtype=t_storage.dtype, device=t_storage.device)
    sh = (C.c_int * len(shape))(*shape)
    st = (C.c_int * len(shape))(*stride)
    _lib.call("sgb_strided_copy_" + _suffix(t_storage), _p(t_storage), _p(out), n, len(shape),
              C.cast(sh, C.c_void_p), C.cast(st, C.c_void_p), _stream())
    return out


# ------------------------------------------------------------------ workspace
def _workspace(like, nbytes):
    """A scratch buffer owned by the host layer (the C ABI never allocates), 256-byte
    aligned by the torch allocator.  Kernels exchange sums through it while they run,
    so calls that may overlap never get the same one: it belongs to the current
    stream and host thread or, during a capture, to the graph that is being made,
    whose replays keep it to themselves for as long as they can run."""
    return _n.workspace(like, nbytes)


def _ws_args(like, nbytes):
    if nbytes == 0:
        return None, 0
    buf = _workspace(like, nbytes)
    return buf.data_ptr(), buf.numel()


# ------------------------------------------------------------------ reductions
def SumRows(M, v=None):
    """core_tensor.i:380 ``SumRows(M, v)``: v[c] = sum_r M[r, c]."""
    return _n.sum_rows(M, v)


def SumColumns(M, v=None):
    """core_tensor.i:379 ``SumColumns(M, v)``: v[r] = sum_c M[r, c]."""
    return _n.sum_columns(M, v)


def Sum(t, axis):
    """core_tensor.i:223 ``Tensor Sum(t, axis)`` (tensor.cc:1229-1240)."""
    if axis == 0:
        return SumRows(t)
    assert axis == 1, "Not support Sum over axis = %d" % axis
    return SumColumns(t)


def SumAll(t):
    """core_tensor.i:226 ``Tensor SumAll(t)`` -> one-element device tensor."""
    return _n.sum_all(t)


_DOT, _ASUM, _NRM2, _AMAX, _AMIN = range(5)


def Dot(a, b):
    """Dot<float, lang::Cuda> (tensor_math_cuda.h:1084-1094, the Tensor*
    overload): one-element DEVICE tensor, no host synchronisation."""
    return _n.blas1(_DOT, a, b)


def Asum(t):
    """Asum<float, lang::Cuda> (tensor_math_cuda.h:1023-1029): sum of |x|."""
    return _n.blas1(_ASUM, t)


def Nrm2(t):
    """Nrm2<float, lang::Cuda> (tensor_math_cuda.h:1097-1102)."""
    return _n.blas1(_NRM2, t)


def Amax(t):
    """Amax<float, lang::Cuda> (tensor_math_cuda.h:1001-1009): 0-based index of
    the first element with the largest magnitude (int32 device tensor)."""
    return _n.blas1(_AMAX, t)


def Amin(t):
    """Amin<float, lang::Cuda> (tensor_math_cuda.h:1012-1020): smallest magnitude."""
    return _n.blas1(_AMIN, t)


def DGMM(side_right, M, v):
    """DGMM<float, lang::Cuda> (tensor_math_cuda.h:1112-1129): M * diag(v) when
    side_right else diag(v) * M, row-major M."""
    return _n.dgmm(bool(side_right), M, v)


def RowMax(t):
    return _n.row_max(t)


def GpuConvBackwardb(dy, b=None, cch=None):
    """model_operation.i:148: db[c] = sum_{n,h,w} dy (NCHW)."""
    return _n.conv_bias_backward(dy)


# ------------------------------------------------------ softmax / cross entropy
def SoftMax(t, axis=None):
    """core_tensor.i:229-230.  ``axis`` reshapes to 2-D as tensor.cc:942-972
    does: rows = prod(shape[:axis]), columns = the rest."""
    if axis is None:
        nrow = t.shape[0] if t.dim() == 2 else 1
    else:
        axis = axis % t.dim()
        nrow = 1
        for s in t.shape[:axis]:
            nrow *= s
    return _n.softmax(t, nrow)


def CrossEntropyFwd(p, t):
    """core_tensor.i:387."""
    return _n.ce_forward(p, t)


def SoftmaxCrossEntropyBwd(p, t):
    """core_tensor.i:388: returns p - target in a new tensor."""
    return _n.ce_backward(p, t)


def SoftmaxCrossEntropyGrad(p, t, scale):
    """Fused SoftmaxCrossEntropyBwd + ``dx *= scale`` (autograd.py:1319-1322
    with scale = float32(1/N))."""
    return _n.ce_grad(p, t, scale)


# ------------------------------------------------------------ operation handles
def SoftMaxCrossEntropyFused(logits, t, scale):
    """The loss head of autograd.SoftMaxCrossEntropy (python/singa/autograd.py:
    1306-1322) for integer targets in one launch.  Returns (prob, loss per
    sample, grad) with grad = (prob - onehot) * scale."""
    return _n.softmax_ce_fused(logits, t, np.float32(scale))


class CudnnBatchNormHandle(object):
    """Shape record with the fields of singa's BatchNormHandle
    (src/model/operation/batchnorm.h:38-60); no cuDNN descriptors are needed."""

    def __init__(self, momentum, x):
        self.factor = momentum
        self.batchsize = x.shape[0]
        self.channels = x.shape[1]
        self.is_2d = x.dim() == 2
        self.height = 1 if self.is_2d else x.shape[2]
        self.width = 1 if self.is_2d else x.shape[3]


def GpuBatchNormForwardTraining(cbnh, x, bnScale, bnBias, running_mean, running_var, eps=0.0):
    """model_operation.i:159: returns [y, mean, var] where ``var`` is the saved
    INVERSE standard deviation 1/sqrt(batch_var + eps); running statistics are
    updated in place with ``cbnh.factor``.  ``eps`` defaults to the value the
    reference passes with cuDNN 9 (CUDNN_BN_MIN_EPSILON == 0)."""
    return _n.bn_forward(x, bnScale, bnBias, running_mean, running_var, cbnh.factor, eps, cbnh.batchsize,
                         cbnh.channels, cbnh.height * cbnh.width)


def GpuBatchNormBackward(cbnh, dy, x, bnScale, mean, var):
    """model_operation.i:165: returns [dx, dscale, dbias].  ``var`` is the
    saved INVERSE standard deviation produced by the forward pass, as in the
    reference (batchnorm.cc:314-321, 390-396)."""
    return _n.bn_backward(dy, None, x, bnScale, mean, var, cbnh.batchsize, cbnh.channels,
                          cbnh.height * cbnh.width)


def GpuBatchNormReLUBackward(cbnh, dy, relu_in, x, bnScale, mean, var):
    """ReLUBackward(dy, relu_in) followed by GpuBatchNormBackward, one pass."""
    return _n.bn_backward(dy, relu_in, x, bnScale, mean, var, cbnh.batchsize, cbnh.channels,
                          cbnh.height * cbnh.width)


def GpuBatchNormAddReLUBackward(cbnh, dy_a, dy_b, relu_in, x, bnScale, mean, var):
    """The end of a residual block in one pass: the gradient join dy_a + dy_b
    (autograd.py:204 "+="), ReLUBackward against relu_in, GpuBatchNormBackward.
    Returns [joined, dx, dbnScale, dbnBias]; ``joined`` is what the shortcut
    branch consumes."""
    return _n.bn_add_relu_backward(dy_a, dy_b, relu_in, x, bnScale, mean, var, cbnh.batchsize, cbnh.channels,
                                   cbnh.height * cbnh.width)


class CudnnPoolingHandle(object):
    """Fields of singa's PoolingHandle (src/model/operation/pooling.h:41-78,
    pooling.cc:27-52)."""

    def __init__(self, x, kernel_size, stride, padding, is_max=True):
        self.kernel_h, self.kernel_w = kernel_size
        self.stride_h, self.stride_w = stride
        self.pad_h, self.pad_w = padding
        self.batchsize, self.channels, self.height, self.width = x.shape
        self.pooled_height = 1
        if self.stride_h > 0:
            self.pooled_height = (self.height + 2 * self.pad_h - self.kernel_h) // self.stride_h + 1
        self.pooled_width = (self.width + 2 * self.pad_w - self.kernel_w) // self.stride_w + 1
        self.is_max_pooling = is_max

    def _geom(self):
        return (self.batchsize, self.channels, self.height, self.width, self.kernel_h,
                self.kernel_w, self.pad_h, self.pad_w, self.stride_h, self.stride_w)


def GpuPoolingForward(cph, x):
    """model_operation.i:189."""
    return _n.pool_forward(x, cph.is_max_pooling, cph._geom(), cph.pooled_height, cph.pooled_width)


def GpuPoolingBackward(cph, dy, x, y):
    """model_operation.i:191."""
    return _n.pool_backward(dy, x, y, cph.is_max_pooling, cph._geom())


def GpuPoolingForwardArgmax(cph, x):
    """Max-pool forward that also returns the arg-max record (one uint8 per
    window: where its first maximum sits) for GpuPoolingBackwardArgmax."""
    assert cph.is_max_pooling
    return _n.pool_forward_argmax(x, cph._geom(), cph.pooled_height, cph.pooled_width)


def GpuPoolingBackwardArgmax(cph, dy, argmax):
    """Max-pool backward from dy and the forward's arg-max record alone (no x,
    no y); equals GpuPoolingBackward bit for bit."""
    return _n.pool_backward_argmax(dy, argmax, cph._geom())


# ------------------------------------------------------------- multi-tensor ops
def _ptr_table(tensors):
    import ctypes as C
    n = len(tensors)
    ptrs = (C.c_void_p * n)(*[t.data_ptr() for t in tensors])
    sizes = (C.c_size_t * n)(*[t.numel() for t in tensors])
    return ptrs, sizes, n


def sgd_update_multi(params, grads, moments, lr, momentum=0.0, dampening=0.0, weight_decay=0.0,
                     nesterov=False, grad_scale=1.0):
    """One launch group for SGD.apply over a list of parameter tensors."""
    _n.sgd_multi(params, grads, moments, lr, momentum, dampening, weight_decay, bool(nesterov), grad_scale)


def pack(tensors, flat, offset=0):
    _n.pack(tensors, flat, offset)


def unpack(flat, tensors, offset=0, scale=1.0):
    _n.unpack(flat, tensors, offset, scale)


# -------------------------------------------------------- sparsification kernels
def sparse_threshold(g, acc, thr):
    """s = g + acc, kept = |s| >= thr; returns (idx 1-based int32, val) of the
    kept non-zero entries in ascending order; ``acc`` (or None) is updated in
    place with the residual.  Synchronises to read the count."""
    _chk(g)
    n = g.numel()
    idx = torch.empty(max(n, 1), dtype=_I32, device=g.device)
    val = torch.empty(max(n, 1), dtype=_F32, device=g.device)
    nnz = torch.zeros(1, dtype=_I32, device=g.device)
    need = _lib.lib().sgb_sparse_workspace_bytes(n)
    ws, wsn = _ws_args(g, need)
    _lib.call("sgb_sparse_threshold_f32", _p(g), None if acc is None else _p(acc), n, float(thr),
              _p(idx), _p(val), _p(nnz), ws, wsn, _stream())
    k = int(nnz.item())
    return idx[:k], val[:k]


def sparse_topk(g, acc, k, mode="magnitude"):
    """The k entries of s = g + acc with the largest key (ties -> lower index),
    as (idx 1-based int32, val) in ascending index order; ``acc`` (or None)
    becomes s with the selected entries zeroed."""
    _chk(g)
    n = g.numel()
    k = min(int(k), n)
    idx = torch.empty(max(k, 1), dtype=_I32, device=g.device)
    val = torch.empty(max(k, 1), dtype=_F32, device=g.device)
    need = _lib.lib().sgb_sparse_workspace_bytes(n)
    ws, wsn = _ws_args(g, need)
    _lib.call("sgb_sparse_topk_f32", _p(g), None if acc is None else _p(acc), None, n, k,
              {"magnitude": 0, "compat": 1}[mode], _p(idx), _p(val), ws, wsn, _stream())
    return idx[:k], val[:k]


def topk_count(ratio, n):
    return int(_lib.lib().sgb_topk_count(float(ratio), int(n)))


def scatter_add(dst, idx, val):
    _chk(dst, idx, val)
    _lib.call("sgb_scatter_add_f32", _p(idx), _p(val), idx.numel(), None, _p(dst), dst.numel(),
              _stream())
    return dst
