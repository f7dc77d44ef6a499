// CPython binding of the Python layer: tensor checks, output allocation, the
// current stream, the C-ABI call and the error are one native function per
// `singa_wrap` name, and a recorded step is a list of C-ABI calls that one
// native loop issues.
//
// Why it exists: on the small layers of a step the GPU needs 2-5 us per call
// and the interpreter path (ctypes conversion of 10-17 arguments, attribute
// lookups, torch.empty_like, torch.cuda.current_stream) needed 10-16 us, so
// the device waited for the host.  Here a call costs its kernel launch plus
// well under a microsecond of argument handling.  Nothing is computed here.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "sgb.h"

namespace {

using at::Tensor;

// ------------------------------------------------------------------- errors
struct PyError {};   // a Python exception has been set

[[noreturn]] void fail(PyObject* type, const std::string& text) {
  PyErr_SetString(type, text.c_str());
  throw PyError{};
}
void require(bool ok, const char* text) {
  if (!ok) fail(PyExc_AssertionError, text);
}

// singa_b200._lib.SgbError(function name, status, text)
[[noreturn]] void fail_status(const char* fn, int status) {
  std::string text = sgb_status_string(status);
  if (status == SGB_ERR_CUDA) text += " cudaError=" + std::to_string(sgb_last_cuda_error());
  PyObject* mod = PyImport_ImportModule("singa_b200._lib");
  PyObject* cls = mod ? PyObject_GetAttrString(mod, "SgbError") : nullptr;
  PyObject* err = cls ? PyObject_CallFunction(cls, "sis", fn, status, text.c_str()) : nullptr;
  if (err) PyErr_SetObject(cls, err);
  Py_XDECREF(err);
  Py_XDECREF(cls);
  Py_XDECREF(mod);
  throw PyError{};
}

using Args = PyObject* const*;

template <PyObject* (*F)(Args, Py_ssize_t), Py_ssize_t Least>
PyObject* guarded(PyObject*, Args a, Py_ssize_t n) {
  if (n < Least) {
    PyErr_Format(PyExc_TypeError, "at least %zd arguments are expected", Least);
    return nullptr;
  }
  try {
    return F(a, n);
  } catch (const PyError&) {
    return nullptr;
  } catch (const std::exception& e) {   // torch's allocator: out of memory, capture errors
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

// ---------------------------------------------------------------- arguments
const Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, "expected a torch.Tensor");
  return THPVariable_Unpack(o);
}
// A CUDA tensor with contiguous storage; what every compute call accepts.
const Tensor& dev(PyObject* o) {
  const Tensor& t = tensor(o);
  if (!t.is_cuda()) fail(PyExc_ValueError, "singa_b200 has no CPU path: tensor is on " + t.device().str());
  if (!t.is_contiguous()) fail(PyExc_ValueError, "tensor must be contiguous");
  return t;
}
bool is_none(PyObject* o) { return o == Py_None; }
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyError{};
  return v;
}
long long whole(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyError{};
  return v;
}
int small(PyObject* o) { return static_cast<int>(whole(o)); }
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PyError{};
  return v != 0;
}
void* address(PyObject* o) {
  if (is_none(o)) return nullptr;
  if (PyBytes_Check(o)) return PyBytes_AS_STRING(o);
  void* p = PyLong_AsVoidPtr(o);
  if (!p && PyErr_Occurred()) throw PyError{};
  return p;
}

const float* f32(const Tensor& t) { return static_cast<const float*>(t.const_data_ptr()); }
float* f32w(const Tensor& t) { return static_cast<float*>(t.mutable_data_ptr()); }
const void* raw(const Tensor& t) { return t.const_data_ptr(); }
void* raww(const Tensor& t) { return t.mutable_data_ptr(); }
size_t count(const Tensor& t) { return static_cast<size_t>(t.numel()); }
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// true: fp16, false: fp32; anything else is a TypeError
bool half_of(const Tensor& t) {
  if (t.scalar_type() == at::kFloat) return false;
  if (t.scalar_type() == at::kHalf) return true;
  fail(PyExc_TypeError, std::string("unsupported dtype ") + c10::toString(t.scalar_type()));
}
Tensor fresh(at::IntArrayRef sizes, at::ScalarType type, const Tensor& like) {
  return Tensor(at::detail::empty_cuda(sizes, type, like.device(), c10::nullopt));
}
Tensor fresh_like(const Tensor& t) { return fresh(t.sizes(), t.scalar_type(), t); }
PyObject* wrap(Tensor t) { return THPVariable_Wrap(std::move(t)); }
PyObject* same(PyObject* o) {
  Py_INCREF(o);
  return o;
}
template <typename... T>
PyObject* list_of(T&&... t) {
  PyObject* out = PyList_New(sizeof...(T));
  if (!out) throw PyError{};
  Py_ssize_t i = 0;
  (PyList_SET_ITEM(out, i++, wrap(std::forward<T>(t))), ...);
  return out;
}

// Runs a C-ABI call without the interpreter lock (a launch can block on a full
// queue) and raises on a non-zero status.
template <typename F>
void issue(const char* name, F&& f) {
  int st;
  Py_BEGIN_ALLOW_THREADS;
  st = f();
  Py_END_ALLOW_THREADS;
  if (st != SGB_OK) fail_status(name, st);
}
#define ISSUE(fn, ...) issue(#fn, [&] { return fn(__VA_ARGS__); })

// ---------------------------------------------------------------- workspace
// Scratch buffers, owned here (the C ABI never allocates).  Kernels exchange sums
// through them while they run, so calls that may overlap never share one: there is
// one per device, stream and host thread (a call of several kernels is not cut in
// two by another thread's on the same stream), and one per capture, which its graph
// keeps for its own replays.  A buffer that a call still holds outlives its place
// here, and what is given back goes to its stream's part of torch's allocator.
struct Scratch {
  cudaStream_t stream;
  unsigned long long thread;
  Tensor buffer;
};
struct CapturedScratch {
  unsigned long long capture;
  cudaStream_t stream;
  unsigned long long thread;
  Tensor buffer;
};
constexpr size_t kMostScratch = 32;          // per device; beyond it the one used least recently goes
constexpr size_t kLeastScratch = size_t{1} << 20;

// Most recently used first.  Never destroyed: the CUDA context may be gone by then.
std::vector<Scratch>& scratch_of(size_t device) {
  static auto* all = new std::vector<std::vector<Scratch>>;
  if (all->size() <= device) all->resize(device + 1);
  return (*all)[device];
}
void cuda_ok(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return;
  cudaGetLastError();
  fail(PyExc_RuntimeError, std::string(what) + ": " + cudaGetErrorString(e));
}
// Captured buffers by number, and the numbers of those whose graph, with all that was
// made of it, is gone.
std::map<unsigned long long, CapturedScratch>& captured_scratch() {
  static auto* m = new std::map<unsigned long long, CapturedScratch>;
  return *m;
}
struct Gone {
  std::mutex guard;
  std::atomic<bool> any{false};
  std::vector<unsigned long long> numbers;
};
Gone& gone() {
  static auto* g = new Gone;
  return *g;
}
void give_back() {
  if (!gone().any.load(std::memory_order_relaxed)) return;
  std::vector<unsigned long long> numbers;
  {
    const std::lock_guard<std::mutex> lock(gone().guard);
    numbers.swap(gone().numbers);
    gone().any = false;
  }
  for (const auto n : numbers) captured_scratch().erase(n);
}
// Buffer of a capture under way: a new one for a request that the capture's others are too small for.
Tensor capture_workspace(const Tensor& like, size_t bytes, cudaStream_t stream, unsigned long long thread) {
  static unsigned long long last = 0;
  cudaStreamCaptureStatus status;
  unsigned long long capture = 0;
  cudaGraph_t graph = nullptr;
  cuda_ok(cudaStreamGetCaptureInfo(stream, &status, &capture, &graph, nullptr, nullptr), "cudaStreamGetCaptureInfo");
  if (status != cudaStreamCaptureStatusActive) fail(PyExc_RuntimeError, "the capture under way has been invalidated");
  for (const auto& [n, c] : captured_scratch())
    if (c.capture == capture && c.stream == stream && c.thread == thread && c.buffer.device() == like.device() &&
        count(c.buffer) >= bytes)
      return c.buffer;
  const Tensor buffer = fresh({static_cast<int64_t>(bytes)}, at::kByte, like);
  const auto destroy = [](void* number) {      // may call nothing of CUDA
    const std::lock_guard<std::mutex> lock(gone().guard);
    gone().numbers.push_back(reinterpret_cast<uintptr_t>(number));
    gone().any = true;
  };
  cudaUserObject_t owner;
  cuda_ok(cudaUserObjectCreate(&owner, reinterpret_cast<void*>(static_cast<uintptr_t>(++last)), destroy, 1,
                               cudaUserObjectNoDestructorSync), "cudaUserObjectCreate");
  captured_scratch().emplace(last, CapturedScratch{capture, stream, thread, buffer});
  const cudaError_t kept = cudaGraphRetainUserObject(graph, owner, 1, cudaGraphUserObjectMove);
  if (kept != cudaSuccess) cudaUserObjectRelease(owner, 1);
  cuda_ok(kept, "cudaGraphRetainUserObject");
  return buffer;
}
// Asked on every call that needs scratch; the driver's own entry takes 80 ns less than
// the runtime's (a look-up of scratch 224 -> 143 ns).
bool capturing(cudaStream_t s) {
  using Query = int (*)(cudaStream_t, int*);
  static const Query query = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    const bool ok = cudaGetDriverEntryPointByVersion("cuStreamIsCapturing", &f, 10000, cudaEnableDefault, &found) ==
                        cudaSuccess &&
                    found == cudaDriverEntryPointSuccess;
    return ok ? reinterpret_cast<Query>(f) : nullptr;
  }();
  int status = 0;
  if (query && query(s, &status) == 0) return status != 0;
  cudaStreamCaptureStatus answer = cudaStreamCaptureStatusNone;
  cuda_ok(cudaStreamIsCapturing(s, &answer), "cudaStreamIsCapturing");
  return answer != cudaStreamCaptureStatusNone;
}
Tensor workspace(const Tensor& like, size_t bytes) {
  static std::atomic<unsigned long long> threads{0};
  thread_local const unsigned long long thread = ++threads;
  const cudaStream_t s = c10::cuda::getCurrentCUDAStream().stream();
  give_back();
  if (capturing(s)) return capture_workspace(like, bytes, s, thread);
  auto& list = scratch_of(static_cast<size_t>(like.device().index()));
  size_t k = 0;
  while (k < list.size() && !(list[k].stream == s && list[k].thread == thread)) ++k;
  if (k == list.size()) {
    if (k == kMostScratch) list.pop_back();
    list.insert(list.begin(), Scratch{s, thread, Tensor()});
  } else if (k) {
    std::rotate(list.begin(), list.begin() + k, list.begin() + k + 1);
  }
  Tensor& buffer = list[0].buffer;
  if (!buffer.defined() || count(buffer) < bytes) {
    buffer = Tensor();
    buffer = fresh({static_cast<int64_t>(std::max(bytes, kLeastScratch))}, at::kByte, like);
  }
  return buffer;
}
struct Ws {                                  // keeps the buffer until its call has been launched
  Tensor held;
  void* ptr = nullptr;
  size_t bytes = 0;
  Ws(const Tensor& like, size_t need) {
    if (!need) return;
    held = workspace(like, need);
    ptr = raww(held);
    bytes = count(held);
  }
};
PyObject* py_workspace(Args a, Py_ssize_t) {   // (tensor on the device, bytes)
  return wrap(workspace(dev(a[0]), static_cast<size_t>(whole(a[1]))));
}

// -------------------------------------------------------------- elementwise
PyObject* py_relu(Args a, Py_ssize_t) {
  const Tensor& t = dev(a[0]);
  const bool h = half_of(t);
  Tensor y = fresh_like(t);
  if (h) ISSUE(sgb_relu_f16, raw(t), raww(y), count(t), stream());
  else ISSUE(sgb_relu_f32, f32(t), f32w(y), count(t), stream());
  return wrap(std::move(y));
}
PyObject* py_relu_backward(Args a, Py_ssize_t) {
  const Tensor &dy = dev(a[0]), &x = dev(a[1]);
  require(dy.sizes() == x.sizes() && dy.scalar_type() == x.scalar_type(), "shapes and dtypes must agree");
  const bool h = half_of(dy);
  Tensor dx = fresh_like(x);
  if (h) ISSUE(sgb_relu_backward_f16, raw(dy), raw(x), raww(dx), count(dy), stream());
  else ISSUE(sgb_relu_backward_f32, f32(dy), f32(x), f32w(dx), count(dy), stream());
  return wrap(std::move(dx));
}
PyObject* py_add_relu_backward(Args a, Py_ssize_t) {
  const Tensor &ga = dev(a[0]), &gb = dev(a[1]), &x = dev(a[2]);
  Tensor dx = fresh_like(x);
  ISSUE(sgb_add_relu_backward_f32, f32(ga), f32(gb), f32(x), f32w(dx), count(x), stream());
  return wrap(std::move(dx));
}
// The result tensor of an elementwise call: `out` when given, else a new one.
struct Out {
  PyObject* given;
  Tensor made;
  Out(PyObject* o, const Tensor& like) : given(is_none(o) ? nullptr : o) {
    if (!given) made = fresh_like(like);
  }
  const Tensor& t() const { return given ? tensor(given) : made; }
  PyObject* done() { return given ? same(given) : wrap(std::move(made)); }
};
PyObject* py_binary(Args a, Py_ssize_t) {   // (op, a, b, out | None)
  const int op = small(a[0]);
  const Tensor &x = dev(a[1]), &y = dev(a[2]);
  require(x.sizes() == y.sizes() && x.scalar_type() == y.scalar_type(), "shapes and dtypes must agree");
  const bool h = half_of(x);
  Out out(a[3], x);
  if (h) ISSUE(sgb_binary_f16, op, raw(x), raw(y), raww(out.t()), count(x), stream());
  else ISSUE(sgb_binary_f32, op, f32(x), f32(y), f32w(out.t()), count(x), stream());
  return out.done();
}
PyObject* py_scalar(Args a, Py_ssize_t) {   // (op, t, x, out | None); op 1 = multiply
  const int op = small(a[0]);
  const Tensor& t = dev(a[1]);
  const float v = static_cast<float>(real(a[2]));
  Out out(a[3], t);
  if (t.scalar_type() == at::kHalf) {
    require(op == 1, "fp16 supports mul only");
    ISSUE(sgb_scalar_mul_f16, raw(t), v, raww(out.t()), count(t), stream());
  } else {
    ISSUE(sgb_scalar_f32, op, f32(t), v, f32w(out.t()), count(t), stream());
  }
  return out.done();
}
PyObject* py_unary(Args a, Py_ssize_t) {    // (op, t, out | None)
  const int op = small(a[0]);
  const Tensor& t = dev(a[1]);
  Out out(a[2], t);
  ISSUE(sgb_unary_f32, op, f32(t), f32w(out.t()), count(t), stream());
  return out.done();
}
PyObject* py_clamp(Args a, Py_ssize_t) {    // (t, low, high, out | None)
  const Tensor& t = dev(a[0]);
  const float lo = static_cast<float>(real(a[1])), hi = static_cast<float>(real(a[2]));
  Out out(a[3], t);
  ISSUE(sgb_clamp_f32, lo, hi, f32(t), f32w(out.t()), count(t), stream());
  return out.done();
}
PyObject* py_set_value(Args a, Py_ssize_t) {
  const Tensor& t = dev(a[0]);
  const float v = static_cast<float>(real(a[1]));
  if (half_of(t)) ISSUE(sgb_set_f16, v, raww(t), count(t), stream());
  else ISSUE(sgb_set_f32, v, f32w(t), count(t), stream());
  return same(a[0]);
}
PyObject* py_cast(Args a, Py_ssize_t) {     // (t, 0 f32->f16 | 1 f16->f32 | 2 f32->i32 | 3 i32->f32)
  const Tensor& t = dev(a[0]);
  const int kind = small(a[1]);
  static const at::ScalarType to[] = {at::kHalf, at::kFloat, at::kInt, at::kFloat};
  Tensor out = fresh(t.sizes(), to[kind & 3], t);
  switch (kind & 3) {
    case 0: ISSUE(sgb_cast_f32_f16, f32(t), raww(out), count(t), stream()); break;
    case 1: ISSUE(sgb_cast_f16_f32, raw(t), f32w(out), count(t), stream()); break;
    case 2: ISSUE(sgb_cast_f32_i32, f32(t), static_cast<int32_t*>(raww(out)), count(t), stream()); break;
    default: ISSUE(sgb_cast_i32_f32, static_cast<const int32_t*>(raw(t)), f32w(out), count(t), stream());
  }
  return wrap(std::move(out));
}
PyObject* py_axpy(Args a, Py_ssize_t) {     // (alpha: float | f32 device tensor, in, out)
  const Tensor &x = dev(a[1]), &y = dev(a[2]);
  const bool h = half_of(x);
  require(x.scalar_type() == y.scalar_type(), "dtypes must agree");
  if (THPVariable_Check(a[0])) {
    const Tensor& al = dev(a[0]);
    if (h) ISSUE(sgb_axpy_dev_alpha_f16, f32(al), raw(x), raww(y), count(x), stream());
    else ISSUE(sgb_axpy_dev_alpha_f32, f32(al), f32(x), f32w(y), count(x), stream());
  } else {
    const float al = static_cast<float>(real(a[0]));
    if (h) ISSUE(sgb_axpy_f16, al, raw(x), raww(y), count(x), stream());
    else ISSUE(sgb_axpy_f32, al, f32(x), f32w(y), count(x), stream());
  }
  return same(a[2]);
}

// --------------------------------------------------------------- reductions
void rows_cols(const Tensor& M, size_t* r, size_t* c) {
  if (M.dim() != 2) fail(PyExc_ValueError, "a 2-D tensor is expected");
  *r = static_cast<size_t>(M.size(0));
  *c = static_cast<size_t>(M.size(1));
}
PyObject* py_sum_rows(Args a, Py_ssize_t) {      // (M, v | None)
  const Tensor& M = dev(a[0]);
  size_t r, c;
  rows_cols(M, &r, &c);
  Tensor made;
  if (is_none(a[1])) made = fresh({M.size(1)}, at::kFloat, M);
  const Tensor& v = made.defined() ? made : tensor(a[1]);
  const Ws ws(M, sgb_sum_rows_workspace_bytes(r, c));
  ISSUE(sgb_sum_rows_f32, f32(M), f32w(v), r, c, ws.ptr, ws.bytes, stream());
  return made.defined() ? wrap(std::move(made)) : same(a[1]);
}
PyObject* py_sum_columns(Args a, Py_ssize_t) {   // (M, v | None)
  const Tensor& M = dev(a[0]);
  size_t r, c;
  rows_cols(M, &r, &c);
  Tensor made;
  if (is_none(a[1])) made = fresh({M.size(0)}, at::kFloat, M);
  const Tensor& v = made.defined() ? made : tensor(a[1]);
  ISSUE(sgb_sum_columns_f32, f32(M), f32w(v), r, c, stream());
  return made.defined() ? wrap(std::move(made)) : same(a[1]);
}
// The first two sizes, whatever else the shape holds (IndexError below two).
void leading_sizes(const Tensor& t, int64_t* n, int64_t* c) {
  if (t.dim() < 2) fail(PyExc_IndexError, "a tensor of at least two dimensions is expected");
  *n = t.size(0);
  *c = t.size(1);
}
// a / b as Python's a // b answers it: an empty batch is an error of the caller
int64_t divide(int64_t a, int64_t b) {
  if (b == 0) fail(PyExc_ZeroDivisionError, "an empty batch has no size per sample");
  return a / b;
}
PyObject* py_row_max(Args a, Py_ssize_t) {
  const Tensor& M = dev(a[0]);
  int64_t r, c;
  leading_sizes(M, &r, &c);
  Tensor v = fresh({r}, at::kFloat, M);
  ISSUE(sgb_row_max_f32, f32(M), f32w(v), static_cast<size_t>(r), static_cast<size_t>(c), stream());
  return wrap(std::move(v));
}
PyObject* py_sum_all(Args a, Py_ssize_t) {
  const Tensor& t = dev(a[0]);
  Tensor out = fresh({1}, at::kFloat, t);
  const size_t need = sgb_sum_all_workspace_bytes(count(t));
  const bool one = need == sizeof(float);          // the only partial sum is the result
  const Ws ws(t, one ? 0 : need);
  ISSUE(sgb_sum_all_f32, f32(t), f32w(out), count(t), one ? raww(out) : ws.ptr, one ? need : ws.bytes, stream());
  return wrap(std::move(out));
}
PyObject* py_blas1(Args a, Py_ssize_t n) {       // (0 dot | 1 asum | 2 nrm2 | 3 amax | 4 amin, x[, y])
  const int which = small(a[0]);
  const Tensor& x = dev(a[1]);
  const size_t k = count(x);
  Tensor out = fresh({1}, which >= 3 ? at::kInt : at::kFloat, x);
  const Ws ws(x, sgb_blas1_workspace_bytes(k));
  int32_t* io = static_cast<int32_t*>(raww(out));
  switch (which) {
    case 0: {
      if (n < 3) fail(PyExc_TypeError, "dot takes two tensors");
      const Tensor& y = dev(a[2]);
      require(count(y) == k, "sizes must agree");
      ISSUE(sgb_dot_f32, f32(x), f32(y), f32w(out), k, ws.ptr, ws.bytes, stream());
      break;
    }
    case 1: ISSUE(sgb_asum_f32, f32(x), f32w(out), k, ws.ptr, ws.bytes, stream()); break;
    case 2: ISSUE(sgb_nrm2_f32, f32(x), f32w(out), k, ws.ptr, ws.bytes, stream()); break;
    case 3: ISSUE(sgb_amax_f32, f32(x), io, k, ws.ptr, ws.bytes, stream()); break;
    default: ISSUE(sgb_amin_f32, f32(x), io, k, ws.ptr, ws.bytes, stream());
  }
  return wrap(std::move(out));
}
PyObject* py_dgmm(Args a, Py_ssize_t) {          // (right, M, v)
  const int right = truth(a[0]);
  const Tensor &M = dev(a[1]), &v = dev(a[2]);
  size_t r, c;
  rows_cols(M, &r, &c);
  require(count(v) == (right ? c : r), "vector length must match the matrix");
  Tensor out = fresh_like(M);
  ISSUE(sgb_dgmm_f32, right, f32(M), f32(v), f32w(out), r, c, stream());
  return wrap(std::move(out));
}
PyObject* py_conv_bias_backward(Args a, Py_ssize_t) {
  const Tensor& dy = dev(a[0]);
  int64_t batch, channels;
  leading_sizes(dy, &batch, &channels);
  const int n = static_cast<int>(batch), c = static_cast<int>(channels);
  const int hw = static_cast<int>(divide(dy.numel(), batch * channels));
  Tensor db = fresh({c}, at::kFloat, dy);
  const Ws ws(dy, sgb_conv_bias_backward_workspace_bytes(n, c, hw));
  ISSUE(sgb_conv_bias_backward_f32, f32(dy), f32w(db), n, c, hw, ws.ptr, ws.bytes, stream());
  return wrap(std::move(db));
}

// ------------------------------------------------------------- loss head
PyObject* py_softmax(Args a, Py_ssize_t) {       // (t, rows)
  const Tensor& t = dev(a[0]);
  const size_t rows = static_cast<size_t>(whole(a[1])), cols = count(t) / (rows ? rows : 1);
  const bool h = half_of(t);
  Tensor y = fresh_like(t);
  if (h) ISSUE(sgb_softmax_rows_f16, raw(t), raww(y), rows, cols, stream());
  else ISSUE(sgb_softmax_rows_f32, f32(t), f32w(y), rows, cols, stream());
  return wrap(std::move(y));
}
struct CeDims {
  size_t batch, dim;
  int int_target;
  CeDims(const Tensor& p, const Tensor& t) {
    batch = p.dim() == 2 ? static_cast<size_t>(p.size(0)) : 1;
    dim = static_cast<size_t>(divide(p.numel(), static_cast<int64_t>(batch)));
    require(t.scalar_type() == at::kInt, "targets are int32 (kInt) tensors");
    int_target = count(t) == batch;
  }
};
PyObject* py_ce_forward(Args a, Py_ssize_t) {
  const Tensor &p = dev(a[0]), &t = dev(a[1]);
  const CeDims d(p, t);
  const bool h = half_of(p);
  const int32_t* ti = static_cast<const int32_t*>(raw(t));
  Tensor loss = fresh({static_cast<int64_t>(d.batch)}, p.scalar_type(), p);
  if (h) ISSUE(sgb_cross_entropy_f16, d.int_target, d.batch, d.dim, raw(p), ti, raww(loss), stream());
  else ISSUE(sgb_cross_entropy_f32, d.int_target, d.batch, d.dim, f32(p), ti, f32w(loss), stream());
  return wrap(std::move(loss));
}
PyObject* py_ce_backward(Args a, Py_ssize_t) {
  const Tensor &p = dev(a[0]), &t = dev(a[1]);
  const CeDims d(p, t);
  const bool h = half_of(p);
  const int32_t* ti = static_cast<const int32_t*>(raw(t));
  Tensor g = fresh_like(p);
  if (h) ISSUE(sgb_softmax_cross_entropy_bwd_f16, d.int_target, d.batch, d.dim, raw(p), ti, raww(g), stream());
  else ISSUE(sgb_softmax_cross_entropy_bwd_f32, d.int_target, d.batch, d.dim, f32(p), ti, f32w(g), stream());
  return wrap(std::move(g));
}
PyObject* py_ce_grad(Args a, Py_ssize_t) {       // (p, t, scale)
  const Tensor &p = dev(a[0]), &t = dev(a[1]);
  const CeDims d(p, t);
  const float scale = static_cast<float>(real(a[2]));
  Tensor g = fresh_like(p);
  ISSUE(sgb_softmax_cross_entropy_grad_f32, d.int_target, d.batch, d.dim, f32(p), static_cast<const int32_t*>(raw(t)),
        scale, f32w(g), stream());
  return wrap(std::move(g));
}
PyObject* py_softmax_ce_fused(Args a, Py_ssize_t) {   // (logits, t, scale)
  const Tensor &x = dev(a[0]), &t = dev(a[1]);
  size_t batch, dim;
  require(t.scalar_type() == at::kInt && t.numel() == x.size(0), "one int32 target per sample");
  rows_cols(x, &batch, &dim);
  const float scale = static_cast<float>(real(a[2]));
  Tensor prob = fresh_like(x), grad = fresh_like(x), loss = fresh({x.size(0)}, at::kFloat, x);
  ISSUE(sgb_softmax_cross_entropy_fused_f32, f32(x), static_cast<const int32_t*>(raw(t)), batch, dim, scale, f32w(prob),
        f32w(loss), f32w(grad), stream());
  PyObject* out = PyTuple_New(3);
  if (!out) throw PyError{};
  PyTuple_SET_ITEM(out, 0, wrap(std::move(prob)));
  PyTuple_SET_ITEM(out, 1, wrap(std::move(loss)));
  PyTuple_SET_ITEM(out, 2, wrap(std::move(grad)));
  return out;
}

// ------------------------------------------------------ batch norm / pooling
PyObject* py_bn_forward(Args a, Py_ssize_t) {    // (x, scale, bias, rmean, rvar, factor, eps, n, c, hw)
  const Tensor &x = dev(a[0]), &sc = dev(a[1]), &bi = dev(a[2]), &rm = dev(a[3]), &rv = dev(a[4]);
  const float factor = static_cast<float>(real(a[5])), eps = static_cast<float>(real(a[6]));
  const int n = small(a[7]), c = small(a[8]), hw = small(a[9]);
  Tensor y = fresh_like(x), mean = fresh_like(rm), inv = fresh_like(rv);
  const Ws ws(x, sgb_bn_backward_workspace_bytes(n, c, hw));
  ISSUE(sgb_bn_forward_training_f32, f32(x), f32(sc), f32(bi), f32w(rm), f32w(rv), factor, eps, f32w(y), f32w(mean),
        f32w(inv), n, c, hw, ws.ptr, ws.bytes, stream());
  return list_of(std::move(y), std::move(mean), std::move(inv));
}
PyObject* py_bn_backward(Args a, Py_ssize_t) {   // (dy, relu_in | None, x, scale, mean, inv, n, c, hw)
  const Tensor &dy = dev(a[0]), &x = dev(a[2]), &sc = dev(a[3]), &mu = dev(a[4]), &inv = dev(a[5]);
  const float* relu_in = is_none(a[1]) ? nullptr : f32(dev(a[1]));
  const int n = small(a[6]), c = small(a[7]), hw = small(a[8]);
  Tensor dx = fresh_like(dy), ds = fresh_like(sc), db = fresh_like(sc);
  const Ws ws(dy, sgb_bn_backward_workspace_bytes(n, c, hw));
  if (relu_in)
    ISSUE(sgb_bn_relu_backward_f32, f32(x), f32(dy), relu_in, f32(sc), f32(mu), f32(inv), f32w(dx), f32w(ds), f32w(db),
          n, c, hw, ws.ptr, ws.bytes, stream());
  else
    ISSUE(sgb_bn_backward_f32, f32(x), f32(dy), f32(sc), f32(mu), f32(inv), f32w(dx), f32w(ds), f32w(db), n, c, hw,
          ws.ptr, ws.bytes, stream());
  return list_of(std::move(dx), std::move(ds), std::move(db));
}
PyObject* py_bn_add_relu_backward(Args a, Py_ssize_t) {   // (dy_a, dy_b, relu_in, x, scale, mean, inv, n, c, hw)
  const Tensor &ga = dev(a[0]), &gb = dev(a[1]), &ri = dev(a[2]), &x = dev(a[3]), &sc = dev(a[4]), &mu = dev(a[5]),
               &inv = dev(a[6]);
  const int n = small(a[7]), c = small(a[8]), hw = small(a[9]);
  Tensor joined = fresh_like(ga), dx = fresh_like(ga), ds = fresh_like(sc), db = fresh_like(sc);
  const Ws ws(ga, sgb_bn_backward_workspace_bytes(n, c, hw));
  ISSUE(sgb_bn_add_relu_backward_f32, f32(x), f32(ga), f32(gb), f32(ri), f32(sc), f32(mu), f32(inv), f32w(joined),
        f32w(dx), f32w(ds), f32w(db), n, c, hw, ws.ptr, ws.bytes, stream());
  return list_of(std::move(joined), std::move(dx), std::move(ds), std::move(db));
}

struct Geometry {   // (n, c, h, w, kh, kw, ph, pw, sh, sw)
  int v[10];
  explicit Geometry(PyObject* tuple) {
    if (!PyTuple_Check(tuple) || PyTuple_GET_SIZE(tuple) != 10) fail(PyExc_TypeError, "pooling geometry: ten integers");
    for (int i = 0; i < 10; ++i) v[i] = small(PyTuple_GET_ITEM(tuple, i));
  }
};
#define GEOM(g) g.v[0], g.v[1], g.v[2], g.v[3], g.v[4], g.v[5], g.v[6], g.v[7], g.v[8], g.v[9]
PyObject* py_pool_forward(Args a, Py_ssize_t) {  // (x, max, geometry, pooled h, pooled w)
  const Tensor& x = dev(a[0]);
  const bool mx = truth(a[1]);
  const Geometry g(a[2]);
  Tensor y = fresh({g.v[0], g.v[1], whole(a[3]), whole(a[4])}, at::kFloat, x);
  if (mx) ISSUE(sgb_maxpool_forward_f32, f32(x), f32w(y), GEOM(g), stream());
  else ISSUE(sgb_avgpool_forward_f32, f32(x), f32w(y), GEOM(g), stream());
  return wrap(std::move(y));
}
PyObject* py_pool_backward(Args a, Py_ssize_t) { // (dy, x, y, max, geometry)
  const Tensor &dy = dev(a[0]), &x = dev(a[1]), &y = dev(a[2]);
  const bool mx = truth(a[3]);
  const Geometry g(a[4]);
  Tensor dx = fresh_like(x);
  if (mx) ISSUE(sgb_maxpool_backward_f32, f32(x), f32(y), f32(dy), f32w(dx), GEOM(g), stream());
  else ISSUE(sgb_avgpool_backward_f32, f32(dy), f32w(dx), GEOM(g), stream());
  return wrap(std::move(dx));
}
PyObject* py_pool_forward_argmax(Args a, Py_ssize_t) {   // (x, geometry, pooled h, pooled w)
  const Tensor& x = dev(a[0]);
  const Geometry g(a[1]);
  const std::array<int64_t, 4> shape{g.v[0], g.v[1], whole(a[2]), whole(a[3])};
  Tensor y = fresh(shape, at::kFloat, x), arg = fresh(shape, at::kByte, x);
  ISSUE(sgb_maxpool_forward_argmax_f32, f32(x), f32w(y), static_cast<unsigned char*>(raww(arg)), GEOM(g), stream());
  PyObject* out = PyTuple_New(2);
  if (!out) throw PyError{};
  PyTuple_SET_ITEM(out, 0, wrap(std::move(y)));
  PyTuple_SET_ITEM(out, 1, wrap(std::move(arg)));
  return out;
}
PyObject* py_pool_backward_argmax(Args a, Py_ssize_t) {  // (dy, argmax, geometry)
  const Tensor &dy = dev(a[0]), &arg = dev(a[1]);
  const Geometry g(a[2]);
  Tensor dx = fresh({g.v[0], g.v[1], g.v[2], g.v[3]}, at::kFloat, dy);
  ISSUE(sgb_maxpool_backward_argmax_f32, f32(dy), static_cast<const unsigned char*>(raw(arg)), f32w(dx), GEOM(g),
        stream());
  return wrap(std::move(dx));
}

// ------------------------------------------------------- multi-tensor / sync
// Pointers and element counts of a list or tuple of tensors.
struct TensorList {
  std::vector<void*> ptrs;
  std::vector<size_t> sizes;
  explicit TensorList(PyObject* o, bool checked = true) {
    PyObject* seq = PySequence_Fast(o, "a sequence of tensors is expected");
    if (!seq) throw PyError{};
    const std::unique_ptr<PyObject, void (*)(PyObject*)> hold(seq, [](PyObject* p) { Py_DECREF(p); });
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
    ptrs.reserve(n);
    sizes.reserve(n);
    for (Py_ssize_t i = 0; i < n; ++i) {
      const Tensor& t = checked ? dev(PySequence_Fast_GET_ITEM(seq, i)) : tensor(PySequence_Fast_GET_ITEM(seq, i));
      ptrs.push_back(raww(t));
      sizes.push_back(count(t));
    }
  }
  size_t n() const { return ptrs.size(); }
};
PyObject* py_sgd_multi(Args a, Py_ssize_t) {
  // (params, grads, moments | None, lr, momentum, dampening, weight decay, nesterov, grad scale)
  const TensorList p(a[0]), g(a[1]);
  const float lr = static_cast<float>(real(a[3])), mom = static_cast<float>(real(a[4])),
              damp = static_cast<float>(real(a[5])), decay = static_cast<float>(real(a[6])),
              scale = static_cast<float>(real(a[8]));
  const int nesterov = truth(a[7]);
  require(g.n() >= p.n(), "one gradient per parameter");
  if (mom != 0.0f) {
    const TensorList m(a[2]);
    require(m.n() >= p.n(), "one momentum buffer per parameter");
    ISSUE(sgb_sgd_update_multi_f32, p.ptrs.data(), g.ptrs.data(), m.ptrs.data(), p.sizes.data(), p.n(), lr, mom, damp,
          decay, nesterov, scale, stream());
  } else {
    ISSUE(sgb_sgd_update_multi_f32, p.ptrs.data(), g.ptrs.data(), nullptr, p.sizes.data(), p.n(), lr, mom, damp, decay,
          nesterov, scale, stream());
  }
  Py_RETURN_NONE;
}
PyObject* py_pack(Args a, Py_ssize_t) {          // (tensors, flat, offset)
  const Tensor& flat = dev(a[1]);
  const TensorList l(a[0]);
  const size_t off = static_cast<size_t>(whole(a[2]));
  if (flat.scalar_type() == at::kFloat)
    ISSUE(sgb_pack_f32, l.ptrs.data(), l.sizes.data(), l.n(), f32w(flat), off, stream());
  else
    ISSUE(sgb_pack_f32_to_f16, l.ptrs.data(), l.sizes.data(), l.n(), raww(flat), off, stream());
  Py_RETURN_NONE;
}
PyObject* py_unpack(Args a, Py_ssize_t) {        // (flat, tensors, offset, scale)
  const Tensor& flat = dev(a[0]);
  const TensorList l(a[1]);
  const size_t off = static_cast<size_t>(whole(a[2]));
  const float scale = static_cast<float>(real(a[3]));
  if (flat.scalar_type() == at::kFloat)
    ISSUE(sgb_unpack_f32, f32(flat), off, l.ptrs.data(), l.sizes.data(), l.n(), scale, stream());
  else
    ISSUE(sgb_unpack_f16_to_f32, raw(flat), off, l.ptrs.data(), l.sizes.data(), l.n(), scale, stream());
  Py_RETURN_NONE;
}
sgb_comm* comm(PyObject* o) { return static_cast<sgb_comm*>(address(o)); }
PyObject* py_comm_synch(Args a, Py_ssize_t) {    // (communicator, tensor)
  const Tensor& t = tensor(a[1]);
  ISSUE(sgb_comm_synch, comm(a[0]), raww(t), count(t), t.scalar_type() == at::kHalf, stream());
  Py_RETURN_NONE;
}
PyObject* py_comm_synch_half(Args a, Py_ssize_t) {
  const Tensor& t = tensor(a[1]);
  require(t.scalar_type() == at::kFloat,
          "only available for 32-bit tensors, which are converted to 16 bits before transmit");
  ISSUE(sgb_comm_synch_half, comm(a[0]), f32w(t), count(t), stream());
  Py_RETURN_NONE;
}
at::ScalarType first_type(PyObject* list) {
  PyObject* first = PySequence_GetItem(list, 0);   // IndexError on an empty list, as ts[0] raises
  if (!first) throw PyError{};
  const std::unique_ptr<PyObject, void (*)(PyObject*)> hold(first, [](PyObject* p) { Py_DECREF(p); });
  return tensor(first).scalar_type();
}
PyObject* py_comm_fused_synch(Args a, Py_ssize_t) {       // (communicator, tensors, send)
  const bool half = first_type(a[1]) == at::kHalf;
  const TensorList l(a[1], false);
  const int send = truth(a[2]);
  ISSUE(sgb_comm_fused_synch, comm(a[0]), l.ptrs.data(), l.sizes.data(), l.n(), half, send, stream());
  Py_RETURN_NONE;
}
PyObject* py_comm_fused_synch_half(Args a, Py_ssize_t) {  // (communicator, tensors, send)
  require(first_type(a[1]) == at::kFloat, "fp32 tensors are expected");
  const TensorList l(a[1], false);
  const int send = truth(a[2]);
  ISSUE(sgb_comm_fused_synch_half, comm(a[0]), l.ptrs.data(), l.sizes.data(), l.n(), send, stream());
  Py_RETURN_NONE;
}
PyObject* py_comm_sparsify(Args a, Py_ssize_t) {  // (communicator, tensors, accumulation | None, spars, topk)
  require(first_type(a[1]) == at::kFloat, "sparsification supports fp32 only");
  const TensorList l(a[1], false);
  float* acc = is_none(a[2]) ? nullptr : f32w(tensor(a[2]));
  const float spars = static_cast<float>(real(a[3]));
  const int topk = truth(a[4]);
  ISSUE(sgb_comm_sparsification, comm(a[0]), l.ptrs.data(), l.sizes.data(), l.n(), acc, spars, topk, stream());
  Py_RETURN_NONE;
}
PyObject* py_comm_sparsify_begin(Args a, Py_ssize_t) {  // as comm_sparsify: the selection half
  require(first_type(a[1]) == at::kFloat, "sparsification supports fp32 only");
  const TensorList l(a[1], false);
  float* acc = is_none(a[2]) ? nullptr : f32w(tensor(a[2]));
  const float spars = static_cast<float>(real(a[3]));
  const int topk = truth(a[4]);
  ISSUE(sgb_comm_sparsification_begin, comm(a[0]), l.ptrs.data(), l.sizes.data(), l.n(), acc, spars, topk, stream());
  Py_RETURN_NONE;
}
PyObject* py_comm_sparsify_buckets(Args a, Py_ssize_t) {  // (communicator, buckets, residuals, threshold) -> done?
  std::vector<void*> ptrs;
  std::vector<size_t> sizes, counts;
  const Py_ssize_t n = PySequence_Size(a[1]);
  if (n < 0) throw PyError{};
  for (Py_ssize_t k = 0; k < n; ++k) {
    const std::unique_ptr<PyObject, void (*)(PyObject*)> bucket(PySequence_GetItem(a[1], k),
                                                                [](PyObject* p) { Py_XDECREF(p); });
    if (!bucket) throw PyError{};
    require(first_type(bucket.get()) == at::kFloat, "sparsification supports fp32 only");
    const TensorList l(bucket.get(), false);
    ptrs.insert(ptrs.end(), l.ptrs.begin(), l.ptrs.end());
    sizes.insert(sizes.end(), l.sizes.begin(), l.sizes.end());
    counts.push_back(l.n());
  }
  const TensorList acc(a[2], false);
  require(acc.n() == counts.size(), "one residual per bucket");
  const float threshold = static_cast<float>(real(a[3]));
  int st = SGB_OK;
  issue("sgb_comm_sparsification_buckets", [&] {
    st = sgb_comm_sparsification_buckets(comm(a[0]), ptrs.data(), sizes.data(), counts.data(),
                                         reinterpret_cast<float* const*>(acc.ptrs.data()), counts.size(), threshold,
                                         stream());
    return st == SGB_ERR_UNSUPPORTED ? SGB_OK : st;
  });
  return PyBool_FromLong(st == SGB_OK);
}
// Tensors that a kernel may take as they are; false otherwise, and the separate
// calls give their own answer.
bool plain_f32(PyObject* seq, const TensorList& l) {
  const Py_ssize_t n = PySequence_Size(seq);
  if (n < 0) throw PyError{};
  if (static_cast<size_t>(n) != l.n()) return false;
  for (Py_ssize_t k = 0; k < n; ++k) {
    PyObject* item = PyList_Check(seq) ? PyList_GET_ITEM(seq, k) : PyTuple_Check(seq) ? PyTuple_GET_ITEM(seq, k) : nullptr;
    if (!item || !THPVariable_Check(item)) return false;
    const Tensor& t = THPVariable_Unpack(item);
    if (t.scalar_type() != at::kFloat || !t.is_cuda() || !t.is_contiguous()) return false;
  }
  return true;
}
struct Hyper {                         // lr, momentum, dampening, weight decay, nesterov, grad scale
  float lr, mom, damp, decay, scale;
  int nesterov;
  explicit Hyper(PyObject* t) {
    if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != 6) fail(PyExc_TypeError, "six hyper-parameters are expected");
    auto v = [&](int k) { return static_cast<float>(real(PyTuple_GET_ITEM(t, k))); };
    lr = v(0);
    mom = v(1);
    damp = v(2);
    decay = v(3);
    nesterov = truth(PyTuple_GET_ITEM(t, 4));
    scale = v(5);
  }
};
// (communicator, params, grads, moments | None, threshold, hyper) -> done?
PyObject* py_comm_update_half(Args a, Py_ssize_t) {
  const TensorList p(a[1], false), g(a[2], false);
  const Hyper h(a[5]);
  std::unique_ptr<TensorList> m;
  if (h.mom != 0.0f) m = std::make_unique<TensorList>(a[3], false);
  bool ok = plain_f32(a[1], p) && plain_f32(a[2], g) && p.sizes == g.sizes && p.n() != 0;
  ok = ok && (!m || (plain_f32(a[3], *m) && m->sizes == p.sizes));
  if (!ok) Py_RETURN_FALSE;
  const double threshold = real(a[4]);
  size_t largest = 0, held = 0;        // of the buckets that a call each would make
  for (const size_t n : g.sizes) {
    if (static_cast<double>(n) > threshold) {
      largest = std::max(largest, n);
      continue;
    }
    held += n;
    largest = std::max(largest, held);
    if (static_cast<double>(held) > threshold) held = 0;
  }
  int st = SGB_OK;
  issue("sgb_comm_update_half", [&] {
    st = sgb_comm_update_half(comm(a[0]), p.ptrs.data(), g.ptrs.data(), m ? m->ptrs.data() : nullptr, g.sizes.data(), g.n(),
                              largest, h.lr, h.mom, h.damp, h.decay, h.nesterov, h.scale, stream());
    return st == SGB_ERR_UNSUPPORTED ? SGB_OK : st;
  });
  return PyBool_FromLong(st == SGB_OK);
}
// (communicator, list of (name, param, grad), bucket threshold, topk) -> worth preparing?
PyObject* py_comm_sparse_update_takes(Args a, Py_ssize_t) {
  if (!PyList_Check(a[1])) Py_RETURN_FALSE;
  const double threshold = real(a[2]);
  const int topk = truth(a[3]);
  if (!topk && PyList_GET_SIZE(a[1]) > SGB_SPARSE_UPDATE_TENSORS) Py_RETURN_FALSE;
  std::vector<void*> ptrs, open;
  std::vector<size_t> sizes, counts, open_sizes;
  size_t held = 0;
  auto flush = [&] {                   // large tensors come before a bucket that is still open
    ptrs.insert(ptrs.end(), open.begin(), open.end());
    sizes.insert(sizes.end(), open_sizes.begin(), open_sizes.end());
    counts.push_back(open.size());
    open.clear();
    open_sizes.clear();
    held = 0;
  };
  for (Py_ssize_t k = 0; k < PyList_GET_SIZE(a[1]); ++k) {
    PyObject* t = PyList_GET_ITEM(a[1], k);
    if (!PyTuple_Check(t) || PyTuple_GET_SIZE(t) != 3 || !THPVariable_Check(PyTuple_GET_ITEM(t, 2))) Py_RETURN_FALSE;
    const Tensor& g = THPVariable_Unpack(PyTuple_GET_ITEM(t, 2));
    if (!g.is_cuda() || g.scalar_type() != at::kFloat) Py_RETURN_FALSE;
    if (static_cast<double>(count(g)) > threshold) {
      ptrs.push_back(raww(g));
      sizes.push_back(count(g));
      counts.push_back(1);
      continue;
    }
    open.push_back(raww(g));
    open_sizes.push_back(count(g));
    held += count(g);
    if (static_cast<double>(held) > threshold) flush();
  }
  if (!open.empty()) flush();
  return PyBool_FromLong(
      sgb_comm_sparse_update_takes(comm(a[0]), ptrs.data(), sizes.data(), counts.data(), counts.size(), topk));
}
// (communicator, buckets, residuals, params, moments | None, spars, topk, hyper) -> done?
PyObject* py_comm_sparse_update(Args a, Py_ssize_t) {
  std::vector<void*> ptrs;
  std::vector<size_t> sizes, counts;
  const Py_ssize_t n = PySequence_Size(a[1]);
  if (n < 0) throw PyError{};
  for (Py_ssize_t k = 0; k < n; ++k) {
    const std::unique_ptr<PyObject, void (*)(PyObject*)> bucket(PySequence_GetItem(a[1], k),
                                                                [](PyObject* p) { Py_XDECREF(p); });
    if (!bucket) throw PyError{};
    const TensorList l(bucket.get(), false);
    if (!plain_f32(bucket.get(), l)) Py_RETURN_FALSE;
    ptrs.insert(ptrs.end(), l.ptrs.begin(), l.ptrs.end());
    sizes.insert(sizes.end(), l.sizes.begin(), l.sizes.end());
    counts.push_back(l.n());
  }
  const TensorList acc(a[2], false), p(a[3], false);
  const float spars = static_cast<float>(real(a[5]));
  const int topk = truth(a[6]);
  const Hyper h(a[7]);
  std::unique_ptr<TensorList> m;
  if (h.mom != 0.0f) m = std::make_unique<TensorList>(a[4], false);
  bool ok = !counts.empty() && acc.n() == counts.size() && plain_f32(a[2], acc) && plain_f32(a[3], p) && p.sizes == sizes;
  ok = ok && (!m || (plain_f32(a[4], *m) && m->sizes == sizes));
  for (size_t k = 0, at = 0; ok && k < counts.size(); ++k) {
    size_t total = 0;
    for (size_t i = 0; i < counts[k]; ++i) total += sizes[at++];
    ok = acc.sizes[k] == total;
  }
  if (!ok) Py_RETURN_FALSE;
  int st = SGB_OK;
  issue("sgb_comm_sparse_update", [&] {
    st = sgb_comm_sparse_update(comm(a[0]), ptrs.data(), sizes.data(), counts.data(),
                                reinterpret_cast<float* const*>(acc.ptrs.data()), counts.size(), spars, topk,
                                p.ptrs.data(), m ? m->ptrs.data() : nullptr, h.lr, h.mom, h.damp, h.decay, h.nesterov,
                                h.scale, stream());
    return st == SGB_ERR_UNSUPPORTED ? SGB_OK : st;
  });
  return PyBool_FromLong(st == SGB_OK);
}
PyObject* py_comm_sparsify_end(Args a, Py_ssize_t) {
  ISSUE(sgb_comm_sparsification_end, comm(a[0]), stream());
  Py_RETURN_NONE;
}
// The dense exchange of a stream of gradients (DistOpt's bucket policy): takes
// (name, param, gradient) triples from an iterator, reduces a gradient above the
// threshold at once and a bucket of smaller ones as soon as it holds more than
// the threshold, while the iterator is still producing the next ones.  Returns
// the names, parameters and gradients as three lists.
PyObject* py_comm_sync_dense(Args a, Py_ssize_t) {   // (communicator, iterable, threshold, half)
  sgb_comm* const c = comm(a[0]);
  const double threshold = real(a[2]);
  const bool half = truth(a[3]);
  using Ref = std::unique_ptr<PyObject, void (*)(PyObject*)>;
  auto drop = [](PyObject* p) { Py_XDECREF(p); };
  const Ref it(PyObject_GetIter(a[1]), drop);
  const Ref names(PyList_New(0), drop), params(PyList_New(0), drop), grads(PyList_New(0), drop);
  if (!it || !names || !params || !grads) throw PyError{};
  std::vector<void*> ptrs;
  std::vector<size_t> sizes;
  size_t held = 0;
  // One rank has nothing to overlap a bucket's rounding with when every
  // gradient exists already: collect the list and round it in one go (161
  // gradients, 25.6e6 elements: 11 launches in 65 us, one in 38).
  bool collect = half && sgb_comm_world_size(c) == 1 &&
                 (Py_TYPE(it.get()) == &PyListIter_Type || Py_TYPE(it.get()) == &PyTupleIter_Type);
  std::vector<void*> all_ptrs;
  std::vector<size_t> all_sizes, ends;                 // `ends`: where each bucket (or large tensor) ends
  size_t largest = 0;
  auto need_f32 = [&](const Tensor& g) {
    require(!half || g.scalar_type() == at::kFloat,
            "only available for 32-bit tensors, which are converted to 16 bits before transmit");
  };
  bool bucket_f16 = false;
  auto flush = [&] {
    if (ptrs.empty()) return;
    if (collect) {
      all_ptrs.insert(all_ptrs.end(), ptrs.begin(), ptrs.end());
      all_sizes.insert(all_sizes.end(), sizes.begin(), sizes.end());
      ends.push_back(all_ptrs.size());
      largest = std::max(largest, held);
    } else for (const int send : {0, 1}) {
      if (half)
        ISSUE(sgb_comm_fused_synch_half, c, ptrs.data(), sizes.data(), ptrs.size(), send, stream());
      else
        ISSUE(sgb_comm_fused_synch, c, ptrs.data(), sizes.data(), ptrs.size(), bucket_f16, send, stream());
    }
    ptrs.clear();
    sizes.clear();
    held = 0;
  };
  while (PyObject* item = PyIter_Next(it.get())) {
    const Ref hold(item, drop);
    const Ref triple(PySequence_Fast(item, "(name, param, grad) triples are expected"), drop);
    if (!triple) throw PyError{};
    if (PySequence_Fast_GET_SIZE(triple.get()) != 3) fail(PyExc_ValueError, "(name, param, grad) triples are expected");
    PyObject** v = PySequence_Fast_ITEMS(triple.get());
    if (PyList_Append(names.get(), v[0]) || PyList_Append(params.get(), v[1]) || PyList_Append(grads.get(), v[2]))
      throw PyError{};
    const Tensor& g = tensor(v[2]);
    need_f32(g);
    const size_t n = count(g);
    if (static_cast<double>(n) > threshold) {
      if (collect) {
        all_ptrs.push_back(raww(g));
        all_sizes.push_back(n);
        ends.push_back(all_ptrs.size());
        largest = std::max(largest, n);
      } else if (half) ISSUE(sgb_comm_synch_half, c, f32w(g), n, stream());
      else ISSUE(sgb_comm_synch, c, raww(g), n, g.scalar_type() == at::kHalf, stream());
      continue;
    }
    if (ptrs.empty()) bucket_f16 = g.scalar_type() == at::kHalf;
    ptrs.push_back(raww(g));
    sizes.push_back(n);
    held += n;
    if (static_cast<double>(held) > threshold) flush();
  }
  if (PyErr_Occurred()) throw PyError{};
  flush();
  if (!all_ptrs.empty()) {
    int st = SGB_OK;
    issue("sgb_comm_round_half", [&] {
      st = sgb_comm_round_half(c, all_ptrs.data(), all_sizes.data(), all_ptrs.size(), largest, stream());
      return st == SGB_ERR_UNSUPPORTED ? SGB_OK : st;
    });
    size_t from = 0;
    if (st == SGB_ERR_UNSUPPORTED)                     // bucket by bucket after all
      for (const size_t end : ends) {
        if (end - from == 1 && static_cast<double>(all_sizes[from]) > threshold)
          ISSUE(sgb_comm_synch_half, c, static_cast<float*>(all_ptrs[from]), all_sizes[from], stream());
        else
          for (const int send : {0, 1})
            ISSUE(sgb_comm_fused_synch_half, c, all_ptrs.data() + from, all_sizes.data() + from, end - from, send,
                  stream());
        from = end;
      }
  }
  PyObject* out = PyTuple_Pack(3, names.get(), params.get(), grads.get());
  if (!out) throw PyError{};
  return out;
}
PyObject* py_comm_wait(Args a, Py_ssize_t) {
  ISSUE(sgb_comm_wait, comm(a[0]), stream());
  Py_RETURN_NONE;
}

// -------------------------------------------------------------- call programs
// A recorded step: C-ABI calls with their arguments converted once.  What
// differs between runs is patched in before each call: the current stream, the
// communicator's result stream (and its number), and three hyper-parameters.
union Slot {
  void* p;
  long long i;
  double d;
};
template <typename T>
Slot to_slot(PyObject* o) {
  Slot s;
  if constexpr (std::is_pointer_v<T>) s.p = address(o);
  else if constexpr (std::is_floating_point_v<T>) s.d = real(o);
  else s.i = whole(o);
  return s;
}
template <typename T>
T from_slot(const Slot& s) {
  if constexpr (std::is_pointer_v<T>) return static_cast<T>(s.p);
  else if constexpr (std::is_floating_point_v<T>) return static_cast<T>(s.d);
  else return static_cast<T>(s.i);
}
struct Callable {
  const char* name;
  size_t arity;
  Slot (*convert)(size_t, PyObject*);
  int (*invoke)(const Slot*);
};
template <auto Fn>
struct Thunk;
template <typename... A, int (*Fn)(A...)>
struct Thunk<Fn> {
  template <size_t... I>
  static int call(const Slot* s, std::index_sequence<I...>) {
    return Fn(from_slot<A>(s[I])...);
  }
  static int invoke(const Slot* s) { return call(s, std::index_sequence_for<A...>{}); }
  static Slot convert(size_t i, PyObject* o) {
    static Slot (*const table[])(PyObject*) = {&to_slot<A>...};
    return table[i](o);
  }
};
#define CALLABLE(fn) \
  Callable { #fn, arity_of(&fn), &Thunk<&fn>::convert, &Thunk<&fn>::invoke }
template <typename... A>
constexpr size_t arity_of(int (*)(A...)) {
  return sizeof...(A);
}
const Callable kCallables[] = {
    CALLABLE(sgb_relu_backward_f32), CALLABLE(sgb_relu_backward_mask_f32), CALLABLE(sgb_add_relu_backward_f32),
    CALLABLE(sgb_add_relu_backward_mask_f32), CALLABLE(sgb_binary_f32), CALLABLE(sgb_scalar_f32),
    CALLABLE(sgb_set_f32), CALLABLE(sgb_bn_backward_f32), CALLABLE(sgb_bn_relu_backward_f32),
    CALLABLE(sgb_bn_relu_backward_mask_f32), CALLABLE(sgb_bn_add_relu_backward_f32),
    CALLABLE(sgb_maxpool_backward_f32), CALLABLE(sgb_maxpool_backward_argmax_f32), CALLABLE(sgb_avgpool_backward_f32),
    CALLABLE(sgb_softmax_rows_f32), CALLABLE(sgb_cross_entropy_f32), CALLABLE(sgb_softmax_cross_entropy_bwd_f32),
    CALLABLE(sgb_softmax_cross_entropy_grad_f32), CALLABLE(sgb_softmax_cross_entropy_fused_f32),
    CALLABLE(sgb_sum_all_f32), CALLABLE(sgb_sum_rows_f32), CALLABLE(sgb_conv_bias_backward_f32),
    CALLABLE(sgb_relu_backward_sum_rows_f32), CALLABLE(sgb_relu_backward_conv_bias_f32),
    CALLABLE(sgb_maxpool_relu_backward_conv_bias_f32), CALLABLE(sgb_loss_head_f32),
    CALLABLE(sgb_unpack_f32), CALLABLE(sgb_sgd_update_multi_f32), CALLABLE(sgb_comm_synch),
    CALLABLE(sgb_comm_synch_half), CALLABLE(sgb_comm_fused_synch), CALLABLE(sgb_comm_fused_synch_half),
    CALLABLE(sgb_comm_sparsification), CALLABLE(sgb_comm_wait), CALLABLE(sgb_comm_profile_mark),
    CALLABLE(sgb_comm_profile_range), CALLABLE(sgb_comm_update_half), CALLABLE(sgb_sgd_update_beside_f32),
    CALLABLE(sgb_comm_wait_captured),
};

enum Patch { kStream, kSideStream, kResultStream, kResultIndex, kLr, kMomentum, kDecay, kPatches };
const char* const kPatchNames[kPatches] = {"STREAM", "SIDE_STREAM", "RESULT_STREAM", "RESULT_INDEX", "LR", "MOMENTUM", "DECAY"};

// When a call of a program is issued: in every run, in timed ones, in runs into a capture,
// in those that are not.  In a capture "fork" and "join" order a side stream behind the main
// one and back, and what a run does there is a branch of the graph.  (One by one, the two
// events of a fork cost the host more than the branch saves.)
enum When { kAlways, kProfiled, kCaptured, kSingle };

constexpr size_t kMaxArguments = 24;
struct Call {
  const Callable* fn;                        // null: a fork or a join
  std::vector<Slot> slots;
  std::vector<std::pair<size_t, int>> patches;
  int when;
  bool join = false;
};
// A side stream and the event that orders it.  It has the priority of ordinary streams,
// which is the lowest there is: what leaves room for the kernels that it runs beside is that
// its own have one block an SM.  A few are kept per device for all programs (one costs more than a millisecond); one that
// takes part in a capture is not lent again before that ends.
struct Side {
  cudaStream_t stream = nullptr;
  cudaEvent_t event = nullptr;
  bool lent = false;
  // Everything of `from` so far, in front of whatever comes to `to`.
  bool order(cudaStream_t from, cudaStream_t to) const {
    return cudaEventRecord(event, from) == cudaSuccess && cudaStreamWaitEvent(to, event, 0) == cudaSuccess;
  }
};
class Sides {
 public:
  // On the current device; null where all are in use.
  static Side* lend() {
    const std::lock_guard<std::mutex> lock(guard());
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return failed();
    auto& sides = all()[device];
    for (const auto& side : sides) {
      cudaStreamCaptureStatus status = cudaStreamCaptureStatusActive;
      if (side->lent) continue;
      if (cudaStreamIsCapturing(side->stream, &status) != cudaSuccess) return failed();
      if (status == cudaStreamCaptureStatusNone) return lent(side.get());
    }
    if (sides.size() == kMost) return nullptr;
    auto side = std::make_unique<Side>();
    if (cudaEventCreateWithFlags(&side->event, cudaEventDisableTiming) != cudaSuccess) return failed();
    if (cudaStreamCreateWithFlags(&side->stream, cudaStreamNonBlocking) != cudaSuccess) {
      cudaEventDestroy(side->event);
      return failed();
    }
    sides.push_back(std::move(side));
    return lent(sides.back().get());
  }
  static void give_back(Side* side) {
    if (!side) return;
    const std::lock_guard<std::mutex> lock(guard());
    side->lent = false;
  }

 private:
  static constexpr size_t kMost = 8;
  static std::mutex& guard() {
    static auto* m = new std::mutex;
    return *m;
  }
  // Never destroyed: the CUDA context may be gone by then.
  static std::map<int, std::vector<std::unique_ptr<Side>>>& all() {
    static auto* m = new std::map<int, std::vector<std::unique_ptr<Side>>>;
    return *m;
  }
  static Side* lent(Side* side) {
    side->lent = true;
    return side;
  }
  static Side* failed() {
    cudaGetLastError();
    return nullptr;
  }
};
// What a recorded step depends on besides its arguments: if this is the same as
// in the run before, so are its launches.
struct Settings {
  double lr, momentum, decay;
  int overlap;
  int device;
  bool operator==(const Settings& o) const {
    return lr == o.lr && momentum == o.momentum && decay == o.decay && overlap == o.overlap && device == o.device;
  }
};
struct Program {
  std::vector<Call> calls;
  sgb_comm* comm = nullptr;
  PyObject* keep = nullptr;   // the argument objects (names stay valid while it lives)
  // A step of small kernels costs the host 1.9 us a launch and the GPU less than
  // that per kernel, so once a program has run twice in a row with the same
  // settings its launches are captured and a run is one graph launch (17 kernels:
  // 32 us launched one by one, 10 us as a graph).  Off for programs whose
  // launches must be made one by one (see HotPathGPU._record_program), while a
  // caller captures, and while the communicator's phases are timed.
  //
  // The settings are part of the launches, so a capture serves only as long as
  // they last, and it costs about as much as kPaysAfter of its replays save (MLP
  // of 8 kernels: 220 us against 6 us a run).  One that was replayed less than
  // that has the next one wait for as many runs, and four times as many each time
  // it happens again: a rate that changes every third run took 85-97 us a run,
  // 14 us launched one by one.
  bool graphable = false;
  Settings seen{};
  unsigned streak = 0;        // runs in a row with `seen`
  unsigned eager = 2;         // of which so many are launched one by one
  unsigned captures = 0;
  cudaGraphExec_t exec = nullptr;
  bool forks = false;         // needs a side stream in a capture
  std::mutex guard;           // of streak, eager, captures, exec, seen
};
constexpr unsigned kEagerRuns = 2, kPaysAfter = 40, kMostEagerRuns = 1u << 16;
const char kProgramTag[] = "singa_b200.program";

void drop_program(PyObject* capsule) {
  auto* p = static_cast<Program*>(PyCapsule_GetPointer(capsule, kProgramTag));
  if (!p) return;
  Py_XDECREF(p->keep);
  if (p->exec) cudaGraphExecDestroy(p->exec);
  delete p;
}

// (list of (function name, argument tuple, when), communicator | None[, graphable]) -> program;
// "fork" and "join" stand for themselves
PyObject* py_program(Args a, Py_ssize_t n) {
  PyObject* seq = PySequence_Fast(a[0], "a list of calls is expected");
  if (!seq) throw PyError{};
  auto prog = std::make_unique<Program>();
  prog->comm = comm(a[1]);
  prog->graphable = n > 2 && truth(a[2]);
  const std::unique_ptr<PyObject, void (*)(PyObject*)> hold(seq, [](PyObject* p) { Py_DECREF(p); });
  for (Py_ssize_t k = 0; k < PySequence_Fast_GET_SIZE(seq); ++k) {
    PyObject* item = PySequence_Fast_GET_ITEM(seq, k);
    const char* name;
    PyObject* args;
    int when;
    if (!PyArg_ParseTuple(item, "sO!i", &name, &PyTuple_Type, &args, &when)) throw PyError{};
    if (when < kAlways || when > kSingle) fail(PyExc_ValueError, "no such time for a call");
    const bool join = !strcmp(name, "join");
    if (join || !strcmp(name, "fork")) {
      prog->calls.push_back(Call{nullptr, {}, {}, kCaptured, join});
      if (!prog->forks) Sides::give_back(Sides::lend());    // made outside captures
      prog->forks = true;
      continue;
    }
    const Callable* fn = nullptr;
    for (const Callable& c : kCallables)
      if (!strcmp(c.name, name)) fn = &c;
    if (!fn) fail(PyExc_ValueError, std::string("no such call in a step: ") + name);
    if (fn->arity > kMaxArguments || static_cast<size_t>(PyTuple_GET_SIZE(args)) != fn->arity)
      fail(PyExc_TypeError, std::string(name) + ": wrong number of arguments");
    Call call{fn, {}, {}, when};
    for (size_t i = 0; i < fn->arity; ++i) {
      PyObject* v = PyTuple_GET_ITEM(args, i);
      Slot s{};
      bool patched = false;
      if (PyUnicode_Check(v)) {
        for (int q = 0; q < kPatches; ++q)
          if (!PyUnicode_CompareWithASCIIString(v, kPatchNames[q])) {
            call.patches.emplace_back(i, q);
            patched = true;
          }
        if (!patched) fail(PyExc_ValueError, std::string(name) + ": unknown placeholder");
      } else {
        s = fn->convert(i, v);
      }
      call.slots.push_back(s);
    }
    prog->calls.push_back(std::move(call));
  }
  prog->keep = same(a[0]);
  PyObject* cap = PyCapsule_New(prog.get(), kProgramTag, drop_program);
  if (!cap) throw PyError{};
  prog.release();
  return cap;
}

// Issues the calls in order on `st`, in a capture with forks to `side`; on a failure `where`
// names the call.
int issue_calls(const Program* prog, const Settings& now, bool profile, void* st, bool captured, const Side* side,
                const char** where) {
  Slot scratch_slots[kMaxArguments];
  for (const Call& c : prog->calls) {
    if (c.when == kProfiled ? !profile : c.when == kCaptured ? !captured : c.when == kSingle && captured) continue;
    if (!c.fn) {
      const cudaStream_t main = static_cast<cudaStream_t>(st);
      if (c.join ? side->order(side->stream, main) : side->order(main, side->stream)) continue;
      *where = c.join ? "join" : "fork";
      return SGB_ERR_CUDA;
    }
    const Slot* slots = c.slots.data();
    if (!c.patches.empty()) {   // patched copies on this thread's stack: a program can run on several threads
      std::copy(c.slots.begin(), c.slots.end(), scratch_slots);
      for (const auto& [i, what] : c.patches) {
        switch (what) {
          case kStream: scratch_slots[i].p = st; break;
          case kSideStream: scratch_slots[i].p = side ? side->stream : st; break;
          case kResultStream: scratch_slots[i].p = sgb_comm_result_stream(prog->comm); break;
          case kResultIndex: {
            void* r = sgb_comm_result_stream(prog->comm);
            int w = 0;
            while (w < 2 && sgb_comm_stream(prog->comm, w) != r) ++w;
            scratch_slots[i].i = w;
            break;
          }
          case kLr: scratch_slots[i].d = now.lr; break;
          case kMomentum: scratch_slots[i].d = now.momentum; break;
          default: scratch_slots[i].d = now.decay;
        }
      }
      slots = scratch_slots;
    }
    const int status = c.fn->invoke(slots);
    if (status != SGB_OK) {
      *where = c.fn->name;
      return status;
    }
  }
  return SGB_OK;
}

// Captures one run on a stream of its own (nothing executes) and instantiates
// it.  False: not possible here; the program then stays with single launches.
bool capture_calls(Program* prog, const Settings& now) {
  cudaStream_t main;
  if (cudaStreamCreateWithFlags(&main, cudaStreamNonBlocking) != cudaSuccess) return false;
  Side* const side = prog->forks ? Sides::lend() : nullptr;
  cudaGraph_t graph = nullptr;
  const char* where = "";
  bool ok = cudaStreamBeginCapture(main, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
  if (ok) {
    ok = issue_calls(prog, now, false, main, !prog->forks || side, side, &where) == SGB_OK;
    ok = cudaStreamEndCapture(main, &graph) == cudaSuccess && ok && graph;
  }
  Sides::give_back(side);
  cudaGraphExec_t exec = nullptr;
  if (ok) ok = cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess;
  if (graph) cudaGraphDestroy(graph);
  cudaStreamDestroy(main);
  if (!ok) {
    cudaGetLastError();      // a refused capture is not an error of the step
    return false;
  }
  if (prog->exec) cudaGraphExecDestroy(prog->exec);
  prog->exec = exec;
  return true;
}

// (program, lr, momentum, weight decay, profile)
PyObject* py_run_program(Args a, Py_ssize_t) {
  auto* prog = static_cast<Program*>(PyCapsule_GetPointer(a[0], kProgramTag));
  if (!prog) throw PyError{};
  const bool profile = truth(a[4]);
  const auto current = c10::cuda::getCurrentCUDAStream();
  const Settings now{real(a[1]), real(a[2]), real(a[3]), sgb_get_option(SGB_OPT_OVERLAP_LAUNCHES),
                     current.device_index()};
  void* const st = current.stream();
  const bool plain = !profile && !sgb_comm_profiling(prog->comm);
  const bool captured = c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
  const bool may_graph = prog->graphable && plain && !captured;
  int status = SGB_OK;
  const char* where = "";
  Py_BEGIN_ALLOW_THREADS;
  bool launched = false;
  if (may_graph) {
    const std::lock_guard<std::mutex> lock(prog->guard);
    if (!(prog->streak && prog->seen == now)) {
      if (prog->streak > prog->eager) {                // there was a capture: did it pay?
        const bool paid = prog->streak - prog->eager >= kPaysAfter;
        prog->eager = paid ? kEagerRuns : std::min(std::max(kPaysAfter, 4 * prog->eager), kMostEagerRuns);
      }
      prog->seen = now;
      prog->streak = 0;
    }
    if (++prog->streak > prog->eager) {
      if (prog->streak == prog->eager + 1) {
        if (capture_calls(prog, now)) ++prog->captures;
        else prog->graphable = false;
      }
      if (prog->graphable) {
        launched = true;
        if (cudaGraphLaunch(prog->exec, static_cast<cudaStream_t>(st)) != cudaSuccess) {
          status = SGB_ERR_CUDA;
          where = "cudaGraphLaunch";
        }
        if (prog->streak > 1u << 30) prog->streak = 1u << 30;
      }
    }
  }
  if (captured && plain) {                             // a caller's capture
    Side* const side = prog->forks ? Sides::lend() : nullptr;
    status = issue_calls(prog, now, profile, st, !prog->forks || side, side, &where);
    Sides::give_back(side);
  } else if (!launched) {
    status = issue_calls(prog, now, profile, st, false, nullptr, &where);
  }
  Py_END_ALLOW_THREADS;
  if (status != SGB_OK) fail_status(where, status);
  Py_RETURN_NONE;
}

PyObject* py_program_captures(Args a, Py_ssize_t) {   // how often the library has captured the program
  auto* prog = static_cast<Program*>(PyCapsule_GetPointer(a[0], kProgramTag));
  if (!prog) throw PyError{};
  const std::lock_guard<std::mutex> lock(prog->guard);
  return PyLong_FromUnsignedLong(prog->captures);
}

// ------------------------------------------------------------------- module
#define METHOD(name, least) \
  { #name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&guarded<py_##name, least>)), METH_FASTCALL, nullptr }
PyMethodDef kMethods[] = {
    METHOD(workspace, 2), METHOD(relu, 1), METHOD(relu_backward, 2), METHOD(add_relu_backward, 3), METHOD(binary, 4), METHOD(scalar, 4),
    METHOD(unary, 3), METHOD(clamp, 4), METHOD(set_value, 2), METHOD(cast, 2), METHOD(axpy, 3), METHOD(sum_rows, 2), METHOD(sum_columns, 2),
    METHOD(row_max, 1), METHOD(sum_all, 1), METHOD(blas1, 2), METHOD(dgmm, 3), METHOD(conv_bias_backward, 1), METHOD(softmax, 2),
    METHOD(ce_forward, 2), METHOD(ce_backward, 2), METHOD(ce_grad, 3), METHOD(softmax_ce_fused, 3), METHOD(bn_forward, 10),
    METHOD(bn_backward, 9), METHOD(bn_add_relu_backward, 10), METHOD(pool_forward, 5), METHOD(pool_backward, 5),
    METHOD(pool_forward_argmax, 4), METHOD(pool_backward_argmax, 3), METHOD(sgd_multi, 9), METHOD(pack, 3), METHOD(unpack, 4),
    METHOD(comm_synch, 2), METHOD(comm_synch_half, 2), METHOD(comm_fused_synch, 3), METHOD(comm_fused_synch_half, 3),
    METHOD(comm_sparsify, 5), METHOD(comm_sparsify_begin, 5), METHOD(comm_sparsify_end, 1), METHOD(comm_sparsify_buckets, 4), METHOD(comm_sync_dense, 4), METHOD(comm_update_half, 6), METHOD(comm_sparse_update, 8), METHOD(comm_sparse_update_takes, 4), METHOD(comm_wait, 1), METHOD(program, 2), METHOD(run_program, 5), METHOD(program_captures, 1),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&kModule); }
