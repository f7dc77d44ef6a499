// Row softmax, per-sample cross entropy and the softmax-cross-entropy gradient.
// The problems on this path are small (batch x classes = 32x1000 ... 256x10),
// so the point of these kernels is to be ONE launch each with few serial steps,
// and to fold the 1/batch scaling into the gradient instead of a clone + edit +
// scale sequence.
//
// A row is read from memory once and stays in registers: its maximum, its sum
// of exponentials and the result come from there (three passes over the row and
// two evaluations of exp per element before: 4.0 us at 256 x 1000).  32 to 1024
// threads work on a row, each with at most 32 elements; short rows share a CTA.
// Rows beyond 32768 elements are re-read instead.
#include <float.h>

#include <type_traits>

#include "common.cuh"
#include "reduce.cuh"

namespace sgb {
namespace {

constexpr int kBlock = 128;

__device__ __forceinline__ float as_float(float v) { return v; }
__device__ __forceinline__ float as_float(__half v) { return __half2float(v); }
__device__ __forceinline__ void put(float* p, float v) { *p = v; }
__device__ __forceinline__ void put(__half* p, float v) { *p = __float2half_rn(v); }

// Sum / maximum over the T threads that share a row; T = 32: a warp, else a CTA.
template <int T, bool MAX>
__device__ __forceinline__ float row_reduce(float v, float* sm) {
  v = MAX ? warp_max(v) : warp_sum(v);
  if (T == 32) return v;
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = v;
  __syncthreads();
  constexpr int kWarps = T / 32;
  const int lane = threadIdx.x & 31;
  v = lane < kWarps ? sm[lane] : (MAX ? -INFINITY : 0.0f);
  return MAX ? warp_max(v) : warp_sum(v);
}
// The sum over twice as many threads: this one stands for itself (a) and for the one T
// further on (b).
template <int T>
__device__ __forceinline__ float row_sum_of_two(float a, float b, float* sm) {
  static_assert(T == 512, "32 partial sums");
  a = warp_sum(a);
  b = warp_sum(b);
  if ((threadIdx.x & 31) == 0) {
    sm[threadIdx.x >> 5] = a;
    sm[(threadIdx.x >> 5) + T / 32] = b;
  }
  __syncthreads();
  return warp_sum(sm[threadIdx.x & 31]);
}

// One row in registers: NV vectors of kL elements per thread.
template <typename V, int T, int NV>
struct Row {
  static constexpr int kL = 16 / sizeof(V);
  // 512 threads with eight vectors add up in the order of 1024 with four, which have the
  // same row where there are fewer (by_length): a row's bits do not depend on the others.
  static constexpr bool kOfTwo = T == 512 && NV == 8;
  float v[NV][kL];
  float sum;

  // Element j of vector k of thread t.  Rows that are not whole vectors are read
  // one element per access, and then neighbouring lanes take neighbouring
  // elements (with the vector order a lane's accesses were kL elements apart:
  // an fp16 head of 953 x 12882 took 112 us instead of 72).
  __device__ __forceinline__ static size_t at(int k, int j, int t, bool vec) {
    return vec ? (static_cast<size_t>(k) * T + t) * kL + j : (static_cast<size_t>(k) * kL + j) * T + t;
  }

  // Loads the row and turns it into exp(x - max); `vec`: 16-byte accesses.
  __device__ __forceinline__ void softmax(const V* __restrict__ x, size_t ncol, bool vec, int t, float* sm) {
    float m = -INFINITY;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      if (vec) {                                   // ncol is a whole number of vectors
        union {
          uint4 u;
          V e[kL];
        } q;
        const size_t i = at(k, 0, t, true);
        if (i < ncol) q.u = ld128(x + i);
#pragma unroll
        for (int j = 0; j < kL; ++j) v[k][j] = i < ncol ? as_float(q.e[j]) : -INFINITY;
      } else {
#pragma unroll
        for (int j = 0; j < kL; ++j) {
          const size_t i = at(k, j, t, false);
          v[k][j] = i < ncol ? as_float(x[i]) : -INFINITY;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int j = 0; j < kL; ++j) m = fmaxf(m, v[k][j]);
    m = row_reduce<T, true>(m, sm);
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int j = 0; j < kL; ++j) {
        v[k][j] = at(k, j, t, vec) < ncol ? expf(v[k][j] - m) : 0.0f;
        if (!kOfTwo) s += v[k][j];
      }
    if constexpr (kOfTwo) {
      float of[2] = {0.f, 0.f};
      if (vec) {                                   // every second vector is the other thread's
#pragma unroll
        for (int k = 0; k < NV; ++k)
#pragma unroll
          for (int j = 0; j < kL; ++j) of[k & 1] += v[k][j];
      } else {                                     // every second element
#pragma unroll
        for (int k = 0; k < NV; ++k)
#pragma unroll
          for (int j = 0; j < kL; ++j) of[j & 1] += v[k][j];
      }
      sum = row_sum_of_two<T>(of[0], of[1], sm + 32);
    } else {
      sum = row_reduce<T, false>(s, sm + 32);
    }
  }
  __device__ __forceinline__ static void store(V* __restrict__ y, size_t ncol, bool vec, int k, int t,
                                               const float (&e)[kL]) {
    if (vec) {
      union {
        uint4 u;
        V e[kL];
      } q;
#pragma unroll
      for (int j = 0; j < kL; ++j) put(&q.e[j], e[j]);
      const size_t i = at(k, 0, t, true);
      if (i < ncol) st128(y + i, q.u);
    } else {
#pragma unroll
      for (int j = 0; j < kL; ++j) {
        const size_t i = at(k, j, t, false);
        if (i < ncol) put(y + i, e[j]);
      }
    }
  }
};

// expf and the division are the full-precision forms (the "accurate" softmax
// mode); fp16 rows are computed in fp32 with one rounding on store.
template <typename V, int T, int NV>
__global__ void __launch_bounds__(T == 32 ? 128 : T, T == 32 ? 8 : 1024 / T)
softmax_rows_kernel(const V* __restrict__ x, V* __restrict__ y, size_t nrow, size_t ncol, bool vec) {
  __shared__ float sm[64];
  dependency_wait();
  release_dependents();
  const size_t row = T == 32 ? blockIdx.x * 4ull + (threadIdx.x >> 5) : blockIdx.x;
  const int t = T == 32 ? threadIdx.x & 31 : threadIdx.x;
  if (row >= nrow) return;
  Row<V, T, NV> r;
  r.softmax(x + row * ncol, ncol, vec, t, sm);
#pragma unroll
  for (int k = 0; k < NV; ++k) {
#pragma unroll
    for (int j = 0; j < Row<V, T, NV>::kL; ++j) r.v[k][j] = r.v[k][j] / r.sum;
    r.store(y + row * ncol, ncol, vec, k, t, r.v[k]);
  }
}

// The whole loss head for integer targets in one launch: row softmax, the
// sample's loss -log(max(p[t], FLT_MIN)) and the scaled gradient
// (p - onehot) * scale.  Every value is formed by the same fp32 operations as
// in the separate kernels, so results are identical bit for bit.
template <int T, int NV>
__global__ void __launch_bounds__(T == 32 ? 128 : T, T == 32 ? 8 : 1024 / T)
softmax_ce_fused_kernel(const float* __restrict__ x, const int* __restrict__ tgt, float* __restrict__ prob,
                        float* __restrict__ loss, float* __restrict__ grad, size_t nrow, size_t ncol, float scale,
                        bool vec) {
  __shared__ float sm[64];
  dependency_wait();
  release_dependents();
  const size_t row = T == 32 ? blockIdx.x * 4ull + (threadIdx.x >> 5) : blockIdx.x;
  const int t = T == 32 ? threadIdx.x & 31 : threadIdx.x;
  if (row >= nrow) return;
  // a label out of range is no slot's number: the threads hold more slots than the row has elements
  const int label = tgt[row];
  const bool known = label >= 0 && static_cast<size_t>(label) < ncol;
  const size_t hot = known ? static_cast<size_t>(label) : ~size_t{0};
  if (!known && t == 0) loss[row] = __int_as_float(0x7fc00000);        // NaN, not stale memory
  Row<float, T, NV> r;
  r.softmax(x + row * ncol, ncol, vec, t, sm);
#pragma unroll
  for (int k = 0; k < NV; ++k) {
#pragma unroll
    for (int j = 0; j < 4; ++j) r.v[k][j] = r.v[k][j] / r.sum;
    if (prob) r.store(prob + row * ncol, ncol, vec, k, t, r.v[k]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float g = r.v[k][j];
      if (r.at(k, j, t, vec) == hot) {
        loss[row] = -logf(fmaxf(g, FLT_MIN));
        g = g - 1.0f;
      }
      r.v[k][j] = g * scale;
    }
    r.store(grad + row * ncol, ncol, vec, k, t, r.v[k]);
  }
}

// Rows too long for registers: three passes over the row.
template <typename V>
__global__ void __launch_bounds__(1024)
softmax_long_kernel(const V* __restrict__ x, V* __restrict__ y, size_t ncol) {
  __shared__ float sm[64];
  dependency_wait();
  release_dependents();
  const V* xr = x + blockIdx.x * ncol;
  V* yr = y + blockIdx.x * ncol;
  float m = -INFINITY;
  for (size_t c = threadIdx.x; c < ncol; c += 1024) m = fmaxf(m, as_float(xr[c]));
  m = row_reduce<1024, true>(m, sm);
  float s = 0.f;
  for (size_t c = threadIdx.x; c < ncol; c += 1024) s += expf(as_float(xr[c]) - m);
  s = row_reduce<1024, false>(s, sm + 32);
  for (size_t c = threadIdx.x; c < ncol; c += 1024) put(yr + c, expf(as_float(xr[c]) - m) / s);
}
__global__ void __launch_bounds__(1024)
softmax_ce_long_kernel(const float* __restrict__ x, const int* __restrict__ t, float* __restrict__ prob,
                       float* __restrict__ loss, float* __restrict__ grad, size_t ncol, float scale) {
  __shared__ float sm[64];
  dependency_wait();
  release_dependents();
  const size_t row = blockIdx.x;
  const float* xr = x + row * ncol;
  float m = -INFINITY;
  for (size_t c = threadIdx.x; c < ncol; c += 1024) m = fmaxf(m, xr[c]);
  m = row_reduce<1024, true>(m, sm);
  float s = 0.f;
  for (size_t c = threadIdx.x; c < ncol; c += 1024) s += expf(xr[c] - m);
  s = row_reduce<1024, false>(s, sm + 32);
  const size_t hot = static_cast<size_t>(t[row]);
  if (hot >= ncol && threadIdx.x == 0) loss[row] = __int_as_float(0x7fc00000);
  for (size_t c = threadIdx.x; c < ncol; c += 1024) {
    const float p = expf(xr[c] - m) / s;
    if (prob) prob[row * ncol + c] = p;
    float g = p;
    if (c == hot) {
      g = g - 1.0f;
      loss[row] = -logf(fmaxf(p, FLT_MIN));
    }
    grad[row * ncol + c] = g * scale;
  }
}

// Threads per row and vectors per thread: a warp up to 512 elements (no barrier at
// all), then the smallest CTA whose threads hold the row with four vectors each.  A CTA of
// 1024 threads has its SM to itself, so where there are more rows than SMs half the threads
// take eight vectors each: one row's sums overlap another's loads, and twice the bytes are
// in flight, with the same additions in the same order (us, 517 rows of 12384 24.0 -> 17.9, with
// loss and gradient 29.5 -> 24.4, 149 11.4 -> 9.0, 1000 of 16000 40.6 -> 31.6, 400 of 8194 16.9 ->
// 13.5; shorter rows, of which an SM holds several anyhow, lost: 4096 of 3000 26.5 -> 32.0, 297
// of 6000 7.9 -> 10.1).  F is called with the two constants.
template <typename V, typename F>
int by_length(size_t nrow, size_t ncol, F f) {
  constexpr size_t kL = 16 / sizeof(V);
  const size_t vecs = ceil_div(ncol, kL);
#define SGB_ROW(T, NV)                                                            \
  if (vecs <= static_cast<size_t>(T) * (NV)) return f(std::integral_constant<int, T>{}, std::integral_constant<int, NV>{});
  SGB_ROW(32, 1)
  SGB_ROW(32, 2)
  SGB_ROW(32, 4)
  SGB_ROW(128, 2)
  SGB_ROW(128, 4)
  SGB_ROW(256, 4)
  SGB_ROW(512, 4)
  if constexpr (kL == 4) {
    if (nrow > static_cast<size_t>(sm_count())) { SGB_ROW(512, 8) }
  }
  SGB_ROW(1024, 4)
  if constexpr (kL == 4) { SGB_ROW(1024, 8) }
#undef SGB_ROW
  return -1000;          // longer
}

template <typename V>
int softmax_rows(const V* x, V* y, size_t nrow, size_t ncol, void* stream) {
  if (nrow == 0 || ncol == 0) return SGB_OK;
  if (!x || !y) return SGB_ERR_NULL;
  if (nrow > 0x7fffffffu) return SGB_ERR_SIZE;
  const bool vec = ncol % (16 / sizeof(V)) == 0 && aligned16(x) && aligned16(y);
  const int st = by_length<V>(nrow, ncol, [&](auto T, auto NV) {
    constexpr int kT = decltype(T)::value, kNV = decltype(NV)::value;
    const unsigned grid = static_cast<unsigned>(kT == 32 ? ceil_div(nrow, 4) : nrow);
    return launch_ex(softmax_rows_kernel<V, kT, kNV>, dim3(grid), dim3(kT == 32 ? 128 : kT), 0, as_stream(stream), 0,
                     true, x, y, nrow, ncol, vec);
  });
  if (st != -1000) return st;
  return launch_ex(softmax_long_kernel<V>, dim3(static_cast<unsigned>(nrow)), dim3(1024), 0, as_stream(stream), 0, true,
                   x, y, ncol);
}

// loss[i] = -log(max(p[i, t[i]], FLT_MIN)) or the weighted form for array
// targets; one thread per sample like the reference (batch is small).
__global__ void ce_fwd_kernel(int int_target, size_t batch, size_t dim,
                              const float* __restrict__ p, const int* __restrict__ t,
                              float* __restrict__ loss) {
  dependency_wait();
  release_dependents();
  size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (i >= batch) return;
  if (int_target) {
    // a label outside [0, dim) reads nothing: the sample's loss is NaN
    const int ti = t[i];
    if (static_cast<unsigned>(ti) >= dim) {
      loss[i] = __int_as_float(0x7fc00000);
      return;
    }
    float pt = p[i * dim + ti];
    loss[i] = -logf(fmaxf(pt, FLT_MIN));
  } else {
    float sum = 0.f;
    for (size_t j = 0; j < dim; ++j) sum += t[i * dim + j];
    float l = 0.f;
    for (size_t j = 0; j < dim; ++j)
      l -= t[i * dim + j] / sum * logf(fmaxf(p[i * dim + j], FLT_MIN));
    loss[i] = l;
  }
}

// grad = (p - onehot) * scale over the flattened matrix, one 16-byte vector
// per thread whatever the row length is (a vector lies in at most two rows);
// with SCALE == false the multiply is skipped, so the values equal the
// reference's in-place kernel bit for bit, with SCALE the extra multiply is
// the same fp32 product the reference forms in its separate "dx /= batch" pass.
// VEC: the pointers are aligned and a row is at least a vector long.
__device__ __forceinline__ float less_one(float v) { return v - 1.0f; }
__device__ __forceinline__ __half less_one(__half v) { return __hsub(v, __int2half_rn(1)); }
template <typename V, bool SCALE, bool VEC>
__global__ void __launch_bounds__(256)
ce_bwd_int_kernel(size_t dim, size_t total, const V* __restrict__ p, const int* __restrict__ t, V* __restrict__ grad,
                  float scale) {
  constexpr int kL = VEC ? 16 / sizeof(V) : 1;
  dependency_wait();
  release_dependents();
  const size_t i = (blockIdx.x * 256ull + threadIdx.x) * kL;
  if (i >= total) return;
  const size_t row = total <= 0xffffffffu ? static_cast<unsigned>(i) / static_cast<unsigned>(dim) : i / dim;
  const size_t c = i - row * dim;
  // where this row's and the next row's target lie, counted from this vector's row start
  const size_t hot = static_cast<size_t>(t[row]);
  size_t hot_next = static_cast<size_t>(-1);
  if (VEC && c + kL > dim && i + (dim - c) < total) {
    const unsigned next = static_cast<unsigned>(t[row + 1]);
    if (next < dim) hot_next = dim + next;
  }
  const bool whole = i + kL <= total;
  union {
    uint4 u;
    V e[kL];
  } q;
  if (VEC && whole) {
    q.u = ld128(p + i);
  } else {
#pragma unroll
    for (int j = 0; j < kL; ++j) q.e[j] = i + j < total ? p[i + j] : p[i];
  }
#pragma unroll
  for (int j = 0; j < kL; ++j) {
    if ((c + j < dim && c + j == hot) || (VEC && c + j == hot_next)) q.e[j] = less_one(q.e[j]);
    if (SCALE) q.e[j] = static_cast<V>(static_cast<float>(q.e[j]) * scale);   // fp32 only
  }
  if (VEC && whole) {
    st128(grad + i, q.u);
  } else {
#pragma unroll
    for (int j = 0; j < kL; ++j)
      if (i + j < total) grad[i + j] = q.e[j];
  }
}
template <typename V, bool SCALE>
int ce_bwd_int(size_t batch, size_t dim, const V* p, const int* t, V* grad, float scale, void* stream) {
  constexpr size_t kL = 16 / sizeof(V);
  const bool vec = dim >= kL && aligned16(p) && aligned16(grad);
  const size_t total = batch * dim, work = vec ? ceil_div(total, kL) : total;
  if (ceil_div(work, 256) > 0x7fffffffu) return SGB_ERR_SIZE;
  return launch_ex(vec ? ce_bwd_int_kernel<V, SCALE, true> : ce_bwd_int_kernel<V, SCALE, false>,
                   dim3(static_cast<unsigned>(ceil_div(work, 256))), dim3(256), 0, as_stream(stream), 0, true, dim, total,
                   p, t, grad, scale);
}

// The same for array targets (weights normalised per row), one CTA per sample row.
template <bool SCALE>
__global__ void __launch_bounds__(kBlock)
ce_bwd_array_kernel(size_t dim, const float* __restrict__ p, const int* __restrict__ t, float* __restrict__ grad,
                    float scale) {
  __shared__ float sm[32];
  dependency_wait();
  release_dependents();
  const size_t row = blockIdx.x;
  const float* pr = p + row * dim;
  float* gr = grad + row * dim;
  const int* tr = t + row * dim;
  // the reference adds the integer weights serially in fp32; sums of small
  // integers are exact in any order
  float part = 0.f;
  for (size_t j = threadIdx.x; j < dim; j += kBlock) part += tr[j];
  const float sum = block_sum(part, sm);
  for (size_t j = threadIdx.x; j < dim; j += kBlock) {
    float g = pr[j] - tr[j] / sum;
    gr[j] = SCALE ? g * scale : g;
  }
}
template <bool SCALE>
int ce_bwd(int int_target, size_t batch, size_t dim, const float* p, const int32_t* t, float scale, float* grad,
           void* stream) {
  if (batch == 0 || dim == 0) return SGB_OK;
  if (!p || !t || !grad) return SGB_ERR_NULL;
  if (batch > 0x7fffffffu) return SGB_ERR_SIZE;
  if (int_target) return ce_bwd_int<float, SCALE>(batch, dim, p, t, grad, scale, stream);
  return launch_ex(ce_bwd_array_kernel<SCALE>, dim3(static_cast<unsigned>(batch)), dim3(kBlock), 0, as_stream(stream), 0,
                   true, dim, p, t, grad, scale);
}

// ------------------------------------------------------------------- fp16
// fp16 cross entropy with the arithmetic of the fp16 kernel it replaces: all
// steps in half precision, probabilities floored at half(1e-7), integer
// weights converted with round-down, the per-sample sums formed serially.
__global__ void ce_fwd_f16_kernel(int int_target, size_t batch, size_t dim,
                                  const __half* __restrict__ p, const int* __restrict__ t,
                                  __half* __restrict__ loss) {
  dependency_wait();
  release_dependents();
  size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (i >= batch) return;
  const __half eps = __float2half_rn(0.0000001f);
  if (int_target) {
    const int ti = t[i];
    if (static_cast<unsigned>(ti) >= dim) {      // label out of range: NaN, no read
      loss[i] = __ushort_as_half(0x7e00);
      return;
    }
    const __half pt = p[i * dim + ti];
    loss[i] = __hneg(hlog(__hgt(pt, eps) ? pt : eps));
  } else {
    __half sum = __float2half_rn(0.f);
    for (size_t j = 0; j < dim; ++j) sum = __hadd(sum, __int2half_rd(t[i * dim + j]));
    __half l = __float2half_rn(0.f);
    for (size_t j = 0; j < dim; ++j) {
      const __half pj = p[i * dim + j];
      l = __hsub(l, __hmul(__hdiv(__int2half_rd(t[i * dim + j]), sum), hlog(__hgt(pj, eps) ? pj : eps)));
    }
    loss[i] = l;
  }
}

// grad = p - target in half precision for array targets; one CTA per sample
// row.  The integer weights are small, so their half sum is exact in any order
// as long as it stays below 2048.
__global__ void __launch_bounds__(kBlock)
ce_bwd_array_f16_kernel(size_t dim, const __half* __restrict__ p, const int* __restrict__ t, __half* __restrict__ grad) {
  __shared__ __half total;
  dependency_wait();
  release_dependents();
  const size_t row = blockIdx.x;
  const __half* pr = p + row * dim;
  __half* gr = grad + row * dim;
  const int* tr = t + row * dim;
  if (threadIdx.x == 0) {
    __half sum = __float2half_rn(0.f);
    for (size_t j = 0; j < dim; ++j) sum = __hadd(sum, __int2half_rd(tr[j]));
    total = sum;
  }
  __syncthreads();
  for (size_t j = threadIdx.x; j < dim; j += kBlock)
    gr[j] = __hsub(pr[j], __hdiv(__int2half_rd(tr[j]), total));
}

}  // namespace
}  // namespace sgb

using namespace sgb;

extern "C" {

int sgb_softmax_rows_f32(const float* x, float* y, size_t nrow, size_t ncol, void* stream) {
  return softmax_rows<float>(x, y, nrow, ncol, stream);
}

int sgb_cross_entropy_f32(int int_target, size_t batch, size_t dim, const float* p,
                          const int32_t* t, float* loss, void* stream) {
  if (batch == 0) return SGB_OK;
  if (!p || !t || !loss) return SGB_ERR_NULL;
  if (dim == 0) return SGB_ERR_SIZE;
  return launch_ex(ce_fwd_kernel, dim3(static_cast<unsigned>(ceil_div(batch, 128))), dim3(128), 0, as_stream(stream), 0,
                   true, int_target, batch, dim, p, t, loss);
}

int sgb_softmax_cross_entropy_bwd_f32(int int_target, size_t batch, size_t dim, const float* p,
                                      const int32_t* t, float* grad, void* stream) {
  return ce_bwd<false>(int_target, batch, dim, p, t, 1.0f, grad, stream);
}

int sgb_softmax_cross_entropy_grad_f32(int int_target, size_t batch, size_t dim, const float* p,
                                       const int32_t* t, float scale, float* grad, void* stream) {
  return ce_bwd<true>(int_target, batch, dim, p, t, scale, grad, stream);
}

int sgb_softmax_cross_entropy_fused_f32(const float* logits, const int32_t* t, size_t batch, size_t dim,
                                        float scale, float* prob, float* loss, float* grad,
                                        void* stream) {
  if (batch == 0 || dim == 0) return SGB_OK;
  if (!logits || !t || !loss || !grad) return SGB_ERR_NULL;
  if (batch > 0x7fffffffu) return SGB_ERR_SIZE;
  const bool vec = dim % 4 == 0 && aligned16(logits) && (!prob || aligned16(prob)) && aligned16(grad);
  const int st = by_length<float>(batch, dim, [&](auto T, auto NV) {
    constexpr int kT = decltype(T)::value, kNV = decltype(NV)::value;
    const unsigned grid = static_cast<unsigned>(kT == 32 ? ceil_div(batch, 4) : batch);
    return launch_ex(softmax_ce_fused_kernel<kT, kNV>, dim3(grid), dim3(kT == 32 ? 128 : kT), 0, as_stream(stream), 0,
                     true, logits, t, prob, loss, grad, batch, dim, scale, vec);
  });
  if (st != -1000) return st;
  return launch_ex(softmax_ce_long_kernel, dim3(static_cast<unsigned>(batch)), dim3(1024), 0, as_stream(stream), 0, true,
                   logits, t, prob, loss, grad, dim, scale);
}

int sgb_loss_head_f32(const float* logits, const int32_t* t, size_t batch, size_t dim, float scale, float* prob,
                      float* loss, float* grad, float* total, float* bias_grad, void* ws, size_t ws_bytes, void* stream) {
  int st = sgb_softmax_cross_entropy_fused_f32(logits, t, batch, dim, scale, prob, loss, grad, stream);
  if (st != SGB_OK) return st;
  if (batch && dim && total && bias_grad)
    return sum_rows_beside_total(grad, bias_grad, batch, dim, loss, total, ws, ws_bytes, stream);
  st = sgb_sum_all_f32(loss, total, batch, ws, ws_bytes, stream);
  return st != SGB_OK ? st : sgb_sum_rows_f32(grad, bias_grad, batch, dim, ws, ws_bytes, stream);
}

int sgb_softmax_rows_f16(const void* x, void* y, size_t nrow, size_t ncol, void* stream) {
  return softmax_rows<__half>(static_cast<const __half*>(x), static_cast<__half*>(y), nrow, ncol, stream);
}

int sgb_cross_entropy_f16(int int_target, size_t batch, size_t dim, const void* p, const int32_t* t,
                          void* loss, void* stream) {
  if (batch == 0) return SGB_OK;
  if (!p || !t || !loss) return SGB_ERR_NULL;
  if (dim == 0) return SGB_ERR_SIZE;
  return launch_ex(ce_fwd_f16_kernel, dim3(static_cast<unsigned>(ceil_div(batch, 128))), dim3(128), 0,
                   as_stream(stream), 0, true, int_target, batch, dim, static_cast<const __half*>(p), t,
                   static_cast<__half*>(loss));
}

int sgb_softmax_cross_entropy_bwd_f16(int int_target, size_t batch, size_t dim, const void* p,
                                      const int32_t* t, void* grad, void* stream) {
  if (batch == 0 || dim == 0) return SGB_OK;
  if (!p || !t || !grad) return SGB_ERR_NULL;
  if (batch > 0x7fffffffu) return SGB_ERR_SIZE;
  if (int_target)
    return ce_bwd_int<__half, false>(batch, dim, static_cast<const __half*>(p), t, static_cast<__half*>(grad), 1.0f,
                                     stream);
  return launch_ex(ce_bwd_array_f16_kernel, dim3(static_cast<unsigned>(batch)), dim3(kBlock), 0, as_stream(stream), 0,
                   true, dim, static_cast<const __half*>(p), t, static_cast<__half*>(grad));
}

}  // extern "C"
