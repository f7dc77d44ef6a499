// Reductions of the backward path: bias gradients (column sums of a row-major
// matrix), row sums, per-channel sums of an NCHW tensor (convolution bias
// gradient), the scalar sum behind SumAll and the per-row maximum.
//
// All sums are formed in a fixed order (per-thread strided accumulation, warp
// shuffles, then a fixed-order combine of per-CTA partials), so results are
// identical from run to run; none uses atomics.
#include <cooperative_groups.h>
#include <float.h>

#include "common.cuh"
#include "reduce.cuh"

namespace cg = cooperative_groups;

namespace sgb {
namespace {

constexpr int kBlock = 256;
constexpr int kWarps = kBlock / 32;
constexpr int kMaxCluster = 8;

// A second, small sum (SumAll of at most kBlock * 16 elements) that rides in a grid.
struct Beside {
  const float* x;
  float* out;
  size_t n;
};
// Part `part` of `parts` of the sum of x (grid-stride), by one CTA.  sm: 32 floats.
__device__ __forceinline__ void cta_total(const float* x, float* out, size_t n, size_t parts, size_t part, float* sm) {
  float acc = 0.f;
#pragma unroll 8
  for (size_t i = part * kBlock + threadIdx.x; i < n; i += parts * kBlock) acc += x[i];
  acc = block_sum(acc, sm);
  if (threadIdx.x == 0) *out = acc;
}

// ---------------------------------------------------------------- column sums
// v[c] = sum_r M[r][c].  A CTA owns a block of adjacent columns and a slice of
// the rows; its 8 warps stride over the rows.  A lane owns one column (or four
// adjacent ones, VEC); matrices narrower than a warp put 32 / width rows side
// by side in a warp (`shift` = log2 of the lanes per row).  Eight loads per
// lane are in flight.  The slices of a column block are the CTAs of one
// thread-block cluster: their partial sums meet in the first CTA's shared
// memory and are added in rank order, so a call is one launch (it was two: the
// problems here are a few microseconds, a launch is half of that).  With more
// slices than a cluster holds, the CTAs leave partial rows in `out` and
// colsum_finish_kernel adds them.
//
// RELU: M is the gradient behind a ReLU with input `x`; what is summed is the
// gradient in front of it, which is also written to `dx` (every element passes
// through exactly one lane).  The terms and their order are those of the two
// calls it stands for, so the sums are the same bits.  256x4096: 6.9 us in two
// calls, 4.6 in one; 64x32x24x24 (channels): 5.3 and 4.0.
template <bool VEC, bool RELU>
__global__ void __launch_bounds__(kBlock, 4)
colsum_kernel(const float* __restrict__ M, const float* __restrict__ x, float* __restrict__ dx, float* __restrict__ out, size_t nrow, size_t ncol, size_t rows_per_slice,
              int slices, int shift, bool clustered, const Beside beside) {
  constexpr int kW = VEC ? 4 : 1;
  __shared__ float sm[kWarps][32 * kW];
  __shared__ float part[kMaxCluster][32 * kW];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const size_t block = blockIdx.x / slices;
  const int slice = static_cast<int>(blockIdx.x - block * slices);
  if (!RELU && beside.x && block + 1 == gridDim.x / slices) {   // the last block (a cluster of its own)
    dependency_wait();
    release_dependents();
    if (slice == 0) cta_total(beside.x, beside.out, beside.n, 1, 0, &sm[0][0]);
    return;
  }
  const int lanes = 1 << shift, rows_abreast = 32 >> shift;
  const size_t c = (block * lanes + (lane & (lanes - 1))) * kW;
  const size_t r0 = slice * rows_per_slice;
  const size_t r1 = r0 + rows_per_slice < nrow ? r0 + rows_per_slice : nrow;
  const size_t step = static_cast<size_t>(kWarps) * rows_abreast;
  constexpr int kBatch = RELU ? 4 : 8;                 // two operands: half the loads of each
  float acc[kW];
#pragma unroll
  for (int k = 0; k < kW; ++k) acc[k] = 0.f;
  auto keep4 = [&](float4& v, const float4& m, size_t at) {
    v.x = m.x > 0.f ? v.x : 0.f;
    v.y = m.y > 0.f ? v.y : 0.f;
    v.z = m.z > 0.f ? v.z : 0.f;
    v.w = m.w > 0.f ? v.w : 0.f;
    *reinterpret_cast<float4*>(dx + at) = v;
  };
  auto keep1 = [&](float& v, float m, size_t at) {
    v = m > 0.f ? v : 0.f;
    dx[at] = v;
  };
  if (RELU && c < ncol) {
    size_t r = r0 + w * rows_abreast + (lane >> shift);
#pragma unroll
    for (int k = 0; k < kBatch; ++k)
      if (r + k * step < r1) prefetch_l2(x + c + (r + k * step) * ncol);
  }
  dependency_wait();
  release_dependents();
  if (c < ncol) {
    const float* p = M + c;
    size_t r = r0 + w * rows_abreast + (lane >> shift);
    for (; r + (kBatch - 1) * step < r1; r += kBatch * step) {
      if (VEC) {
        float4 v[kBatch], m[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          v[k] = *reinterpret_cast<const float4*>(p + (r + k * step) * ncol);
          if (RELU) m[k] = *reinterpret_cast<const float4*>(x + c + (r + k * step) * ncol);
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          if (RELU) keep4(v[k], m[k], c + (r + k * step) * ncol);
          acc[0] += v[k].x;
          acc[1 % kW] += v[k].y;
          acc[2 % kW] += v[k].z;
          acc[3 % kW] += v[k].w;
        }
      } else {
        float v[kBatch], m[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          v[k] = p[(r + k * step) * ncol];
          if (RELU) m[k] = x[c + (r + k * step) * ncol];
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
          if (RELU) keep1(v[k], m[k], c + (r + k * step) * ncol);
          acc[0] += v[k];
        }
      }
    }
#pragma unroll 4
    for (; r < r1; r += step) {
      if (VEC) {
        float4 v = *reinterpret_cast<const float4*>(p + r * ncol);
        if (RELU) keep4(v, *reinterpret_cast<const float4*>(x + c + r * ncol), c + r * ncol);
        acc[0] += v.x;
        acc[1 % kW] += v.y;
        acc[2 % kW] += v.z;
        acc[3 % kW] += v.w;
      } else {
        float v = p[r * ncol];
        if (RELU) keep1(v, x[c + r * ncol], c + r * ncol);
        acc[0] += v;
      }
    }
  }
  if (!VEC)
    for (int o = lanes; o < 32; o <<= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
#pragma unroll
  for (int k = 0; k < kW; ++k) sm[w][lane * kW + k] = acc[k];
  cg::cluster_group cluster = cg::this_cluster();
  if (clustered) cluster.barrier_arrive();             // completed before the first remote store below
  __syncthreads();
  float s[kW];
#pragma unroll
  for (int k = 0; k < kW; ++k) {
    s[k] = 0.f;
    if (w == 0)
#pragma unroll
      for (int q = 0; q < kWarps; ++q) s[k] += sm[q][lane * kW + k];
  }
  if (clustered) {
    cluster.barrier_wait();
    if (w == 0) {
      float* first = cluster.map_shared_rank(&part[slice][0], 0);
#pragma unroll
      for (int k = 0; k < kW; ++k) first[lane * kW + k] = s[k];
    }
    cluster.sync();
    if (slice != 0) return;
    if (w == 0)
#pragma unroll
      for (int k = 0; k < kW; ++k) {
        s[k] = 0.f;
        for (int q = 0; q < slices; ++q) s[k] += part[q][lane * kW + k];
      }
  }
  if (w == 0 && c < ncol && lane < lanes) {
    float* o = out + (clustered ? 0 : slice * ncol) + c;
#pragma unroll
    for (int k = 0; k < kW; ++k) o[k] = s[k];
  }
}

__global__ void __launch_bounds__(kBlock)
colsum_finish_kernel(const float* __restrict__ partial, float* __restrict__ v,
                     size_t ncol, int slices) {
  dependency_wait();
  release_dependents();
  const size_t c = blockIdx.x * static_cast<size_t>(kBlock) + threadIdx.x;
  if (c >= ncol) return;
  float s = 0.f;
#pragma unroll 8
  for (int k = 0; k < slices; ++k) s += partial[k * ncol + c];
  v[c] = s;
}

struct ColsumPlan {
  int shift, slices;
  bool vec, clustered;
  size_t blocks;
};
ColsumPlan colsum_plan(size_t nrow, size_t ncol, bool can_vec) {
  ColsumPlan p;
  p.shift = 5;
  while (p.shift > 0 && (static_cast<size_t>(1) << (p.shift - 1)) >= ncol) --p.shift;
  // four columns per lane once that still leaves a column block for most SMs
  p.vec = can_vec && ncol >= 4096;
  p.blocks = ceil_div(ncol, (p.vec ? 4u : 1u) << p.shift);
  const size_t rows_per_pass = static_cast<size_t>(kWarps) << (5 - p.shift);   // rows a CTA reads with one load per lane
  const size_t useful = ceil_div(nrow, rows_per_pass);                           // more slices than this have no row
  const size_t target = ceil_div(static_cast<size_t>(sm_count()) * 4, p.blocks);
  size_t s = useful < target ? useful : target;
  // A cluster covers up to 8 slices; beyond 64 loads per lane a second launch
  // with more slices is the faster way.
  p.clustered = s <= kMaxCluster || useful <= kMaxCluster * 64;
  if (p.clustered) {
    size_t c = 1;
    while (c * 2 <= kMaxCluster && c < s) c *= 2;
    s = c;
  } else if (s > 256) {
    s = 256;
  }
  p.slices = static_cast<int>(s < 1 ? 1 : s);
  if (p.slices == 1) p.clustered = true;      // a single CTA per column block: nothing to exchange
  return p;
}

// ------------------------------------------------------------------- row sums
// v[r] = sum_c M[r][c]; one warp per row, lanes stride over the columns.
__global__ void __launch_bounds__(kBlock)
rowsum_kernel(const float* __restrict__ M, float* __restrict__ v, size_t nrow, size_t ncol) {
  dependency_wait();
  release_dependents();
  const int lane = threadIdx.x & 31;
  const size_t r = (blockIdx.x * static_cast<size_t>(kBlock) + threadIdx.x) >> 5;
  if (r >= nrow) return;
  const float* row = M + r * ncol;
  float acc = 0.f;
#pragma unroll 4
  for (size_t c = lane; c < ncol; c += 32) acc += row[c];
  acc = warp_sum(acc);
  if (lane == 0) v[r] = acc;
}

__global__ void __launch_bounds__(kBlock)
rowmax_kernel(const float* __restrict__ M, float* __restrict__ v, size_t nrow, size_t ncol) {
  dependency_wait();
  release_dependents();
  const int lane = threadIdx.x & 31;
  const size_t r = (blockIdx.x * static_cast<size_t>(kBlock) + threadIdx.x) >> 5;
  if (r >= nrow) return;
  const float* row = M + r * ncol;
  float m = row[0];  // seeded with the first element, as the CUDA reference does
#pragma unroll 4
  for (size_t c = lane; c < ncol; c += 32) m = fmaxf(m, row[c]);
  m = warp_max(m);
  if (lane == 0) v[r] = m;
}

// ---------------------------------------------------- per-channel NCHW reduce
// db[c] = sum over n and the HW plane of dy[n][c][:].  A CTA walks its slice of
// the channel's flattened (n, i) index space; with up to eight slices per
// channel they form a cluster and the call is one launch (see above), else the
// partials are added by chansum_finish_kernel.  RELU as in colsum_kernel.
//
// POOL: dy is the gradient behind a max pooling of 2x2 windows, stride 2, without
// padding, and what goes through the ReLU is the gradient in front of it, which is
// written to pool_dx as well.  Windows do not overlap: an element finds its
// window's first maximum in the window's two rows (the other row's vector is a
// neighbour's, so it comes from L1).  Same values and order as the three calls.
// Planes whose width is a multiple of four only.
struct Pool22 {
  int W, OH, OW;
  FastDiv width;
  // First maximum of a window; a NaN wins and then sticks, as in the pooling kernels.
  __device__ __forceinline__ static int winner(float a, float b, float c, float d) {
    const float v[4] = {a, b, c, d};
    float best = -FLT_MAX;
    int at = -1;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (v[k] > best || (v[k] != v[k] && best == best)) {
        best = v[k];
        at = k;
      }
    return at;
  }
  // The vector at element `pos` of plane `plane`, whose offset is plane0: what its
  // gradient takes, and the gradient.
  struct Windows {
    float4 a, b;
    float g0, g1;
    int r;                                           // its row of the windows' two; -1: no window covers it
  };
  __device__ __forceinline__ Windows load(const float* __restrict__ px, const float* __restrict__ dy, size_t plane,
                                          size_t plane0, int pos) const {
    Windows v;
    const int h = static_cast<int>(width.quot(static_cast<unsigned>(pos))), w = pos - h * W, oh = h >> 1;
    v.r = oh < OH ? h & 1 : -1;
    if (oh >= OH) return v;                          // a last row
    const float* row = px + plane0 + static_cast<size_t>(h - v.r) * W + w;
    const float* gp = dy + (plane * OH + oh) * OW + (w >> 1);
    v.a = *reinterpret_cast<const float4*>(row);
    v.b = *reinterpret_cast<const float4*>(row + W);
    v.g0 = gp[0];
    v.g1 = gp[1];
    return v;
  }
  __device__ __forceinline__ static float4 gradient(const Windows& v) {
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
    if (v.r < 0) return g;
    const int at0 = winner(v.a.x, v.a.y, v.b.x, v.b.y), at1 = winner(v.a.z, v.a.w, v.b.z, v.b.w);
    g.x = 0.0f + (at0 == 2 * v.r ? v.g0 : 0.0f);
    g.y = 0.0f + (at0 == 2 * v.r + 1 ? v.g0 : 0.0f);
    g.z = 0.0f + (at1 == 2 * v.r ? v.g1 : 0.0f);
    g.w = 0.0f + (at1 == 2 * v.r + 1 ? v.g1 : 0.0f);
    return g;
  }
};
template <bool VEC, bool RELU, bool POOL = false>
__global__ void __launch_bounds__(kBlock, RELU ? 4 : 0)
chansum_kernel(const float* __restrict__ dy, const float* __restrict__ x, float* __restrict__ dx,
               float* __restrict__ out, int N, int C,
               int HW, int per_slice, int slices, bool clustered, const Pool22 pool,
               const float* __restrict__ pool_x, float* __restrict__ pool_dx) {
  __shared__ float sm[32];
  __shared__ float part[kMaxCluster];
  const int c = static_cast<int>(blockIdx.x / slices), slice = static_cast<int>(blockIdx.x - c * slices);
  constexpr int kW = VEC ? 4 : 1;
  const int hwu = HW / kW, total = N * hwu;
  const int i0 = min(slice * per_slice, total), i1 = min(i0 + per_slice, total);
  float acc = 0.f;
  // (sample, position) of the unit is advanced without a division per step
  int n = (i0 + static_cast<int>(threadIdx.x)) / hwu, q = (i0 + static_cast<int>(threadIdx.x)) - n * hwu;
  const int dn = kBlock / hwu, dq = kBlock - dn * hwu;
  if (RELU && first_wave(4)) {      // (8 asked ahead for CTAs that start later: 64x256x14x14 from L2 8.6 us, 8.2 so)
    int pn = n, pq = q;
    for (int k = 0, i = i0 + threadIdx.x; k < 4 && i < i1; ++k, i += kBlock) {
      const size_t at = (static_cast<size_t>(pn) * C + c) * HW + static_cast<size_t>(pq) * kW;
      prefetch_l2(x + at);
      if (POOL) prefetch_l2(pool_x + at);
      pn += dn;
      pq += dq;
      if (pq >= hwu) {
        pq -= hwu;
        ++pn;
      }
    }
  }
  dependency_wait();
  release_dependents();
  if constexpr (!RELU) {
#pragma unroll 4
    for (int i = i0 + threadIdx.x; i < i1; i += kBlock) {
      const size_t at = (static_cast<size_t>(n) * C + c) * HW + static_cast<size_t>(q) * kW;
      if (VEC) {
        const float4 v = *reinterpret_cast<const float4*>(dy + at);
        acc += (v.x + v.y) + (v.z + v.w);
      } else {
        acc += dy[at];
      }
      n += dn;
      q += dq;
      if (q >= hwu) {
        q -= hwu;
        ++n;
      }
    }
  } else {
    // The loads of several units ahead of the first one's stores, which the compiler does
    // not move them across (us, 512x16x24x24 with a ReLU 26.8 -> 14.8, with a pooling as well
    // 31.8 -> 21.3; 64x32x24x24 6.1 -> 5.0 and 9.3 -> 8.5).  Four CTAs an SM: with more units
    // of a pooling there are fewer (64x64x24x24 11.0 -> 16.1, with these 10.6).
    constexpr int kBatch = POOL ? 2 : 4;
    for (int i = i0 + threadIdx.x; i < i1; i += kBatch * kBlock) {
      size_t at[kBatch];
      Pool22::Windows p[POOL ? kBatch : 1];
      float4 v[kBatch], m[kBatch];
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        if (i + k * kBlock < i1) {
          const size_t plane = static_cast<size_t>(n) * C + c;
          at[k] = plane * HW + static_cast<size_t>(q) * kW;
          if (POOL) p[POOL ? k : 0] = pool.load(pool_x, dy, plane, plane * HW, q * kW);
          else if (VEC) v[k] = *reinterpret_cast<const float4*>(dy + at[k]);
          else v[k].x = dy[at[k]];
          if (VEC) m[k] = *reinterpret_cast<const float4*>(x + at[k]);
          else m[k].x = x[at[k]];
        }
        n += dn;
        q += dq;
        if (q >= hwu) {
          q -= hwu;
          ++n;
        }
      }
#pragma unroll
      for (int k = 0; k < kBatch; ++k) {
        if (i + k * kBlock >= i1) break;
        if (POOL) *reinterpret_cast<float4*>(pool_dx + at[k]) = v[k] = Pool22::gradient(p[POOL ? k : 0]);
        v[k].x = m[k].x > 0.f ? v[k].x : 0.f;
        if (VEC) {
          v[k].y = m[k].y > 0.f ? v[k].y : 0.f;
          v[k].z = m[k].z > 0.f ? v[k].z : 0.f;
          v[k].w = m[k].w > 0.f ? v[k].w : 0.f;
          *reinterpret_cast<float4*>(dx + at[k]) = v[k];
          acc += (v[k].x + v[k].y) + (v[k].z + v[k].w);
        } else {
          dx[at[k]] = v[k].x;
          acc += v[k].x;
        }
      }
    }
  }
  cg::cluster_group cluster = cg::this_cluster();
  if (clustered) cluster.barrier_arrive();
  acc = block_sum(acc, sm);
  if (!clustered) {
    if (threadIdx.x == 0) out[static_cast<size_t>(c) * slices + slice] = acc;
    return;
  }
  cluster.barrier_wait();
  if (threadIdx.x == 0) *cluster.map_shared_rank(&part[slice], 0) = acc;
  cluster.sync();
  if (slice == 0 && threadIdx.x == 0) {
    float s = 0.f;
    for (int k = 0; k < slices; ++k) s += part[k];
    out[c] = s;
  }
}

__global__ void chansum_finish_kernel(const float* __restrict__ partial,
                                      float* __restrict__ db, int C, int slices) {
  dependency_wait();
  release_dependents();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  float s = 0.f;
#pragma unroll 8
  for (int k = 0; k < slices; ++k) s += partial[static_cast<size_t>(c) * slices + k];
  db[c] = s;
}

int chan_slices(int N, int C, int HW, bool* clustered) {
  const long long per_channel = static_cast<long long>(N) * HW;
  long long s = ceil_div(static_cast<size_t>(sm_count()) * 8, static_cast<size_t>(C));
  const long long max_s = (per_channel + 4095) / 4096;  // >= 4096 elements per slice
  if (s > max_s) s = max_s;
  if (s > 64) s = 64;
  // eight slices of one cluster, unless that leaves more than 64K elements to each
  *clustered = s <= kMaxCluster || per_channel <= kMaxCluster * 65536LL;
  if (*clustered) {
    int c = 1;
    while (c * 2 <= kMaxCluster && c < s) c *= 2;
    s = c;
  }
  return static_cast<int>(s < 1 ? 1 : s);
}

// ------------------------------------------------------------------ total sum
__global__ void __launch_bounds__(kBlock)
sumall_partial_kernel(const float* __restrict__ x, float* __restrict__ partial, size_t n) {
  __shared__ float sm[32];
  dependency_wait();
  release_dependents();
  cta_total(x, partial + blockIdx.x, n, gridDim.x, blockIdx.x, sm);
}
__global__ void __launch_bounds__(kBlock)
sumall_finish_kernel(const float* __restrict__ partial, float* __restrict__ out, int parts) {
  __shared__ float sm[32];
  dependency_wait();
  release_dependents();
  float acc = 0.f;
  for (int i = threadIdx.x; i < parts; i += kBlock) acc += partial[i];
  acc = block_sum(acc, sm);
  if (threadIdx.x == 0) out[0] = acc;
}
int sumall_parts(size_t n) {
  size_t p = ceil_div(n, static_cast<size_t>(kBlock) * 16);
  size_t cap = static_cast<size_t>(sm_count()) * 8;
  if (p > cap) p = cap;
  return static_cast<int>(p < 1 ? 1 : p);
}

}  // namespace
}  // namespace sgb

using namespace sgb;

namespace {
// The column sums of M, or (RELU) of dx = x > 0 ? M : 0, which is written as well.
template <bool RELU>
int column_sums(const float* M, const float* x, float* dx, float* v, size_t nrow, size_t ncol, void* ws,
                size_t ws_bytes, cudaStream_t s, const Beside& beside = Beside{nullptr, nullptr, 0}) {
  const ColsumPlan p = colsum_plan(nrow, ncol, ncol % 4 == 0 && aligned16(RELU ? dx : M));
  const size_t blocks = p.blocks + (beside.x ? 1 : 0);
  if (blocks * p.slices > 0x7fffffffu) return SGB_ERR_SIZE;
  const dim3 grid(static_cast<unsigned>(blocks * p.slices));
  float* out = v;
  if (!p.clustered) {
    if (!ws || ws_bytes < static_cast<size_t>(p.slices) * ncol * sizeof(float)) return SGB_ERR_WORKSPACE;
    out = static_cast<float*>(ws);
  }
  const int st = launch_ex(p.vec ? colsum_kernel<true, RELU> : colsum_kernel<false, RELU>, grid, dim3(kBlock), 0, s,
                           p.clustered && p.slices > 1 ? p.slices : 0, true, M, x, dx, out, nrow, ncol,
                           ceil_div(nrow, p.slices), p.slices, p.shift, p.clustered && p.slices > 1, beside);
  if (st != SGB_OK || p.clustered) return st;
  return launch_ex(colsum_finish_kernel, dim3(static_cast<unsigned>(ceil_div(ncol, kBlock))), dim3(kBlock), 0, s, 0,
                   true, static_cast<const float*>(out), v, ncol, p.slices);
}

// The same over the channels of an NCHW tensor.
struct PoolOf {                        // what the gradient passes first, null: nothing
  const float* x = nullptr;
  float* dx = nullptr;
  int W = 1;
};
template <bool RELU, bool POOL = false>
int channel_sums(const float* dy, const float* x, float* dx, float* db, int N, int C, int HW, void* ws,
                 size_t ws_bytes, cudaStream_t s, const PoolOf& pool = PoolOf()) {
  if (static_cast<long long>(N) * HW > 0x7fffffffLL || C > 65535) return SGB_ERR_SIZE;
  bool clustered;
  const int slices = chan_slices(N, C, HW, &clustered);
  if (!ws || ws_bytes < static_cast<size_t>(slices) * C * sizeof(float)) return SGB_ERR_WORKSPACE;
  const bool vec = (HW % 4 == 0) && aligned16(RELU ? dx : dy);
  const int total = vec ? N * (HW / 4) : N * HW;
  const int per_slice = static_cast<int>(ceil_div(total, slices));
  if (slices == 1) clustered = false;     // the CTA's sum is the result
  float* out = clustered || slices == 1 ? db : static_cast<float*>(ws);
  const Pool22 p{pool.W, HW / pool.W / 2, pool.W / 2, FastDiv(static_cast<unsigned>(pool.W))};
  auto go = [&](auto kernel) {
    return launch_ex(kernel, dim3(static_cast<unsigned>(slices) * C), dim3(kBlock), 0, s, clustered ? slices : 0, true,
                     dy, x, dx, out, N, C, HW, per_slice, slices, clustered, p, pool.x, pool.dx);
  };
  const int st = POOL || vec ? go(chansum_kernel<true, RELU, POOL>) : go(chansum_kernel<false, RELU>);
  if (st != SGB_OK || out == db) return st;
  return launch_ex(chansum_finish_kernel, dim3(static_cast<unsigned>(ceil_div(C, 128))), dim3(128), 0, s, 0, true,
                   static_cast<const float*>(out), db, C, slices);
}
}  // namespace

namespace sgb {
int sum_rows_beside_total(const float* M, float* v, size_t nrow, size_t ncol, const float* x, float* total, void* ws,
                          size_t ws_bytes, void* stream) {
  // one launch where either sum alone is one
  if (sumall_parts(nrow) == 1 && colsum_plan(nrow, ncol, ncol % 4 == 0 && aligned16(M)).clustered)
    return column_sums<false>(M, nullptr, nullptr, v, nrow, ncol, ws, ws_bytes, as_stream(stream),
                              Beside{x, total, nrow});
  const int st = sgb_sum_all_f32(x, total, nrow, ws, ws_bytes, stream);
  return st != SGB_OK ? st : sgb_sum_rows_f32(M, v, nrow, ncol, ws, ws_bytes, stream);
}
}  // namespace sgb

extern "C" {

size_t sgb_sum_rows_workspace_bytes(size_t nrow, size_t ncol) {
  if (nrow == 0 || ncol == 0) return 0;
  // what either alignment may need
  size_t need = 0;
  for (const bool can_vec : {false, true}) {
    const ColsumPlan p = colsum_plan(nrow, ncol, can_vec);
    if (!p.clustered && static_cast<size_t>(p.slices) * ncol * sizeof(float) > need)
      need = static_cast<size_t>(p.slices) * ncol * sizeof(float);
  }
  return need;
}

int sgb_sum_rows_f32(const float* M, float* v, size_t nrow, size_t ncol, void* ws,
                     size_t ws_bytes, void* stream) {
  if (ncol == 0) return SGB_OK;
  if (!v) return SGB_ERR_NULL;
  if (nrow == 0) return sgb_set_f32(0.f, v, ncol, stream);
  if (!M) return SGB_ERR_NULL;
  return column_sums<false>(M, nullptr, nullptr, v, nrow, ncol, ws, ws_bytes, as_stream(stream));
}

int sgb_relu_backward_sum_rows_f32(const float* dy, const float* x, float* dx, float* v, size_t nrow, size_t ncol,
                                   void* ws, size_t ws_bytes, void* stream) {
  if (nrow && ncol && (!dy || !x || !dx)) return SGB_ERR_NULL;
  // vectors or not is decided by dx, as when it is summed by itself
  if (nrow == 0 || ncol == 0 || !v || (aligned16(dx) && !(aligned16(dy) && aligned16(x)))) {
    const int st = sgb_relu_backward_f32(dy, x, dx, nrow * ncol, stream);
    return st != SGB_OK ? st : sgb_sum_rows_f32(dx, v, nrow, ncol, ws, ws_bytes, stream);
  }
  return column_sums<true>(dy, x, dx, v, nrow, ncol, ws, ws_bytes, as_stream(stream));
}

int sgb_sum_columns_f32(const float* M, float* v, size_t nrow, size_t ncol, void* stream) {
  if (nrow == 0) return SGB_OK;
  if (!v) return SGB_ERR_NULL;
  if (ncol == 0) return sgb_set_f32(0.f, v, nrow, stream);
  if (!M) return SGB_ERR_NULL;
  return launch_ex(rowsum_kernel, dim3(static_cast<unsigned>(ceil_div(nrow * 32, kBlock))), dim3(kBlock), 0,
                   as_stream(stream), 0, true, M, v, nrow, ncol);
}

int sgb_row_max_f32(const float* M, float* v, size_t nrow, size_t ncol, void* stream) {
  if (nrow == 0) return SGB_OK;
  if (!M || !v) return SGB_ERR_NULL;
  if (ncol == 0) return SGB_ERR_SIZE;
  return launch_ex(rowmax_kernel, dim3(static_cast<unsigned>(ceil_div(nrow * 32, kBlock))), dim3(kBlock), 0,
                   as_stream(stream), 0, true, M, v, nrow, ncol);
}

size_t sgb_conv_bias_backward_workspace_bytes(int N, int C, int HW) {
  if (N <= 0 || C <= 0 || HW <= 0) return 0;
  bool clustered;
  return static_cast<size_t>(chan_slices(N, C, HW, &clustered)) * C * sizeof(float);
}

int sgb_conv_bias_backward_f32(const float* dy, float* db, int N, int C, int HW, void* ws,
                               size_t ws_bytes, void* stream) {
  if (C <= 0) return C == 0 ? SGB_OK : SGB_ERR_SIZE;
  if (N < 0 || HW < 0) return SGB_ERR_SIZE;
  if (!db) return SGB_ERR_NULL;
  if (N == 0 || HW == 0) return sgb_set_f32(0.f, db, C, stream);
  if (!dy) return SGB_ERR_NULL;
  return channel_sums<false>(dy, nullptr, nullptr, db, N, C, HW, ws, ws_bytes, as_stream(stream));
}

int sgb_relu_backward_conv_bias_f32(const float* dy, const float* x, float* dx, float* db, int N, int C, int HW,
                                    void* ws, size_t ws_bytes, void* stream) {
  if (N < 0 || C < 0 || HW < 0) return SGB_ERR_SIZE;
  const size_t n = static_cast<size_t>(N) * C * HW;
  if (n && (!dy || !x || !dx)) return SGB_ERR_NULL;
  if (n == 0 || !db || (aligned16(dx) && !(aligned16(dy) && aligned16(x)))) {
    const int st = sgb_relu_backward_f32(dy, x, dx, n, stream);
    return st != SGB_OK ? st : sgb_conv_bias_backward_f32(dx, db, N, C, HW, ws, ws_bytes, stream);
  }
  return channel_sums<true>(dy, x, dx, db, N, C, HW, ws, ws_bytes, as_stream(stream));
}

int sgb_maxpool_relu_backward_conv_bias_f32(const float* pool_x, const float* pool_y, const float* dy, float* pool_dx,
                                            int N, int C, int H, int W, int kh, int kw, int ph, int pw, int sh, int sw,
                                            const float* x, float* dx, float* db, void* ws, size_t ws_bytes,
                                            void* stream) {
  const int HW = H > 0 && W > 0 && static_cast<long long>(H) * W <= 0x7fffffffLL ? H * W : 0;
  // One launch and one read of the pooling's gradient less, for the winners found
  // twice and in the order of the channel sums, where the pooling's own kernel reads
  // whole rows.  It pays while a CTA's threads have their few vectors in flight at once
  // and the grid is one wave (elements per CTA, CTAs: the two calls / one, with the
  // operands in L2, as a step of small layers has them, and from DRAM):
  //   1024, 64     16x64x8x8     3.0 / 1.8    3.0 / 1.8
  //   2304, 256    32x32x24x24   5.2 / 4.5    5.5 / 5.6
  //   2304, 512    32x64x24x24   6.9 / 5.7    7.6 / 6.7
  //   4608, 64     64x8x24x24    4.7 / 5.0    5.5 / 6.6
  //   4608, 128    64x16x24x24   5.6 / 5.4    6.5 / 7.2
  //   4608, 256    64x32x24x24   7.2 / 6.1    7.6 / 8.3
  //   4608, 512    256x64x12x12  9.4 / 8.2   10.7 / 10.8
  //   2304, 1024   32x128x24x24 10.7 / 11.0  11.8 / 13.0
  //   9216, 64     128x8x24x24   6.6 / 7.4    7.6 / 10.7
  //   9216, 256    128x32x24x24 10.0 / 9.3   11.3 / 13.5
  //   36864, 96    512x12x24x24 15.1 / 27.8  19.1 / 37.8
  // (64x8x24x24 is the one shape on this side that loses from L2.)  A form with single
  // accesses, for other widths, lost (64x32x13x13 8.1 / 10.2, 256x8x15x15 13.5 / 21.9).
  bool clustered, pays = kh == 2 && kw == 2 && sh == 2 && sw == 2 && ph == 0 && pw == 0 && N > 0 && C > 0 && H >= 2 &&
                         HW && W % 4 == 0 && pool_x && dy && pool_dx && x && dx && db && aligned16(pool_x) &&
                         aligned16(pool_dx) && aligned16(x) && aligned16(dx) && C <= 65535;
  if (pays) {
    const long long slices = chan_slices(N, C, HW, &clustered);
    pays = static_cast<long long>(N) * HW <= 4608 * slices && slices * C <= 4LL * sm_count();
  }
  if (pays)
    return channel_sums<true, true>(dy, x, dx, db, N, C, HW, ws, ws_bytes, as_stream(stream), PoolOf{pool_x, pool_dx, W});
  const int st = sgb_maxpool_backward_f32(pool_x, pool_y, dy, pool_dx, N, C, H, W, kh, kw, ph, pw, sh, sw, stream);
  return st != SGB_OK ? st : sgb_relu_backward_conv_bias_f32(pool_dx, x, dx, db, N, C, H * W, ws, ws_bytes, stream);
}

size_t sgb_sum_all_workspace_bytes(size_t n) {
  return n ? static_cast<size_t>(sumall_parts(n)) * sizeof(float) : 0;
}

int sgb_sum_all_f32(const float* x, float* out, size_t n, void* ws, size_t ws_bytes, void* stream) {
  if (!out) return SGB_ERR_NULL;
  if (n == 0) return sgb_set_f32(0.f, out, 1, stream);
  if (!x) return SGB_ERR_NULL;
  const int parts = sumall_parts(n);
  if (!ws || ws_bytes < parts * sizeof(float)) return SGB_ERR_WORKSPACE;
  cudaStream_t s = as_stream(stream);
  float* partial = static_cast<float*>(ws);
  if (parts == 1) {
    // one CTA covers everything: its block sum IS the result (adding the zeros
    // of a second pass would not change a bit), so write it straight to `out`
    return launch_ex(sumall_partial_kernel, dim3(1), dim3(kBlock), 0, s, 0, true, x, out, n);
  }
  const int st = launch_ex(sumall_partial_kernel, dim3(parts), dim3(kBlock), 0, s, 0, true, x, partial, n);
  if (st != SGB_OK) return st;
  return launch_ex(sumall_finish_kernel, dim3(1), dim3(kBlock), 0, s, 0, true, static_cast<const float*>(partial), out,
                   parts);
}

}  // extern "C"
