// Batch-norm forward in training mode, the partner of the backward kernels:
// batch statistics, normalisation and running statistics.  Emits what the
// backward consumes: save_mean and save_invstd = 1/sqrt(biased_var + eps).
// Running statistics follow cuDNN: r = (1-f)*r + f*batch_value, with the
// UNBIASED variance (M/(M-1)).
//
// Variances are sums of squared differences from a mean (of the whole channel,
// or of a part of it, parts being merged by the pairwise formula
//   n = na + nb,  mean = ma + d nb/n,  m2 = m2a + m2b + d^2 na nb/n,  d = mb - ma:
// T. F. Chan, G. H. Golub, R. J. LeVeque, 1983), never E[x^2] - E[x]^2.
//
// Four forms, by the size of a channel and of the call:
//   registers   up to 8192 floats: one CTA (or a warp) per channel, one pass;
//   cluster     up to 8 CTAs' shared memory: one pass; every CTA works out the
//               moments of its share and the CTAs exchange them ONCE (sum, m2
//               and count in one asynchronous store per pair of CTAs);
//   two visits  large channels of large calls (fwd_revisit_pays): one kernel that
//               reads its data twice, the second time out of L2;
//   two passes  anything else: per-slice moments, then normalisation, which
//               adds the slices up itself (2 launches; 5 before).
// Units are 16-byte vectors, also where planes are not a multiple of four
// floats (RaggedUnit); single floats only for misaligned tensors and tiny planes.
#include "bn_revisit.cuh"

namespace cg = cooperative_groups;

namespace sgb {
namespace {

// Bit 0: the wait for the peers' moments ran out of iterations (that launch's
// outputs are void).
__device__ unsigned g_forward_faults;

enum UnitKind { kScalar = 0, kVec = 1, kRagged = 2 };

__host__ __device__ inline int units_per_plane(int kind, int hw) {
  return kind == kScalar ? hw : kind == kVec ? hw / 4 : ragged_units(hw);
}
template <int KIND>
struct Unit {
  static constexpr int kW = KIND == kScalar ? 1 : 4;
  size_t off;
  unsigned valid;
  __device__ __forceinline__ Unit(size_t plane_off, int q, int hw) {
    if (KIND == kRagged) {
      const RaggedUnit r(plane_off, q, hw);
      off = r.off;
      valid = r.valid;
    } else {
      off = plane_off + static_cast<size_t>(q) * kW;
      valid = KIND == kVec ? 15u : 1u;
    }
  }
  __device__ __forceinline__ Vec4f load(const float* p, size_t numel) const {
    Vec4f v;
    if (KIND == kVec) {
      v.u = ld128(p + off);
    } else if (KIND == kRagged) {
      v.u = make_uint4(0, 0, 0, 0);
      if (valid) v = ragged_load(p, off, numel);
    } else {
      v.f[0] = p[off];
    }
    return v;
  }
  __device__ __forceinline__ void store(float* p, const Vec4f& v) const {
    if (KIND == kScalar) {
      p[off] = v.f[0];
    } else if (KIND == kVec || valid == 15u) {
      st128(p + off, v.u);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (valid >> j & 1u) p[off + j] = v.f[j];
    }
  }
};

struct FwdArgs {
  const float* x;
  const float* scale;
  const float* bias;
  float* running_mean;
  float* running_var;
  float factor, eps;
  float* y;
  float* save_mean;
  float* save_invstd;
  BnShape sh;
  size_t numel;
};

// One thread per channel: everything that is written once per channel.
__device__ __forceinline__ void finish_channel(const FwdArgs& a, int c, float mu, float var, float invstd) {
  const float m = static_cast<float>(a.sh.N) * static_cast<float>(a.sh.HW);
  const float unbiased = m > 1.0f ? var * (m / (m - 1.0f)) : var;
  a.save_mean[c] = mu;
  a.save_invstd[c] = invstd;
  a.running_mean[c] = (1.0f - a.factor) * a.running_mean[c] + a.factor * mu;
  a.running_var[c] = (1.0f - a.factor) * a.running_var[c] + a.factor * unbiased;
}

// ------------------------------------------------------------ in registers
template <int G, int NV, bool VEC>
__global__ void __launch_bounds__(G == 32 ? 128 : G)
bn_fwd_small_kernel(const FwdArgs a) {
  constexpr int kW = VEC ? 4 : 1;
  __shared__ float sm[2][2 * G / 32];
  const int c = G == 32 ? blockIdx.x * 4 + (threadIdx.x >> 5) : blockIdx.x;
  const int t = G == 32 ? threadIdx.x & 31 : threadIdx.x;
  dependency_wait();
  release_dependents();
  if (c >= a.sh.C) return;
  const int hwu = a.sh.HW / kW, total = a.sh.N * hwu;
  const size_t plane_stride = static_cast<size_t>(a.sh.C) * a.sh.HW, chan_off = static_cast<size_t>(c) * a.sh.HW;
  float v[NV][kW];
  size_t off[NV];
  UnitWalk w(t, G, hwu);
#pragma unroll
  for (int k = 0; k < NV; ++k, w.next()) {
    off[k] = w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * kW;
    const bool in = t + k * G < total;
    if (VEC) {
      Vec4f q;
      q.u = make_uint4(0, 0, 0, 0);
      if (in) q.u = ld128(a.x + off[k]);
#pragma unroll
      for (int j = 0; j < kW; ++j) v[k][j] = q.f[j];
    } else {
      v[k][0] = in ? a.x[off[k]] : 0.0f;
    }
  }
  const float sc = a.scale[c], b = a.bias[c];
  const float inv_m = 1.0f / (static_cast<float>(a.sh.N) * static_cast<float>(a.sh.HW));
  float s = 0.f, q = 0.f, unused = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int j = 0; j < kW; ++j) s += v[k][j];
  channel_sums<G, false>(s, unused, sm[0]);
  const float mu = s * inv_m;
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int j = 0; j < kW; ++j) {
      const float d = t + k * G < total ? v[k][j] - mu : 0.0f;
      q += d * d;
    }
  channel_sums<G, false>(q, unused, sm[1]);
  const float var = q * inv_m, invstd = 1.0f / sqrtf(var + a.eps), g = sc * invstd;
  if (t == 0) finish_channel(a, c, mu, var, invstd);
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    if (t + k * G >= total) break;
    if (VEC) {
      Vec4f o;
#pragma unroll
      for (int j = 0; j < kW; ++j) o.f[j] = (v[k][j] - mu) * g + b;
      st128(a.y + off[k], o.u);
    } else {
      a.y[off[k]] = (v[k][0] - mu) * g + b;
    }
  }
}

// The CTAs of a cluster exchange (sum, m2, count) of their shares, once, as
// 16-byte asynchronous stores that signal the receivers' mbarriers, and every
// thread merges them in rank order: mean and biased variance of the channel.
// The peers have started (cluster barrier): their memory is addressable.
__device__ __forceinline__ void exchange_moments(const FwdArgs& a, int cs, int rank, float s, float q, float n,
                                                 float4* parts, unsigned long long* parts_in, float& mu, float& var) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    if (lane == 0) mbar_arrive_expect(parts_in, 16u * static_cast<unsigned>(cs));
    if (lane < cs) {
      unsigned slot, bar;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(slot) : "r"(smem_addr(&parts[rank])), "r"(lane));
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(smem_addr(parts_in)), "r"(lane));
      asm volatile(
          "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(slot),
          "r"(__float_as_uint(s)), "r"(__float_as_uint(q)), "r"(__float_as_uint(n)), "r"(0u), "r"(bar)
          : "memory");
    }
  }
  bool in = false;
  for (unsigned it = 0; it < (1u << 24) && !in; ++it) in = mbar_try_wait(parts_in, 0);
  if (!in) atomicOr(&g_forward_faults, 1u);
  const float inv_m = 1.0f / (static_cast<float>(a.sh.N) * static_cast<float>(a.sh.HW));
  float sum = 0.f, m2 = 0.f;
  for (int r = 0; r < cs; ++r) sum += parts[r].x;
  mu = sum * inv_m;
  for (int r = 0; r < cs; ++r) {
    const float4 p = parts[r];
    if (p.z > 0.f) {
      const float d = p.x / p.z - mu;
      m2 += p.y + p.z * (d * d);
    }
  }
  var = m2 * inv_m;
}

// ------------------------------------------------------------- in a cluster
// The CTAs of a cluster share channel blockIdx.x / cs.  x is staged in shared
// memory by 16-byte asynchronous copies; sum and squared differences of the
// share are two passes over the staged copy.
template <int KIND, int T>
__global__ void __launch_bounds__(T)
bn_fwd_cluster_kernel(const FwdArgs a, int per_cta) {
  constexpr int kW = Unit<KIND>::kW;
  extern __shared__ __align__(16) float stage[];
  __shared__ unsigned long long parts_in;              // mbarrier: counts the peers' moments as they land
  __shared__ __align__(16) float4 parts[16];           // (sum, m2, count) of every CTA of the cluster
  __shared__ float sm[2][2 * T / 32];
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = static_cast<int>(cluster.num_blocks());
  const int rank = static_cast<int>(cluster.block_rank());
  const int c = blockIdx.x / cs;
  if (threadIdx.x == 0) {
    mbar_init(&parts_in, 1);
    fence_mbarrier_init();
  }
  cluster.barrier_arrive();                            // matched by barrier_wait before the exchange
  const int upp = units_per_plane(KIND, a.sh.HW), total = a.sh.N * upp;
  const int u0 = min(rank * per_cta, total), u1 = min(u0 + per_cta, total);
  const int first = u0 + threadIdx.x;
  const size_t plane_stride = static_cast<size_t>(a.sh.C) * a.sh.HW, chan_off = static_cast<size_t>(c) * a.sh.HW;
  const int group_units = ((per_cta + T - 1) / T + kCopyGroups - 1) / kCopyGroups;
  dependency_wait();
  {
    UnitWalk w(first, T, upp);
    int u = first;
#pragma unroll
    for (int g = 0; g < kCopyGroups; ++g) {
      for (int k = 0; k < group_units && u < u1; ++k, u += T, w.next()) {
        const Unit<KIND> r(w.n * plane_stride + chan_off, w.q, a.sh.HW);
        float* dst = stage + (u - u0) * kW;
        if (KIND == kVec) cp_async16(dst, a.x + r.off);
        else if (KIND == kScalar) *dst = a.x[r.off];
        else if (r.valid) ragged_copy(dst, a.x, r.off, a.numel);
      }
      cp_async_commit();
    }
  }
  const float sc = a.scale[c], b = a.bias[c];
  // sum and count of the share, copy group by copy group as the groups land
  float s = 0.f, n = 0.f;
  {
    UnitWalk w(first, T, upp);
    int u = first;
    auto sum_copy_group = [&]() {
      for (int k = 0; k < group_units && u < u1; ++k, u += T) {
        const float* src = stage + (u - u0) * kW;
        if (KIND == kScalar) {
          s += *src;
        } else if (KIND == kVec) {
          Vec4f v;
          v.u = *reinterpret_cast<const uint4*>(src);
          s += (v.f[0] + v.f[1]) + (v.f[2] + v.f[3]);
        } else {
          const Unit<KIND> r(w.n * plane_stride + chan_off, w.q, a.sh.HW);
          w.next();
          if (!r.valid) continue;
          Vec4f v;
          v.u = *reinterpret_cast<const uint4*>(src);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (r.valid >> j & 1u) s += v.f[j];
          n += static_cast<float>(__popc(r.valid));
        }
      }
    };
    static_assert(kCopyGroups == 4, "the waits below are written out for four groups");
    cp_async_wait_pending<3>();
    sum_copy_group();
    cp_async_wait_pending<2>();
    sum_copy_group();
    cp_async_wait_pending<1>();
    sum_copy_group();
    cp_async_wait_pending<0>();
    sum_copy_group();
  }
  channel_sums<T, KIND == kRagged>(s, n, sm[0]);
  if (KIND != kRagged) n = static_cast<float>((u1 - u0) * kW);
  const float mine = n > 0.f ? s / n : 0.f;            // mean of the share
  float q = 0.f, unused = 0.f;
  {
    UnitWalk w(first, T, upp);
    for (int u = first; u < u1; u += T) {
      const float* src = stage + (u - u0) * kW;
      if (KIND == kScalar) {
        const float d = *src - mine;
        q += d * d;
        continue;
      }
      unsigned valid = 15u;
      if (KIND == kRagged) {
        valid = Unit<KIND>(w.n * plane_stride + chan_off, w.q, a.sh.HW).valid;
        w.next();
        if (!valid) continue;
      }
      Vec4f v;
      v.u = *reinterpret_cast<const uint4*>(src);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float d = v.f[j] - mine;
        if (KIND == kVec || (valid >> j & 1u)) q += d * d;
      }
    }
  }
  channel_sums<T, false>(q, unused, sm[1]);
  cluster.barrier_wait();                              // peers have started: their memory is addressable
  float mu, var;
  exchange_moments(a, cs, rank, s, q, n, parts, &parts_in, mu, var);
  const float invstd = 1.0f / sqrtf(var + a.eps), g = sc * invstd;
  if (rank == 0 && threadIdx.x == 0) finish_channel(a, c, mu, var, invstd);
  release_dependents();
  UnitWalk w(first, T, upp);
  for (int u = first; u < u1; u += T, w.next()) {
    const Unit<KIND> r(w.n * plane_stride + chan_off, w.q, a.sh.HW);
    if (!r.valid) continue;
    const float* src = stage + (u - u0) * kW;
    Vec4f v, o;
    if (KIND == kScalar) v.f[0] = *src;
    else v.u = *reinterpret_cast<const uint4*>(src);
#pragma unroll
    for (int j = 0; j < kW; ++j) o.f[j] = (v.f[j] - mu) * g + b;
    r.store(a.y, o);
  }
}

// The same with the first kRegUnits units per thread in registers: three CTAs of
// 256 threads keep 290 KB of an SM's registers and shared memory in flight
// instead of 200 KB.  All loads are issued at once.
constexpr int kRegUnits = 8;
constexpr int kHybridT = 256;
__global__ void __launch_bounds__(kHybridT, 3)
bn_fwd_hybrid_kernel(const FwdArgs a, int per_cta) {
  constexpr int T = kHybridT, R = kRegUnits;
  extern __shared__ __align__(16) float stage[];
  __shared__ unsigned long long parts_in;
  __shared__ __align__(16) float4 parts[16];
  __shared__ float sm[2][2 * T / 32];
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = static_cast<int>(cluster.num_blocks());
  const int rank = static_cast<int>(cluster.block_rank());
  const int c = blockIdx.x / cs;
  if (threadIdx.x == 0) {
    mbar_init(&parts_in, 1);
    fence_mbarrier_init();
  }
  cluster.barrier_arrive();
  const int hwu = a.sh.HW >> 2, total = a.sh.N * hwu;
  const int u0 = min(rank * per_cta, total), u1 = min(u0 + per_cta, total);
  const int first = u0 + threadIdx.x;
  float* const sx = stage + static_cast<size_t>(threadIdx.x) * 4;      // unit k >= R at (k - R) * T * 4
  const size_t plane_stride = static_cast<size_t>(a.sh.C) * a.sh.HW, chan_off = static_cast<size_t>(c) * a.sh.HW;
  dependency_wait();
  Vec4f v[R];
  {
    UnitWalk w(first, T, hwu);
#pragma unroll
    for (int k = 0; k < R; ++k, w.next()) {
      v[k].u = make_uint4(0, 0, 0, 0);
      if (first + k * T < u1) v[k].u = ld128(a.x + w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4);
    }
    float* dst = sx;
    for (int u = first + R * T; u < u1; u += T, w.next(), dst += T * 4)
      cp_async16(dst, a.x + w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4);
    cp_async_commit();
  }
  const float sc = a.scale[c], b = a.bias[c];
  float s = 0.f, q = 0.f, unused = 0.f;
#pragma unroll
  for (int k = 0; k < R; ++k) s += (v[k].f[0] + v[k].f[1]) + (v[k].f[2] + v[k].f[3]);
  cp_async_wait_pending<0>();
  {
    const float* src = sx;
    for (int u = first + R * T; u < u1; u += T, src += T * 4) {
      Vec4f t;
      t.u = *reinterpret_cast<const uint4*>(src);
      s += (t.f[0] + t.f[1]) + (t.f[2] + t.f[3]);
    }
  }
  channel_sums<T, false>(s, unused, sm[0]);
  const float n = static_cast<float>((u1 - u0) * 4), mine = n > 0.f ? s / n : 0.f;
#pragma unroll
  for (int k = 0; k < R; ++k)
    if (first + k * T < u1) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float d = v[k].f[j] - mine;
        q += d * d;
      }
    }
  {
    const float* src = sx;
    for (int u = first + R * T; u < u1; u += T, src += T * 4) {
      Vec4f t;
      t.u = *reinterpret_cast<const uint4*>(src);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float d = t.f[j] - mine;
        q += d * d;
      }
    }
  }
  channel_sums<T, false>(q, unused, sm[1]);
  cluster.barrier_wait();
  float mu, var;
  exchange_moments(a, cs, rank, s, q, n, parts, &parts_in, mu, var);
  const float invstd = 1.0f / sqrtf(var + a.eps), g = sc * invstd;
  if (rank == 0 && threadIdx.x == 0) finish_channel(a, c, mu, var, invstd);
  release_dependents();
  UnitWalk w(first, T, hwu);
  auto emit = [&](const Vec4f& x) {
    Vec4f o;
#pragma unroll
    for (int j = 0; j < 4; ++j) o.f[j] = (x.f[j] - mu) * g + b;
    st128(a.y + w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4, o.u);
  };
#pragma unroll
  for (int k = 0; k < R; ++k, w.next())
    if (first + k * T < u1) emit(v[k]);
  const float* src = sx;
  for (int u = first + R * T; u < u1; u += T, w.next(), src += T * 4) {
    Vec4f t;
    t.u = *reinterpret_cast<const uint4*>(src);
    emit(t);
  }
}

struct Moments {
  float n, mean, m2;
};
__device__ __forceinline__ Moments merge(const Moments& a, const Moments& b) {
  Moments r;
  r.n = a.n + b.n;
  const float f = r.n > 0.f ? b.n / r.n : 0.f, d = b.mean - a.mean;
  r.mean = a.mean + d * f;
  r.m2 = a.m2 + b.m2 + d * d * (a.n * f);
  return r;
}
__device__ __forceinline__ Moments warp_merge(Moments v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Moments t;
    t.n = __shfl_down_sync(0xffffffffu, v.n, o);
    t.mean = __shfl_down_sync(0xffffffffu, v.mean, o);
    t.m2 = __shfl_down_sync(0xffffffffu, v.m2, o);
    v = merge(v, t);
  }
  return v;              // valid in lane 0
}

// ------------------------------------------------------------ in two visits
// See bn_revisit.cuh.  An item leaves its mean and its sum of squared differences.
// One operand only, so a CTA takes more units: of 3 to 6 vectors and 192 to 288
// threads these were the best (32x256x56x56 42.4 us against 43.8-47.6,
// 32x128x57x57 28.7 against 30.2-37.9).
template <bool VEC>
constexpr RevisitShape kFwd = VEC ? RevisitShape{6, 256, 4} : RevisitShape{3, 256, 5};

// Elements of channel c ahead of unit u.
template <bool VEC>
__device__ __forceinline__ unsigned elements_before(const Revisit& r, unsigned c, unsigned u) {
  if (VEC) return 4 * u;
  const unsigned n = r.upp.quot(u), q = u - n * r.upp.d, lead = (n * r.plane_stride + c * r.hw) & 3u;
  return n * r.hw + (4 * q > lead ? min(4 * q - lead, r.hw) : 0u);
}

template <bool VEC>
__global__ void __launch_bounds__(kFwd<VEC>.threads + 32, kFwd<VEC>.per_sm)
bn_fwd_revisit_kernel(const __grid_constant__ FwdArgs a, const __grid_constant__ Revisit r) {
  constexpr int NV = kFwd<VEC>.units, kWarps = kFwd<VEC>.threads / 32;
  __shared__ float sm[2][kWarps];
  __shared__ float coef[3];
  __shared__ bool stopped;
  const unsigned item = blockIdx.x, mine = item - r.delay, threads = blockDim.x - 32;
  const bool summing = static_cast<int>(item) < r.items, finishing = static_cast<int>(item) >= r.delay;
  const unsigned numel = static_cast<unsigned>(a.numel);
  if (threadIdx.x >= threads) {
    dependency_wait();
    release_dependents();
    if (summing) revisit_open(r, item);
    if (!finishing) return;
    const unsigned c = r.parts.quot(mine);
    const float sc = a.scale[c], b = a.bias[c];
    Moments m{0.f, 0.f, 0.f};
    unsigned base;
    const bool got = revisit_gather(r, c, base, [&](unsigned k, float mean, float m2) {
      const unsigned e0 = elements_before<VEC>(r, c, k * r.per), e1 = elements_before<VEC>(r, c, min((k + 1) * r.per, r.total));
      m = merge(m, Moments{static_cast<float>(e1 - e0), mean, m2});
    });
    m = warp_merge(m);
    if ((threadIdx.x & 31) == 0) {
      stopped = !got;
      const float var = m.m2 / (static_cast<float>(a.sh.N) * static_cast<float>(a.sh.HW));
      const float invstd = 1.0f / sqrtf(var + a.eps);
      coef[0] = m.mean;
      coef[1] = sc * invstd;
      coef[2] = b;
      if (got && mine == c * r.parts.d) finish_channel(a, c, m.mean, var, invstd);
    }
    revisit_arrive(2, blockDim.x);
    if (got) revisit_leave(r, c, base);
    return;
  }
  Vec4f v[NV];
  // Sum over the summing threads; every thread adds the warps' sums up itself.
  auto total = [&](float x, float (&s)[kWarps]) {
    x = warp_sum(x);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = x;
    revisit_sync(1, threads);
    x = 0.f;
    for (unsigned w = 0; w < threads / 32; ++w) x += s[w];
    return x;
  };
  if (summing) {
    const RevisitUnits<VEC, NV> u(r, item, threads);
    if (first_wave(kFwd<VEC>.per_sm)) {
#pragma unroll
      for (int k = 0; k < NV; ++k)
        if (u.valid[k] && (VEC || u.off[k] < numel)) prefetch_l2(a.x + u.off[k]);
    }
    dependency_wait();
    const unsigned long long keep = keep_policy();
    float s = 0.f, q = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k)
      if (u.valid[k]) v[k] = u.load(a.x, k, numel, keep);
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (u.valid[k] >> j & 1u) s += v[k].f[j];
    const unsigned e0 = elements_before<VEC>(r, u.c, u.part * r.per),
                   e1 = elements_before<VEC>(r, u.c, min((u.part + 1) * r.per, r.total));
    const float mean = e1 > e0 ? total(s, sm[0]) / static_cast<float>(e1 - e0) : total(s, sm[0]);
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (u.valid[k] >> j & 1u) {
          const float d = v[k].f[j] - mean;
          q += d * d;
        }
    q = total(q, sm[1]);
    if (threadIdx.x == 0) put_entry(r.entries + item, mean, q, r.tag);
  } else {
    dependency_wait();
  }
  if (!finishing) return;
  const RevisitUnits<VEC, NV> u(r, mine, threads);
  const unsigned long long ease = ease_policy();
#pragma unroll
  for (int k = 0; k < NV; ++k)
    if (u.valid[k]) v[k] = u.load(a.x, k, numel, ease);
  revisit_sync(2, blockDim.x);
  if (stopped) return;
  const float mu = coef[0], g = coef[1], b = coef[2];
#pragma unroll
  for (int k = 0; k < NV; ++k)
    if (u.valid[k]) {
      Vec4f o;
#pragma unroll
      for (int j = 0; j < 4; ++j) o.f[j] = (v[k].f[j] - mu) * g + b;
      u.store(a.y, k, o);
    }
}

// One operand is little to overlap with, so only channels that leave clusters with
// large shares or no place at all gain (us, the forms above and below / this one):
//   32x64x112x112 61.5 / 40.5   32x64x56x56 14.9 / 13.3    64x100x40x40  19.4 / 18.5
//   32x512x28x28 25.4 / 24.7    10x256x52x52 15.5 / 14.8   12x200x50x50  12.5 / 13.7
// and odd planes, whose clusters read with masked ends:
//   32x128x57x57 37.3 / 28.6    24x64x71x71 24.4 / 18.4    24x64x57x57   19.1 / 14.8
//   40x32x51x51  13.5 / 10.4    24x64x37x37 10.2 / 9.4     33x128x35x35  17.0 / 15.3
//   12x64x69x69  12.6 / 11.9    40x64x31x31 11.0 / 10.1    18x100x47x47  12.9 / 12.8
//   20x100x47x47 13.7 / 13.7    4x100x99x99 12.7 / 12.1    16x96x49x49   12.6 / 13.2
//   18x256x25x25 11.1 / 11.6 (11,250 elements a channel), 4x128x57x57 8.5 / 8.9 (12,996)
// (the last two are on the other side; of the 22 shapes in this range that were looked at,
// 16x96x49x49 alone lost more than a percent)
// The lower line for whole vectors is from a layer's forward, ReLU and backward in
// sequence: what the second visit leaves in L2 is x, and what comes next reads y
// (elements of a channel: 69,000 134.3 / 136.7, 75,000 145.4 / 147.9, 88,000 149.7 /
// 152.7, 100,000 154.2 / 147.9 and on 64 channels 42.3 / 39.5).
// The upper lines are those of the backward (batchnorm.cu): 4.0e6 elements a channel,
// 8.0e7 in all 175.8 / 172.1, 4.2e6 and 6.7e7 132.3 / 137.9, 8.0e6 and 3.2e7 103.8 /
// 109.7, 1.7e7 and 1.7e7 141.8 / 101.5; odd planes 2.6e6 and 2.1e7 101.5 / 92.0, 2.9e6
// and 3.5e7 142.0 / 156.5, 4.0e6 and 3.2e7 155.7 / 187.4.
inline bool fwd_revisit_pays(int N, int C, int HW) {
  const long long channel = static_cast<long long>(N) * HW, elements = channel * C;
  if (HW % 4)
    return channel <= 2600000 &&
           ((HW >= 900 && elements >= 2000000 && channel >= 32000) || (HW >= 2500 && elements >= 6000000));
  return HW >= 2500 && channel >= 96000 && elements >= 6000000 && (channel <= 4000000 || elements <= 20000000);
}

// SGB_ERR_WORKSPACE and nothing done where the workspace is too small or the problem too large.
template <bool VEC>
int launch_revisit(const FwdArgs& a, void* ws, size_t ws_bytes, cudaStream_t s) {
  const int upp = units_per_plane(VEC ? kVec : kRagged, a.sh.HW);
  const long long units = static_cast<long long>(a.sh.N) * upp;
  RevisitPlan p;
  if (!ws || !aligned16(ws) || !revisit_plan(kFwd<VEC>, units, upp, a.sh.C, &p) || ws_bytes < p.bytes)
    return SGB_ERR_WORKSPACE;
  int st = SGB_OK;
  RevisitState* state = revisit_state(&st);
  if (!state) return st;
  return launch_ex(bn_fwd_revisit_kernel<VEC>, dim3(static_cast<unsigned>(p.items + p.delay)), dim3(p.threads + 32), 0,
                   s, 0, true, a, revisit_args(p, units, upp, a.sh.C, a.sh.HW, ws, state));
}

// ------------------------------------------------------------- in two passes
// Pass 1, grid (slices, C): moments of a slice.  A thread works out those of
// four units at a time (in registers) and merges them into its own.
template <int KIND>
__global__ void __launch_bounds__(kBlock)
bn_fwd_moments_kernel(const FwdArgs a, float4* __restrict__ partial, int per_slice) {
  constexpr int kW = Unit<KIND>::kW;
  __shared__ float4 sm[kBlock / 32];
  dependency_wait();
  release_dependents();
  const int c = blockIdx.y, slice = blockIdx.x;
  const int upp = units_per_plane(KIND, a.sh.HW), total = a.sh.N * upp;
  const int i0 = min(slice * per_slice, total), i1 = min(i0 + per_slice, total);
  const size_t plane_stride = static_cast<size_t>(a.sh.C) * a.sh.HW, chan_off = static_cast<size_t>(c) * a.sh.HW;
  Moments acc{0.f, 0.f, 0.f};
  UnitWalk w(i0 + threadIdx.x, kBlock, upp);
  for (int i = i0 + threadIdx.x; i < i1;) {
    Vec4f v[4];
    unsigned valid[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      valid[k] = 0;
      if (i < i1) {
        const Unit<KIND> r(w.n * plane_stride + chan_off, w.q, a.sh.HW);
        valid[k] = r.valid;
        v[k] = r.load(a.x, a.numel);
        i += kBlock;
        w.next();
      }
    }
    Moments b{0.f, 0.f, 0.f};
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int j = 0; j < kW; ++j)
        if (valid[k] >> j & 1u) {
          s += v[k].f[j];
          b.n += 1.f;
        }
    if (b.n == 0.f) continue;
    b.mean = s / b.n;
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int j = 0; j < kW; ++j)
        if (valid[k] >> j & 1u) {
          const float d = v[k].f[j] - b.mean;
          b.m2 += d * d;
        }
    acc = merge(acc, b);
  }
  acc = warp_merge(acc);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = make_float4(acc.n, acc.mean, acc.m2, 0.f);
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < kBlock / 32; ++k) acc = merge(acc, Moments{sm[k].x, sm[k].y, sm[k].z});
    partial[static_cast<size_t>(c) * gridDim.x + slice] = make_float4(acc.n, acc.mean, acc.m2, 0.f);
  }
}

// Pass 2, grid (tiles, C): a warp of every CTA merges the channel's slices (the
// same order everywhere), then the CTA normalises its tile.  Channels in
// descending order: what pass 1 read last is still in L2.
constexpr int kNormUnits = 4;
template <int KIND>
__global__ void __launch_bounds__(kBlock)
bn_fwd_normalize_kernel(const FwdArgs a, const float4* __restrict__ partial, int slices) {
  constexpr int kW = Unit<KIND>::kW;
  __shared__ float coef[2];
  const int c = a.sh.C - 1 - blockIdx.y;
  const int upp = units_per_plane(KIND, a.sh.HW), total = a.sh.N * upp;
  const size_t plane_stride = static_cast<size_t>(a.sh.C) * a.sh.HW, chan_off = static_cast<size_t>(c) * a.sh.HW;
  const int unit0 = blockIdx.x * (kBlock * kNormUnits) + threadIdx.x;
  UnitWalk w(min(unit0, total - 1), kBlock, upp);
  Vec4f v[kNormUnits];
  UnitWalk w2 = w;
  dependency_wait();
#pragma unroll
  for (int k = 0; k < kNormUnits; ++k)
    if (unit0 + k * kBlock < total) {
      v[k] = Unit<KIND>(w.n * plane_stride + chan_off, w.q, a.sh.HW).load(a.x, a.numel);
      w.next();
    }
  if (threadIdx.x < 32) {
    Moments m{0.f, 0.f, 0.f};
    for (int k = threadIdx.x; k < slices; k += 32) {
      const float4 p = partial[static_cast<size_t>(c) * slices + k];
      m = merge(m, Moments{p.x, p.y, p.z});
    }
    m = warp_merge(m);
    if (threadIdx.x == 0) {
      const float var = m.m2 / (static_cast<float>(a.sh.N) * static_cast<float>(a.sh.HW));
      const float invstd = 1.0f / sqrtf(var + a.eps);
      coef[0] = m.mean;
      coef[1] = a.scale[c] * invstd;
      if (blockIdx.x == 0) finish_channel(a, c, m.mean, var, invstd);
    }
  }
  __syncthreads();
  release_dependents();
  const float mu = coef[0], g = coef[1], b = a.bias[c];
#pragma unroll
  for (int k = 0; k < kNormUnits; ++k) {
    if (unit0 + k * kBlock >= total) break;
    const Unit<KIND> r(w2.n * plane_stride + chan_off, w2.q, a.sh.HW);
    w2.next();
    if (!r.valid) continue;
    Vec4f o;
#pragma unroll
    for (int j = 0; j < kW; ++j) o.f[j] = (v[k].f[j] - mu) * g + b;
    r.store(a.y, o);
  }
}

template <int KIND, int T>
int launch_cluster_t(const FwdArgs& a, int cs, int per_cta, cudaStream_t s) {
  auto kernel = bn_fwd_cluster_kernel<KIND, T>;
  static std::atomic<bool> attr_set[64];
  const int ready = opt_in_once(kernel, attr_set, true);
  if (ready != SGB_OK) return ready;
  return launch_ex(kernel, dim3(static_cast<unsigned>(a.sh.C) * cs), dim3(T),
                   static_cast<size_t>(per_cta) * Unit<KIND>::kW * 4, s, cs, true, a, per_cta);
}
// A cluster where the channel fits one, else two passes.
template <int KIND>
int launch_large(const FwdArgs& a, void* ws, size_t ws_bytes, cudaStream_t s) {
  const int total = a.sh.N * units_per_plane(KIND, a.sh.HW);
  int per_cta = 0;
  if (KIND == kVec) {
    // registers and shared memory together, where that still leaves two CTAs for
    // every SM (32x256x56x56: 47.4 -> 44.4 us, 32x512x28x28 26.0 -> 24.8)
    for (int hcs = 1; hcs <= 8; hcs *= 2) {
      const int share = (total + hcs - 1) / hcs, rest = share - kRegUnits * kHybridT;
      if (rest * 16 > 74 * 1024) continue;
      if (rest < 0 || static_cast<long long>(a.sh.C) * hcs < 2LL * sm_count()) break;
      static std::atomic<bool> attr_set[64];
      const int ready = opt_in_once(bn_fwd_hybrid_kernel, attr_set, true);
      if (ready != SGB_OK) return ready;
      return launch_ex(bn_fwd_hybrid_kernel, dim3(static_cast<unsigned>(a.sh.C) * hcs), dim3(kHybridT),
                       static_cast<size_t>(rest) * 16, s, hcs, true, a, share);
    }
  }
  const int cs = cluster_plan(total, Unit<KIND>::kW * 4, 8192, &per_cta, a.sh.C);
  if (cs > 0 && static_cast<long long>(a.sh.C) * cs <= 0x7fffffffLL)
    return per_cta > 2048 ? launch_cluster_t<KIND, 512>(a, cs, per_cta, s) : launch_cluster_t<KIND, 256>(a, cs, per_cta, s);
  // half the slices of the backward passes: a slice leaves 16 bytes in the workspace, not 8
  int slices = bn_slices_for(static_cast<long long>(a.sh.N) * a.sh.HW, a.sh.C, sm_count());
  if (slices > kMaxSlices / 2) slices = kMaxSlices / 2;
  if (!ws || ws_bytes < static_cast<size_t>(slices) * a.sh.C * sizeof(float4) || !aligned16(ws)) return SGB_ERR_WORKSPACE;
  float4* partial = static_cast<float4*>(ws);
  const int st = launch_ex(bn_fwd_moments_kernel<KIND>, dim3(slices, a.sh.C), dim3(kBlock), 0, s, 0, true, a, partial,
                           static_cast<int>(ceil_div(total, slices)));
  if (st != SGB_OK) return st;
  return launch_ex(bn_fwd_normalize_kernel<KIND>,
                   dim3(static_cast<unsigned>(ceil_div(total, kBlock * kNormUnits)), a.sh.C), dim3(kBlock), 0, s, 0,
                   true, a, static_cast<const float4*>(partial), slices);
}

}  // namespace

size_t bn_forward_workspace_bytes(int N, int C, int HW) {
  const int upp = units_per_plane(HW % 4 ? kRagged : kVec, HW);
  RevisitPlan p;
  if (!fwd_revisit_pays(N, C, HW)) return 0;
  return revisit_plan(HW % 4 ? kFwd<false> : kFwd<true>, static_cast<long long>(N) * upp, upp, C, &p) ? p.bytes : 0;
}

int bn_forward_faults(unsigned* flags) {
  const cudaError_t e = cudaMemcpyFromSymbol(flags, g_forward_faults, sizeof(unsigned));
  return e == cudaSuccess ? SGB_OK : note_cuda_error(e);
}

}  // namespace sgb

using namespace sgb;

extern "C" {

int sgb_bn_forward_training_f32(const float* x, const float* scale, const float* bias,
                                float* running_mean, float* running_var, float factor, float eps,
                                float* y, float* save_mean, float* save_invstd, int N, int C,
                                int HW, void* ws, size_t ws_bytes, void* stream) {
  if (N < 0 || C < 0 || HW < 0) return SGB_ERR_SIZE;
  if (N == 0 || C == 0 || HW == 0) return SGB_OK;
  if (!x || !scale || !bias || !running_mean || !running_var || !y || !save_mean || !save_invstd) return SGB_ERR_NULL;
  const long long per_channel = static_cast<long long>(N) * HW;
  if (per_channel > 0x7fffffffLL || C > 65535) return SGB_ERR_SIZE;
  cudaStream_t s = as_stream(stream);
  const FwdArgs a{x, scale, bias, running_mean, running_var, factor, eps, y, save_mean, save_invstd,
                  BnShape{N, C, HW}, static_cast<size_t>(per_channel) * C};
  const bool bases = aligned16(x) && aligned16(y), vec = HW % 4 == 0 && bases;
  int st = SGB_OK;
  if (bases && fwd_revisit_pays(N, C, HW)) {
    st = vec ? launch_revisit<true>(a, ws, ws_bytes, s) : launch_revisit<false>(a, ws, ws_bytes, s);
    if (st != SGB_ERR_WORKSPACE) return st;
    st = SGB_OK;
  }
  auto small = [&](auto g, auto nv, auto v) {
    constexpr int kG = decltype(g)::value, kNV = decltype(nv)::value;
    st = launch_ex(bn_fwd_small_kernel<kG, kNV, decltype(v)::value>,
                   dim3(static_cast<unsigned>(kG == 32 ? (C + 3) / 4 : C)), dim3(kG == 32 ? 128 : kG), 0, s, 0, true, a);
  };
  if (vec ? small_plan<true, 8>(per_channel / 4, [&](auto g, auto nv) { small(g, nv, std::true_type{}); })
          : small_plan<false, 8>(per_channel, [&](auto g, auto nv) { small(g, nv, std::false_type{}); }))
    return st;
  if (vec) return launch_large<kVec>(a, ws, ws_bytes, s);
  // below eight elements a plane has more edge units than whole ones
  if (bases && HW >= 8 && static_cast<long long>(N) * ragged_units(HW) <= 0x7fffffffLL)
    return launch_large<kRagged>(a, ws, ws_bytes, s);
  return launch_large<kScalar>(a, ws, ws_bytes, s);
}

}  // extern "C"
