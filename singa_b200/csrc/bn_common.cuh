// What the batch-norm forward and backward kernels share: the walk over a
// channel's units, ReLU decisions, asynchronous copies, units of planes that
// are not a multiple of four floats, and launch helpers.
#pragma once
#include <cooperative_groups.h>

#include <atomic>
#include <type_traits>

#include "bulk_copy.cuh"
#include "common.cuh"

namespace sgb {

// Sticky fault word of the forward cluster kernel (0: none), see batchnorm.cu.
int bn_forward_faults(unsigned* flags);
// What the forward form needs beyond the partial sums of two passes.
size_t bn_forward_workspace_bytes(int N, int C, int HW);

namespace {

constexpr int kBlock = 256;
constexpr int kMaxSlices = 64;

// Opts a kernel in to more than 48 KB of dynamic shared memory (and, for the
// cluster kernels, to non-portable cluster sizes) once per device: the
// attribute sticks to the function in that device's context, so later
// launches - including launches under stream capture - issue no attribute
// call.  `done` is one flag per device ordinal; ordinals beyond the table are
// set every time.  Racing first calls from two host threads both set the
// same attribute, which is harmless.
template <typename K>
int opt_in_once(K kernel, std::atomic<bool>* done, bool cluster) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
  const bool tracked = dev >= 0 && dev < 64;
  if (tracked && done[dev].load(std::memory_order_acquire)) return SGB_OK;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
  if (e != cudaSuccess) return note_cuda_error(e);
  if (cluster) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return note_cuda_error(e);
  }
  if (tracked) done[dev].store(true, std::memory_order_release);
  return SGB_OK;
}

struct BnShape {
  int N, C, HW;
};

// Walks the units u0 + tid, u0 + tid + T, ... of a share and keeps the
// (plane n, position q) decomposition up to date without a division per step.
struct UnitWalk {
  int n, q, dn, dq, hwu;
  __device__ __forceinline__ UnitWalk(int u, int step, int hwu_) : hwu(hwu_) {
    n = u / hwu_;
    q = u - n * hwu_;
    dn = step / hwu_;
    dq = step - dn * hwu_;
  }
  __device__ __forceinline__ void next() {
    n += dn;
    q += dq;
    if (q >= hwu) {
      q -= hwu;
      ++n;
    }
  }
};

// How the fused ReLU backward learns which gradients to keep.  MASK 0: no ReLU.
// MASK 1: from the ReLU's stored input (keep where it is > 0).  MASK 2: from the
// forward partner's record, one bit per element in element order (bit i & 7 of
// byte i >> 3; 1 = the input was > 0), passed through the same pointer.
// `off` is the element offset; for the 4-wide forms it is a multiple of 4.
template <int MASK>
__device__ __forceinline__ unsigned keep4(const float* relu_in, size_t off) {
  if (MASK == 2) {
    const unsigned char b = reinterpret_cast<const unsigned char*>(relu_in)[off >> 3];
    return (b >> (off & 4)) & 15u;
  }
  Vec4f v;
  v.u = ld128(relu_in + off);
  unsigned bits = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) bits |= (v.f[k] > 0 ? 1u : 0u) << k;
  return bits;
}
template <int MASK>
__device__ __forceinline__ bool keep1(const float* relu_in, size_t off) {
  if (MASK == 2) return (reinterpret_cast<const unsigned char*>(relu_in)[off >> 3] >> (off & 7)) & 1u;
  return relu_in[off] > 0;
}

__host__ __device__ inline int bn_slices_for(long long per_channel, int C, int sms) {
  long long s = (static_cast<long long>(sms) * 16 + C - 1) / C;
  const long long max_s = (per_channel + 2047) / 2048;  // >= 2048 elements per slice
  if (s > max_s) s = max_s;
  if (s > kMaxSlices) s = kMaxSlices;
  return static_cast<int>(s < 1 ? 1 : s);
}

__device__ __forceinline__ void cp_async16(float* smem_dst, const float* gmem_src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Returns once at most PENDING of this thread's most recent copy groups are still in flight.
template <int PENDING>
__device__ __forceinline__ void cp_async_wait_pending() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}
// A thread issues its copies in kCopyGroups groups, so that it can start adding
// up the units of the first group while the later ones are still in flight
// (a thread only ever reads back what it staged itself: no barrier needed).
constexpr int kCopyGroups = 4;


// Planes that are not a multiple of four floats, moved in 16-byte units all the
// same: unit q of plane (n, c) is the q-th ALIGNED vector that touches the
// plane, so its first element lies (plane offset mod 4) elements before the
// plane when q = 0.  The few elements of the neighbouring planes in the first
// and last unit are masked.
struct RaggedUnit {
  size_t off;        // element offset of the vector, a multiple of 4
  unsigned valid;    // which of its four elements belong to the plane
  __device__ __forceinline__ RaggedUnit(size_t plane_off, int q, int hw) {
    const int lead = static_cast<int>(plane_off & 3), e = 4 * q - lead;
    off = plane_off - lead + 4 * static_cast<size_t>(q);
    if (e >= 0 && e + 4 <= hw) {
      valid = 15u;
    } else {
      valid = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) valid |= e + j >= 0 && e + j < hw ? 1u << j : 0u;
    }
  }
};
__host__ __device__ inline int ragged_units(int hw) { return (hw + 6) / 4; }   // per plane, whatever its lead

// The vector at off (0 where it lies behind the tensor's last element).
__device__ __forceinline__ Vec4f ragged_load(const float* p, size_t off, size_t numel) {
  Vec4f v;
  if (off + 4 <= numel) {
    v.u = ld128(p + off);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) v.f[j] = off + j < numel ? p[off + j] : 0.0f;
  }
  return v;
}
__device__ __forceinline__ void ragged_store(float* p, const RaggedUnit& u, const Vec4f& v) {
  if (u.valid == 15u) {
    st128(p + u.off, v.u);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (u.valid >> j & 1u) p[u.off + j] = v.f[j];
  }
}
// Asynchronous copy of the vector into shared memory; the one that reaches
// behind the tensor goes element by element (the same thread reads it back).
__device__ __forceinline__ void ragged_copy(float* smem, const float* p, size_t off, size_t numel) {
  if (off + 4 <= numel) {
    cp_async16(smem, p + off);
  } else {
    *reinterpret_cast<uint4*>(smem) = ragged_load(p, off, numel).u;
  }
}

// Sums over the G threads that share a channel; valid in all of them.  G = 32:
// a warp, else the CTA (sm: 2 * G / 32 floats, used once per kernel and slot).
template <int G, bool TWO>
__device__ __forceinline__ void channel_sums(float& a, float& b, float* sm) {
  a = warp_sum(a);
  if (TWO) b = warp_sum(b);
  if (G == 32) return;
  constexpr int kWarps = G / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    sm[wid] = a;
    if (TWO) sm[kWarps + wid] = b;
  }
  __syncthreads();
  a = 0.f;
  if (TWO) b = 0.f;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    a += sm[w];
    if (TWO) b += sm[kWarps + w];
  }
}

// Cluster size (1, 2, 4 or 8) and per-CTA share for the single-pass kernels;
// returns 0 when a channel does not fit 8 CTAs' shared memory.  unit_bytes:
// what staging one unit of all operands takes.  max_units: per CTA (a fused
// mask keeps the decisions of 16 units per thread of a 512-thread CTA).
inline int cluster_plan(long long units_per_channel, int unit_bytes, int max_units, int* per_cta, int channels) {
  constexpr int max_cs = 8;      // portable cluster size (16-CTA clusters with 50 KB shares measured slower)
  for (const long long cap : {50 * 1024LL, 100 * 1024LL}) {   // preferred: four CTAs per SM; at most: two
    for (int cs = 1; cs <= max_cs; cs *= 2) {
      long long share = (units_per_channel + cs - 1) / cs;
      if (share * unit_bytes <= cap && share <= max_units) {
        // Few channels: a grid that leaves SMs idle is latency bound, so the
        // channel is split further while a share still keeps every thread of a
        // 256-thread CTA busy and there are less than two CTAs per SM
        // (17x48x35x29: 9.4 -> 7.4 us fused, 6.0 -> 5.4; three or more change
        // nothing or cost up to a tenth: 32x128x28x28 13.5 -> 15.7).
        while (cs * 2 <= max_cs && static_cast<long long>(channels) * cs < 2LL * sm_count() &&
               (units_per_channel + 2 * cs - 1) / (2 * cs) >= 512) {
          cs *= 2;
          share = (units_per_channel + cs - 1) / cs;
        }
        *per_cta = static_cast<int>(share);
        return cs;
      }
    }
  }
  return 0;
}

// The number of threads and of units per thread that hold a channel of `units`
// in registers (at most MOST vectors per thread); F is called with them as
// constants.  False: too large.
template <bool VEC, int MOST, typename F>
bool small_plan(long long units, F f) {
  constexpr int kM = VEC ? 1 : 2;     // a scalar unit takes a quarter of the registers
#define SGB_BN_SMALL(G, NV)                                                     \
  if (units <= static_cast<long long>(G) * (NV)) {                              \
    f(std::integral_constant<int, G>{}, std::integral_constant<int, (NV)>{});   \
    return true;                                                                \
  }
  SGB_BN_SMALL(32, 1 * kM)
  SGB_BN_SMALL(32, 2 * kM)
  SGB_BN_SMALL(32, 4 * kM)
  SGB_BN_SMALL(128, 2 * kM)
  SGB_BN_SMALL(128, 4 * kM)
  SGB_BN_SMALL(256, 4 * kM)
  SGB_BN_SMALL(256, MOST * kM)
#undef SGB_BN_SMALL
  return false;
}

}  // namespace
}  // namespace sgb
