// Shared device/host helpers for the sm_100a kernels behind the C ABI.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <utility>

#include "sgb.h"

namespace sgb {

// Number of SMs of the current device (148 on B200), cached per device.
int sm_count();

// Records a CUDA runtime error so sgb_last_cuda_error() can report it.
int note_cuda_error(cudaError_t e);

// Returns SGB_OK or SGB_ERR_CUDA after a kernel launch (launch errors only;
// nothing here synchronises).
inline int launch_status() {
  cudaError_t e = cudaPeekAtLastError();
  return e == cudaSuccess ? SGB_OK : note_cuda_error(cudaGetLastError());
}

inline bool aligned16(const void* p) {
  return (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
}

inline cudaStream_t as_stream(void* s) { return static_cast<cudaStream_t>(s); }

inline size_t ceil_div(size_t a, size_t b) { return (a + b - 1) / b; }

// Library-wide switches (sgb_set_option); read on the host at launch time.
int option(int which);

// Launch with optional attributes: a thread-block cluster of `cluster` CTAs
// along x (0 = none) and, when SGB_OPT_OVERLAP_LAUNCHES is on and the kernel
// is `dependent_aware`, programmatic stream serialisation: the grid may be
// scheduled while the previous kernel of the stream drains, and the kernel
// itself waits (dependency_wait) before it touches global memory.  Only
// kernels that contain that wait - in every thread, before any exit - may pass
// dependent_aware = true.  Such a launch also costs the host less (1.9 us
// against 2.5 us for a plain one, measured back to back on an idle stream).
template <typename... KArgs, typename... Args>
inline int launch_ex(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                     int cluster, bool dependent_aware, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (cluster > 0) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = static_cast<unsigned>(cluster);
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (dependent_aware && option(SGB_OPT_OVERLAP_LAUNCHES)) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
  if (e != cudaSuccess) return note_cuda_error(e);
  return launch_status();
}

// Grid for a grid-stride kernel: enough CTAs for the work, capped at
// ctas_per_sm resident CTAs on every SM so the grid is a multiple of the SM
// count when the problem is large.
inline unsigned capped_grid(size_t work_items, size_t per_cta, int ctas_per_sm) {
  size_t need = ceil_div(work_items, per_cta);
  size_t cap = static_cast<size_t>(sm_count()) * ctas_per_sm;
  if (need < 1) need = 1;
  return static_cast<unsigned>(need < cap ? need : cap);
}

// n / d for n < 2^31 by multiplication with ceil(2^(31 + l) / d), l = ceil(log2 d):
// division by invariant integers (T. Granlund, P. L. Montgomery, 1994).
struct FastDiv {
  unsigned d, mul, shift;
  explicit FastDiv(unsigned div) : d(div) {
    unsigned l = 0;
    while ((1ull << l) < div) ++l;
    shift = 31 + l;
    mul = static_cast<unsigned>(((1ull << shift) + div - 1) / div);
  }
  __device__ __forceinline__ unsigned quot(unsigned n) const {
    return static_cast<unsigned>((static_cast<unsigned long long>(n) * mul) >> shift);
  }
};

// ---------------------------------------------------------------- device side
// Programmatic dependent launch.  dependency_wait: returns once every kernel
// this grid depends on has completed and its writes are visible (a no-op for
// a grid launched without the attribute).  It must precede the first access
// to global memory.  release_dependents: this CTA no longer needs the SM's
// free resources for CTAs of its own grid; once every CTA of the grid has
// said so (or exited), the next kernel of the stream may be scheduled.
__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void release_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Before dependency_wait() a kernel may still ask for lines to be brought into
// L2: that reads no value, so it cannot see a stale one, and whatever an earlier
// kernel of the stream writes goes through the same L2.  The CTAs of the first
// wave ask for the operands that no running kernel is likely to produce
// (activations, parameters, momentum) and so wait for DRAM while the previous
// kernel drains.  Later waves find that kernel finished and load at once.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ bool first_wave(unsigned ctas_per_sm) {
  unsigned sms;
  asm("mov.u32 %0, %%nsmid;" : "=r"(sms));
  return blockIdx.x < sms * ctas_per_sm;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Block-wide sum with a fixed combination order (deterministic run to run).
// smem must hold 32 floats.  Result valid in every thread.
__device__ __forceinline__ float block_sum(float v, float* smem) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int nwarp = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();  // protects smem reuse across consecutive calls
  if (lane == 0) smem[wid] = v;
  __syncthreads();
  float r = lane < nwarp ? smem[lane] : 0.0f;
  r = warp_sum(r);
  return r;
}

// 128-bit global accesses.  "Streaming" forms mark the line evict-first: the
// gradient tensors on this path are touched once per step.
__device__ __forceinline__ uint4 ld128(const void* p) {
  return *reinterpret_cast<const uint4*>(p);
}
__device__ __forceinline__ uint4 ld128_stream(const void* p) {
  return __ldcs(reinterpret_cast<const uint4*>(p));
}
__device__ __forceinline__ void st128(void* p, uint4 v) {
  *reinterpret_cast<uint4*>(p) = v;
}
__device__ __forceinline__ void st128_stream(void* p, uint4 v) {
  __stcs(reinterpret_cast<uint4*>(p), v);
}

union Vec4f {
  uint4 u;
  float f[4];
  int i[4];
};
// Four floats at an address that need not be a vector's (the same alignment in all
// lanes): tensors of any length lie back to back in a gradient arena.
__device__ __forceinline__ Vec4f ld4(const float* p) {
  Vec4f v;
  const unsigned at = static_cast<unsigned>(reinterpret_cast<uintptr_t>(p));
  if ((at & 15u) == 0) {
    v.u = ld128(p);
  } else if ((at & 7u) == 0) {
    const float2 a = *reinterpret_cast<const float2*>(p), b = *reinterpret_cast<const float2*>(p + 2);
    v.f[0] = a.x; v.f[1] = a.y; v.f[2] = b.x; v.f[3] = b.y;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) v.f[j] = p[j];
  }
  return v;
}
__device__ __forceinline__ void st4(float* p, const Vec4f& v) {
  const unsigned at = static_cast<unsigned>(reinterpret_cast<uintptr_t>(p));
  if ((at & 15u) == 0) {
    st128(p, v.u);
  } else if ((at & 7u) == 0) {
    *reinterpret_cast<float2*>(p) = make_float2(v.f[0], v.f[1]);
    *reinterpret_cast<float2*>(p + 2) = make_float2(v.f[2], v.f[3]);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) p[j] = v.f[j];
  }
}

union Vec8h {
  uint4 u;
  __half h[8];
  __half2 h2[4];
};

}  // namespace sgb
