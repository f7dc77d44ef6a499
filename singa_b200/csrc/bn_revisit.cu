// Batch-norm backward in two visits (see bn_revisit.cuh): the sums of a channel's
// items, then dx from the same operands, out of L2.
#include "bn_revisit.cuh"

#include <chrono>


namespace sgb {

unsigned long long revisit_tag() {
  static const unsigned long long salt =
      static_cast<unsigned long long>(std::chrono::steady_clock::now().time_since_epoch().count()) ^ 0x5851f42d4c957f2dull;
  static std::atomic<unsigned long long> launches{0};
  // the mixer of SplitMix64 (G. L. Steele, D. Lea, C. H. Flood, 2014), a bijection: the tags differ
  unsigned long long z = salt + 0x9e3779b97f4a7c15ull * ++launches;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  z ^= z >> 31;
  return z ? z : 1;                    // 0 is a tag taken away
}

namespace {

__device__ RevisitState g_revisit_state;

// Four vectors of x, dy and the ReLU's input are 48 registers, and four CTAs of
// 256 threads fill an SM; the masked ends of ragged planes need registers for
// themselves.  Of 1 to 4 vectors, 192 to 320 threads and 3 to 7 CTAs (us, the form
// that a channel took before / this one / the range of the others):
//   32x64x112x112 with ReLU 101.1 / 73.4 / 73.9-78.0, without 79.1 / 54.0 / 53.9-55.5
//   32x256x56x56            76.0 / 70.5 / 71.5-77.3            57.8 / 53.8 / 54.6-55.8
//   32x512x28x28            45.6 / 37.9 / 38.8-41.0            34.1 / 30.3 / 30.1-31.1
//   32x64x56x56             24.6 / 20.6 / 21.1-21.9            18.3 / 16.4 / 16.8-17.6
//   32x128x57x57            66.0 / 45.8 / 47.8-53.3            46.6 / 38.5 / 40.4-47.4
// (Those are from when the exchange had fences, see bn_revisit.cuh; now, with / without:
// 32x256x56x56 68.0 / 51.2, 32x512x28x28 36.4 / 28.2, 32x64x56x56 19.8 / 15.4, 32x128x57x57
// 42.0 / 32.5.)
template <bool MASKED, bool VEC>
constexpr RevisitShape kBwd = VEC ? RevisitShape{4, 224, 4} : RevisitShape{2, 288, MASKED ? 4 : 5};

// Whether what is to be finished is asked for before the CTA's warps meet to add up, and
// so is on its way while they do.  Odd planes, whose masked ends make a CTA's reduction
// long: 32x128x57x57 38.5 -> 35.3 us, with a ReLU (and four CTAs, for the registers) 44.9
// -> 43.4; 24x64x71x71 23.9 -> 22.6 and 27.9 -> 27.4.  Whole vectors gain nothing (53.3 ->
// 53.2), and with a ReLU the registers that it takes cost more (69.8 -> 71.9).
//
// What did not help either (us, 32x256x56x56 with / without a ReLU, 69.7 / 53.4): the second
// visit through shared memory by asynchronous copies that start with the first (74.1 /
// 54.9); a join in front taken into both visits (124.4 with its 24 bytes an element, the
// join and this kernel apart 110.0: four operands leave too little of them in L2).
template <bool VEC>
constexpr bool kEarly = !VEC;

struct BwdArgs {
  const float *x, *dy, *relu, *scale, *mean, *invstd;
  float *dx, *dscale, *dbias;
  unsigned numel;
  float inv_m;
  Revisit r;
};

// The last warp fetches the sums and forms the coefficients of the item to be
// finished while the others load and add up the item to be summed.
template <int MASK, bool VEC>
__global__ void __launch_bounds__(kBwd<MASK != 0, VEC>.threads + 32, kBwd<MASK != 0, VEC>.per_sm)
bn_bwd_revisit_kernel(const __grid_constant__ BwdArgs a) {
  constexpr int NV = kBwd<MASK != 0, VEC>.units;
  __shared__ float2 sm[kBwd<MASK != 0, VEC>.threads / 32];
  __shared__ float4 coef;
  __shared__ bool stopped;
  const unsigned item = blockIdx.x, mine = item - a.r.delay, threads = blockDim.x - 32;
  const bool summing = static_cast<int>(item) < a.r.items, finishing = static_cast<int>(item) >= a.r.delay;
  if (threadIdx.x >= threads) {
    dependency_wait();
    release_dependents();
    if (summing) revisit_open(a.r, item);
    if (!finishing) return;
    const unsigned c = a.r.parts.quot(mine);
    const float sc = a.scale[c], r = a.invstd[c], mu = a.mean[c];
    float s = 0.f, t = 0.f;
    unsigned base;
    const bool got = revisit_gather(a.r, c, base, [&](unsigned, float p, float q) {
      s += p;
      t += q;
    });
    s = warp_sum(s);
    t = warp_sum(t);
    if ((threadIdx.x & 31) == 0) {
      stopped = !got;
      const float ds = t * r;
      coef = make_float4(sc * r, s * a.inv_m, ds * r * a.inv_m, mu);
      if (got && mine == c * a.r.parts.d) {
        a.dscale[c] = ds;
        a.dbias[c] = s;
      }
    }
    revisit_arrive(2, blockDim.x);
    if (got) revisit_leave(a.r, c, base);
    return;
  }
  // loads of all units at once; what is not there is 0
  Vec4f vx[NV], vg[NV], vm[NV];
  auto load = [&](const RevisitUnits<VEC, NV>& u, unsigned long long policy) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      vx[k].u = vg[k].u = vm[k].u = make_uint4(0, 0, 0, 0);
      if (u.valid[k]) {
        vx[k] = u.load(a.x, k, a.numel, policy);
        vg[k] = u.load(a.dy, k, a.numel, policy);
        if (MASK == 1) vm[k] = u.load(a.relu, k, a.numel, policy);
        if (MASK == 2) vm[k].i[0] = static_cast<int>(keep4<2>(a.relu, u.off[k]));
      }
    }
  };
  auto gradient = [&](int k, int j) {
    const float g = vg[k].f[j];
    if (MASK == 1) return vm[k].f[j] > 0 ? g : 0.0f;
    if (MASK == 2) return (vm[k].i[0] >> j) & 1 ? g : 0.0f;
    return g;
  };
  float s = 0.f, t = 0.f;
  if (summing) {
    const RevisitUnits<VEC, NV> u(a.r, item, threads);
    // the first CTAs wait for DRAM while the previous kernel drains; dy may be its output
    if (first_wave(kBwd<MASK != 0, VEC>.per_sm)) {
#pragma unroll
      for (int k = 0; k < NV; ++k)
        if (u.valid[k] && (VEC || u.off[k] < a.numel)) {
          prefetch_l2(a.x + u.off[k]);
          if (MASK == 1) prefetch_l2(a.relu + u.off[k]);
        }
    }
    dependency_wait();
    load(u, keep_policy());
    const float mu = a.mean[u.c];
#pragma unroll
    for (int k = 0; k < NV; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (VEC || u.valid[k] >> j & 1u) {
          const float g = gradient(k, j);              // 0 where there is no unit
          s += g;
          t += g * (vx[k].f[j] - mu);
        }
  } else {
    dependency_wait();
  }
  // What is to be finished is asked for before the warps meet: it is on its way while
  // they add up, and while the slowest of them still waits for its operands.
  RevisitUnits<VEC, NV> u(a.r, finishing ? mine : item, threads);
  if (kEarly<VEC> && finishing) load(u, drop_policy());
  if (summing) {
    s = warp_sum(s);
    t = warp_sum(t);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = make_float2(s, t);
    revisit_sync(1, threads);
    if (threadIdx.x == 0) {
      s = t = 0.f;
      for (unsigned w = 0; w < threads / 32; ++w) {
        s += sm[w].x;
        t += sm[w].y;
      }
      put_entry(a.r.entries + item, s, t, a.r.tag);
    }
  }
  if (!finishing) return;
  if (!kEarly<VEC>) load(u, drop_policy());
  revisit_sync(2, blockDim.x);
  if (stopped) return;
  const float k_ = coef.x, am = coef.y, bm = coef.z, mu = coef.w;
#pragma unroll
  for (int k = 0; k < NV; ++k)
    if (u.valid[k]) {
      Vec4f o;
#pragma unroll
      for (int j = 0; j < 4; ++j) o.f[j] = k_ * (gradient(k, j) - am - (vx[k].f[j] - mu) * bm);
      u.store(a.dx, k, o);
    }
}

}  // namespace

RevisitState* revisit_state(int* status) {
  static std::atomic<RevisitState*> cached[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) {
    *status = e != cudaSuccess ? note_cuda_error(e) : SGB_ERR_UNSUPPORTED;
    return nullptr;
  }
  *status = SGB_OK;
  RevisitState* p = cached[dev].load(std::memory_order_acquire);
  if (p) return p;
  void* q = nullptr;
  e = cudaGetSymbolAddress(&q, g_revisit_state);
  if (e != cudaSuccess) {
    *status = note_cuda_error(e);
    return nullptr;
  }
  cached[dev].store(static_cast<RevisitState*>(q), std::memory_order_release);
  return static_cast<RevisitState*>(q);
}

int revisit_faults(unsigned* flags) {
  const cudaError_t e = cudaMemcpyFromSymbol(flags, g_revisit_state, sizeof(unsigned));
  return e == cudaSuccess ? SGB_OK : note_cuda_error(e);
}

size_t bn_revisit_workspace_bytes(int N, int C, int HW) {
  const int upp = HW % 4 ? ragged_units(HW) : HW / 4;
  RevisitPlan p;
  return revisit_plan(HW % 4 ? kBwd<false, false> : kBwd<false, true>, static_cast<long long>(N) * upp, upp, C, &p) ? p.bytes : 0;
}

int bn_revisit_backward(int mask, const float* x, const float* dy, const float* relu, const float* scale,
                        const float* mean, const float* invstd, float* dx, float* dscale, float* dbias, int N, int C,
                        int HW, void* ws, size_t ws_bytes, cudaStream_t s) {
  const bool vec = HW % 4 == 0;
  const int upp = vec ? HW / 4 : ragged_units(HW);
  const long long units = static_cast<long long>(N) * upp;
  const RevisitShape shape = vec ? (mask ? kBwd<true, true> : kBwd<false, true>)
                                 : (mask ? kBwd<true, false> : kBwd<false, false>);
  RevisitPlan p;
  if (!ws || !aligned16(ws) || !revisit_plan(shape, units, upp, C, &p) || ws_bytes < p.bytes) return SGB_ERR_WORKSPACE;
  int st = SGB_OK;
  RevisitState* state = revisit_state(&st);
  if (!state) return st;
  const BwdArgs a{x, dy, relu, scale, mean, invstd, dx, dscale, dbias,
                  static_cast<unsigned>(N) * static_cast<unsigned>(C) * static_cast<unsigned>(HW),
                  1.0f / (static_cast<float>(N) * static_cast<float>(HW)),
                  revisit_args(p, units, upp, C, HW, ws, state)};
  auto kernel = mask == 0   ? (vec ? bn_bwd_revisit_kernel<0, true> : bn_bwd_revisit_kernel<0, false>)
                : mask == 1 ? (vec ? bn_bwd_revisit_kernel<1, true> : bn_bwd_revisit_kernel<1, false>)
                            : (vec ? bn_bwd_revisit_kernel<2, true> : bn_bwd_revisit_kernel<2, false>);
  return launch_ex(kernel, dim3(static_cast<unsigned>(p.items + p.delay)), dim3(p.threads + 32), 0, s, 0, true, a);
}

}  // namespace sgb
