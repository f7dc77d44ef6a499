// Batch-normalisation backward (training mode) with saved mean and saved
// inverse standard deviation:
//   dbias[c]  = sum dy
//   dscale[c] = sum dy * (x - mean[c]) * invstd[c]
//   dx        = scale[c] * invstd[c] *
//               (dy - dbias[c]/M - (x - mean[c]) * invstd[c] * dscale[c] / M)
// M = N*H*W (spatial mode, NCHW) or N (per-activation mode, N x D).
//
// One pass over HBM (12 bytes per element) wherever a channel can be held while
// its two sums form, in this order of preference:
//   registers  a warp or a CTA holds a channel of up to a few thousand elements
//              (bn_bwd_small_kernel);
//   groups     planes that are no multiple of four floats: a CTA stages the 2 or
//              4 adjacent channels that make an aligned run (bn_bwd_group_kernel;
//              also ahead of the registers for larger calls without a mask, see
//              bn_backward);
//   ragged     such planes when a channel needs a cluster: the aligned vectors
//              that touch a plane, ends masked (bn_bwd_ragged_kernel);
//   hybrid     a cluster of up to 8 CTAs shares a channel, part of the gradient
//              stays in registers: three CTAs per SM where shared memory alone
//              would leave two (bn_bwd_hybrid_kernel);
//   cluster    the same with all of x and dy staged in shared memory by 16-byte
//              asynchronous copies (cp.async, no register staging): every CTA
//              reduces its share with warp shuffles, the CTAs exchange their two
//              partial sums through distributed shared memory, and dx is computed
//              from the staged copy; two to four CTAs per SM, so that the load
//              phase of one overlaps the store phase of another
//              (bn_bwd_cluster_kernel);
//   streaming  channels too large for a cluster (e.g. 32 x 112 x 112) and calls
//              whose workspace is too small for the form below: persistent
//              small CTAs take 50 KB items of a channel from a ticket counter and
//              meet through counters in global memory (bn_stream.cu).
// Ahead of them all, for large calls whose channels are not too large (revisit_pays):
// two visits to the data in one kernel, the second out of L2 (bn_revisit.cu).
//
// Two passes (20 bytes of HBM traffic per element when the tensor does not fit
// L2) for what is left: ragged planes too large for a cluster, misaligned
// operands or planes below eight floats too large for one, channels that the
// streaming kernel cannot cut or more than 4096 of them, and the entry point
// without workspace:
//   pass 1  grid (slices, C): a CTA walks its slice of the channel's flattened
//           (n, hw) space, with 128-bit loads where it can, and leaves two partial
//           sums in the workspace (no atomics, fixed order -> run-to-run identical);
//   pass 2  grid (tiles, C): every CTA first adds the channel's <= 64 partials
//           in one warp (the same order in every CTA), then streams
//           dx for its 1024-unit tile.  CTAs with blockIdx.x == 0 also store
//           dscale/dbias.
// The optional ReLU mask fuses "dy = relu_in > 0 ? dy : 0" (the backward of
// the ReLU that follows the BN layer) into every form, which removes one
// full write + read of the intermediate gradient.
#include "bn_common.cuh"
#include "bn_revisit.cuh"
#include "bn_stream.cuh"

namespace cg = cooperative_groups;

namespace sgb {
namespace {

template <bool VEC, int MASK>
__global__ void __launch_bounds__(kBlock)
bn_bwd_reduce_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                     const float* __restrict__ relu_in, const float* __restrict__ mean,
                     float2* __restrict__ partial, BnShape sh, int per_slice) {
  __shared__ float sm[32];
  const int c = blockIdx.y, slice = blockIdx.x;
  dependency_wait();
  const float mu = mean[c];
  float s_dy = 0.f, s_dyx = 0.f;
  if (VEC) {
    const int hw4 = sh.HW >> 2, total = sh.N * hw4;
    const int i0 = slice * per_slice, i1 = min(i0 + per_slice, total);
    UnitWalk w(i0 + threadIdx.x, kBlock, hw4);
    for (int i = i0 + threadIdx.x; i < i1; i += kBlock, w.next()) {
      const size_t off = (static_cast<size_t>(w.n) * sh.C + c) * sh.HW + 4 * w.q;
      Vec4f vx, vg, vm;
      vx.u = ld128(x + off);
      vg.u = ld128(dy + off);
      unsigned bits = 15u;
      if (MASK == 1) vm.u = ld128(relu_in + off);
      if (MASK == 2) bits = keep4<2>(relu_in, off);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float g = vg.f[k];
        if (MASK == 1) g = vm.f[k] > 0 ? g : 0.0f;
        if (MASK == 2) g = (bits >> k) & 1u ? g : 0.0f;
        s_dy += g;
        s_dyx += g * (vx.f[k] - mu);
      }
    }
  } else {
    const int total = sh.N * sh.HW;
    const int i0 = slice * per_slice, i1 = min(i0 + per_slice, total);
    for (int i = i0 + threadIdx.x; i < i1; i += kBlock) {
      const int n = i / sh.HW, q = i - n * sh.HW;
      const size_t off = (static_cast<size_t>(n) * sh.C + c) * sh.HW + q;
      float g = dy[off];
      if (MASK) g = keep1<MASK>(relu_in, off) ? g : 0.0f;
      s_dy += g;
      s_dyx += g * (x[off] - mu);
    }
  }
  release_dependents();
  s_dy = block_sum(s_dy, sm);
  s_dyx = block_sum(s_dyx, sm);
  if (threadIdx.x == 0)
    partial[static_cast<size_t>(c) * gridDim.x + slice] = make_float2(s_dy, s_dyx);
}

// Units (16-byte vectors, or floats when !VEC) per thread of the apply pass:
// the coefficient lookup and the barrier are paid once per CTA, so more units
// per CTA make them cheaper per byte.
constexpr int kApplyUnits = 4;

template <bool VEC, int MASK>
__global__ void __launch_bounds__(kBlock)
bn_bwd_apply_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                    const float* __restrict__ relu_in, const float* __restrict__ scale,
                    const float* __restrict__ mean, const float* __restrict__ invstd,
                    const float2* __restrict__ partial, int slices, float* __restrict__ dx,
                    float* __restrict__ dscale, float* __restrict__ dbias, BnShape sh) {
  __shared__ float coef[4];
  // channels in DESCENDING order: the reduce pass walked them ascending, so the
  // last ones it touched are the ones most likely still in L2
  const int c = sh.C - 1 - blockIdx.y;
  // issue this thread's loads first, so that their latency overlaps the
  // partial-sum lookup below
  constexpr int kW = VEC ? 4 : 1;
  const int hwu = sh.HW / kW, total = sh.N * hwu;
  const int unit0 = blockIdx.x * (kBlock * kApplyUnits) + threadIdx.x;
  size_t off[kApplyUnits];
  Vec4f vx[kApplyUnits], vg[kApplyUnits], vm[kApplyUnits];
  UnitWalk w(min(unit0, total - 1), kBlock, hwu);
  dependency_wait();
#pragma unroll
  for (int j = 0; j < kApplyUnits; ++j) {
    vx[j].f[0] = vg[j].f[0] = vm[j].f[0] = 0.f;
    off[j] = 0;
    if (unit0 + j * kBlock < total) {
      off[j] = (static_cast<size_t>(w.n) * sh.C + c) * sh.HW + static_cast<size_t>(w.q) * kW;
      if (VEC) {
        vx[j].u = ld128(x + off[j]);
        vg[j].u = ld128(dy + off[j]);
        if (MASK == 1) vm[j].u = ld128(relu_in + off[j]);
        if (MASK == 2) vm[j].i[0] = static_cast<int>(keep4<2>(relu_in, off[j]));
      } else {
        vx[j].f[0] = x[off[j]];
        vg[j].f[0] = dy[off[j]];
        if (MASK == 1) vm[j].f[0] = relu_in[off[j]];
        if (MASK == 2) vm[j].i[0] = keep1<2>(relu_in, off[j]) ? 1 : 0;
      }
      w.next();
    }
  }
  if (threadIdx.x < 32) {
    // add the channel's partials: lanes take slices lane, lane+32; fixed order
    float a = 0.f, b = 0.f;
    for (int k = threadIdx.x; k < slices; k += 32) {
      const float2 p = partial[static_cast<size_t>(c) * slices + k];
      a += p.x;
      b += p.y;
    }
    a = warp_sum(a);
    b = warp_sum(b);
    if (threadIdx.x == 0) {
      const float r = invstd[c];
      const float inv_m = 1.0f / (static_cast<float>(sh.N) * static_cast<float>(sh.HW));
      const float ds = b * r;
      coef[0] = scale[c] * r;       // k
      coef[1] = a * inv_m;          // mean of dy
      coef[2] = ds * r * inv_m;     // slope on (x - mean)
      coef[3] = mean[c];
      if (blockIdx.x == 0) {
        dscale[c] = ds;
        dbias[c] = a;
      }
    }
  }
  __syncthreads();
  release_dependents();
  const float k = coef[0], a = coef[1], b = coef[2], mu = coef[3];
#pragma unroll
  for (int j = 0; j < kApplyUnits; ++j) {
    if (unit0 + j * kBlock >= total) break;
    if (VEC) {
      Vec4f o;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float g = vg[j].f[i];
        if (MASK == 1) g = vm[j].f[i] > 0 ? g : 0.0f;
        if (MASK == 2) g = (vm[j].i[0] >> i) & 1 ? g : 0.0f;
        o.f[i] = k * (g - a - (vx[j].f[i] - mu) * b);
      }
      st128(dx + off[j], o.u);
    } else {
      float g = vg[j].f[0];
      if (MASK == 1) g = vm[j].f[0] > 0 ? g : 0.0f;
      if (MASK == 2) g = vm[j].i[0] & 1 ? g : 0.0f;
      dx[off[j]] = k * (g - a - (vx[j].f[0] - mu) * b);
    }
  }
}

// ----------------------------------------------------------- single pass
// CTA size of the single-pass kernel: 512 threads for large shares (fewer
// serial iterations per thread), 256 for small ones.

// Sticky fault word of the cluster kernel's exchange: bit 0 = the wait for the
// peers' pairs ran out of iterations (that launch's outputs are void).
__device__ unsigned g_cluster_faults;

// grid.x = C * CS with cluster dimension CS: the CS CTAs of a cluster share
// channel blockIdx.x / CS.  A "unit" is one float4 (VEC) or one float.
// Dynamic shared memory: 2 * per_cta units (x share, then dy share).
// ADD (only with VEC): the incoming gradient is the join dy + dy_b masked by
// the ReLU input; it is formed while staging, kept in shared memory for the
// two later phases and ALSO written to `joined` for the other consumers of the
// join (the shortcut branch), which replaces a separate join+ReLU kernel.
// This thread's units of a share, for L2 (see prefetch_l2): x and, where there
// is one, the ReLU's input.
__device__ __forceinline__ void prefetch_share(const float* x, const float* relu_in, int first, int u1, int threads,
                                               int hwu, size_t plane_stride, size_t chan_off) {

  UnitWalk w(first, threads, hwu);
  for (int u = first; u < u1; u += threads, w.next()) {
    const size_t off = w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4;
    prefetch_l2(x + off);
    if (relu_in) prefetch_l2(relu_in + off);
  }
}

template <bool VEC, int MASK, int T, bool ADD = false>
__global__ void __launch_bounds__(T)
bn_bwd_cluster_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                      const float* __restrict__ relu_in, const float* __restrict__ scale,
                      const float* __restrict__ mean, const float* __restrict__ invstd,
                      float* __restrict__ dx, float* __restrict__ dscale,
                      float* __restrict__ dbias, BnShape sh, int per_cta,
                      bool early, const float* __restrict__ dy_b = nullptr, float* __restrict__ joined = nullptr) {
  extern __shared__ __align__(16) float stage[];
  __shared__ unsigned long long pairs_in;          // mbarrier: counts the peers' pairs as they land
  __shared__ float red[2 * T / 32];
  __shared__ float2 parts[16];   // (sum dy, sum dy*(x-mean)) of every CTA of the cluster
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = static_cast<int>(cluster.num_blocks());
  const int rank = static_cast<int>(cluster.block_rank());
  const int c = blockIdx.x / cs;
  if (threadIdx.x == 0) {
    mbar_init(&pairs_in, 1);
    fence_mbarrier_init();                            // visible to the peers once the cluster barrier completes
  }
  cluster.barrier_arrive();                           // matched by barrier_wait before the exchange
  constexpr int kW = VEC ? 4 : 1;                     // floats per unit
  const int hwu = sh.HW / kW;                         // units per plane
  const int total = sh.N * hwu;
  const int u0 = min(rank * per_cta, total), u1 = min(u0 + per_cta, total);
  const int first = u0 + threadIdx.x;
  float* sx = stage;
  float* sg = stage + static_cast<size_t>(per_cta) * kW;
  const size_t plane_stride = static_cast<size_t>(sh.C) * sh.HW;
  const size_t chan_off = static_cast<size_t>(c) * sh.HW;
  if (VEC && first_wave(2)) prefetch_share(x, MASK == 1 || ADD ? relu_in : nullptr, first, u1, T, hwu, plane_stride, chan_off);
  dependency_wait();                                  // first access to global memory follows
  // see leaves_room()
  if (early) release_dependents();
  const float mu = mean[c];
  // units of one copy group per thread (the same in every thread: kCopyGroups * group_units covers a share)
  const int group_units = ((per_cta + T - 1) / T + kCopyGroups - 1) / kCopyGroups;

  // phase 1: stage this CTA's share (asynchronous 16-byte copies, all in flight at once)
  if (VEC && ADD) {
    UnitWalk w(first, T, hwu);
    for (int u = first; u < u1;) {
      // two units per round: x by asynchronous copy, the three gradient-side
      // operands through registers (six independent 16-byte loads in flight)
      Vec4f va[2], vb[2], vr[2];
      size_t offs[2];
      int ls[2], cnt = 0;
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (u < u1) {
          offs[j] = w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4;
          ls[j] = (u - u0) * 4;
          cp_async16(sx + ls[j], x + offs[j]);
          va[j].u = ld128(dy + offs[j]);
          vb[j].u = ld128(dy_b + offs[j]);
          vr[j].u = ld128(relu_in + offs[j]);
          u += T;
          w.next();
          cnt = j + 1;
        }
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (j < cnt) {
          Vec4f g;
#pragma unroll
          for (int k = 0; k < 4; ++k) g.f[k] = vr[j].f[k] > 0 ? (va[j].f[k] + vb[j].f[k]) : 0.0f;
          *reinterpret_cast<uint4*>(sg + ls[j]) = g.u;
          st128(joined + offs[j], g.u);
        }
      }
    }
  } else if (VEC) {
    UnitWalk w(first, T, hwu);
    int u = first;
#pragma unroll
    for (int g = 0; g < kCopyGroups; ++g) {
      for (int k = 0; k < group_units && u < u1; ++k, u += T, w.next()) {
        const size_t off = w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4;
        const int l = (u - u0) * 4;
        cp_async16(sx + l, x + off);
        cp_async16(sg + l, dy + off);
      }
      cp_async_commit();
    }
  } else {
    UnitWalk w(first, T, hwu);
    for (int u = first; u < u1; u += T, w.next()) {
      const size_t off = w.n * plane_stride + chan_off + static_cast<size_t>(w.q);
      const int l = u - u0;
      float g = dy[off];
      if (MASK) g = keep1<MASK>(relu_in, off) ? g : 0.0f;
      sx[l] = x[off];
      sg[l] = g;
    }
  }
  // fused ReLU: while the copies fly, read the ReLU input and keep only the
  // sign decisions, 4 bits per unit (a share is at most 16 units per thread)
  unsigned long long keep = 0;
  if (VEC && MASK == 2 && !ADD) {
    // bit record: one byte holds the decisions of two units
    UnitWalk w(first, T, hwu);
    int slot = 0;
    for (int u = first; u < u1;) {
      // the byte loads of up to 8 units are issued together, then combined
      unsigned char rec[8];
      unsigned shift[8];
      int cnt = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (u < u1) {
          const size_t off = w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4;
          rec[j] = reinterpret_cast<const unsigned char*>(relu_in)[off >> 3];
          shift[j] = static_cast<unsigned>(off & 4);
          u += T;
          w.next();
          cnt = j + 1;
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j < cnt) {
          keep |= static_cast<unsigned long long>((rec[j] >> shift[j]) & 15u) << slot;
          slot += 4;
        }
      }
    }
  } else if (VEC && MASK && !ADD) {
    UnitWalk w(first, T, hwu);
    int slot = 0;
    for (int u = first; u < u1;) {
      // up to 8 independent 16-byte loads in flight per thread, then the sign tests
      Vec4f vm[8];
      int cnt = 0;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (u < u1) {
          const size_t off = w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4;
          vm[j].u = ld128(relu_in + off);
          u += T;
          w.next();
          cnt = j + 1;
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j < cnt) {
          unsigned bits = 0;
#pragma unroll
          for (int k = 0; k < 4; ++k) bits |= (vm[j].f[k] > 0 ? 1u : 0u) << k;
          keep |= static_cast<unsigned long long>(bits) << slot;
          slot += 4;
        }
      }
    }
  }
  if (VEC && ADD) cp_async_wait_all();

  // phase 2: partial sums over the share (each thread re-reads what it staged),
  // copy group by copy group as the groups land; the order of the additions is
  // the order of the units, whatever the grouping
  float s_dy = 0.f, s_dyx = 0.f;
  if (VEC) {
    int slot = 0, u = first;
    auto sum_copy_group = [&]() {
      for (int k = 0; k < group_units && u < u1; ++k, u += T, slot += 4) {
        const int l = (u - u0) * 4;
        Vec4f vx, vg;
        vx.u = *reinterpret_cast<const uint4*>(sx + l);
        vg.u = *reinterpret_cast<const uint4*>(sg + l);
        if (MASK && !ADD) {
          const unsigned bits = static_cast<unsigned>(keep >> slot);
#pragma unroll
          for (int q = 0; q < 4; ++q) vg.f[q] = (bits >> q) & 1u ? vg.f[q] : 0.0f;
          *reinterpret_cast<uint4*>(sg + l) = vg.u;    // keep the masked gradient for phase 3
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          s_dy += vg.f[q];
          s_dyx += vg.f[q] * (vx.f[q] - mu);
        }
      }
    };
    static_assert(kCopyGroups == 4, "the waits below are written out for four groups");
    if (!ADD) cp_async_wait_pending<3>();
    sum_copy_group();
    if (!ADD) cp_async_wait_pending<2>();
    sum_copy_group();
    if (!ADD) cp_async_wait_pending<1>();
    sum_copy_group();
    if (!ADD) cp_async_wait_pending<0>();
    sum_copy_group();
  } else {
    for (int u = first; u < u1; u += T) {
      const int l = u - u0;
      s_dy += sg[l];
      s_dyx += sg[l] * (sx[l] - mu);
    }
  }
  // one block reduction for both sums (fixed order), then every CTA pushes its
  // pair into the slot `parts[rank]` of all peers through distributed shared
  // memory; each CTA then owns a full copy, so nobody reads a peer's memory
  // afterwards.
  {
    constexpr int kWarps = T / 32;
    static_assert(kWarps <= 32, "one warp finishes the reduction");
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    s_dy = warp_sum(s_dy);
    s_dyx = warp_sum(s_dyx);
    if (lane == 0) {
      red[wid] = s_dy;
      red[kWarps + wid] = s_dyx;
    }
    __syncthreads();
    if (wid == 0) {
      float p0 = lane < kWarps ? red[lane] : 0.0f;
      float p1 = lane < kWarps ? red[kWarps + lane] : 0.0f;
      p0 = warp_sum(p0);
      p1 = warp_sum(p1);
      cluster.barrier_wait();                       // peers have started: their memory is addressable
      // every pair travels as one asynchronous 8-byte store that also signals the receiver's
      // mbarrier: no second cluster barrier, a CTA goes on as soon as its cs pairs are in
      if (lane == 0) mbar_arrive_expect(&pairs_in, 8u * static_cast<unsigned>(cs));
      if (lane < cs) {
        unsigned remote_slot, remote_bar;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote_slot) : "r"(smem_addr(&parts[rank])), "r"(lane));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote_bar) : "r"(smem_addr(&pairs_in)), "r"(lane));
        const unsigned long long bits = (static_cast<unsigned long long>(__float_as_uint(p1)) << 32) |
                                        static_cast<unsigned long long>(__float_as_uint(p0));
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(remote_slot),
                     "l"(bits), "r"(remote_bar)
                     : "memory");
      }
    } else {
      cluster.barrier_wait();
    }
  }
  // No CTA writes to a peer after this point and none exits before all pairs
  // addressed to it have landed, so the CTAs retire independently.
  {
    bool in = false;
    for (unsigned it = 0; it < (1u << 24) && !in; ++it) in = mbar_try_wait(&pairs_in, 0);
    if (!in) atomicOr(&g_cluster_faults, 1u);
  }

  float a = 0.f, b = 0.f;
  for (int r = 0; r < cs; ++r) {                    // rank order: same totals in every CTA
    a += parts[r].x;
    b += parts[r].y;
  }
  const float r_ = invstd[c];
  const float inv_m = 1.0f / (static_cast<float>(sh.N) * static_cast<float>(sh.HW));
  const float ds = b * r_;
  const float k_ = scale[c] * r_, am = a * inv_m, bm = ds * r_ * inv_m;
  if (rank == 0 && threadIdx.x == 0) {
    dscale[c] = ds;
    dbias[c] = a;
  }

  // phase 3: dx from the staged copy.  From here on this CTA only drains: the
  // next kernel of the stream may take the SM slots that free up.
  if (!early) release_dependents();
  {
    UnitWalk w(first, T, hwu);
    for (int u = first; u < u1; u += T, w.next()) {
      const size_t off = w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * kW;
      const int l = (u - u0) * kW;
      if (VEC) {
        Vec4f vx, vg, o;
        vx.u = *reinterpret_cast<const uint4*>(sx + l);
        vg.u = *reinterpret_cast<const uint4*>(sg + l);
#pragma unroll
        for (int j = 0; j < 4; ++j) o.f[j] = k_ * (vg.f[j] - am - (vx.f[j] - mu) * bm);
        st128(dx + off, o.u);
      } else {
        dx[off] = k_ * (sg[l] - am - (sx[l] - mu) * bm);
      }
    }
  }
}

// ------------------------------------------- single pass, channel groups
// Planes whose size is not a multiple of four floats (7x7 = 49) cannot be
// moved with 16-byte accesses one channel at a time, but G = 4 / gcd(HW, 4)
// ADJACENT channels of one sample form a contiguous, 16-byte aligned run of
// G*HW floats.  One CTA stages the G channels of all N samples (G*N*HW*8
// bytes of shared memory) with 16-byte copies, reduces every channel with a
// sub-group of its threads from shared memory and forms dx from the staged
// copies on the way out: four elements belong to two channels at most.  Such a
// call is one wave that loads, reduces and stores, so each step between counts: with
// the channel's scalars fetched behind the copies and dx formed in place by a pass
// of its own 32x2048x7x7 took 12.8 us (now 10.6), 64x512x7x7 9.8 (7.2); with the
// masked gradient brought in through registers, four units a round, 13.1 (9.7).
constexpr int kGroupBytes = 100 * 1024;               // the two staged operands of a group at most
template <int MASK, int G>
__global__ void __launch_bounds__(kBlock, 4)
bn_bwd_group_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                    const float* __restrict__ relu_in, const float* __restrict__ scale,
                    const float* __restrict__ mean, const float* __restrict__ invstd,
                    float* __restrict__ dx, float* __restrict__ dscale,
                    float* __restrict__ dbias, BnShape sh) {
  extern __shared__ __align__(16) float stage[];
  constexpr int kSub = kBlock / G;                    // threads per channel
  __shared__ float red[2][kBlock / 32];
  __shared__ float4 coef[G];
  const int c0 = blockIdx.x * G;
  const int run = G * sh.HW;                          // floats per sample, multiple of 4
  const int run4 = run >> 2;
  const int units = sh.N * run4;
  float* sx = stage;
  float* sg = stage + static_cast<size_t>(sh.N) * run;
  const size_t sample_stride = static_cast<size_t>(sh.C) * sh.HW;
  const size_t base = static_cast<size_t>(c0) * sh.HW;
  const UnitWalk start(threadIdx.x, kBlock, run4);
  UnitWalk wl = start;
  if (first_wave(2)) prefetch_share(x, MASK == 1 ? relu_in : nullptr, threadIdx.x, units, kBlock, run4, sample_stride, base);
  // channel g is handled by threads [g*kSub, (g+1)*kSub)
  const int g = threadIdx.x / kSub, t = threadIdx.x - g * kSub;
  const int c = c0 + g;
  UnitWalk w(t, kSub, sh.HW);                         // (sample, position) without a division per step
  dependency_wait();
  const float mu = mean[c], r = invstd[c], gain = scale[c];     // on their way with the operands
  for (int u = threadIdx.x; u < units; u += kBlock, wl.next()) {
    const size_t off = wl.n * sample_stride + base + 4 * static_cast<size_t>(wl.q);
    cp_async16(sx + 4 * u, x + off);
    cp_async16(sg + 4 * u, dy + off);
  }
  if (MASK) {
    // what the ReLU keeps of the thread's own units, four bits each, eight loads at a
    // time while the copies are on their way
    constexpr int kWords = (kGroupBytes / 32 + 8 * kBlock - 1) / (8 * kBlock);
    unsigned keep[kWords];
    wl = start;
    int u = threadIdx.x;
#pragma unroll
    for (int k = 0; k < kWords; ++k) {
      keep[k] = 0;
      if (8 * k * kBlock >= units) break;
      Vec4f vm[8];
      unsigned bits[8];
#pragma unroll
      for (int j = 0; j < 8; ++j, u += kBlock, wl.next()) {
        if (u >= units) continue;
        const size_t off = wl.n * sample_stride + base + 4 * static_cast<size_t>(wl.q);
        if (MASK == 1) vm[j].u = ld128(relu_in + off);
        if (MASK == 2) bits[j] = keep4<2>(relu_in, off);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (static_cast<int>(threadIdx.x) + (8 * k + j) * kBlock >= units) continue;
        if (MASK == 1) {
          bits[j] = 0;
#pragma unroll
          for (int i = 0; i < 4; ++i) bits[j] |= (vm[j].f[i] > 0 ? 1u : 0u) << i;
        }
        keep[k] |= (bits[j] & 15u) << (4 * j);
      }
    }
    cp_async_wait_all();
#pragma unroll
    for (int j = 0; j < 8 * kWords; ++j) {
      const int own = threadIdx.x + j * kBlock;
      if (own >= units) break;
      uint4* const at = reinterpret_cast<uint4*>(sg + 4 * own);
      Vec4f v;
      v.u = *at;
#pragma unroll
      for (int i = 0; i < 4; ++i) v.f[i] = (keep[j / 8] >> (4 * (j % 8) + i)) & 1u ? v.f[i] : 0.0f;
      *at = v.u;
    }
  } else {
    cp_async_wait_all();
  }
  __syncthreads();
  // element (n, i) of the channel sits at staged offset n*run + g*HW + i
  const int per = sh.N * sh.HW;
  float s_dy = 0.f, s_dyx = 0.f;
  int e = t;
  for (constexpr int kAhead = 4; e + (kAhead - 1) * kSub < per; e += kAhead * kSub) {
    float vg[kAhead], vx[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j, w.next()) {
      const int l = w.n * run + g * sh.HW + w.q;
      vg[j] = sg[l];
      vx[j] = sx[l];
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      s_dy += vg[j];
      s_dyx += vg[j] * (vx[j] - mu);
    }
  }
  for (; e < per; e += kSub, w.next()) {
    const int l = w.n * run + g * sh.HW + w.q;
    s_dy += sg[l];
    s_dyx += sg[l] * (sx[l] - mu);
  }
  // reduce inside the sub-group (kSub is a multiple of 32: whole warps per channel)
  s_dy = warp_sum(s_dy);
  s_dyx = warp_sum(s_dyx);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    red[0][wid] = s_dy;
    red[1][wid] = s_dyx;
  }
  __syncthreads();
  if (t == 0) {
    constexpr int kWarpsPer = kSub / 32;
    float a = 0.f, b = 0.f;
    for (int w = 0; w < kWarpsPer; ++w) {
      a += red[0][g * kWarpsPer + w];
      b += red[1][g * kWarpsPer + w];
    }
    const float inv_m = 1.0f / (static_cast<float>(sh.N) * static_cast<float>(sh.HW));
    const float ds = b * r;
    coef[g] = make_float4(gain * r, a * inv_m, ds * r * inv_m, mu);
    dscale[c] = ds;
    dbias[c] = a;
  }
  __syncthreads();
  release_dependents();
  wl = start;
  for (int u = threadIdx.x; u < units; u += kBlock, wl.next()) {
    const size_t off = wl.n * sample_stride + base + 4 * static_cast<size_t>(wl.q);
    const int i = 4 * wl.q;
    int first = 0;                                    // the channel of element i
#pragma unroll
    for (int j = 1; j < G; ++j) first += i >= j * sh.HW;
    const int next = (first + 1) * sh.HW - i;         // so many elements are its own
    const float4 k0 = coef[first], k1 = coef[first + 1 < G ? first + 1 : first];
    Vec4f vx, vg, o;
    vx.u = *reinterpret_cast<const uint4*>(sx + 4 * u);
    vg.u = *reinterpret_cast<const uint4*>(sg + 4 * u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool own = j < next;
      o.f[j] = (own ? k0.x : k1.x) * (vg.f[j] - (own ? k0.y : k1.y) - (vx.f[j] - (own ? k0.w : k1.w)) * (own ? k0.z : k1.z));
    }
    st128(dx + off, o.u);
  }
}

// ------------------------------------------- single pass, channels in registers
// Small channels (one sample of a 40x40 plane, a small batch of 10x10 or 5x5
// planes): 32, 128 or 256 threads hold a channel's operands in registers, so
// there is nothing between the loads and the stores but the reduction - no
// staging, no cluster, for a warp (four channels per CTA) not even a barrier.
// Such calls are latency, not bandwidth: what they cost is the length of this
// chain.  3x1024x10x10: 5.3 -> 2.3 us, fused with ReLU 8.3 -> 3.8 us.
// NV units (float4, or float when !VEC) per thread and operand.  MASK 3: the
// incoming gradient is the join dy + dy_b, masked by the ReLU's input and also
// written to `joined`.
template <int MASK, int G, int NV, bool VEC>
__global__ void __launch_bounds__(G == 32 ? 128 : G)
bn_bwd_small_kernel(const float* __restrict__ x, const float* __restrict__ dy, const float* __restrict__ relu_in,
                    const float* __restrict__ scale, const float* __restrict__ mean, const float* __restrict__ invstd,
                    float* __restrict__ dx, float* __restrict__ dscale, float* __restrict__ dbias, BnShape sh,
                    const float* __restrict__ dy_b, float* __restrict__ joined) {
  constexpr int kW = VEC ? 4 : 1;
  __shared__ float sm[2 * G / 32];
  const int c = G == 32 ? blockIdx.x * 4 + (threadIdx.x >> 5) : blockIdx.x;
  const int t = G == 32 ? threadIdx.x & 31 : threadIdx.x;
  const int hwu = sh.HW / kW, total = sh.N * hwu;
  const size_t plane_stride = static_cast<size_t>(sh.C) * sh.HW, chan_off = static_cast<size_t>(c) * sh.HW;
  float vx[NV][kW], vg[NV][kW];
  size_t off[NV];
  UnitWalk w(t, G, hwu);
#pragma unroll
  for (int k = 0; k < NV; ++k, w.next()) {
    off[k] = w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * kW;
    if (c < sh.C && t + k * G < total) {
      prefetch_l2(x + off[k]);
      if (MASK == 1 || MASK == 3) prefetch_l2(relu_in + off[k]);
      if (MASK == 3) prefetch_l2(dy_b + off[k]);
    }
  }
  if (c < sh.C && t < 3) prefetch_l2((t == 0 ? mean : t == 1 ? invstd : scale) + c);
  dependency_wait();
  release_dependents();
  if (c >= sh.C) return;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    const bool in = t + k * G < total;
    if (VEC) {
      Vec4f a, b, m, e;
      a.u = b.u = m.u = e.u = make_uint4(0, 0, 0, 0);
      unsigned bits = 15u;
      if (in) {
        a.u = ld128(x + off[k]);
        b.u = ld128(dy + off[k]);
        if (MASK == 3) e.u = ld128(dy_b + off[k]);
        if (MASK == 1 || MASK == 3) m.u = ld128(relu_in + off[k]);
        if (MASK == 2) bits = keep4<2>(relu_in, off[k]);
      }
#pragma unroll
      for (int j = 0; j < kW; ++j) {
        vx[k][j] = a.f[j];
        vg[k][j] = b.f[j];
        if (MASK == 3) vg[k][j] = m.f[j] > 0 ? (b.f[j] + e.f[j]) : 0.0f;
        if (MASK == 1) vg[k][j] = m.f[j] > 0 ? vg[k][j] : 0.0f;
        if (MASK == 2) vg[k][j] = (bits >> j) & 1u ? vg[k][j] : 0.0f;
      }
    } else {
      vx[k][0] = vg[k][0] = 0.0f;
      if (in) {
        vx[k][0] = x[off[k]];
        vg[k][0] = dy[off[k]];
        if (MASK == 3) vg[k][0] += dy_b[off[k]];
        if (MASK) vg[k][0] = keep1<MASK == 3 ? 1 : MASK>(relu_in, off[k]) ? vg[k][0] : 0.0f;
      }
    }
  }
  const float mu = mean[c], r = invstd[c], sc = scale[c];
  float a = 0.f, b = 0.f;
#pragma unroll
  for (int k = 0; k < NV; ++k)
#pragma unroll
    for (int j = 0; j < kW; ++j) {     // outside the channel both are 0 (a test here would split the loads above)
      a += vg[k][j];
      b += vg[k][j] * (vx[k][j] - mu);
    }
  channel_sums<G, true>(a, b, sm);
  const float inv_m = 1.0f / (static_cast<float>(sh.N) * static_cast<float>(sh.HW));
  const float ds = b * r, k_ = sc * r, am = a * inv_m, bm = ds * r * inv_m;
  if (t == 0) {
    dscale[c] = ds;
    dbias[c] = a;
  }
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    if (t + k * G >= total) break;
    if (VEC) {
      Vec4f o;
#pragma unroll
      for (int j = 0; j < kW; ++j) o.f[j] = k_ * (vg[k][j] - am - (vx[k][j] - mu) * bm);
      st128(dx + off[k], o.u);
      if (MASK == 3) {
#pragma unroll
        for (int j = 0; j < kW; ++j) o.f[j] = vg[k][j];
        st128(joined + off[k], o.u);
      }
    } else {
      dx[off[k]] = k_ * (vg[k][0] - am - (vx[k][0] - mu) * bm);
      if (MASK == 3) joined[off[k]] = vg[k][0];
    }
  }
}

template <int MASK, int G, int NV, bool VEC>
int launch_small(const float* x, const float* dy, const float* relu_in, const float* scale, const float* mean,
                 const float* invstd, float* dx, float* dscale, float* dbias, BnShape sh, cudaStream_t s,
                 const float* dy_b = nullptr, float* joined = nullptr) {
  const unsigned grid = static_cast<unsigned>(G == 32 ? (sh.C + 3) / 4 : sh.C);
  return launch_ex(bn_bwd_small_kernel<MASK, G, NV, VEC>, dim3(grid), dim3(G == 32 ? 128 : G), 0, s, 0, true, x, dy,
                   relu_in, scale, mean, invstd, dx, dscale, dbias, sh, dy_b, joined);
}

template <int MASK, int G>
int launch_group(const float* x, const float* dy, const float* relu_in, const float* scale,
                 const float* mean, const float* invstd, float* dx, float* dscale, float* dbias,
                 BnShape sh, cudaStream_t s) {
  auto kernel = bn_bwd_group_kernel<MASK, G>;
  const size_t smem = static_cast<size_t>(G) * sh.N * sh.HW * 8;
  static std::atomic<bool> attr_set[64];
  const int ready = opt_in_once(kernel, attr_set, false);
  if (ready != SGB_OK) return ready;
  return launch_ex(kernel, dim3(sh.C / G), dim3(kBlock), smem, s, 0, true, x, dy, relu_in, scale, mean, invstd,
                   dx, dscale, dbias, sh);
}

// One warp: this CTA's pair of sums goes to the slot parts[rank] of all `cs`
// CTAs of the cluster as asynchronous 8-byte stores that signal the receiver's
// mbarrier: a CTA goes on as soon as its cs pairs are in.  The peers have
// started (cluster barrier): their memory is addressable.
__device__ __forceinline__ void exchange_pairs(int cs, int rank, float p0, float p1, float2* parts,
                                               unsigned long long* pairs_in) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) mbar_arrive_expect(pairs_in, 8u * static_cast<unsigned>(cs));
  if (lane < cs) {
    unsigned remote_slot, remote_bar;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote_slot) : "r"(smem_addr(&parts[rank])), "r"(lane));
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote_bar) : "r"(smem_addr(pairs_in)), "r"(lane));
    const unsigned long long bits = (static_cast<unsigned long long>(__float_as_uint(p1)) << 32) |
                                    static_cast<unsigned long long>(__float_as_uint(p0));
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(remote_slot),
                 "l"(bits), "r"(remote_bar)
                 : "memory");
  }
}
// All threads: the totals over the cluster, in rank order, once every pair has
// landed (bounded wait; a run-out sets the sticky fault word).
__device__ __forceinline__ void pair_totals(int cs, const float2* parts, unsigned long long* pairs_in, float& a,
                                            float& b) {
  bool in = false;
  for (unsigned it = 0; it < (1u << 24) && !in; ++it) in = mbar_try_wait(pairs_in, 0);
  if (!in) atomicOr(&g_cluster_faults, 1u);
  a = b = 0.f;
  for (int r = 0; r < cs; ++r) {
    a += parts[r].x;
    b += parts[r].y;
  }
}

// ---------------------------------- planes that are not a multiple of four floats
// The cluster scheme over the aligned vectors that touch a plane (RaggedUnit);
// with one float per access the loads of a CTA were a quarter as wide.
template <int MASK, int T>
__global__ void __launch_bounds__(T)
bn_bwd_ragged_kernel(const float* __restrict__ x, const float* __restrict__ dy, const float* __restrict__ relu_in,
                     const float* __restrict__ scale, const float* __restrict__ mean, const float* __restrict__ invstd,
                     float* __restrict__ dx, float* __restrict__ dscale, float* __restrict__ dbias, BnShape sh,
                     int per_cta, size_t numel) {
  extern __shared__ __align__(16) float stage[];
  __shared__ unsigned long long pairs_in;
  __shared__ float red[2 * T / 32];
  __shared__ float2 parts[16];
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = static_cast<int>(cluster.num_blocks());
  const int rank = static_cast<int>(cluster.block_rank());
  const int c = blockIdx.x / cs;
  if (threadIdx.x == 0) {
    mbar_init(&pairs_in, 1);
    fence_mbarrier_init();
  }
  cluster.barrier_arrive();
  const int upp = ragged_units(sh.HW), total = sh.N * upp;
  const int u0 = min(rank * per_cta, total), u1 = min(u0 + per_cta, total);
  const int first = u0 + threadIdx.x;
  float* sx = stage;
  float* sg = stage + static_cast<size_t>(per_cta) * 4;
  const size_t plane_stride = static_cast<size_t>(sh.C) * sh.HW, chan_off = static_cast<size_t>(c) * sh.HW;
  if (first_wave(2)) {
    UnitWalk w(first, T, upp);
    for (int u = first; u < u1; u += T, w.next()) {
      const RaggedUnit r(w.n * plane_stride + chan_off, w.q, sh.HW);
      if (r.valid && r.off < numel) {
        prefetch_l2(x + r.off);
        if (MASK == 1) prefetch_l2(relu_in + r.off);
      }
    }
  }
  dependency_wait();
  const float mu = mean[c];
  const int group_units = ((per_cta + T - 1) / T + kCopyGroups - 1) / kCopyGroups;
  {
    UnitWalk w(first, T, upp);
    int u = first;
#pragma unroll
    for (int g = 0; g < kCopyGroups; ++g) {
      for (int k = 0; k < group_units && u < u1; ++k, u += T, w.next()) {
        const RaggedUnit r(w.n * plane_stride + chan_off, w.q, sh.HW);
        const int l = (u - u0) * 4;
        if (r.valid) {
          ragged_copy(sx + l, x, r.off, numel);
          ragged_copy(sg + l, dy, r.off, numel);
        }
      }
      cp_async_commit();
    }
  }
  // ReLU decisions, 4 bits per unit (a share is at most 16 units per thread)
  unsigned long long keep = 0;
  if (MASK) {
    UnitWalk w(first, T, upp);
    int slot = 0;
    for (int u = first; u < u1;) {
      Vec4f vm[4];
      unsigned bits[4];
      int cnt = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        bits[j] = 0;
        vm[j].u = make_uint4(0, 0, 0, 0);
        if (u < u1) {
          const RaggedUnit r(w.n * plane_stride + chan_off, w.q, sh.HW);
          if (r.valid) {
            if (MASK == 1) vm[j] = ragged_load(relu_in, r.off, numel);
            else bits[j] = keep4<2>(relu_in, r.off);
          }
          u += T;
          w.next();
          cnt = j + 1;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j < cnt) {
          if (MASK == 1)
#pragma unroll
            for (int k = 0; k < 4; ++k) bits[j] |= (vm[j].f[k] > 0 ? 1u : 0u) << k;
          keep |= static_cast<unsigned long long>(bits[j] & 15u) << slot;
          slot += 4;
        }
      }
    }
  }
  float s_dy = 0.f, s_dyx = 0.f;
  {
    UnitWalk w(first, T, upp);
    int slot = 0, u = first;
    auto sum_copy_group = [&]() {
      for (int k = 0; k < group_units && u < u1; ++k, u += T, slot += 4, w.next()) {
        const RaggedUnit r(w.n * plane_stride + chan_off, w.q, sh.HW);
        if (!r.valid) continue;
        const int l = (u - u0) * 4;
        Vec4f vx, vg;
        vx.u = *reinterpret_cast<const uint4*>(sx + l);
        vg.u = *reinterpret_cast<const uint4*>(sg + l);
        if (MASK) {
          const unsigned bits = static_cast<unsigned>(keep >> slot);
#pragma unroll
          for (int q = 0; q < 4; ++q) vg.f[q] = (bits >> q) & 1u ? vg.f[q] : 0.0f;
          *reinterpret_cast<uint4*>(sg + l) = vg.u;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (r.valid >> q & 1u) {
            s_dy += vg.f[q];
            s_dyx += vg.f[q] * (vx.f[q] - mu);
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
  channel_sums<T, true>(s_dy, s_dyx, red);
  cluster.barrier_wait();
  if (threadIdx.x < 32) exchange_pairs(cs, rank, s_dy, s_dyx, parts, &pairs_in);
  // no CTA writes to a peer after this and none exits before all pairs addressed to it have landed
  float a, b;
  pair_totals(cs, parts, &pairs_in, a, b);
  const float r_ = invstd[c];
  const float inv_m = 1.0f / (static_cast<float>(sh.N) * static_cast<float>(sh.HW));
  const float ds = b * r_, k_ = scale[c] * r_, am = a * inv_m, bm = ds * r_ * inv_m;
  if (rank == 0 && threadIdx.x == 0) {
    dscale[c] = ds;
    dbias[c] = a;
  }
  release_dependents();
  UnitWalk w(first, T, upp);
  for (int u = first; u < u1; u += T, w.next()) {
    const RaggedUnit r(w.n * plane_stride + chan_off, w.q, sh.HW);
    if (!r.valid) continue;
    const int l = (u - u0) * 4;
    Vec4f vx, vg, o;
    vx.u = *reinterpret_cast<const uint4*>(sx + l);
    vg.u = *reinterpret_cast<const uint4*>(sg + l);
#pragma unroll
    for (int j = 0; j < 4; ++j) o.f[j] = k_ * (vg.f[j] - am - (vx.f[j] - mu) * bm);
    ragged_store(dx, r, o);
  }
}

// Two passes over the same units, for channels that no cluster holds.
template <int MASK>
__global__ void __launch_bounds__(kBlock, 4)
bn_bwd_ragged_reduce_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                            const float* __restrict__ relu_in, const float* __restrict__ mean,
                            float2* __restrict__ partial, BnShape sh, int per_slice, size_t numel) {
  __shared__ float sm[2 * kBlock / 32];
  constexpr int kFlight = MASK == 1 ? 2 : 4;         // units of each operand in flight
  const int c = blockIdx.y, slice = blockIdx.x;
  dependency_wait();
  release_dependents();
  const float mu = mean[c];
  const int upp = ragged_units(sh.HW), total = sh.N * upp;
  const int i0 = slice * per_slice, i1 = min(i0 + per_slice, total);
  const size_t plane_stride = static_cast<size_t>(sh.C) * sh.HW, chan_off = static_cast<size_t>(c) * sh.HW;
  float s_dy = 0.f, s_dyx = 0.f;
  UnitWalk w(i0 + threadIdx.x, kBlock, upp);
  for (int i = i0 + threadIdx.x; i < i1;) {
    Vec4f vx[kFlight], vg[kFlight], vm[kFlight];
    unsigned valid[kFlight], bits[kFlight];
#pragma unroll
    for (int k = 0; k < kFlight; ++k) {
      valid[k] = 0;
      bits[k] = 15u;
      if (i < i1) {
        const RaggedUnit r(w.n * plane_stride + chan_off, w.q, sh.HW);
        valid[k] = r.valid;
        if (r.valid) {
          vx[k] = ragged_load(x, r.off, numel);
          vg[k] = ragged_load(dy, r.off, numel);
          if (MASK == 1) vm[k] = ragged_load(relu_in, r.off, numel);
          if (MASK == 2) bits[k] = keep4<2>(relu_in, r.off);
        }
        i += kBlock;
        w.next();
      }
    }
#pragma unroll
    for (int k = 0; k < kFlight; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (valid[k] >> j & 1u) {
          float g = vg[k].f[j];
          if (MASK == 1) g = vm[k].f[j] > 0 ? g : 0.0f;
          if (MASK == 2) g = (bits[k] >> j) & 1u ? g : 0.0f;
          s_dy += g;
          s_dyx += g * (vx[k].f[j] - mu);
        }
  }
  channel_sums<kBlock, true>(s_dy, s_dyx, sm);
  if (threadIdx.x == 0) partial[static_cast<size_t>(c) * gridDim.x + slice] = make_float2(s_dy, s_dyx);
}

template <int MASK>
__global__ void __launch_bounds__(kBlock, 4)
bn_bwd_ragged_apply_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                           const float* __restrict__ relu_in, const float* __restrict__ scale,
                           const float* __restrict__ mean, const float* __restrict__ invstd,
                           const float2* __restrict__ partial, int slices, float* __restrict__ dx,
                           float* __restrict__ dscale, float* __restrict__ dbias, BnShape sh, size_t numel) {
  __shared__ float coef[4];
  const int c = sh.C - 1 - blockIdx.y;               // descending: what the first pass touched last is still in L2
  const int upp = ragged_units(sh.HW), total = sh.N * upp;
  const size_t plane_stride = static_cast<size_t>(sh.C) * sh.HW, chan_off = static_cast<size_t>(c) * sh.HW;
  const int unit0 = blockIdx.x * (kBlock * kApplyUnits) + threadIdx.x;
  Vec4f vx[kApplyUnits], vg[kApplyUnits];
  UnitWalk w(min(unit0, total - 1), kBlock, upp);
  UnitWalk w2 = w;
  dependency_wait();
#pragma unroll
  for (int j = 0; j < kApplyUnits; ++j) {
    vx[j].u = vg[j].u = make_uint4(0, 0, 0, 0);
    if (unit0 + j * kBlock < total) {
      const RaggedUnit r(w.n * plane_stride + chan_off, w.q, sh.HW);
      if (r.valid) {
        vx[j] = ragged_load(x, r.off, numel);
        vg[j] = ragged_load(dy, r.off, numel);
        unsigned bits = 15u;
        Vec4f vm;
        if (MASK == 1) vm = ragged_load(relu_in, r.off, numel);
        if (MASK == 2) bits = keep4<2>(relu_in, r.off);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (MASK == 1) vg[j].f[k] = vm.f[k] > 0 ? vg[j].f[k] : 0.0f;
          if (MASK == 2) vg[j].f[k] = (bits >> k) & 1u ? vg[j].f[k] : 0.0f;
        }
      }
      w.next();
    }
  }
  if (threadIdx.x < 32) {
    float a = 0.f, b = 0.f;
    for (int k = threadIdx.x; k < slices; k += 32) {
      const float2 p = partial[static_cast<size_t>(c) * slices + k];
      a += p.x;
      b += p.y;
    }
    a = warp_sum(a);
    b = warp_sum(b);
    if (threadIdx.x == 0) {
      const float r = invstd[c];
      const float inv_m = 1.0f / (static_cast<float>(sh.N) * static_cast<float>(sh.HW));
      const float ds = b * r;
      coef[0] = scale[c] * r;
      coef[1] = a * inv_m;
      coef[2] = ds * r * inv_m;
      coef[3] = mean[c];
      if (blockIdx.x == 0) {
        dscale[c] = ds;
        dbias[c] = a;
      }
    }
  }
  __syncthreads();
  release_dependents();
  const float k_ = coef[0], am = coef[1], bm = coef[2], mu = coef[3];
#pragma unroll
  for (int j = 0; j < kApplyUnits; ++j) {
    if (unit0 + j * kBlock >= total) break;
    const RaggedUnit r(w2.n * plane_stride + chan_off, w2.q, sh.HW);
    w2.next();
    if (!r.valid) continue;
    Vec4f o;
#pragma unroll
    for (int i = 0; i < 4; ++i) o.f[i] = k_ * (vg[j].f[i] - am - (vx[j].f[i] - mu) * bm);
    ragged_store(dx, r, o);
  }
}

template <int MASK, int T>
int launch_ragged_t(const float* x, const float* dy, const float* relu_in, const float* scale, const float* mean,
                    const float* invstd, float* dx, float* dscale, float* dbias, BnShape sh, int cs, int per_cta,
                    cudaStream_t s) {
  auto kernel = bn_bwd_ragged_kernel<MASK, T>;
  static std::atomic<bool> attr_set[64];
  const int ready = opt_in_once(kernel, attr_set, true);
  if (ready != SGB_OK) return ready;
  return launch_ex(kernel, dim3(static_cast<unsigned>(sh.C) * cs), dim3(T), static_cast<size_t>(per_cta) * 32, s, cs,
                   true, x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias, sh, per_cta,
                   static_cast<size_t>(sh.N) * sh.C * sh.HW);
}
// One pass with a cluster where the channel fits one, else two passes.
template <int MASK>
int launch_ragged(const float* x, const float* dy, const float* relu_in, const float* scale, const float* mean,
                  const float* invstd, float* dx, float* dscale, float* dbias, BnShape sh, void* ws, size_t ws_bytes,
                  cudaStream_t s) {
  const int total = sh.N * ragged_units(sh.HW);
  int per_cta = 0;
  const int cs = cluster_plan(total, 32, 8192, &per_cta, sh.C);
  if (cs > 0 && static_cast<long long>(sh.C) * cs <= 0x7fffffffLL)
    return per_cta > 2048 ? launch_ragged_t<MASK, 512>(x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias, sh, cs,
                                                       per_cta, s)
                          : launch_ragged_t<MASK, 256>(x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias, sh, cs,
                                                       per_cta, s);
  const size_t numel = static_cast<size_t>(sh.N) * sh.C * sh.HW;
  const int slices = bn_slices_for(static_cast<long long>(sh.N) * sh.HW, sh.C, sm_count());
  if (!ws || ws_bytes < static_cast<size_t>(slices) * sh.C * sizeof(float2) || !aligned16(ws)) return SGB_ERR_WORKSPACE;
  float2* partial = static_cast<float2*>(ws);
  const int st = launch_ex(bn_bwd_ragged_reduce_kernel<MASK>, dim3(slices, sh.C), dim3(kBlock), 0, s, 0, true, x, dy,
                           relu_in, mean, partial, sh, static_cast<int>(ceil_div(total, slices)), numel);
  if (st != SGB_OK) return st;
  return launch_ex(bn_bwd_ragged_apply_kernel<MASK>,
                   dim3(static_cast<unsigned>(ceil_div(total, kBlock * kApplyUnits)), sh.C), dim3(kBlock), 0, s, 0, true,
                   x, dy, relu_in, scale, mean, invstd, static_cast<const float2*>(partial), slices, dx, dscale, dbias,
                   sh, numel);
}

// ------------------------ single pass, gradient in registers, x in shared memory
// For shares of which shared memory alone holds only two CTAs' worth per SM:
// the first kRegUnits units per thread of the gradient stay in registers, so
// THREE CTAs of 256 threads fit an SM and half as many bytes again are staged.
// (A CTA spends 3.3 us taking its share in and 4.2 us on reduction, exchange
// and dx; with two CTAs the SM's input idles part of the time.)  32x256x56x56,
// cluster form / this one: 67.0 / 56.7 us, 0.83 of the copy bandwidth.
// All loads have to be issued at once: a second, dependent batch waits behind
// everything that is queued already (gradient after x: 4 % slower).  A ReLU's input
// has no registers left to go to, so it passes through the place of x and leaves
// four bits per unit behind; x follows it unit by unit.  With the ReLU's input:
// 88.3 / 75.0 us (0.84); in batches of four registers it was 40 % slower.
// The sums are formed exactly as by bn_bwd_cluster_kernel with 512 threads
// (thread t stands in for its threads t and t + 256), so that a fused call and
// its unfused parts agree bit for bit whichever kernels they take.
constexpr int kRegUnits = 8;
constexpr int kHybridT = 256;

template <bool RELU>
__global__ void __launch_bounds__(kHybridT, 3)
bn_bwd_hybrid_kernel(const float* __restrict__ x, const float* __restrict__ dy, const float* __restrict__ relu_in,
                     const float* __restrict__ scale, const float* __restrict__ mean, const float* __restrict__ invstd, float* __restrict__ dx,
                     float* __restrict__ dscale, float* __restrict__ dbias, BnShape sh, int per_cta) {
  constexpr int T = kHybridT, R = kRegUnits;
  extern __shared__ __align__(16) float stage[];
  __shared__ unsigned long long pairs_in;
  __shared__ float red[2][2 * T / 32];
  __shared__ float2 parts[16];
  cg::cluster_group cluster = cg::this_cluster();
  const int cs = static_cast<int>(cluster.num_blocks());
  const int rank = static_cast<int>(cluster.block_rank());
  const int c = blockIdx.x / cs;
  if (threadIdx.x == 0) {
    mbar_init(&pairs_in, 1);
    fence_mbarrier_init();
  }
  cluster.barrier_arrive();
  const int hwu = sh.HW >> 2, total = sh.N * hwu;
  const int u0 = min(rank * per_cta, total), u1 = min(u0 + per_cta, total);
  const int first = u0 + threadIdx.x;
  float* const sx = stage + static_cast<size_t>(threadIdx.x) * 4;                             // unit k at k * T * 4
  float* const sg = stage + static_cast<size_t>(per_cta) * 4 + static_cast<size_t>(threadIdx.x) * 4;   // k >= R, at (k - R) * T * 4
  const size_t plane_stride = static_cast<size_t>(sh.C) * sh.HW, chan_off = static_cast<size_t>(c) * sh.HW;
  if (first_wave(1)) prefetch_share(x, RELU ? relu_in : nullptr, first, u1, T, hwu, plane_stride, chan_off);
  dependency_wait();
  const float mu = mean[c];
  Vec4f g[R];
  unsigned long long keep = 0;       // RELU: 4 bits per unit
  if (RELU) {
    // The ReLU's input passes through the place of x, also by asynchronous copies:
    // loads to registers would share the 28 KB that the staging leaves to L1.
    UnitWalk w(first, T, hwu);
    int k = 0;
    for (int u = first; u < u1; u += T, w.next(), ++k)
      cp_async16(sx + k * (T * 4), relu_in + w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4);
    cp_async_commit();
  }
  {
    UnitWalk w(first, T, hwu);
#pragma unroll
    for (int k = 0; k < R; ++k, w.next()) {
      g[k].u = make_uint4(0, 0, 0, 0);
      if (first + k * T < u1) {
        const size_t off = w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4;
        g[k].u = ld128(dy + off);
        if (!RELU) cp_async16(sx + k * (T * 4), x + off);
      }
      if (!RELU && k == R / 2 - 1) cp_async_commit();
    }
    if (!RELU) cp_async_commit();
    int k = R;
    for (int u = first + R * T; u < u1; u += T, w.next(), ++k) {
      const size_t off = w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4;
      if (!RELU) cp_async16(sx + k * (T * 4), x + off);
      cp_async16(sg + (k - R) * (T * 4), dy + off);
    }
    cp_async_commit();
  }
  if (RELU) {
    cp_async_wait_pending<1>();
    UnitWalk w(first, T, hwu);
#pragma unroll
    for (int k = 0; k < 16; ++k, w.next()) {
      if (first + k * T < u1) {
        Vec4f m;
        m.u = *reinterpret_cast<const uint4*>(sx + k * (T * 4));
        unsigned bits = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) bits |= (m.f[q] > 0 ? 1u : 0u) << q;
        keep |= static_cast<unsigned long long>(bits) << (4 * k);
        cp_async16(sx + k * (T * 4), x + w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4);
      }
      if (k == R / 2 - 1 || k == R - 1) cp_async_commit();
    }
    cp_async_commit();
#pragma unroll
    for (int k = 0; k < R; ++k)
#pragma unroll
      for (int q = 0; q < 4; ++q) g[k].f[q] = (keep >> (4 * k + q)) & 1u ? g[k].f[q] : 0.0f;
  }
  // sums, in the order of the units; [0]: even units (thread t), [1]: odd ones (thread t + 256)
  float s_dy[2] = {0.f, 0.f}, s_dyx[2] = {0.f, 0.f};
  auto add = [&](int half, const Vec4f& vx, const Vec4f& vg) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      s_dy[half] += vg.f[q];
      s_dyx[half] += vg.f[q] * (vx.f[q] - mu);
    }
  };
  cp_async_wait_pending<2>();
#pragma unroll
  for (int k = 0; k < R; ++k) {
    if (k == R / 2) cp_async_wait_pending<1>();
    if (first + k * T < u1) {
      Vec4f vx;
      vx.u = *reinterpret_cast<const uint4*>(sx + k * (T * 4));
      add(k & 1, vx, g[k]);
    }
  }
  cp_async_wait_pending<0>();
#pragma unroll
  for (int k = R; k < 16; ++k) {
    if (first + k * T >= u1) break;
    Vec4f vx, vg;
    vx.u = *reinterpret_cast<const uint4*>(sx + k * (T * 4));
    vg.u = *reinterpret_cast<const uint4*>(sg + (k - R) * (T * 4));
    if (RELU) {
#pragma unroll
      for (int q = 0; q < 4; ++q) vg.f[q] = (keep >> (4 * k + q)) & 1u ? vg.f[q] : 0.0f;
      *reinterpret_cast<uint4*>(sg + (k - R) * (T * 4)) = vg.u;
    }
    add(k & 1, vx, vg);
  }
  {
    constexpr int kWarps = 2 * T / 32;                 // of the 512 threads
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const float p0 = warp_sum(s_dy[half]), p1 = warp_sum(s_dyx[half]);
      if (lane == 0) {
        red[0][half * (T / 32) + wid] = p0;
        red[1][half * (T / 32) + wid] = p1;
      }
    }
    __syncthreads();
    cluster.barrier_wait();
    if (wid == 0) {
      const float p0 = warp_sum(lane < kWarps ? red[0][lane] : 0.0f);
      const float p1 = warp_sum(lane < kWarps ? red[1][lane] : 0.0f);
      exchange_pairs(cs, rank, p0, p1, parts, &pairs_in);
    }
  }
  const float r_ = invstd[c], sc = scale[c];
  float a, b;
  pair_totals(cs, parts, &pairs_in, a, b);
  const float inv_m = 1.0f / (static_cast<float>(sh.N) * static_cast<float>(sh.HW));
  const float ds = b * r_, k_ = sc * r_, am = a * inv_m, bm = ds * r_ * inv_m;
  if (rank == 0 && threadIdx.x == 0) {
    dscale[c] = ds;
    dbias[c] = a;
  }
  release_dependents();
  auto emit = [&](size_t off, const Vec4f& vx, const Vec4f& vg) {
    Vec4f o;
#pragma unroll
    for (int j = 0; j < 4; ++j) o.f[j] = k_ * (vg.f[j] - am - (vx.f[j] - mu) * bm);
    st128(dx + off, o.u);
  };
  UnitWalk w(first, T, hwu);
#pragma unroll
  for (int k = 0; k < R; ++k, w.next()) {
    if (first + k * T < u1) {
      Vec4f vx;
      vx.u = *reinterpret_cast<const uint4*>(sx + k * (T * 4));
      emit(w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4, vx, g[k]);
    }
  }
  int k = R;
  for (int u = first + R * T; u < u1; u += T, w.next(), ++k) {
    Vec4f vx, vg;
    vx.u = *reinterpret_cast<const uint4*>(sx + k * (T * 4));
    vg.u = *reinterpret_cast<const uint4*>(sg + (k - R) * (T * 4));
    emit(w.n * plane_stride + chan_off + static_cast<size_t>(w.q) * 4, vx, vg);
  }
}

inline size_t hybrid_smem(long long units) {
  const long long rest = units - kRegUnits * kHybridT;
  return (static_cast<size_t>(units) + (rest > 0 ? rest : 0)) * 16;
}
// A share that the cluster kernel would give 512 threads, and that fits three
// times into an SM this way.
inline bool hybrid_share(int units) {
  return units > 2048 && units <= 16 * kHybridT && hybrid_smem(units) <= 74 * 1024;
}
template <bool RELU>
int launch_hybrid(const float* x, const float* dy, const float* relu_in, const float* scale, const float* mean,
                  const float* invstd, float* dx, float* dscale, float* dbias, BnShape sh, int cs, int per_cta,
                  cudaStream_t s) {
  auto kernel = bn_bwd_hybrid_kernel<RELU>;
  static std::atomic<bool> attr_set[64];
  const int ready = opt_in_once(kernel, attr_set, true);
  if (ready != SGB_OK) return ready;
  return launch_ex(kernel, dim3(static_cast<unsigned>(sh.C) * cs), dim3(kHybridT), hybrid_smem(per_cta), s, cs, true, x,
                   dy, relu_in, scale, mean, invstd, dx, dscale, dbias, sh, per_cta);
}

// Whether a grid lets the next kernel's CTAs in, to prefetch, as soon as all of
// its own have started, and not only when it has nothing left to do but store:
// if it takes at most half of the slots that the SMs have for it by shared memory
// and threads.  With more, the waiting CTAs take the places of kernels behind
// them.  A ResNet-50 step in us, never / this rule / one full wave / always:
//   batch 4   398.2  397.9  415.0  415.0      batch 32  1695.9  1692.1  1702.8  1725.6
//   batch 8   598.2  587.4  592.3  596.6      batch 33  1905.1  1897.7  1899.8  1940.7
//   batch 16  974.9  969.4  974.3  983.0      batch 40  2240.5  2241.6  2231.8  2270.5
//   batch 24 1331.4 1326.9 1318.6 1339.3      batch 64  3443.3  3443.6  3462.3  3502.0
// and on images of 160 at batch 16: 613.7  602.9  609.1  613.6.
inline bool leaves_room(long long ctas, size_t smem, int threads) {
  const long long by_smem = 227 * 1024 / (static_cast<long long>(smem) + 2048), by_threads = 2048 / threads;
  return 2 * ctas <= (by_smem < by_threads ? by_smem : by_threads) * sm_count();
}

template <bool VEC, int MASK, int T, bool ADD = false>
int launch_cluster_t(const float* x, const float* dy, const float* relu_in, const float* scale,
                     const float* mean, const float* invstd, float* dx, float* dscale,
                     float* dbias, BnShape sh, int cs, int per_cta, cudaStream_t s,
                     const float* dy_b = nullptr, float* joined = nullptr) {
  auto kernel = bn_bwd_cluster_kernel<VEC, MASK, T, ADD>;
  const size_t smem = static_cast<size_t>(per_cta) * (VEC ? 16 : 4) * 2;
  static std::atomic<bool> attr_set[64];
  const int ready = opt_in_once(kernel, attr_set, true);
  if (ready != SGB_OK) return ready;
  return launch_ex(kernel, dim3(static_cast<unsigned>(sh.C) * cs), dim3(T), smem, s, cs, true, x, dy, relu_in,
                   scale, mean, invstd, dx, dscale, dbias, sh, per_cta,
                   leaves_room(static_cast<long long>(sh.C) * cs, smem, T), dy_b, joined);
}

template <bool VEC, int MASK>
int launch_cluster(const float* x, const float* dy, const float* relu_in, const float* scale,
                   const float* mean, const float* invstd, float* dx, float* dscale,
                   float* dbias, BnShape sh, int cs, int per_cta, cudaStream_t s) {
  // at most 16 units per thread (the fused mask keeps 4 bits per unit in 64 bits)
  if (per_cta > 2048)
    return launch_cluster_t<VEC, MASK, 512>(x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias,
                                            sh, cs, per_cta, s);
  return launch_cluster_t<VEC, MASK, 256>(x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias, sh,
                                          cs, per_cta, s);
}

// Per-activation mode (N x D, one statistic per feature): a thread owns one
// feature, so warp accesses are coalesced along D; it walks the N rows twice.
__global__ void __launch_bounds__(128)
bn_bwd_peract_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                     const float* __restrict__ scale, const float* __restrict__ mean,
                     const float* __restrict__ invstd, float* __restrict__ dx,
                     float* __restrict__ dscale, float* __restrict__ dbias, int N, int D) {
  const int d = blockIdx.x * 128 + threadIdx.x;
  if (d >= D) return;
  const float mu = mean[d], r = invstd[d];
  float s_dy = 0.f, s_dyx = 0.f;
  for (int n = 0; n < N; ++n) {
    const float g = dy[static_cast<size_t>(n) * D + d];
    s_dy += g;
    s_dyx += g * (x[static_cast<size_t>(n) * D + d] - mu);
  }
  const float ds = s_dyx * r, inv_m = 1.0f / static_cast<float>(N);
  dscale[d] = ds;
  dbias[d] = s_dy;
  const float k = scale[d] * r, a = s_dy * inv_m, b = ds * r * inv_m;
  for (int n = 0; n < N; ++n) {
    const size_t off = static_cast<size_t>(n) * D + d;
    dx[off] = k * (dy[off] - a - (x[off] - mu) * b);
  }
}

// join + ReLU backward + batch-norm backward.  Uses the single-pass cluster
// kernel when the shape allows it; otherwise the three steps run as separate
// kernels (same values).
int bn_add_relu_backward(const float* x, const float* dy_a, const float* dy_b, const float* relu_in,
                         const float* scale, const float* mean, const float* invstd, float* joined,
                         float* dx, float* dscale, float* dbias, int N, int C, int HW, void* ws,
                         size_t ws_bytes, void* stream);

// The cluster size of the single-pass kernel for a channel, 0 if none holds it
// (what the registers hold, a cluster holds too).
int takes_cluster(long long per_channel, bool vec, int C, int* per_cta) {
  int share = 0;
  const int cs = cluster_plan(vec ? per_channel / 4 : per_channel, vec ? 32 : 8, 8192, &share, C);
  if (per_cta) *per_cta = share;
  return static_cast<long long>(C) * cs <= 0x7fffffffLL ? cs : 0;
}

// Whether a call takes the form that visits its data twice (bn_revisit.cu).  It
// overlaps everything but its first loads and last stores, which a call has to be
// large enough for; the line is the same whatever the mask, so that a fused call
// and its parts agree bit for bit, and lies where a call with a ReLU gains a microsecond or
// more, and one without at best as much and at worst loses 0.4.
// Time of the forms below / of this one, with and without a ReLU:
//   24x40x56x56   (3.0e6 elements)  12.9 / 10.8    9.2 /  9.6
//   16x64x56x56   (3.2e6)           14.2 / 11.1   10.4 /  9.6
//   32x128x28x28  (3.2e6)           14.2 / 11.4   10.0 /  9.9
//   32x512x14x14  (3.2e6)           13.8 / 11.9    9.5 /  9.9
//   8x512x28x28   (3.2e6)           13.9 / 11.7    9.9 /  9.4
//   32x256x20x20  (3.3e6)           14.5 / 12.0   10.0 /  9.8
//   9x30x112x112  (3.4e6)           21.6 / 12.0   16.0 /  9.9
//   6x48x112x112  (3.6e6)           14.1 / 13.0   10.3 / 10.5
//   12x48x80x80   (3.7e6)           13.9 / 13.1   10.5 / 10.3
//   32x1024x14x14 (6.4e6)           24.1 / 20.7   18.3 / 16.8
//   12x200x50x50  (6.0e6)           25.4 / 19.2   17.4 / 15.4
// smaller ones: 10x256x30x30 (2.3e6) 10.8 / 9.5, 7.8 / 8.2; 8x256x32x32 (2.1e6) 10.3 / 8.9,
// 7.5 / 8.3; 16x128x28x28 (1.6e6) 8.3 / 6.9, 6.3 / 6.0; and channels that one CTA's
// registers hold: 4x512x32x32 6.8 / 8.9, 4.9 / 7.5; 24x1024x8x8 5.4 / 7.3, 4.1 / 6.8.
// Planes that are no multiple of four pay for their masked ends twice:
//   24x64x71x71   (7.7e6)           40.0 / 26.4   27.6 / 20.4
//   12x64x79x79   (4.8e6)           29.8 / 18.0   17.0 / 14.8
//   18x256x33x33  (5.0e6)           25.1 / 19.0   16.2 / 15.3
//   16x512x25x25  (5.1e6)           25.7 / 19.6   16.3 / 15.1
//   24x128x39x39  (4.7e6)           24.3 / 17.8   16.4 / 14.2
// smaller ones: 24x64x45x45 (3.1e6) 16.0 / 13.6, 10.4 / 11.1; 16x64x51x51 (2.7e6) 14.6 / 12.5,
// 9.7 / 10.4.
// Two costs grow with the items of a channel: the lead of the first visit over the
// second (what lies between them has to stay in L2), and every CTA's reading of all
// the channel's sums.  Large channels therefore take the forms below, unless the
// whole call is small (elements of a channel, of the call):
//   64x12x224x224   3.2e6, 3.9e7  172.8 / 143.1   117.8 / 103.0
//   80x20x224x224   4.0e6, 8.0e7  340.9 / 328.8   245.2 / 235.5
//   1x8x2048x2048   4.2e6, 3.4e7  152.2 / 155.8   107.9 / 107.2
//   1x4x2828x2828   8.0e6, 3.2e7  173.1 / 182.5   136.7 / 149.2
//   4x1x4096x4096   6.7e7, 6.7e7  781.8 / 1482.6  695.8 / 1435.5
//   128x3x224x224   6.4e6, 1.9e7  115.4 / 106.3    94.6 / 83.9
//   1x1x4096x4096   1.7e7, 1.7e7  201.7 / 151.1   160.3 / 131.3
// Odd planes have smaller items and a better form of two passes:
//   16x32x223x223   8.0e5, 2.5e7  115.8 / 83.7     78.7 / 70.1
//   2x16x723x723    1.0e6, 1.7e7   75.5 / 61.4     51.3 / 54.6
//   32x16x223x223   1.6e6, 2.5e7  118.9 / 104.8    80.1 / 92.2
//   6x8x597x599     2.1e6, 1.7e7   81.7 / 95.3     55.1 / 86.3
//   32x3x397x397    5.0e6, 1.5e7   86.3 / 141.0    58.2 / 128.1
inline bool revisit_pays(int N, int C, int HW, bool aligned, bool groups) {
  const long long channel = static_cast<long long>(N) * HW, elements = channel * C;
  const bool shared = channel > 6144;                  // a channel is more than one CTA's registers hold
  if (HW % 4)
    return aligned && !groups && channel <= 1000000 &&
           ((HW >= 400 && elements >= 4400000 && shared) || (HW >= 2500 && elements >= 6000000));
  return aligned && HW >= 8 && (elements >= 4000000 || (elements >= 3000000 && shared)) &&
         (channel <= 4000000 || elements <= 20000000);
}

// Whether channels that fit a CTA's registers, read one float an access, go through groups of
// G all the same: above 2e6 elements, where the call is bound by bytes and no longer by
// latency, unless a channel nearly fills the threads' 512, 1024 or 2048 slots, or is so small
// that a group's threads find little to do.  Cold inputs, us in registers / in groups, 2.3e6
// elements if not said:
//   elements of a channel   plain                   ReLU's input          its bits
//     49                   13.2 / 36.1             13.9 / 49.9           13.7 / 49.7
//    294 (of 512)          10.9 / 12.1             13.9 / 14.5           14.2 / 14.1
//    441, 1e7              30.0 / 33.4             39.6 / 41.2           43.9 / 40.8
//    567 (of 1024)          9.8 /  9.2             12.2 / 10.9           14.7 / 10.3
//    637                    9.0 /  9.4             11.4 / 11.1           13.8 / 10.6
//    686                    8.7 /  9.3             10.7 / 10.9           14.3 / 10.2
//    735, 3.6e6 and 5e6    12.1 / 12.6, 16.2 / 16.0  15.6 / 15.2, 20.8 / 19.4  19.8 / 14.5, 27.1 / 18.4
//    833, 5e6 and 7.5e6    15.2 / 16.4, 21.6 / 22.3  19.3 / 19.5, 28.2 / 26.8  26.3 / 18.8, 37.1 / 26.1
//   1014, 1.3e7            30.9 / 34.7             40.7 / 41.8           58.7 / 40.7
//   1617 (of 2048)          9.8 /  9.1             12.5 / 12.2           16.0 / 10.3
//   1764, and 3.6e6         9.6 /  9.6, 13.4 / 12.4  11.0 / 13.1, 17.1 / 17.0  16.2 / 10.9, 22.4 / 14.4
//   1960, 3.6e6 and 7.5e6  12.7 / 13.3, 24.0 / 21.5  16.9 / 17.4, 31.9 / 28.6  23.4 / 15.6, 41.8 / 26.3
//   2025, 5e6 and 7.5e6    16.1 / 17.1, 22.8 / 22.2  21.4 / 21.8, 31.2 / 28.9  29.9 / 19.7, 42.2 / 26.5
//   2997 (of 3072)         11.1 / 10.8             17.3 / 15.0           24.5 / 12.8
// and in groups of two, which are half as large:
//    600, 5e6              18.3 / 21.9             22.4 / 28.1           28.0 / 27.3
//    900, 5e6              14.2 / 19.3             18.4 / 24.0           26.3 / 22.6
//   1050                   12.1 /  9.2             14.8 / 11.2           16.6 / 10.6
//   1800, 5e6              17.1 / 16.0             22.6 / 20.1           28.7 / 18.3
//   3000                    8.1 /  8.8             12.0 / 11.8           17.1 / 10.0
// A ReLU's input and its bits take the same side, so that they have the same bits; it is
// the side of the input.
inline bool groups_pay(long long channel, long long elements, int G, bool masked) {
  if (channel <= 512 || (G == 2 && channel <= 1024)) return false;
  if (channel <= 640) return elements > 2000000;
  if (channel <= 768) return elements > 4000000;
  if (channel <= 1024) return masked && channel <= 960 && elements > 6000000;
  if (channel <= 1680) return elements > 2000000;
  if (channel <= 1920) return elements > 3500000;
  if (channel <= 2048) return elements > 6000000;
  return elements > 2000000;
}

template <int MASK>
int bn_backward(const float* x, const float* dy, const float* relu_in, const float* scale,
                const float* mean, const float* invstd, float* dx, float* dscale,
                float* dbias, int N, int C, int HW, void* ws, size_t ws_bytes, void* stream) {
  if (N < 0 || C < 0 || HW < 0) return SGB_ERR_SIZE;
  if (N == 0 || C == 0 || HW == 0) return SGB_OK;
  if (!x || !dy || !scale || !mean || !invstd || !dx || !dscale || !dbias ||
      (MASK && !relu_in))
    return SGB_ERR_NULL;
  const long long per_channel = static_cast<long long>(N) * HW;
  if (per_channel > 0x7fffffffLL || C > 65535) return SGB_ERR_SIZE;
  cudaStream_t s = as_stream(stream);
  if (HW == 1 && !MASK) {
    bn_bwd_peract_kernel<<<static_cast<unsigned>(ceil_div(C, 128)), 128, 0, s>>>(
        x, dy, scale, mean, invstd, dx, dscale, dbias, N, C);
    return launch_status();
  }
  const bool vec = (HW % 4 == 0) && aligned16(x) && aligned16(dy) && aligned16(dx) &&
                   (MASK != 1 || aligned16(relu_in));
  const BnShape sh{N, C, HW};
  const bool bases_aligned = aligned16(x) && aligned16(dy) && aligned16(dx) && (MASK != 1 || aligned16(relu_in));
  // groups of G adjacent channels make 16-byte runs of odd planes (7x7 layers)
  const int G = (HW % 2) ? 4 : 2;
  const bool groups = !vec && HW > 1 && bases_aligned && (HW * G) % 4 == 0 && C % G == 0 &&
                      static_cast<long long>(G) * per_channel * 8 <= kGroupBytes;
  if (revisit_pays(N, C, HW, bases_aligned, groups)) {
    const int st = bn_revisit_backward(MASK, x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias, N, C, HW, ws,
                                       ws_bytes, s);
    if (st != SGB_ERR_WORKSPACE) return st;            // a smaller workspace: the forms below
  }
  // Channels that fit a CTA's registers need no staging.
  const bool grouped = groups && groups_pay(per_channel, per_channel * C, G, MASK != 0);
  if (!grouped) {
    int st = SGB_OK;
    auto go = [&](auto g, auto nv, auto v) {
      st = launch_small<MASK, decltype(g)::value, decltype(nv)::value, decltype(v)::value>(
          x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias, sh, s);
    };
    if (vec ? small_plan<true, 6>(per_channel / 4, [&](auto g, auto nv) { go(g, nv, std::true_type{}); })
            : small_plan<false, 6>(per_channel, [&](auto g, auto nv) { go(g, nv, std::false_type{}); }))
      return st;
  }
  if (!vec && HW > 1 && bases_aligned) {
    if (groups) {
      if (G == 4)
        return launch_group<MASK, 4>(x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias, sh, s);
      return launch_group<MASK, 2>(x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias, sh, s);
    }
    // below eight elements a plane has more edge units than whole ones
    if (HW >= 8 && static_cast<long long>(N) * ragged_units(HW) <= 0x7fffffffLL)
      return launch_ragged<MASK>(x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias, sh, ws, ws_bytes, s);
  }
  {
    int per_cta = 0;
    const int cs = takes_cluster(per_channel, vec, C, &per_cta);
    if (cs > 0) {
      // two CTAs' worth of work per SM at least, or there is nothing for a third to overlap with
      if (vec && MASK != 2 && hybrid_share(per_cta) && static_cast<long long>(C) * cs >= 2LL * sm_count())
        return launch_hybrid<MASK == 1>(x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias, sh, cs, per_cta, s);
      return vec ? launch_cluster<true, MASK>(x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias,
                                              sh, cs, per_cta, s)
                 : launch_cluster<false, MASK>(x, dy, relu_in, scale, mean, invstd, dx, dscale,
                                               dbias, sh, cs, per_cta, s);
    }
  }
  // channels too large for a cluster: one pass over HBM with the streaming
  // kernel where its plan applies, else two passes
  if (vec && ws && aligned16(ws) && ws_bytes >= bn_stream_workspace_bytes(N, C, HW) &&
      (MASK != 2 || aligned16(relu_in))) {
    BnStreamPlan plan;
    if (bn_stream_plan(N, C, HW, MASK, &plan))
      return bn_stream_backward(MASK, x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias, N, C, HW, plan, ws, s);
  }
  const int slices = bn_slices_for(per_channel, C, sm_count());
  if (!ws || ws_bytes < static_cast<size_t>(slices) * C * sizeof(float2) || !aligned16(ws))
    return SGB_ERR_WORKSPACE;
  float2* partial = static_cast<float2*>(ws);
  const int total = static_cast<int>(vec ? per_channel / 4 : per_channel);
  const int per_slice = static_cast<int>(ceil_div(total, slices));
  const dim3 g1(slices, C), g2(static_cast<unsigned>(ceil_div(total, kBlock * kApplyUnits)), C);
  int st;
  if (vec) {
    st = launch_ex(bn_bwd_reduce_kernel<true, MASK>, g1, dim3(kBlock), 0, s, 0, true, x, dy, relu_in, mean, partial,
                   sh, per_slice);
    if (st != SGB_OK) return st;
    st = launch_ex(bn_bwd_apply_kernel<true, MASK>, g2, dim3(kBlock), 0, s, 0, true, x, dy, relu_in, scale, mean,
                   invstd, partial, slices, dx, dscale, dbias, sh);
  } else {
    st = launch_ex(bn_bwd_reduce_kernel<false, MASK>, g1, dim3(kBlock), 0, s, 0, true, x, dy, relu_in, mean,
                   partial, sh, per_slice);
    if (st != SGB_OK) return st;
    st = launch_ex(bn_bwd_apply_kernel<false, MASK>, g2, dim3(kBlock), 0, s, 0, true, x, dy, relu_in, scale, mean,
                   invstd, partial, slices, dx, dscale, dbias, sh);
  }
  return st;
}

int bn_add_relu_backward(const float* x, const float* dy_a, const float* dy_b, const float* relu_in,
                         const float* scale, const float* mean, const float* invstd, float* joined,
                         float* dx, float* dscale, float* dbias, int N, int C, int HW, void* ws,
                         size_t ws_bytes, void* stream) {
  if (N < 0 || C < 0 || HW < 0) return SGB_ERR_SIZE;
  if (N == 0 || C == 0 || HW == 0) return SGB_OK;
  if (!x || !dy_a || !dy_b || !relu_in || !scale || !mean || !invstd || !joined || !dx || !dscale ||
      !dbias)
    return SGB_ERR_NULL;
  const long long per_channel = static_cast<long long>(N) * HW;
  if (per_channel > 0x7fffffffLL || C > 65535) return SGB_ERR_SIZE;
  const bool vec = (HW % 4 == 0) && aligned16(x) && aligned16(dy_a) && aligned16(dy_b) &&
                   aligned16(relu_in) && aligned16(joined) && aligned16(dx);
  if (vec && !revisit_pays(N, C, HW, true, false)) {
    const BnShape sh{N, C, HW};
    cudaStream_t s = as_stream(stream);
    // the same forms as without the join (same sums, bit for bit)
    int st = SGB_OK;
    if (small_plan<true, 6>(per_channel / 4, [&](auto g, auto nv) {
          st = launch_small<3, decltype(g)::value, decltype(nv)::value, true>(
              x, dy_a, relu_in, scale, mean, invstd, dx, dscale, dbias, sh, s, dy_b, joined);
        }))
      return st;
    int per_cta = 0;
    const int cs = takes_cluster(per_channel, true, C, &per_cta);
    if (cs > 0) {
      if (per_cta > 2048)
        return launch_cluster_t<true, true, 512, true>(x, dy_a, relu_in, scale, mean, invstd, dx, dscale,
                                                       dbias, sh, cs, per_cta, s, dy_b, joined);
      return launch_cluster_t<true, true, 256, true>(x, dy_a, relu_in, scale, mean, invstd, dx, dscale,
                                                     dbias, sh, cs, per_cta, s, dy_b, joined);
    }
  }
  // Planes that are no multiple of four, where the call without the join takes
  // the scalar form of the small kernel too (3x2048x5x5: 3.4 us in two calls, 2.4 in one).
  if (HW > 1 && HW % 4 != 0 && per_channel * C <= 2000000LL) {
    int st = SGB_OK;
    if (small_plan<false, 6>(per_channel, [&](auto g, auto nv) {
          st = launch_small<3, decltype(g)::value, decltype(nv)::value, false>(
              x, dy_a, relu_in, scale, mean, invstd, dx, dscale, dbias, BnShape{N, C, HW}, as_stream(stream), dy_b,
              joined);
        }))
      return st;
  }
  int st = sgb_add_relu_backward_f32(dy_a, dy_b, relu_in, joined, static_cast<size_t>(N) * C * HW, stream);
  if (st != SGB_OK) return st;
  return bn_backward<0>(x, joined, nullptr, scale, mean, invstd, dx, dscale, dbias, N, C, HW, ws,
                        ws_bytes, stream);
}

// ------------------------------------------------ variant with built-in scratch
// Partial sums of the two-pass scheme for callers that cannot provide a
// workspace: a fixed array that lives in the library's device image.  Every
// GPU that loads the library holds these 2 MiB until the process exits.
constexpr int kNoAllocMaxChannels = 4096;
static __device__ __align__(256) float2 g_bn_static_scratch[kMaxSlices * kNoAllocMaxChannels];

// In host code `g_bn_static_scratch` is only a handle for the symbol, not an
// address a kernel could use; the device address is looked up once per device
// (with that device current) and cached here.
float2* static_scratch_address(int* status) {
  static std::atomic<float2*> cached[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    *status = note_cuda_error(e);
    return nullptr;
  }
  if (dev < 0 || dev >= 64) {
    *status = SGB_ERR_UNSUPPORTED;
    return nullptr;
  }
  if (!cached[dev].load(std::memory_order_acquire)) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_bn_static_scratch);
    if (e != cudaSuccess || !ptr) {
      *status = note_cuda_error(e != cudaSuccess ? e : cudaErrorInvalidSymbol);
      return nullptr;
    }
    cached[dev].store(static_cast<float2*>(ptr), std::memory_order_release);
  }
  *status = SGB_OK;
  return cached[dev].load(std::memory_order_acquire);
}

int bn_backward_static(const float* x, const float* dy, const float* scale, const float* mean,
                       const float* invstd, float* dx, float* dscale, float* dbias, int N, int C,
                       int HW, void* stream) {
  if (N < 0 || C < 0 || HW < 0) return SGB_ERR_SIZE;
  if (N == 0 || C == 0 || HW == 0) return SGB_OK;
  if (!x || !dy || !scale || !mean || !invstd || !dx || !dscale || !dbias) return SGB_ERR_NULL;
  if (C > kNoAllocMaxChannels) return SGB_ERR_LIMIT;   // the built-in scratch holds 4096 channels
  const long long per_channel = static_cast<long long>(N) * HW;
  if (per_channel > 0x7fffffffLL) return SGB_ERR_SIZE;
  int st = SGB_OK;
  float2* partial = static_scratch_address(&st);
  if (!partial) return st;
  cudaStream_t s = as_stream(stream);
  const int slices = bn_slices_for(per_channel, C, sm_count());   // <= kMaxSlices
  const bool vec = (HW % 4 == 0) && aligned16(x) && aligned16(dy) && aligned16(dx);
  const BnShape sh{N, C, HW};
  const int total = static_cast<int>(vec ? per_channel / 4 : per_channel);
  const int per_slice = static_cast<int>(ceil_div(total, slices));
  const dim3 g1(slices, C), g2(static_cast<unsigned>(ceil_div(total, kBlock * kApplyUnits)), C);
  // pass 1 writes partial[c * slices + k] for every k < slices before pass 2
  // (same stream) reads exactly those entries, so nothing has to be cleared
  if (vec) {
    bn_bwd_reduce_kernel<true, false><<<g1, kBlock, 0, s>>>(x, dy, nullptr, mean, partial, sh, per_slice);
    bn_bwd_apply_kernel<true, false><<<g2, kBlock, 0, s>>>(x, dy, nullptr, scale, mean, invstd, partial,
                                                           slices, dx, dscale, dbias, sh);
  } else {
    bn_bwd_reduce_kernel<false, false><<<g1, kBlock, 0, s>>>(x, dy, nullptr, mean, partial, sh, per_slice);
    bn_bwd_apply_kernel<false, false><<<g2, kBlock, 0, s>>>(x, dy, nullptr, scale, mean, invstd, partial,
                                                            slices, dx, dscale, dbias, sh);
  }
  return launch_status();
}

}  // namespace
}  // namespace sgb

using namespace sgb;

extern "C" {

size_t sgb_bn_backward_workspace_bytes(int N, int C, int HW) {
  if (N <= 0 || C <= 0 || HW <= 0) return 0;
  size_t need = static_cast<size_t>(kMaxSlices) * C * sizeof(float2);
  const size_t backward = revisit_pays(N, C, HW, true, false) ? bn_revisit_workspace_bytes(N, C, HW) : 0;
  const size_t forward = bn_forward_workspace_bytes(N, C, HW);
  if (backward > need) need = backward;
  return forward > need ? forward : need;
}

int sgb_bn_backward_faults(unsigned* flags) {
  if (!flags) return SGB_ERR_NULL;
  unsigned streaming = 0, cluster = 0;
  const int st = bn_stream_faults(&streaming);
  if (st != SGB_OK) return st;
  cudaError_t e = cudaMemcpyFromSymbol(&cluster, g_cluster_faults, sizeof(unsigned));
  if (e != cudaSuccess) return note_cuda_error(e);
  unsigned forward = 0;
  const int fs = bn_forward_faults(&forward);
  if (fs != SGB_OK) return fs;
  unsigned revisit = 0;
  const int rs = revisit_faults(&revisit);
  if (rs != SGB_OK) return rs;
  *flags = streaming | (cluster << 8) | (forward << 16) | (revisit << 24);
  return SGB_OK;
}

int sgb_bn_backward_streams(int N, int C, int HW, int mask) {
  if (N <= 0 || C <= 0 || HW <= 0 || HW % 4 != 0 || mask < 0 || mask > 2) return 0;
  const long long per_channel = static_cast<long long>(N) * HW;
  if (per_channel > 0x7fffffffLL || takes_cluster(per_channel, true, C, nullptr)) return 0;
  BnStreamPlan plan;
  return bn_stream_plan(N, C, HW, mask, &plan) ? 1 : 0;
}

int sgb_bn_backward_draws_table(int N, int C, int HW, int mask, size_t ws_bytes) {
  if (!sgb_bn_backward_streams(N, C, HW, mask)) return 0;
  const size_t need = revisit_pays(N, C, HW, true, false) ? bn_revisit_workspace_bytes(N, C, HW) : 0;
  return need == 0 || ws_bytes < need;
}

int sgb_bn_backward_stream_plan(int N, int C, int HW, int mask, int* plan6) {
  if (!plan6) return SGB_ERR_NULL;
  BnStreamPlan p;
  if (!bn_stream_plan(N, C, HW, mask, &p)) return 0;
  plan6[0] = p.P;
  plan6[1] = p.Lp;
  plan6[2] = p.S;
  plan6[3] = p.parts;
  plan6[4] = p.depth;
  plan6[5] = p.arrays;
  return 1;
}

int sgb_bn_backward_f32(const float* x, const float* dy, const float* scale, const float* mean,
                        const float* invstd, float* dx, float* dscale, float* dbias, int N,
                        int C, int HW, void* ws, size_t ws_bytes, void* stream) {
  return bn_backward<0>(x, dy, nullptr, scale, mean, invstd, dx, dscale, dbias, N, C, HW,
                        ws, ws_bytes, stream);
}

int sgb_bn_add_relu_backward_f32(const float* x, const float* dy_a, const float* dy_b,
                                 const float* relu_in, const float* scale, const float* mean,
                                 const float* invstd, float* joined, float* dx, float* dscale,
                                 float* dbias, int N, int C, int HW, void* ws, size_t ws_bytes,
                                 void* stream) {
  return bn_add_relu_backward(x, dy_a, dy_b, relu_in, scale, mean, invstd, joined, dx, dscale, dbias, N,
                              C, HW, ws, ws_bytes, stream);
}

int sgb_bn_backward_noalloc_f32(const float* x, const float* dy, const float* scale,
                                const float* mean, const float* invstd, float* dx, float* dscale,
                                float* dbias, int N, int C, int HW, void* stream) {
  return bn_backward_static(x, dy, scale, mean, invstd, dx, dscale, dbias, N, C, HW, stream);
}

int sgb_bn_relu_backward_mask_f32(const float* x, const float* dy, const void* relu_mask,
                                  const float* scale, const float* mean, const float* invstd,
                                  float* dx, float* dscale, float* dbias, int N, int C, int HW,
                                  void* ws, size_t ws_bytes, void* stream) {
  return bn_backward<2>(x, dy, static_cast<const float*>(relu_mask), scale, mean, invstd, dx, dscale, dbias, N, C,
                        HW, ws, ws_bytes, stream);
}

int sgb_bn_relu_backward_f32(const float* x, const float* dy, const float* relu_in,
                             const float* scale, const float* mean, const float* invstd,
                             float* dx, float* dscale, float* dbias, int N, int C, int HW,
                             void* ws, size_t ws_bytes, void* stream) {
  return bn_backward<1>(x, dy, relu_in, scale, mean, invstd, dx, dscale, dbias, N, C, HW,
                        ws, ws_bytes, stream);
}

}  // extern "C"
