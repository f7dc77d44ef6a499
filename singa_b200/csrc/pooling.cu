// 2-D pooling (NCHW): max and average (divisor excludes padding), forward and
// backward.  Backward is written as a GATHER: every dx element visits the
// output windows that cover it, in raster order, and adds the gradients it is
// owed.  No atomics, so results are deterministic, and the order of additions
// equals that of a serial window-by-window scatter, which makes the result
// bit-identical to the CPU statement of the reference.
//
// Max backward credits, per window, the FIRST maximum in raster order (strict
// '>' while scanning, padding never wins).
#include <float.h>

#include <type_traits>

#include "common.cuh"

namespace sgb {
namespace {

constexpr int kBlock = 256;

struct PoolShape {
  int N, C, H, W, OH, OW, kh, kw, ph, pw, sh, sw;
};

__device__ __forceinline__ void window(const PoolShape& p, int oh, int ow, int& h0, int& h1,
                                       int& w0, int& w1) {
  h0 = oh * p.sh - p.ph;
  w0 = ow * p.sw - p.pw;
  h1 = min(h0 + p.kh, p.H);
  w1 = min(w0 + p.kw, p.W);
  h0 = max(h0, 0);
  w0 = max(w0, 0);
}

// Range of output rows whose window contains input row h (same for columns).
__device__ __forceinline__ void covering(int h, int pad, int k, int stride, int out, int& lo,
                                         int& hi) {
  const int t = h + pad - k + 1;
  lo = t > 0 ? (t + stride - 1) / stride : 0;
  hi = min((h + pad) / stride, out - 1);
}

template <bool MAX>
__global__ void __launch_bounds__(kBlock)
pool_fwd_kernel(const float* __restrict__ x, float* __restrict__ y, PoolShape p, size_t total) {
  dependency_wait();
  release_dependents();
  const size_t i = blockIdx.x * static_cast<size_t>(kBlock) + threadIdx.x;
  if (i >= total) return;
  const int ow = static_cast<int>(i % p.OW);
  const int oh = static_cast<int>((i / p.OW) % p.OH);
  const size_t plane = i / (static_cast<size_t>(p.OW) * p.OH);
  const float* xp = x + plane * p.H * p.W;
  int h0, h1, w0, w1;
  window(p, oh, ow, h0, h1, w0, w1);
  if (MAX) {
    float best = -FLT_MAX;
    for (int h = h0; h < h1; ++h)
      for (int w = w0; w < w1; ++w) {
        const float v = xp[h * p.W + w];
        // a NaN in the window is the window's result (the reference's pooling
        // descriptor asks for CUDNN_PROPAGATE_NAN, src/model/operation/pooling.h:90):
        // the first NaN sticks, since nothing compares greater than it
        if (v > best || v != v) best = v;
      }
    y[i] = best;
  } else {
    float s = 0.f;
    for (int h = h0; h < h1; ++h)
      for (int w = w0; w < w1; ++w) s += xp[h * p.W + w];
    y[i] = s / static_cast<float>((h1 - h0) * (w1 - w0));
  }
}

// Max backward, one band of dx rows of one (n, c) plane per CTA.
//   phase 0: the x rows touched by the band's covering windows are staged in
//            shared memory with coalesced (128-bit when aligned) loads;
//   phase 1: every covering window finds its winner (first maximum in raster
//            order) in shared memory and parks the flat plane index;
//   phase 2: every dx element of the band gathers, in raster order, the dy of
//            the covering windows whose parked winner it is, and is stored
//            with a coalesced write.
// x is read from HBM once plus a one-window halo per band, dy and dx once.
struct BandPlan {
  int rows;        // dx rows per band
  int bands;       // bands per plane
  int max_xrows;   // x rows staged per band (upper bound)
  int max_orows;   // window rows per band (upper bound)
};

__global__ void __launch_bounds__(kBlock)
maxpool_bwd_band_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                        float* __restrict__ dx, PoolShape p, BandPlan bp) {
  extern __shared__ float smem[];
  float* xs = smem;                                            // max_xrows * W
  int* winner = reinterpret_cast<int*>(smem + bp.max_xrows * p.W);  // max_orows * OW
  dependency_wait();
  release_dependents();
  const size_t plane = blockIdx.x;
  const int h_lo = blockIdx.y * bp.rows, h_hi = min(h_lo + bp.rows, p.H);  // dx rows [h_lo, h_hi)
  int o_lo, o_hi, unused;
  covering(h_lo, p.ph, p.kh, p.sh, p.OH, o_lo, unused);
  covering(h_hi - 1, p.ph, p.kh, p.sh, p.OH, unused, o_hi);    // window rows [o_lo, o_hi]
  const float* xp = x + plane * p.H * p.W;
  const float* gp = dy + plane * p.OH * p.OW;
  float* dp = dx + plane * p.H * p.W;
  if (o_hi >= o_lo) {
    const int xr_lo = max(o_lo * p.sh - p.ph, 0);
    const int xr_hi = min(o_hi * p.sh - p.ph + p.kh, p.H);     // x rows [xr_lo, xr_hi)
    const int nx = (xr_hi - xr_lo) * p.W;
    const float* src = xp + xr_lo * p.W;
    if ((reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
      const int nv = nx >> 2;
      for (int v = threadIdx.x; v < nv; v += kBlock)
        reinterpret_cast<float4*>(xs)[v] = reinterpret_cast<const float4*>(src)[v];
      for (int i = (nv << 2) + threadIdx.x; i < nx; i += kBlock) xs[i] = src[i];
    } else {
      for (int i = threadIdx.x; i < nx; i += kBlock) xs[i] = src[i];
    }
    __syncthreads();
    const int nwin = (o_hi - o_lo + 1) * p.OW;
    for (int o = threadIdx.x; o < nwin; o += kBlock) {
      const int r = o / p.OW, ow = o - r * p.OW, oh = o_lo + r;
      int h0, h1, w0, w1;
      window(p, oh, ow, h0, h1, w0, w1);
      float best = -FLT_MAX;
      int bi = -1;
      for (int h = h0; h < h1; ++h) {
        const float* row = xs + (h - xr_lo) * p.W;
        for (int w = w0; w < w1; ++w) {
          const float v = row[w];
          if (v > best || (v != v && best == best)) {   // first maximum; a NaN wins and then sticks, as in cuDNN
            best = v;
            bi = h * p.W + w;
          }
        }
      }
      winner[o] = bi;
    }
  }
  __syncthreads();
  const int nin = (h_hi - h_lo) * p.W;
  for (int j = threadIdx.x; j < nin; j += kBlock) {
    const int r = j / p.W, w = j - r * p.W, h = h_lo + r;
    const int i = h * p.W + w;
    int oh_lo, oh_hi, ow_lo, ow_hi;
    covering(h, p.ph, p.kh, p.sh, p.OH, oh_lo, oh_hi);
    covering(w, p.pw, p.kw, p.sw, p.OW, ow_lo, ow_hi);
    float acc = 0.f;
    for (int oh = oh_lo; oh <= oh_hi; ++oh)
      for (int ow = ow_lo; ow <= ow_hi; ++ow)
        if (winner[(oh - o_lo) * p.OW + ow] == i) acc += gp[oh * p.OW + ow];
    dp[i] = acc;
  }
}

// Same scheme with the geometry (square kernel K, stride S, padding P) known
// at compile time: window loops unroll, the divisions by the stride become
// shifts, dy rows are staged in shared memory as well, and every thread
// produces four consecutive dx values of one row (one 128-bit store).  For the
// square windows that have no form of their own further down (3x3 / 2 / 0 and
// 2x2 / 1 / 0); it needs W % 4 == 0.  About 60 instructions per dx element
// instead of ~200.
template <int K, int S, int P>
__global__ void __launch_bounds__(kBlock)
maxpool_bwd_band_fast_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                             float* __restrict__ dx, PoolShape p, BandPlan bp) {
  extern __shared__ float smem[];
  float* xs = smem;
  int* winner = reinterpret_cast<int*>(xs + bp.max_xrows * p.W);
  float* gs = reinterpret_cast<float*>(winner + bp.max_orows * p.OW);
  dependency_wait();
  release_dependents();
  const size_t plane = blockIdx.x;
  const int H = p.H, W = p.W, OH = p.OH, OW = p.OW;
  const int h_lo = blockIdx.y * bp.rows, h_hi = min(h_lo + bp.rows, H);
  const int t_lo = h_lo + P - K + 1;
  const int o_lo = t_lo > 0 ? (t_lo + S - 1) / S : 0;
  const int o_hi = min((h_hi - 1 + P) / S, OH - 1);
  const float* xp = x + plane * H * W;
  const float* gp = dy + plane * OH * OW;
  float* dp = dx + plane * H * W;
  const int xr_lo = max(o_lo * S - P, 0);
  if (o_hi >= o_lo) {
    const int xr_hi = min(o_hi * S - P + K, H);
    const int nv = ((xr_hi - xr_lo) * W) >> 2;                 // W % 4 == 0
    const float4* src = reinterpret_cast<const float4*>(xp + xr_lo * W);
    for (int v = threadIdx.x; v < nv; v += kBlock) reinterpret_cast<float4*>(xs)[v] = src[v];
    const int nwin = (o_hi - o_lo + 1) * OW;
    const float* gsrc = gp + o_lo * OW;
    for (int o = threadIdx.x; o < nwin; o += kBlock) gs[o] = gsrc[o];
    __syncthreads();
    for (int o = threadIdx.x; o < nwin; o += kBlock) {
      const int r = o / OW, ow = o - r * OW, oh = o_lo + r;
      float best = -FLT_MAX;
      int bi = -1;
#pragma unroll
      for (int i = 0; i < K; ++i) {
        const int h = oh * S - P + i;
        if (h < 0 || h >= H) continue;
        const float* row = xs + (h - xr_lo) * W;
#pragma unroll
        for (int j = 0; j < K; ++j) {
          const int w = ow * S - P + j;
          if (w < 0 || w >= W) continue;
          const float v = row[w];
          if (v > best || (v != v && best == best)) {   // first maximum; a NaN wins and then sticks, as in cuDNN
            best = v;
            bi = h * W + w;
          }
        }
      }
      winner[o] = bi;
    }
  }
  __syncthreads();
  constexpr int kCover = (K + S - 1) / S;                       // windows covering one row/column
  const int w4 = W >> 2, nq = (h_hi - h_lo) * w4;
  for (int q = threadIdx.x; q < nq; q += kBlock) {
    const int r = q / w4, c4 = q - r * w4, h = h_lo + r;
    const int th = h + P - K + 1;
    const int oh_lo = th > 0 ? (th + S - 1) / S : 0;
    const int oh_hi = min((h + P) / S, OH - 1);
    float out[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int w = 4 * c4 + e, i = h * W + w;
      const int tw = w + P - K + 1;
      const int ow_lo = tw > 0 ? (tw + S - 1) / S : 0;
      const int ow_hi = min((w + P) / S, OW - 1);
      float acc = 0.f;
#pragma unroll
      for (int a = 0; a < kCover; ++a) {
        const int oh = oh_lo + a;
        if (oh > oh_hi) break;
#pragma unroll
        for (int b = 0; b < kCover; ++b) {
          const int ow = ow_lo + b;
          if (ow > ow_hi) break;
          const int widx = (oh - o_lo) * OW + ow;
          if (winner[widx] == i) acc += gs[widx];
        }
      }
      out[e] = acc;
    }
    *reinterpret_cast<float4*>(dp + h * W + 4 * c4) = make_float4(out[0], out[1], out[2], out[3]);
  }
}

// ------------------------------------------------ arg-max forward partner
// Max-pool forward that also records, per window, WHERE its (first, in raster
// order) maximum sits: one byte, row offset in the high nibble and column
// offset in the low nibble, both relative to the window's unclipped top-left
// corner (oh*sh - ph, ow*sw - pw).  With that record the backward pass needs
// neither x nor y: it reads dy and one byte per window.
__global__ void __launch_bounds__(kBlock)
maxpool_fwd_argmax_kernel(const float* __restrict__ x, float* __restrict__ y,
                          unsigned char* __restrict__ arg, PoolShape p, size_t total) {
  dependency_wait();
  release_dependents();
  const size_t i = blockIdx.x * static_cast<size_t>(kBlock) + threadIdx.x;
  if (i >= total) return;
  const int ow = static_cast<int>(i % p.OW);
  const int oh = static_cast<int>((i / p.OW) % p.OH);
  const size_t plane = i / (static_cast<size_t>(p.OW) * p.OH);
  const float* xp = x + plane * p.H * p.W;
  int h0, h1, w0, w1;
  window(p, oh, ow, h0, h1, w0, w1);
  const int hs = oh * p.sh - p.ph, ws = ow * p.sw - p.pw;
  float best = -FLT_MAX;
  int code = 0xff;                                  // matches no cell (empty or all -FLT_MAX window)
  for (int h = h0; h < h1; ++h)
    for (int w = w0; w < w1; ++w) {
      const float v = xp[h * p.W + w];
      if (v > best || (v != v && best == best)) {   // first maximum, or the first NaN (which then sticks)
        best = v;
        code = ((h - hs) << 4) | (w - ws);
      }
    }
  y[i] = best;
  arg[i] = static_cast<unsigned char>(code);
}

// Backward from the record, any geometry: one dx element per thread gathers,
// in raster order of the windows, the dy of every covering window whose
// record points at it.
__global__ void __launch_bounds__(kBlock)
maxpool_bwd_argmax_kernel(const float* __restrict__ dy, const unsigned char* __restrict__ arg,
                          float* __restrict__ dx, PoolShape p, size_t total) {
  dependency_wait();
  release_dependents();
  const size_t i = blockIdx.x * static_cast<size_t>(kBlock) + threadIdx.x;
  if (i >= total) return;
  const int w = static_cast<int>(i % p.W);
  const int h = static_cast<int>((i / p.W) % p.H);
  const size_t plane = i / (static_cast<size_t>(p.W) * p.H);
  const float* gp = dy + plane * p.OH * p.OW;
  const unsigned char* ap = arg + plane * p.OH * p.OW;
  int oh_lo, oh_hi, ow_lo, ow_hi;
  covering(h, p.ph, p.kh, p.sh, p.OH, oh_lo, oh_hi);
  covering(w, p.pw, p.kw, p.sw, p.OW, ow_lo, ow_hi);
  float acc = 0.f;
  for (int oh = oh_lo; oh <= oh_hi; ++oh)
    for (int ow = ow_lo; ow <= ow_hi; ++ow) {
      const int code = ap[oh * p.OW + ow];
      const int wh = oh * p.sh - p.ph + (code >> 4), ww = ow * p.sw - p.pw + (code & 15);
      if (code != 0xff && wh == h && ww == w) acc += gp[oh * p.OW + ow];
    }
  dx[i] = acc;
}

// ------------------------------------------------ 3x3 / stride 2 / pad 1, all passes
// The ResNet stem's geometry, any plane size.  A lane owns four adjacent input
// columns, which are the two windows 2q and 2q + 1 (columns 4q-1 .. 4q+3); a
// warp walks down the rows of one or more planes.  Everything is in registers:
// the row above is kept from the step before, the column to the left comes
// from the neighbour lane, and the first window of the lane to the right is
// fetched with a shuffle where a gradient needs it.  No shared memory and no
// barrier; the next two rows are in flight while the current ones are worked
// on.  (The form with staged rows spent its time on shared-memory traffic and
// index arithmetic: 67 us forward, 59 us backward at 32x64x112x112, where the
// bytes take 20 and 35 us.)  Planes wider than 128 columns are cut into
// segments of 30 lanes with one halo lane on each side.
enum StripMode { kMaxFwd = 0, kMaxFwdRecord = 1, kMaxBwd = 2, kMaxBwdRecord = 3, kAvgFwd = 4, kAvgBwd = 5 };

struct StripArgs {
  const float* x;          // input planes (kMaxFwd*, kMaxBwd, kAvgFwd)
  const float* dy;         // output gradient (backward modes)
  float* out;              // y or dx
  unsigned char* record;   // written by kMaxFwdRecord, read by kMaxBwdRecord
  int planes, H, W, OH, OW;
  int quads;               // lanes a row needs: ceil(W / 4)
  int abreast;             // planes side by side in a warp
  int segments;            // warps a row needs
  int rows;                // window rows per band
  int bands;
};

constexpr int kNoCell = -1;

// The first maximum of a window in raster order, in two steps: of the three cells of
// each row, which serves every window that holds them, then of the three rows (a row's
// winner counts only if it is strictly greater than the rows above).  NANS: a NaN wins
// and then sticks, as in cuDNN; warps that have seen none (nor an infinity) take the
// plain comparisons.  (us, 32x64x112x112 by 3/2/1, nine comparisons a window -> this:
// forward 24.7 -> 23.9, with the record 32.0 -> 29.6, backward 45.0 -> 42.2.)
template <bool NANS>
__device__ __forceinline__ bool beats(float v, float best) {
  return v > best || (NANS && v != v && best == best);
}
template <bool NANS>
__device__ __forceinline__ void first_of_cells(float c0, float c1, float c2, float& best, int& at) {
  bool p = beats<NANS>(c1, c0);
  best = p ? c1 : c0;
  at = p ? 1 : 0;
  p = beats<NANS>(c2, best);
  best = p ? c2 : best;
  at = p ? 2 : at;
}
// Index 0..8 of the winner; kNoCell (and -FLT_MAX) if no cell exceeds -FLT_MAX.
template <bool NANS>
__device__ __forceinline__ void first_of_rows(const float (&v)[3], const int (&col)[3], float& best, int& at) {
  best = v[0];
  at = col[0];
#pragma unroll
  for (int r = 1; r < 3; ++r) {
    const bool p = beats<NANS>(v[r], best);
    best = p ? v[r] : best;
    at = p ? 3 * r + col[r] : at;
  }
  const bool some = beats<NANS>(best, -FLT_MAX);
  best = some ? best : -FLT_MAX;
  at = some ? at : kNoCell;
}

template <int MODE, bool VEC>
__global__ void __launch_bounds__(kBlock, 4)
pool_k3s2p1_kernel(const StripArgs a) {
  constexpr bool kBackward = MODE == kMaxBwd || MODE == kMaxBwdRecord || MODE == kAvgBwd;
  constexpr bool kNeedsX = MODE != kMaxBwdRecord && MODE != kAvgBwd;
  constexpr bool kMax = MODE <= kMaxBwdRecord;
  constexpr unsigned kAll = 0xffffffffu;
  dependency_wait();
  release_dependents();
  const int lane = threadIdx.x & 31;
  const unsigned task = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5);
  const unsigned rest = task / a.bands;
  const int band = static_cast<int>(task - rest * a.bands);
  const int group = static_cast<int>(rest / a.segments), seg = static_cast<int>(rest - group * a.segments);
  int q, plane;
  bool active, owner;
  if (a.segments > 1) {
    q = seg * 30 - 1 + lane;
    plane = group;
    active = q >= 0 && q < a.quads && plane < a.planes;
    owner = active && lane >= 1 && lane <= 30;
  } else {
    const int pl = lane / a.quads;
    q = lane - pl * a.quads;
    plane = group * a.abreast + pl;
    active = pl < a.abreast && plane < a.planes;
    owner = active;
  }
  if (!active) plane = 0;
  const int H = a.H, W = a.W, OH = a.OH, OW = a.OW, c = 4 * q;
  const float* xp = a.x + static_cast<size_t>(plane) * H * W + c;
  const size_t window0 = static_cast<size_t>(plane) * OH * OW + 2 * q;   // window (row 0, column 2q)
  float* dxp = a.out + static_cast<size_t>(plane) * H * W + c;
  const bool has_left = q > 0, has_right = q + 1 < a.quads;
  const bool w1_exists = 2 * q + 1 < OW;
  const float kPad = kMax ? -FLT_MAX : 0.0f;

  const int m0 = band * a.rows, m1 = min(m0 + a.rows, OH);
  // backward: the odd row above window row m1 also takes from it
  const int last = kBackward ? min(m1, OH - 1) : m1 - 1;
  auto load_row = [&](int h, float (&v)[4]) {
    const bool in = active && h >= 0 && h < H;
    if (VEC) {
      float4 t = make_float4(kPad, kPad, kPad, kPad);
      if (in) t = *reinterpret_cast<const float4*>(xp + static_cast<size_t>(h) * W);
      v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = in && c + j < W ? xp[static_cast<size_t>(h) * W + j] : kPad;
    }
  };
  auto load_windows = [&](int m, float (&g)[2], unsigned (&code)[2]) {
    const size_t i = window0 + static_cast<size_t>(m) * OW;
    if (VEC) {                                       // W % 4 == 0: both windows exist, i is even
      if (kBackward) {
        const float2 t = active ? *reinterpret_cast<const float2*>(a.dy + i) : make_float2(0.f, 0.f);
        g[0] = t.x;
        g[1] = t.y;
      }
      if (MODE == kMaxBwdRecord) {
        const unsigned t = active ? *reinterpret_cast<const unsigned short*>(a.record + i) : 0xffffu;
        code[0] = t & 0xffu;
        code[1] = t >> 8;
      }
      return;
    }
    if (kBackward) {
      g[0] = active ? a.dy[i] : 0.0f;
      g[1] = active && w1_exists ? a.dy[i + 1] : 0.0f;
    }
    if (MODE == kMaxBwdRecord) {
      code[0] = active ? a.record[i] : 0xffu;
      code[1] = active && w1_exists ? a.record[i + 1] : 0xffu;
    }
  };
  // What window row m needs, into L2: the registers hold one row pair ahead, which is
  // 29 KB in flight per SM where the rate takes 47.  32x64x112x112: forward 27.5 ->
  // 25.7 us, backward 48.1 -> 46.1, with the record 31.9 -> 28.7, average backward
  // 39.8 -> 32.7; two rows further ahead it is 26.7 and more.  The backward pass that
  // finds its winners again has no registers to spare: not on odd rows (111x111 49.8 ->
  // 50.9) and small problems (16x512x14x14 7.7 -> 8.2; 64 channels of 112x112, 6.4e6
  // elements 14.8 -> 15.1, 9.6e6 20.6 -> 20.6, 1.28e7 26.6 -> 26.2, 1.45e7 28.1 -> 28.7,
  // 1.6e7 32.1 -> 31.2, 1.9e7 37.4 -> 36.0; 56x56 1.28e7 26.9 -> 26.3, 1.6e7 32.5 -> 31.3;
  // 160x160 1.31e7 32.4 -> 34.2; 28x28 1.28e7 27.7 -> 27.8).
  const bool far = MODE != kMaxBwd || (VEC && static_cast<long long>(a.planes) * H * W >= 16000000);
  auto ahead = [&](int m) {
    if (!far || !active || m > last) return;
    if (kNeedsX) {
      const float* p = xp + static_cast<size_t>(2 * m) * W;
      if (2 * m < H) prefetch_l2(p);
      if (2 * m + 1 < H) prefetch_l2(p + W);
    }
    if (kBackward) prefetch_l2(a.dy + window0 + static_cast<size_t>(m) * OW);
  };
  auto store_row = [&](int h, const float (&v)[4]) {
    if (!owner || h >= H) return;
    float* p = dxp + static_cast<size_t>(h) * W;
    if (VEC) {
      *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c + j < W) p[j] = v[j];
    }
  };

  float above[4], above_left = kPad, r0[4], r1[4], n0[4], n1[4], g[2] = {0.f, 0.f}, ng[2] = {0.f, 0.f};
  float top[2] = {kPad, kPad};     // maxima: what the two windows hold in the row above
  int top_at[2] = {0, 0};
  unsigned code[2] = {0, 0}, ncode[2] = {0, 0};
  bool odd_above = false;          // something in the row above that only the NaN-aware comparison may decide
  auto unordered = [](const float (&v)[4]) {
    const float s = (v[0] + v[1]) + (v[2] + v[3]);   // NaN, or inf - inf: rare enough
    return s != s;
  };
  if (kNeedsX) {
    load_row(2 * m0 - 1, above);
    load_row(2 * m0, n0);
    load_row(2 * m0 + 1, n1);
    above_left = __shfl_up_sync(kAll, above[3], 1);
    if (!has_left) above_left = kPad;
    if (kMax) {
      odd_above = __any_sync(kAll, unordered(above));
      first_of_cells<true>(above_left, above[0], above[1], top[0], top_at[0]);
      first_of_cells<true>(above[1], above[2], above[3], top[1], top_at[1]);
    }
  }
  load_windows(m0, ng, ncode);
  ahead(m0 + 1);
  float pend[4] = {0.f, 0.f, 0.f, 0.f};   // gradient of row 2m - 1 so far
  for (int m = m0; m <= last; ++m) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      r0[j] = n0[j];
      r1[j] = n1[j];
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      g[j] = ng[j];
      code[j] = ncode[j];
    }
    if (m < last) {
      if (kNeedsX) {
        load_row(2 * m + 2, n0);
        load_row(2 * m + 3, n1);
      }
      load_windows(m + 1, ng, ncode);
      ahead(m + 2);
    }
    int at0 = kNoCell, at1 = kNoCell;
    float best0 = 0.f, best1 = 0.f;
    if (kNeedsX) {
      float l0 = __shfl_up_sync(kAll, r0[3], 1), l1 = __shfl_up_sync(kAll, r1[3], 1);
      if (!has_left) l0 = l1 = kPad;
      if (kMax) {
        const bool odd0 = __any_sync(kAll, unordered(r0)), odd1 = __any_sync(kAll, unordered(r1));
        auto windows = [&](auto nans) {
          constexpr bool kNans = decltype(nans)::value;
          float v[2][3] = {{top[0]}, {top[1]}};
          int col[2][3] = {{top_at[0]}, {top_at[1]}};
          first_of_cells<kNans>(l0, r0[0], r0[1], v[0][1], col[0][1]);
          first_of_cells<kNans>(r0[1], r0[2], r0[3], v[1][1], col[1][1]);
          first_of_cells<kNans>(l1, r1[0], r1[1], v[0][2], col[0][2]);
          first_of_cells<kNans>(r1[1], r1[2], r1[3], v[1][2], col[1][2]);
          first_of_rows<kNans>(v[0], col[0], best0, at0);
          first_of_rows<kNans>(v[1], col[1], best1, at1);
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            top[j] = v[j][2];
            top_at[j] = col[j][2];
          }
        };
        if (odd_above || odd0 || odd1) windows(std::true_type{});
        else windows(std::false_type{});
        odd_above = odd1;
      } else {
        const float w0[9] = {above_left, above[0], above[1], l0, r0[0], r0[1], l1, r1[0], r1[1]};
        const float w1[9] = {above[1], above[2], above[3], r0[1], r0[2], r0[3], r1[1], r1[2], r1[3]};
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          best0 += w0[k];
          best1 += w1[k];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) above[j] = r1[j];
        above_left = l1;
      }
    }
    if (MODE == kMaxBwdRecord) {
      at0 = code[0] == 0xffu ? kNoCell : static_cast<int>(code[0] >> 4) * 3 + static_cast<int>(code[0] & 15u);
      at1 = code[1] == 0xffu ? kNoCell : static_cast<int>(code[1] >> 4) * 3 + static_cast<int>(code[1] & 15u);
    }
    if (!kMax) {
      // cells inside the plane: the divisor excludes the padding
      const int rows_in = 3 - (m == 0) - (2 * m + 1 >= H);
      const float n_0 = static_cast<float>(rows_in * (3 - (c == 0) - (c + 1 >= W)));
      const float n_1 = static_cast<float>(rows_in * (3 - (c + 3 >= W)));
      if (kBackward) {
        g[0] = g[0] / n_0;
        g[1] = w1_exists ? g[1] / n_1 : 0.0f;
      } else {
        best0 = best0 / n_0;
        best1 = best1 / n_1;
      }
    }
    if (!kBackward) {
      if (owner) {
        const size_t i = window0 + static_cast<size_t>(m) * OW;
        if (VEC) {
          *reinterpret_cast<float2*>(a.out + i) = make_float2(best0, best1);
        } else {
          a.out[i] = best0;
          if (w1_exists) a.out[i + 1] = best1;
        }
        if (MODE == kMaxFwdRecord) {
          const unsigned c0 = at0 < 0 ? 0xffu : static_cast<unsigned>((at0 / 3) << 4 | at0 % 3);
          const unsigned c1 = at1 < 0 ? 0xffu : static_cast<unsigned>((at1 / 3) << 4 | at1 % 3);
          if (VEC) {
            *reinterpret_cast<unsigned short*>(a.record + i) = static_cast<unsigned short>(c0 | c1 << 8);
          } else {
            a.record[i] = static_cast<unsigned char>(c0);
            if (w1_exists) a.record[i + 1] = static_cast<unsigned char>(c1);
          }
        }
      }
    } else {
      if (!w1_exists) at1 = kNoCell;
      int at2 = __shfl_down_sync(kAll, at0, 1);
      float g2 = __shfl_down_sync(kAll, g[0], 1);
      if (!has_right) {
        at2 = kNoCell;
        g2 = 0.0f;
      }
      // gradient of the four columns in window row DR of the three, windows in raster order
      auto row_of = [&](int dr, float (&v)[4]) {
        if (kMax) {
          v[0] = v[0] + (at0 == 3 * dr + 1 ? g[0] : 0.0f);
          v[1] = (v[1] + (at0 == 3 * dr + 2 ? g[0] : 0.0f)) + (at1 == 3 * dr ? g[1] : 0.0f);
          v[2] = v[2] + (at1 == 3 * dr + 1 ? g[1] : 0.0f);
          v[3] = (v[3] + (at1 == 3 * dr + 2 ? g[1] : 0.0f)) + (at2 == 3 * dr ? g2 : 0.0f);
        } else {
          v[0] = v[0] + g[0];
          v[1] = (v[1] + g[0]) + g[1];
          v[2] = v[2] + g[1];
          v[3] = (v[3] + g[1]) + g2;
        }
      };
      if (m > m0) {
        row_of(0, pend);
        store_row(2 * m - 1, pend);
      }
      if (m < m1) {
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        row_of(1, v);
        store_row(2 * m, v);
#pragma unroll
        for (int j = 0; j < 4; ++j) pend[j] = 0.f;
        row_of(2, pend);
      }
    }
  }
  if (kBackward && m1 == OH) store_row(2 * OH - 1, pend);   // below it there is no further window
}

StripArgs strip_args(const float* x, const float* dy, float* out, unsigned char* record, const PoolShape& p,
                     long long warps_per_sm = 96) {
  StripArgs a;
  a.x = x;
  a.dy = dy;
  a.out = out;
  a.record = record;
  a.planes = p.N * p.C;
  a.H = p.H;
  a.W = p.W;
  a.OH = p.OH;
  a.OW = p.OW;
  a.quads = (p.W + 3) / 4;
  a.abreast = a.quads <= 32 ? 32 / a.quads : 1;
  a.segments = a.quads <= 32 ? 1 : (a.quads + 29) / 30;
  // A band re-reads the row above it (and, backward, works out the window rows
  // at its edges twice), so bands are as tall as leaves about three warps per
  // slot of the machine (32 per SM), at least four window rows.  Where the extra
  // rows cost the most (`warps_per_sm`, see launch_k3s1p1) they are taller.
  const long long strips = static_cast<long long>((a.planes + a.abreast - 1) / a.abreast) * a.segments;
  const long long want = (static_cast<long long>(sm_count()) * warps_per_sm + strips - 1) / strips;   // bands wanted
  long long rows = (p.OH + want - 1) / want;
  if (rows < 4) rows = 4;
  if (rows > p.OH) rows = p.OH;
  a.bands = static_cast<int>((p.OH + rows - 1) / rows);
  a.rows = (p.OH + a.bands - 1) / a.bands;       // even heights
  a.bands = (p.OH + a.rows - 1) / a.rows;
  return a;
}
long long strip_ctas(const StripArgs& a) {
  const long long strips = static_cast<long long>((a.planes + a.abreast - 1) / a.abreast) * a.segments;
  return (strips * a.bands + kBlock / 32 - 1) / (kBlock / 32);
}
template <int MODE>
int launch_k3s2p1(const float* x, const float* dy, float* out, unsigned char* record, const PoolShape& p, cudaStream_t s) {
  const StripArgs a = strip_args(x, dy, out, record, p);
  const long long ctas = strip_ctas(a);
  if (ctas > 0x7fffffffLL) return SGB_ERR_SIZE;
  const bool vec = p.W % 4 == 0 && (!x || aligned16(x)) && (!dy || aligned16(dy)) && aligned16(out) &&
                   (reinterpret_cast<uintptr_t>(record) & 1u) == 0;
  return launch_ex(vec ? pool_k3s2p1_kernel<MODE, true> : pool_k3s2p1_kernel<MODE, false>,
                   dim3(static_cast<unsigned>(ctas)), dim3(kBlock), 0, s, 0, true, a);
}
inline bool is_k3s2p1(const PoolShape& p) {
  return p.kh == 3 && p.kw == 3 && p.sh == 2 && p.sw == 2 && p.ph == 1 && p.pw == 1;
}

// ------------------------------------------------ 3x3 / stride 1 / pad 1, max passes
// Same layout: a lane owns four columns and the four windows centred on them.
// The first maximum of three adjacent cells of a row is worked out once and
// serves the three windows it belongs to (5 comparisons per window instead of
// 9: two for a row's winner, two between the rows, one against the lowest value).
// Was 231 us forward and 276 us backward at 32x64x112x112, where the bytes take 31 and 47 us,
// and 56.5 and 104.2 when all comparisons looked for NaNs and began at the lowest value; now
// 47.7 and 90.2.  The backward pass of rows off a vector's boundary has registers for three
// CTAs an SM only (64x512x14x14 38.0 us with four and spilled ones, 30.1 with three;
// 64x64x35x35 33.2 and 27.4).
struct RowBest {
  float v[4];
  int at[4];               // column offset 0..2 of the winner
};

template <int MODE, bool VEC>
__global__ void __launch_bounds__(kBlock, MODE == kMaxBwd && !VEC ? 3 : 4)
pool_k3s1p1_kernel(const StripArgs a) {
  constexpr bool kBackward = MODE == kMaxBwd || MODE == kMaxBwdRecord;
  constexpr bool kNeedsX = MODE != kMaxBwdRecord;
  constexpr unsigned kAll = 0xffffffffu;
  dependency_wait();
  release_dependents();
  const int lane = threadIdx.x & 31;
  const unsigned task = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5);
  const unsigned rest = task / a.bands;
  const int band = static_cast<int>(task - rest * a.bands);
  const int group = static_cast<int>(rest / a.segments), seg = static_cast<int>(rest - group * a.segments);
  int q, plane;
  bool active, owner;
  if (a.segments > 1) {
    q = seg * 30 - 1 + lane;
    plane = group;
    active = q >= 0 && q < a.quads && plane < a.planes;
    owner = active && lane >= 1 && lane <= 30;
  } else {
    const int pl = lane / a.quads;
    q = lane - pl * a.quads;
    plane = group * a.abreast + pl;
    active = pl < a.abreast && plane < a.planes;
    owner = active;
  }
  if (!active) plane = 0;
  const int H = a.H, W = a.W, c = 4 * q;
  const size_t origin = static_cast<size_t>(plane) * H * W + c;      // input and output planes have one size
  const bool has_left = q > 0, has_right = q + 1 < a.quads;

  auto load4 = [&](const float* p, int h, float pad, float (&v)[4]) {
    const bool in = active && h >= 0 && h < H;
    const float* r = p + origin + static_cast<ptrdiff_t>(h) * W;
    if (VEC) {
      float4 t = make_float4(pad, pad, pad, pad);
      if (in) t = *reinterpret_cast<const float4*>(r);
      v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = in && c + j < W ? r[j] : pad;
    }
  };
  auto store4 = [&](float* p, int h, const float (&v)[4]) {
    if (!owner || h < 0 || h >= H) return;
    float* r = p + origin + static_cast<size_t>(h) * W;
    if (VEC) {
      *reinterpret_cast<float4*>(r) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c + j < W) r[j] = v[j];
    }
  };
  // the winner of each window's three cells in one row, and whether the row
  // (of the whole warp) holds anything that needs the NaN-aware comparison
  auto row_best = [&](const float (&v)[4], RowBest& b) -> bool {
    float left = __shfl_up_sync(kAll, v[3], 1), right = __shfl_down_sync(kAll, v[0], 1);
    if (!has_left) left = -FLT_MAX;
    if (!has_right) right = -FLT_MAX;
    const float s = (v[0] + v[1]) + (v[2] + v[3]);
    const bool nans = __any_sync(kAll, s != s);
    const float cell[6] = {left, v[0], v[1], v[2], v[3], right};
    auto work_out = [&](auto kind) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        first_of_cells<decltype(kind)::value>(cell[j], cell[j + 1], cell[j + 2], b.v[j], b.at[j]);
    };
    if (nans) work_out(std::true_type{});
    else work_out(std::false_type{});
    return nans;
  };

  // forward: output rows [m0, m1); backward: window rows m0 - 1 .. m1 feed dx rows [m0, m1)
  const int m0 = band * a.rows, m1 = min(m0 + a.rows, H);
  const int first = kBackward ? max(m0 - 1, 0) : m0, last = kBackward ? min(m1, H - 1) : m1 - 1;
  RowBest up, mid, low;
  bool nan_up = false, nan_mid = false, nan_low = false;
  float v[4], ahead[4], g[4], g_ahead[4];
  unsigned code_ahead[4] = {0, 0, 0, 0}, code[4];
  auto load_codes = [&](int m, unsigned (&k)[4]) {
    const unsigned char* r = a.record + origin + static_cast<size_t>(m) * W;
    if (VEC) {
      const unsigned t = active ? *reinterpret_cast<const unsigned*>(r) : 0xffffffffu;
#pragma unroll
      for (int j = 0; j < 4; ++j) k[j] = t >> (8 * j) & 0xffu;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) k[j] = active && c + j < W ? r[j] : 0xffu;
    }
  };
  if (kNeedsX) {
    load4(a.x, first - 1, -FLT_MAX, v);
    load4(a.x, first, -FLT_MAX, ahead);
    nan_up = row_best(v, up);
    nan_mid = row_best(ahead, mid);
    load4(a.x, first + 1, -FLT_MAX, ahead);
  }
  if (kBackward) load4(a.dy, first, 0.0f, g_ahead);
  if (MODE == kMaxBwdRecord) load_codes(first, code_ahead);
  float acc0[4] = {0.f, 0.f, 0.f, 0.f}, acc1[4] = {0.f, 0.f, 0.f, 0.f};   // dx rows m - 1 and m so far
  for (int m = first; m <= last; ++m) {
    int win[4];
    float best[4];
    if (kNeedsX) {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = ahead[j];
      if (m < last) load4(a.x, m + 2, -FLT_MAX, ahead);
    }
    if (kBackward) {
#pragma unroll
      for (int j = 0; j < 4; ++j) g[j] = g_ahead[j];
      if (m < last) load4(a.dy, m + 1, 0.0f, g_ahead);
    }
    if (MODE == kMaxBwdRecord) {
#pragma unroll
      for (int j = 0; j < 4; ++j) code[j] = code_ahead[j];
      if (m < last) load_codes(m + 1, code_ahead);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        win[j] = code[j] == 0xffu ? kNoCell : static_cast<int>(code[j] >> 4) * 3 + static_cast<int>(code[j] & 15u);
    }
    if (kNeedsX) {
      nan_low = row_best(v, low);
      auto windows = [&](auto kind) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float rows[3] = {up.v[j], mid.v[j], low.v[j]};
          const int col[3] = {up.at[j], mid.at[j], low.at[j]};
          first_of_rows<decltype(kind)::value>(rows, col, best[j], win[j]);
          if (kBackward && c + j >= W) win[j] = kNoCell;
        }
      };
      if (nan_up || nan_mid || nan_low) windows(std::true_type{});
      else windows(std::false_type{});
      up = mid;
      mid = low;
      nan_up = nan_mid;
      nan_mid = nan_low;
    }
    if (!kBackward) {
      store4(a.out, m, best);
      if (MODE == kMaxFwdRecord && owner) {
        unsigned char* r = a.record + origin + static_cast<size_t>(m) * W;
        unsigned packed = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const unsigned k = win[j] < 0 ? 0xffu : static_cast<unsigned>((win[j] / 3) << 4 | win[j] % 3);
          packed |= k << (8 * j);
          if (!VEC && c + j < W) r[j] = static_cast<unsigned char>(k);
        }
        if (VEC) *reinterpret_cast<unsigned*>(r) = packed;
      }
      continue;
    }
    // the windows centred on columns c-1 .. c+4
    int w[6];
    float gw[6];
    w[0] = __shfl_up_sync(kAll, win[3], 1);
    gw[0] = __shfl_up_sync(kAll, g[3], 1);
    w[5] = __shfl_down_sync(kAll, win[0], 1);
    gw[5] = __shfl_down_sync(kAll, g[0], 1);
    if (!has_left) w[0] = kNoCell;
    if (!has_right) w[5] = kNoCell;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      w[j + 1] = win[j];
      gw[j + 1] = g[j];
    }
    // column c + j lies in the windows j, j + 1, j + 2 of that list, at column offsets 2, 1, 0
    auto add_row = [&](int dr, float (&t)[4]) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int k = 0; k < 3; ++k) t[j] += w[j + k] == 3 * dr + 2 - k ? gw[j + k] : 0.0f;
    };
    add_row(0, acc0);
    if (m - 1 >= m0) store4(a.out, m - 1, acc0);
    add_row(1, acc1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      acc0[j] = acc1[j];
      acc1[j] = 0.f;
    }
    add_row(2, acc1);
  }
  if (kBackward && m1 == H) store4(a.out, H - 1, acc0);     // below it there is no further window row
}

template <int MODE>
int launch_k3s1p1(const float* x, const float* dy, float* out, unsigned char* record, const PoolShape& p, cudaStream_t s) {
  // Backward, a band works out two window rows more than it owns, and comparisons
  // are what bounds it: bands twice as tall (1.5 warps per slot) were as fast or
  // faster on each of ten shapes: 32x64x112x112 115.0 -> 104.8 us, 16x128x56x56
  // 43.5 -> 38.1, 64x512x14x14 44.8 -> 34.7; fewer warps than that idle the machine.
  constexpr bool kBackward = MODE == kMaxBwd || MODE == kMaxBwdRecord;
  const StripArgs a = strip_args(x, dy, out, record, p, kBackward ? 48 : 96);
  const long long ctas = strip_ctas(a);
  if (ctas > 0x7fffffffLL) return SGB_ERR_SIZE;
  const bool vec = p.W % 4 == 0 && (!x || aligned16(x)) && (!dy || aligned16(dy)) && aligned16(out) &&
                   (reinterpret_cast<uintptr_t>(record) & 3u) == 0;
  return launch_ex(vec ? pool_k3s1p1_kernel<MODE, true> : pool_k3s1p1_kernel<MODE, false>,
                   dim3(static_cast<unsigned>(ctas)), dim3(kBlock), 0, s, 0, true, a);
}

// ------------------------------------------------ 2x2 / stride 2 / no padding
// The windows do not overlap: a thread owns four columns of two rows, i.e. two
// whole windows.  Rows and columns that no window covers (odd sizes) get zero
// gradient.  One 16-byte access per row where the width allows it.
struct PairArgs {
  const float* x;
  const float* dy;
  float* out;
  unsigned char* record;
  unsigned work;           // planes * row pairs * quads, < 2^31
  int H, W, OH, OW;
  FastDiv quads, pairs;    // quads per row, row pairs per plane
};

template <int MODE, bool VEC>
__global__ void __launch_bounds__(kBlock)
pool_k2s2_kernel(const PairArgs a) {
  constexpr bool kBackward = MODE == kMaxBwd || MODE == kMaxBwdRecord || MODE == kAvgBwd;
  constexpr bool kNeedsX = MODE != kMaxBwdRecord && MODE != kAvgBwd;
  constexpr bool kMax = MODE <= kMaxBwdRecord;
  const unsigned i = blockIdx.x * static_cast<unsigned>(kBlock) + threadIdx.x;
  const unsigned line = a.quads.quot(i);
  const int c = 4 * static_cast<int>(i - line * a.quads.d);
  const unsigned plane = a.pairs.quot(line);
  const int m = static_cast<int>(line - plane * a.pairs.d), h = 2 * m;
  const size_t in0 = (static_cast<size_t>(plane) * a.H + h) * a.W + c;
  const size_t win = (static_cast<size_t>(plane) * a.OH + m) * a.OW + c / 2;
  const bool second_row = h + 1 < a.H;
  const bool exists[2] = {second_row && c + 1 < a.W, second_row && c + 3 < a.W};
  if (kBackward && kNeedsX && i < a.work) {
    prefetch_l2(a.x + in0);
    if (second_row) prefetch_l2(a.x + in0 + a.W);
  }
  dependency_wait();
  release_dependents();
  if (i >= a.work) return;
  float v[2][4];
  if (kNeedsX) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      if (VEC) {
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r == 0 || second_row) t = *reinterpret_cast<const float4*>(a.x + in0 + static_cast<size_t>(r) * a.W);
        v[r][0] = t.x; v[r][1] = t.y; v[r][2] = t.z; v[r][3] = t.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          v[r][j] = (r == 0 || second_row) && c + j < a.W ? a.x[in0 + static_cast<size_t>(r) * a.W + j] : 0.0f;
      }
    }
  }
  float o[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    if (!exists[w]) continue;
    int at = kNoCell;
    float best = kMax ? -FLT_MAX : 0.0f;
    if (kNeedsX) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float t = v[k >> 1][2 * w + (k & 1)];
        if (kMax) {
          if (t > best || (t != t && best == best)) {   // first maximum; a NaN wins and then sticks, as in cuDNN
            best = t;
            at = k;
          }
        } else {
          best += t;
        }
      }
    }
    if (!kBackward) {
      a.out[win + w] = kMax ? best : best / 4.0f;
      if (MODE == kMaxFwdRecord)
        a.record[win + w] = at < 0 ? 0xff : static_cast<unsigned char>((at >> 1) << 4 | (at & 1));
      continue;
    }
    float g = a.dy[win + w];
    if (MODE == kMaxBwdRecord) {
      const unsigned code = a.record[win + w];
      at = code == 0xffu ? kNoCell : static_cast<int>(code >> 4) * 2 + static_cast<int>(code & 15u);
    }
    if (MODE == kAvgBwd) g = g / 4.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k >> 1][2 * w + (k & 1)] = 0.0f + (!kMax || at == k ? g : 0.0f);
  }
  if (!kBackward) return;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    if (r == 1 && !second_row) break;
    float* p = a.out + in0 + static_cast<size_t>(r) * a.W;
    if (VEC) {
      *reinterpret_cast<float4*>(p) = make_float4(o[r][0], o[r][1], o[r][2], o[r][3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c + j < a.W) p[j] = o[r][j];
    }
  }
}

inline bool is_k2s2(const PoolShape& p) {
  const long long work = static_cast<long long>(p.N) * p.C * ((p.H + 1) / 2) * ((p.W + 3) / 4);
  return p.kh == 2 && p.kw == 2 && p.sh == 2 && p.sw == 2 && p.ph == 0 && p.pw == 0 && work < 0x7fffffffLL;
}
template <int MODE>
int launch_k2s2(const float* x, const float* dy, float* out, unsigned char* record, const PoolShape& p, cudaStream_t s) {
  const unsigned quads = (p.W + 3) / 4, pairs = (p.H + 1) / 2;
  const unsigned work = static_cast<unsigned>(p.N) * p.C * pairs * quads;
  const PairArgs a{x, dy, out, record, work, p.H, p.W, p.OH, p.OW, FastDiv(quads), FastDiv(pairs)};
  const bool backward = MODE == kMaxBwd || MODE == kMaxBwdRecord || MODE == kAvgBwd;
  const bool vec = p.W % 4 == 0 && (!x || aligned16(x)) && (!backward || aligned16(out));
  return launch_ex(vec ? pool_k2s2_kernel<MODE, true> : pool_k2s2_kernel<MODE, false>,
                   dim3(static_cast<unsigned>(ceil_div(work, kBlock))), dim3(kBlock), 0, s, 0, true, a);
}

// Global average (one window = the whole plane): a warp adds up one plane.
__global__ void __launch_bounds__(kBlock)
avgpool_fwd_global_kernel(const float* __restrict__ x, float* __restrict__ y, int planes, int hw) {
  dependency_wait();
  release_dependents();
  const int plane = static_cast<int>(blockIdx.x) * (kBlock / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (plane >= planes) return;
  const float* p = x + static_cast<size_t>(plane) * hw;
  float s = 0.f;
#pragma unroll 8
  for (int i = lane; i < hw; i += 32) s += p[i];
  s = warp_sum(s);
  if (lane == 0) y[plane] = s / static_cast<float>(hw);
}

// The geometries above, if `p` is one of them; `done` tells.
template <int MODE>
int launch_known(const float* x, const float* dy, float* out, unsigned char* record, const PoolShape& p, cudaStream_t s,
                 bool* done) {
  *done = true;
  if (is_k3s2p1(p) && static_cast<long long>(p.N) * p.C <= 0x7fffffffLL)
    return launch_k3s2p1<MODE>(x, dy, out, record, p, s);
  if (is_k2s2(p)) return launch_k2s2<MODE>(x, dy, out, record, p, s);
  if constexpr (MODE <= kMaxBwdRecord)
    if (p.kh == 3 && p.kw == 3 && p.sh == 1 && p.sw == 1 && p.ph == 1 && p.pw == 1 &&
        static_cast<long long>(p.N) * p.C <= 0x7fffffffLL)
      return launch_k3s1p1<MODE>(x, dy, out, record, p, s);
  *done = false;
  return SGB_OK;
}

// Band height: the largest power-of-two-ish row count whose staging fits
// `budget` bytes of shared memory; 0 rows means even one row does not fit.
BandPlan plan_bands(const PoolShape& p, size_t budget) {
  BandPlan bp{0, 0, 0, 0};
  for (int rows = p.H; rows >= 1; rows = (rows > 64 ? (rows + 1) / 2 : rows - 1)) {
    // windows covering `rows` consecutive dx rows, and the x rows they touch
    const int orows = min((rows + p.kh - 2) / p.sh + 2, p.OH);
    const int xrows = min((orows - 1) * p.sh + p.kh, p.H);
    const size_t bytes = (static_cast<size_t>(xrows) * p.W + 2 * static_cast<size_t>(orows) * p.OW) * 4;
    if (bytes <= budget) {
      bp.rows = rows;
      bp.bands = (p.H + rows - 1) / rows;
      bp.max_xrows = xrows;
      bp.max_orows = orows;
      return bp;
    }
  }
  return bp;
}

// Fallback for planes whose winner table does not fit shared memory: every dx
// element re-derives the winner of each covering window from x.
__global__ void __launch_bounds__(kBlock)
maxpool_bwd_kernel(const float* __restrict__ x, const float* __restrict__ dy,
                   float* __restrict__ dx, PoolShape p) {
  dependency_wait();
  release_dependents();
  const size_t plane = blockIdx.x;
  const int i = blockIdx.y * kBlock + threadIdx.x;
  if (i >= p.H * p.W) return;
  const int h = i / p.W, w = i - h * p.W;
  const float* xp = x + plane * p.H * p.W;
  const float* gp = dy + plane * p.OH * p.OW;
  const float mine = xp[i];
  int oh_lo, oh_hi, ow_lo, ow_hi;
  covering(h, p.ph, p.kh, p.sh, p.OH, oh_lo, oh_hi);
  covering(w, p.pw, p.kw, p.sw, p.OW, ow_lo, ow_hi);
  float acc = 0.f;
  for (int oh = oh_lo; oh <= oh_hi; ++oh)
    for (int ow = ow_lo; ow <= ow_hi; ++ow) {
      int h0, h1, w0, w1;
      window(p, oh, ow, h0, h1, w0, w1);
      // (h, w) wins this window iff nothing before it (raster order) is >= it
      // and nothing after it is > it, and it beats the -FLT_MAX seed.
      bool win = mine > -FLT_MAX;
      for (int hh = h0; hh < h1 && win; ++hh)
        for (int ww = w0; ww < w1; ++ww) {
          const float v = xp[hh * p.W + ww];
          const bool before = hh < h || (hh == h && ww < w);
          if (before ? (v >= mine) : (v > mine)) {
            win = false;
            break;
          }
        }
      if (win) acc += gp[oh * p.OW + ow];
    }
  dx[plane * p.H * p.W + i] = acc;
}

// Average backward: one thread per dx element over the flattened tensor
// (chunks of < 2^31 elements so the index arithmetic stays 32-bit).
__global__ void __launch_bounds__(kBlock)
avgpool_bwd_kernel(const float* __restrict__ dy, float* __restrict__ dx, PoolShape p,
                   unsigned total) {
  dependency_wait();
  release_dependents();
  const unsigned i = blockIdx.x * static_cast<unsigned>(kBlock) + threadIdx.x;
  if (i >= total) return;
  const unsigned hw = static_cast<unsigned>(p.H * p.W);
  const unsigned plane = i / hw, r = i - plane * hw;
  const int h = static_cast<int>(r / static_cast<unsigned>(p.W)), w = static_cast<int>(r) - h * p.W;
  const float* gp = dy + static_cast<size_t>(plane) * p.OH * p.OW;
  int oh_lo, oh_hi, ow_lo, ow_hi;
  covering(h, p.ph, p.kh, p.sh, p.OH, oh_lo, oh_hi);
  covering(w, p.pw, p.kw, p.sw, p.OW, ow_lo, ow_hi);
  float acc = 0.f;
  for (int oh = oh_lo; oh <= oh_hi; ++oh)
    for (int ow = ow_lo; ow <= ow_hi; ++ow) {
      int h0, h1, w0, w1;
      window(p, oh, ow, h0, h1, w0, w1);
      acc += gp[oh * p.OW + ow] / static_cast<float>((h1 - h0) * (w1 - w0));
    }
  dx[i] = acc;
}

// Global average pooling (one window = the whole plane, no padding): every dx
// element of a plane is dy[plane] / (H*W).  Four consecutive elements per
// thread, one 128-bit store; the plane index advances without extra divisions.
__global__ void __launch_bounds__(kBlock)
avgpool_bwd_global_kernel(const float* __restrict__ dy, float* __restrict__ dx, unsigned hw,
                          unsigned total4) {
  dependency_wait();
  release_dependents();
  const unsigned v = blockIdx.x * static_cast<unsigned>(kBlock) + threadIdx.x;
  if (v >= total4) return;
  const unsigned i = 4u * v;
  unsigned plane = i / hw, r = i - plane * hw;
  const float inv = static_cast<float>(hw);
  float out[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    out[e] = dy[plane] / inv;
    if (++r == hw) {
      r = 0;
      ++plane;
    }
  }
  *reinterpret_cast<float4*>(dx + i) = make_float4(out[0], out[1], out[2], out[3]);
}

int make_shape(PoolShape& p, int N, int C, int H, int W, int kh, int kw, int ph, int pw, int sh,
               int sw) {
  if (N < 0 || C < 0 || H <= 0 || W <= 0 || kh <= 0 || kw <= 0 || ph < 0 || pw < 0 || sh <= 0 ||
      sw <= 0)
    return SGB_ERR_SIZE;
  if (ph >= kh || pw >= kw) return SGB_ERR_SIZE;  // a window must touch the image
  if (H + 2 * ph < kh || W + 2 * pw < kw) return SGB_ERR_SIZE;
  p = PoolShape{N, C, H, W, (H + 2 * ph - kh) / sh + 1, (W + 2 * pw - kw) / sw + 1,
                kh, kw, ph, pw, sh, sw};
  return SGB_OK;
}

unsigned blocks_for(size_t total) { return static_cast<unsigned>(ceil_div(total, kBlock)); }

}  // namespace
}  // namespace sgb

using namespace sgb;

extern "C" {

int sgb_pool_out_size(int in, int kernel, int pad, int stride) {
  if (stride <= 0) return 1;
  return (in + 2 * pad - kernel) / stride + 1;
}

#define POOL_PROLOGUE(OUT_IS_Y)                                                        \
  PoolShape p;                                                                         \
  int st = make_shape(p, N, C, H, W, kh, kw, ph, pw, sh, sw);                          \
  if (st != SGB_OK) return st;                                                         \
  const size_t in_total = static_cast<size_t>(N) * C * H * W;                          \
  const size_t out_total = static_cast<size_t>(N) * C * p.OH * p.OW;                   \
  (void)in_total; (void)out_total;                                                     \
  if (in_total == 0) return SGB_OK;                                                    \
  if (ceil_div(in_total, kBlock) > 0x7fffffffu) return SGB_ERR_SIZE;

int sgb_maxpool_forward_f32(const float* x, float* y, int N, int C, int H, int W, int kh, int kw,
                            int ph, int pw, int sh, int sw, void* stream) {
  POOL_PROLOGUE(1)
  if (!x || !y) return SGB_ERR_NULL;
  bool done;
  const int r = launch_known<kMaxFwd>(x, nullptr, y, nullptr, p, as_stream(stream), &done);
  if (done) return r;
  return launch_ex(pool_fwd_kernel<true>, dim3(blocks_for(out_total)), dim3(kBlock), 0, as_stream(stream), 0, true, x, y,
                   p, out_total);
}

int sgb_avgpool_forward_f32(const float* x, float* y, int N, int C, int H, int W, int kh, int kw,
                            int ph, int pw, int sh, int sw, void* stream) {
  POOL_PROLOGUE(1)
  if (!x || !y) return SGB_ERR_NULL;
  if (p.OH == 1 && p.OW == 1 && ph == 0 && pw == 0 && kh == H && kw == W &&
      static_cast<long long>(N) * C <= 0x7fffffffLL && static_cast<long long>(H) * W <= 0x7fffffffLL)
    return launch_ex(avgpool_fwd_global_kernel, dim3(static_cast<unsigned>(ceil_div(out_total, kBlock / 32))),
                     dim3(kBlock), 0, as_stream(stream), 0, true, x, y, N * C, H * W);
  bool done;
  const int r = launch_known<kAvgFwd>(x, nullptr, y, nullptr, p, as_stream(stream), &done);
  if (done) return r;
  return launch_ex(pool_fwd_kernel<false>, dim3(blocks_for(out_total)), dim3(kBlock), 0, as_stream(stream), 0, true, x,
                   y, p, out_total);
}

int sgb_maxpool_backward_f32(const float* x, const float* y, const float* dy, float* dx, int N,
                             int C, int H, int W, int kh, int kw, int ph, int pw, int sh, int sw,
                             void* stream) {
  (void)y;  // the winner is recomputed from x; y is accepted for interface parity
  POOL_PROLOGUE(0)
  if (!x || !dy || !dx) return SGB_ERR_NULL;
  const size_t planes = static_cast<size_t>(N) * C;
  if (planes > 0x7fffffffu || static_cast<long long>(H) * W > 0x7fffffffLL) return SGB_ERR_SIZE;
  cudaStream_t s = as_stream(stream);
  bool done;
  const int r = launch_known<kMaxBwd>(x, dy, dx, nullptr, p, s, &done);
  if (done) return r;
  const BandPlan bp = plan_bands(p, 24 * 1024);
  if (bp.rows > 0 && bp.bands <= 65535) {
    const size_t smem = (static_cast<size_t>(bp.max_xrows) * W +
                         2 * static_cast<size_t>(bp.max_orows) * p.OW) * sizeof(float);
    const dim3 grid(static_cast<unsigned>(planes), bp.bands);
    const bool square = kh == kw && sh == sw && ph == pw && W % 4 == 0 && aligned16(x) && aligned16(dx);
#define SGB_POOL_FAST(KK, SS, PP)                                                       \
  if (square && kh == KK && sh == SS && ph == PP)                                       \
    return launch_ex(maxpool_bwd_band_fast_kernel<KK, SS, PP>, grid, dim3(kBlock), smem, s, 0, true, x, dy, dx, p, bp);
    SGB_POOL_FAST(3, 2, 0)
    SGB_POOL_FAST(2, 1, 0)
#undef SGB_POOL_FAST
    return launch_ex(maxpool_bwd_band_kernel, grid, dim3(kBlock), smem, s, 0, true, x, dy, dx, p, bp);
  }
  const unsigned by = blocks_for(static_cast<size_t>(H) * W);
  if (by > 65535) return SGB_ERR_SIZE;
  return launch_ex(maxpool_bwd_kernel, dim3(static_cast<unsigned>(planes), by), dim3(kBlock), 0, s, 0, true, x, dy, dx, p);
}

int sgb_maxpool_forward_argmax_f32(const float* x, float* y, unsigned char* argmax, int N, int C, int H,
                                   int W, int kh, int kw, int ph, int pw, int sh, int sw, void* stream) {
  POOL_PROLOGUE(1)
  if (!x || !y || !argmax) return SGB_ERR_NULL;
  if (kh > 15 || kw > 15) return SGB_ERR_UNSUPPORTED;           // offsets are stored in nibbles; 15|15 is "none"
  bool done;
  const int r = launch_known<kMaxFwdRecord>(x, nullptr, y, argmax, p, as_stream(stream), &done);
  if (done) return r;
  return launch_ex(maxpool_fwd_argmax_kernel, dim3(blocks_for(out_total)), dim3(kBlock), 0, as_stream(stream), 0, true,
                   x, y, argmax, p, out_total);
}

int sgb_maxpool_backward_argmax_f32(const float* dy, const unsigned char* argmax, float* dx, int N, int C,
                                    int H, int W, int kh, int kw, int ph, int pw, int sh, int sw,
                                    void* stream) {
  POOL_PROLOGUE(0)
  if (!dy || !argmax || !dx) return SGB_ERR_NULL;
  if (kh > 15 || kw > 15) return SGB_ERR_UNSUPPORTED;
  cudaStream_t s = as_stream(stream);
  bool done;
  const int r = launch_known<kMaxBwdRecord>(nullptr, dy, dx, const_cast<unsigned char*>(argmax), p, s, &done);
  if (done) return r;
  return launch_ex(maxpool_bwd_argmax_kernel, dim3(blocks_for(in_total)), dim3(kBlock), 0, s, 0, true, dy, argmax, dx, p,
                   in_total);
}

int sgb_avgpool_backward_f32(const float* dy, float* dx, int N, int C, int H, int W, int kh,
                             int kw, int ph, int pw, int sh, int sw, void* stream) {
  POOL_PROLOGUE(0)
  if (!dy || !dx) return SGB_ERR_NULL;
  const size_t planes = static_cast<size_t>(N) * C;
  if (static_cast<long long>(H) * W > 0x7fffffffLL) return SGB_ERR_SIZE;
  if (p.OH == 1 && p.OW == 1 && ph == 0 && pw == 0 && kh == H && kw == W && aligned16(dx) &&
      in_total % 4 == 0 && in_total < 0x7fffffffu) {
    const unsigned total4 = static_cast<unsigned>(in_total / 4);
    return launch_ex(avgpool_bwd_global_kernel, dim3(blocks_for(total4)), dim3(kBlock), 0, as_stream(stream), 0, true,
                     dy, dx, static_cast<unsigned>(H * W), total4);
  }
  bool done;
  const int r = launch_known<kAvgBwd>(nullptr, dy, dx, nullptr, p, as_stream(stream), &done);
  if (done) return r;
  // whole planes per launch, each launch below 2^31 elements
  const size_t hw = static_cast<size_t>(H) * W;
  const size_t planes_per_launch = (0x7fffffffu - kBlock) / hw;
  if (planes_per_launch == 0) return SGB_ERR_SIZE;
  for (size_t p0 = 0; p0 < planes; p0 += planes_per_launch) {
    const size_t np = planes - p0 < planes_per_launch ? planes - p0 : planes_per_launch;
    const unsigned total = static_cast<unsigned>(np * hw);
    const int e = launch_ex(avgpool_bwd_kernel, dim3(blocks_for(total)), dim3(kBlock), 0, as_stream(stream), 0, true,
                            dy + p0 * p.OH * p.OW, dx + p0 * hw, p, total);
    if (e != SGB_OK) return e;
  }
  return launch_status();
}

}  // extern "C"
