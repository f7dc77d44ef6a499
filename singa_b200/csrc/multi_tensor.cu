// Multi-tensor kernels: one launch covers a whole list of parameter tensors.
//   * fused SGD update (weight decay, momentum, dampening, Nesterov, 1/world
//     gradient scaling) - one pass over p, g, m instead of the reference's
//     chain of 8-10 BLAS-1 / elementwise launches per tensor;
//   * bucket pack / unpack between a list of gradient tensors and the
//     communicator's flat staging buffer, with the fp32->fp16 cast on the way
//     in and the fp16->fp32 cast (+ scale) on the way out.
// The tensor table (pointers, sizes, first-tile index) travels in the kernel
// argument buffer, so there is no host-to-device table copy and no
// allocation.  Two table sizes: lists of up to 72 tensors stay below 4 KB of
// arguments, longer ones use the large buffer of this architecture (448
// tensors, 18 KB: all 161 of ResNet-50 in one launch instead of three), and
// only beyond that are several launches made.
// Every CTA handles one 1024-element tile and finds its tensor with a binary
// search over the table.
#include <type_traits>

#include "sgd.cuh"

namespace sgb {
namespace {

constexpr int kBlock = 256;
constexpr int kTile = 1024;       // elements per CTA (one float4 per thread)
constexpr int kSmallTable = 72, kLargeTable = 448;

template <int N>
struct Table {
  static constexpr int kMost = N;
  int count;
  unsigned first_tile[N + 1];
  unsigned long long n[N];
  void* a[N];  // param            | packed tensor
  void* b[N];  // grad             | (unused)
  void* c[N];  // momentum buffer  | (unused)
};
// flat-buffer element offset of tensor k (pack / unpack)
template <int N>
struct Offsets {
  unsigned long long off[N];
};

template <int N>
__device__ __forceinline__ int find_tensor(const Table<N>& t, unsigned tile) {
  int lo = 0, hi = t.count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.first_tile[mid] <= tile) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// ROUND: the gradient is rounded to fp16 and widened again on the way, and written
// back: what a one-rank exchange in half precision does to it.  One pass over p, g
// and m (24 B/element) instead of one over g and one over all three (28).
//
// ANY: some tensor is off a vector's boundary (tensors of any length lie back to back in
// a gradient arena), and four elements are still accessed together, as far as they can be.
// (us, the gradient off by one element: 1.2e6 elements 8.8 element by element, 5.0 so;
// 1.7e7 84.0 and 49.2.  In a kernel for both kinds the aligned lists took 5.0 instead of 4.4.)
template <int N, bool ROUND, bool ANY>
__global__ void __launch_bounds__(kBlock)
sgd_multi_kernel(const __grid_constant__ Table<N> t, const SgdArgs a) {
  const int k = find_tensor(t, blockIdx.x);
  const size_t n = t.n[k];
  const size_t base = static_cast<size_t>(blockIdx.x - t.first_tile[k]) * kTile;
  float* p = static_cast<float*>(t.a[k]);
  float* g = static_cast<float*>(t.b[k]);
  float* m = static_cast<float*>(t.c[k]);
  const size_t i = base + 4 * threadIdx.x;
  auto load = [](const float* from) {
    if (ANY) return ld4(from);
    Vec4f v;
    v.u = ld128(from);
    return v;
  };
  auto store = [](float* to, const Vec4f& v) {
    if (ANY) st4(to, v);
    else st128(to, v.u);
  };
  if (i + 4 <= n && first_wave(8)) {
    prefetch_l2(p + i);
    if (a.use_momentum) prefetch_l2(m + i);
  }
  dependency_wait();
  if (i + 4 <= n) {
    Vec4f vp = load(p + i), vg = load(g + i), vm;
    if (a.use_momentum) vm = load(m + i);
    release_dependents();
    if (ROUND) {
#pragma unroll
      for (int j = 0; j < 4; ++j) vg.f[j] = __half2float(__float2half_rn(vg.f[j]));
      store(g + i, vg);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) sgd_one(vp.f[j], vg.f[j], vm.f[j], a);
    store(p + i, vp);
    if (a.use_momentum) store(m + i, vm);
  } else {
    for (size_t j = i; j < n && j < i + 4; ++j) {
      float pv = p[j], gv = g[j], mv = a.use_momentum ? m[j] : 0.f;
      if (ROUND) g[j] = gv = __half2float(__float2half_rn(gv));
      sgd_one(pv, gv, mv, a);
      p[j] = pv;
      if (a.use_momentum) m[j] = mv;
    }
  }
}

// The same by one CTA an SM that walks the tiles, two at a time: for an update beside a
// chain of small kernels, which finds room on every SM.  A ResNet-50 step at batch 2 and
// images of 159, us: the update behind the chain 240, on a branch with all the CTAs that the
// SMs hold 228, with four an SM 239, three 230, two 227, one 206.
template <int N, bool ROUND>
__global__ void __launch_bounds__(kBlock)
sgd_beside_kernel(const __grid_constant__ Table<N> t, const SgdArgs a) {
  constexpr int kAbreast = 2;
  dependency_wait();
  release_dependents();
  const unsigned tiles = t.first_tile[t.count];
  for (unsigned first = blockIdx.x; first < tiles; first += kAbreast * gridDim.x) {
    float *p[kAbreast], *g[kAbreast], *m[kAbreast];
    int left[kAbreast];                                // elements from this thread's first on
    Vec4f vp[kAbreast], vg[kAbreast], vm[kAbreast];
#pragma unroll
    for (int k = 0; k < kAbreast; ++k) {
      const unsigned tile = first + k * gridDim.x;
      left[k] = 0;
      if (tile >= tiles) continue;
      const int j = find_tensor(t, tile);
      const size_t i = static_cast<size_t>(tile - t.first_tile[j]) * kTile + 4 * threadIdx.x;
      if (i >= t.n[j]) continue;
      left[k] = t.n[j] - i < 4 ? static_cast<int>(t.n[j] - i) : 4;
      p[k] = static_cast<float*>(t.a[j]) + i;
      g[k] = static_cast<float*>(t.b[j]) + i;
      m[k] = a.use_momentum ? static_cast<float*>(t.c[j]) + i : nullptr;
      if (left[k] < 4) continue;
      vp[k] = ld4(p[k]);
      vg[k] = ld4(g[k]);
      if (a.use_momentum) vm[k] = ld4(m[k]);
    }
#pragma unroll
    for (int k = 0; k < kAbreast; ++k) {
      if (left[k] == 4) {
        if (ROUND) {
#pragma unroll
          for (int j = 0; j < 4; ++j) vg[k].f[j] = __half2float(__float2half_rn(vg[k].f[j]));
          st4(g[k], vg[k]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) sgd_one(vp[k].f[j], vg[k].f[j], vm[k].f[j], a);
        st4(p[k], vp[k]);
        if (a.use_momentum) st4(m[k], vm[k]);
      } else {
        for (int j = 0; j < left[k]; ++j) {
          float pv = p[k][j], gv = g[k][j], mv = a.use_momentum ? m[k][j] : 0.f;
          if (ROUND) g[k][j] = gv = __half2float(__float2half_rn(gv));
          sgd_one(pv, gv, mv, a);
          p[k][j] = pv;
          if (a.use_momentum) m[k][j] = mv;
        }
      }
    }
  }
}

// kRoundF16: the tensors are rounded to fp16 and widened again where they are
// (what packing, a one-rank all-reduce and unpacking do to them).
enum PackMode { kPackF32 = 0, kPackF32ToF16 = 1, kUnpackF32 = 2, kUnpackF16ToF32 = 3, kRoundF16 = 4 };

// ANY: as in sgd_multi_kernel.
template <int MODE, int N, bool ANY>
__global__ void __launch_bounds__(kBlock)
pack_multi_kernel(const __grid_constant__ Table<N> t, const __grid_constant__ Offsets<N> o,
                  void* flat, float scale, int use_scale) {
  dependency_wait();
  release_dependents();
  const int k = find_tensor(t, blockIdx.x);
  const size_t n = t.n[k];
  const size_t i = static_cast<size_t>(blockIdx.x - t.first_tile[k]) * kTile + 4 * threadIdx.x;
  if (i >= n) return;
  float* tensor = static_cast<float*>(t.a[k]);
  const bool full = i + 4 <= n;
  auto load = [](const float* from) {
    if (ANY) return ld4(from);
    Vec4f v;
    v.u = ld128(from);
    return v;
  };
  auto store = [](float* to, const Vec4f& v) {
    if (ANY) st4(to, v);
    else st128(to, v.u);
  };
  if (MODE == kRoundF16) {
    if (full) {
      Vec4f v = load(tensor + i);
#pragma unroll
      for (int j = 0; j < 4; ++j) v.f[j] = __half2float(__float2half_rn(v.f[j]));
      store(tensor + i, v);
    } else {
      for (size_t j = 0; j < 4 && i + j < n; ++j) tensor[i + j] = __half2float(__float2half_rn(tensor[i + j]));
    }
    return;
  }
  const size_t fo = o.off[k] + i;
  if (MODE == kPackF32 || MODE == kUnpackF32) {
    float* fl = static_cast<float*>(flat) + fo;
    if (MODE == kPackF32) {
      if (full) store(fl, load(tensor + i));
      else for (size_t j = 0; j < 4 && i + j < n; ++j) fl[j] = tensor[i + j];
    } else {
      if (full) {
        Vec4f v = load(fl);
        if (use_scale) {
#pragma unroll
          for (int j = 0; j < 4; ++j) v.f[j] = v.f[j] * scale;
        }
        store(tensor + i, v);
      } else {
        for (size_t j = 0; j < 4 && i + j < n; ++j)
          tensor[i + j] = use_scale ? fl[j] * scale : fl[j];
      }
    }
  } else {
    __half* fl = static_cast<__half*>(flat) + fo;
    const bool vec = full && (reinterpret_cast<uintptr_t>(fl) & 7u) == 0;
    if (MODE == kPackF32ToF16) {
      if (vec) {
        const Vec4f v = load(tensor + i);
        union { uint2 u; __half h[4]; } h;
#pragma unroll
        for (int j = 0; j < 4; ++j) h.h[j] = __float2half_rn(v.f[j]);
        *reinterpret_cast<uint2*>(fl) = h.u;
      } else {
        for (size_t j = 0; j < 4 && i + j < n; ++j) fl[j] = __float2half_rn(tensor[i + j]);
      }
    } else {
      if (vec) {
        union { uint2 u; __half h[4]; } h;
        h.u = *reinterpret_cast<const uint2*>(fl);
        Vec4f v;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float f = __half2float(h.h[j]);
          v.f[j] = use_scale ? f * scale : f;
        }
        store(tensor + i, v);
      } else {
        for (size_t j = 0; j < 4 && i + j < n; ++j) {
          const float f = __half2float(fl[j]);
          tensor[i + j] = use_scale ? f * scale : f;
        }
      }
    }
  }
}

// Fills a table with tensors [first, first+count) and returns the tile count.
template <int N>
unsigned fill_table(Table<N>& t, Offsets<N>* o, void* const* a, void* const* b, void* const* c,
                    const size_t* sizes, size_t first, int count, size_t flat_off0) {
  t.count = count;
  unsigned tiles = 0;
  size_t off = flat_off0;
  for (int k = 0; k < count; ++k) {
    t.first_tile[k] = tiles;
    t.n[k] = sizes[first + k];
    t.a[k] = a[first + k];
    t.b[k] = b ? b[first + k] : nullptr;
    t.c[k] = c ? c[first + k] : nullptr;
    if (o) o->off[k] = off;
    off += sizes[first + k];
    tiles += static_cast<unsigned>(ceil_div(sizes[first + k], kTile));
  }
  t.first_tile[count] = tiles;
  return tiles;
}

template <int N>
int pack_list(int mode, void* const* tensors, const size_t* sizes, size_t count, void* flat,
              size_t flat_offset, float scale, int use_scale, void* stream) {
  if (count == 0) return SGB_OK;
  if (!tensors || !sizes || (!flat && mode != kRoundF16)) return SGB_ERR_NULL;
  cudaStream_t s = as_stream(stream);
  size_t off = flat_offset;
  for (size_t first = 0; first < count;) {
    // take as many tensors as fit the table, skipping empty ones
    Table<N> t;
    Offsets<N> o;
    void* ptrs[N];
    size_t ns[N];
    int cnt = 0;
    size_t chunk_off = off;
    unsigned long long tiles64 = 0;
    while (first < count && cnt < N) {
      const size_t n = sizes[first];
      if (n && !tensors[first]) return SGB_ERR_NULL;
      const unsigned long long tl = ceil_div(n, kTile);
      if (tiles64 + tl > 0x7fffffffull) {
        if (cnt == 0) return SGB_ERR_SIZE;
        break;
      }
      if (n) {
        // empty tensors keep their place in the flat buffer (0 elements)
        ptrs[cnt] = tensors[first];
        ns[cnt] = n;
        if (cnt == 0) chunk_off = off;
        ++cnt;
        tiles64 += tl;
      }
      off += n;
      ++first;
      if (n == 0) continue;
    }
    if (cnt == 0) continue;
    // offsets inside the chunk are contiguous because empty tensors add 0
    const unsigned tiles = fill_table<N>(t, &o, ptrs, nullptr, nullptr, ns, 0, cnt, chunk_off);
    bool any = mode != kRoundF16 && !aligned16(flat);
    for (int k = 0; k < cnt; ++k) any = any || !aligned16(ptrs[k]) || (mode != kRoundF16 && (o.off[k] & 3u));
    auto pick = [&](auto off) {
      constexpr bool kAny = decltype(off)::value;
      return mode == kPackF32        ? pack_multi_kernel<kPackF32, N, kAny>
             : mode == kPackF32ToF16 ? pack_multi_kernel<kPackF32ToF16, N, kAny>
             : mode == kUnpackF32    ? pack_multi_kernel<kUnpackF32, N, kAny>
             : mode == kRoundF16     ? pack_multi_kernel<kRoundF16, N, kAny>
                                     : pack_multi_kernel<kUnpackF16ToF32, N, kAny>;
    };
    auto kernel = any ? pick(std::true_type{}) : pick(std::false_type{});
    const int st = launch_ex(kernel, dim3(tiles), dim3(kBlock), 0, s, 0, true, t, o, flat, scale, use_scale);
    if (st != SGB_OK) return st;
  }
  return launch_status();
}

int pack_common(int mode, void* const* tensors, const size_t* sizes, size_t count, void* flat,
                size_t flat_offset, float scale, int use_scale, void* stream) {
  return count <= kSmallTable
             ? pack_list<kSmallTable>(mode, tensors, sizes, count, flat, flat_offset, scale, use_scale, stream)
             : pack_list<kLargeTable>(mode, tensors, sizes, count, flat, flat_offset, scale, use_scale, stream);
}

// One launch for as many tensors as the table holds.
template <int N, bool ROUND>
int sgd_list(void* const* params, void* const* grads, void* const* moments, const size_t* sizes, size_t count,
             const SgdArgs& a, bool beside, cudaStream_t s) {
  const bool use_m = a.use_momentum;
  for (size_t first = 0; first < count;) {
    Table<N> t;
    void *pa[N], *pb[N], *pc[N];
    size_t ns[N];
    int cnt = 0;
    bool any = false;
    unsigned long long tiles64 = 0;
    while (first < count && cnt < N) {
      const size_t n = sizes[first];
      if (n) {
        if (!params[first] || !grads[first] || (use_m && !moments[first])) return SGB_ERR_NULL;
        const unsigned long long tl = ceil_div(n, kTile);
        if (tiles64 + tl > 0x7fffffffull) {
          if (cnt == 0) return SGB_ERR_SIZE;
          break;
        }
        pa[cnt] = params[first];
        pb[cnt] = grads[first];
        pc[cnt] = use_m ? moments[first] : nullptr;
        any = any || !aligned16(pa[cnt]) || !aligned16(pb[cnt]) || !aligned16(pc[cnt]);
        ns[cnt] = n;
        ++cnt;
        tiles64 += tl;
      }
      ++first;
    }
    if (cnt == 0) continue;
    const unsigned tiles = fill_table<N>(t, nullptr, pa, pb, pc, ns, 0, cnt, 0);
    const unsigned few = static_cast<unsigned>(sm_count());
    const int st = launch_ex(beside ? sgd_beside_kernel<N, ROUND>
                             : any  ? sgd_multi_kernel<N, ROUND, true>
                                    : sgd_multi_kernel<N, ROUND, false>,
                             dim3(beside && few < tiles ? few : tiles), dim3(kBlock), 0, s, 0, true, t, a);
    if (st != SGB_OK) return st;
  }
  return launch_status();
}

template <bool ROUND>
int sgd_any(void* const* params, void* const* grads, void* const* moments, const size_t* sizes, size_t count,
            const SgdArgs& a, bool beside, cudaStream_t s) {
  return count <= kSmallTable ? sgd_list<kSmallTable, ROUND>(params, grads, moments, sizes, count, a, beside, s)
                              : sgd_list<kLargeTable, ROUND>(params, grads, moments, sizes, count, a, beside, s);
}

}  // namespace

int sgd_round_f16_multi(void* const* params, void* const* grads, void* const* moments, const size_t* sizes, size_t count,
                        const SgdArgs& a, cudaStream_t s) {
  return sgd_any<true>(params, grads, moments, sizes, count, a, false, s);
}

int round_f16_multi(void* const* tensors, const size_t* sizes, size_t count, cudaStream_t s) {
  return pack_common(kRoundF16, tensors, sizes, count, nullptr, 0, 1.f, 0, s);
}

}  // namespace sgb

using namespace sgb;

extern "C" {

int sgb_sgd_update_multi_f32(void* const* params, void* const* grads, void* const* moments,
                             const size_t* sizes, size_t count, float lr, float momentum,
                             float dampening, float weight_decay, int nesterov, float grad_scale,
                             void* stream) {
  if (count == 0) return SGB_OK;
  if (!params || !grads || !sizes) return SGB_ERR_NULL;
  SgdArgs a;
  const int st = sgd_args(&a, moments, lr, momentum, dampening, weight_decay, nesterov, grad_scale);
  if (st != SGB_OK) return st;
  return sgd_any<false>(params, grads, moments, sizes, count, a, false, as_stream(stream));
}

int sgb_sgd_update_beside_f32(void* const* params, void* const* grads, void* const* moments, const size_t* sizes,
                              size_t count, float lr, float momentum, float dampening, float weight_decay, int nesterov,
                              float grad_scale, int round_f16, void* stream) {
  if (count == 0) return SGB_OK;
  if (!params || !grads || !sizes) return SGB_ERR_NULL;
  SgdArgs a;
  const int st = sgd_args(&a, moments, lr, momentum, dampening, weight_decay, nesterov, grad_scale);
  if (st != SGB_OK) return st;
  return round_f16 ? sgd_any<true>(params, grads, moments, sizes, count, a, true, as_stream(stream))
                   : sgd_any<false>(params, grads, moments, sizes, count, a, true, as_stream(stream));
}

int sgb_sgd_update_f32(float* param, const float* grad, float* moment, size_t n, float lr,
                       float momentum, float dampening, float weight_decay, int nesterov,
                       float grad_scale, void* stream) {
  void* p[1] = {param};
  void* g[1] = {const_cast<float*>(grad)};
  void* m[1] = {moment};
  size_t ns[1] = {n};
  return sgb_sgd_update_multi_f32(p, g, m, ns, 1, lr, momentum, dampening, weight_decay,
                                  nesterov, grad_scale, stream);
}

int sgb_pack_f32(void* const* tensors, const size_t* sizes, size_t count, float* flat,
                 size_t flat_offset, void* stream) {
  return pack_common(kPackF32, tensors, sizes, count, flat, flat_offset, 1.f, 0, stream);
}
int sgb_pack_f32_to_f16(void* const* tensors, const size_t* sizes, size_t count, void* flat_f16,
                        size_t flat_offset, void* stream) {
  return pack_common(kPackF32ToF16, tensors, sizes, count, flat_f16, flat_offset, 1.f, 0, stream);
}
int sgb_unpack_f32(const float* flat, size_t flat_offset, void* const* tensors,
                   const size_t* sizes, size_t count, float scale, void* stream) {
  return pack_common(kUnpackF32, tensors, sizes, count, const_cast<float*>(flat), flat_offset,
                     scale, scale != 1.0f, stream);
}
int sgb_unpack_f16_to_f32(const void* flat_f16, size_t flat_offset, void* const* tensors,
                          const size_t* sizes, size_t count, float scale, void* stream) {
  return pack_common(kUnpackF16ToF32, tensors, sizes, count, const_cast<void*>(flat_f16),
                     flat_offset, scale, scale != 1.0f, stream);
}

}  // extern "C"
