// Batch norm in two visits to the data inside one kernel: what the backward and
// the forward form share.
//
// The grid is one CTA per item (a run of units of one channel) and `delay` more.
// CTA i forms the sums of item i and publishes them, then finishes item
// i - delay: the sums of that item's channel have been published by then, and its
// operands come from L2, where the first visit asked for them to be kept.  So HBM
// sees every operand once, as if a channel were held on the chip, but nothing is
// staged: thousands of small CTAs overlap loads, sums and stores, and every SM slot is
// used whatever the shape.  A channel of very many items puts its visits too far apart
// (revisit_pays and fwd_revisit_pays have the lines).
//
// What bounds it: HBM and the latency of a CTA's life (load, reduce, load again,
// store), which the number of CTAs in flight has to cover.  A loop of persistent
// CTAs, one warp fewer (its waits then delayed the sums that others wait for),
// bulk copies to shared memory and acquire / release accesses to the exchange
// were all slower by 10 to 40 %.
//
// The exchange is in the caller's workspace, whose contents are unknown when the
// kernel starts and which serves one launch at a time.  An item's two sums and the
// launch's tag, a 64-bit number that no other launch of the process has, travel in
// one 16-byte access: an entry counts once it shows the tag.  A graph replays a launch
// with the same tag, so the last reader of a channel takes the tags away again.
//
// Progress: a CTA waits for CTAs with lower numbers only, and for a part of them
// that waits for nobody.  CTAs are started in order, so however few are resident,
// the lowest one can always go on.  (CUDA does not promise that order.  As the CTAs
// that are waited for lie a full wave behind, more than a wave of disorder would be
// needed for all resident CTAs to wait for ones that have no place.)  The waits are
// bounded all the same: a CTA whose wait runs out sets the sticky fault word and names
// the launch as stopped; the launch's other CTAs see that while they poll, and none
// of them finishes its item.
#pragma once
#include "bn_common.cuh"

namespace sgb {

// A number that no other launch of this process has, and that data do not show by chance.
unsigned long long revisit_tag();
struct RevisitState {                  // one per device
  unsigned faults;                     // sticky fault word
  unsigned long long stopped;          // tag of the last launch whose wait ran out
};
// Its address on the current device; null on an error.
RevisitState* revisit_state(int* status);
int revisit_faults(unsigned* flags);

// Backward: planes of any size from eight floats on, all pointers 16-byte aligned.
// mask: 0 none, 1 ReLU input as floats, 2 ReLU bit record.  SGB_ERR_WORKSPACE and
// nothing done where the workspace is too small or the problem too large.
int bn_revisit_backward(int mask, const float* x, const float* dy, const float* relu, const float* scale,
                        const float* mean, const float* invstd, float* dx, float* dscale, float* dbias, int N, int C,
                        int HW, void* ws, size_t ws_bytes, cudaStream_t s);
size_t bn_revisit_workspace_bytes(int N, int C, int HW);    // 0: too large

namespace {

struct __align__(16) RevisitEntry {
  float a, b;
  unsigned long long tag;
};

// Units per thread, most summing threads per CTA (one warp more fetches the
// channel's sums) and resident CTAs per SM.  The summing CTAs lead the finishing
// ones by that many waves: with less the latter wait, with more what they come
// back to has left the part of L2 that is fast (about 30 MB).
struct RevisitShape {
  int units, threads, per_sm;
};
struct RevisitPlan {
  int parts, per;                      // items per channel, units per item
  int items, delay, threads;
  size_t readers, bytes;               // of workspace: where the counters lie, how much
};
// False: too many items for a launch, or elements for 32-bit offsets.
inline bool revisit_plan(const RevisitShape& shape, long long units, int upp, int channels, RevisitPlan* p) {
  const long long target = static_cast<long long>(shape.units) * shape.threads;
  const long long least = (units + target - 1) / target, per = (units + least - 1) / least;
  const long long parts = (units + per - 1) / per, items = parts * channels;
  const long long delay = parts + static_cast<long long>(shape.per_sm) * sm_count();
  if (items + delay > 0x7fffffffLL || units > 0x7fffffffLL || units * channels > 0x1fffffffLL || upp < 1) return false;
  p->parts = static_cast<int>(parts);
  p->per = static_cast<int>(per);
  p->items = static_cast<int>(items);
  p->delay = static_cast<int>(delay);
  p->threads = static_cast<int>((per + 32 * shape.units - 1) / (32 * shape.units)) * 32;
  p->readers = sizeof(RevisitEntry) * static_cast<size_t>(items + channels);
  p->bytes = p->readers + 4 * static_cast<size_t>(channels);
  return true;
}

struct Revisit {
  RevisitEntry* entries;               // one per item, then one per channel
  unsigned* readers;                   // per channel: items finished, ever
  unsigned long long tag;
  RevisitState* state;
  FastDiv parts;
  unsigned per, total;                 // units per item, per channel
  int items, delay;
  FastDiv upp;                         // units per plane
  unsigned hw, plane_stride;           // plane_stride: elements per sample
};
inline Revisit revisit_args(const RevisitPlan& p, long long units, int upp, int C, int HW, void* ws,
                            RevisitState* state) {
  char* const base = static_cast<char*>(ws);
  return Revisit{reinterpret_cast<RevisitEntry*>(base), reinterpret_cast<unsigned*>(base + p.readers), revisit_tag(),
                 state, FastDiv(static_cast<unsigned>(p.parts)), static_cast<unsigned>(p.per),
                 static_cast<unsigned>(units), p.items, p.delay, FastDiv(static_cast<unsigned>(upp)),
                 static_cast<unsigned>(HW), static_cast<unsigned>(C) * static_cast<unsigned>(HW)};
}

// Loads of the first visit ask L2 to keep the lines, those of the second give them
// up: at once, or (what is wanted again, by the backward pass) like any other line.
// (32x256x56x56 with ReLU, between other kernels: 77 us; 90 with ordinary loads in
// the second visit.)
__device__ __forceinline__ unsigned long long keep_policy() {
  unsigned long long p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ unsigned long long drop_policy() {
  unsigned long long p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ unsigned long long ease_policy() {
  unsigned long long p;
  asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint4 ld128_hint(const void* p, unsigned long long policy) {
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p), "l"(policy));
  return v;
}

// One access each: the value and the tag cannot be seen apart.
__device__ __forceinline__ void put_entry(RevisitEntry* p, float a, float b, unsigned long long tag) {
  const unsigned long long v = static_cast<unsigned long long>(__float_as_uint(b)) << 32 | __float_as_uint(a);
  asm volatile("{\n.reg .b128 e;\nmov.b128 e, {%1, %2};\nst.relaxed.gpu.global.b128 [%0], e;\n}" ::"l"(p), "l"(v),
               "l"(tag)
               : "memory");
}
__device__ __forceinline__ bool get_entry(const RevisitEntry* p, unsigned long long tag, float& a, float& b) {
  unsigned long long v, got;
  asm volatile("{\n.reg .b128 e;\nld.relaxed.gpu.global.b128 e, [%2];\nmov.b128 {%0, %1}, e;\n}"
               : "=l"(v), "=l"(got)
               : "l"(p)
               : "memory");
  a = __uint_as_float(static_cast<unsigned>(v));
  b = __uint_as_float(static_cast<unsigned>(v >> 32));
  return got == tag;
}

// The readers of a channel are counted from whatever its counter holds, which the CTA of
// the channel's first item passes on in an entry of its own: nobody counts before having
// seen that entry, so it is what earlier launches left, and no store to the counter has to
// be ordered with the counting.  (With a counter set to zero by the first item, and fences
// on both sides, calls took 0.7 to 2 us longer: 32x256x56x56 53.3 -> 51.2, forward 42.2 ->
// 40.5; 32x1024x14x14 18.6 -> 16.8; 12x200x50x50 16.3 -> 15.4.)  By the warp that fetches
// sums, first of all.
__device__ __forceinline__ void revisit_open(const Revisit& r, unsigned item) {
  const unsigned c = r.parts.quot(item);
  if (item != c * r.parts.d || (threadIdx.x & 31) != 0) return;
  // a graph's launches share a tag: an earlier one's stop is not this one's
  if (item == 0 && *static_cast<volatile unsigned long long*>(&r.state->stopped) == r.tag) r.state->stopped = 0;
  put_entry(r.entries + r.items + c, __uint_as_float(*static_cast<volatile unsigned*>(r.readers + c)), 0.f, r.tag);
}

constexpr unsigned kMostPolls = 1u << 20;   // of half a microsecond and more

// One warp: calls fold(k, a, b) with the channel's entries k = lane, lane + 32, ...;
// all entries of a batch are asked for at once.  `base` (in lane 0): what the channel's
// counter held.  False (in all lanes): the launch has been stopped.
template <typename F>
__device__ __forceinline__ bool revisit_gather(const Revisit& r, unsigned c, unsigned& base, F fold) {
  constexpr int kBatch = 4;
  const unsigned parts = r.parts.d;
  const RevisitEntry* const e = r.entries + static_cast<size_t>(c) * parts;
  const RevisitEntry* const counted = r.entries + r.items + c;
  float first = 0.f, none;
  bool got = true;
  for (unsigned k0 = threadIdx.x & 31; got && k0 < parts; k0 += 32 * kBatch) {
    float a[kBatch], b[kBatch];
    unsigned missing = 0;
#pragma unroll
    for (int q = 0; q < kBatch; ++q)
      if (k0 + 32 * q < parts && !get_entry(e + k0 + 32 * q, r.tag, a[q], b[q])) missing |= 1u << q;
    if (k0 == 0 && !get_entry(counted, r.tag, first, none)) missing |= 1u << kBatch;
    for (unsigned n = 1; missing && got; ++n) {
#pragma unroll
      for (int q = 0; q < kBatch; ++q)
        if (missing >> q & 1u && get_entry(e + k0 + 32 * q, r.tag, a[q], b[q])) missing &= ~(1u << q);
      if (missing >> kBatch && get_entry(counted, r.tag, first, none)) missing &= (1u << kBatch) - 1;
      if (n % 256 == 0 && missing) {
        got = *static_cast<volatile unsigned long long*>(&r.state->stopped) != r.tag;
        if (got && n >= kMostPolls) {
          r.state->stopped = r.tag;
          atomicOr(&r.state->faults, 1u);
          got = false;
        }
      }
    }
    if (!got) break;
#pragma unroll
    for (int q = 0; q < kBatch; ++q)
      if (k0 + 32 * q < parts) fold(k0 + 32 * q, a[q], b[q]);
  }
  base = __float_as_uint(first);
  return __all_sync(0xffffffffu, got);
}
// The same warp, once it has the sums: the last reader takes the channel's tags away.
// (No fence: a reader counts only once all its lanes have seen the tags.)
__device__ __forceinline__ void revisit_leave(const Revisit& r, unsigned c, unsigned base) {
  const unsigned parts = r.parts.d, lane = threadIdx.x & 31;
  unsigned before = 0;
  if (lane == 0) before = atomicAdd(r.readers + c, 1u) - base;
  before = __shfl_sync(0xffffffffu, before, 0);
  if (before + 1 != parts) return;
  for (unsigned k = lane; k < parts; k += 32) r.entries[static_cast<size_t>(c) * parts + k].tag = 0;
  if (lane == 0) r.entries[r.items + c].tag = 0;
}

// This thread's units of an item.  VEC: whole vectors of a plane; else the aligned
// vectors that touch it (RaggedUnit).  valid == 0: no unit.
template <bool VEC, int NV>
struct RevisitUnits {
  unsigned c, part;
  unsigned off[NV], valid[NV];
  __device__ __forceinline__ RevisitUnits(const Revisit& r, unsigned item, unsigned threads) {
    c = r.parts.quot(item);
    part = item - c * r.parts.d;
    const unsigned u1 = min((part + 1) * r.per, r.total);
    unsigned u = part * r.per + threadIdx.x;
#pragma unroll
    for (int k = 0; k < NV; ++k, u += threads) {
      const unsigned n = r.upp.quot(u), q = u - n * r.upp.d, plane = n * r.plane_stride + c * r.hw;
      if (VEC) {
        off[k] = plane + q * 4;
        valid[k] = u < u1 ? 15u : 0u;
      } else {
        const RaggedUnit x(plane, static_cast<int>(q), static_cast<int>(r.hw));
        off[k] = static_cast<unsigned>(x.off);
        valid[k] = u < u1 ? x.valid : 0u;
      }
    }
  }
  // The vector of unit k (which is there); behind the tensor's last element: 0.
  __device__ __forceinline__ Vec4f load(const float* p, int k, unsigned numel, unsigned long long policy) const {
    Vec4f v;
    if (VEC || off[k] + 4 <= numel) {
      v.u = ld128_hint(p + off[k], policy);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) v.f[j] = off[k] + j < numel ? p[off[k] + j] : 0.0f;
    }
    return v;
  }
  __device__ __forceinline__ void store(float* p, int k, const Vec4f& v) const {
    if (VEC || valid[k] == 15u) {
      st128_stream(p + off[k], v.u);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (valid[k] >> j & 1u) p[off[k] + j] = v.f[j];
    }
  }
};

// Named barriers: 1 among the summing warps, 2 with the warp that fetches the sums.
__device__ __forceinline__ void revisit_sync(int id, unsigned threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void revisit_arrive(int id, unsigned threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

}  // namespace
}  // namespace sgb
