// Gradient sparsification kernels of the communicator:
//   * threshold selection with residual correction and ORDER-PRESERVING
//     compaction into a [1-based index | value] payload;
//   * top-K selection by radix select on a 32-bit key (no sort), ties broken
//     by lower index, with the same compaction;
//   * the dense sum of the received payloads.
//
// Each selection is ONE cooperative kernel.  The elements are split into chunks
// of eight runs (one per warp) of one or four 512-element tiles; what a warp
// selects in its run goes to a private list in the workspace in ascending index
// order, so that after one device-wide barrier (all counts are known) the lists
// are copied to their final place: no scan kernel, no second read of the
// gradient.  A CTA draws its next chunk from a ticket counter while it works on
// the current one: with a fixed share per CTA the slowest SMs finished 40 us
// after the others at 1e8 elements (SMs do not get equal bandwidth).  Inside a
// chunk warps do not wait for one another.  The device-wide barriers are
// cooperative-launch grid barriers (all CTAs of the grid are co-resident by
// construction).  A list that fills up (a run in which more than about one
// element in six is selected) costs no correctness: the warp notes how many
// tiles were listed and reads the others again.
//
// What bounds them: HBM.  g and the residual are read once, the residual is
// written once (12 B/element); the top-K form reads the residual once more
// (4 B/element) after the first radix digit is decided, unless a sample has
// bounded the k-th key before (large gradients).  All index arithmetic
// that reaches the payload is 1-based int32, the reference's wire format.
#include <cooperative_groups.h>

#include <atomic>
#include <cmath>
#include <vector>

#include <type_traits>

#include "sgd.cuh"
#include "sparse.cuh"

namespace cg = cooperative_groups;

namespace sgb {
namespace {

constexpr int kBlock = 256;
constexpr int kWarps = kBlock / 32;
constexpr int kRounds = 4;                             // float4 vectors per lane and tile
constexpr int kTile = 32 * kRounds * 4;                // 512 elements, a warp's unit of work
constexpr int kBins1 = 3072, kBins23 = 1024;           // 12 + 10 + 10 key bits; no key is above 2^31, bin 2048
// 4 CTAs per SM: 128 KB of loads in flight per SM already saturate HBM, and a
// cooperative grid that does not need every slot can start beside the kernels
// of another stream.
constexpr int kCtasPerSm = 4;
constexpr int kMaxGrid = 1024;

struct Counters {        // zeroed before a call that uses them
  unsigned ticket[4];    // chunks drawn so far, one counter per pass
  unsigned max_key;      // largest key of pass 0
  unsigned arrived;      // at the barriers of a part of the grid
  unsigned pad[2];
  unsigned hist0[kBins1], hist1[kBins23], hist2[kBins23], sample[kBins1];
};

__host__ __device__ inline size_t align256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }
inline size_t tiles_of(size_t n) { return ceil_div(n, kTile); }
inline size_t max_grid() {
  const size_t g = static_cast<size_t>(sm_count()) * kCtasPerSm;
  return g < kMaxGrid ? g : kMaxGrid;
}
// How the tiles are cut.  One tile per warp and chunk until every CTA has four
// chunks, then four: fewer counts to add up, less to draw.
struct Work {
  unsigned chunks, grid;
  unsigned run;          // tiles per warp and chunk
  unsigned capacity;     // list entries per warp and chunk
  bool dynamic;          // chunks are drawn from the ticket counter
};
inline Work work_for(size_t n, size_t g = max_grid()) {
  const size_t tiles = tiles_of(n);
  Work w;
  w.run = tiles > 4 * kWarps * g ? 4 : 1;
  w.capacity = w.run == 4 ? 352 : 128;
  w.chunks = static_cast<unsigned>(ceil_div(tiles, kWarps * w.run));
  w.grid = static_cast<unsigned>(w.chunks < g ? w.chunks : g);
  w.dynamic = w.chunks > 2 * w.grid;
  return w;
}

struct Workspace {
  Counters* counters;
  unsigned* chunk_a;     // per chunk: selected, or keys above the threshold
  unsigned* chunk_b;     //            keys equal to the threshold
  unsigned* run_meta;    // per warp and chunk, see pack_meta
  unsigned* run_counts;  // per warp and chunk: keys above / equal to the threshold (16 bits each)
  int* list_idx;         // chunks * kWarps segments of `capacity` entries
  float* list_val;
};
inline size_t lists_bytes(const Work& w) {
  const size_t runs = static_cast<size_t>(w.chunks) * kWarps;
  return 2 * align256(w.chunks * sizeof(unsigned)) + 2 * align256(runs * sizeof(unsigned)) +
         2 * align256(runs * w.capacity * sizeof(int));
}
inline size_t workspace_bytes_exact(size_t n) {
  return align256(sizeof(Counters)) + lists_bytes(work_for(n));
}
// Monotonic in n (a workspace for n serves any smaller call): where the cut
// changes from one tile to four, the shorter runs need the larger lists.
inline size_t workspace_bytes(size_t n) {
  const size_t turn = 4 * kWarps * max_grid() * static_cast<size_t>(kTile);
  size_t b = workspace_bytes_exact(n);
  if (n > turn && workspace_bytes_exact(turn) > b) b = workspace_bytes_exact(turn);
  return b;
}
// The counters at `counters`, the rest from `lists` on.
__host__ __device__ inline Workspace carve_at(char* counters, char* lists, const Work& k) {
  char* p = lists;
  const size_t runs = static_cast<size_t>(k.chunks) * kWarps;
  Workspace w;
  w.counters = reinterpret_cast<Counters*>(counters);
  w.chunk_a = reinterpret_cast<unsigned*>(p); p += align256(k.chunks * sizeof(unsigned));
  w.chunk_b = reinterpret_cast<unsigned*>(p); p += align256(k.chunks * sizeof(unsigned));
  w.run_meta = reinterpret_cast<unsigned*>(p); p += align256(runs * sizeof(unsigned));
  w.run_counts = reinterpret_cast<unsigned*>(p); p += align256(runs * sizeof(unsigned));
  w.list_idx = reinterpret_cast<int*>(p); p += align256(runs * k.capacity * sizeof(int));
  w.list_val = reinterpret_cast<float*>(p);
  return w;
}
inline Workspace carve(void* ws, const Work& k) {
  char* p = static_cast<char*>(ws);
  return carve_at(p, p + align256(sizeof(Counters)), k);
}
// ------------------------------------------------------------- tile helpers
// Element order inside a tile: vector v = r * 32 + lane (round r), elements
// 4v .. 4v+3.  Loads are fully coalesced; ranks below follow this order, which
// is ascending element index.
__device__ __forceinline__ size_t vec_at(size_t tile, int r) {
  return tile * kTile + (r * 32 + (threadIdx.x & 31)) * 4;
}

// The values of elements i .. i+3; out-of-range lanes get 0.  `vec` (host-checked
// 16-byte alignment of every operand) allows 128-bit accesses.
__device__ __forceinline__ void load4(const float* p, size_t i, size_t n, bool vec, float (&s)[4]) {
  if (vec && i + 4 <= n) {
    const float4 a = *reinterpret_cast<const float4*>(p + i);
    s[0] = a.x; s[1] = a.y; s[2] = a.z; s[3] = a.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] = i + j < n ? p[i + j] : 0.0f;
  }
}
__device__ __forceinline__ void store4(float* p, size_t i, size_t n, bool vec, const float (&v)[4]) {
  if (vec && i + 4 <= n) {
    *reinterpret_cast<float4*>(p + i) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (i + j < n) p[i + j] = v[j];
  }
}
// s = g + acc for one tile, all loads issued before the first use.
__device__ __forceinline__ void load_tile(const float* g, const float* acc, size_t tile, size_t n, bool vec,
                                          float (&s)[kRounds][4]) {
  float b[kRounds][4];
#pragma unroll
  for (int r = 0; r < kRounds; ++r) load4(g, vec_at(tile, r), n, vec, s[r]);
  if (!acc) return;
#pragma unroll
  for (int r = 0; r < kRounds; ++r) load4(acc, vec_at(tile, r), n, vec, b[r]);
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[r][j] += b[r][j];
}

// The gradient as a list of tensors that need not lie back to back: element i
// of the bucket is ptr[k][i - off[k]] for the k with off[k] <= i < off[k + 1].
// Selecting straight from the list saves the copy into one buffer (8 B/element
// and a launch per bucket).
constexpr int kPieces = 256;
struct Pieces {
  int count;
  unsigned off[kPieces + 1];
  const float* ptr[kPieces];
};
// A part of such a list that lies elsewhere in the kernel's arguments.
struct PieceView {
  int count;
  const unsigned* off;
  const float* const* ptr;
};
struct NoPieces {};
// Where a tile lies in the lists: searched for once per run of tiles, then
// walked.  (A search is up to thirteen dependent loads ahead of the tile's own.)
struct Cursor {
  int piece = 0, bucket = 0;
};
__device__ __forceinline__ void seek(const NoPieces&, Cursor&, size_t) {}
__device__ __forceinline__ void advance(const NoPieces&, Cursor&, size_t) {}
template <typename P>
__device__ __forceinline__ void seek_piece(const P& p, Cursor& c, size_t tile) {
  const unsigned e0 = static_cast<unsigned>(tile * kTile);
  int lo = 0, hi = p.count - 1;
  while (lo < hi) {                                    // the same in all lanes
    const int mid = (lo + hi + 1) >> 1;
    if (p.off[mid] <= e0) lo = mid; else hi = mid - 1;
  }
  c.piece = lo;
}
template <typename P>
__device__ __forceinline__ void advance_piece(const P& p, Cursor& c, size_t tile) {
  const unsigned e0 = static_cast<unsigned>(tile * kTile);
  while (c.piece + 1 < p.count && p.off[c.piece + 1] <= e0) ++c.piece;
}
__device__ __forceinline__ void seek(const Pieces& p, Cursor& c, size_t tile) { seek_piece(p, c, tile); }
__device__ __forceinline__ void advance(const Pieces& p, Cursor& c, size_t tile) { advance_piece(p, c, tile); }
__device__ __forceinline__ void seek(const PieceView& p, Cursor& c, size_t tile) { seek_piece(p, c, tile); }
__device__ __forceinline__ void advance(const PieceView& p, Cursor& c, size_t tile) { advance_piece(p, c, tile); }
__device__ __forceinline__ void load_tile(const NoPieces&, const Cursor&, const float* g, const float* acc, size_t tile,
                                          size_t n, bool vec, float (&s)[kRounds][4]) {
  load_tile(g, acc, tile, n, vec, s);
}
// s = gradient + acc for one tile.  A tile inside one tensor is loaded as above,
// one that crosses an end element by element.  acc is there and aligned.
template <typename P>
__device__ __forceinline__ void load_pieces(const P& p, const Cursor& c, const float* acc, size_t tile, size_t n,
                                            float (&s)[kRounds][4]) {
  const unsigned e0 = static_cast<unsigned>(tile * kTile), e1 = e0 + kTile;
  const int lo = c.piece;
  const float* base = p.ptr[lo] - p.off[lo];           // only used where it points into the tensor
  if (e1 <= p.off[lo + 1] && (reinterpret_cast<uintptr_t>(base + e0) & 15u) == 0) {
    load_tile(base, acc, tile, n, true, s);
    return;
  }
  if (e1 <= p.off[lo + 1] && e1 <= n) {
    // inside one tensor, but not at a vector's start (a list of odd-sized tensors): single
    // loads of it, without a look at the list for each
    float b[kRounds][4];
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[r][j] = base[vec_at(tile, r) + j];
#pragma unroll
    for (int r = 0; r < kRounds; ++r) load4(acc, vec_at(tile, r), n, true, b[r]);
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[r][j] += b[r][j];
    return;
  }
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const unsigned i = static_cast<unsigned>(vec_at(tile, r));
    int k = lo;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s[r][j] = 0.0f;
      if (i + j < n) {
        while (i + j >= p.off[k + 1]) ++k;
        s[r][j] = p.ptr[k][i + j - p.off[k]] + acc[i + j];
      }
    }
  }
}

__device__ __forceinline__ void load_tile(const Pieces& p, const Cursor& c, const float*, const float* acc, size_t tile,
                                          size_t n, bool, float (&s)[kRounds][4]) {
  load_pieces(p, c, acc, tile, n, s);
}
__device__ __forceinline__ void load_tile(const PieceView& p, const Cursor& c, const float*, const float* acc, size_t tile,
                                          size_t n, bool, float (&s)[kRounds][4]) {
  load_pieces(p, c, acc, tile, n, s);
}

// Several buckets, each with its own residual, as one index space in which
// every bucket starts on a tile (the gaps are beyond its end and never selected).
constexpr int kBuckets = 32;
struct Buckets {
  int count;
  unsigned tile[kBuckets];       // first tile
  unsigned end[kBuckets];        // one past the last element
  float* acc[kBuckets];
  Pieces pieces;                 // offsets in the joint space; a bucket's last piece takes in the gap
};
__device__ __forceinline__ void seek(const Buckets& b, Cursor& c, size_t tile) {
  seek(b.pieces, c, tile);
  int lo = 0, hi = b.count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (b.tile[mid] <= tile) lo = mid; else hi = mid - 1;
  }
  c.bucket = lo;
}
__device__ __forceinline__ void advance(const Buckets& b, Cursor& c, size_t tile) {
  advance(b.pieces, c, tile);
  while (c.bucket + 1 < b.count && b.tile[c.bucket + 1] <= tile) ++c.bucket;
}
__device__ __forceinline__ void load_tile(const Buckets& b, const Cursor& c, const float* g, const float* acc,
                                          size_t tile, size_t n, bool vec, float (&s)[kRounds][4]) {
  load_tile(b.pieces, c, g, acc, tile, n, vec, s);
}
// The residual (indexed like the elements) and the end of what a tile belongs to.
struct View {
  float* acc;
  size_t n;
};
template <typename Source>
__device__ __forceinline__ View view(const Source&, const Cursor&, float* acc, size_t n) {
  return View{acc, n};
}
__device__ __forceinline__ View view(const Buckets& b, const Cursor& c, float*, size_t) {
  return View{b.acc[c.bucket] - static_cast<size_t>(b.tile[c.bucket]) * kTile, b.end[c.bucket]};
}

// Exclusive offsets, in element order, of this lane's counts inside the tile:
// `mine` holds the counts of the four rounds, one byte each (<= 4; a warp's
// total of a round is at most 128), so one scan serves all rounds.  Returns
// the tile total.
__device__ __forceinline__ unsigned tile_exclusive(unsigned mine, unsigned (&excl)[kRounds]) {
  static_assert(kRounds == 4, "one byte per round");
  const int lane = threadIdx.x & 31;
  unsigned incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  const unsigned totals = __shfl_sync(0xffffffffu, incl, 31);
  const unsigned before = incl - mine;      // bytes cannot borrow: incl >= mine in each
  unsigned base = 0;
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    excl[r] = base + ((before >> (8 * r)) & 0xffu);
    base += (totals >> (8 * r)) & 0xffu;
  }
  return base;
}
// One bit per element of a tile (bit 4r + j) -> the four counts, one byte each.
__device__ __forceinline__ unsigned round_counts(unsigned m) {
  return __popc(m & 0xfu) | __popc(m & 0xf0u) << 8 | __popc(m & 0xf00u) << 16 | __popc(m & 0xf000u) << 24;
}
// The bits of elements below n (all of them except in the last tile).
__device__ __forceinline__ unsigned in_range(size_t tile, size_t n) {
  if ((tile + 1) * kTile <= n) return 0xffffu;
  unsigned m = 0;
#pragma unroll
  for (int r = 0; r < kRounds; ++r)
#pragma unroll
    for (int j = 0; j < 4; ++j) m |= vec_at(tile, r) + j < n ? 1u << (4 * r + j) : 0u;
  return m;
}

// Writes a tile's selected elements (bit 4r + j of `m`) to list[at ...] in
// element order.  They pass through the warp's shared-memory slots so that the
// list is written in full sectors: straight from the lanes every store would
// carry one or two of them.  A tile with more than `slots` goes straight.
__device__ __forceinline__ void list_tile(const float (&s)[kRounds][4], unsigned m, const unsigned (&excl)[kRounds],
                                          unsigned total, size_t tile, int* list_idx, float* list_val, int* slot_idx,
                                          float* slot_val, unsigned slots) {
  const bool staged = total <= slots;
  int* const di = staged ? slot_idx : list_idx;
  float* const dv = staged ? slot_val : list_val;
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    unsigned pos = excl[r];
    const int i1 = static_cast<int>(vec_at(tile, r) + 1);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (m >> (4 * r + j) & 1u) {
        di[pos] = i1 + j;
        dv[pos] = s[r][j];
        ++pos;
      }
  }
  if (!staged) return;
  __syncwarp();
  for (unsigned e = threadIdx.x & 31; e < total; e += 32) {
    list_idx[e] = slot_idx[e];
    list_val[e] = slot_val[e];
  }
  __syncwarp();
}

// Sum over the CTA of one unsigned per thread (two at once); valid in every thread.
__device__ __forceinline__ uint2 cta_sum2(unsigned a, unsigned b, uint2* sm) {
  a = __reduce_add_sync(0xffffffffu, a);
  b = __reduce_add_sync(0xffffffffu, b);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = make_uint2(a, b);
  __syncthreads();
  uint2 t = make_uint2(0, 0);
#pragma unroll
  for (int k = 0; k < kWarps; ++k) {
    t.x += sm[k].x;
    t.y += sm[k].y;
  }
  return t;
}

// What one warp left behind for its run of a chunk: elements selected (<= 2048),
// list entries written (<= 352) and tiles listed (the first ones of the run).
__device__ __forceinline__ unsigned pack_meta(unsigned count, unsigned used, unsigned listed) {
  return count | used << 12 | listed << 24;
}
__device__ __forceinline__ unsigned meta_count(unsigned m) { return m & 0xfffu; }
__device__ __forceinline__ unsigned meta_used(unsigned m) { return m >> 12 & 0xfffu; }
__device__ __forceinline__ unsigned meta_listed(unsigned m) { return m >> 24; }

// This warp's tiles [lo, hi) of a chunk.
__device__ __forceinline__ void run_tiles(const Work& k, unsigned chunk, size_t n, size_t& lo, size_t& hi) {
  const size_t tiles = (n + kTile - 1) / kTile;
  lo = (static_cast<size_t>(chunk) * kWarps + (threadIdx.x >> 5)) * k.run;
  hi = lo + k.run < tiles ? lo + k.run : tiles;
  if (lo > hi) lo = hi;
}
// Calls body(chunk) in all warps of the CTA for each of its chunks, and then,
// behind a barrier, after(chunk, parity) in all warps; `parity` alternates, so
// that what the warps hand to `after` in shared memory can be double-buffered.
// Every CTA's first chunk is its own number; the counter hands out the rest.
template <bool DESCENDING, typename Body, typename After>
__device__ __forceinline__ void for_chunks(const Work& k, unsigned rank, unsigned* ticket, unsigned* sm_next, Body body,
                                           After after) {
  unsigned c = rank, parity = 0;
  while (c < k.chunks) {
    unsigned next = c + k.grid;
    if (k.dynamic && threadIdx.x == 0) next = k.grid + atomicAdd(ticket, 1u);
    const unsigned chunk = DESCENDING ? k.chunks - 1 - c : c;
    body(chunk, parity);
    if (k.dynamic && threadIdx.x == 0) sm_next[parity] = next;
    __syncthreads();
    after(chunk, parity);
    c = k.dynamic ? sm_next[parity] : next;
    parity ^= 1;
  }
  __syncthreads();
}
// After a grid barrier the chunks are walked in contiguous shares: this CTA's
// [first, last), and how much one or two counts per chunk add up to before it.
__device__ __forceinline__ void my_chunks(const Work& k, unsigned rank, unsigned& first, unsigned& last) {
  first = static_cast<unsigned>(static_cast<unsigned long long>(k.chunks) * rank / k.grid);
  last = static_cast<unsigned>(static_cast<unsigned long long>(k.chunks) * (rank + 1) / k.grid);
}
struct Before {
  unsigned before, total;
};
__device__ __forceinline__ Before counts_before(const unsigned* counts, unsigned chunks, unsigned first, uint2* sm) {
  unsigned b = 0, t = 0;
#pragma unroll 8
  for (unsigned k = threadIdx.x; k < chunks; k += kBlock) {
    const unsigned v = __ldcg(counts + k);
    t += v;
    b += k < first ? v : 0u;
  }
  const uint2 s = cta_sum2(b, t, sm);
  return Before{s.x, s.y};
}

// ------------------------------------------------------------ threshold mode
// s = g (+ acc); kept = |s| >= thr ? s : 0; sent iff kept != 0; acc = s - kept.
// BOUNDED: the payload layout is fixed, [idx(cap) | val(cap)], and only the
// first `cap` selected entries (index order) are sent; the others go back into
// the residual (without one they are lost) and their number is added to
// *dropped, so the caller knows the length of the exchange before the count.
struct ThrArgs {
  const float* g;
  float* acc;
  size_t n;
  float thr;
  Work work;
  Workspace ws;
  int* idx_out;
  float* val_out;        // null: right behind the indices (packed payload)
  int* nnz_dev;
  unsigned cap;          // BOUNDED only
  unsigned long long* dropped;
  bool vec;
};

template <bool BOUNDED, typename Source>
__global__ void __launch_bounds__(kBlock, kCtasPerSm)
thr_select_kernel(const ThrArgs a, const __grid_constant__ Source source) {
  constexpr unsigned kSlots = 192;
  __shared__ int slot_idx[kWarps][kSlots];
  __shared__ float slot_val[kWarps][kSlots];
  __shared__ uint2 sm[kWarps];
  __shared__ unsigned warp_counts[2][kWarps], next[2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for_chunks<false>(
      a.work, blockIdx.x, a.ws.counters->ticket, next,
      [&](unsigned chunk, unsigned parity) {
        size_t lo, hi;
        run_tiles(a.work, chunk, a.n, lo, hi);
        const size_t run = static_cast<size_t>(chunk) * kWarps + warp;
        int* const list_idx = a.ws.list_idx + run * a.work.capacity;
        float* const list_val = a.ws.list_val + run * a.work.capacity;
        unsigned used = 0, count = 0;
        size_t unlisted = hi;           // tiles [unlisted, hi) are counted only; acc keeps s there
        Cursor at;
        if (lo < hi) seek(source, at, lo);
        for (size_t tile = lo; tile < hi; ++tile) {
          float s[kRounds][4];
          const View v = view(source, at, a.acc, a.n);
          load_tile(source, at, a.g, v.acc, tile, v.n, a.vec, s);
          if (tile + 1 < hi) {
            // the residual of the next tile, into L2 while this one is worked on
            // (2.56e7 elements: 72.6 -> 66.2 us)
            advance(source, at, tile + 1);
            const View next = view(source, at, a.acc, a.n);
            if (next.acc && (tile + 2) * kTile <= next.n) {
#pragma unroll
              for (int r = 0; r < kRounds; ++r) prefetch_l2(next.acc + vec_at(tile + 1, r));
            }
          }
          unsigned m = 0, excl[kRounds];  // out-of-range lanes are 0 and never selected
#pragma unroll
          for (int r = 0; r < kRounds; ++r)
#pragma unroll
            for (int j = 0; j < 4; ++j)
              m |= (fabsf(s[r][j]) >= a.thr && s[r][j] != 0.0f) ? 1u << (4 * r + j) : 0u;
          const unsigned total = tile_exclusive(round_counts(m), excl);
          if (unlisted == hi && used + total > a.work.capacity) unlisted = tile;
          const bool listed = unlisted == hi;
          if (v.acc) {
#pragma unroll
            for (int r = 0; r < kRounds; ++r) {
              float res[4];
#pragma unroll
              for (int j = 0; j < 4; ++j)
                res[j] = listed && fabsf(s[r][j]) >= a.thr ? s[r][j] - s[r][j] : s[r][j];
              store4(v.acc, vec_at(tile, r), v.n, a.vec, res);
            }
          }
          count += total;
          if (!listed || !total) continue;
          list_tile(s, m, excl, total, tile, list_idx + used, list_val + used, slot_idx[warp], slot_val[warp], kSlots);
          used += total;
        }
        if (lane == 0) {
          a.ws.run_meta[run] = pack_meta(count, used, static_cast<unsigned>(unlisted - lo));
          warp_counts[parity][warp] = count;
        }
      },
      [&](unsigned chunk, unsigned parity) {
        if (threadIdx.x != 0) return;
        unsigned t = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) t += warp_counts[parity][w];
        a.ws.chunk_a[chunk] = t;
      });
  cg::this_grid().sync();

  unsigned first, last;
  my_chunks(a.work, blockIdx.x, first, last);
  const Before b = counts_before(a.ws.chunk_a, a.work.chunks, first, sm);
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.nnz_dev = static_cast<int>(b.total);
  float* const val_out = a.val_out ? a.val_out : reinterpret_cast<float*>(a.idx_out) + (BOUNDED ? a.cap : b.total);
  unsigned lost = 0, chunk_at = b.before;
  for (unsigned chunk = first; chunk < last; ++chunk) {
    const size_t run = static_cast<size_t>(chunk) * kWarps + warp;
    const int* const list_idx = a.ws.list_idx + run * a.work.capacity;
    const float* const list_val = a.ws.list_val + run * a.work.capacity;
    const unsigned meta = lane < kWarps ? __ldcg(a.ws.run_meta + run - warp + lane) : 0u;
    // the first 128 entries are fetched beside the count (they are inside the
    // segment whatever it is): one round trip per chunk instead of two
    int idx[4];
    float val[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      idx[q] = __ldcg(list_idx + lane + 32 * q);
      val[q] = __ldcg(list_val + lane + 32 * q);
    }
    const unsigned mine = __shfl_sync(0xffffffffu, meta, warp), used = meta_used(mine);
    unsigned base = chunk_at + __reduce_add_sync(0xffffffffu, lane < warp ? meta_count(meta) : 0u);
    chunk_at += __reduce_add_sync(0xffffffffu, meta_count(meta));
    for (unsigned e0 = lane; e0 < used; e0 += 128) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (e0 >= 128 && e0 + 32 * q < used) {
          idx[q] = __ldcg(list_idx + e0 + 32 * q);
          val[q] = __ldcg(list_val + e0 + 32 * q);
        }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (e0 + 32 * q >= used) break;
        const unsigned pos = base + e0 + 32 * q;
        if (!BOUNDED || pos < a.cap) {
          a.idx_out[pos] = idx[q];
          val_out[pos] = val[q];
        } else {
          if (a.acc) a.acc[idx[q] - 1] = val[q];
          ++lost;
        }
      }
    }
    // tiles that did not fit the list: acc (or g) still holds s
    base += used;
    size_t lo, hi;
    run_tiles(a.work, chunk, a.n, lo, hi);
    for (size_t tile = lo + meta_listed(mine); tile < hi; ++tile) {
      float s[kRounds][4];
      Cursor at;
      seek(source, at, tile);
      const View v = view(source, at, a.acc, a.n);
      load_tile(v.acc ? v.acc : a.g, nullptr, tile, v.n, a.vec, s);
      unsigned m = 0, excl[kRounds];
#pragma unroll
      for (int r = 0; r < kRounds; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          m |= (fabsf(s[r][j]) >= a.thr && s[r][j] != 0.0f) ? 1u << (4 * r + j) : 0u;
      const unsigned total = tile_exclusive(round_counts(m), excl);
#pragma unroll
      for (int r = 0; r < kRounds; ++r) {
        const size_t i = vec_at(tile, r);
        unsigned pos = base + excl[r];
        bool sent = false;
        float res[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          res[j] = s[r][j];
          if (!(fabsf(s[r][j]) >= a.thr)) continue;
          if (s[r][j] == 0.0f) {                     // thr == 0: not sent, s - kept is still +0
            res[j] = 0.0f;
            sent = true;
            continue;
          }
          if (!BOUNDED || pos < a.cap) {
            a.idx_out[pos] = static_cast<int>(i + j + 1);
            val_out[pos] = s[r][j];
            res[j] = s[r][j] - s[r][j];
            sent = true;
          } else {
            ++lost;
          }
          ++pos;
        }
        if (v.acc && sent) store4(v.acc, i, v.n, a.vec, res);
      }
      base += total;
    }
  }
  if (BOUNDED) {
    lost = __reduce_add_sync(0xffffffffu, lost);
    if (lane == 0 && lost) atomicAdd(a.dropped, static_cast<unsigned long long>(lost));
  }
}

// ---------------------------------------------------------------- top-K mode
// mode 0 "magnitude": key = bits of |s| (monotonic in |s| for non-NaN);
// mode 1 "compat":    key = |(int)s|, the value the reference's comparator
//                     actually compares (both operands truncated to int).
template <int MODE>
__device__ __forceinline__ unsigned make_key(float s) {
  if (MODE == 0) return __float_as_uint(s) & 0x7fffffffu;
  const int t = static_cast<int>(s);  // saturating truncation toward zero
  return t < 0 ? 0u - static_cast<unsigned>(t) : static_cast<unsigned>(t);
}

// Adds the four keys of one vector to a shared-memory histogram.  Fast path:
// every lane of the warp takes all four of its elements and they fall into one
// bin (always true when every key ties): one atomic per warp for 128 elements.
__device__ __forceinline__ void tally4(unsigned* sh, const unsigned (&bin)[4], const bool (&take)[4]) {
  const bool mine_same = take[0] && take[1] && take[2] && take[3] && bin[0] == bin[1] && bin[1] == bin[2] &&
                         bin[2] == bin[3];
  const unsigned b0 = __shfl_sync(0xffffffffu, bin[0], 0);
  if (__all_sync(0xffffffffu, mine_same && bin[0] == b0)) {
    if ((threadIdx.x & 31) == 0) atomicAdd(&sh[b0], 128u);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (take[j]) atomicAdd(&sh[bin[j]], 1u);
  }
}

template <int BINS>
__device__ __forceinline__ void clear_bins(unsigned* sh) {
  for (int b = threadIdx.x; b < BINS; b += kBlock) sh[b] = 0;
  __syncthreads();
}
template <int BINS>
__device__ __forceinline__ void flush_bins(const unsigned* sh, unsigned* global) {
  __syncthreads();
  for (int b = threadIdx.x; b < BINS; b += kBlock)
    if (sh[b]) atomicAdd(&global[b], sh[b]);
}

// The bin, counted from the top, in which the cumulative count reaches
// `remaining`, and how many elements are still to be taken from it.  Every CTA
// works it out for itself from the global histogram.  If the total is short
// (cannot happen for k <= n) the lowest bin takes whatever is left.
template <int BINS>
__device__ __forceinline__ void pick_bin(const unsigned* hist, unsigned& remaining, unsigned& bin, unsigned* sm) {
  constexpr int kPer = BINS / kBlock;                // consecutive bins per thread, descending
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned mine[kPer], local = 0;
#pragma unroll
  for (int j = 0; j < kPer; j += 4) {
    // bins kBins-1 - (t*kPer + j) and the three below it: one aligned vector, reversed
    const uint4 v = __ldcg(reinterpret_cast<const uint4*>(hist + BINS - 4 - (threadIdx.x * kPer + j)));
    mine[j] = v.w; mine[j + 1] = v.z; mine[j + 2] = v.y; mine[j + 3] = v.x;
  }
#pragma unroll
  for (int j = 0; j < kPer; ++j) local += mine[j];
  unsigned incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) sm[w] = incl;
  __syncthreads();
  unsigned above = incl - local;
  for (int k = 0; k < w; ++k) above += sm[k];
  const bool last = threadIdx.x == kBlock - 1;
  if (above < remaining && (remaining <= above + local || last)) {   // exactly one thread
    unsigned left = remaining - above;
    int b = BINS - 1 - threadIdx.x * kPer;
    bool found = false;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      if (!found && (mine[j] >= left || (last && j == kPer - 1))) {
        found = true;
        b -= j;
      }
      if (!found) left -= mine[j];
    }
    sm[kWarps] = static_cast<unsigned>(b);
    sm[kWarps + 1] = left;
  }
  __syncthreads();
  bin = sm[kWarps];
  remaining = sm[kWarps + 1];
  __syncthreads();
}

struct TopkArgs {
  const float* g;
  float* acc;
  size_t n;
  unsigned k;
  unsigned sample_target;  // rank in the sample that bounds the k-th key from below; 0: no sample
  Work work;
  Workspace ws;
  int* idx_out;
  float* val_out;
  bool vec;
  unsigned index_base;     // added to the indices that are sent
};

// s of one element.
__device__ __forceinline__ float element(const NoPieces&, const float* g, const float* acc, size_t i) {
  return acc ? g[i] + acc[i] : g[i];
}
template <typename P>
__device__ __forceinline__ float element(const P& p, const float*, const float* acc, size_t i) {
  int lo = 0, hi = p.count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (p.off[mid] <= i) lo = mid; else hi = mid - 1;
  }
  return p.ptr[lo][i - p.off[lo]] + acc[i];
}

// One warp's list while it goes through the tiles of a run.
struct RunList {
  int* idx;
  float* val;
  unsigned capacity, used;
  size_t unlisted;       // tiles from here on are not in the list
};
// Appends the tile's elements of mask `m` while there is room, and calls
// tally(value) for each of them in any case.  Few per lane (about one element
// in sixty): walking the set bits, with the value picked from the registers,
// beats sixteen predicated blocks.
template <typename Tally>
__device__ __forceinline__ void list_keys(const float (&s)[kRounds][4], unsigned m, size_t tile, size_t hi,
                                          RunList& list, int* slot_idx, float* slot_val, unsigned slots, Tally tally) {
  if (!__any_sync(0xffffffffu, m)) return;
  const int lane = threadIdx.x & 31;
  bool room = list.unlisted == hi;
  unsigned excl[kRounds], total = 0;
  if (room) {
    total = tile_exclusive(round_counts(m), excl);
    if (list.used + total > list.capacity) {
      list.unlisted = tile;
      room = false;
    }
  }
  const bool staged = total <= slots;
  int* const di = staged ? slot_idx : list.idx + list.used;
  float* const dv = staged ? slot_val : list.val + list.used;
  unsigned long long at = 0;                           // next position of each round, 16 bits each
  if (room) {
#pragma unroll
    for (int r = 0; r < kRounds; ++r) at |= static_cast<unsigned long long>(excl[r]) << (16 * r);
  }
  for (unsigned left = m; left; left &= left - 1) {
    const int q = __ffs(left) - 1;
    float v = 0.0f;
#pragma unroll
    for (int e = 0; e < 4 * kRounds; ++e) v = e == q ? s[e >> 2][e & 3] : v;
    tally(v);
    if (room) {
      const unsigned pos = static_cast<unsigned>(at >> (16 * (q >> 2))) & 0xffffu;
      at += 1ull << (16 * (q >> 2));
      di[pos] = static_cast<int>(vec_at(tile, q >> 2) + (q & 3) + 1);
      dv[pos] = v;
    }
  }
  if (!room) return;
  if (staged) {
    __syncwarp();
    for (unsigned e = lane; e < total; e += 32) {
      list.idx[list.used + e] = slot_idx[e];
      list.val[list.used + e] = slot_val[e];
    }
    __syncwarp();
  }
  list.used += total;
}

// Radix selection over 12 + 10 + 10 key bits, one cooperative launch:
//   sample  128 elements per warp bound the k-th key from below (large n only)
//   pass 0  s = g + acc; histogram of the top digit; with a bound, the keys at
//           or above it go to the lists, and only they are counted
//   pass 1  the middle digit inside the chosen bin: from the lists, or without
//           a bound (or if it turned out too high) from s, which fills the lists
//   pass 2  the last digit, from the lists; then count and copy out.
// HBM-bound: pass 0 moves 12 B/element, pass 1 over s another 4, of which the
// sample (8 us) saves the most and four in five of the shared-memory atomics.
//
// `rank` of a.work.grid CTAs, which sync() brings together: the whole grid, or the
// part of it that works on one of several buckets.  Where sync() says false the others
// did not come: what they should have written is not there, and the CTA leaves.
template <int MODE, typename Source, typename Sync>
__device__ __forceinline__ void topk_select(const TopkArgs& a, const Source& source, const unsigned rank, Sync sync) {
  constexpr unsigned kSlots = 96;
  __shared__ unsigned sh[kBins1];
  __shared__ int slot_idx_all[kWarps][kSlots];
  __shared__ float slot_val_all[kWarps][kSlots];
  __shared__ uint2 sm2[kWarps];
  __shared__ unsigned sm[kWarps + 2], next[2];
  const unsigned ranks = a.work.grid;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int* const slot_idx = slot_idx_all[warp];
  float* const slot_val = slot_val_all[warp];
  Counters* const cnt = a.ws.counters;
  const size_t n = a.n;
  const unsigned capacity = a.work.capacity;
  const float* const sum = a.acc ? a.acc : a.g;      // s after pass 0
  auto nothing = [](unsigned, unsigned) {};
  auto run_list = [&](size_t run, size_t hi) {
    return RunList{a.ws.list_idx + run * capacity, a.ws.list_val + run * capacity, capacity, 0, hi};
  };

  unsigned floor_bin = 0;                            // bins from here on are listed in pass 0; 0: none
  if (MODE == 0 && a.sample_target) {
    clear_bins<kBins1>(sh);
    const unsigned warps = ranks * kWarps;
    const size_t e0 = n / warps * (rank * kWarps + warp) + lane;   // n / warps >= 128: see the host's rule
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = element(source, a.g, a.acc, e0 + 32 * q);
    unsigned bin[4];
    const bool take[4] = {true, true, true, true};
#pragma unroll
    for (int q = 0; q < 4; ++q) bin[q] = make_key<MODE>(v[q]) >> 20;
    tally4(sh, bin, take);
    flush_bins<kBins1>(sh, cnt->sample);
    if (!sync()) return;
    unsigned left = a.sample_target, b;
    pick_bin<kBins1>(cnt->sample, left, b, sm);
    // more than an eighth at or above the bound (ties, a crowded bin) would not fit the lists
    const unsigned taken = a.sample_target - left + __ldcg(&cnt->sample[b]);
    if (taken <= warps * (128 / 8)) floor_bin = b;
  }

  // pass 0: fold the gradient into the residual, histogram of the top 12 key bits
  clear_bins<kBins1>(sh);
  unsigned top = 0;
  for_chunks<false>(
      a.work, rank, &cnt->ticket[0], next,
      [&](unsigned chunk, unsigned) {
        size_t lo, hi;
        run_tiles(a.work, chunk, n, lo, hi);
        const size_t run = static_cast<size_t>(chunk) * kWarps + warp;
        RunList list = run_list(run, hi);
        Cursor at;
        if (lo < hi) seek(source, at, lo);
        for (size_t tile = lo; tile < hi; ++tile, advance(source, at, tile)) {
          float s[kRounds][4];
          load_tile(source, at, a.g, a.acc, tile, n, a.vec, s);
          if (a.acc) {
#pragma unroll
            for (int r = 0; r < kRounds; ++r) store4(a.acc, vec_at(tile, r), n, a.vec, s[r]);
          }
          if (floor_bin) {
            unsigned m = 0;                          // out-of-range lanes have key 0
#pragma unroll
            for (int r = 0; r < kRounds; ++r)
#pragma unroll
              for (int j = 0; j < 4; ++j) m |= make_key<MODE>(s[r][j]) >> 20 >= floor_bin ? 1u << (4 * r + j) : 0u;
            list_keys(s, m, tile, hi, list, slot_idx, slot_val, kSlots,
                      [&](float v) { atomicAdd(&sh[make_key<MODE>(v) >> 20], 1u); });
            continue;
          }
          const unsigned valid = in_range(tile, n);
#pragma unroll
          for (int r = 0; r < kRounds; ++r) {
            unsigned bin[4];
            bool take[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const unsigned key = make_key<MODE>(s[r][j]);  // 0 outside the range
              take[j] = valid >> (4 * r + j) & 1u;
              top = max(top, key);
              bin[j] = key >> 20;
            }
            tally4(sh, bin, take);
          }
        }
        if (floor_bin && lane == 0)
          a.ws.run_meta[run] = pack_meta(0, list.used, static_cast<unsigned>(list.unlisted - lo));
      },
      nothing);
  flush_bins<kBins1>(sh, cnt->hist0);
  top = __reduce_max_sync(0xffffffffu, top);
  if (lane == 0) sm[warp] = top;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < kWarps; ++k) top = max(top, sm[k]);
    if (top) atomicMax(&cnt->max_key, top);
  }
  if (!sync()) return;

  unsigned remaining = a.k, bin;
  pick_bin<kBins1>(cnt->hist0, remaining, bin, sm);
  const bool listed = floor_bin && bin >= floor_bin;
  if (floor_bin && !listed) {
    // fewer than k keys at or above the bound: count the others as well
    clear_bins<kBins1>(sh);
    for_chunks<true>(
        a.work, rank, &cnt->ticket[2], next,
        [&](unsigned chunk, unsigned) {
          size_t lo, hi;
          run_tiles(a.work, chunk, n, lo, hi);
          for (size_t tile = lo; tile < hi; ++tile) {
            float s[kRounds][4];
            load_tile(sum, nullptr, tile, n, a.vec, s);
            const unsigned valid = in_range(tile, n);
#pragma unroll
            for (int r = 0; r < kRounds; ++r) {
              unsigned low[4];
              bool take[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                low[j] = make_key<MODE>(s[r][j]) >> 20;
                take[j] = (valid >> (4 * r + j) & 1u) && low[j] < floor_bin;
              }
              tally4(sh, low, take);
            }
          }
        },
        nothing);
    flush_bins<kBins1>(sh, cnt->hist0);
    if (!sync()) return;
    remaining = a.k;
    pick_bin<kBins1>(cnt->hist0, remaining, bin, sm);
  }
  // the sample has seen a key of floor_bin
  const unsigned max_key = floor_bin ? floor_bin << 20 : __ldcg(&cnt->max_key);
  if (max_key == 0) {
    // every key is 0 (small gradients under integer-truncated keys): the first
    // k elements are sent, and the whole grid shares the work
    for (size_t i = rank * static_cast<size_t>(kBlock) + threadIdx.x; i < a.k;
         i += static_cast<size_t>(ranks) * kBlock) {
      a.idx_out[i] = static_cast<int>(i + 1 + a.index_base);
      a.val_out[i] = __ldcg(sum + i);                // written by another CTA in pass 0
      if (a.acc) a.acc[i] = 0.0f;
    }
    return;
  }

  // Once there are lists only they are looked at, and the tiles that are not in
  // one: calls entry(value) for each listed entry and tile_fn(values, tile) for
  // each other tile of this warp's runs, and done(run) after each run.  The
  // next run's count and first 64 entries are fetched ahead (they are inside
  // the segment whatever the count).
  unsigned first, last;
  my_chunks(a.work, rank, first, last);
  auto visit = [&](auto entry, auto tile_fn, auto done) {
    unsigned meta = 0;
    float v0 = 0.0f, v1 = 0.0f;
    auto fetch = [&](unsigned chunk) {
      const size_t run = static_cast<size_t>(chunk) * kWarps + warp;
      meta = __ldcg(a.ws.run_meta + run);
      v0 = __ldcg(a.ws.list_val + run * capacity + lane);
      v1 = __ldcg(a.ws.list_val + run * capacity + lane + 32);
    };
    if (first < last) fetch(first);
    for (unsigned chunk = first; chunk < last; ++chunk) {
      const size_t run = static_cast<size_t>(chunk) * kWarps + warp;
      const float* const list_val = a.ws.list_val + run * capacity;
      const unsigned now = meta, used = meta_used(now);
      const float w0 = v0, w1 = v1;
      if (chunk + 1 < last) fetch(chunk + 1);
      if (lane < used) entry(w0);
      if (lane + 32 < used) entry(w1);
      for (unsigned e = lane + 64; e < used; e += 32) entry(__ldcg(list_val + e));
      size_t lo, hi;
      run_tiles(a.work, chunk, n, lo, hi);
      for (size_t tile = lo + meta_listed(now); tile < hi; ++tile) {
        float s[kRounds][4];
        load_tile(sum, nullptr, tile, n, a.vec, s);
        tile_fn(s, tile);
      }
      done(run);
    }
  };
  auto no_done = [](size_t) {};
  // pass 1: the histogram of the next digit inside the bin
  const bool low_only = max_key < (1u << 10);        // the middle digit is zero everywhere
  const int shift = low_only ? 0 : 10;
  unsigned prefix = bin << 20;
  // The lowest bin takes in everything: no use listing it, and its keys tend
  // to tie, which is what tally4 is for.
  const bool everything = prefix == 0;
  clear_bins<kBins23>(sh);
  auto tally_tile = [&](const float (&s)[kRounds][4], size_t tile) {
    const unsigned valid = in_range(tile, n);
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      unsigned digit[4];
      bool take[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const unsigned key = make_key<MODE>(s[r][j]);
        take[j] = (valid >> (4 * r + j) & 1u) && key >> 20 == bin;
        digit[j] = (key >> shift) & (kBins23 - 1);
      }
      tally4(sh, digit, take);
    }
  };
  auto tally_key = [&](float v) {
    const unsigned key = make_key<MODE>(v);
    if (key >> 20 == bin) atomicAdd(&sh[(key >> shift) & (kBins23 - 1)], 1u);
  };
  if (listed) {
    // pass 0 has streamed the lists out of L2: ask for all of them at once
    for (unsigned chunk = first + lane; chunk < last; chunk += 32) {
      const size_t run = static_cast<size_t>(chunk) * kWarps + warp;
      prefetch_l2(a.ws.run_meta + run);
      prefetch_l2(a.ws.list_val + run * capacity);
      prefetch_l2(a.ws.list_val + run * capacity + 32);
      prefetch_l2(a.ws.list_idx + run * capacity);
      prefetch_l2(a.ws.list_idx + run * capacity + 32);
    }
    visit(tally_key, tally_tile, no_done);
  } else {
    // chunks in descending order: what pass 0 touched last is still in L2
    for_chunks<true>(
        a.work, rank, &cnt->ticket[1], next,
        [&](unsigned chunk, unsigned) {
          size_t lo, hi;
          run_tiles(a.work, chunk, n, lo, hi);
          const size_t run = static_cast<size_t>(chunk) * kWarps + warp;
          RunList list = run_list(run, hi);
          if (everything) list.unlisted = lo;
          for (size_t tile = lo; tile < hi; ++tile) {
            float s[kRounds][4];
            load_tile(sum, nullptr, tile, n, a.vec, s);
            if (everything) {
              tally_tile(s, tile);
              continue;
            }
            unsigned m = 0;                          // out-of-range lanes have key 0 < prefix
#pragma unroll
            for (int r = 0; r < kRounds; ++r)
#pragma unroll
              for (int j = 0; j < 4; ++j) m |= make_key<MODE>(s[r][j]) >= prefix ? 1u << (4 * r + j) : 0u;
            list_keys(s, m, tile, hi, list, slot_idx, slot_val, kSlots, tally_key);
          }
          if (lane == 0)
            a.ws.run_meta[run] = pack_meta(0, list.used, static_cast<unsigned>(list.unlisted - lo));
        },
        nothing);
  }
  flush_bins<kBins23>(sh, cnt->hist1);
  if (!sync()) return;
  pick_bin<kBins23>(cnt->hist1, remaining, bin, sm);
  prefix |= bin << shift;

  if (!low_only) {
    // pass 2: the last digit
    clear_bins<kBins23>(sh);
    visit(
          [&](float v) {
            const unsigned key = make_key<MODE>(v);
            if ((key & ~(kBins23 - 1u)) == prefix) atomicAdd(&sh[key & (kBins23 - 1)], 1u);
          },
          [&](const float (&s)[kRounds][4], size_t tile) {
            const unsigned valid = in_range(tile, n);
#pragma unroll
            for (int r = 0; r < kRounds; ++r) {
              unsigned digit[4];
              bool take[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const unsigned key = make_key<MODE>(s[r][j]);
                take[j] = (valid >> (4 * r + j) & 1u) && (key & ~(kBins23 - 1u)) == prefix;
                digit[j] = key & (kBins23 - 1);
              }
              tally4(sh, digit, take);
            }
          },
          no_done);
    flush_bins<kBins23>(sh, cnt->hist2);
    if (!sync()) return;
    pick_bin<kBins23>(cnt->hist2, remaining, bin, sm);
    prefix |= bin;
  }

  // T = prefix: keys above T are sent, and the first `quota` keys equal to T
  const unsigned T = prefix, quota = remaining;
  auto masks = [&](const float (&s)[kRounds][4], size_t tile, unsigned& mg, unsigned& me) {
    mg = me = 0;
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const unsigned key = make_key<MODE>(s[r][j]);
        mg |= key > T ? 1u << (4 * r + j) : 0u;
        me |= key == T ? 1u << (4 * r + j) : 0u;
      }
    me &= in_range(tile, n);                         // out-of-range lanes have key 0: never above T
  };
  // counts per run, greater in the high half (a run has <= 2048 elements), kept
  // for the positions below; sums per CTA for the other CTAs
  unsigned c = 0, c_gt = 0, c_eq = 0;
  visit(
      [&](float v) {
        const unsigned key = make_key<MODE>(v);
        c += key > T ? 0x10000u : key == T ? 1u : 0u;
      },
      [&](const float (&s)[kRounds][4], size_t tile) {
        unsigned mg, me;
        masks(s, tile, mg, me);
        c += __popc(mg) << 16 | __popc(me);
      },
      [&](size_t run) {
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) {
          a.ws.run_counts[run] = c;
          c_gt += c >> 16;
          c_eq += c & 0xffffu;
        }
        c = 0;
      });
  const uint2 mine_all = cta_sum2(c_gt, c_eq, sm2);
  if (threadIdx.x == 0) {
    a.ws.chunk_a[rank] = mine_all.x;
    a.ws.chunk_b[rank] = mine_all.y;
  }
  if (!sync()) return;
  unsigned g_chunk = counts_before(a.ws.chunk_a, ranks, rank, sm2).before;
  unsigned e_chunk = counts_before(a.ws.chunk_b, ranks, rank, sm2).before;

  // payload position = (#greater before) + min(#equal before, quota)
  auto send = [&](size_t index1, float v, unsigned ng, unsigned ne) {
    const unsigned pos = ng + (ne < quota ? ne : quota);
    a.idx_out[pos] = static_cast<int>(index1 + a.index_base);
    a.val_out[pos] = v;
    if (a.acc) a.acc[index1 - 1] = 0.0f;             // s - s
  };
  const unsigned below = (1u << lane) - 1u;
  unsigned next_c = 0, next_meta = 0;
  float next_v = 0.0f;
  int next_i = 0;
  auto fetch = [&](unsigned chunk) {
    const size_t run = static_cast<size_t>(chunk) * kWarps + warp;
    next_c = lane < kWarps ? __ldcg(a.ws.run_counts + run - warp + lane) : 0u;
    next_meta = __ldcg(a.ws.run_meta + run);
    next_v = __ldcg(a.ws.list_val + run * capacity + lane);
    next_i = __ldcg(a.ws.list_idx + run * capacity + lane);
  };
  if (first < last) fetch(first);
  for (unsigned chunk = first; chunk < last; ++chunk) {
    const size_t run = static_cast<size_t>(chunk) * kWarps + warp;
    const int* const list_idx = a.ws.list_idx + run * capacity;
    const float* const list_val = a.ws.list_val + run * capacity;
    const unsigned c = next_c, meta = next_meta, used = meta_used(meta);
    float v_now = next_v;
    int i_now = next_i;
    if (chunk + 1 < last) fetch(chunk + 1);
    const unsigned mine = __shfl_sync(0xffffffffu, c, warp);
    unsigned g_at = g_chunk + __reduce_add_sync(0xffffffffu, lane < warp ? c >> 16 : 0u);
    unsigned e_at = e_chunk + __reduce_add_sync(0xffffffffu, lane < warp ? c & 0xffffu : 0u);
    g_chunk += __reduce_add_sync(0xffffffffu, c >> 16);
    e_chunk += __reduce_add_sync(0xffffffffu, c & 0xffffu);
    if (mine >> 16 == 0 && ((mine & 0xffffu) == 0 || e_at >= quota)) continue;   // this run sends nothing
    for (unsigned base = 0; base < used; base += 32) {   // the list, 32 entries at a time, in order
      const bool in = base + lane < used;
      const float v = v_now;
      const int idx = i_now;
      if (base + 32 + lane < used) {
        v_now = __ldcg(list_val + base + 32 + lane);
        i_now = __ldcg(list_idx + base + 32 + lane);
      }
      const unsigned key = make_key<MODE>(v);
      const bool is_gt = in && key > T, is_eq = in && key == T;
      const unsigned mg = __ballot_sync(0xffffffffu, is_gt), me = __ballot_sync(0xffffffffu, is_eq);
      const unsigned ng = g_at + __popc(mg & below), ne = e_at + __popc(me & below);
      if (is_gt || (is_eq && ne < quota)) send(static_cast<size_t>(idx), v, ng, ne);
      g_at += __popc(mg);
      e_at += __popc(me);
    }
    size_t lo, hi;
    run_tiles(a.work, chunk, n, lo, hi);
    for (size_t tile = lo + meta_listed(meta); tile < hi; ++tile) {
      float s[kRounds][4];
      load_tile(sum, nullptr, tile, n, a.vec, s);
      unsigned mg, me, xg[kRounds], xe[kRounds];
      masks(s, tile, mg, me);
      const unsigned tg = tile_exclusive(round_counts(mg), xg), te = tile_exclusive(round_counts(me), xe);
#pragma unroll
      for (int r = 0; r < kRounds; ++r) {
        const size_t i = vec_at(tile, r);
        unsigned ng = g_at + xg[r], ne = e_at + xe[r];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool is_gt = mg >> (4 * r + j) & 1u, is_eq = me >> (4 * r + j) & 1u;
          if (is_gt || (is_eq && ne < quota)) send(i + j + 1, s[r][j], ng, ne);
          ng += is_gt;
          ne += is_eq;
        }
      }
      g_at += tg;
      e_at += te;
    }
  }
}

template <int MODE, typename Source>
__global__ void __launch_bounds__(kBlock, kCtasPerSm)
topk_select_kernel(const TopkArgs a, const __grid_constant__ Source source) {
  topk_select<MODE>(a, source, blockIdx.x, [] {
    cg::this_grid().sync();
    return true;
  });
}

// Several buckets at once, each by its own part of a cooperative grid: a bucket of
// 2e5 elements keeps 54 CTAs busy for a tenth of the 14 us that its barriers take
// (2.56e7 elements in 11 buckets: 547 -> 210 us a pass, in 25: 727 -> 206; 2e6 in
// four: 93 -> 42).
// The parts do not wait for one another.  Their barrier counts arrivals; all CTAs
// are resident, and the wait is bounded: one that runs out sets the sticky fault word
// (sgb_sparse_faults) and marks the barrier, and the part's CTAs leave.
struct TopkBuckets {
  int count;
  unsigned first_cta[kBuckets + 1];
  unsigned n[kBuckets], k[kBuckets], sample_target[kBuckets], at[kBuckets], index_base[kBuckets];   // at: in the payload
  Work work[kBuckets];
  size_t ws_off[kBuckets];         // of a bucket's lists in the workspace, behind the counters of all
  float* acc[kBuckets];
  int first_piece[kBuckets + 1];   // a bucket's offsets start at first_piece + its number (one more than pieces)
  unsigned off[kPieces + kBuckets];
  const float* ptr[kPieces];
  char* ws;
  int* idx_out;
  float* val_out;
};
__device__ unsigned g_topk_faults;
template <int MODE>
__global__ void __launch_bounds__(kBlock, kCtasPerSm)
topk_buckets_kernel(const __grid_constant__ TopkBuckets b) {
  int g = 0;
  for (int hi = b.count - 1; g < hi;) {
    const int mid = (g + hi + 1) >> 1;
    if (b.first_cta[mid] <= blockIdx.x) g = mid; else hi = mid - 1;
  }
  const PieceView source{b.first_piece[g + 1] - b.first_piece[g], b.off + b.first_piece[g] + g, b.ptr + b.first_piece[g]};
  const TopkArgs a{nullptr, b.acc[g], b.n[g], b.k[g], b.sample_target[g], b.work[g],
                   carve_at(b.ws + g * align256(sizeof(Counters)), b.ws + b.ws_off[g], b.work[g]), b.idx_out + b.at[g],
                   b.val_out + b.at[g], true, b.index_base[g]};
  unsigned* const arrived = &a.ws.counters->arrived;
  unsigned target = 0;
  topk_select<MODE>(a, source, blockIdx.x - b.first_cta[g], [&] {
    constexpr unsigned kLeft = 1u << 31, kMostPolls = 1u << 21;   // polls of half a microsecond and more
    target += a.work.grid;
    __syncthreads();
    bool in = false;
    if (threadIdx.x == 0) {
      __threadfence();
      atomicAdd(arrived, 1u);
      unsigned v = 0;
      for (unsigned q = 0; q < kMostPolls && v < target; ++q)
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrived) : "memory");
      in = v >= target && v < kLeft;
      if (v < target) {
        atomicOr(arrived, kLeft);
        atomicOr(&g_topk_faults, 1u);
      }
      __threadfence();
    }
    return __syncthreads_or(in) != 0;
  });
}

// -------------------------------------------------------- dense sum of payloads
// The dense gradient is built tile by tile in shared memory: zeros, plus each
// rank's entries of that tile in ascending rank order (the additions of the
// reference's scatter, rank after rank), then one coalesced store to the
// tensors the tile overlaps.  It replaces a fill of the dense buffer, one
// scatter pass per rank that re-reads and re-writes scattered sectors of it,
// and the copy back into the tensors: 4 B/element written, the payload read.
// Payloads are in ascending index order, so a CTA finds its start in each with
// one search and then walks forward.
constexpr int kDenseTargets = 200;   // below 4 KB of kernel arguments
constexpr int kDenseTile = 4096;   // elements: 16 KB of shared memory
struct DenseArgs {
  const int* payload;          // rank r: [idx | val] at payload + r * stride
  size_t stride;
  size_t val_off;              // 0: the values follow the rank's own count
  const int* counts_dev;       // counts on the device, clamped to most; null: counts[]
  unsigned most;
  int world;
  int counts[kMaxDenseRanks];
  size_t first, last;          // element range of this launch
  uint4* clear;                // set to 0 on the way, for the next selection
  unsigned clear_vecs;
  int targets;
  size_t off[kDenseTargets + 1];   // first element of each target tensor; off[targets] == last
  float* ptr[kDenseTargets];
};
// Parameter and momentum of each target, for the form that ends in the update.
struct DenseUpdate {
  SgdArgs sgd;
  float* p[kDenseTargets];
  float* m[kDenseTargets];
};
struct NoUpdate {};

// A position at most `slack` before the first whose index is >= want (1-based,
// ascending): one warp, 32-ary.  The last rounds of a search cost as much as the
// first (0.7 us each) and save less than one window.
__device__ __forceinline__ unsigned warp_lower_bound(const int* idx, unsigned count, long long want,
                                                     unsigned slack) {
  const unsigned lane = threadIdx.x & 31;
  unsigned lo = 0, hi = count;                       // the answer is in [lo, hi]
  while (hi - lo > slack) {
    const unsigned step = (hi - lo + 31) / 32;
    const unsigned at = lo + lane * step;
    const bool less = at < hi && static_cast<long long>(idx[at]) < want;
    const unsigned m = __ballot_sync(0xffffffffu, less);
    if (m == 0) return lo;
    const unsigned top = 31 - __clz(m);              // probes below the answer are a prefix of the lanes
    const unsigned base = lo + top * step;
    hi = base + step < hi ? base + step : hi;
    lo = base + 1;
  }
  return lo;
}

// g = src (in shared memory), and the update of p and m with it; by all threads of the
// CTA: what is not a whole tile of one tensor.  Vectors start where the tensors' addresses
// are aligned, wherever that is in the tile.
__device__ __forceinline__ void update_run(const SgdArgs& a, float* p, float* g, float* m, const float* src, int len) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(g);
  const uintptr_t apart = (reinterpret_cast<uintptr_t>(p) ^ at) | (a.use_momentum ? reinterpret_cast<uintptr_t>(m) ^ at : 0);
  const int lead = static_cast<int>((0u - static_cast<unsigned>(at >> 2)) & 3u);
  const bool vectors = (apart & 15u) == 0 && lead < len;
  const int head = vectors ? lead : 0, nv = vectors ? (len - lead) >> 2 : 0;
  for (int v = threadIdx.x; v < nv; v += kBlock) {
    const int i = head + 4 * v;
    Vec4f vp, vg, vm;
    vp.u = ld128(p + i);
    if (a.use_momentum) vm.u = ld128(m + i);
#pragma unroll
    for (int j = 0; j < 4; ++j) vg.f[j] = src[i + j];
    st128(g + i, vg.u);
#pragma unroll
    for (int j = 0; j < 4; ++j) sgd_one(vp.f[j], vg.f[j], vm.f[j], a);
    st128(p + i, vp.u);
    if (a.use_momentum) st128(m + i, vm.u);
  }
  for (int e = threadIdx.x; e < len - 4 * nv; e += kBlock) {
    const int i = e < head ? e : e + 4 * nv;
    float pv = p[i], mv = a.use_momentum ? m[i] : 0.f;
    const float gv = src[i];
    g[i] = gv;
    sgd_one(pv, gv, mv, a);
    p[i] = pv;
    if (a.use_momentum) m[i] = mv;
  }
}

// Entries pass through windows of 1024, four per thread, indices and values
// fetched together: with 256 at a time a tile of a dense payload was a chain of
// three to four round trips.  A single rank's window stays in registers over the
// tiles that it serves.  11 buckets of 2.3e6 elements, 15 % of them sent:
// 5.4 us each; 2.56e7 at once: 31.4 -> 24.9 us with the window, the binary
// search for the first target and all 8 CTAs of an SM resident; 1e8 elements,
// 1 % sent: 81.4 -> 80.0 us.
//
// Update: the tile's parameters and momentum are updated with it on the way, so
// that the dense gradient is not read back (a pass of 1e8 elements, 1 % sent:
// 652 -> 644 us; of 3.6e6 62 -> 56, of 4.4e5 34 -> 30).
constexpr int kUpdateCtas = 4;
constexpr size_t kMostTiles = 4;
constexpr size_t kUpdateStage = 2 * kDenseTile * sizeof(float);
__device__ __forceinline__ void stage16(uint4* to, const float* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(to))),
               "l"(from)
               : "memory");
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
template <bool ALONE, typename Update>
__global__ void __launch_bounds__(kBlock, std::is_same_v<Update, NoUpdate> ? 8 : kUpdateCtas)
dense_from_payloads_kernel(const __grid_constant__ DenseArgs a, unsigned tiles_per_cta, const __grid_constant__ Update u) {
  constexpr unsigned kPer = 4, kWindow = kPer * kBlock;
  constexpr bool kUpdate = std::is_same_v<Update, DenseUpdate>;
  constexpr int kVecs = kDenseTile / (4 * kBlock);     // of a thread and tile
  __shared__ __align__(16) float out[kDenseTile];
  [[maybe_unused]] extern __shared__ uint4 staged[];   // kUpdate: the tile's parameters, and its momentum
  __shared__ unsigned cursor[kMaxDenseRanks], count[kMaxDenseRanks];
  dependency_wait();
  release_dependents();
  for (unsigned i = blockIdx.x * kBlock + threadIdx.x; i < a.clear_vecs; i += gridDim.x * kBlock)
    a.clear[i] = make_uint4(0, 0, 0, 0);
  const size_t begin = a.first + static_cast<size_t>(blockIdx.x) * tiles_per_cta * kDenseTile;
  const size_t end = begin + static_cast<size_t>(tiles_per_cta) * kDenseTile < a.last
                         ? begin + static_cast<size_t>(tiles_per_cta) * kDenseTile : a.last;
  for (int r = threadIdx.x >> 5; r < a.world; r += kWarps) {
    int c = a.counts_dev ? a.counts_dev[r] : a.counts[r];
    if (c < 0) c = 0;
    if (static_cast<unsigned>(c) > a.most) c = static_cast<int>(a.most);
    const unsigned at = warp_lower_bound(a.payload + r * a.stride, static_cast<unsigned>(c),
                                         static_cast<long long>(begin) + 1, kBlock);
    if ((threadIdx.x & 31) == 0) {
      cursor[r] = at;
      count[r] = static_cast<unsigned>(c);
    }
  }
  int target = 0;
  for (int hi = a.targets - 1; target < hi;) {
    const int mid = (target + hi + 1) >> 1;
    if (a.off[mid] <= begin) target = mid; else hi = mid - 1;
  }
  unsigned wi[kPer];
  float wv[kPer];
  bool have = false;                                 // ALONE: the window at cursor[0] is in wi, wv
  for (size_t base = begin; base < end; base += kDenseTile) {
    const size_t stop = base + kDenseTile < end ? base + kDenseTile : end;
    // A whole tile of one tensor, whose parameters and momentum lie like its gradient
    // modulo a vector: what its update reads is on its way while the tile is put together.
    [[maybe_unused]] float *pt = nullptr, *gt = nullptr, *mt = nullptr;
    [[maybe_unused]] int head = 0;
    bool whole = false;
    if constexpr (kUpdate) {
      if (base + kDenseTile == stop && a.off[target + 1] >= stop && a.ptr[target]) {
        const size_t in = base - a.off[target];
        gt = a.ptr[target] + in;
        pt = u.p[target] + in;
        mt = u.sgd.use_momentum ? u.m[target] + in : gt;
        const uintptr_t at = reinterpret_cast<uintptr_t>(gt);
        whole = (((reinterpret_cast<uintptr_t>(pt) ^ at) | (reinterpret_cast<uintptr_t>(mt) ^ at)) & 15u) == 0;
        head = static_cast<int>((0u - static_cast<unsigned>(at >> 2)) & 3u);
      }
      if (whole) {
#pragma unroll
        for (int k = 0; k < kVecs; ++k) {
          const int i = head + 4 * (k * kBlock + static_cast<int>(threadIdx.x));
          if (i + 4 <= kDenseTile) {                   // all but the last thread's last vector, if head > 0
            stage16(staged + k * kBlock + threadIdx.x, pt + i);
            if (u.sgd.use_momentum) stage16(staged + (kVecs + k) * kBlock + threadIdx.x, mt + i);
          }
        }
      }
    }
    __syncthreads();                                 // cursors set; the previous tile has been stored
#pragma unroll
    for (int r = 0; r < kDenseTile / (4 * kBlock); ++r)
      reinterpret_cast<float4*>(out)[r * kBlock + threadIdx.x] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    for (int r = 0; r < (ALONE ? 1 : a.world); ++r) {
      const int* idx = a.payload + r * a.stride;
      const unsigned cnt = count[r];
      const float* val = reinterpret_cast<const float*>(idx) + (a.val_off ? a.val_off : cnt);
      unsigned c = cursor[r];
      for (;;) {
        if (!ALONE || !have) {
#pragma unroll
          for (unsigned q = 0; q < kPer; ++q) {
            const unsigned j = c + q * kBlock + threadIdx.x;
            const int i = j < cnt ? idx[j] : 0;
            wv[q] = j < cnt ? val[j] : 0.0f;
            wi[q] = i > 0 ? static_cast<unsigned>(i) : 0xffffffffu;     // padding is beyond every tile
          }
          have = true;
        }
#pragma unroll
        for (unsigned q = 0; q < kPer; ++q)          // indices are unique within a payload
          if (wi[q] > base && wi[q] <= stop) out[wi[q] - 1 - base] += wv[q];
        if (__syncthreads_or(wi[kPer - 1] > stop)) break;               // the window reaches past the tile
        c += kWindow;
        have = false;
        if (threadIdx.x == 0) cursor[r] = c;         // read again behind a barrier
      }
    }
    if constexpr (kUpdate) {
      if (whole) {
        stage_wait();                                  // a thread reads what it has asked for itself
#pragma unroll
        for (int k = 0; k < kVecs; ++k) {
          const int i = head + 4 * (k * kBlock + static_cast<int>(threadIdx.x));
          if (i + 4 > kDenseTile) break;
          Vec4f vp, vg, vm;
          vp.u = staged[k * kBlock + threadIdx.x];
          if (u.sgd.use_momentum) vm.u = staged[(kVecs + k) * kBlock + threadIdx.x];
          if (head == 0) {
            vg.u = *reinterpret_cast<const uint4*>(out + i);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) vg.f[j] = out[i + j];
          }
          st128(gt + i, vg.u);
#pragma unroll
          for (int j = 0; j < 4; ++j) sgd_one(vp.f[j], vg.f[j], vm.f[j], u.sgd);
          st128(pt + i, vp.u);
          if (u.sgd.use_momentum) st128(mt + i, vm.u);
        }
        if (head != 0 && threadIdx.x < 4) {            // the elements ahead of the vectors and behind them
          const int t = static_cast<int>(threadIdx.x), i = t < head ? t : kDenseTile - 4 + t;
          float pv = pt[i], mv = u.sgd.use_momentum ? mt[i] : 0.f;
          const float gv = out[i];
          gt[i] = gv;
          sgd_one(pv, gv, mv, u.sgd);
          pt[i] = pv;
          if (u.sgd.use_momentum) mt[i] = mv;
        }
        if (a.off[target + 1] == stop && target + 1 < a.targets) ++target;
        continue;
      }
    }
    // store the tile to the tensors it overlaps
    for (size_t at = base; at < stop;) {
      const size_t seg_end = a.off[target + 1] < stop ? a.off[target + 1] : stop;
      float* dst = a.ptr[target] + (at - a.off[target]);
      const float* src = out + (at - base);
      const int len = static_cast<int>(seg_end - at);
      if (!a.ptr[target]) {                            // a gap between buckets
      } else if constexpr (kUpdate) {
        const size_t in = at - a.off[target];
        update_run(u.sgd, u.p[target] + in, dst, u.sgd.use_momentum ? u.m[target] + in : nullptr, src, len);
      } else if (((reinterpret_cast<uintptr_t>(dst) | static_cast<uintptr_t>((at - base) * 4)) & 15u) == 0) {
        const int nv = len >> 2;
        for (int v = threadIdx.x; v < nv; v += kBlock)
          reinterpret_cast<float4*>(dst)[v] = reinterpret_cast<const float4*>(src)[v];
        for (int v = (nv << 2) + threadIdx.x; v < len; v += kBlock) dst[v] = src[v];
      } else {
        for (int v = threadIdx.x; v < len; v += kBlock) dst[v] = src[v];
      }
      at = seg_end;
      if (seg_end == a.off[target + 1] && target + 1 < a.targets) ++target;
    }
  }
}

// ------------------------------------------------------------- scatter-add
// dst[idx-1] += val for one rank's payload; the count lives on the device when
// count_dev != NULL (entry `rank_slot`), else `count` is used.  Index 0 marks
// padding and is skipped; indices are unique within a payload, so there are
// no conflicting updates inside one launch.
__global__ void __launch_bounds__(kBlock)
scatter_add_kernel(const int* __restrict__ idx, const float* __restrict__ val, size_t count,
                   const int* __restrict__ count_dev, float* __restrict__ dst, size_t n) {
  size_t m = count;
  if (count_dev) {                                  // the host count is then the capacity of idx / val
    const int dv = *count_dev;
    const size_t d = dv > 0 ? static_cast<size_t>(dv) : 0;
    m = d < count ? d : count;
  }
  for (size_t j = blockIdx.x * static_cast<size_t>(kBlock) + threadIdx.x; j < m;
       j += static_cast<size_t>(gridDim.x) * kBlock) {
    const int i = idx[j];
    if (i > 0 && static_cast<size_t>(i) <= n) dst[i - 1] += val[j];
  }
}

int check_common(const float* g, size_t n, const void* idx_out, void* ws, size_t ws_bytes) {
  if (!g || !idx_out) return SGB_ERR_NULL;
  if (n > 0x7fffffffu) return SGB_ERR_SIZE;  // 1-based int32 indices on the wire
  if (!ws || ws_bytes < workspace_bytes(n) || (reinterpret_cast<uintptr_t>(ws) & 255u))
    return SGB_ERR_WORKSPACE;
  return SGB_OK;
}

// Lets a kernel have `bytes` of dynamic shared memory beside its own, once per device.
template <typename K>
int more_shared_memory(K kernel, size_t bytes, std::atomic<bool>* done) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
  const bool tracked = dev >= 0 && dev < 64;
  if (tracked && done[dev].load(std::memory_order_acquire)) return SGB_OK;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  if (e != cudaSuccess) return note_cuda_error(e);
  if (tracked) done[dev].store(true, std::memory_order_release);
  return SGB_OK;
}

// A grid whose CTAs wait for one another: all of them are resident or the
// launch fails.  work_for() asks for at most kCtasPerSm CTAs per SM, which the
// launch bounds and the shared memory of both kernels allow.
template <typename A, typename S>
int launch_cooperative(void (*kernel)(A, S), unsigned grid, const A& args, const S& source, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kBlock);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args, source);
  if (e != cudaSuccess) return note_cuda_error(e);
  return launch_status();
}

// The gradient behind a selection: one array, or a list of tensors.
struct Gradient {
  const float* flat = nullptr;
  Pieces pieces;
  size_t n = 0;
};
// Fills in `g` from a tensor list; false where the list has to be packed first
// (too many tensors, or no residual buffer to hold their sum).
bool gather(Gradient* g, float* const* tensors, const size_t* sizes, size_t count, const float* acc) {
  g->flat = nullptr;
  g->n = 0;
  g->pieces.count = 0;
  bool joined = true;                                  // back to back in memory
  for (size_t k = 0; k < count; ++k) {
    if (!sizes[k]) continue;
    Pieces& p = g->pieces;
    if (p.count && p.ptr[p.count - 1] + (g->n - p.off[p.count - 1]) == tensors[k]) {
      g->n += sizes[k];
      continue;
    }
    if (p.count) joined = false;
    if (p.count == kPieces) return false;
    p.off[p.count] = static_cast<unsigned>(g->n);
    p.ptr[p.count++] = tensors[k];
    g->n += sizes[k];
  }
  if (g->n > 0x7fffffffu) return false;
  g->pieces.off[g->pieces.count] = static_cast<unsigned>(g->n);
  if (joined) {
    g->flat = g->pieces.count ? g->pieces.ptr[0] : nullptr;
    return true;
  }
  return acc && aligned16(acc);
}

int threshold_select(const Gradient& source, float* acc, float thr, int* idx_out, float* val_out, int* nnz_dev,
                     size_t cap, unsigned long long* dropped, void* ws, size_t ws_bytes, cudaStream_t s) {
  const size_t n = source.n;
  const float* g = source.flat ? source.flat : acc;
  if (!nnz_dev) return SGB_ERR_NULL;
  if (n == 0) {
    cudaError_t e = cudaMemsetAsync(nnz_dev, 0, sizeof(int), s);
    return e == cudaSuccess ? SGB_OK : note_cuda_error(e);
  }
  const int st = check_common(g, n, idx_out, ws, ws_bytes);
  if (st != SGB_OK) return st;
  const Work work = work_for(n);
  ThrArgs a{g, acc, n, thr, work, carve(ws, work), idx_out, val_out, nnz_dev, static_cast<unsigned>(cap), dropped,
            aligned16(g) && (!acc || aligned16(acc))};
  if (work.dynamic) {
    cudaError_t e = cudaMemsetAsync(a.ws.counters->ticket, 0, sizeof(a.ws.counters->ticket), s);
    if (e != cudaSuccess) return note_cuda_error(e);
  }
  if (!source.flat)
    return cap ? launch_cooperative(thr_select_kernel<true, Pieces>, work.grid, a, source.pieces, s)
               : launch_cooperative(thr_select_kernel<false, Pieces>, work.grid, a, source.pieces, s);
  return cap ? launch_cooperative(thr_select_kernel<true, NoPieces>, work.grid, a, NoPieces{}, s)
             : launch_cooperative(thr_select_kernel<false, NoPieces>, work.grid, a, NoPieces{}, s);
}

bool gather_buckets(Buckets* b, const SparseBucket* buckets, size_t count, size_t* span) {
  size_t at = 0;
  b->count = 0;
  b->pieces.count = 0;
  Gradient g;
  for (size_t k = 0; k < count; ++k) {
    const SparseBucket& from = buckets[k];
    // (a bucket that lies back to back is one piece, with or without a residual)
    if (!from.acc || !aligned16(from.acc) || !gather(&g, from.tensors, from.sizes, from.count, from.acc)) return false;
    if (g.n == 0) continue;
    if (b->count == kBuckets || b->pieces.count + g.pieces.count > kPieces || at + g.n > kMaxBucketSpan) return false;
    b->tile[b->count] = static_cast<unsigned>(at / kTile);
    b->end[b->count] = static_cast<unsigned>(at + g.n);
    b->acc[b->count++] = from.acc;
    for (int p = 0; p < g.pieces.count; ++p) {
      b->pieces.off[b->pieces.count] = static_cast<unsigned>(at) + g.pieces.off[p];
      b->pieces.ptr[b->pieces.count++] = g.pieces.ptr[p];
    }
    at = (at + g.n + kTile - 1) / kTile * kTile;
  }
  b->pieces.off[b->pieces.count] = static_cast<unsigned>(at);
  *span = at;
  return at > 0;
}

// The sample takes 8 us, and pass 1 over s 16 us per 10^7 elements: it pays
// from there on, where every warp has two KB or more of elements to sample
// from.  k up to n / 12, so that bound and margin stay inside the lists (352
// entries per 2048 elements).  Margin: an eighth and four standard deviations.
// Not for integer keys, which are mostly 0 or tied.
inline unsigned sample_target(size_t n, size_t k, int mode, const Work& work) {
  if (mode != 0 || work.run != 4 || k > n / 12) return 0;
  double target = static_cast<double>(k) / static_cast<double>(n) * (work.grid * kWarps * 128.0);
  target += target / 8 + 4 * std::sqrt(target) + 16;
  return static_cast<unsigned>(target);
}

int topk_launch(const Gradient& source, float* acc, size_t k, int mode, int* idx_out, float* val_out, void* ws,
                size_t ws_bytes, cudaStream_t s, bool cleared = false) {
  const size_t n = source.n;
  if (n == 0 || k == 0) return SGB_OK;
  if (mode != 0 && mode != 1) return SGB_ERR_UNSUPPORTED;
  if (!val_out) return SGB_ERR_NULL;
  const float* g = source.flat ? source.flat : acc;
  const int st = check_common(g, n, idx_out, ws, ws_bytes);
  if (st != SGB_OK) return st;
  if (k > n) k = n;
  const Work work = work_for(n);
  TopkArgs a{g, acc, n, static_cast<unsigned>(k), sample_target(n, k, mode, work), work, carve(ws, work), idx_out, val_out,
             aligned16(g) && (!acc || aligned16(acc)), 0};
  if (!cleared) {
    const cudaError_t e = cudaMemsetAsync(a.ws.counters, 0, sizeof(Counters), s);
    if (e != cudaSuccess) return note_cuda_error(e);
  }
  if (!source.flat)
    return mode == 0 ? launch_cooperative(topk_select_kernel<0, Pieces>, work.grid, a, source.pieces, s)
                     : launch_cooperative(topk_select_kernel<1, Pieces>, work.grid, a, source.pieces, s);
  return mode == 0 ? launch_cooperative(topk_select_kernel<0, NoPieces>, work.grid, a, NoPieces{}, s)
                   : launch_cooperative(topk_select_kernel<1, NoPieces>, work.grid, a, NoPieces{}, s);
}

}  // namespace

// ---- forms used by the communicator (declared in sparse.cuh) ---------------
size_t sparse_buckets_span(const SparseBucket* buckets, size_t count) {
  Buckets b;
  size_t span = 0;
  return gather_buckets(&b, buckets, count, &span) ? span : 0;
}

size_t sparse_counter_bytes(size_t buckets) { return buckets * align256(sizeof(Counters)); }

int sparse_threshold_buckets(const SparseBucket* buckets, size_t count, float thr, int* payload, int* nnz_dev, void* ws,
                             size_t ws_bytes, cudaStream_t s, bool cleared) {
  Buckets b;
  size_t n = 0;
  if (!gather_buckets(&b, buckets, count, &n)) return SGB_ERR_UNSUPPORTED;
  const int st = check_common(b.acc[0], n, payload, ws, ws_bytes);
  if (st != SGB_OK) return st;
  const Work work = work_for(n);
  ThrArgs a{nullptr, nullptr, n, thr, work, carve(ws, work), payload, nullptr, nnz_dev, 0, nullptr, true};
  if (work.dynamic && !cleared) {
    cudaError_t e = cudaMemsetAsync(a.ws.counters->ticket, 0, sizeof(a.ws.counters->ticket), s);
    if (e != cudaSuccess) return note_cuda_error(e);
  }
  return launch_cooperative(thr_select_kernel<false, Buckets>, work.grid, a, b, s);
}

// The plan of a joint top-K selection; false where it takes a launch per bucket.
static bool topk_plan(const SparseBucket* buckets, const size_t* ks, size_t count, int mode, TopkBuckets* b, size_t* bytes,
                      size_t* sent) {
  if (count < 1 || count > kBuckets) return false;
  size_t total = 0;
  std::vector<size_t> sizes;
  for (size_t k = 0; k < count; ++k) {
    size_t n = 0;
    for (size_t t = 0; t < buckets[k].count; ++t) n += buckets[k].sizes[t];
    sizes.push_back(n);
    total += n;
  }
  if (total == 0) return false;
  const size_t most = max_grid();
  size_t index = 0, lists = 0, payload = 0, ctas = 0, pieces = 0;
  Gradient g;
  b->count = 0;
  for (size_t k = 0; k < count; ++k) {
    const size_t n = sizes[k];
    if (n && ks[k]) {
      if (!buckets[k].acc || !aligned16(buckets[k].acc) ||
          !gather(&g, buckets[k].tensors, buckets[k].sizes, buckets[k].count, buckets[k].acc) ||
          pieces + g.pieces.count > kPieces)
        return false;
      const int i = b->count++;
      size_t share = (most - count) * n / total;       // (each gets at least one)
      if (share < 1) share = 1;
      b->work[i] = work_for(n, share);
      b->first_cta[i] = static_cast<unsigned>(ctas);
      ctas += b->work[i].grid;
      b->n[i] = static_cast<unsigned>(n);
      b->k[i] = static_cast<unsigned>(ks[k] < n ? ks[k] : n);
      b->sample_target[i] = sample_target(n, b->k[i], mode, b->work[i]);
      b->at[i] = static_cast<unsigned>(payload);
      b->index_base[i] = static_cast<unsigned>(index);
      b->ws_off[i] = lists;
      b->acc[i] = buckets[k].acc;
      b->first_piece[i] = static_cast<int>(pieces);
      for (int p = 0; p <= g.pieces.count; ++p) b->off[pieces + i + p] = g.pieces.off[p];
      for (int p = 0; p < g.pieces.count; ++p) b->ptr[pieces + p] = g.pieces.ptr[p];
      pieces += g.pieces.count;
      b->first_piece[i + 1] = static_cast<int>(pieces);
      lists += lists_bytes(b->work[i]);
      payload += b->k[i];
    }
    index = (index + n + kTile - 1) / kTile * kTile;
  }
  if (index > kMaxBucketSpan || ctas > most) return false;
  b->first_cta[b->count] = static_cast<unsigned>(ctas);
  const size_t counters = sparse_counter_bytes(b->count);
  for (int i = 0; i < b->count; ++i) b->ws_off[i] += counters;
  *bytes = counters + lists;
  *sent = payload;
  return true;
}

// A list that one launch cannot take goes through several, of about as many buckets
// each (2.56e7 elements, the largest 1.8 % of 35 buckets: 1105 us a pass with a call per
// bucket, 270 in two groups).  Below 2^20 elements a list that one launch does not take
// keeps its calls, as sgb.h says.
constexpr size_t kLeastCut = size_t{1} << 20;
bool sparse_topk_buckets_cut(float* const* tensors, const size_t* sizes, const size_t* counts, size_t nbuckets,
                             std::vector<size_t>* ends) {
  if (nbuckets < 2) return false;
  const size_t launches = ceil_div(nbuckets, kBuckets), most = ceil_div(nbuckets, launches);
  size_t cuts = 0, total = 0, first = 0, span = 0, pieces = 0, t = 0;
  for (size_t k = 0; k < nbuckets; ++k) {
    const float* end = nullptr;
    size_t n = 0, runs = 0;
    for (const size_t last = t + counts[k]; t < last; ++t) {
      if (!sizes[t]) continue;
      runs += tensors[t] != end;                       // back to back with the one before: the same piece
      end = tensors[t] + sizes[t];
      n += sizes[t];
    }
    const size_t room = (n + kTile - 1) / kTile * kTile;
    if (room > kMaxBucketSpan || runs > kPieces) return false;
    if (k - first == most || span + room > kMaxBucketSpan || pieces + runs > kPieces) {
      if (ends) ends->push_back(k);
      ++cuts;
      first = k;
      span = pieces = 0;
    }
    span += room;
    pieces += runs;
    total += n;
  }
  if (ends) ends->push_back(nbuckets);
  return cuts == 0 || total >= kLeastCut;
}

size_t sparse_topk_buckets_bytes(const SparseBucket* buckets, const size_t* ks, size_t count, int mode, size_t* counters) {
  TopkBuckets b;
  size_t bytes = 0, sent = 0;
  if (!topk_plan(buckets, ks, count, mode, &b, &bytes, &sent)) return 0;
  *counters = sparse_counter_bytes(b.count);
  return bytes + 256;
}

int sparse_topk_buckets(const SparseBucket* buckets, const size_t* ks, size_t count, int mode, int* payload, int* sent,
                        void* ws, size_t ws_bytes, cudaStream_t s, bool cleared) {
  TopkBuckets b;
  size_t bytes = 0, total = 0;
  if (!topk_plan(buckets, ks, count, mode, &b, &bytes, &total)) return SGB_ERR_UNSUPPORTED;
  if (!ws || ws_bytes < bytes || (reinterpret_cast<uintptr_t>(ws) & 255u)) return SGB_ERR_WORKSPACE;
  *sent = static_cast<int>(total);
  if (b.count == 0) return SGB_OK;
  b.ws = static_cast<char*>(ws);
  b.idx_out = payload;
  b.val_out = reinterpret_cast<float*>(payload) + total;
  cudaError_t e = cleared ? cudaSuccess : cudaMemsetAsync(ws, 0, sparse_counter_bytes(b.count), s);
  if (e != cudaSuccess) return note_cuda_error(e);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(b.first_cta[b.count]);
  cfg.blockDim = dim3(kBlock);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;       // all CTAs are resident, or the launch fails
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  e = mode == 0 ? cudaLaunchKernelEx(&cfg, topk_buckets_kernel<0>, b) : cudaLaunchKernelEx(&cfg, topk_buckets_kernel<1>, b);
  return e == cudaSuccess ? launch_status() : note_cuda_error(e);
}

int sparse_dense_buckets(const int* payload, int known, const int* nnz_dev, const SparseBucket* buckets, size_t count,
                         cudaStream_t s, const SparseUpdate* update, const SparseClear& clear) {
  std::vector<float*> tensors, params, moments;
  std::vector<size_t> sizes;
  const int none[1] = {known};
  size_t at = 0;
  for (size_t k = 0; k < count; ++k) {
    size_t n = 0;
    for (size_t t = 0; t < buckets[k].count; ++t, ++at) {
      tensors.push_back(buckets[k].tensors[t]);
      sizes.push_back(buckets[k].sizes[t]);
      if (update) params.push_back(update->params[at]);
      if (update) moments.push_back(update->moments ? update->moments[at] : nullptr);
      n += buckets[k].sizes[t];
    }
    tensors.push_back(nullptr);                        // the gap up to the next tile
    params.push_back(nullptr);
    moments.push_back(nullptr);
    sizes.push_back((kTile - n % kTile) % kTile);
  }
  const SparseUpdate joint{update ? update->sgd : nullptr, params.data(), moments.data()};
  return sparse_dense_sum(payload, 0, 0, none, nnz_dev, 1, tensors.data(), sizes.data(), tensors.size(), s,
                          update ? &joint : nullptr, clear);
}

int sparse_faults(unsigned* flags) {
  const cudaError_t e = cudaMemcpyFromSymbol(flags, g_topk_faults, sizeof(unsigned));
  return e == cudaSuccess ? SGB_OK : note_cuda_error(e);
}

bool sparse_selects_from(float* const* tensors, const size_t* sizes, size_t count, const float* acc) {
  Gradient g;
  return gather(&g, tensors, sizes, count, acc);
}

int sparse_threshold_packed(float* const* tensors, const size_t* sizes, size_t count, float* acc, float thr,
                            int* payload, int* nnz_dev, void* ws, size_t ws_bytes, cudaStream_t s) {
  Gradient g;
  if (!gather(&g, tensors, sizes, count, acc)) return SGB_ERR_UNSUPPORTED;
  return threshold_select(g, acc, thr, payload, nullptr, nnz_dev, 0, nullptr, ws, ws_bytes, s);
}

int sparse_threshold_bounded(float* const* tensors, const size_t* sizes, size_t count, float* acc, float thr,
                             int* payload, size_t cap, int* nnz_dev, unsigned long long* dropped_dev, void* ws,
                             size_t ws_bytes, cudaStream_t s) {
  if (cap == 0 || cap > 0x7fffffffu || !dropped_dev) return SGB_ERR_SIZE;
  Gradient g;
  if (!gather(&g, tensors, sizes, count, acc)) return SGB_ERR_UNSUPPORTED;
  return threshold_select(g, acc, thr, payload, nullptr, nnz_dev, cap, dropped_dev, ws, ws_bytes, s);
}

int sparse_topk(float* const* tensors, const size_t* sizes, size_t count, float* acc, size_t k, int mode, int* idx_out,
                float* val_out, void* ws, size_t ws_bytes, cudaStream_t s, bool cleared) {
  Gradient g;
  if (!gather(&g, tensors, sizes, count, acc)) return SGB_ERR_UNSUPPORTED;
  return topk_launch(g, acc, k, mode, idx_out, val_out, ws, ws_bytes, s, cleared);
}

int sparse_dense_sum(const int* payload, size_t stride, size_t val_off, const int* counts, const int* counts_dev,
                     int world, float* const* tensors, const size_t* sizes, size_t ntensors, cudaStream_t s,
                     const SparseUpdate* update, const SparseClear& clear) {
  DenseArgs a;
  DenseUpdate u;
  if (update && world != 1) return SGB_ERR_UNSUPPORTED;
  if (update) u.sgd = *update->sgd;
  if (world < 1 || world > kMaxDenseRanks) return SGB_ERR_UNSUPPORTED;
  if (clear.bytes > clear.room) return SGB_ERR_WORKSPACE;
  a.clear = static_cast<uint4*>(clear.at);
  a.clear_vecs = static_cast<unsigned>(clear.bytes / sizeof(uint4));
  a.payload = payload;
  a.stride = stride;
  a.val_off = val_off;
  a.counts_dev = counts_dev;
  size_t n = 0;
  for (size_t k = 0; k < ntensors; ++k) n += sizes[k];
  a.most = static_cast<unsigned>(val_off ? val_off : n);
  a.world = world;
  for (int r = 0; r < world; ++r) a.counts[r] = counts_dev ? 0 : counts[r];
  size_t at = 0;
  for (size_t k = 0; k < ntensors;) {
    a.first = at;
    a.targets = 0;
    while (k < ntensors && a.targets < kDenseTargets) {
      if (sizes[k]) {
        // tensors that lie back to back are one target
        const int last = a.targets - 1;
        const size_t run = a.targets ? at - a.off[last] : 0;
        const bool joined = a.targets && a.ptr[last] && a.ptr[last] + run == tensors[k] &&
                            (!update || (u.p[last] + run == update->params[k] &&
                                         (!u.sgd.use_momentum || u.m[last] + run == update->moments[k])));
        if (!joined) {
          if (update) {
            u.p[a.targets] = update->params[k];
            u.m[a.targets] = u.sgd.use_momentum ? update->moments[k] : nullptr;
          }
          a.off[a.targets] = at;
          a.ptr[a.targets++] = tensors[k];
        }
        at += sizes[k];
      }
      ++k;
    }
    if (!a.targets) continue;
    a.last = at;
    a.off[a.targets] = at;
    const size_t tiles = ceil_div(a.last - a.first, kDenseTile);
    // A CTA's tiles: few enough that those whose entries crowd (the first elements of a
    // bucket whose keys tie) are spread over the GPU, where they are updated as well.  As many
    // as fill the GPU once, 16, 8 and 4 of them: 3.1e7 elements, the first 4.8 % sent, 218 / 218 /
    // 195 / 185 us a pass; 1e8, 1 % anywhere, 629 / 609 / 601 / 594; 2.56e7 in 16 buckets 172 /
    // 172 / 170 / 165.  Without the update 5e7 elements at 2.6 standard deviations took 323
    // instead of 317.
    const size_t even = ceil_div(tiles, static_cast<size_t>(sm_count()) * (update ? kUpdateCtas : 8));
    const unsigned per = static_cast<unsigned>(update && even > kMostTiles ? kMostTiles : even);
    const dim3 grid(static_cast<unsigned>(ceil_div(tiles, per)));
    int st;
    if (update) {
      static std::atomic<bool> ready[64];
      st = more_shared_memory(dense_from_payloads_kernel<true, DenseUpdate>, kUpdateStage, ready);
      if (st == SGB_OK)
        st = launch_ex(dense_from_payloads_kernel<true, DenseUpdate>, grid, dim3(kBlock), kUpdateStage, s, 0, true, a, per, u);
    } else {
      st = launch_ex(world == 1 ? dense_from_payloads_kernel<true, NoUpdate> : dense_from_payloads_kernel<false, NoUpdate>,
                     grid, dim3(kBlock), 0, s, 0, true, a, per, NoUpdate{});
    }
    if (st != SGB_OK) return st;
    a.clear_vecs = 0;
  }
  return launch_status();
}

}  // namespace sgb

using namespace sgb;

extern "C" {

size_t sgb_sparse_workspace_bytes(size_t n) { return n ? workspace_bytes(n) : 256; }

size_t sgb_sparse_topk_plan(const size_t* sizes, const size_t* ks, size_t nbuckets, int mode, size_t* counters) {
  if (!sizes || !ks || !counters || nbuckets > kBuckets) return 0;
  float* const somewhere = reinterpret_cast<float*>(static_cast<uintptr_t>(256));   // never followed
  std::vector<SparseBucket> buckets;
  for (size_t k = 0; k < nbuckets; ++k) buckets.push_back({&somewhere, sizes + k, 1, somewhere});
  return sparse_topk_buckets_bytes(buckets.data(), ks, nbuckets, mode, counters);
}

int sgb_topk_count(float ratio, size_t n) {
  // (int)ceil(threshold * num) evaluated in fp32, as the reference does
  // (float * size_t -> float).
  const float prod = ratio * static_cast<float>(n);
  float c = ceilf(prod);
  if (c < 0.f) c = 0.f;
  if (c > static_cast<float>(n)) return static_cast<int>(n);
  return static_cast<int>(c);
}

int sgb_sparse_threshold_f32(const float* g, float* acc, size_t n, float thr, int32_t* idx_out,
                             float* val_out, int32_t* nnz_dev, void* ws, size_t ws_bytes,
                             void* stream) {
  if (n && (!g || !val_out)) return SGB_ERR_NULL;
  Gradient source;
  source.flat = g;
  source.n = n;
  return threshold_select(source, acc, thr, idx_out, val_out, nnz_dev, 0, nullptr, ws, ws_bytes, as_stream(stream));
}

int sgb_sparse_topk_f32(const float* g, float* acc, float* sum_scratch, size_t n, size_t k,
                        int mode, int32_t* idx_out, float* val_out, void* ws, size_t ws_bytes,
                        void* stream) {
  (void)sum_scratch;   // kept in the signature; the sum lives in acc (or is g itself without a residual)
  if (n && k && !g) return SGB_ERR_NULL;
  Gradient source;
  source.flat = g;
  source.n = n;
  return topk_launch(source, acc, k, mode, idx_out, val_out, ws, ws_bytes, as_stream(stream));
}

int sgb_sparse_faults(unsigned* flags) { return flags ? sparse_faults(flags) : SGB_ERR_NULL; }

int sgb_scatter_add_f32(const int32_t* idx, const float* val, size_t count,
                        const int32_t* count_dev, float* dst, size_t n, void* stream) {
  if (!count_dev && count == 0) return SGB_OK;
  if (!idx || !val || !dst) return SGB_ERR_NULL;
  const size_t guess = count_dev ? (count ? count : n) : count;
  unsigned grid = capped_grid(guess, kBlock, 8);
  scatter_add_kernel<<<grid, kBlock, 0, as_stream(stream)>>>(idx, val, count, count_dev, dst, n);
  return launch_status();
}

}  // extern "C"
