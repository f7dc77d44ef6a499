// Internal interface of the sparsifiers, used by the communicator.
#pragma once
#include <vector>

#include "sgd.cuh"

namespace sgb {

constexpr int kMaxDenseRanks = 64;

// Whether the selectors can read this bucket from its tensors: they lie back to
// back, or there are at most 256 runs of them and an aligned residual buffer.
bool sparse_selects_from(float* const* tensors, const size_t* sizes, size_t count, const float* acc);

// Threshold selection with residual update and packed payload [idx(nnz) | val(nnz)]
// (int32 view); the payload length lands in *nnz_dev.
int sparse_threshold_packed(float* const* tensors, const size_t* sizes, size_t count, float* acc, float thr,
                            int* payload, int* nnz_dev, void* ws, size_t ws_bytes, cudaStream_t s);

// Capacity-bounded form: payload [idx(cap) | val(cap)]; selected entries beyond
// the first `cap` (index order) stay in the residual and are counted in
// *dropped_dev (a device counter the caller owns).  *nnz_dev is the full count.
int sparse_threshold_bounded(float* const* tensors, const size_t* sizes, size_t count, float* acc, float thr,
                             int* payload, size_t cap, int* nnz_dev, unsigned long long* dropped_dev, void* ws,
                             size_t ws_bytes, cudaStream_t s);

// Several buckets at once, each with an aligned residual, as one selection: the
// payload's indices are in a joint space of sparse_buckets_span() elements in
// which bucket k starts at the next multiple of 512 behind bucket k - 1.  The
// span is 0 where the list has to be cut (more than 32 buckets, 256 runs of
// tensors or kMaxBucketSpan elements).
struct SparseBucket {
  float* const* tensors;
  const size_t* sizes;
  size_t count;
  float* acc;
};
constexpr size_t kMaxBucketSpan = size_t{1} << 25;
size_t sparse_buckets_span(const SparseBucket* buckets, size_t count);
int sparse_threshold_buckets(const SparseBucket* buckets, size_t count, float thr, int* payload, int* nnz_dev, void* ws,
                             size_t ws_bytes, cudaStream_t s, bool cleared = false);
// The counters of a selection are the first bytes of its workspace and are 0 when it
// starts: set so ahead of it, unless the caller says that they are (`cleared`).  A dense
// sum behind the selection does that for the next one on its way (`clear`).
size_t sparse_counter_bytes(size_t buckets);
struct SparseClear {
  void* at = nullptr;
  size_t bytes = 0;      // a multiple of 256
  size_t room = 0;       // what there is at `at`; more than that is refused
};
// The SGD update that a dense sum ends in: parameters (and momentum buffers) of the
// tensors, in their order.
struct SparseUpdate {
  const SgdArgs* sgd;
  float* const* params;
  float* const* moments;   // null without momentum
};
// Top-K of several buckets (the first ks[k] of bucket k by size) by one launch, into
// a payload of the same joint space; *sent: its length.  sparse_topk_buckets_bytes:
// of workspace, 0 where one launch does not take them, and how much of its start is
// counters: those of the buckets that it selects from (one without elements, or of
// which nothing is sent, has none).  sparse_topk_buckets_cut: whether
// launches of several buckets each take a list, by sizes and places alone, before
// anything is prepared, and where each ends (`ends` may be null).
bool sparse_topk_buckets_cut(float* const* tensors, const size_t* sizes, const size_t* counts, size_t nbuckets,
                             std::vector<size_t>* ends);
size_t sparse_topk_buckets_bytes(const SparseBucket* buckets, const size_t* ks, size_t count, int mode, size_t* counters);
int sparse_topk_buckets(const SparseBucket* buckets, const size_t* ks, size_t count, int mode, int* payload, int* sent,
                        void* ws, size_t ws_bytes, cudaStream_t s, bool cleared = false);
// The dense gradients of such a payload, back into the buckets' tensors; its length
// is on the device, or (nnz_dev null) `known`.
int sparse_dense_buckets(const int* payload, int known, const int* nnz_dev, const SparseBucket* buckets, size_t count,
                         cudaStream_t s, const SparseUpdate* update = nullptr, const SparseClear& clear = {});

// Top-K selection (see sgb_sparse_topk_f32) from a tensor list.
int sparse_topk(float* const* tensors, const size_t* sizes, size_t count, float* acc, size_t k, int mode, int* idx_out,
                float* val_out, void* ws, size_t ws_bytes, cudaStream_t s, bool cleared = false);

// Dense sum of `world` payloads (ascending indices, rank r at payload + r *
// stride words) into the tensors, which cover the index space in list order.
// Values start val_off words behind the indices, or, with val_off == 0, right
// behind the rank's own count.  counts: host array, or counts_dev on the device
// (then clamped to val_off, or to the size of the index space).  update: one rank only.
int sparse_dense_sum(const int* payload, size_t stride, size_t val_off, const int* counts, const int* counts_dev,
                     int world, float* const* tensors, const size_t* sizes, size_t ntensors, cudaStream_t s,
                     const SparseUpdate* update = nullptr, const SparseClear& clear = {});

// Rounds the tensors to fp16 and back, in place (multi_tensor.cu).
int round_f16_multi(void* const* tensors, const size_t* sizes, size_t count, cudaStream_t s);

}  // namespace sgb
