// Data-parallel gradient communicator: dense all-reduce (direct and bucketed),
// fp16-compressed all-reduce, and sparsified all-gather (threshold / top-K with
// residual correction), one process per GPU over NCCL on NVLink / NVSwitch.
//
// It keeps the reference communicator's observable structure - a compute
// stream plus three side streams (c1: pre-processing, s: NCCL, c2:
// post-processing) chained by events, staging buffers of maxSize elements,
// sum semantics (the caller divides by the world size) - and replaces the
// per-tensor memcpy / cast / thrust / cuSPARSE passes around the collectives
// by the fused kernels of this library:
//   stage   = one multi-tensor pack (+ fp32->fp16 cast) launch per call
//   flush   = collective + one multi-tensor unpack (+ fp16->fp32 cast) launch
//   sparse  = residual + select + order-preserving compaction, radix select
//             instead of a full sort, one scatter-add launch per rank.
// Each cross-stream edge has its own event.  No kernel here touches another
// GPU's memory: remote data reaches local HBM through NCCL only.
#include <nccl.h>

#include <atomic>
#include <cstring>
#include <new>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include <string>

#include "comm_order.h"
#include "common.cuh"
#include "sparse.cuh"

namespace {
std::atomic<int> g_last_nccl_error{0};

int nccl_fail(ncclResult_t r) {
  g_last_nccl_error.store(static_cast<int>(r));
  return SGB_ERR_NCCL;
}
}  // namespace

#define CU(call)                                            \
  do {                                                      \
    cudaError_t e__ = (call);                               \
    if (e__ != cudaSuccess) return sgb::note_cuda_error(e__); \
  } while (0)
#define NC(call)                                   \
  do {                                             \
    ncclResult_t r__ = (call);                     \
    if (r__ != ncclSuccess) return nccl_fail(r__); \
  } while (0)
#define OK(call)                     \
  do {                               \
    int s__ = (call);                \
    if (s__ != SGB_OK) return s__;   \
  } while (0)

struct sgb_comm {
  int rank = 0, world = 1, device = 0;
  ncclComm_t nccl = nullptr;
  size_t max_elems = 0;
  float* send = nullptr;   // fusedSendBuff
  float* recv = nullptr;   // fusedRecvBuff
  __half* send_h = nullptr;    // staging bucket in fp16
  __half* recv_h = nullptr;
  __half* dsend_h = nullptr;   // direct (unbucketed) fp16 synch: never aliases a half-filled bucket
  __half* drecv_h = nullptr;
  // sparse path (allocated at first use)
  int* pay_recv = nullptr;     // world * 2 * max_elems words
  void* ws = nullptr;
  size_t ws_bytes = 0;
  // A sparse exchange between its selection and its all-gather.  Two may be
  // open at a time, so that the next bucket's selection runs while the host
  // waits for this one's counts.
  struct Sparse {
    int* pay_send = nullptr;     // [idx | val], 2 * max_elems words
    int* nnz_dev = nullptr;      // [0] own count, [1 .. world] all ranks
    int* nnz_host = nullptr;     // pinned, world entries
    cudaEvent_t selected = nullptr;  // behind the selection on c1
    cudaEvent_t counted = nullptr;   // behind the counts' copy to the host
    cudaEvent_t consumed = nullptr;  // behind the dense sum on c2 that read pay_send (one rank)
    size_t n = 0, nnz_max = 0, capacity = 0;
    int topk = 0;
    const char* op_name = "";
    std::vector<float*> tensors;
    std::vector<size_t> sizes;
  };
  Sparse sparse[2];
  // One rank's joint selection over several buckets; grows with the largest span
  // that was asked for (at most kMaxBucketSpan), freed with the communicator.
  int *joint_pay = nullptr, *joint_nnz = nullptr;
  void* joint_ws = nullptr;
  size_t joint_elems = 0, joint_ws_bytes = 0;
  // How many bytes of counters at the start of a workspace the last exchange's dense sum
  // has set to 0; never again once a graph holds the workspace (its replays use it too).
  struct Cleared {
    size_t bytes = 0;
    bool captured = false;
  } ws_clear, joint_clear;
  std::vector<void*> joint_retired;
  unsigned sparse_begun = 0, sparse_ended = 0;
  unsigned long long* dropped_dev = nullptr;   // entries the bounded threshold form left for later calls
  int topk_mode = 1;           // 1 = the reference comparator's key, 0 = |value|
  cudaStream_t s = nullptr, c1 = nullptr, c2 = nullptr;
  bool own_streams = true;     // false after sgb_comm_use_streams: the caller's streams are not destroyed
  cudaEvent_t ev_compute = nullptr, ev_c1 = nullptr, ev_s = nullptr, ev_c2 = nullptr,
              ev_c2_done = nullptr;
  size_t send_off = 0;         // elements staged since the last flush
  // Which side streams received work since the last wait() (only those are
  // joined, so a wait() issued while the compute stream is being captured
  // never touches a stream outside the capture) and whether c2 still reads a
  // receive buffer: the state of the edge planner in comm_order.h.
  sgb::order::State order;
  int result_stream = sgb::order::kStreamS;   // where the last call's result can be consumed
  // Per-phase device timing (off by default; never during stream capture):
  // one event pair per phase on the stream that runs it, named like the
  // reference's operations ("Dist_s_fusedSynch_allreduce", ...), measured
  // from an origin event on the compute stream.
  bool profiling = false;
  cudaEvent_t prof_origin = nullptr;
  struct Range {
    std::string name;
    cudaEvent_t start, end;
  };
  std::vector<Range> ranges;
  size_t open_range = 0;
  std::vector<void*> registered;   // ncclCommRegister handles (user buffers reduced in place)
  // Staging is deferred: a stage call only records the tensors; the bytes are
  // gathered by ONE multi-tensor pack launch when the bucket is flushed (the
  // tensors must stay alive until then anyway - the flush writes into them).
  std::vector<void*> pend_ptrs;
  std::vector<size_t> pend_sizes;
  size_t pend_off = 0;         // staging-buffer offset of the first pending tensor
  int pend_half = 0;           // pending tensors go to the fp16 staging buffer
};

namespace {

int edge(cudaEvent_t ev, cudaStream_t from, cudaStream_t to) {
  CU(cudaEventRecord(ev, from));
  CU(cudaStreamWaitEvent(to, ev, 0));
  return SGB_OK;
}

cudaStream_t side(const sgb_comm* c, int which) {
  return which == sgb::order::kStreamS ? c->s : (which == sgb::order::kStreamC1 ? c->c1 : c->c2);
}

// Emits the edges of one phase of a planned call (see comm_order.h), in a
// fixed order.  Every edge re-records its event; a wait takes the state of the
// event at the time of the wait, so an event can serve many edges in a row.
int emit(sgb_comm* c, unsigned edges, cudaStream_t compute, int slot = 0) {
  using namespace sgb::order;
  if (edges & kComputeToC1) OK(edge(c->ev_compute, compute, c->c1));
  if (edges & kComputeToS) OK(edge(c->ev_compute, compute, c->s));
  if (edges & kC1ToS) OK(edge(c->ev_c1, c->c1, c->s));
  if (edges & kC2DoneToS) CU(cudaStreamWaitEvent(c->s, c->ev_c2_done, 0));
  if (edges & (kSToC1 | kSToC2)) {
    CU(cudaEventRecord(c->ev_s, c->s));
    if (edges & kSToC1) CU(cudaStreamWaitEvent(c->c1, c->ev_s, 0));
    if (edges & kSToC2) CU(cudaStreamWaitEvent(c->c2, c->ev_s, 0));
  }
  if (edges & kMarkC2Done) CU(cudaEventRecord(c->ev_c2_done, c->c2));
  const sgb_comm::Sparse& x = c->sparse[slot];
  if (edges & kConsumedToC1) CU(cudaStreamWaitEvent(c->c1, x.consumed, 0));
  if (edges & kMarkSelected) CU(cudaEventRecord(x.selected, c->c1));
  if (edges & kSelectedToS) CU(cudaStreamWaitEvent(c->s, x.selected, 0));
  if (edges & kSelectedToC2) CU(cudaStreamWaitEvent(c->c2, x.selected, 0));
  if (edges & kMarkConsumed) CU(cudaEventRecord(x.consumed, c->c2));
  if (edges & kSToCompute) OK(edge(c->ev_s, c->s, compute));
  if (edges & kC1ToCompute) OK(edge(c->ev_c1, c->c1, compute));
  if (edges & kC2ToCompute) OK(edge(c->ev_c2, c->c2, compute));
  return SGB_OK;
}

sgb::order::Step plan_call(sgb_comm* c, int call) {
  sgb::order::Step p = sgb::order::plan(c->order, call);
  c->result_stream = p.result_stream;
  return p;
}

// True also if the question fails (the default stream beside another stream's
// capture): no place for a timing event or an allocation either.
bool capturing(cudaStream_t s) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) == cudaSuccess) return st != cudaStreamCaptureStatusNone;
  cudaGetLastError();
  return true;
}

// A named phase on one of the side streams: an NVTX range around the enqueue
// and, while profiling is on, an event pair on that stream.
struct Phase {
  sgb_comm* c;
  cudaStream_t stream;
  bool timed = false;
  size_t slot = 0;
  Phase(sgb_comm* comm, const char* name, int which) : c(comm), stream(side(comm, which)) {
    nvtxRangePushA(name);
    if (!c->profiling || capturing(stream)) return;
    sgb_comm::Range r;
    r.name = name;
    if (cudaEventCreate(&r.start) != cudaSuccess) return;
    if (cudaEventCreate(&r.end) != cudaSuccess) {
      cudaEventDestroy(r.start);
      return;
    }
    cudaEventRecord(r.start, stream);
    slot = c->ranges.size();
    c->ranges.push_back(r);
    timed = true;
  }
  ~Phase() {
    if (timed) cudaEventRecord(c->ranges[slot].end, stream);
    nvtxRangePop();
  }
};

void drop_ranges(sgb_comm* c) {
  for (auto& r : c->ranges) {
    cudaEventDestroy(r.start);
    if (r.end) cudaEventDestroy(r.end);
  }
  c->ranges.clear();
}

// Packs the deferred tensors into the staging buffer on c1.  The caller has
// emitted compute -> c1 for this call already (every staged gradient was
// produced before this point).
int pack_pending(sgb_comm* c, const char* name) {
  if (c->pend_ptrs.empty()) return SGB_OK;
  Phase ph(c, name, sgb::order::kStreamC1);
  if (c->pend_half)
    OK(sgb_pack_f32_to_f16(c->pend_ptrs.data(), c->pend_sizes.data(), c->pend_ptrs.size(), c->send_h,
                           c->pend_off, c->c1));
  else
    OK(sgb_pack_f32(c->pend_ptrs.data(), c->pend_sizes.data(), c->pend_ptrs.size(), c->send,
                    c->pend_off, c->c1));
  c->pend_ptrs.clear();
  c->pend_sizes.clear();
  return SGB_OK;
}

// A bucket of the other precision is still pending: it is packed now, ordered
// after the compute stream.
int pack_other_kind(sgb_comm* c, cudaStream_t compute, const char* name) {
  OK(emit(c, plan_call(c, sgb::order::kStageCopy).pre, compute));
  return pack_pending(c, name);
}

void defer(sgb_comm* c, void* const* tensors, const size_t* sizes, size_t count, int half) {
  if (c->pend_ptrs.empty()) {
    c->pend_off = c->send_off;
    c->pend_half = half;
  }
  for (size_t i = 0; i < count; ++i) {
    c->pend_ptrs.push_back(tensors[i]);
    c->pend_sizes.push_back(sizes[i]);
  }
}

// One rank, and the flush hands back exactly the tensors that were staged.
bool alone(const sgb_comm* c, void* const* tensors, const size_t* sizes, size_t count, size_t total, int half) {
  if (c->world != 1 || c->pend_half != half || c->pend_off != 0 || c->pend_ptrs.size() != count || c->send_off != total)
    return false;
  for (size_t i = 0; i < count; ++i)
    if (c->pend_ptrs[i] != tensors[i] || c->pend_sizes[i] != sizes[i]) return false;
  return true;
}

int half_init(sgb_comm* c) {
  if (c->send_h) return SGB_OK;
  CU(cudaMalloc(&c->send_h, c->max_elems * sizeof(__half)));
  CU(cudaMalloc(&c->recv_h, c->max_elems * sizeof(__half)));
  CU(cudaMalloc(&c->dsend_h, c->max_elems * sizeof(__half)));
  CU(cudaMalloc(&c->drecv_h, c->max_elems * sizeof(__half)));
  return SGB_OK;
}

int sparse_init(sgb_comm* c) {
  if (c->dropped_dev) return SGB_OK;
  const size_t n = c->max_elems;
  c->ws_bytes = sgb_sparse_workspace_bytes(n);
  CU(cudaMalloc(&c->ws, c->ws_bytes));
  for (sgb_comm::Sparse& x : c->sparse) {
    CU(cudaMalloc(&x.pay_send, 2 * n * sizeof(int)));
    CU(cudaMalloc(&x.nnz_dev, sizeof(int) * (c->world + 1)));
    CU(cudaMallocHost(&x.nnz_host, sizeof(int) * c->world));
    // the host polls for the counts: it has the next calls to issue, and a
    // blocking wait woke it 50-100 us late
    CU(cudaEventCreateWithFlags(&x.selected, cudaEventDisableTiming));
    CU(cudaEventCreateWithFlags(&x.counted, cudaEventDisableTiming));
    CU(cudaEventCreateWithFlags(&x.consumed, cudaEventDisableTiming));
  }
  if (c->world > 1) CU(cudaMalloc(&c->pay_recv, 2 * n * sizeof(int) * static_cast<size_t>(c->world)));
  CU(cudaMalloc(&c->dropped_dev, sizeof(unsigned long long)));
  CU(cudaMemset(c->dropped_dev, 0, sizeof(unsigned long long)));
  return SGB_OK;
}

size_t total_of(const size_t* sizes, size_t count) {
  size_t t = 0;
  for (size_t i = 0; i < count; ++i) t += sizes[i];
  return t;
}

int check_list(void* const* tensors, const size_t* sizes, size_t count) {
  if (count == 0) return SGB_ERR_SIZE;  // the reference CHECKs t.size() > 0
  if (!tensors || !sizes) return SGB_ERR_NULL;
  for (size_t i = 0; i < count; ++i)
    if (sizes[i] && !tensors[i]) return SGB_ERR_NULL;
  return SGB_OK;
}

}  // namespace

extern "C" {

int sgb_last_nccl_error(void) { return g_last_nccl_error.load(); }

int sgb_comm_unique_id_bytes(void) { return static_cast<int>(sizeof(ncclUniqueId)); }

int sgb_comm_get_unique_id(void* id_out) {
  if (!id_out) return SGB_ERR_NULL;
  ncclUniqueId id;
  NC(ncclGetUniqueId(&id));
  std::memcpy(id_out, &id, sizeof(id));
  return SGB_OK;
}

int sgb_comm_create(sgb_comm** out, int rank, int world, const void* unique_id, size_t max_elems) {
  return sgb_comm_create_ex(out, rank, world, unique_id, max_elems, 0, 0);
}

int sgb_comm_register(sgb_comm* c, void* buffer, size_t bytes) {
  if (!c || !buffer) return SGB_ERR_NULL;
  if (bytes == 0) return SGB_ERR_SIZE;
  void* handle = nullptr;
  NC(ncclCommRegister(c->nccl, buffer, bytes, &handle));
  c->registered.push_back(handle);
  return SGB_OK;
}

int sgb_comm_create_ex(sgb_comm** out, int rank, int world, const void* unique_id, size_t max_elems,
                       int min_ctas, int max_ctas) {
  if (!out || !unique_id) return SGB_ERR_NULL;
  if (world < 1 || rank < 0 || rank >= world || max_elems == 0) return SGB_ERR_SIZE;
  if (max_elems > 0x7fffffffu) return SGB_ERR_SIZE;  // collective counts and 1-based indices are int32
  sgb_comm* c = new (std::nothrow) sgb_comm();
  if (!c) return SGB_ERR_STATE;
  c->rank = rank;
  c->world = world;
  c->max_elems = max_elems;
  *out = c;  // handed out early so a failed create can still be destroyed
  CU(cudaGetDevice(&c->device));
  ncclUniqueId id;
  std::memcpy(&id, unique_id, sizeof(id));
  if (min_ctas > 0 || max_ctas > 0) {
    ncclConfig_t cfg = NCCL_CONFIG_INITIALIZER;
    if (min_ctas > 0) cfg.minCTAs = min_ctas;
    if (max_ctas > 0) cfg.maxCTAs = max_ctas;
    NC(ncclCommInitRankConfig(&c->nccl, world, id, rank, &cfg));
  } else {
    NC(ncclCommInitRank(&c->nccl, world, id, rank));
  }
  CU(cudaMalloc(&c->send, max_elems * sizeof(float)));
  CU(cudaMalloc(&c->recv, max_elems * sizeof(float)));
  // Highest priority: the collectives and their small pack / unpack kernels
  // should start as soon as their inputs exist instead of queueing behind the
  // large backward kernels of the compute stream.
  int prio_lo = 0, prio_hi = 0;
  CU(cudaDeviceGetStreamPriorityRange(&prio_lo, &prio_hi));
  CU(cudaStreamCreateWithPriority(&c->s, cudaStreamNonBlocking, prio_hi));
  CU(cudaStreamCreateWithPriority(&c->c1, cudaStreamNonBlocking, prio_hi));
  CU(cudaStreamCreateWithPriority(&c->c2, cudaStreamNonBlocking, prio_hi));
  cudaEvent_t* evs[] = {&c->ev_compute, &c->ev_c1, &c->ev_s, &c->ev_c2, &c->ev_c2_done};
  for (cudaEvent_t* e : evs) CU(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  return SGB_OK;
}

int sgb_comm_destroy(sgb_comm* c) {
  if (!c) return SGB_OK;
  if (c->s) cudaStreamSynchronize(c->s);
  if (c->c1) cudaStreamSynchronize(c->c1);
  if (c->c2) cudaStreamSynchronize(c->c2);
  if (c->nccl) {
    for (void* h : c->registered) ncclCommDeregister(c->nccl, h);
    ncclCommDestroy(c->nccl);
  }
  void* bufs[] = {c->send, c->recv, c->send_h, c->recv_h, c->dsend_h, c->drecv_h, c->pay_recv, c->ws};
  for (void* b : bufs)
    if (b) cudaFree(b);
  for (sgb_comm::Sparse& x : c->sparse) {
    if (x.pay_send) cudaFree(x.pay_send);
    if (x.nnz_dev) cudaFree(x.nnz_dev);
    if (x.nnz_host) cudaFreeHost(x.nnz_host);
    if (x.selected) cudaEventDestroy(x.selected);
    if (x.counted) cudaEventDestroy(x.counted);
    if (x.consumed) cudaEventDestroy(x.consumed);
  }
  if (c->dropped_dev) cudaFree(c->dropped_dev);
  if (c->joint_pay) cudaFree(c->joint_pay);
  if (c->joint_nnz) cudaFree(c->joint_nnz);
  if (c->joint_ws) cudaFree(c->joint_ws);
  for (void* b : c->joint_retired) cudaFree(b);
  drop_ranges(c);
  cudaEvent_t evs[] = {c->ev_compute, c->ev_c1, c->ev_s, c->ev_c2, c->ev_c2_done, c->prof_origin};
  for (cudaEvent_t e : evs)
    if (e) cudaEventDestroy(e);
  cudaStream_t ss[] = {c->s, c->c1, c->c2};
  for (cudaStream_t st : ss)
    if (st && c->own_streams) cudaStreamDestroy(st);
  delete c;
  return SGB_OK;
}

int sgb_comm_use_streams(sgb_comm* c, void* s, void* c1, void* c2) {
  if (!c || !s || !c1 || !c2) return SGB_ERR_NULL;
  if (s == c1 || s == c2 || c1 == c2) return SGB_ERR_UNSUPPORTED;
  if (c->order.dirty_s || c->order.dirty_c1 || c->order.dirty_c2 || !c->pend_ptrs.empty() ||
      c->sparse_begun != c->sparse_ended)
    return SGB_ERR_STATE;
  if (c->own_streams) {
    cudaStream_t ss[] = {c->s, c->c1, c->c2};
    for (cudaStream_t st : ss)
      if (st) {
        CU(cudaStreamSynchronize(st));
        CU(cudaStreamDestroy(st));
      }
  }
  c->s = sgb::as_stream(s);
  c->c1 = sgb::as_stream(c1);
  c->c2 = sgb::as_stream(c2);
  c->own_streams = false;
  return SGB_OK;
}

int sgb_comm_rank(const sgb_comm* c) { return c ? c->rank : -1; }
int sgb_comm_world_size(const sgb_comm* c) { return c ? c->world : -1; }
size_t sgb_comm_staged_elems(const sgb_comm* c) { return c ? c->send_off : 0; }

int sgb_comm_set_topk_mode(sgb_comm* c, int mode) {
  if (!c) return SGB_ERR_NULL;
  if (mode != 0 && mode != 1) return SGB_ERR_UNSUPPORTED;
  c->topk_mode = mode;
  return SGB_OK;
}

/* The three side streams, for callers that profile or order against them:
 * which = 0 (s, NCCL), 1 (c1), 2 (c2). */
void* sgb_comm_stream(const sgb_comm* c, int which) {
  if (!c) return nullptr;
  return which == 0 ? c->s : (which == 1 ? c->c1 : (which == 2 ? c->c2 : nullptr));
}

int sgb_comm_wait(sgb_comm* c, void* compute_stream) {
  if (!c) return SGB_ERR_NULL;
  if (c->sparse_begun != c->sparse_ended) return SGB_ERR_STATE;   // an exchange is still to be ended
  return emit(c, plan_call(c, sgb::order::kWait).before, sgb::as_stream(compute_stream));
}

// The capture that a stream takes part in; 0 where it takes part in none.
static unsigned long long capture_of(cudaStream_t s) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamGetCaptureInfo(s, &st, &id) == cudaSuccess && st == cudaStreamCaptureStatusActive) return id;
  cudaGetLastError();
  return 0;
}

int sgb_comm_wait_captured(sgb_comm* c, void* compute_stream) {
  if (!c) return SGB_ERR_NULL;
  const cudaStream_t compute = sgb::as_stream(compute_stream);
  const unsigned long long mine = capture_of(compute);
  if (!mine) return sgb_comm_wait(c, compute_stream);
  if (c->sparse_begun != c->sparse_ended) return SGB_ERR_STATE;
  // what was queued before the capture stays as it is noted
  sgb::order::State before;
  before.dirty_s = c->order.dirty_s && capture_of(c->s) != mine;
  before.dirty_c1 = c->order.dirty_c1 && capture_of(c->c1) != mine;
  before.dirty_c2 = c->order.dirty_c2 && capture_of(c->c2) != mine;
  if (before.dirty_c2) {
    before.c2_reads_recv = c->order.c2_reads_recv;
    before.sparse = c->order.sparse;
  }
  c->order.dirty_s &= !before.dirty_s;
  c->order.dirty_c1 &= !before.dirty_c1;
  c->order.dirty_c2 &= !before.dirty_c2;
  const int st = emit(c, plan_call(c, sgb::order::kWait).before, compute);
  c->order = before;
  return st;
}

void* sgb_comm_result_stream(const sgb_comm* c) { return c ? side(c, c->result_stream) : nullptr; }

int sgb_comm_order_plan(unsigned char* state, int call, unsigned* edges, int* result_stream) {
  using namespace sgb::order;
  if (!state || !edges) return SGB_ERR_NULL;
  const bool both = call == 5;     // the two halves of a sparse exchange, one behind the other
  if (!both && !(call >= kSynch && call <= kWait) && !(call >= kSparseSelect && call <= kSparseLocal) &&
      call != kSparseUpdate)
    return SGB_ERR_UNSUPPORTED;
  State st;
  st.dirty_s = state[0];
  st.dirty_c1 = state[1];
  st.dirty_c2 = state[2];
  st.c2_reads_recv = state[3] & 1;
  st.sparse = state[3] >> 1;
  Step p = plan(st, both ? kSparseSelect : call);
  if (both) {
    const unsigned pre = p.pre, selected = p.post;
    p = plan(st, kSparseExchange);
    p.pre = pre | selected;        // recorded behind the selection, ahead of the exchange half
  }
  state[0] = st.dirty_s;
  state[1] = st.dirty_c1;
  state[2] = st.dirty_c2;
  state[3] = static_cast<unsigned char>(st.c2_reads_recv | st.sparse << 1);
  edges[0] = p.pre;
  edges[1] = p.before;
  edges[2] = p.after;
  edges[3] = p.post;
  if (result_stream) *result_stream = p.result_stream;
  return SGB_OK;
}

int sgb_comm_profile_begin(sgb_comm* c, void* compute_stream) {
  if (!c) return SGB_ERR_NULL;
  drop_ranges(c);
  if (!c->prof_origin) CU(cudaEventCreate(&c->prof_origin));
  CU(cudaEventRecord(c->prof_origin, sgb::as_stream(compute_stream)));
  c->profiling = true;
  return SGB_OK;
}

int sgb_comm_profiling(const sgb_comm* c) { return c && c->profiling ? 1 : 0; }

int sgb_comm_profile_range(sgb_comm* c, const char* name, int which, int begin) {
  if (!c || !name) return SGB_ERR_NULL;
  if (which < 0 || which > 2) return SGB_ERR_UNSUPPORTED;
  if (!c->profiling || capturing(side(c, which))) return SGB_OK;
  if (begin) {
    sgb_comm::Range r;
    r.name = name;
    CU(cudaEventCreate(&r.start));
    CU(cudaEventCreate(&r.end));
    CU(cudaEventRecord(r.start, side(c, which)));
    c->open_range = c->ranges.size();
    c->ranges.push_back(r);
  } else if (c->open_range < c->ranges.size()) {
    CU(cudaEventRecord(c->ranges[c->open_range].end, side(c, which)));
  }
  return SGB_OK;
}

int sgb_comm_profile_mark(sgb_comm* c, const char* name, void* stream) {
  if (!c || !name) return SGB_ERR_NULL;
  if (!c->profiling || capturing(sgb::as_stream(stream))) return SGB_OK;
  sgb_comm::Range r;
  r.name = name;
  CU(cudaEventCreate(&r.start));
  CU(cudaEventRecord(r.start, sgb::as_stream(stream)));
  r.end = nullptr;   // a mark has no extent
  c->ranges.push_back(r);
  return SGB_OK;
}

int sgb_comm_profile_end(sgb_comm* c, char* names, size_t name_stride, float* start_ms, float* end_ms,
                         size_t capacity, size_t* count) {
  if (!c || !count) return SGB_ERR_NULL;
  c->profiling = false;
  CU(cudaDeviceSynchronize());
  *count = c->ranges.size();
  for (size_t i = 0; i < c->ranges.size() && i < capacity; ++i) {
    const sgb_comm::Range& r = c->ranges[i];
    if (names && name_stride) {
      std::strncpy(names + i * name_stride, r.name.c_str(), name_stride - 1);
      names[i * name_stride + name_stride - 1] = 0;
    }
    if (start_ms) CU(cudaEventElapsedTime(start_ms + i, c->prof_origin, r.start));
    if (end_ms) CU(cudaEventElapsedTime(end_ms + i, c->prof_origin, r.end ? r.end : r.start));
  }
  drop_ranges(c);
  return SGB_OK;
}

int sgb_comm_synch(sgb_comm* c, void* data, size_t n, int is_half, void* compute_stream) {
  if (!c) return SGB_ERR_NULL;
  if (n == 0) return SGB_OK;
  if (!data) return SGB_ERR_NULL;
  if (n > 0x7fffffffu) return SGB_ERR_SIZE;
  const sgb::order::Step p = plan_call(c, sgb::order::kSynch);
  OK(emit(c, p.before, sgb::as_stream(compute_stream)));
  {
    Phase ph(c, "Dist_s_synch_allreduce", sgb::order::kStreamS);
    if (c->world > 1) NC(ncclAllReduce(data, data, n, is_half ? ncclHalf : ncclFloat, ncclSum, c->nccl, c->s));
  }
  return emit(c, p.after, nullptr);
}

int sgb_comm_fused_synch(sgb_comm* c, void* const* tensors, const size_t* sizes, size_t count,
                         int is_half, int send, void* compute_stream) {
  if (!c) return SGB_ERR_NULL;
  OK(check_list(tensors, sizes, count));
  cudaStream_t compute = sgb::as_stream(compute_stream);
  const size_t esz = is_half ? sizeof(__half) : sizeof(float);
  if (!send) {
    const size_t total = total_of(sizes, count);
    if (c->send_off + total > c->max_elems) return SGB_ERR_CAPACITY;
    if (!is_half) {
      if (!c->pend_ptrs.empty() && c->pend_half)
        OK(pack_other_kind(c, compute, "Dist_c1_fusedSynchHalf_filling"));
      defer(c, tensors, sizes, count, 0);
    } else {
      OK(emit(c, plan_call(c, sgb::order::kStageCopy).pre, compute));
      Phase ph(c, "Dist_c1_fusedSynch_filling", sgb::order::kStreamC1);
      size_t off = c->send_off;
      for (size_t i = 0; i < count; ++i) {
        CU(cudaMemcpyAsync(reinterpret_cast<char*>(c->send) + off * esz, tensors[i],
                           sizes[i] * esz, cudaMemcpyDeviceToDevice, c->c1));
        off += sizes[i];
      }
    }
    c->send_off += total;
    return SGB_OK;
  }
  // flush: everything staged so far is reduced; `tensors` receive the result
  const size_t total = total_of(sizes, count);
  if (total > c->max_elems) return SGB_ERR_CAPACITY;
  // Gradients that already sit back to back in memory (a gradient arena) need
  // neither the pack nor the unpack pass: the bucket is reduced in place, on s,
  // ordered directly after the compute stream that produced it.
  if (!is_half && !c->pend_half && c->pend_off == 0 && c->pend_ptrs.size() == count &&
      c->send_off == total) {
    bool in_place = true;
    for (size_t i = 0; i < count && in_place; ++i) {
      in_place = c->pend_ptrs[i] == tensors[i] && c->pend_sizes[i] == sizes[i] &&
                 (i + 1 == count ||
                  static_cast<char*>(tensors[i]) + sizes[i] * sizeof(float) == tensors[i + 1]);
    }
    if (in_place) {
      c->pend_ptrs.clear();
      c->pend_sizes.clear();
      c->send_off = 0;
      const sgb::order::Step p = plan_call(c, sgb::order::kFlushInPlace);
      OK(emit(c, p.before, compute));
      {
        Phase ph(c, "Dist_s_fusedSynch_allreduce", sgb::order::kStreamS);
        if (c->world > 1) NC(ncclAllReduce(tensors[0], tensors[0], total, ncclFloat, ncclSum, c->nccl, c->s));
      }
      return emit(c, p.after, nullptr);
    }
  }
  const sgb::order::Step p = plan_call(c, sgb::order::kFlushPacked);
  OK(emit(c, p.pre, compute));
  if (alone(c, tensors, sizes, count, total, 0)) {
    // One rank: the tensors hold their sum already.  Streams, events and phases
    // are those of any world size; nothing is packed, reduced or copied back.
    c->pend_ptrs.clear();
    c->pend_sizes.clear();
    c->send_off = 0;
    { Phase ph(c, "Dist_c1_fusedSynch_filling", sgb::order::kStreamC1); }
    OK(emit(c, p.before, compute));
    { Phase ph(c, "Dist_s_fusedSynch_allreduce", sgb::order::kStreamS); }
    OK(emit(c, p.after, nullptr));
    Phase ph(c, "Dist_c1_fusedSynch_copyBackToTensor", sgb::order::kStreamC1);
    return SGB_OK;
  }
  OK(pack_pending(c, "Dist_c1_fusedSynch_filling"));
  OK(emit(c, p.before, compute));
  if (c->send_off) {
    Phase ph(c, "Dist_s_fusedSynch_allreduce", sgb::order::kStreamS);
    NC(ncclAllReduce(c->send, c->recv, c->send_off, is_half ? ncclHalf : ncclFloat, ncclSum,
                     c->nccl, c->s));
  }
  c->send_off = 0;
  OK(emit(c, p.after, nullptr));
  Phase ph(c, "Dist_c1_fusedSynch_copyBackToTensor", sgb::order::kStreamC1);
  if (!is_half) {
    OK(sgb_unpack_f32(c->recv, 0, tensors, sizes, count, 1.0f, c->c1));
  } else {
    size_t off = 0;
    for (size_t i = 0; i < count; ++i) {
      CU(cudaMemcpyAsync(tensors[i], reinterpret_cast<char*>(c->recv) + off * esz, sizes[i] * esz,
                         cudaMemcpyDeviceToDevice, c->c1));
      off += sizes[i];
    }
  }
  return SGB_OK;
}

int sgb_comm_synch_half(sgb_comm* c, float* data, size_t n, void* compute_stream) {
  if (!c) return SGB_ERR_NULL;
  if (n == 0) return SGB_OK;
  if (!data) return SGB_ERR_NULL;
  if (n > c->max_elems) return SGB_ERR_CAPACITY;
  OK(half_init(c));
  cudaStream_t compute = sgb::as_stream(compute_stream);
  const sgb::order::Step p = plan_call(c, sgb::order::kSynchHalf);
  const bool one = c->world == 1;     // the sum of one rank's fp16 values is those values: round in place
  OK(emit(c, p.pre, compute));
  {
    Phase ph(c, "Dist_c1_synchHalf_float2half", sgb::order::kStreamC1);
    if (one) {
      void* const t[1] = {data};
      const size_t sz[1] = {n};
      OK(sgb::round_f16_multi(t, sz, 1, c->c1));
    } else {
      OK(sgb_cast_f32_f16(data, c->dsend_h, n, c->c1));
    }
  }
  OK(emit(c, p.before, compute));
  {
    Phase ph(c, "Dist_s_synchHalf_allreduce", sgb::order::kStreamS);
    if (!one) NC(ncclAllReduce(c->dsend_h, c->drecv_h, n, ncclHalf, ncclSum, c->nccl, c->s));
  }
  OK(emit(c, p.after, nullptr));
  {
    Phase ph(c, "Dist_c2_synchHalf_half2float", sgb::order::kStreamC2);
    if (!one) OK(sgb_cast_f16_f32(c->drecv_h, data, n, c->c2));
  }
  return emit(c, p.post, nullptr);
}

int sgb_comm_fused_synch_half(sgb_comm* c, void* const* tensors, const size_t* sizes,
                              size_t count, int send, void* compute_stream) {
  if (!c) return SGB_ERR_NULL;
  OK(check_list(tensors, sizes, count));
  OK(half_init(c));
  cudaStream_t compute = sgb::as_stream(compute_stream);
  const size_t total = total_of(sizes, count);
  if (!send) {
    if (c->send_off + total > c->max_elems) return SGB_ERR_CAPACITY;
    // copy + float2half of the reference collapse into one pack-and-cast pass at flush time
    if (!c->pend_ptrs.empty() && !c->pend_half)
      OK(pack_other_kind(c, compute, "Dist_c1_fusedSynch_filling"));
    defer(c, tensors, sizes, count, 1);
    c->send_off += total;
    return SGB_OK;
  }
  if (total > c->max_elems) return SGB_ERR_CAPACITY;
  if (alone(c, tensors, sizes, count, total, 1)) {
    // one rank: rounded where they are (see sgb_comm_synch_half), all of it on c1
    c->pend_ptrs.clear();
    c->pend_sizes.clear();
    c->send_off = 0;
    OK(emit(c, plan_call(c, sgb::order::kStageCopy).pre, compute));
    Phase ph(c, "Dist_c1_fusedSynchHalf_float2half", sgb::order::kStreamC1);
    return sgb::round_f16_multi(tensors, sizes, count, c->c1);
  }
  const sgb::order::Step p = plan_call(c, sgb::order::kFlushHalf);
  OK(emit(c, p.pre, compute));
  OK(pack_pending(c, "Dist_c1_fusedSynchHalf_float2half"));
  OK(emit(c, p.before, compute));
  if (c->send_off) {
    Phase ph(c, "Dist_s_fusedSynchHalf_allreduce", sgb::order::kStreamS);
    NC(ncclAllReduce(c->send_h, c->recv_h, c->send_off, ncclHalf, ncclSum, c->nccl, c->s));
  }
  c->send_off = 0;
  OK(emit(c, p.after, nullptr));
  {
    Phase ph(c, "Dist_c2_fusedSynchHalf_half2floatcopy", sgb::order::kStreamC2);
    OK(sgb_unpack_f16_to_f32(c->recv_h, 0, tensors, sizes, count, 1.0f, c->c2));
  }
  return emit(c, p.post, nullptr);
}

int sgb_comm_round_half(sgb_comm* c, void* const* tensors, const size_t* sizes, size_t count, size_t largest,
                        void* compute_stream) {
  if (!c) return SGB_ERR_NULL;
  OK(check_list(tensors, sizes, count));
  if (c->world != 1 || c->profiling || c->send_off || !c->pend_ptrs.empty() || largest > c->max_elems)
    return SGB_ERR_UNSUPPORTED;
  if (count == 0) return SGB_OK;
  OK(emit(c, plan_call(c, sgb::order::kStageCopy).pre, sgb::as_stream(compute_stream)));
  Phase ph(c, "Dist_c1_fusedSynchHalf_float2half", sgb::order::kStreamC1);
  return sgb::round_f16_multi(tensors, sizes, count, c->c1);
}

// Whether the first `bytes` of a workspace are clear, which they no longer count as: the
// selection uses them.  (Two microseconds of a pass went by between the call that cleared
// them and the selection.)
static bool take_cleared(sgb_comm* c, sgb_comm::Cleared* w, size_t bytes, cudaStream_t compute) {
  w->captured = w->captured || capturing(compute) || capturing(c->c1);
  const bool clear = !w->captured && w->bytes >= bytes;
  w->bytes = 0;
  return clear;
}
// The dense sum that clears them has been launched.
static void now_cleared(sgb_comm::Cleared* w, size_t bytes) { w->bytes = w->captured ? 0 : bytes; }

// The selection half.  capacity == 0: the reference's exchange (the payload is
// as long as the largest count, which the host reads back).  capacity > 0
// (threshold mode): every rank sends exactly `capacity` slots, no host round trip.
static int sparse_begin(sgb_comm* c, void* const* tensors, const size_t* sizes, size_t count,
                        float* accumulation, float spars, int topk, size_t capacity, void* compute_stream) {
  if (!c) return SGB_ERR_NULL;
  OK(check_list(tensors, sizes, count));
  const size_t n = total_of(sizes, count);
  if (n > c->max_elems) return SGB_ERR_CAPACITY;
  if (capacity > c->max_elems) return SGB_ERR_CAPACITY;
  if (c->sparse_begun - c->sparse_ended >= 2) return SGB_ERR_STATE;
  OK(sparse_init(c));
  const unsigned char slots = c->order.sparse;
  const sgb::order::Step p = plan_call(c, sgb::order::kSparseSelect);
  sgb_comm::Sparse& x = c->sparse[p.slot];
  x.n = n;
  x.nnz_max = 0;
  x.capacity = capacity;
  x.topk = topk;
  x.op_name = count > 1 ? "Dist_c1c2_fusedSparsification" : "Dist_c1c2_sparsification";
  x.tensors.clear();
  x.sizes.clear();
  for (size_t i = 0; i < count; ++i) {
    x.tensors.push_back(static_cast<float*>(tensors[i]));
    x.sizes.push_back(sizes[i]);
  }
  const int st = [&] {
    OK(emit(c, p.pre, sgb::as_stream(compute_stream), p.slot));
    if (n == 0) return emit(c, p.post, nullptr, p.slot);
    Phase ph(c, x.op_name, sgb::order::kStreamC1);
    // The selection reads the tensors where they are; only a long list, or one
    // without a residual buffer, is copied together first.
    float* const* grads = x.tensors.data();
    const size_t* grad_sizes = x.sizes.data();
    size_t ngrads = count;
    if (!sgb::sparse_selects_from(grads, grad_sizes, ngrads, accumulation)) {
      OK(sgb_pack_f32(tensors, sizes, count, c->send, 0, c->c1));
      grads = &c->send;
      grad_sizes = &x.n;
      ngrads = 1;
    }
    take_cleared(c, &c->ws_clear, 0, sgb::as_stream(compute_stream));   // (clears for itself, and leaves its own behind)
    if (topk) {
      x.nnz_max = static_cast<size_t>(sgb_topk_count(spars, n));
      for (int r = 0; r < c->world; ++r) x.nnz_host[r] = static_cast<int>(x.nnz_max);
      if (x.nnz_max)
        OK(sgb::sparse_topk(grads, grad_sizes, ngrads, accumulation, x.nnz_max, c->topk_mode, x.pay_send,
                            reinterpret_cast<float*>(x.pay_send) + x.nnz_max, c->ws, c->ws_bytes, c->c1));
    } else if (capacity) {
      x.nnz_max = capacity;
      OK(sgb::sparse_threshold_bounded(grads, grad_sizes, ngrads, accumulation, spars, x.pay_send, capacity, x.nnz_dev,
                                       c->dropped_dev, c->ws, c->ws_bytes, c->c1));
      // the counts travel on the device only; receivers clamp them to the capacity
      if (c->world > 1) NC(ncclAllGather(x.nnz_dev, x.nnz_dev + 1, 1, ncclInt, c->nccl, c->c1));
    } else if (c->world == 1) {
      // nobody to tell: the dense sum reads the payload and its count where they are
      OK(sgb::sparse_threshold_packed(grads, grad_sizes, ngrads, accumulation, spars, x.pay_send, x.nnz_dev, c->ws,
                                      c->ws_bytes, c->c1));
    } else {
      OK(sgb::sparse_threshold_packed(grads, grad_sizes, ngrads, accumulation, spars, x.pay_send, x.nnz_dev, c->ws,
                                      c->ws_bytes, c->c1));
      NC(ncclAllGather(x.nnz_dev, x.nnz_dev + 1, 1, ncclInt, c->nccl, c->c1));
      CU(cudaMemcpyAsync(x.nnz_host, x.nnz_dev + 1, sizeof(int) * c->world, cudaMemcpyDeviceToHost, c->c1));
      CU(cudaEventRecord(x.counted, c->c1));
    }
    return emit(c, p.post, nullptr, p.slot);
  }();
  if (st != SGB_OK) {
    c->order.sparse = slots;         // not begun: the slot stays free
    return st;
  }
  ++c->sparse_begun;
  return SGB_OK;
}

// The exchange half of the oldest exchange that is open.
static int sparse_end(sgb_comm* c, void* compute_stream) {
  if (!c) return SGB_ERR_NULL;
  if (c->sparse_begun == c->sparse_ended) return SGB_ERR_STATE;
  ++c->sparse_ended;
  const int W = c->world;
  const sgb::order::Step p = plan_call(c, W == 1 ? sgb::order::kSparseLocal : sgb::order::kSparseExchange);
  sgb_comm::Sparse& x = c->sparse[p.slot];
  if (W == 1) {
    // The payload is read where it lies: no all-gather, no count on the host.
    OK(emit(c, p.before, sgb::as_stream(compute_stream), p.slot));
    if (x.n == 0) return emit(c, p.post, nullptr, p.slot);
    Phase ph(c, x.op_name, sgb::order::kStreamC2);
    OK(sgb::sparse_dense_sum(x.pay_send, 0, x.capacity, x.nnz_host, x.topk ? nullptr : x.nnz_dev, 1, x.tensors.data(),
                             x.sizes.data(), x.tensors.size(), c->c2));
    return emit(c, p.post, nullptr, p.slot);
  }
  if (x.n && !x.topk && !x.capacity) {
    CU(cudaEventSynchronize(x.counted));
    for (int r = 0; r < W; ++r) {
      if (x.nnz_host[r] < 0 || static_cast<size_t>(x.nnz_host[r]) > x.n) return SGB_ERR_STATE;
      if (static_cast<size_t>(x.nnz_host[r]) > x.nnz_max) x.nnz_max = x.nnz_host[r];
    }
  }
  OK(emit(c, p.before, sgb::as_stream(compute_stream), p.slot));
  {
    Phase ph(c, "Dist_s_sparsification_allgather", sgb::order::kStreamS);
    if (x.nnz_max) NC(ncclAllGather(x.pay_send, c->pay_recv, 2 * x.nnz_max, ncclFloat, c->nccl, c->s));
  }
  OK(emit(c, p.after, nullptr));
  if (x.n) {
    Phase ph(c, x.op_name, sgb::order::kStreamC2);
    const size_t stride = 2 * x.nnz_max;
    if (W <= sgb::kMaxDenseRanks) {
      OK(sgb::sparse_dense_sum(c->pay_recv, stride, x.capacity, x.nnz_host, x.capacity ? x.nnz_dev + 1 : nullptr, W,
                               x.tensors.data(), x.sizes.data(), x.tensors.size(), c->c2));
    } else {
      // more ranks than the dense kernel's table holds: fill, then add rank after rank
      CU(cudaMemsetAsync(c->recv, 0, x.n * sizeof(float), c->c2));
      for (int r = 0; r < W && x.nnz_max; ++r) {
        const int* seg = c->pay_recv + static_cast<size_t>(r) * stride;
        const size_t cnt = x.capacity ? x.capacity : static_cast<size_t>(x.nnz_host[r]);
        OK(sgb_scatter_add_f32(seg, reinterpret_cast<const float*>(seg) + cnt, cnt,
                               x.capacity ? x.nnz_dev + 1 + r : nullptr, c->recv, x.n, c->c2));
      }
      OK(sgb_unpack_f32(c->recv, 0, reinterpret_cast<void* const*>(x.tensors.data()), x.sizes.data(),
                        x.tensors.size(), 1.0f, c->c2));
    }
  }
  return emit(c, p.post, nullptr);
}

// Room for a joint selection over `span` elements, ahead of any work of the call
// (c1 has not joined a capture of the compute stream yet).  Outgrown buffers are
// kept until the communicator goes: their addresses may sit in a captured graph
// or in queued work.  Doubling keeps their sum below twice the size of the last one.
static int joint_reserve(sgb_comm* c, size_t span, cudaStream_t compute, size_t ws_least = 0) {
  if (span <= c->joint_elems && ws_least <= c->joint_ws_bytes) return SGB_OK;
  if (capturing(compute) || capturing(c->c1)) return SGB_ERR_UNSUPPORTED;
  size_t elems = 2 * c->joint_elems;
  if (elems > sgb::kMaxBucketSpan) elems = sgb::kMaxBucketSpan;
  if (elems < span) elems = span;
  size_t ws_bytes = sgb_sparse_workspace_bytes(elems);
  if (ws_bytes < ws_least) ws_bytes = ws_least;
  int* pay = nullptr;
  void* ws = nullptr;
  if (!c->joint_nnz) CU(cudaMalloc(&c->joint_nnz, sizeof(int)));
  CU(cudaMalloc(&pay, 2 * elems * sizeof(int)));
  if (c->joint_pay) c->joint_retired.push_back(c->joint_pay);
  c->joint_pay = pay;
  c->joint_elems = 0;              // until the workspace is there as well
  CU(cudaMalloc(&ws, ws_bytes));
  if (c->joint_ws) c->joint_retired.push_back(c->joint_ws);
  c->joint_ws = ws;
  c->joint_ws_bytes = ws_bytes;
  c->joint_clear = {};
  c->joint_elems = elems;
  return SGB_OK;
}

// One rank has no transport to overlap a bucket's selection with, so all buckets
// are selected by one launch and written back by another: per bucket the two
// took 14 + 5 us, of which 4 + 2 were memory traffic.
static int threshold_buckets(sgb_comm* c, const std::vector<sgb::SparseBucket>& list, float threshold,
                             const sgb::SparseUpdate* update, cudaStream_t compute) {
  // cut the list into groups that one launch can take
  std::vector<size_t> ends;
  size_t widest = 0;
  for (size_t k = 0; k < list.size();) {
    size_t end = k, span = 0;
    while (end < list.size()) {
      const size_t more = sgb::sparse_buckets_span(list.data() + k, end + 1 - k);
      if (!more) break;
      span = more;
      ++end;
    }
    if (end == k) return SGB_ERR_UNSUPPORTED;
    ends.push_back(end);
    widest = span > widest ? span : widest;
    k = end;
  }
  OK(joint_reserve(c, widest, compute));
  OK(emit(c, plan_call(c, sgb::order::kStageCopy).pre, compute));
  Phase ph(c, "Dist_c1c2_fusedSparsification", sgb::order::kStreamC1);
  size_t k = 0, tensor = 0;
  for (const size_t end : ends) {
    const size_t counters = sgb::sparse_counter_bytes(1);
    OK(sgb::sparse_threshold_buckets(list.data() + k, end - k, threshold, c->joint_pay, c->joint_nnz, c->joint_ws,
                                     c->joint_ws_bytes, c->c1, take_cleared(c, &c->joint_clear, counters, compute)));
    sgb::SparseUpdate part{};
    if (update)
      part = {update->sgd, update->params + tensor, update->moments ? update->moments + tensor : nullptr};
    OK(sgb::sparse_dense_buckets(c->joint_pay, 0, c->joint_nnz, list.data() + k, end - k, c->c1, update ? &part : nullptr,
                                 {c->joint_ws, counters, c->joint_ws_bytes}));
    now_cleared(&c->joint_clear, counters);
    for (; k < end; ++k) tensor += list[k].count;
  }
  return SGB_OK;
}

// The buckets of a joint call; SGB_ERR_UNSUPPORTED where it takes a call per bucket.
static int joint_list(sgb_comm* c, void* const* tensors, const size_t* sizes, const size_t* counts,
                      float* const* accumulations, size_t nbuckets, std::vector<sgb::SparseBucket>* list) {
  if (!c) return SGB_ERR_NULL;
  if (!counts || !accumulations) return SGB_ERR_NULL;
  if (c->world != 1 || c->profiling || c->sparse_begun != c->sparse_ended) return SGB_ERR_UNSUPPORTED;
  size_t at = 0;
  for (size_t k = 0; k < nbuckets; ++k) {
    OK(check_list(tensors + at, sizes + at, counts[k]));
    if (total_of(sizes + at, counts[k]) > c->max_elems) return SGB_ERR_UNSUPPORTED;
    list->push_back({reinterpret_cast<float* const*>(tensors + at), sizes + at, counts[k], accumulations[k]});
    at += counts[k];
  }
  return SGB_OK;
}

int sgb_comm_sparsification_buckets(sgb_comm* c, void* const* tensors, const size_t* sizes, const size_t* counts,
                                    float* const* accumulations, size_t nbuckets, float threshold,
                                    void* compute_stream) {
  std::vector<sgb::SparseBucket> list;
  OK(joint_list(c, tensors, sizes, counts, accumulations, nbuckets, &list));
  return threshold_buckets(c, list, threshold, nullptr, sgb::as_stream(compute_stream));
}

// Which lists of one rank the joint call takes.  Several buckets by size: whatever
// one launch can, since their selections are one launch then (us a pass, a call per
// bucket and update / joint: 4 buckets of 12 tensors, 2e6 elements in all 70.9 / 32.6, 12
// of 160, 2.4e7 355.3 / 186.7).  Else only the update is saved a launch and a read of
// the gradients, for tiles in which a tensor's update waits for its neighbour's and a
// longer list of arguments: the line is at few tensors and, by threshold, few elements.
//   by size, one bucket of 1e6: in 1 tensor 30.0 / 21.8, 12 35.5 / 32.7, 50 33.8 / 53.5
//   by threshold, 1e6:   in 1 tensor 20.6 / 16.4, 5 21.3 / 18.1, 12 22.8 / 24.8, 50 27.1 / 31.3
//   3e6 elements in 1 tensor 36.9 / 33.3, 5e6 53.5 / 45.9, 8e6 70.3 / 66.0, 1.6e7 116 / 109;
//   in 6 3.4e6 35.4 / 33.2, 4.6e6 54.6 / 53.4, 5.8e6 63.2 / 65.3, 8.2e6 77 / 86; 2.56e7 in 161
//   182 / 174, but 27 us more of the host
static bool sparse_update_pays(size_t elements, size_t tensors, size_t nbuckets, int topk) {
  if (topk) return nbuckets > 1 || tensors <= 16;
  return tensors == 1 ? elements <= sgb::kMaxBucketSpan : tensors <= SGB_SPARSE_UPDATE_TENSORS && elements <= 4000000;
}

int sgb_comm_sparse_update_takes(const sgb_comm* c, void* const* tensors, const size_t* sizes, const size_t* counts,
                                 size_t nbuckets, int topk) {
  if (!c || !tensors || !sizes || !counts || c->world != 1 || c->profiling) return 0;
  size_t count = 0;
  for (size_t k = 0; k < nbuckets; ++k) count += counts[k];
  return sparse_update_pays(total_of(sizes, count), count, nbuckets, topk) &&
         (!topk || nbuckets == 1 ||
          sgb::sparse_topk_buckets_cut(reinterpret_cast<float* const*>(tensors), sizes, counts, nbuckets, nullptr));
}

int sgb_comm_sparse_update(sgb_comm* c, void* const* tensors, const size_t* sizes, const size_t* counts,
                           float* const* accumulations, size_t nbuckets, float spars, int topk, void* const* params,
                           void* const* moments, float lr, float momentum, float dampening, float weight_decay,
                           int nesterov, float grad_scale, void* compute_stream) {
  std::vector<sgb::SparseBucket> list;
  OK(joint_list(c, tensors, sizes, counts, accumulations, nbuckets, &list));
  if (!params) return SGB_ERR_NULL;
  sgb::SgdArgs sgd;
  OK(sgb::sgd_args(&sgd, moments, lr, momentum, dampening, weight_decay, nesterov, grad_scale));
  size_t total = 0;
  for (const sgb::SparseBucket& b : list) total += b.count;
  for (size_t k = 0; k < total; ++k)
    if (sizes[k] && (!params[k] || (sgd.use_momentum && !moments[k]))) return SGB_ERR_NULL;
  cudaStream_t compute = sgb::as_stream(compute_stream);
  const sgb::SparseUpdate update{&sgd, reinterpret_cast<float* const*>(params),
                                 sgd.use_momentum ? reinterpret_cast<float* const*>(moments) : nullptr};
  if (!sparse_update_pays(total_of(sizes, total), total, nbuckets, topk)) return SGB_ERR_UNSUPPORTED;
  if (!topk) return threshold_buckets(c, list, spars, &update, compute);
  for (const sgb::SparseBucket& b : list)
    if (!sgb::sparse_selects_from(b.tensors, b.sizes, b.count, b.acc)) return SGB_ERR_UNSUPPORTED;
  // several buckets: one launch selects from as many as it can take, the next updates them
  if (nbuckets > 1) {
    std::vector<size_t> ends, ks, counters;            // counters: bytes of them, per launch
    if (!sgb::sparse_topk_buckets_cut(reinterpret_cast<float* const*>(tensors), sizes, counts, nbuckets, &ends))
      return SGB_ERR_UNSUPPORTED;
    size_t widest = 0, ws_bytes = 0, k = 0, tensor = 0;
    for (const size_t end : ends) {
      size_t span = 0;
      const size_t first = k;
      for (; k < end; ++k) {
        const size_t n = total_of(list[k].sizes, list[k].count);
        ks.push_back(static_cast<size_t>(sgb_topk_count(spars, n)));
        span += n + 512;
      }
      size_t of_these = 0;
      const size_t need =
          sgb::sparse_topk_buckets_bytes(list.data() + first, ks.data() + first, k - first, c->topk_mode, &of_these);
      if (!need) return SGB_ERR_UNSUPPORTED;
      counters.push_back(of_these);
      widest = span > widest ? span : widest;
      ws_bytes = need > ws_bytes ? need : ws_bytes;
    }
    OK(joint_reserve(c, widest, compute, ws_bytes));
    OK(emit(c, plan_call(c, sgb::order::kStageCopy).pre, compute));
    Phase ph(c, "Dist_c1c2_fusedSparsification", sgb::order::kStreamC1);
    k = 0;
    for (size_t part = 0; part < ends.size(); ++part) {
      const size_t end = ends[part], used = counters[part];
      int sent = 0;
      OK(sgb::sparse_topk_buckets(list.data() + k, ks.data() + k, end - k, c->topk_mode, c->joint_pay, &sent,
                                  c->joint_ws, c->joint_ws_bytes, c->c1,
                                  take_cleared(c, &c->joint_clear, used, compute)));
      const sgb::SparseUpdate behind{&sgd, update.params + tensor, update.moments ? update.moments + tensor : nullptr};
      OK(sgb::sparse_dense_buckets(c->joint_pay, sent, nullptr, list.data() + k, end - k, c->c1, &behind,
                                   {c->joint_ws, used, c->joint_ws_bytes}));
      now_cleared(&c->joint_clear, used);
      for (; k < end; ++k) tensor += list[k].count;
    }
    return SGB_OK;
  }
  if (nbuckets != 1 || (!c->dropped_dev && (capturing(compute) || capturing(c->c1)))) return SGB_ERR_UNSUPPORTED;
  OK(sparse_init(c));
  const sgb::order::Step p = plan_call(c, sgb::order::kSparseUpdate);
  const sgb_comm::Sparse& x = c->sparse[p.slot];
  OK(emit(c, p.pre, compute, p.slot));
  Phase ph(c, "Dist_c1c2_fusedSparsification", sgb::order::kStreamC1);
  const sgb::SparseBucket& b = list[0];
  const size_t n = total_of(b.sizes, b.count), k = static_cast<size_t>(sgb_topk_count(spars, n));
  const int sent[1] = {static_cast<int>(k)};
  const size_t counters = sgb::sparse_counter_bytes(1);
  if (k)
    OK(sgb::sparse_topk(b.tensors, b.sizes, b.count, b.acc, k, c->topk_mode, x.pay_send,
                        reinterpret_cast<float*>(x.pay_send) + k, c->ws, c->ws_bytes, c->c1,
                        take_cleared(c, &c->ws_clear, counters, compute)));
  OK(sgb::sparse_dense_sum(x.pay_send, 0, 0, sent, nullptr, 1, b.tensors, b.sizes, b.count, c->c1, &update,
                           {c->ws, k ? counters : 0, c->ws_bytes}));
  if (k) now_cleared(&c->ws_clear, counters);
  return SGB_OK;
}

int sgb_comm_update_half(sgb_comm* c, void* const* params, void* const* grads, void* const* moments,
                         const size_t* sizes, size_t count, size_t largest, float lr, float momentum, float dampening,
                         float weight_decay, int nesterov, float grad_scale, void* compute_stream) {
  if (!c) return SGB_ERR_NULL;
  OK(check_list(grads, sizes, count));
  if (!params) return SGB_ERR_NULL;
  if (c->world != 1 || c->profiling || c->send_off || !c->pend_ptrs.empty() || largest > c->max_elems)
    return SGB_ERR_UNSUPPORTED;
  sgb::SgdArgs sgd;
  OK(sgb::sgd_args(&sgd, moments, lr, momentum, dampening, weight_decay, nesterov, grad_scale));
  // no buffer of the communicator takes part: behind what its streams still do, on the caller's
  OK(sgb_comm_wait_captured(c, compute_stream));
  return sgb::sgd_round_f16_multi(params, grads, moments, sizes, count, sgd, sgb::as_stream(compute_stream));
}

static int sparsify(sgb_comm* c, void* const* tensors, const size_t* sizes, size_t count, float* accumulation,
                    float spars, int topk, size_t capacity, void* compute_stream) {
  if (c && c->sparse_begun != c->sparse_ended) return SGB_ERR_STATE;
  OK(sparse_begin(c, tensors, sizes, count, accumulation, spars, topk, capacity, compute_stream));
  return sparse_end(c, compute_stream);
}

int sgb_comm_sparsification(sgb_comm* c, void* const* tensors, const size_t* sizes, size_t count,
                            float* accumulation, float spars, int topk, void* compute_stream) {
  return sparsify(c, tensors, sizes, count, accumulation, spars, topk, 0, compute_stream);
}

int sgb_comm_sparsification_begin(sgb_comm* c, void* const* tensors, const size_t* sizes, size_t count,
                                  float* accumulation, float spars, int topk, void* compute_stream) {
  return sparse_begin(c, tensors, sizes, count, accumulation, spars, topk, 0, compute_stream);
}

int sgb_comm_sparsification_end(sgb_comm* c, void* compute_stream) { return sparse_end(c, compute_stream); }

int sgb_comm_sparsification_bounded(sgb_comm* c, void* const* tensors, const size_t* sizes, size_t count,
                                    float* accumulation, float threshold, size_t capacity,
                                    void* compute_stream) {
  if (capacity == 0) return SGB_ERR_SIZE;
  return sparsify(c, tensors, sizes, count, accumulation, threshold, 0, capacity, compute_stream);
}

int sgb_comm_sparse_dropped(sgb_comm* c, unsigned long long* dropped) {
  if (!c || !dropped) return SGB_ERR_NULL;
  *dropped = 0;
  if (!c->dropped_dev) return SGB_OK;               // no sparse call yet
  // on the stream that runs the selection, so that every call issued so far is counted
  CU(cudaMemcpyAsync(dropped, c->dropped_dev, sizeof(unsigned long long), cudaMemcpyDeviceToHost, c->c1));
  CU(cudaStreamSynchronize(c->c1));
  return SGB_OK;
}

}  // extern "C"
