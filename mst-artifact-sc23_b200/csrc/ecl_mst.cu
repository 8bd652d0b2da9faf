// B200 (sm_100a) engine of the ECL-MST minimum spanning forest: host side
// of the single-graph solve (context, launch sequence, C ABI). The kernels
// and their mapping to the reference's gpuMST (ECL-MST/ECL_MST.cu:265-362)
// are in mst_device.cuh.
#include <cuda_runtime.h>
#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <utility>

#include "ecl_mst.h"
#include "internal.h"
#include "mst_device.cuh"
#include "rounds_device.cuh"
#include "scan_device.cuh"
#include "group_device.cuh"
#include "cluster_device.cuh"
#include <vector>

// Learned threshold/split (learned.cu). ecl_learned_sample uploads changed
// weights and sorts the weight sample; ecl_learned_apply computes the
// features from it and from k_prep's degree statistics and runs the trained
// MLP, writing DevState::threshold, filtered, quantile and split.
int ecl_learned_sample(ecl_mst_ctx* c, const ecl_graph* d_graph, cudaStream_t s);
int ecl_learned_apply(ecl_mst_ctx* c, const ecl_graph* d_graph, cudaStream_t s, void* st, int lists);
int ecl_learned_upload(ecl_mst_ctx* c, cudaStream_t s);
unsigned ecl_learned_weights_version();
// The same for the graphs of a batch, all in two launches.
int ecl_learned_batch_prepare();
int ecl_learned_batch(ecl_mst_ctx* c, const ecl::GraphDesc* graphs, int count, int least, const int* nindex,
                      const int* eweight, ecl::FeatAcc* acc, ecl::LearnedChoice* choice, cudaStream_t s);

using namespace ecl;

namespace {
constexpr int kDefaultSplit = 8;
constexpr unsigned kDefaultSmallTail = 4096;
constexpr int kDefaultMinTiles = 1;  // round CTAs kept: one per tile of the round's worklist
constexpr int64_t kWlSlack = 1 << 19;  // worklist slots beyond `edges` (scan chunk tails)
constexpr int kLearnedMinEdges = 1 << 20;
// Single graphs up to this many entries are solved in one launch (k_group):
// RMAT-14 156 us against 200 with a launch per pass, ER 200k 295 against 327.
// At 4.0M entries ER 500k takes 338 against 360 and RMAT-16 207 against 219, but
// a grid 437 against 416; at 4.5M 367 against 388, 219 against 221 and 463
// against 437; at 8.0M ER 1M 505 against 491, a geometric graph 479 against 461
// and a grid 663 against 625.
constexpr int kGroupEdges = 1 << 22;
// and of up to this many entries and vertices by one cluster (k_cluster), alone
// on one CTA up to kClusterShare entries
constexpr int kClusterEdges = 1 << 16, kClusterNodes = 1 << 15;
constexpr int kClusterShare = 1 << 14;
}  // namespace

// =================================================================== host
struct ecl_mst_ctx {
  int device = 0;
  int sm_count = 0;
  int64_t max_nodes = 0, max_edges = 0;
  cudaStream_t stream = nullptr;
  // the learned schedule's sample sort (beside k_prep) and MLP run on `side`
  cudaStream_t side = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr, prep_done = nullptr;
  // the last solve's key, and the captured solve (CUDA graph) with its key
  std::vector<long long> last_key, exec_key;
  cudaGraphExec_t exec = nullptr;
  // [minv0 | minv1 | parent] in one allocation, laid out per solve for the
  // graph's vertex count (minv0 = slots, minv1 = minv0 + n, parent after
  // minv1), so one L2 access-policy window covers exactly the 20n bytes used
  void* slots = nullptr;
  // L2 persistence (ECL_FLAG_L2_PERSIST): the device's persisting set-aside
  // and window limits, and the set-aside this context raised (restored at
  // destroy)
  size_t l2_persist_max = 0, l2_window_max = 0;
  size_t l2_limit_prev = 0;
  bool l2_limit_set = false;
  int4* wl[2] = {nullptr, nullptr};
  unsigned wl_cap = 0;
  // false: each list holds max_edges / 2 entries plus slack (every symmetric
  // input); true: max_edges plus slack (any input). A solve whose scan
  // overflows the half-size lists is repeated after they are grown.
  bool wl_full = false;
  // the last device solve, kept so ecl_mst_ctx_sync can repeat it after a
  // worklist overflow
  bool pending = false;
  ecl_graph pend_graph = {};
  unsigned char* pend_out = nullptr;
  mst_opts pend_opts = {};
  cudaStream_t pend_stream = nullptr;
  bool resolved = false;  // the last ecl_mst_ctx_sync repeated the solve
  // pipelined host-buffer solves (ecl_mst_ctx_run_host_async): two device
  // buffer sets used in turn (set 0 is the one run_host uses), a copy-in and a
  // copy-out stream, the events that order them, a sticky device error word
  // and the calls since the last ecl_mst_ctx_wait (repeated after a
  // worklist overflow)
  struct HostSet {
    int* nindex = nullptr;
    int* nlist = nullptr;
    int* eweight = nullptr;
    unsigned char* inMST = nullptr;
    cudaEvent_t in_done = nullptr, solved = nullptr, out_done = nullptr;
    bool used = false;
  };
  HostSet hs[2];
  cudaStream_t cin = nullptr, cout = nullptr;
  unsigned async_seq = 0;
  unsigned* sticky = nullptr;
  struct AsyncCall {
    ecl_graph g;
    uint8_t* out;
    mst_opts opts;
  };
  std::vector<AsyncCall> async_calls;
  int* slist = nullptr;    // ECL_FLAG_NO_TUPLES: vertex of every CSR entry (allocated on first use)
  int vertex_grid = 0;     // ECL_FLAG_NO_EDGE_BASED: cooperative grid of the vertex-centric rounds
  int* first_v = nullptr;  // task -> row table of the scans
  unsigned* tree_bits = nullptr;  // bit v: v lies in the light phase's largest tree
  int first_v_cap = 0;
  DevState* st = nullptr;
  DevState* st_host = nullptr;  // statistics of the last solve
  int round_grid = 0;  // most co-resident CTAs of k_round
  int abl_grid = 0;    // the same of k_rounds (ablation variants)
  int group_grid = 0;  // the same of k_group
  // device CSR + output for host-buffer runs (allocated on first use)
  int* d_nindex = nullptr;
  int* d_nlist = nullptr;
  int* d_eweight = nullptr;
  unsigned char* d_inMST = nullptr;
  // timed solves: start, light scan end, light rounds end, heavy scan end, end,
  // prep end, flatten end
  cudaEvent_t ev[7] = {};
  // learned schedule: MLP parameters (and the load they came from), the 16
  // features, degree accumulators, the sorted 4096-entry weight sample
  float* ml_params = nullptr;
  unsigned ml_version = ~0u;
  float* ml_feat = nullptr;  // the features of the last learned solve
  bool ml_features_set = false;
  void* ml_acc = nullptr;
  int* ml_sample = nullptr;
};

namespace {

int cuda_status(cudaError_t e) {
  if (e == cudaSuccess) return ECL_OK;
  if (e == cudaErrorMemoryAllocation) return ECL_ERR_ALLOC;
  if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) return ECL_ERR_NO_DEVICE;
  return ECL_ERR_CUDA;
}

#define ECL_CUDA_TRY(call)                         \
  do {                                             \
    cudaError_t e_ = (call);                       \
    if (e_ != cudaSuccess) return cuda_status(e_); \
  } while (0)

int device_error_status(unsigned err) {
  if (err & kErrTimeout) return ECL_ERR_TIMEOUT;
  if (err & (kErrFormat | kErrIds)) return ECL_ERR_FORMAT;
  if (err & kErrOverflow) return ECL_ERR_OVERFLOW;
  if (err & kErrRounds) return ECL_ERR_OVERFLOW;
  return ECL_OK;
}

int coop_grid(const void* fn, int threads, int sm_count) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0) != cudaSuccess)
    return 0;
  return per_sm * sm_count;
}

// The solve's slot arrays inside ctx->slots, packed for n vertices.
struct Slots {
  u64* minv0;
  u64* minv1;
  int* parent;
  size_t bytes;  // 20n
};
Slots slots_for(void* base, int n) {
  Slots sl;
  sl.minv0 = (u64*)base;
  sl.minv1 = sl.minv0 + n;
  sl.parent = (int*)(sl.minv1 + n);
  sl.bytes = (size_t)n * (2 * sizeof(u64) + sizeof(int));
  return sl;
}

// Launch `kernel` with optional launch attributes: cooperative (grid-wide
// barriers) and an L2 access-policy window. Without either it is a plain
// launch.
template <typename... KArgs, typename... Args>
int launch_ex(void (*kernel)(KArgs...), int grid, int threads, size_t smem, cudaStream_t s, bool coop,
              const cudaAccessPolicyWindow* win, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  unsigned na = 0;
  if (coop) {
    at[na].id = cudaLaunchAttributeCooperative;
    at[na].val.cooperative = 1;
    na++;
  }
  if (win) {
    at[na].id = cudaLaunchAttributeAccessPolicyWindow;
    at[na].val.accessPolicyWindow = *win;
    na++;
  }
  cfg.attrs = na ? at : nullptr;
  cfg.numAttrs = na;
  return cuda_status(cudaLaunchKernelEx(&cfg, kernel, args...));
}

// Launch `clusters` clusters of `size` CTAs.
template <typename... KArgs, typename... Args>
int launch_cluster(void (*kernel)(KArgs...), int size, int clusters, int threads, size_t smem, cudaStream_t s,
                   Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(size * clusters);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = size;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cuda_status(cudaLaunchKernelEx(&cfg, kernel, args...));
}

int prepare_scan_kernels();
int prepare_cluster_kernels();
int prepare_round_kernels();

// Bytes of the vertex bits for up to `nodes` vertices.
constexpr size_t tree_bits_bytes(int64_t nodes) { return (size_t)(nodes + 31) / 32 * sizeof(unsigned); }

// Entries of the task->row table for up to `edges` CSR entries.
int64_t first_v_entries(int64_t edges) { return edges / kGran + 2; }

int enqueue_prep(const PrepArgs& pa, int sm_count, cudaStream_t s, const cudaAccessPolicyWindow* win = nullptr) {
  const int grid = (int)std::min<int64_t>(((int64_t)pa.nodes + kThreads - 1) / kThreads, (int64_t)sm_count * 16);
  return launch_ex(k_prep, std::max(grid, 1), kThreads, 0, s, false, win, pa);
}

// Round-kernel ablation bits from the option flags.
unsigned round_ablation(int flags) {
  return ((flags & ECL_FLAG_NO_GUARDS) ? kAblNoGuards : 0u) | ((flags & ECL_FLAG_NO_WARP_COOP) ? kAblNoCoop : 0u) |
         ((flags & ECL_FLAG_DEDUP) ? kDedup : 0u) | ((flags & ECL_FLAG_NO_FIND_CACHE) ? kAblNoFindCache : 0u) |
         ((flags & ECL_FLAG_NO_IMPLICIT_COMPRESSION) ? kAblNoIPC : 0u) |
         ((flags & ECL_FLAG_NO_TUPLES) ? kAblNoTuples : 0u) | ((flags & ECL_FLAG_NO_DATA_DRIVEN) ? kAblNoDD : 0u) |
         ((flags & ECL_FLAG_VARIANT_BASE) ? kAblBase : 0u);
}

// The reference's later ablation steps, which only the single-graph engine runs.
constexpr int kDeoptFlags = ECL_FLAG_NO_IMPLICIT_COMPRESSION | ECL_FLAG_NO_TUPLES | ECL_FLAG_NO_DATA_DRIVEN |
                            ECL_FLAG_NO_EDGE_BASED;

}  // namespace

namespace {

// A phase's worklist holds one entry per one-direction CSR entry
// (nlist[j] > v) at most. That is edges / 2 for a symmetric input (the size
// the reference gives it, ECL_MST.cu:279) and up to `edges` otherwise; the
// lists start at the symmetric size and grow to the full one when a solve
// overflows them. Both carry slack for the unused tails of the scan warps'
// slot chunks.
int alloc_worklists(ecl_mst_ctx* c, bool full) {
  cudaFree(c->wl[0]);  // holds both
  c->wl[0] = c->wl[1] = nullptr;
  const int64_t keep = full ? c->max_edges : c->max_edges / 2;
  c->wl_cap = (unsigned)std::max<int64_t>(keep + std::min<int64_t>(c->max_edges, kWlSlack), 1);
  c->wl_full = full;
  ECL_CUDA_TRY(cudaMalloc(&c->wl[0], 2 * (size_t)c->wl_cap * sizeof(int4)));
  c->wl[1] = c->wl[0] + c->wl_cap;
  return ECL_OK;
}

}  // namespace

extern "C" void ecl_default_opts(mst_opts* o) {
  if (!o) return;
  memset(o, 0, sizeof(*o));
  o->threshold_mode = ECL_THRESH_HEURISTIC;
  o->quantile = 1.0f;
}

// `full`: worklists for any input from the start.
static int ctx_create(int device, int64_t max_nodes, int64_t max_edges, bool full, ecl_mst_ctx** out) {
  if (!out || max_nodes < 1 || max_edges < 0 || max_nodes > INT32_MAX || max_edges > INT32_MAX)
    return ECL_ERR_INVALID_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return ECL_ERR_NO_DEVICE;
  if (device < 0 || device >= ndev) return ECL_ERR_INVALID_ARG;
  ECL_CUDA_TRY(cudaSetDevice(device));
  ecl_mst_ctx* c = new (std::nothrow) ecl_mst_ctx();
  if (!c) return ECL_ERR_ALLOC;
  c->device = device;
  c->max_nodes = max_nodes;
  c->max_edges = max_edges;
  int st = ECL_OK;
  auto fail = [&](int s) {
    ecl_mst_ctx_destroy(c);
    return s;
  };
  int coop = 0, persist = 0, window = 0;
  for (const auto& q : {std::make_pair(&coop, cudaDevAttrCooperativeLaunch),
                        std::make_pair(&c->sm_count, cudaDevAttrMultiProcessorCount),
                        std::make_pair(&persist, cudaDevAttrMaxPersistingL2CacheSize),
                        std::make_pair(&window, cudaDevAttrMaxAccessPolicyWindowSize)})
    if ((st = cuda_status(cudaDeviceGetAttribute(q.first, q.second, device)))) return fail(st);
  if (!coop) return fail(ECL_ERR_UNSUPPORTED);
  if ((st = cuda_status(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking)))) return fail(st);
  if ((st = cuda_status(cudaStreamCreateWithFlags(&c->side, cudaStreamNonBlocking)))) return fail(st);
  if ((st = cuda_status(cudaEventCreateWithFlags(&c->fork, cudaEventDisableTiming)))) return fail(st);
  if ((st = cuda_status(cudaEventCreateWithFlags(&c->join, cudaEventDisableTiming)))) return fail(st);
  if ((st = cuda_status(cudaEventCreateWithFlags(&c->prep_done, cudaEventDisableTiming)))) return fail(st);
  c->l2_persist_max = (size_t)std::max(persist, 0);
  c->l2_window_max = (size_t)std::max(window, 0);
  c->first_v_cap = (int)first_v_entries(max_edges);
  // one allocation (its pointer is c->slots) for everything but the worklists,
  // which may grow: an allocation and its release take 0.7 ms together
  size_t bytes = 0;
  auto carve = [&](size_t size) {
    const size_t at = bytes;
    bytes += (size + 255) & ~(size_t)255;
    return at;
  };
  carve((size_t)max_nodes * (2 * sizeof(u64) + sizeof(int)));
  const size_t first_v = carve((size_t)c->first_v_cap * sizeof(int)), bits = carve(tree_bits_bytes(max_nodes));
  const size_t state = carve(sizeof(DevState)), params = carve(ECL_MLP_PARAMS * sizeof(float));
  const size_t feat = carve(ECL_MLP_INPUTS * sizeof(float)), acc = carve(sizeof(FeatAcc));
  const size_t sample = carve(4096 * sizeof(int));
  if ((st = cuda_status(cudaMalloc(&c->slots, bytes)))) return fail(st);
  unsigned char* base = static_cast<unsigned char*>(c->slots);
  c->first_v = reinterpret_cast<int*>(base + first_v);
  c->tree_bits = reinterpret_cast<unsigned*>(base + bits);
  c->st = reinterpret_cast<DevState*>(base + state);
  c->ml_params = reinterpret_cast<float*>(base + params);
  c->ml_feat = reinterpret_cast<float*>(base + feat);
  c->ml_acc = base + acc;
  c->ml_sample = reinterpret_cast<int*>(base + sample);
  if ((st = alloc_worklists(c, full))) return fail(st);
  c->st_host = new (std::nothrow) DevState();  // not pinned: that takes 2 ms, a copy to it 10 us
  if (!c->st_host) return fail(ECL_ERR_ALLOC);
  for (auto& e : c->ev)
    if ((st = cuda_status(cudaEventCreate(&e)))) return fail(st);
  // every CTA of a round pass writes one segment of the round's output list
  c->round_grid = std::min(coop_grid((const void*)k_round, kBorThreads, c->sm_count), kMaxRoundCtas);
  c->abl_grid = std::min(coop_grid((const void*)k_rounds, kRoundThreads, c->sm_count), kMaxRoundCtas);
  c->group_grid = coop_grid((const void*)k_group, kGroupThreads, c->sm_count);
  c->vertex_grid = coop_grid((const void*)k_rounds_vertex, kRoundThreads, c->sm_count);
  if ((st = prepare_scan_kernels())) return fail(st);
  if ((st = prepare_round_kernels())) return fail(st);
  if ((st = prepare_cluster_kernels())) return fail(st);
  if (c->round_grid <= 0 || c->abl_grid <= 0 || c->group_grid <= 0 || c->vertex_grid <= 0) return fail(ECL_ERR_CUDA);
  *out = c;
  return ECL_OK;
}

extern "C" int ecl_mst_ctx_create(int device, int64_t max_nodes, int64_t max_edges,
                                  ecl_mst_ctx** out) {
  return ctx_create(device, max_nodes, max_edges, false, out);
}

extern "C" void ecl_mst_ctx_destroy(ecl_mst_ctx* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  if (c->l2_limit_set) {  // hand the persisting set-aside back as it was
    cudaCtxResetPersistingL2Cache();
    cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, c->l2_limit_prev);
  }
  cudaFree(c->slots);     // and what lies behind the slots
  cudaFree(c->wl[0]);     // both lists
  cudaFree(c->slist);
  delete c->st_host;
  cudaFree(c->d_nindex);  // all four arrays
  if (c->cin) cudaStreamSynchronize(c->cin);
  if (c->cout) cudaStreamSynchronize(c->cout);
  cudaFree(c->hs[1].nindex);
  cudaFree(c->sticky);
  for (auto& h : c->hs)
    for (cudaEvent_t e : {h.in_done, h.solved, h.out_done})
      if (e) cudaEventDestroy(e);
  if (c->cin) cudaStreamDestroy(c->cin);
  if (c->cout) cudaStreamDestroy(c->cout);
  for (auto& e : c->ev)
    if (e) cudaEventDestroy(e);
  if (c->side) cudaStreamSynchronize(c->side);
  if (c->exec) cudaGraphExecDestroy(c->exec);
  if (c->fork) cudaEventDestroy(c->fork);
  if (c->join) cudaEventDestroy(c->join);
  if (c->prep_done) cudaEventDestroy(c->prep_done);
  if (c->side) cudaStreamDestroy(c->side);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

extern "C" void* ecl_mst_ctx_stream(ecl_mst_ctx* c) { return c ? (void*)c->stream : nullptr; }

extern "C" int ecl_mst_ctx_learned_features(ecl_mst_ctx* c, float* out16) {
  if (!c || !out16) return ECL_ERR_INVALID_ARG;
  if (!c->ml_features_set) return ECL_ERR_UNSUPPORTED;
  ECL_CUDA_TRY(cudaSetDevice(c->device));
  ECL_CUDA_TRY(cudaStreamSynchronize(c->side));
  ECL_CUDA_TRY(cudaMemcpy(out16, c->ml_feat, ECL_MLP_INPUTS * sizeof(float), cudaMemcpyDeviceToHost));
  return ECL_OK;
}

extern "C" int ecl_mst_ctx_l2_reset(ecl_mst_ctx* c) {
  if (!c) return ECL_ERR_INVALID_ARG;
  ECL_CUDA_TRY(cudaSetDevice(c->device));
  ECL_CUDA_TRY(cudaCtxResetPersistingL2Cache());
  return ECL_OK;
}

namespace {
int run_device_once(ecl_mst_ctx* c, const ecl_graph* g, uint8_t* d_inMST, const mst_opts* opts, void* stream,
                    ecl_mst_stats* stats);
int grow_worklists(ecl_mst_ctx* c);
}  // namespace

extern "C" int ecl_mst_ctx_sync(ecl_mst_ctx* c) {
  if (!c) return ECL_ERR_INVALID_ARG;
  ECL_CUDA_TRY(cudaSetDevice(c->device));
  c->resolved = false;
  cudaStream_t s = c->pending ? c->pend_stream : c->stream;
  ECL_CUDA_TRY(cudaStreamSynchronize(s));
  if (s != c->stream) ECL_CUDA_TRY(cudaStreamSynchronize(c->stream));
  unsigned err = 0;
  ECL_CUDA_TRY(cudaMemcpy(&err, &c->st->error, sizeof(unsigned), cudaMemcpyDeviceToHost));
  if ((err & kErrOverflow) && c->pending && !c->wl_full) {
    // the input had more one-direction entries than half its CSR entries:
    // solve it again with worklists that hold every entry
    c->pending = false;
    int st = grow_worklists(c);
    if (st) return st;
    if ((st = run_device_once(c, &c->pend_graph, c->pend_out, &c->pend_opts, c->pend_stream, nullptr))) return st;
    c->resolved = true;
    ECL_CUDA_TRY(cudaStreamSynchronize(c->pend_stream));
    ECL_CUDA_TRY(cudaMemcpy(&err, &c->st->error, sizeof(unsigned), cudaMemcpyDeviceToHost));
  }
  c->pending = false;
  return device_error_status(err);
}

namespace {

// Opt the scans into their shared memory (once per device).
int prepare_scan_kernels() {
  for (auto k : {k_scan_light<false>, k_scan_light<true>})
    ECL_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ScanSmem<true>)));
  for (auto k : {k_scan_heavy<false>, k_scan_heavy<true>})
    ECL_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ScanSmem<false>)));
  return ECL_OK;
}

// Shared memory an SM sets aside while the rounds and the kernels between the
// scans run, in per cent. An SM changes the split between shared memory and L1
// only when it is idle, so with several streams a kernel of the smallest
// split waits for the SMs that run another's scan (3 x 72 KB) to drain: a
// batch of 39 large graphs on 8 streams 8.0 ms at 25 to 60 per cent, 9.1 with
// the driver's choice; one solve at a time is the same (RMAT-22 1.47 ms) but at
// 12 or 100, where k_round's CTAs or its L1 hits go missing (1.57, 1.83).
constexpr int kCarveout = 40;
int prepare_round_kernels() {
  for (const void* k : {(const void*)k_round, (const void*)k_round_tail, (const void*)k_prep, (const void*)k_flatten,
                        (const void*)k_group})
    ECL_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, kCarveout));
  return ECL_OK;
}

// Persistent scan: as many CTAs as can be resident at once, or one per
// kScanWarps tasks. The CTAs' slot chunk is sized so that the unused chunk
// tails (at most chunk - 1 per CTA and list, two lists to an array) fit in the
// worklist's slack; 0 = slots are reserved exactly.
int launch_scan(int kind, const ScanArgs& sa, int sm_count, unsigned wl_slack, cudaStream_t s,
                const cudaAccessPolicyWindow* win = nullptr) {
  const int blocks = std::max(1, std::min((sa.tiles + kScanWarps - 1) / kScanWarps, kScanBlocks * sm_count));
  ScanArgs a = sa;
  a.chunk = std::min(kScanMaxChunk, wl_slack / (unsigned)(2 * blocks));
  if (a.chunk < kScanMinChunk) a.chunk = 0;
  const bool vec = (((uintptr_t)(kind == kLight ? sa.eweight : sa.nlist)) & 15) == 0;
  if (kind == kLight)
    return launch_ex(vec ? k_scan_light<true> : k_scan_light<false>, blocks, kScanThreads, sizeof(ScanSmem<true>), s,
                     false, win, a);
  return launch_ex(vec ? k_scan_heavy<true> : k_scan_heavy<false>, blocks, kScanThreads, sizeof(ScanSmem<false>), s,
                   false, win, a);
}

// Flattened parent[] and the largest tree's vertex bits.
int launch_flatten(int list, int* parent, int n, const DevState* st, unsigned* tree_bits, int sm_count, cudaStream_t s,
                   const cudaAccessPolicyWindow* win = nullptr) {
  const int grid = (int)std::min<int64_t>(((int64_t)n + 4 * kThreads - 1) / (4 * kThreads), (int64_t)sm_count * 4);
  return launch_ex(k_flatten, std::max(grid, 1), kThreads, 0, s, false, win, parent, n, st, tree_bits, list);
}

// One phase's Boruvka rounds: the grid-wide kernel, then the cluster kernel
// that ends the phase. The ablation switches run the variants kept in
// k_rounds. `per_sm`: the caller's limit on CTAs per SM (0 = none).
int enqueue_rounds(const RoundArgs& ra, int list, int edges, int sm_count, int per_sm, int round_grid, int abl_grid,
                   cudaStream_t s, const cudaAccessPolicyWindow* win) {
  const int limit = per_sm > 0 ? per_sm * sm_count : INT_MAX;
  if (ra.abl) {
    const int grid = std::max(1, std::min({abl_grid, limit, (edges / 2 + kRoundThreads - 1) / kRoundThreads + 1}));
    return launch_ex(k_rounds, grid, kRoundThreads, 0, s, true, win, ra);
  }
  constexpr int tile = kBorThreads * kBorEpt;
  BorArgs ba{};
  ba.phase = ra.phase;
  ba.nodes = ra.nodes;
  ba.list = list;
  ba.wl0 = ra.wl0;
  ba.wl1 = ra.wl1;
  ba.wl_cap = ra.wl_cap;
  ba.parent = ra.parent;
  ba.minv = ra.minv0;
  ba.roots0 = reinterpret_cast<int*>(ra.minv1);  // the second min array's space holds the root lists
  ba.roots1 = ba.roots0 + ra.nodes;
  ba.inMST = ra.inMST;
  ba.st = ra.st;
  ba.solo = ra.small_tail;
  ba.tail = ra.small_tail ? std::max(ra.small_tail, kTailEntries) : 0u;
  ba.min_tiles = ra.min_tiles;
  ba.count_atomics = ra.count_atomics;
  const int grid = std::max(1, std::min({round_grid, limit, (edges / 2 + tile - 1) / tile + 1}));
  const int st = launch_ex(k_round, grid, kBorThreads, 0, s, true, win, ba);
  if (st) return st;
  return launch_ex(k_round_tail, kTailCtas, kTailThreads, 0, s, false, win, ba);
}

// Opt the one-CTA kernels into their shared memory (once per device).
int prepare_cluster_kernels() {
  ECL_CUDA_TRY(cudaFuncSetAttribute(k_cluster<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClSmem));
  ECL_CUDA_TRY(cudaFuncSetAttribute(k_batch_cluster<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClSmem));
  return ECL_OK;
}

// CTAs of the cluster that solves a graph alone (k_cluster), 0 = k_group does.
// One CTA up to kClusterShare entries and what its shared memory holds, else
// one per quarter of that, in entries or vertices: the roots pass looks at every
// vertex, and a thread's unions and walks follow one another (the path of 16 000
// equal weights 55 us on 8 CTAs, 85 on 4; ER 3000 98 against 108). Measured
// against k_group: ER of 1000 vertices 57 us (one CTA) against 99, ER 4000 107
// (4 CTAs) against 156, 16 000-vertex grid (8 CTAs) 138 against 165; from 128K
// entries on k_group is the faster one, and beyond kClusterNodes vertices with
// few entries too (0.2 per vertex: 40 000 57 us against 82, 60 000 64 against
// 122; 32 000 84 against 59 on 8 CTAs).
int cluster_ctas(int n, int m, unsigned wl_cap) {
  if (m > kClusterEdges || n > kClusterNodes || (unsigned)m > wl_cap) return 0;
  if (m <= kClusterShare && n <= kClVertices) return 1;
  int c = 2;
  while (c < kClMaxCtas && std::max(m, n) > c * (kClusterShare / 4)) c *= 2;
  return c;
}

int enqueue_cluster(ClArgs ca, int ctas, const mst_opts* o, cudaStream_t s) {
  ca.mode = o->threshold_mode;
  ca.explicit_thr = o->threshold;
  ca.split = o->degree_split > 0 ? o->degree_split : kDefaultSplit;
  ca.quantile = o->quantile;
  ca.count_atomics = (o->flags & ECL_FLAG_STATS) ? 1 : 0;
  if (ctas == 1) return launch_cluster(k_cluster<true>, 1, 1, kClThreads, kClSmem, s, ca);
  return launch_cluster(k_cluster<false>, ctas, 1, kClThreads, 0, s, ca);
}

// A whole solve in one launch (k_group), on one CTA per kGroupCtaTiles scan
// tiles of the graph; `per_sm` is the caller's limit on CTAs per SM (0 = none)
// and `wl_slack` what the worklists hold beyond the entries a scan can keep.
// 1, 2, 4, 8 tiles per CTA: RMAT-14 163, 156, 162, 191 us; ER 200k 292, 295,
// 309, 337; the 1000 x 1000 grid 455, 456, 454, 475.
constexpr int kGroupCtaTiles = 2;
int enqueue_group(GroupArgs ga, const mst_opts* o, unsigned wl_slack, int sm_count, int group_grid, cudaStream_t s,
                  const cudaAccessPolicyWindow* win) {
  constexpr int per_cta = kGroupCtaTiles * kGroupTile;
  const int limit = o->ctas_per_sm > 0 ? o->ctas_per_sm * sm_count : INT_MAX;
  const int grid = std::max(1, std::min({group_grid, limit, std::max((ga.edges + per_cta - 1) / per_cta,
                                                                     (int)(((int64_t)ga.nodes + per_cta - 1) / per_cta))}));
  ga.mode = o->threshold_mode;
  ga.explicit_thr = o->threshold;
  ga.split = o->degree_split > 0 ? o->degree_split : kDefaultSplit;
  ga.quantile = o->quantile;
  ga.solo = o->small_tail < 0 ? 0u : (o->small_tail == 0 ? kDefaultSmallTail : (unsigned)o->small_tail);
  if (o->flags & ECL_FLAG_NO_SMALL_TAIL) ga.solo = 0;
  ga.min_tiles = o->round_min_tiles < 0 ? 0 : (o->round_min_tiles == 0 ? kDefaultMinTiles : o->round_min_tiles);
  ga.count_atomics = (o->flags & ECL_FLAG_STATS) ? 1 : 0;
  ga.chunk = std::min(256u, wl_slack / (unsigned)grid);
  if (ga.chunk < 128) ga.chunk = 0;  // a warp may append 128 entries at once
  return launch_ex(k_group, grid, kGroupThreads, 0, s, grid > 1, win, ga);
}

// The L2 access-policy window of a solve (ECL_FLAG_L2_PERSIST): the packed
// min-slot and parent arrays (20n bytes; the min slots alone when the window
// limit is smaller), with the share of lines the persisting set-aside can
// hold marked persisting and the rest left normal.
bool l2_window(const ecl_mst_ctx* c, const Slots& sl, bool parent_only, cudaAccessPolicyWindow* w) {
  if (!c->l2_limit_set || c->l2_window_max == 0) return false;
  memset(w, 0, sizeof(*w));
  w->base_ptr = parent_only ? (void*)sl.parent : (void*)sl.minv0;
  size_t bytes = parent_only ? (sl.bytes / 5) : sl.bytes;  // parent is 4n of the 20n
  bytes = std::min(bytes, c->l2_window_max);
  if (bytes == 0) return false;
  w->num_bytes = bytes;
  size_t persist = 0;
  cudaDeviceGetLimit(&persist, cudaLimitPersistingL2CacheSize);
  w->hitRatio = (float)std::min(1.0, (double)persist / (double)bytes);
  w->hitProp = cudaAccessPropertyPersisting;
  w->missProp = cudaAccessPropertyStreaming;
  return true;
}

// The learned schedule's steps around k_prep. The weight sample is sorted on
// `side` from the start of the solve (ecl_learned_sample); k_prep gathers the
// degree statistics into `acc` on the solve's stream; the MLP then runs on
// `side`, and the light scan waits for it.
struct LearnedPlan {
  cudaStream_t side;
  cudaEvent_t prep_done, join;
  FeatAcc* acc;
};

// Start of a learned solve on stream q: zero the degree accumulator (before
// k_prep adds to it), then fork the side stream and sort the weight sample
// there. Fills lp->acc.
int learned_fork(ecl_mst_ctx* c, const ecl_graph* g, cudaStream_t q, LearnedPlan* lp) {
  lp->acc = static_cast<FeatAcc*>(c->ml_acc);
  c->ml_features_set = true;
  ECL_CUDA_TRY(cudaMemsetAsync(lp->acc, 0, sizeof(FeatAcc), q));
  ECL_CUDA_TRY(cudaEventRecord(c->fork, q));
  ECL_CUDA_TRY(cudaStreamWaitEvent(lp->side, c->fork, 0));
  return ecl_learned_sample(c, g, lp->side);
}

// The share of the entries that the light phase will take, as far as the host
// can tell: the reference heuristic's expectation where the threshold is
// chosen on the device.
double light_share(const mst_opts* o, int n, int m) {
  if (o->threshold_mode == ECL_THRESH_NONE) return 1.0;
  if (o->threshold_mode == ECL_THRESH_QUANTILE) return std::min(1.0, (double)o->quantile);
  return m / n < 4 ? 1.0 : (std::min(19, (int)(3.0 * n * 20 / m)) + 1) / 21.0;
}

int enqueue_solve(ecl_mst_ctx* c, const ecl_graph* g, unsigned char* d_inMST, const mst_opts* o,
                  cudaStream_t s, bool timed, const LearnedPlan* lp = nullptr) {
  const int n = g->nodes, m = g->edges;
  const int split = o->degree_split > 0 ? o->degree_split : kDefaultSplit;
  const int tiles = (int)(((int64_t)m + kGran - 1) / kGran);
  const Slots sl = slots_for(c->slots, n);
  // L2 persistence: k_prep writes the slots and parent, the rounds hammer
  // them, the flatten pass and the heavy scan gather parent[]
  cudaAccessPolicyWindow w_all, w_par;
  const bool l2 = (o->flags & ECL_FLAG_L2_PERSIST) != 0;
  const cudaAccessPolicyWindow* win_all = l2 && l2_window(c, sl, false, &w_all) ? &w_all : nullptr;
  const cudaAccessPolicyWindow* win_par = l2 && l2_window(c, sl, true, &w_par) ? &w_par : nullptr;
  const bool one_launch = !lp && !round_ablation(o->flags) && !(o->flags & ECL_FLAG_NO_EDGE_BASED);
  if (const int ctas = one_launch && o->ctas_per_sm == 0 && !(o->flags & ECL_FLAG_NO_SMALL_TAIL)
                           ? cluster_ctas(n, m, c->wl_cap) : 0) {
    ClArgs ca{};
    ca.nodes = n;
    ca.edges = m;
    ca.nindex = g->nindex;
    ca.nlist = g->nlist;
    ca.eweight = g->eweight;
    ca.inMST = d_inMST;
    ca.wl0 = c->wl[0];
    ca.wl1 = c->wl[1];
    ca.parent = sl.parent;
    ca.minv = sl.minv0;
    ca.st = c->st;
    const int r = enqueue_cluster(ca, ctas, o, s);
    if (r) return r;
    if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[4], s));
    return ECL_OK;
  }
  if (m <= kGroupEdges && one_launch) {
    GroupArgs ga{};
    ga.nodes = n;
    ga.edges = m;
    ga.nindex = g->nindex;
    ga.nlist = g->nlist;
    ga.eweight = g->eweight;
    ga.inMST = d_inMST;
    ga.parent = sl.parent;
    ga.minv = sl.minv0;
    ga.roots0 = reinterpret_cast<int*>(sl.minv1);
    ga.roots1 = ga.roots0 + n;
    ga.wl0 = c->wl[0];
    ga.wl1 = c->wl[1];
    ga.wl_cap = c->wl_cap;
    ga.st = c->st;
    const int r = enqueue_group(ga, o, c->wl_cap - (unsigned)(c->wl_full ? m : m / 2), c->sm_count, c->group_grid, s,
                                win_all);
    if (r) return r;
    if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[4], s));
    return ECL_OK;
  }
  PrepArgs pa{};
  pa.nodes = n;
  pa.edges = m;
  pa.nindex = g->nindex;
  pa.eweight = g->eweight;
  pa.parent = sl.parent;
  pa.minv0 = sl.minv0;
  pa.minv1 = sl.minv1;
  pa.first_v = c->first_v;
  pa.tiles = tiles;
  pa.mode = o->threshold_mode;
  pa.explicit_thr = o->threshold;
  pa.split = split;
  pa.quantile = o->quantile;
  pa.st = c->st;
  pa.feat = lp ? lp->acc : nullptr;
  const unsigned abl = round_ablation(o->flags);
  pa.both_slots = abl != 0;
  // The launches that lists split by weight need (split_ranks): about 20 us if
  // the device then splits none. Below six entries per vertex it does not pay (a
  // 1500 x 2000 grid 0.94 ms against 0.82), and the ablation variants keep one
  // list per phase.
  const bool lists = abl == 0 && !(o->flags & ECL_FLAG_NO_EDGE_BASED) && m / n >= 6 &&
                     (n >= kMidNodes || light_share(o, n, m) * 0.5 * m >= kSplitMin);
  pa.use_lists = lists;
  // whether the heavy phase can run at all (the device may still decide not)
  const bool two_phases = o->threshold_mode == ECL_THRESH_LEARNED || o->threshold_mode == ECL_THRESH_EXPLICIT ||
                          (o->threshold_mode == ECL_THRESH_QUANTILE && o->quantile < 1.0f) ||
                          (o->threshold_mode == ECL_THRESH_HEURISTIC && m / n >= 4);
  int st;
  if ((st = enqueue_prep(pa, c->sm_count, s, win_all))) return st;
  if (lp) {  // the network, once k_prep's degree statistics are complete
    ECL_CUDA_TRY(cudaEventRecord(lp->prep_done, s));
    ECL_CUDA_TRY(cudaStreamWaitEvent(lp->side, lp->prep_done, 0));
    if ((st = ecl_learned_apply(c, g, lp->side, c->st, lists))) return st;
    ECL_CUDA_TRY(cudaEventRecord(lp->join, lp->side));
    ECL_CUDA_TRY(cudaStreamWaitEvent(s, lp->join, 0));
  }
  const bool no_tuples = (o->flags & (ECL_FLAG_NO_TUPLES | ECL_FLAG_NO_EDGE_BASED)) == ECL_FLAG_NO_TUPLES;
  if (no_tuples) {  // the vertex of every entry, for the gathers of the rounds
    const int sgrid = (int)std::min<int64_t>(((int64_t)m + kThreads - 1) / kThreads, (int64_t)c->sm_count * 16);
    k_slist<<<std::max(sgrid, 1), kThreads, 0, s>>>(g->nindex, c->first_v, c->slist, m, c->st);
    ECL_CUDA_TRY(cudaGetLastError());
  }
  ScanArgs sa{};
  sa.nodes = n;
  sa.edges = m;
  sa.nindex = g->nindex;
  sa.nlist = g->nlist;
  sa.eweight = g->eweight;
  sa.first_v = c->first_v;
  sa.tiles = tiles;
  sa.parent = sl.parent;
  sa.wl0 = c->wl[0];
  sa.wl1 = c->wl[1];
  sa.wl_cap = c->wl_cap;
  sa.tree_bits = c->tree_bits;
  // a scan keeps at most m entries, m / 2 for the symmetric input the
  // half-size lists assume (more overflows, and the solve is repeated)
  const unsigned wl_slack = c->wl_cap - (unsigned)(c->wl_full ? m : m / 2);
  sa.inMST = d_inMST;
  sa.zero_vec = (((uintptr_t)d_inMST) & 15) == 0;
  sa.st = c->st;
  sa.ids = no_tuples ? 1 : 0;
  RoundArgs ra{};
  ra.nodes = n;
  ra.wl0 = c->wl[0];
  ra.wl1 = c->wl[1];
  ra.wl_cap = c->wl_cap;
  ra.parent = sl.parent;
  ra.minv0 = sl.minv0;
  ra.minv1 = sl.minv1;
  ra.inMST = d_inMST;
  ra.st = c->st;
  ra.small_tail = o->small_tail < 0 ? 0u : (o->small_tail == 0 ? kDefaultSmallTail : (unsigned)o->small_tail);
  if (o->flags & ECL_FLAG_NO_SMALL_TAIL) ra.small_tail = 0;
  ra.count_atomics = (o->flags & ECL_FLAG_STATS) ? 1 : 0;
  ra.abl = abl;
  ra.nlist = g->nlist;
  ra.eweight = g->eweight;
  ra.slist = c->slist;
  // entries that keep their endpoints clear the whole previous min array
  // each round, which one CTA of a small tail would do alone
  if (ra.abl & kAblKeepEnds) ra.small_tail = 0;
  ra.min_tiles = o->round_min_tiles < 0 ? 0 : (o->round_min_tiles == 0 ? kDefaultMinTiles : o->round_min_tiles);
  if (o->flags & ECL_FLAG_NO_EDGE_BASED) {
    // vertex-centric rounds straight over the CSR: no scans, no worklists
    if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[5], s));
    ECL_CUDA_TRY(cudaMemsetAsync(d_inMST, 0, (size_t)m, s));
    if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[1], s));
    ra.phase = 0;
    if ((st = launch_ex(k_rounds_vertex, c->vertex_grid, kRoundThreads, 0, s, true, nullptr, ra, g->nindex)))
      return st;
    if (timed) {
      ECL_CUDA_TRY(cudaEventRecord(c->ev[2], s));
      ECL_CUDA_TRY(cudaEventRecord(c->ev[6], s));
      ECL_CUDA_TRY(cudaEventRecord(c->ev[3], s));
    }
    ra.phase = 1;
    if ((st = launch_ex(k_rounds_vertex, c->vertex_grid, kRoundThreads, 0, s, true, nullptr, ra, g->nindex)))
      return st;
    if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[4], s));
    return ECL_OK;
  }
  if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[5], s));
  if ((st = launch_scan(kLight, sa, c->sm_count, wl_slack, s))) return st;
  if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[1], s));
  ra.phase = 0;
  auto rounds = [&](int list) {
    return enqueue_rounds(ra, list, m, c->sm_count, o->ctas_per_sm, c->round_grid, c->abl_grid, s, win_all);
  };
  auto flatten = [&](int list) {
    return launch_flatten(list, sl.parent, n, c->st, c->tree_bits, c->sm_count, s, win_par);
  };
  if ((st = rounds(kListLight0))) return st;
  if (lists && ((st = flatten(kListLight1)) || (st = rounds(kListLight1)))) return st;
  if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[2], s));
  ra.phase = 1;
  if (two_phases) {
    if (lists && n >= kMidNodes && ((st = flatten(kListMid)) || (st = rounds(kListMid)))) return st;
    if ((st = flatten(kListHeavy))) return st;
    if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[6], s));
    if ((st = launch_scan(kHeavy, sa, c->sm_count, wl_slack, s, win_par))) return st;
    if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[3], s));
    if ((st = rounds(kListHeavy))) return st;
  } else if (timed) {
    ECL_CUDA_TRY(cudaEventRecord(c->ev[6], s));
    ECL_CUDA_TRY(cudaEventRecord(c->ev[3], s));
  }
  if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[4], s));
  return ECL_OK;
}

int fill_stats(ecl_mst_ctx* c, ecl_mst_stats* stats, bool timed, bool breakdown = true) {
  ECL_CUDA_TRY(cudaMemcpyAsync(c->st_host, c->st, sizeof(DevState), cudaMemcpyDeviceToHost, c->stream));
  ECL_CUDA_TRY(cudaStreamSynchronize(c->stream));
  const DevState& h = *c->st_host;
  memset(stats, 0, sizeof(*stats));
  stats->threshold = h.threshold;
  stats->filtered = h.filtered;
  stats->degree_split = h.split;
  stats->rounds[0] = h.rounds[0];
  stats->rounds[1] = h.rounds[1];
  stats->status = (int32_t)h.error;
  for (int p = 0; p < 2; p++) {
    stats->scan_kept[p] = (int64_t)h.lists[2 * p].kept + h.lists[2 * p + 1].kept;
    for (int r = 0; r < ECL_MAX_ROUNDS; r++) {
      stats->wl_in[p][r] = h.wl_count[p][r];
      stats->wl_real[p][r] = h.wl_kept[p][r];
    }
  }
  stats->atomics = (int64_t)h.atomics;
  for (int p = 0; p < 2; p++) {
    u64 prev = h.t_round_start[p];
    for (int r = 0; r < h.rounds[p] && r < ECL_MAX_ROUNDS; r++) {
      for (int k : {2 * p, 2 * p + 1})  // a scan or a flattening pass lies before a list's rounds
        if (h.t_list[k] && h.r_list[k] == r) prev = h.t_list[k];
      const u64 a = h.t_round[p][2 * r], b = h.t_round[p][2 * r + 1];
      if (a && prev) stats->us_round[p][r][0] = (a - prev) * 1e-3f;
      if (b && a) stats->us_round[p][r][1] = (b - a) * 1e-3f;
      prev = b ? b : a;
    }
  }
  if (timed && !breakdown) {  // a replayed graph: only the whole solve is timed
    cudaEventElapsedTime(&stats->ms_total, c->ev[0], c->ev[4]);
  } else if (timed && h.t_step[kStepStart]) {  // one launch: the kernel's own times
    cudaEventElapsedTime(&stats->ms_total, c->ev[0], c->ev[4]);
    auto us = [](u64 from, u64 to) { return from && to > from ? (float)(to - from) * 1e-3f : 0.f; };
    const u64 *t = h.t_step, *r = h.t_round_start;
    auto end = [&](int p) {  // of the phase's rounds
      const int last = std::min(h.rounds[p], ECL_MAX_ROUNDS) - 1;
      return last < 0 ? r[p] : h.t_round[p][2 * last];
    };
    float(*sc)[3] = stats->us_scan;
    sc[0][1] = us(t[kStepStart], t[kStepPrep]);
    sc[0][2] = us(t[kStepPrep], r[0]);
    sc[1][1] = t[kStepFlatten] ? us(end(0), t[kStepFlatten]) : 0.f;
    sc[1][2] = us(t[kStepFlatten], r[1]);
    for (int p = 0; p < 2; p++) sc[p][0] = sc[p][1] + sc[p][2];
    stats->ms_rounds = (us(r[0], end(0)) + us(r[1], end(1))) * 1e-3f;
    stats->ms_scan = std::max(0.f, stats->ms_total - stats->ms_rounds);
  } else if (timed) {
    float t01, t12, t23, t34, t04;
    cudaEventElapsedTime(&t01, c->ev[0], c->ev[1]);
    cudaEventElapsedTime(&t12, c->ev[1], c->ev[2]);
    cudaEventElapsedTime(&t23, c->ev[2], c->ev[3]);
    cudaEventElapsedTime(&t34, c->ev[3], c->ev[4]);
    cudaEventElapsedTime(&t04, c->ev[0], c->ev[4]);
    stats->ms_scan = t01 + t23;
    stats->ms_rounds = t12 + t34;
    stats->ms_total = t04;
    float t05, t26;
    cudaEventElapsedTime(&t05, c->ev[0], c->ev[5]);
    cudaEventElapsedTime(&t26, c->ev[2], c->ev[6]);
    // the rounds of the heavy list set aside run between flatten's events
    const int mid_end = h.t_list[kListHeavy] ? h.r_list[kListHeavy] : h.rounds[1];
    if (h.t_list[kListMid] && mid_end > 0 && mid_end <= ECL_MAX_ROUNDS) {
      const u64 end = h.t_round[1][2 * mid_end - 2];
      const float ms = end > h.t_list[kListMid] ? (float)(end - h.t_list[kListMid]) * 1e-6f : 0.f;
      stats->ms_scan -= ms;
      stats->ms_rounds += ms;
      t23 -= ms;
      t26 -= ms;
    }
    stats->us_scan[0][0] = t01 * 1e3f;
    stats->us_scan[0][1] = t05 * 1e3f;
    stats->us_scan[0][2] = (t01 - t05) * 1e3f;
    stats->us_scan[1][0] = t23 * 1e3f;
    stats->us_scan[1][1] = t26 * 1e3f;
    stats->us_scan[1][2] = (t23 - t26) * 1e3f;
  }
  return device_error_status(h.error);
}

int check_graph_args(const ecl_mst_ctx* c, const ecl_graph* g, const void* inMST) {
  if (!c || !g || !inMST) return ECL_ERR_INVALID_ARG;
  if (g->nodes < 1 || g->edges < 0) return ECL_ERR_INVALID_ARG;
  if (g->nodes > c->max_nodes || g->edges > c->max_edges) return ECL_ERR_TOO_LARGE;
  if (!g->nindex || (g->edges > 0 && (!g->nlist || !g->eweight))) return ECL_ERR_INVALID_ARG;
  return ECL_OK;
}

int check_opts(const mst_opts* o) {
  if (o->threshold_mode < ECL_THRESH_HEURISTIC || o->threshold_mode > ECL_THRESH_LEARNED)
    return ECL_ERR_INVALID_ARG;
  if (o->degree_split < 0 || o->degree_split > (1 << 20)) return ECL_ERR_INVALID_ARG;
  if (o->ctas_per_sm < 0) return ECL_ERR_INVALID_ARG;
  if (o->batch_large_streams < 0 || o->batch_large_streams > 8) return ECL_ERR_INVALID_ARG;
  if (o->threshold_mode == ECL_THRESH_QUANTILE && !(o->quantile >= 0.0f)) return ECL_ERR_INVALID_ARG;
  return ECL_OK;
}

}  // namespace

int ecl_ctx_learned_buffers(ecl_mst_ctx* c, float** params, float** feat, void** acc, int** sample,
                            unsigned** version, int* sm_count) {
  *sample = c->ml_sample;
  *version = &c->ml_version;
  *params = c->ml_params;
  *feat = c->ml_feat;
  *acc = c->ml_acc;
  *sm_count = c->sm_count;
  return ECL_OK;
}

namespace {

int run_device_once(ecl_mst_ctx* c, const ecl_graph* g, uint8_t* d_inMST, const mst_opts* opts, void* stream,
                    ecl_mst_stats* stats) {
  int st = check_graph_args(c, g, d_inMST);
  if (st) return st;
  mst_opts o;
  if (opts) o = *opts;
  else ecl_default_opts(&o);
  if ((st = check_opts(&o))) return st;
  ECL_CUDA_TRY(cudaSetDevice(c->device));
  cudaStream_t s = stream ? (cudaStream_t)stream : c->stream;
  if (g->edges == 0) {
    if (stats) {
      memset(stats, 0, sizeof(*stats));
      stats->threshold = INT_MAX;
    }
    return ECL_OK;
  }
  // Graphs below kLearnedMinEdges CSR entries keep the reference heuristic:
  // there the feature pass costs about as much as any schedule can save.
  // Without loaded weights the heuristic is the fallback.
  if (o.threshold_mode == ECL_THRESH_LEARNED && (g->edges < kLearnedMinEdges || !ecl_learned_has_weights()))
    o.threshold_mode = ECL_THRESH_HEURISTIC;
  const bool timed = stats != nullptr;
  if ((o.flags & ECL_FLAG_NO_TUPLES) && !c->slist)  // the ablation's per-entry vertex list, once
    ECL_CUDA_TRY(cudaMalloc(&c->slist, (size_t)std::max<int64_t>(c->max_edges, 1) * sizeof(int)));
  if (o.flags & ECL_FLAG_L2_PERSIST) {
    // Persisting set-aside for this process's context, sized for the solve's
    // slot arrays (20n bytes) up to the device maximum; set before any
    // capture, restored when the context is destroyed.
    const size_t want = std::min(c->l2_persist_max, (size_t)g->nodes * (2 * sizeof(u64) + sizeof(int)));
    size_t cur = 0;
    ECL_CUDA_TRY(cudaDeviceGetLimit(&cur, cudaLimitPersistingL2CacheSize));
    if (!c->l2_limit_set) c->l2_limit_prev = cur;
    if (want > cur) ECL_CUDA_TRY(cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, want));
    c->l2_limit_set = want > 0 || c->l2_limit_set;
  }
  // inner_events: the per-phase timing events (not inside a captured graph)
  auto enqueue_all = [&](cudaStream_t q, bool inner_events) -> int {
    ECL_CUDA_TRY(cudaMemsetAsync(c->st, 0, sizeof(DevState), q));
    // the timed window starts before the learned schedule's feature pass
    if (inner_events) ECL_CUDA_TRY(cudaEventRecord(c->ev[0], q));
    if (o.threshold_mode != ECL_THRESH_LEARNED) return enqueue_solve(c, g, d_inMST, &o, q, inner_events);
    LearnedPlan lp{c->side, c->prep_done, c->join, nullptr};
    const int r = learned_fork(c, g, q, &lp);
    return r ? r : enqueue_solve(c, g, d_inMST, &o, q, inner_events, &lp);
  };
  // A solve repeated with the same graph, buffers and options (benchmarks,
  // iterative callers) is captured once as a CUDA graph and then replayed
  // with a single launch: the first repeat captures, later ones replay. A
  // replay is timed as a whole (events around the launch), so its stats have
  // ms_total but no per-phase breakdown; ECL_FLAG_NO_GRAPH keeps the direct
  // launches and the breakdown.
  int32_t qbits;  // the quantile's bit pattern
  memcpy(&qbits, &o.quantile, sizeof(qbits));
  const std::vector<long long> key = {
      g->nodes, g->edges, (long long)(uintptr_t)g->nindex, (long long)(uintptr_t)g->nlist,
      (long long)(uintptr_t)g->eweight, (long long)(uintptr_t)d_inMST, o.threshold_mode, o.threshold,
      (long long)qbits, o.degree_split, o.small_tail, o.flags, o.round_min_tiles, o.ctas_per_sm,
      (long long)(uintptr_t)c->wl[0], (long long)ecl_learned_weights_version()};
  const bool graph_ok = !(o.flags & ECL_FLAG_NO_GRAPH);
  bool replayed = false;
  auto replay = [&]() -> int {
    if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[0], s));
    ECL_CUDA_TRY(cudaGraphLaunch(c->exec, s));
    if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[4], s));
    replayed = true;
    return ECL_OK;
  };
  if (graph_ok && c->exec && c->exec_key == key) {
    if ((st = replay())) return st;
  } else if (graph_ok && key == c->last_key) {
    if (c->exec) {
      cudaGraphExecDestroy(c->exec);
      c->exec = nullptr;
    }
    cudaGraph_t graph = nullptr;
    bool captured = false;
    if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
      const int r = enqueue_all(s, false);
      const cudaError_t e = cudaStreamEndCapture(s, &graph);
      if (r == ECL_OK && e == cudaSuccess && graph && cudaGraphInstantiate(&c->exec, graph, 0) == cudaSuccess) {
        captured = true;
        c->exec_key = key;
      }
      if (graph) cudaGraphDestroy(graph);
    }
    cudaGetLastError();  // clear a failed capture's error state
    if (captured) {
      if ((st = replay())) return st;
    } else {
      c->exec = nullptr;
      if ((st = enqueue_all(s, timed))) return st;
    }
  } else {
    if ((st = enqueue_all(s, timed))) return st;
  }
  c->last_key = key;
  if (stats) {
    if (s != c->stream) {
      ECL_CUDA_TRY(cudaStreamSynchronize(s));
    }
    return fill_stats(c, stats, true, !replayed);
  }
  return ECL_OK;
}

// Worklists grown to hold every CSR entry; the captured solve refers to the
// old lists and is dropped.
int grow_worklists(ecl_mst_ctx* c) {
  ECL_CUDA_TRY(cudaSetDevice(c->device));
  ECL_CUDA_TRY(cudaDeviceSynchronize());
  if (c->exec) {
    cudaGraphExecDestroy(c->exec);
    c->exec = nullptr;
  }
  c->exec_key.clear();
  c->last_key.clear();
  return alloc_worklists(c, true);
}

}  // namespace

extern "C" int ecl_mst_run_device(ecl_mst_ctx* c, const ecl_graph* g, uint8_t* d_inMST,
                                  const mst_opts* opts, void* stream, ecl_mst_stats* stats) {
  int st = run_device_once(c, g, d_inMST, opts, stream, stats);
  if (!c) return st;
  if (stats) {
    // The solve has finished: an input with more one-direction entries than
    // the half-size worklists hold is solved again with full-size ones.
    c->pending = false;
    if (st == ECL_ERR_OVERFLOW && !c->wl_full && (c->st_host->error & kErrOverflow)) {
      if ((st = grow_worklists(c))) return st;
      st = run_device_once(c, g, d_inMST, opts, stream, stats);
    }
    return st;
  }
  if (st == ECL_OK) {  // enqueued: ecl_mst_ctx_sync checks it and repeats it on overflow
    c->pending = true;
    c->pend_graph = *g;
    c->pend_out = d_inMST;
    if (opts) c->pend_opts = *opts;
    else ecl_default_opts(&c->pend_opts);
    c->pend_stream = stream ? (cudaStream_t)stream : c->stream;
  }
  return st;
}

namespace {

// Device CSR and inMST buffers for host-buffer solves, allocated on first use.
int host_buffers(ecl_mst_ctx* c, int** ni, int** nl, int** ew, unsigned char** out) {
  if (*ni) return ECL_OK;
  // one allocation, whose pointer is *ni
  auto align = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const size_t m = (size_t)std::max<int64_t>(c->max_edges, 1);
  const size_t nb = align(((size_t)c->max_nodes + 1) * 4), eb = align(m * 4);
  ECL_CUDA_TRY(cudaMalloc(ni, nb + 2 * eb + align(m)));
  *nl = reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(*ni) + nb);
  *ew = reinterpret_cast<int*>(reinterpret_cast<unsigned char*>(*nl) + eb);
  *out = reinterpret_cast<unsigned char*>(*ew) + eb;
  return ECL_OK;
}

}  // namespace

extern "C" int ecl_mst_ctx_run_host(ecl_mst_ctx* c, const ecl_graph* g, uint8_t* inMST,
                                    const mst_opts* opts, ecl_mst_stats* stats) {
  int st = check_graph_args(c, g, inMST);
  if (st) return st;
  ECL_CUDA_TRY(cudaSetDevice(c->device));
  if ((st = host_buffers(c, &c->d_nindex, &c->d_nlist, &c->d_eweight, &c->d_inMST))) return st;
  const int n = g->nodes, m = g->edges;
  ECL_CUDA_TRY(cudaMemcpyAsync(c->d_nindex, g->nindex, ((size_t)n + 1) * 4, cudaMemcpyHostToDevice, c->stream));
  if (m > 0) {
    ECL_CUDA_TRY(cudaMemcpyAsync(c->d_nlist, g->nlist, (size_t)m * 4, cudaMemcpyHostToDevice, c->stream));
    ECL_CUDA_TRY(cudaMemcpyAsync(c->d_eweight, g->eweight, (size_t)m * 4, cudaMemcpyHostToDevice, c->stream));
  }
  ecl_graph dg = {n, m, c->d_nindex, c->d_nlist, c->d_eweight};
  if ((st = ecl_mst_run_device(c, &dg, c->d_inMST, opts, c->stream, stats))) return st;
  if (m > 0)
    ECL_CUDA_TRY(cudaMemcpyAsync(inMST, c->d_inMST, (size_t)m, cudaMemcpyDeviceToHost, c->stream));
  if ((st = ecl_mst_ctx_sync(c))) return st;
  if (c->resolved && m > 0) {  // the solve was repeated after a worklist overflow
    ECL_CUDA_TRY(cudaMemcpyAsync(inMST, c->d_inMST, (size_t)m, cudaMemcpyDeviceToHost, c->stream));
    ECL_CUDA_TRY(cudaStreamSynchronize(c->stream));
  }
  if (stats) {
    int64_t fe = 0;
    uint64_t fw = 0;
    for (int j = 0; j < m; j++)
      if (inMST[j]) {
        fe++;
        fw += (uint64_t)(int64_t)g->eweight[j];
      }
    stats->forest_edges = fe;
    stats->forest_weight = fw;
  }
  return ECL_OK;
}

namespace {

__global__ void k_sticky_or(const DevState* st, unsigned* sticky) {
  const unsigned e = ld_volatile(&st->error);
  if (e) atomicOr(sticky, e);
}

// Streams, events, the second buffer set and the sticky error word of the
// pipelined solves, created on first use.
int async_setup(ecl_mst_ctx* c) {
  if (c->cin) return ECL_OK;
  int st;
  if ((st = host_buffers(c, &c->d_nindex, &c->d_nlist, &c->d_eweight, &c->d_inMST))) return st;
  c->hs[0].nindex = c->d_nindex;
  c->hs[0].nlist = c->d_nlist;
  c->hs[0].eweight = c->d_eweight;
  c->hs[0].inMST = c->d_inMST;
  if ((st = host_buffers(c, &c->hs[1].nindex, &c->hs[1].nlist, &c->hs[1].eweight, &c->hs[1].inMST))) return st;
  for (auto& h : c->hs)
    for (cudaEvent_t* e : {&h.in_done, &h.solved, &h.out_done})
      ECL_CUDA_TRY(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
  ECL_CUDA_TRY(cudaMalloc(&c->sticky, sizeof(unsigned)));
  ECL_CUDA_TRY(cudaMemset(c->sticky, 0, sizeof(unsigned)));
  ECL_CUDA_TRY(cudaStreamCreateWithFlags(&c->cout, cudaStreamNonBlocking));
  ECL_CUDA_TRY(cudaStreamCreateWithFlags(&c->cin, cudaStreamNonBlocking));
  return ECL_OK;
}

}  // namespace

extern "C" int ecl_mst_ctx_run_host_async(ecl_mst_ctx* c, const ecl_graph* g, uint8_t* inMST,
                                          const mst_opts* opts) {
  int st = check_graph_args(c, g, inMST);
  if (st) return st;
  ECL_CUDA_TRY(cudaSetDevice(c->device));
  if ((st = async_setup(c))) return st;
  auto& h = c->hs[c->async_seq++ & 1];
  const int n = g->nodes, m = g->edges;
  // copy in, once the solve that last read this set's CSR has finished
  if (h.used) ECL_CUDA_TRY(cudaStreamWaitEvent(c->cin, h.solved, 0));
  ECL_CUDA_TRY(cudaMemcpyAsync(h.nindex, g->nindex, ((size_t)n + 1) * 4, cudaMemcpyHostToDevice, c->cin));
  if (m > 0) {
    ECL_CUDA_TRY(cudaMemcpyAsync(h.nlist, g->nlist, (size_t)m * 4, cudaMemcpyHostToDevice, c->cin));
    ECL_CUDA_TRY(cudaMemcpyAsync(h.eweight, g->eweight, (size_t)m * 4, cudaMemcpyHostToDevice, c->cin));
  }
  ECL_CUDA_TRY(cudaEventRecord(h.in_done, c->cin));
  // solve on the context's stream once the inputs are in and the set's
  // previous inMST has been copied out; its device errors accumulate
  ECL_CUDA_TRY(cudaStreamWaitEvent(c->stream, h.in_done, 0));
  if (h.used) ECL_CUDA_TRY(cudaStreamWaitEvent(c->stream, h.out_done, 0));
  ecl_graph dg = {n, m, h.nindex, h.nlist, h.eweight};
  if ((st = run_device_once(c, &dg, h.inMST, opts, c->stream, nullptr))) return st;
  k_sticky_or<<<1, 1, 0, c->stream>>>(c->st, c->sticky);
  ECL_CUDA_TRY(cudaGetLastError());
  ECL_CUDA_TRY(cudaEventRecord(h.solved, c->stream));
  // copy out beside the next graph's copy in and solve
  ECL_CUDA_TRY(cudaStreamWaitEvent(c->cout, h.solved, 0));
  if (m > 0) ECL_CUDA_TRY(cudaMemcpyAsync(inMST, h.inMST, (size_t)m, cudaMemcpyDeviceToHost, c->cout));
  ECL_CUDA_TRY(cudaEventRecord(h.out_done, c->cout));
  h.used = true;
  ecl_mst_ctx::AsyncCall call;
  call.g = *g;
  call.out = inMST;
  if (opts) call.opts = *opts;
  else ecl_default_opts(&call.opts);
  c->async_calls.push_back(call);
  c->pending = false;
  return ECL_OK;
}

extern "C" int ecl_mst_ctx_wait(ecl_mst_ctx* c) {
  if (!c) return ECL_ERR_INVALID_ARG;
  ECL_CUDA_TRY(cudaSetDevice(c->device));
  if (!c->cin) return ECL_OK;
  ECL_CUDA_TRY(cudaStreamSynchronize(c->cin));
  ECL_CUDA_TRY(cudaStreamSynchronize(c->stream));
  ECL_CUDA_TRY(cudaStreamSynchronize(c->cout));
  unsigned err = 0;
  ECL_CUDA_TRY(cudaMemcpy(&err, c->sticky, sizeof(unsigned), cudaMemcpyDeviceToHost));
  ECL_CUDA_TRY(cudaMemset(c->sticky, 0, sizeof(unsigned)));
  std::vector<ecl_mst_ctx::AsyncCall> calls;
  calls.swap(c->async_calls);
  if ((err & kErrOverflow) && !c->wl_full) {
    // an input had more one-direction entries than half its CSR entries:
    // grow the worklists and solve the calls since the last wait again
    int st = grow_worklists(c);
    if (st) return st;
    for (auto& call : calls)
      if ((st = ecl_mst_ctx_run_host(c, &call.g, call.out, &call.opts, nullptr))) return st;
    return ECL_OK;
  }
  return device_error_status(err);
}

extern "C" int ecl_mst_run(const ecl_graph* g, uint8_t* inMST, const mst_opts* opts,
                           ecl_mst_stats* stats) {
  if (!g || !inMST || g->nodes < 1 || g->edges < 0) return ECL_ERR_INVALID_ARG;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return ECL_ERR_NO_DEVICE;
  ecl_mst_ctx* c = nullptr;
  int st = ecl_mst_ctx_create(dev, g->nodes, g->edges, &c);
  if (st) return st;
  st = ecl_mst_ctx_run_host(c, g, inMST, opts, stats);
  ecl_mst_ctx_destroy(c);
  return st;
}

extern "C" int ecl_host_alloc_pinned(size_t bytes, void** out) {
  if (!out) return ECL_ERR_INVALID_ARG;
  *out = nullptr;
  ECL_CUDA_TRY(cudaHostAlloc(out, bytes ? bytes : 1, cudaHostAllocDefault));
  return ECL_OK;
}

extern "C" void ecl_host_free_pinned(void* p) {
  if (p) cudaFreeHost(p);
}

// ===================================================== allocation-free solve
// Some callers cannot allocate device memory: code that runs inside a host
// allocator hook or a memory-pool callback, an embedding that owns every
// allocation of the process, or a service whose device memory budget is
// fixed at start-up. ecl_mst_run_device_noalloc serves them: its scratch
// (min slots, parent array, worklists, control block) is one file-scope
// device array, created when the module loads and kept until the process
// exits, on every GPU that loads this library. The caller passes only the
// device CSR and the device inMST output.
#include <mutex>

namespace {

constexpr int64_t kNaMaxNodes = 1 << 18;              // 262,144 vertices
constexpr int64_t kNaMaxEdges = 1 << 20;              // 1,048,576 directed CSR entries
constexpr int64_t kNaWlCap = kNaMaxEdges / 2;         // one-direction entries per worklist
constexpr int64_t kNaTiles = kNaMaxEdges / kGran + 2;  // task -> row table entries

constexpr size_t na_align(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kNaOffState = 0;
constexpr size_t kNaOffMinv0 = na_align(kNaOffState + sizeof(DevState));
constexpr size_t kNaOffMinv1 = na_align(kNaOffMinv0 + sizeof(u64) * kNaMaxNodes);
constexpr size_t kNaOffParent = na_align(kNaOffMinv1 + sizeof(u64) * kNaMaxNodes);
constexpr size_t kNaOffFirstV = na_align(kNaOffParent + sizeof(int) * kNaMaxNodes);
constexpr size_t kNaOffBits = na_align(kNaOffFirstV + sizeof(int) * kNaTiles);
constexpr size_t kNaOffWl0 = na_align(kNaOffBits + tree_bits_bytes(kNaMaxNodes));
constexpr size_t kNaOffWl1 = na_align(kNaOffWl0 + sizeof(int4) * kNaWlCap);
constexpr size_t kNaBytes = na_align(kNaOffWl1 + sizeof(int4) * kNaWlCap);  // about 21 MB

// The scratch itself. In host code this name is only a stand-in for the
// symbol, never a device address: the address comes from
// cudaGetSymbolAddress, once per device.
static __device__ __align__(256) unsigned char g_na_scratch[kNaBytes];

struct NaDevice {
  bool ready = false;
  unsigned char* base = nullptr;  // device address of g_na_scratch on this device
  int sm_count = 0;
  int round_grid = 0, abl_grid = 0, group_grid = 0;
};
constexpr int kNaMaxDevices = 64;
NaDevice g_na_dev[kNaMaxDevices];
std::mutex g_na_mu;

// Once per device, with that device current: resolve the scratch address and
// the cooperative grid size. No allocation happens here.
int na_setup(int dev, NaDevice** out) {
  if (dev < 0 || dev >= kNaMaxDevices) return ECL_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(g_na_mu);
  NaDevice& d = g_na_dev[dev];
  // The scratch array's address is looked up on every call: a device reset
  // reloads the module, and the array then lives elsewhere.
  void* p = nullptr;
  ECL_CUDA_TRY(cudaGetSymbolAddress(&p, g_na_scratch));
  d.base = (unsigned char*)p;
  if (!d.ready) {
    int coop = 0;
    ECL_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    if (!coop) return ECL_ERR_UNSUPPORTED;
    ECL_CUDA_TRY(cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev));
    d.round_grid = std::min(coop_grid((const void*)k_round, kBorThreads, d.sm_count), kMaxRoundCtas);
    d.abl_grid = std::min(coop_grid((const void*)k_rounds, kRoundThreads, d.sm_count), kMaxRoundCtas);
    d.group_grid = coop_grid((const void*)k_group, kGroupThreads, d.sm_count);
    int ps = prepare_scan_kernels();
    if (ps || (ps = prepare_round_kernels()) || (ps = prepare_cluster_kernels())) return ps;
    if (d.round_grid <= 0 || d.abl_grid <= 0 || d.group_grid <= 0) return ECL_ERR_CUDA;
    d.ready = true;
  }
  *out = &d;
  return ECL_OK;
}

}  // namespace

extern "C" int ecl_mst_run_device_noalloc(const ecl_graph* g, uint8_t* d_inMST,
                                          const mst_opts* opts, void* stream) {
  if (!g || !d_inMST || g->nodes < 1 || g->edges < 0) return ECL_ERR_INVALID_ARG;
  if (g->nodes > kNaMaxNodes || g->edges > kNaMaxEdges) return ECL_ERR_TOO_LARGE;
  if (!g->nindex || (g->edges > 0 && (!g->nlist || !g->eweight))) return ECL_ERR_INVALID_ARG;
  mst_opts o;
  if (opts) o = *opts;
  else ecl_default_opts(&o);
  int st = check_opts(&o);
  if (st) return st;
  // The learned schedule's feature pass needs scratch this entry point does
  // not hold; it takes the reference heuristic, as ecl_mst_run_device does
  // below its learned-schedule cut-off.
  if (o.threshold_mode == ECL_THRESH_LEARNED) o.threshold_mode = ECL_THRESH_HEURISTIC;
  if (o.flags & kDeoptFlags) return ECL_ERR_UNSUPPORTED;  // single-graph contexts only
  if (g->edges == 0) return ECL_OK;
  int dev = 0;
  ECL_CUDA_TRY(cudaGetDevice(&dev));
  NaDevice* d = nullptr;
  if ((st = na_setup(dev, &d))) return st;
  cudaStream_t s = (cudaStream_t)stream;
  const int n = g->nodes, m = g->edges;
  DevState* dst = (DevState*)(d->base + kNaOffState);
  int* parent = (int*)(d->base + kNaOffParent);
  u64* minv0 = (u64*)(d->base + kNaOffMinv0);
  u64* minv1 = (u64*)(d->base + kNaOffMinv1);
  int* first_v = (int*)(d->base + kNaOffFirstV);
  int4* wl0 = (int4*)(d->base + kNaOffWl0);
  int4* wl1 = (int4*)(d->base + kNaOffWl1);
  // The array keeps the previous call's contents: the control block (error
  // word, worklist counters, barrier) must start at zero (k_cluster clears it
  // itself); the kernels initialise parent[] and the min arrays.
  const int ctas = round_ablation(o.flags) || (o.flags & ECL_FLAG_NO_SMALL_TAIL)
                       ? 0 : cluster_ctas(n, m, (unsigned)kNaWlCap);
  if (!ctas) ECL_CUDA_TRY(cudaMemsetAsync(dst, 0, sizeof(DevState), s));
  auto finish = [&]() -> int {
    // Report device-side errors (malformed CSR, worklist overflow) to the caller.
    unsigned err = 0;
    ECL_CUDA_TRY(cudaMemcpyAsync(&err, &dst->error, sizeof(err), cudaMemcpyDeviceToHost, s));
    ECL_CUDA_TRY(cudaStreamSynchronize(s));
    return device_error_status(err);
  };
  if (ctas) {
    ClArgs ca{};
    ca.nodes = n;
    ca.edges = m;
    ca.nindex = g->nindex;
    ca.nlist = g->nlist;
    ca.eweight = g->eweight;
    ca.inMST = d_inMST;
    ca.wl0 = wl0;
    ca.wl1 = wl1;
    ca.parent = parent;
    ca.minv = minv0;
    ca.st = dst;
    if ((st = enqueue_cluster(ca, ctas, &o, s))) return st;
    return finish();
  }
  if (!round_ablation(o.flags)) {
    GroupArgs ga{};
    ga.nodes = n;
    ga.edges = m;
    ga.nindex = g->nindex;
    ga.nlist = g->nlist;
    ga.eweight = g->eweight;
    ga.inMST = d_inMST;
    ga.parent = parent;
    ga.minv = minv0;
    ga.roots0 = reinterpret_cast<int*>(minv1);
    ga.roots1 = ga.roots0 + n;
    ga.wl0 = wl0;
    ga.wl1 = wl1;
    ga.wl_cap = (unsigned)kNaWlCap;
    ga.st = dst;
    // within the stated limit a scan keeps at most m / 2 entries
    o.ctas_per_sm = 0;
    const unsigned slack = (unsigned)std::max<int64_t>(0, kNaWlCap - m / 2);
    if ((st = enqueue_group(ga, &o, slack, d->sm_count, d->group_grid, s, nullptr))) return st;
    return finish();
  }
  const int split = o.degree_split > 0 ? o.degree_split : kDefaultSplit;
  const int tiles = (int)(((int64_t)m + kGran - 1) / kGran);
  PrepArgs pa{};
  pa.nodes = n;
  pa.edges = m;
  pa.nindex = g->nindex;
  pa.eweight = g->eweight;
  pa.parent = parent;
  pa.minv0 = minv0;
  pa.minv1 = minv1;
  pa.first_v = first_v;
  pa.tiles = tiles;
  pa.mode = o.threshold_mode;
  pa.explicit_thr = o.threshold;
  pa.split = split;
  pa.quantile = o.quantile;
  pa.both_slots = round_ablation(o.flags) != 0;
  pa.st = dst;
  if ((st = enqueue_prep(pa, d->sm_count, s))) return st;
  ScanArgs sa{};
  sa.nodes = n;
  sa.edges = m;
  sa.nindex = g->nindex;
  sa.nlist = g->nlist;
  sa.eweight = g->eweight;
  sa.first_v = first_v;
  sa.tiles = tiles;
  sa.parent = parent;
  sa.wl0 = wl0;
  sa.wl1 = wl1;
  sa.wl_cap = (unsigned)kNaWlCap;
  sa.tree_bits = (const unsigned*)(d->base + kNaOffBits);
  // within the stated limit a scan keeps at most m / 2 entries
  const unsigned wl_slack = (unsigned)std::max<int64_t>(0, kNaWlCap - m / 2);
  sa.inMST = d_inMST;
  sa.zero_vec = (((uintptr_t)d_inMST) & 15) == 0;
  sa.st = dst;
  RoundArgs ra{};
  ra.nodes = n;
  ra.wl0 = wl0;
  ra.wl1 = wl1;
  ra.wl_cap = (unsigned)kNaWlCap;
  ra.parent = parent;
  ra.minv0 = minv0;
  ra.minv1 = minv1;
  ra.inMST = d_inMST;
  ra.st = dst;
  ra.small_tail = o.small_tail < 0 ? 0u : (o.small_tail == 0 ? kDefaultSmallTail : (unsigned)o.small_tail);
  if (o.flags & ECL_FLAG_NO_SMALL_TAIL) ra.small_tail = 0;
  ra.count_atomics = (o.flags & ECL_FLAG_STATS) ? 1 : 0;
  ra.abl = round_ablation(o.flags);
  ra.min_tiles = kDefaultMinTiles;
  if ((st = launch_scan(kLight, sa, d->sm_count, wl_slack, s))) return st;
  ra.phase = 0;
  if ((st = enqueue_rounds(ra, kListLight0, m, d->sm_count, 0, d->round_grid, d->abl_grid, s, nullptr))) return st;
  if ((st = launch_flatten(kListHeavy, parent, n, dst, (unsigned*)sa.tree_bits, d->sm_count, s))) return st;
  if ((st = launch_scan(kHeavy, sa, d->sm_count, wl_slack, s))) return st;
  ra.phase = 1;
  if ((st = enqueue_rounds(ra, kListHeavy, m, d->sm_count, 0, d->round_grid, d->abl_grid, s, nullptr))) return st;
  return finish();
}

// ============================================================== batched mode
namespace {

__global__ void k_or_error(const DevState* src, DevState* dst) {
  const unsigned e = ld_volatile(&src->error);
  if (e) atomicOr(&dst->error, e);
}

constexpr int kBatchDefaultCap = 1 << 19;
constexpr int kMaxLargeStreams = 8;      // concurrent streams for a batch's large graphs
// Graphs of up to kTeamEdges entries are solved by teams (k_batch_group) where
// at least kTeamMin of a batch's large graphs are that small, or half as many
// and no others; the rest by the engines, K streams side by side. 39 large
// graphs (17 by teams) 8.45 -> 7.95 ms on 8 streams, 33 (18) 6.36 -> 5.59, 55
// (53) 5.57 -> 3.62, 5 (5) 1.07 -> 0.97. Two graphs alone are the faster on the
// engines (0.22 ms against 0.27), and three by teams before five others only
// delay those (2.05 -> 2.15). With kTeamEdges 2^22 the largest graph of a team
// takes as long as on the whole chip alone (8.44 ms, 5.65, 3.54). Teams of fewer
// than kTeamMinCtas CTAs gain nothing, and on one stream a graph has the chip
// to itself as it is.
constexpr int kTeamEdges = 1 << 21;
constexpr int kTeamMin = 8;
constexpr int kTeamMinCtas = 6;
constexpr int64_t kTeamGraphCost = 1 << 18;  // of the rounds' latency, in entries
constexpr int kDefaultLargeStreams = 4;  // measured: 957 large graphs of the mixed batch 1.5x faster than on one

}  // namespace

// Size classes of a batch's small graphs (batch_small) and the CTAs of their
// clusters. The last one keeps parent[] and the slots in shared memory.
constexpr int kBatchClasses = 5;
constexpr int kClassCtas[kBatchClasses] = {8, 4, 2, 1, 1};

struct ecl_batch_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  int sm_count = 0;
  int max_graphs = 0;
  int64_t max_nodes = 0, max_edges = 0;
  int cap = 0;        // per-CTA scratch: vertices and CSR entries
  // scratch for small_grid graphs of `cap` vertices and entries; a run divides
  // it among the clusters of its size classes (at most sm_count / size each,
  // state_count in all)
  int small_grid = 0, state_count = 0;
  int* parent_pool = nullptr;
  u64* minv_pool = nullptr;
  int4* wl_pool = nullptr;
  DevState* states = nullptr;   // a control block per cluster
  GraphDesc* d_graphs = nullptr;
  unsigned* d_queue = nullptr;  // one per size class
  cudaStream_t cls_stream[kBatchClasses - 1] = {};  // the classes beside the first
  cudaEvent_t cls_fork = nullptr, cls_join[kBatchClasses - 1] = {};
  DevState* st = nullptr;
  // grid-wide engines for the graphs beyond the cutoff, one per concurrent
  // stream: [0] is made with the context, the others when a solve asks for
  // more streams (opts batch_large_streams)
  ecl_mst_ctx* big[kMaxLargeStreams] = {};
  cudaEvent_t large_fork = nullptr, large_join[kMaxLargeStreams] = {};
  // the graphs that teams of CTAs solve (k_batch_group): descriptors, degree
  // statistics and learned schedules by graph, barriers and control blocks by team
  GraphDesc* d_team_graphs = nullptr;
  FeatAcc* d_team_feat = nullptr;
  LearnedChoice* d_team_choice = nullptr;
  TeamWords* d_team_words = nullptr;
  DevState* d_team_states = nullptr;
  int team_grid = 0;
  cudaEvent_t ev[3] = {};
  // the large-graph launch sequence captured as a CUDA graph, keyed by the batch
  cudaGraphExec_t exec = nullptr;
  std::vector<long long> exec_key;
};

// Grid-wide engine k of a batch context, sized for its largest graph. The
// batch's solves are captured and replayed without a host check in between,
// so its lists hold every entry of any input.
static int batch_big_ctx(ecl_batch_ctx* c, int k) {
  if (c->big[k]) return ECL_OK;
  return ctx_create(c->device, c->max_nodes, std::max<int64_t>(c->max_edges, 1), true, &c->big[k]);
}

extern "C" void ecl_batch_ctx_destroy(ecl_batch_ctx* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  if (c->exec) cudaGraphExecDestroy(c->exec);
  cudaFree(c->parent_pool);
  cudaFree(c->minv_pool);
  cudaFree(c->wl_pool);
  for (cudaStream_t q : c->cls_stream)
    if (q) cudaStreamDestroy(q);
  for (cudaEvent_t e : c->cls_join)
    if (e) cudaEventDestroy(e);
  if (c->cls_fork) cudaEventDestroy(c->cls_fork);
  cudaFree(c->states);
  cudaFree(c->d_graphs);
  cudaFree(c->d_queue);
  cudaFree(c->d_team_graphs);
  cudaFree(c->d_team_feat);
  cudaFree(c->d_team_choice);
  cudaFree(c->d_team_words);
  cudaFree(c->d_team_states);
  cudaFree(c->st);
  for (auto& e : c->ev)
    if (e) cudaEventDestroy(e);
  if (c->large_fork) cudaEventDestroy(c->large_fork);
  for (auto& e : c->large_join)
    if (e) cudaEventDestroy(e);
  for (ecl_mst_ctx* b : c->big) ecl_mst_ctx_destroy(b);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

extern "C" int ecl_batch_ctx_create(int device, int32_t max_graphs, int64_t max_graph_nodes,
                                    int64_t max_graph_edges, int32_t small_cap, ecl_batch_ctx** out) {
  if (!out || max_graphs < 1 || max_graph_nodes < 1 || max_graph_edges < 0 || small_cap < 0)
    return ECL_ERR_INVALID_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return ECL_ERR_NO_DEVICE;
  if (device < 0 || device >= ndev) return ECL_ERR_INVALID_ARG;
  ECL_CUDA_TRY(cudaSetDevice(device));
  ecl_batch_ctx* c = new (std::nothrow) ecl_batch_ctx();
  if (!c) return ECL_ERR_ALLOC;
  c->device = device;
  c->max_graphs = max_graphs;
  c->max_nodes = max_graph_nodes;
  c->max_edges = max_graph_edges;
  c->cap = small_cap > 0 ? small_cap : kBatchDefaultCap;
  int st;
  auto fail = [&](int s) {
    ecl_batch_ctx_destroy(c);
    return s;
  };
  if ((st = cuda_status(cudaDeviceGetAttribute(&c->sm_count, cudaDevAttrMultiProcessorCount, device))))
    return fail(st);
  if ((st = cuda_status(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking)))) return fail(st);
  c->small_grid = 2 * c->sm_count;
  for (int size : kClassCtas) c->state_count += std::max(1, c->sm_count / size);
  if ((st = prepare_cluster_kernels())) return fail(st);
  const size_t ctas = (size_t)c->small_grid, cap = (size_t)c->cap;
  if ((st = cuda_status(cudaMalloc(&c->parent_pool, ctas * cap * sizeof(int))))) return fail(st);
  if ((st = cuda_status(cudaMalloc(&c->minv_pool, ctas * cap * sizeof(u64))))) return fail(st);
  if ((st = cuda_status(cudaMalloc(&c->wl_pool, ctas * 2 * cap * sizeof(int4))))) return fail(st);
  if ((st = cuda_status(cudaMalloc(&c->states, (size_t)c->state_count * sizeof(DevState))))) return fail(st);
  if ((st = cuda_status(cudaMalloc(&c->d_graphs, (size_t)max_graphs * sizeof(GraphDesc))))) return fail(st);
  if ((st = cuda_status(cudaMalloc(&c->d_queue, kBatchClasses * sizeof(unsigned))))) return fail(st);
  for (auto& q : c->cls_stream)
    if ((st = cuda_status(cudaStreamCreateWithFlags(&q, cudaStreamNonBlocking)))) return fail(st);
  if ((st = cuda_status(cudaEventCreateWithFlags(&c->cls_fork, cudaEventDisableTiming)))) return fail(st);
  for (auto& e : c->cls_join)
    if ((st = cuda_status(cudaEventCreateWithFlags(&e, cudaEventDisableTiming)))) return fail(st);
  if ((st = cuda_status(cudaMalloc(&c->st, sizeof(DevState))))) return fail(st);
  for (auto& e : c->ev)
    if ((st = cuda_status(cudaEventCreate(&e)))) return fail(st);
  if ((st = cuda_status(cudaEventCreateWithFlags(&c->large_fork, cudaEventDisableTiming)))) return fail(st);
  for (auto& e : c->large_join)
    if ((st = cuda_status(cudaEventCreateWithFlags(&e, cudaEventDisableTiming)))) return fail(st);
  if (max_graph_edges > c->cap || max_graph_nodes > c->cap) {
    if ((st = batch_big_ctx(c, 0))) return fail(st);
    if ((st = cuda_status(cudaMalloc(&c->d_team_graphs, (size_t)max_graphs * sizeof(GraphDesc))))) return fail(st);
    if ((st = cuda_status(cudaMalloc(&c->d_team_feat, (size_t)max_graphs * sizeof(FeatAcc))))) return fail(st);
    if ((st = cuda_status(cudaMalloc(&c->d_team_choice, (size_t)max_graphs * sizeof(LearnedChoice))))) return fail(st);
    if ((st = cuda_status(cudaMalloc(&c->d_team_words, kMaxTeams * sizeof(TeamWords))))) return fail(st);
    if ((st = cuda_status(cudaMalloc(&c->d_team_states, kMaxTeams * sizeof(DevState))))) return fail(st);
    if ((st = ecl_learned_batch_prepare())) return fail(st);
    c->team_grid = coop_grid((const void*)k_batch_group, kGroupThreads, c->sm_count);
    if (c->team_grid <= 0) return fail(ECL_ERR_CUDA);
  }
  *out = c;
  return ECL_OK;
}

namespace {

// The graphs solved by clusters. A graph's cluster has two CTAs or more if one
// cannot hold its vertices (kClVertices), and as many as its share of the
// batch's work asks for (entries, or vertices where these are more), so that no
// graph is worked on much longer than an even split of the batch over the chip
// takes (twice that share, rounded up to 1, 2, 4 or 8): a batch of thousands
// runs one CTA to a graph, a few graphs run on as much of the chip as they can
// use. Sparse graphs that one CTA cannot hold run on one all the same: latency
// is what they cost, and twice as many side by side hide it (400 of 17 000
// vertices and 1000 edges 0.12 ms against 0.25 on two CTAs each; for graphs of
// more entries than vertices the rule loses where a batch has few of them, 398 of
// 1000 to 60 000 vertices 2.16 ms against 2.11). Largest first within a class; the
// classes run side by side, the largest clusters launched first. Those 398
// graphs took 7.1 ms with one CTA to every graph.
int batch_small(ecl_batch_ctx* c, const ecl_batch* b, const std::vector<int>& small, uint8_t* d_inMST,
                const mst_opts* o, cudaStream_t s) {
  const int S = (int)small.size();
  auto fits = [&](int g) { return b->nodes[g] <= kClVertices; };
  auto work = [&](int g) { return (int64_t)(fits(g) ? b->edges[g] : std::max(b->edges[g], b->nodes[g])); };
  int64_t total = 0;
  for (int g : small) total += work(g);
  const int64_t share = std::max<int64_t>(kClTile, total / (2 * c->sm_count));
  auto class_of = [&](int g) {
    if (fits(g) && work(g) <= share) return kBatchClasses - 1;
    int k = !fits(g) && b->edges[g] < b->nodes[g] ? 3 : 2;
    while (k > 0 && work(g) > kClassCtas[k] * share) k--;
    return k;
  };
  std::vector<int> order(small);
  std::vector<int> cls(b->num_graphs);
  for (int g : small) cls[g] = class_of(g);
  std::sort(order.begin(), order.end(), [&](int x, int y) {
    return cls[x] != cls[y] ? cls[x] < cls[y] : b->edges[x] > b->edges[y];
  });
  std::vector<GraphDesc> descs(S);
  int first[kBatchClasses + 1] = {};
  for (int i = 0; i < S; i++) {
    const int g = order[i];
    descs[i] = GraphDesc{b->nindex_off[g], b->edge_off[g], b->nodes[g], b->edges[g]};
    for (int k = cls[g] + 1; k <= kBatchClasses; k++) first[k] = i + 1;
  }
  ECL_CUDA_TRY(cudaMemsetAsync(c->d_queue, 0, kBatchClasses * sizeof(unsigned), s));
  ECL_CUDA_TRY(cudaMemcpyAsync(c->d_graphs, descs.data(), (size_t)S * sizeof(GraphDesc), cudaMemcpyHostToDevice, s));
  BatchArgs ba{};
  ba.nindex = b->nindex;
  ba.nlist = b->nlist;
  ba.eweight = b->eweight;
  ba.inMST = d_inMST;
  ba.st = c->st;
  ba.mode = o->threshold_mode == ECL_THRESH_LEARNED ? ECL_THRESH_HEURISTIC : o->threshold_mode;
  ba.explicit_thr = o->threshold;
  ba.quantile = o->quantile;
  ba.count_atomics = (o->flags & ECL_FLAG_STATS) ? 1 : 0;
  // clusters of every class and the graph size their scratch is for; all of a
  // class at once if the pool has room, else its part of the pool
  int64_t cap[kBatchClasses], want[kBatchClasses], needed = 0, least = 0;
  for (int k = 0; k < kBatchClasses; k++) {
    cap[k] = 0;
    for (int i = first[k]; i < first[k + 1]; i++) cap[k] = std::max<int64_t>(cap[k], std::max(descs[i].nodes, descs[i].edges));
    cap[k] = (cap[k] + 3) & ~(int64_t)3;
    want[k] = std::min(first[k + 1] - first[k], std::max(1, c->sm_count / kClassCtas[k]));
    needed += want[k] * cap[k];
    least += cap[k];
  }
  const int64_t pool = (int64_t)c->small_grid * c->cap;
  int64_t used = 0;  // pool entries given out
  int states = 0, forked = 0;
  ECL_CUDA_TRY(cudaEventRecord(c->cls_fork, s));
  for (int k = 0; k < kBatchClasses; k++) {
    const int count = first[k + 1] - first[k], size = kClassCtas[k];
    if (count <= 0) continue;
    // (more than the pool: the parts add up to pool - least, one cluster each to least)
    const int clusters = (int)(needed <= pool ? want[k] : std::max<int64_t>(1, want[k] * (pool - least) / needed));
    ba.graphs = c->d_graphs + first[k];
    ba.count = count;
    ba.queue = c->d_queue + k;
    ba.states = c->states + states;
    ba.parent_pool = c->parent_pool + used;
    ba.minv_pool = c->minv_pool + used;
    ba.wl_pool = c->wl_pool + 2 * used;
    ba.cap = cap[k];
    used += clusters * cap[k];
    states += clusters;
    cudaStream_t q = s;
    if (first[k + 1] < S) {  // the last class runs on the caller's stream
      q = c->cls_stream[forked];
      ECL_CUDA_TRY(cudaStreamWaitEvent(q, c->cls_fork, 0));
    }
    const int st = k == kBatchClasses - 1 ? launch_cluster(k_batch_cluster<true>, 1, clusters, kClThreads, kClSmem, q, ba)
                             : launch_cluster(k_batch_cluster<false>, size, clusters, kClThreads, 0, q, ba);
    if (st) return st;
    if (q != s) ECL_CUDA_TRY(cudaEventRecord(c->cls_join[forked++], q));
  }
  for (int i = 0; i < forked; i++) ECL_CUDA_TRY(cudaStreamWaitEvent(s, c->cls_join[i], 0));
  return ECL_OK;
}

// Which graphs a batch's teams solve, on what scratch and how many CTAs.
struct TeamPlan {
  std::vector<GraphDesc> descs;  // by team
  Team team[kMaxTeams + 1];
  int teams = 0, ctas = 0;
};

// `graphs` (largest first) on as many teams as the scratch of `engines` engines
// has room for: every graph goes to the team with the least work so far, a
// team's share of the CTAs is its share of the work, and a graph's work is its
// entries and kTeamGraphCost for the rounds' latency.
TeamPlan plan_teams(ecl_batch_ctx* c, const ecl_batch* b, const std::vector<int>& graphs, int engines, int max_ctas) {
  TeamPlan plan;
  const int total_ctas = c->team_grid;
  int T = (int)std::min<size_t>(graphs.size(), (size_t)std::min(kMaxTeams, total_ctas / kTeamMinCtas));
  auto cap_of = [&](int g) { return b->edges[g] + std::min<int64_t>(b->edges[g], kWlSlack) / 4; };
  for (;; T--) {  // (one team always fits)
    // no more teams than lists fit: team t's first graph, its largest, is graph t
    int64_t room = 0;
    for (int t = 0; t < T; t++) room += cap_of(graphs[t]);
    if (T > 1 && room > engines * (int64_t)c->big[0]->wl_cap) continue;
    std::vector<std::vector<int>> lists(T);
    std::vector<int64_t> work(T, 0);
    std::vector<int> nmax(T, 0);
    for (int g : graphs) {
      const int t = (int)(std::min_element(work.begin(), work.end()) - work.begin());
      lists[t].push_back(g);
      work[t] += b->edges[g] + kTeamGraphCost;
      nmax[t] = std::max(nmax[t], b->nodes[g]);
    }
    // the teams' scratch, first fit
    std::vector<int64_t> slots_used(engines, 0), wl_used(engines, 0);
    bool fits = true;
    for (int t = 0; t < T && fits; t++) {
      const int64_t n = nmax[t], cap = cap_of(lists[t][0]);
      int k = 0;
      while (k < engines && (slots_used[k] + n > c->max_nodes || wl_used[k] + cap > c->big[k]->wl_cap)) k++;
      if (!(fits = k < engines)) break;
      Team& tm = plan.team[t];  // 20 bytes of slots a vertex, from an 8-byte boundary
      tm.slots = reinterpret_cast<u64*>(static_cast<char*>(c->big[k]->slots) + 20 * slots_used[k]);
      tm.wl0 = c->big[k]->wl[0] + wl_used[k];
      tm.wl1 = c->big[k]->wl[1] + wl_used[k];
      tm.wl_cap = (unsigned)cap;
      slots_used[k] += (n + 1) & ~1;
      wl_used[k] += cap;
    }
    if (!fits) continue;
    int64_t total = 0;
    for (int64_t w : work) total += w;
    std::vector<int> ctas(T);
    int used = 0;
    for (int t = 0; t < T; t++) {
      ctas[t] = std::max(1, std::min(max_ctas, (int)((total_ctas - T) * work[t] / total)));
      used += ctas[t];
    }
    for (; used < total_ctas; used++) {  // the rest one by one to the team with the most work per CTA
      int best = -1;
      for (int t = 0; t < T; t++)
        if (ctas[t] < max_ctas && (best < 0 || work[t] * ctas[best] > work[best] * ctas[t])) best = t;
      if (best < 0) break;
      ctas[best]++;
    }
    for (int t = 0; t < T; t++) {
      plan.team[t].first_graph = (int)plan.descs.size();
      plan.team[t].first_cta = plan.ctas;
      plan.ctas += ctas[t];
      for (int g : lists[t]) plan.descs.push_back(GraphDesc{b->nindex_off[g], b->edge_off[g], b->nodes[g], b->edges[g]});
    }
    plan.team[T] = Team{};
    plan.team[T].first_graph = (int)plan.descs.size();
    plan.team[T].first_cta = plan.ctas;
    plan.teams = T;
    return plan;
  }
}

// The plan's graphs, whose descriptors are in c->d_team_graphs.
int batch_teams(ecl_batch_ctx* c, const ecl_batch* b, const TeamPlan& plan, bool learned, uint8_t* d_inMST,
                const mst_opts* o, cudaStream_t s) {
  TeamArgs ta{};
  ta.graphs = c->d_team_graphs;
  ta.choice = c->d_team_choice;
  ta.teams = plan.teams;
  for (int t = 0; t <= plan.teams; t++) ta.team[t] = plan.team[t];
  ta.learned_min = kLearnedMinEdges;
  ta.words = c->d_team_words;
  ta.states = c->d_team_states;
  ta.nindex = b->nindex;
  ta.nlist = b->nlist;
  ta.eweight = b->eweight;
  ta.inMST = d_inMST;
  ta.st = c->st;
  ta.mode = o->threshold_mode;
  ta.explicit_thr = o->threshold;
  ta.split = o->degree_split > 0 ? o->degree_split : kDefaultSplit;
  ta.quantile = o->quantile;
  ta.solo = o->small_tail < 0 ? 0u : (o->small_tail == 0 ? kDefaultSmallTail : (unsigned)o->small_tail);
  if (o->flags & ECL_FLAG_NO_SMALL_TAIL) ta.solo = 0;
  ta.min_tiles = o->round_min_tiles < 0 ? 0 : (o->round_min_tiles == 0 ? kDefaultMinTiles : o->round_min_tiles);
  ta.count_atomics = (o->flags & ECL_FLAG_STATS) ? 1 : 0;
  ECL_CUDA_TRY(cudaMemsetAsync(c->d_team_words, 0, kMaxTeams * sizeof(TeamWords), s));
  ECL_CUDA_TRY(cudaMemsetAsync(c->d_team_states, 0, kMaxTeams * sizeof(DevState), s));
  if (learned) {
    const int r = ecl_learned_batch(c->big[0], c->d_team_graphs, (int)plan.descs.size(), kLearnedMinEdges, b->nindex,
                                    b->eweight, c->d_team_feat, c->d_team_choice, s);
    if (r) return r;
  }
  return launch_ex(k_batch_group, plan.ctas, kGroupThreads, 0, s, true, nullptr, ta);
}

int batch_enqueue(ecl_batch_ctx* c, const ecl_batch* b, uint8_t* d_inMST, const mst_opts* o,
                  cudaStream_t s, bool timed, ecl_batch_stats* stats) {
  const int G = b->num_graphs;
  const int cutoff = std::min(o->batch_small_edges > 0 ? o->batch_small_edges : c->cap, c->cap);
  std::vector<int> small, large;
  int64_t edges_total = 0;
  for (int g = 0; g < G; g++) {
    const int n = b->nodes[g], m = b->edges[g];
    if (n < 1 || m < 0) return ECL_ERR_INVALID_ARG;
    if (n > c->max_nodes || m > c->max_edges) return ECL_ERR_TOO_LARGE;
    edges_total += m;
    if (m <= cutoff && n <= c->cap) small.push_back(g);
    else large.push_back(g);
  }
  if (!large.empty() && !c->big[0]) return ECL_ERR_TOO_LARGE;
  const int S = (int)small.size();
  ECL_CUDA_TRY(cudaMemsetAsync(c->st, 0, sizeof(DevState), s));
  if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[0], s));
  if (S > 0) {
    const int r = batch_small(c, b, small, d_inMST, o, s);
    if (r) return r;
  }
  if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[1], s));
  bool replayed = false;
  if (!large.empty()) {
    // The large graphs' launch sequence (no host round trip) is captured once
    // per batch layout as a CUDA graph and replayed; if capture is unavailable
    // it is enqueued.
    std::vector<long long> key;
    key.push_back((long long)(uintptr_t)b->nindex);
    key.push_back((long long)(uintptr_t)b->nlist);
    key.push_back((long long)(uintptr_t)b->eweight);
    key.push_back((long long)(uintptr_t)d_inMST);
    key.push_back(o->threshold_mode);
    key.push_back(o->threshold);
    key.push_back((long long)(o->quantile * 1e6f));
    key.push_back(o->degree_split);
    key.push_back(o->small_tail);
    key.push_back(o->flags);
    key.push_back(o->round_min_tiles);
    key.push_back(o->ctas_per_sm);
    key.push_back(o->batch_large_streams);
    key.push_back((long long)ecl_learned_weights_version());
    for (int g : large) {
      key.push_back(g);
      key.push_back(b->nindex_off[g]);
      key.push_back(b->edge_off[g]);
      key.push_back(b->nodes[g]);
      key.push_back(b->edges[g]);
    }
    // The learned schedule runs for the large graphs it serves (as the
    // single-graph solve: at least kLearnedMinEdges entries, weights loaded),
    // its feature pass on the engine's side stream beside k_prep; the others
    // take the reference heuristic.
    mst_opts lo = *o;
    const bool learned = lo.threshold_mode == ECL_THRESH_LEARNED && ecl_learned_has_weights();
    if (lo.threshold_mode == ECL_THRESH_LEARNED && !learned) lo.threshold_mode = ECL_THRESH_HEURISTIC;
    // K concurrent streams, each with its own engine; the graphs go largest
    // first, each to the stream with the fewest entries so far. With several
    // streams the round kernels take one CTA per SM unless ctas_per_sm says
    // otherwise, so the streams' rounds run side by side.
    int K = std::max(1, std::min((int)large.size(), o->batch_large_streams > 0
                                                       ? std::min(o->batch_large_streams, kMaxLargeStreams)
                                                       : kDefaultLargeStreams));
    for (int k = 0; k < K; k++) {
      int r = batch_big_ctx(c, k);
      if (r == ECL_ERR_ALLOC && k > 0) {  // no room for another engine: fewer streams
        cudaGetLastError();
        K = k;
        break;
      }
      if (!r && learned) r = ecl_learned_upload(c->big[k], s);  // before any capture
      if (r) return r;
    }
    if (K > 1 && lo.ctas_per_sm == 0) lo.ctas_per_sm = 1;
    key.push_back(K);  // the streams in use (fewer than asked when memory ran short)
    std::vector<int> order(large), team;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return b->edges[x] > b->edges[y]; });
    if (K > 1 && !round_ablation(lo.flags)) {
      const auto rest = std::find_if(order.begin(), order.end(), [&](int g) { return b->edges[g] <= kTeamEdges; });
      if (order.end() - rest >= (rest == order.begin() ? kTeamMin / 2 : kTeamMin)) {
        team.assign(rest, order.end());
        order.erase(rest, order.end());
      }
    }
    std::vector<int> lane_of(order.size());
    {
      std::vector<int64_t> load(K, 0);
      for (size_t i = 0; i < order.size(); i++) {
        const int k = (int)(std::min_element(load.begin(), load.end()) - load.begin());
        lane_of[i] = k;
        load[k] += b->edges[order[i]];
      }
    }
    TeamPlan plan;
    if (!team.empty() && !(c->exec && c->exec_key == key)) {
      plan = plan_teams(c, b, team, K, lo.ctas_per_sm > 0 ? lo.ctas_per_sm * c->sm_count : INT_MAX);
      ECL_CUDA_TRY(cudaMemcpyAsync(c->d_team_graphs, plan.descs.data(), plan.descs.size() * sizeof(GraphDesc),
                                   cudaMemcpyHostToDevice, s));
    }
    auto enqueue_large = [&](cudaStream_t q) -> int {
      if (!team.empty()) {
        const int r = batch_teams(c, b, plan, learned, d_inMST, &lo, q);
        if (r) return r;
      }
      if (order.empty()) return ECL_OK;
      if (K > 1) {
        ECL_CUDA_TRY(cudaEventRecord(c->large_fork, q));
        for (int k = 0; k < K; k++) ECL_CUDA_TRY(cudaStreamWaitEvent(c->big[k]->stream, c->large_fork, 0));
      }
      for (size_t i = 0; i < order.size(); i++) {
        const int g = order[i];
        ecl_mst_ctx* e = c->big[lane_of[i]];
        const cudaStream_t sq = K > 1 ? e->stream : q;
        ecl_graph dg = {b->nodes[g], b->edges[g], b->nindex + b->nindex_off[g], b->nlist + b->edge_off[g],
                        b->eweight + b->edge_off[g]};
        ECL_CUDA_TRY(cudaMemsetAsync(e->st, 0, sizeof(DevState), sq));
        mst_opts go = lo;
        LearnedPlan lp{e->side, e->prep_done, e->join, nullptr};
        const LearnedPlan* plan = nullptr;
        if (learned && dg.edges >= kLearnedMinEdges) {
          const int r = learned_fork(e, &dg, sq, &lp);
          if (r) return r;
          plan = &lp;
        } else if (go.threshold_mode == ECL_THRESH_LEARNED) {
          go.threshold_mode = ECL_THRESH_HEURISTIC;
        }
        int r = enqueue_solve(e, &dg, d_inMST + b->edge_off[g], &go, sq, false, plan);
        if (r) return r;
        k_or_error<<<1, 1, 0, sq>>>(e->st, c->st);
        ECL_CUDA_TRY(cudaGetLastError());
      }
      if (K > 1)
        for (int k = 0; k < K; k++) {
          ECL_CUDA_TRY(cudaEventRecord(c->large_join[k], c->big[k]->stream));
          ECL_CUDA_TRY(cudaStreamWaitEvent(q, c->large_join[k], 0));
        }
      return ECL_OK;
    };
    if (c->exec && c->exec_key == key) {
      ECL_CUDA_TRY(cudaGraphLaunch(c->exec, s));
      replayed = true;
    } else {
      if (c->exec) {
        cudaGraphExecDestroy(c->exec);
        c->exec = nullptr;
      }
      cudaGraph_t graph = nullptr;
      bool captured = false;
      if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
        const int r = enqueue_large(s);
        const cudaError_t e = cudaStreamEndCapture(s, &graph);
        if (r == ECL_OK && e == cudaSuccess && graph &&
            cudaGraphInstantiate(&c->exec, graph, 0) == cudaSuccess) {
          captured = true;
          c->exec_key = key;
        }
        if (graph) cudaGraphDestroy(graph);
      }
      cudaGetLastError();  // clear a failed capture's error state
      if (captured) {
        ECL_CUDA_TRY(cudaGraphLaunch(c->exec, s));
        replayed = true;
      } else {
        c->exec = nullptr;
        int r = enqueue_large(s);
        if (r) return r;
      }
    }
  }
  if (timed) ECL_CUDA_TRY(cudaEventRecord(c->ev[2], s));
  if (stats) {
    memset(stats, 0, sizeof(*stats));
    stats->graphs_small = S;
    stats->graphs_large = (int)large.size();
    stats->graph_replay = replayed ? 1 : 0;
    stats->edges_total = edges_total;
  }
  return ECL_OK;
}

int batch_finish(ecl_batch_ctx* c, cudaStream_t s, ecl_batch_stats* stats) {
  ECL_CUDA_TRY(cudaStreamSynchronize(s));
  unsigned err = 0;
  ECL_CUDA_TRY(cudaMemcpy(&err, &c->st->error, sizeof(unsigned), cudaMemcpyDeviceToHost));
  if (stats) {
    stats->status = (int32_t)err;
    cudaEventElapsedTime(&stats->ms_small, c->ev[0], c->ev[1]);
    cudaEventElapsedTime(&stats->ms_large, c->ev[1], c->ev[2]);
    cudaEventElapsedTime(&stats->ms_total, c->ev[0], c->ev[2]);
  }
  return device_error_status(err);
}

}  // namespace

extern "C" int ecl_mst_run_batch_device(ecl_batch_ctx* c, const ecl_batch* b, uint8_t* d_inMST,
                                        const mst_opts* opts, void* stream, ecl_batch_stats* stats) {
  if (!c || !b || !d_inMST || b->num_graphs < 0 || !b->nodes || !b->edges || !b->nindex_off ||
      !b->edge_off || !b->nindex)
    return ECL_ERR_INVALID_ARG;
  if (b->num_graphs > c->max_graphs) return ECL_ERR_TOO_LARGE;
  mst_opts o;
  if (opts) o = *opts;
  else ecl_default_opts(&o);
  int st = check_opts(&o);
  if (st) return st;
  if (o.flags & kDeoptFlags) return ECL_ERR_UNSUPPORTED;  // single-graph contexts only
  ECL_CUDA_TRY(cudaSetDevice(c->device));
  cudaStream_t s = stream ? (cudaStream_t)stream : c->stream;
  if ((st = batch_enqueue(c, b, d_inMST, &o, s, stats != nullptr, stats))) return st;
  if (stats) return batch_finish(c, s, stats);
  return ECL_OK;
}

extern "C" int ecl_batch_autotune(ecl_batch_ctx* c, const ecl_batch* b, uint8_t* d_inMST,
                                  const mst_opts* base, mst_opts* best, float* best_ms) {
  if (!c || !b || !best) return ECL_ERR_INVALID_ARG;
  mst_opts o0;
  if (base) o0 = *base;
  else ecl_default_opts(&o0);
  float best_t = 1e30f;
  mst_opts best_o = o0;
  // one candidate: a warm-up run (which also captures), then a timed one
  auto trial = [&](const mst_opts& o) -> int {
    float t = 0.f;
    for (int rep = 0; rep < 2; rep++) {
      ecl_batch_stats bs;
      const int st = ecl_mst_run_batch_device(c, b, d_inMST, &o, nullptr, &bs);
      if (st) return st;
      if (rep > 0) t += bs.ms_total;
    }
    if (t < best_t) {
      best_t = t;
      best_o = o;
    }
    return ECL_OK;
  };
  int st;
  const int cutoffs[] = {c->cap / 8, c->cap / 4, c->cap / 2, c->cap};
  // 1. small-graph cutoff and schedule. The learned schedule (large graphs
  //    only) is kept only where it beats the reference heuristic on this
  //    batch. (degree_split changes no kernel's work and stays as in *base.)
  const int modes[] = {o0.threshold_mode, ECL_THRESH_HEURISTIC};
  const int nmodes = o0.threshold_mode == ECL_THRESH_LEARNED ? 2 : 1;
  for (int mi = 0; mi < nmodes; mi++)
    for (int cut : cutoffs) {
      if (cut < 1) continue;
      mst_opts o = o0;
      o.threshold_mode = modes[mi];
      o.batch_small_edges = cut;
      if ((st = trial(o))) return st;
    }
  // 2. the large graphs' streams and round CTAs per SM, unless *base sets them
  if (best_o.batch_large_streams == 0 && best_o.ctas_per_sm == 0) {
    const mst_opts o1 = best_o;
    for (int k : {1, 2, 4, 8})
      for (int cps : {1, 2}) {
        mst_opts o = o1;
        o.batch_large_streams = k;
        o.ctas_per_sm = cps;
        if ((st = trial(o))) return st;
      }
    // 3. the cutoff again, now that the large graphs run concurrently
    const mst_opts o2 = best_o;
    for (int cut : cutoffs) {
      if (cut < 1 || cut == o2.batch_small_edges) continue;
      mst_opts o = o2;
      o.batch_small_edges = cut;
      if ((st = trial(o))) return st;
    }
  }
  *best = best_o;
  if (best_ms) *best_ms = best_t;
  return ECL_OK;
}
