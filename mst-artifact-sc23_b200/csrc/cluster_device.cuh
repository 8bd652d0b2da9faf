// A whole solve (ECL-MST/ECL_MST.cu:305-340) by one thread-block cluster, for
// graphs so small that the latency of a round's dependent accesses and its
// barriers is all there is: a cluster barrier takes 0.32 us, a grid barrier
// 1.2. One CTA keeps parent[] and the min slots in its shared memory; two to
// eight reach them in L2. (Spread over the cluster's shared memories they were
// slower, 2-4 cycles per remote atomic and SM: RMAT-14 224 against 154 us.)
// Every CTA keeps the worklist entries it scanned, so a round needs no list
// exchange, and the roots pass looks at every vertex the CTA owns (v mod C), so
// there is no root list. Three barriers per round:
//
//   offer   entries to reps, drop the ones inside a tree, offer the rest
//   mark    entries that hold a minimum: union, inMST
//   roots   offered vertices clear their slot and point to their new root
#pragma once
#include <cstddef>

#include "group_device.cuh"

namespace ecl {

constexpr int kClThreads = 1024;
constexpr int kClVertices = 16384;         // vertices a CTA alone can hold: 12 bytes each
constexpr int kClTile = kClThreads * 4;    // CSR entries a CTA scans at a time
constexpr int kClMaxCtas = 8;              // CTAs of a cluster
// Vertices per CTA from which a short list's roots pass takes the ends of its
// entries instead of looking at every vertex. 400 graphs of 40 000 vertices and
// 2000 edges 0.35 ms against 0.44, one of 500 000 and 50 000 0.20 against 0.26; on
// 3000 vertices per CTA it is 7 % slower (one graph of 24 000, 12 000 entries).
constexpr int kClManyVertices = 8 * kClThreads;
constexpr size_t kClSmem = (size_t)kClVertices * (sizeof(u64) + sizeof(int));

struct ClArgs {
  int nodes, edges;
  const int* nindex;
  const int* nlist;
  const int* eweight;
  unsigned char* inMST;
  int4* wl0;  // room for `edges` entries each
  int4* wl1;
  int* parent;  // two CTAs and more
  u64* minv;
  DevState* st;
  int mode, explicit_thr, split;
  float quantile;
  int count_atomics;
  int batch;
};

struct ClSmem {
  int samp[4096];      // choose_threshold
  unsigned cursor;     // entries of this CTA's list
  unsigned total[3];   // entries of all lists, by pass
};

// parent[] and the min slots: in shared memory (kOne, one CTA) or in L2.
template <bool kOne>
struct ClMem {
  unsigned rank, log;  // of the cluster's CTAs; log2 of their number
  int* par;
  u64* min;
  __device__ __forceinline__ int parent(int v) const { return kOne ? ((volatile int*)par)[v] : ld_ca(par + v); }
  // `settled`: nobody writes the slots before the next barrier
  __device__ __forceinline__ u64 minv(int v, bool settled) const {
    if (kOne) return ((volatile u64*)min)[v];
    return settled ? ld_ca64(min + v) : __ldcg(min + v);
  }
  __device__ __forceinline__ void set_parent(int v, int x) const {
    if (kOne) ((volatile int*)par)[v] = x;
    else __stcg(par + v, x);
  }
  __device__ __forceinline__ void set_minv(int v, u64 x) const {
    if (kOne) ((volatile u64*)min)[v] = x;
    else __stcg(min + v, x);
  }
  __device__ __forceinline__ int root(int v) const {
    for (int p = parent(v); p != v; p = parent(v)) v = p;
    return v;
  }
  // As cas_union (mst_kernels.cuh).
  __device__ __forceinline__ void join(int a, int b) const {
    while (a != b) {
      if (uf_prio(a) > uf_prio(b)) {
        const int t = a;
        a = b;
        b = t;
      }
      const int old = atomicCAS(par + a, a, b);
      if (old == a) return;
      a = old;
    }
  }
  // Adds `x` to the same shared-memory counter of every CTA (one thread).
  __device__ __forceinline__ void add_all(unsigned* counter, unsigned x) const {
    if (kOne || log == 0) *counter += x;
    else for (unsigned r = 0; r < (1u << log); r++) {
      unsigned a;
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(counter)), "r"(r));
      asm volatile("red.shared::cluster.add.u32 [%0], %1;" ::"r"(a), "r"(x) : "memory");
    }
  }
};

// A batch graph's quantile threshold: 64 hashed samples, sorted by insertion
// (one thread).
__device__ __noinline__ void batch_quantile(DevState* st, const int* eweight, int edges, float quantile) {
  int s[64];
  const int ns = edges < 64 ? edges : 64;
  for (int i = 0; i < ns; i++) {
    const uint64_t r = ecl_mix64(0x5EED0000ull + (uint64_t)i);
    const int x = eweight[(unsigned)(r % (uint64_t)(unsigned)edges)];
    int k = i - 1;
    while (k >= 0 && s[k] > x) {
      s[k + 1] = s[k];
      k--;
    }
    s[k + 1] = x;
  }
  const int idx = (int)(quantile * (float)(ns - 1));
  st->filtered = 1;
  st->threshold = s[idx < 0 ? 0 : (idx > ns - 1 ? ns - 1 : idx)];
}

// initWL by a cluster: as group_scan, but into the CTA's own list (`out`).
template <int KIND, bool kOne>
__device__ void cl_scan(const ClArgs& g, const ClMem<kOne>& M, unsigned ctas, int thr, int4* out, ClSmem& sm) {
  const int n = g.nodes, m = g.edges, lane = threadIdx.x & 31;
  const bool vec = ((((uintptr_t)g.nlist) | ((uintptr_t)g.eweight)) & 15) == 0;
  const bool zero_vec = (((uintptr_t)g.inMST) & 3) == 0;
  bool bad = false;
  for (int base = (int)M.rank * kClTile; base < m; base += (int)ctas * kClTile) {
    const int jw = base + ((int)threadIdx.x & ~31) * 4;  // the warp's first entry
    if (jw >= m) continue;                               // (whole warps)
    const int j0 = jw + lane * 4, own = min(4, m - j0);  // own <= 0: none
    int nb[4] = {}, w[4] = {};
    if (own == 4 && vec) {
      const int4 x = __ldg(reinterpret_cast<const int4*>(g.nlist + j0));
      const int4 y = __ldg(reinterpret_cast<const int4*>(g.eweight + j0));
      nb[0] = x.x; nb[1] = x.y; nb[2] = x.z; nb[3] = x.w;
      w[0] = y.x; w[1] = y.y; w[2] = y.z; w[3] = y.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (i < own) {
          nb[i] = __ldg(g.nlist + j0 + i);
          w[i] = __ldg(g.eweight + j0 + i);
        }
    }
    if (KIND == kLight && own > 0) {
      if (own == 4 && zero_vec) *reinterpret_cast<unsigned*>(g.inMST + j0) = 0u;
      else
        for (int i = 0; i < own; i++) g.inMST[j0 + i] = 0;
    }
    int lo, hi;
    warp_rows(g.nindex, n, jw, min(jw + 127, m - 1), lo, hi);
    const int top = hi;
    while (lo < hi && own > 0) {  // the last row starting at or before j0
      const int mid = lo + ((hi - lo + 1) >> 1);
      if (__ldg(g.nindex + mid) <= j0) lo = mid;
      else hi = mid - 1;
    }
    int v = lo, end = own > 0 ? __ldg(g.nindex + v + 1) : 0;
    int4 e[4];
    unsigned pass = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if (i < own) {
        row_on(g.nindex, top, j0 + i, v, end);
        bad |= (unsigned)nb[i] >= (unsigned)n;
        // one direction with a valid id (v < nb < n) as one unsigned compare
        if ((unsigned)nb[i] - (unsigned)v - 1u < (unsigned)(n - v - 1) && (KIND == kLight ? w[i] <= thr : w[i] > thr))
          pass |= 1u << i;
      }
      e[i] = make_int4(v, nb[i], w[i], j0 + i);
    }
    if (KIND == kHeavy) {  // the trees of both ends
#pragma unroll
      for (int i = 0; i < 4; i++)
        if ((pass >> i) & 1u) {
          e[i].x = M.parent(e[i].x);
          e[i].y = M.parent(e[i].y);
        }
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (e[i].x == e[i].y) pass &= ~(1u << i);
    }
    unsigned mask[4], total = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      mask[i] = __ballot_sync(0xffffffffu, (pass >> i) & 1u);
      total += __popc(mask[i]);
    }
    if (!total) continue;
    unsigned pos = 0;
    if (lane == 0) pos = atomicAdd(&sm.cursor, total);
    pos = __shfl_sync(0xffffffffu, pos, 0);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      if ((pass >> i) & 1u) __stcg(out + pos + __popc(mask[i] & ((1u << lane) - 1u)), e[i]);
      pos += __popc(mask[i]);
    }
  }
  if (bad) atomicOr(&g.st->error, kErrIds);  // a neighbour id outside [0, n)
}

// All rounds of one phase over the CTAs' lists in `a` (cursor entries here);
// `b` is the other list array. `skip` offers nothing (rounds_device.cuh).
template <bool kOne>
__device__ void cl_rounds(const ClArgs& g, const ClMem<kOne>& M, ClusterSync& sy, int phase, int skip, int4* a, int4* b,
                          unsigned& pass_no, ClSmem& sm) {
  DevState* st = g.st;
  const int tid = threadIdx.x, lane = tid & 31;
  const bool stamp = M.rank == 0 && tid == 0;
  const unsigned below = (1u << lane) - 1u;
  unsigned atomics = 0;
  // many vertices to a CTA: a list of a quarter as many entries names the offered ones sooner
  const bool few = !kOne && g.nodes >> M.log >= kClManyVertices;
  // entries of all CTAs: counted into every CTA's `total` before a barrier
  auto count = [&]() {
    if (tid == 0 && sm.cursor) M.add_all(&sm.total[pass_no % 3], sm.cursor);
  };
  if (stamp) st->t_round_start[phase] = globaltimer_ns();
  count();
  sy.sync();
  unsigned W = sm.total[pass_no % 3], mine = sm.cursor;
  if (tid == 0) sm.total[(pass_no + 2) % 3] = 0;  // used two passes from now, three barriers away
  pass_no++;
  if (stamp) {
    st->wl_count[phase][0] = W;
    st->wl_kept[phase][0] = W;
    st->lists[phase == 0 ? kListLight0 : kListHeavy].kept = W;
  }
  int r = 0;
  for (; W; r++) {
    if (r >= ECL_MAX_ROUNDS) {
      if (stamp) atomicOr(&st->error, kErrRounds);
      break;
    }
    __syncthreads();  // `mine` read by all
    if (tid == 0) sm.cursor = 0;
    __syncthreads();
    // ---- offer
    int4 next = tid < mine ? __ldcg(a + tid) : make_int4(-1, -1, 0, 0);
    for (unsigned base = 0; base < mine; base += kClThreads) {
      int4 e = next;
      const unsigned ahead = base + kClThreads + tid;
      next = ahead < mine ? __ldcg(a + ahead) : make_int4(-1, -1, 0, 0);
      bool on = e.x >= 0;
      if (r > 0) {
        if (on) {
          e.x = M.parent(e.x);
          e.y = M.parent(e.y);
        }
        on = on && e.x != e.y;
        const unsigned mask = __ballot_sync(0xffffffffu, on);
        unsigned pos = 0;
        if (lane == 0 && mask) pos = atomicAdd(&sm.cursor, (unsigned)__popc(mask));
        pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(mask & below);
        if (on) __stcg(b + pos, e);
      }
      const u64 key = edge_key(e.z, e.w);
#pragma unroll
      for (int side = 0; side < 2; side++) {
        const int rep = side ? e.y : e.x;
        bool offer = on && rep != skip;
        u64 val = key;
        const int id = offer ? rep : -2 - lane;
        const int up = __shfl_up_sync(0xffffffffu, id, 1);
        if (__any_sync(0xffffffffu, lane > 0 && up == id)) {  // equal neighbours: the warp reduces first
          const unsigned grp = __match_any_sync(0xffffffffu, id);
          if (offer && (grp & (grp - 1))) {
            const unsigned khi = (unsigned)(key >> 32);
            const unsigned hi = __reduce_min_sync(grp, khi);
            const unsigned lo = __reduce_min_sync(grp, khi == hi ? (unsigned)key : 0xffffffffu);
            val = ((u64)hi << 32) | lo;
            offer = lane == __ffs(grp) - 1;
          }
        }
        const u64 seen = offer ? M.minv(rep, false) : 0ull;
        if (seen > val) {
          atomicMin(M.min + rep, val);
          atomics++;
        }
      }
    }
    __syncthreads();
    if (r > 0) {
      count();
    } else if (tid == 0) {
      sm.cursor = mine;  // the first round keeps its list as it is
    }
    sy.sync();
    if (stamp) st->t_round[phase][2 * r] = globaltimer_ns();
    const unsigned W2 = r > 0 ? sm.total[pass_no % 3] : W;
    if (r > 0) {
      if (tid == 0) sm.total[(pass_no + 2) % 3] = 0;
      pass_no++;
    }
    if (stamp) {
      st->wl_count[phase][r + 1] = W2;
      st->wl_kept[phase][r + 1] = W2;
    }
    if (r > 0) {
      int4* t = a;
      a = b;
      b = t;
      mine = sm.cursor;
    }
    if (W2 == 0) {
      r++;
      break;
    }
    W = W2;
    // ---- mark
    next = tid < mine ? __ldcg(a + tid) : make_int4(-1, -1, 0, 0);
    for (unsigned base = 0; base < mine; base += kClThreads) {
      const int4 e = next;
      const unsigned ahead = base + kClThreads + tid;
      next = ahead < mine ? __ldcg(a + ahead) : make_int4(-1, -1, 0, 0);
      if (e.x < 0) continue;
      const u64 key = edge_key(e.z, e.w);
      const u64 mx = e.x != skip ? M.minv(e.x, true) : kNoEdge, my = e.y != skip ? M.minv(e.y, true) : kNoEdge;
      if (key == mx || key == my) {
        M.join(e.x, e.y);
        g.inMST[e.w] = 1;
      }
    }
    sy.sync();
    // ---- roots: the vertices this CTA holds, or the ends of its entries
    auto flat = [&](int v) {
      const int p = M.parent(v);
      if (p == v) return;
      const int root = M.root(p);
      if (root != p) M.set_parent(v, root);
    };
    if (few && 4ull * W <= (u64)(unsigned)g.nodes) {
      for (unsigned i = tid; i < mine; i += kClThreads) {
        const int4 e = __ldcg(a + i);
#pragma unroll
        for (int side = 0; side < 2; side++) {
          const int v = side ? e.y : e.x;  // of an end's entries, the one that takes the key goes on
          if (v != skip && atomicExch(M.min + v, kNoEdge) != kNoEdge) flat(v);
        }
      }
      if (stamp && skip >= 0) flat(skip);
    } else {
      for (unsigned v = M.rank + (tid << M.log); v < (unsigned)g.nodes; v += kClThreads << M.log) {
        if (M.minv((int)v, true) == kNoEdge && (int)v != skip) continue;
        M.set_minv((int)v, kNoEdge);
        flat((int)v);
      }
    }
    sy.sync();
    if (stamp) st->t_round[phase][2 * r + 1] = globaltimer_ns();
    if (skip >= 0) skip = M.parent(skip);
  }
  if (stamp) st->rounds[phase] = r;
  if (g.count_atomics && atomics) atomicAdd(&st->atomics, (u64)atomics);
}

// One solve by the cluster. Every thread of it calls this; the control block
// is cleared here.
template <bool kOne>
__device__ void cl_solve(const ClArgs& g, ClusterSync& sy, const ClMem<kOne>& M, ClSmem& sm) {
  DevState* st = g.st;
  const unsigned ctas = sy.ctas, tid = threadIdx.x, rank = M.rank;
  const int n = g.nodes, m = g.edges;
  if (m == 0) return;
  for (unsigned i = rank * kClThreads + tid; i < sizeof(DevState) / sizeof(unsigned); i += ctas * kClThreads)
    if (i != offsetof(DevState, graph) / sizeof(unsigned)) reinterpret_cast<unsigned*>(st)[i] = 0u;
  if (tid < 3) sm.total[tid] = 0;
  if (tid == 0) sm.cursor = 0;
  // a step's end is read before a barrier and stored after it: neither is waited for
  const bool stamp = rank == 0 && tid == 0;
  auto now = [&]() { return stamp ? globaltimer_ns() : 0ull; };
  auto step_done = [&](int step, u64 t) {
    if (stamp) st->t_step[step] = t;
  };
  u64 t = now();
  sy.sync();
  step_done(kStepStart, t);
  if (rank == 0 && g.batch && g.mode == ECL_THRESH_QUANTILE && g.quantile < 1.0f) {
    if (tid == 0) batch_quantile(st, g.eweight, m, g.quantile);
  } else if (rank == 0) {
    PrepArgs pa{};
    pa.nodes = n;
    pa.edges = m;
    pa.eweight = g.eweight;
    pa.mode = g.mode;
    pa.explicit_thr = g.explicit_thr;
    pa.split = g.split;
    pa.quantile = g.quantile;
    pa.st = st;
    choose_threshold(pa, sm.samp);
  }
  bool bad = false;
  for (unsigned v = rank + (tid << M.log); v < (unsigned)n; v += kClThreads << M.log) {
    M.set_parent((int)v, (int)v);
    M.set_minv((int)v, kNoEdge);
    const int b = __ldg(g.nindex + v), e = __ldg(g.nindex + v + 1);
    bad |= b < 0 || e < b || e > m;
  }
  if (rank == 0 && tid == 0) bad |= __ldg(g.nindex) != 0 || __ldg(g.nindex + n) != m;
  if (bad) atomicOr(&st->error, kErrFormat);
  t = now();
  sy.sync();
  step_done(kStepPrep, t);
  if (ld_volatile(&st->error) & kErrFormat) return;  // only set before the barrier: the whole cluster
  const int thr = (int)ld_volatile((const unsigned*)&st->threshold);
  const int filtered = (int)ld_volatile((const unsigned*)&st->filtered);
  // every CTA's lists start behind the entries the CTAs before it may scan
  const unsigned region = share_region((unsigned)m, kClTile, rank, ctas);
  int4* l0 = g.wl0 + region;
  int4* l1 = g.wl1 + region;
  unsigned pass_no = 0;
  cl_scan<kLight>(g, M, ctas, thr, l0, sm);
  __syncthreads();
  cl_rounds(g, M, sy, 0, -1, l0, l1, pass_no, sm);
  if (!filtered) return;
  __syncthreads();
  if (tid == 0) sm.cursor = 0;
  // parent[v] = root(v), and the tree most entries point into (a vote of 32)
  for (unsigned v = rank + (tid << M.log); v < (unsigned)n; v += kClThreads << M.log) {
    const int p = M.parent((int)v);
    const int r = M.root(p);
    if (r != p) M.set_parent((int)v, r);
  }
  if (rank == 0 && tid < 32) {
    int v = __ldg(g.nlist + (unsigned)(((u64)uf_prio((int)tid + 1) * (u64)m) >> 32));
    v = (unsigned)v < (unsigned)n ? v : 0;
    const int r = M.root(v);
    const unsigned same = __popc(__match_any_sync(0xffffffffu, r));
    if (same == __reduce_max_sync(0xffffffffu, same)) st->giant = r;  // any of the largest groups
  }
  t = now();
  sy.sync();
  step_done(kStepFlatten, t);
  const int giant = (int)ld_volatile((const unsigned*)&st->giant);
  cl_scan<kHeavy>(g, M, ctas, thr, l0, sm);
  __syncthreads();
  cl_rounds(g, M, sy, 1, giant, l0, l1, pass_no, sm);
}

template <bool kOne>
__device__ __forceinline__ void cl_setup(ClusterSync& sy, ClMem<kOne>& M, unsigned ctas, void* dyn, int* par, u64* min) {
  sy.init(ctas);
  M.rank = sy.rank;
  M.log = (unsigned)(31 - __clz((int)ctas));
  M.min = kOne ? reinterpret_cast<u64*>(dyn) : min;
  M.par = kOne ? reinterpret_cast<int*>(M.min + kClVertices) : par;
}

// One graph on one cluster.
template <bool kOne>
__global__ void __launch_bounds__(kClThreads, 1) k_cluster(ClArgs g) {
  extern __shared__ __align__(16) unsigned char cl_dyn[];
  __shared__ ClSmem sm;
  ClusterSync sy;
  ClMem<kOne> M;
  cl_setup(sy, M, gridDim.x, cl_dyn, g.parent, g.minv);
  cl_solve(g, sy, M, sm);
  sy.sync();  // no CTA leaves while another may add to its counters
}

// ------------------------------------------------------------------ batch
// One size class of a batch: `count` graphs, largest first, each solved by
// the next free cluster. Every cluster has its own control block and its own
// share of the scratch pools, for graphs of up to `cap` vertices and entries.
struct BatchArgs {
  const GraphDesc* graphs;
  int count;
  unsigned* queue;
  const int* nindex;
  const int* nlist;
  const int* eweight;
  unsigned char* inMST;
  DevState* states;  // per cluster
  int* parent_pool;  // per cluster: cap
  u64* minv_pool;    // per cluster: cap
  int4* wl_pool;     // per cluster: 2 * cap
  long long cap;
  DevState* st;      // the batch's error word and atomics counter
  int mode, explicit_thr;
  float quantile;
  int count_atomics;
};

// The clusters of a class take its graphs from a queue.
template <bool kOne>
__global__ void __launch_bounds__(kClThreads, 1) k_batch_cluster(BatchArgs b) {
  extern __shared__ __align__(16) unsigned char cl_dyn[];
  __shared__ ClSmem sm;
  ClusterSync sy;
  ClMem<kOne> M;
  unsigned ctas, cluster;
  asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(ctas));
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(cluster));
  cl_setup(sy, M, ctas, cl_dyn, b.parent_pool + (size_t)cluster * b.cap, b.minv_pool + (size_t)cluster * b.cap);
  ClArgs g{};
  g.wl0 = b.wl_pool + (size_t)cluster * 2 * b.cap;
  g.wl1 = g.wl0 + b.cap;
  g.st = b.states + cluster;
  g.mode = b.mode;
  g.explicit_thr = b.explicit_thr;
  g.quantile = b.quantile;
  g.count_atomics = b.count_atomics;
  g.batch = 1;
  for (;;) {
    if (sy.rank == 0 && threadIdx.x == 0) g.st->graph = atomicAdd(b.queue, 1u);
    sy.sync();
    const unsigned i = ld_volatile(&g.st->graph);
    if (i >= (unsigned)b.count) break;
    const GraphDesc d = b.graphs[i];
    g.nodes = d.nodes;
    g.edges = d.edges;
    g.nindex = b.nindex + d.nindex_off;
    g.nlist = b.nlist + d.edge_off;
    g.eweight = b.eweight + d.edge_off;
    g.inMST = b.inMST + d.edge_off;
    cl_solve(g, sy, M, sm);
    sy.sync();
    if (sy.rank == 0 && threadIdx.x == 0 && d.edges) {
      if (g.st->error) atomicOr(&b.st->error, g.st->error);
      if (b.count_atomics && g.st->atomics) atomicAdd(&b.st->atomics, g.st->atomics);
    }
    sy.sync();  // before the control block is cleared again
  }
}

}  // namespace ecl
