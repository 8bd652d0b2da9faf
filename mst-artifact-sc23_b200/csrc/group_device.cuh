// A whole solve (initPM, initWL<true>, rounds, initWL<false>, rounds:
// ECL-MST/ECL_MST.cu:305-340) in one launch, for a graph of up to kGroupEdges
// entries, on a grid of as many CTAs as its size asks for. At these sizes the
// ten launches of the separate kernels cost more than their work: an empty one
// takes 5-8 us.
#pragma once
#include "rounds_device.cuh"

namespace ecl {

// 512 threads, two worklist entries each, two CTAs per SM: the scans and the
// rounds together take 64 registers.
constexpr int kGroupThreads = 512, kGroupEpt = 2, kGroupBlocks = 2;
constexpr int kGroupTile = kGroupThreads * 4;  // CSR entries a CTA scans at a time

struct GroupArgs {
  int nodes, edges;
  const int* nindex;
  const int* nlist;
  const int* eweight;
  unsigned char* inMST;
  int* parent;
  u64* minv;
  int* roots0;  // nodes entries each
  int* roots1;
  int4* wl0;
  int4* wl1;
  unsigned wl_cap;
  unsigned chunk;  // worklist slots a CTA reserves at once, 0 = exactly what it needs
  DevState* st;
  int mode, explicit_thr, split;
  float quantile;
  unsigned solo;
  int min_tiles;
  int count_atomics;
};

struct GroupSmem {
  union {
    BorSmem bor;
    int samp[4096];
  };
  u64 chunk;  // the CTA's current slots: first << 32 | given out
  unsigned kept;
};

// The row that holds entry `jl` and the one that holds `jh` >= jl, found by
// the whole warp: every step probes 32 rows of each range.
__device__ __forceinline__ void warp_rows(const int* nindex, int n, int jl, int jh, int& lo, int& hi) {
  const int lane = threadIdx.x & 31;
  int len_l = n, len_h = n;
  lo = hi = 0;
  while (len_l > 1 || len_h > 1) {
    const int sl = (int)(((unsigned)len_l + 31u) >> 5), sh = (int)(((unsigned)len_h + 31u) >> 5);  // n up to INT_MAX
    const int pl = lane * sl, ph = lane * sh;
    const bool bl = pl < len_l && (lane == 0 || __ldg(nindex + lo + pl) <= jl);
    const bool bh = ph < len_h && (lane == 0 || __ldg(nindex + hi + ph) <= jh);
    const int kl = __popc(__ballot_sync(0xffffffffu, bl)) - 1, kh = __popc(__ballot_sync(0xffffffffu, bh)) - 1;
    lo += kl * sl;
    len_l = min(sl, len_l - kl * sl);
    hi += kh * sh;
    len_h = min(sh, len_h - kh * sh);
  }
}

// row_on over the CSR itself. The search is out of line: in line at every entry of
// a scan it cost the one-cluster solve of 1000 vertices 1 us of 72, by its size.
__device__ __noinline__ int last_row_of(const int* nindex, int lo, int hi, int j) {
  return last_row([&](int r) { return __ldg(nindex + r); }, lo, hi, j);
}
__device__ __forceinline__ void row_on(const int* nindex, int top, int j, int& v, int& end) {
  row_on([&](int r) { return __ldg(nindex + r); }, [&](int lo, int hi) { return last_row_of(nindex, lo, hi, j); }, top,
         j, v, end);
}

// initWL by a group: every thread takes four consecutive entries, looks for
// the row of the first between the rows its warp spans, and walks on from
// there; appends as tuples, in chunks of slots the CTA's warps share.
template <int KIND>
__device__ void group_scan(const GroupArgs& g, unsigned rank, unsigned ctas, GroupSmem& sm) {
  const int n = g.nodes, m = g.edges, lane = threadIdx.x & 31;
  const int thr = g.st->threshold;
  const bool vec = ((((uintptr_t)g.nlist) | ((uintptr_t)g.eweight)) & 15) == 0;
  const bool zero_vec = (((uintptr_t)g.inMST) & 3) == 0;
  ListCount& list = g.st->lists[KIND == kLight ? kListLight0 : kListHeavy];
  if (threadIdx.x == 0) {
    sm.chunk = g.chunk;
    sm.kept = 0;
  }
  __syncthreads();
  bool bad = false;
  for (long long base = (long long)rank * kGroupTile; base < m; base += (long long)ctas * kGroupTile) {
    const int jw = (int)base + ((int)threadIdx.x & ~31) * 4;  // the warp's first entry
    if (jw >= m) continue;                                    // (whole warps)
    const int j0 = jw + lane * 4, own = min(4, m - j0);       // own <= 0: none
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
    if (KIND == kHeavy) {  // the trees of both ends, all loads in flight together
#pragma unroll
      for (int i = 0; i < 4; i++)
        if ((pass >> i) & 1u) {
          e[i].x = ld_ca(g.parent + e[i].x);
          e[i].y = ld_ca(g.parent + e[i].y);
        }
#pragma unroll
      for (int i = 0; i < 4; i++)
        if (e[i].x == e[i].y) pass &= ~(1u << i);
    }
    // the warp's slots
    unsigned mask[4], total = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      mask[i] = __ballot_sync(0xffffffffu, (pass >> i) & 1u);
      total += __popc(mask[i]);
    }
    if (!total) continue;
    unsigned pos = 0, avail = 0, fresh = 0;
    if (lane == 0) {
      chunk_take(&sm.chunk, g.chunk, &list.slots, total, pos, avail, fresh, g.st, g.wl_cap);
      atomicAdd(&sm.kept, total);
    }
    pos = __shfl_sync(0xffffffffu, pos, 0);
    avail = __shfl_sync(0xffffffffu, avail, 0);
    fresh = __shfl_sync(0xffffffffu, fresh, 0);
    unsigned before = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const unsigned r = before + __popc(mask[i] & ((1u << lane) - 1u));
      before += __popc(mask[i]);
      if (!((pass >> i) & 1u)) continue;
      const unsigned slot = r < avail ? pos + r : fresh + (r - avail);
      if (slot >= g.wl_cap) atomicOr(&g.st->error, kErrOverflow);
      else __stcg(g.wl0 + slot, e[i]);
    }
  }
  if (bad) atomicOr(&g.st->error, kErrIds);  // a neighbour id outside [0, n)
  __syncthreads();
  const unsigned first = (unsigned)(sm.chunk >> 32);  // null entries in the slots not given out
  for (unsigned p = (unsigned)sm.chunk + threadIdx.x; p < g.chunk; p += kGroupThreads)
    if (first + p < g.wl_cap) g.wl0[first + p] = make_int4(-1, -1, 0, 0);
  if (threadIdx.x == 0 && sm.kept) atomicAdd(&list.kept, sm.kept);
}

// The rounds of one phase by the group, then the whole group again.
__device__ bool group_rounds(const GroupArgs& g, int phase, int skip, GridSync& sy, GroupSmem& sm) {
  BorArgs a{};
  a.phase = phase;
  a.nodes = g.nodes;
  a.list = phase == 0 ? kListLight0 : kListHeavy;
  a.wl0 = g.wl0;
  a.wl1 = g.wl1;
  a.wl_cap = g.wl_cap;
  a.parent = g.parent;
  a.minv = g.minv;
  a.roots0 = g.roots0;
  a.roots1 = g.roots1;
  a.inMST = g.inMST;
  a.st = g.st;
  a.solo = g.solo;
  a.min_tiles = g.min_tiles;
  a.count_atomics = g.count_atomics;
  BorState b = {};
  b.W = min(ld_volatile(&g.st->lists[a.list].slots), g.wl_cap);
  b.first = 1;
  b.skip = skip;
  __syncthreads();  // the scan's use of the shared memory is over
  bor_smem_init(sm.bor);
  __syncthreads();
  if (sy.rank == 0 && threadIdx.x == 0) {
    g.st->t_round_start[phase] = globaltimer_ns();
    g.st->wl_count[phase][0] = b.W;
    g.st->wl_kept[phase][0] = ld_volatile(&g.st->lists[a.list].kept);
  }
  bool left;
  bor_rounds<kGroupThreads, kGroupEpt, true, false>(a, b, sy, sm.bor, left);
  if (sy.rank == 0 && threadIdx.x == 0) g.st->rounds[phase] = b.r;
  return sy.regroup(left);
}

// One solve; the control block's counters are zero. False if a barrier timed
// out. Every thread of the group calls this.
__device__ bool group_solve(const GroupArgs& g, GridSync& sy, GroupSmem& sm) {
  DevState* st = g.st;
  const unsigned rank = sy.rank, ctas = sy.active, tid = threadIdx.x;
  const unsigned gid = rank * kGroupThreads + tid, stride = ctas * kGroupThreads;
  const int n = g.nodes, m = g.edges;
  if (m == 0) return true;
  // a step's end is read before a barrier and stored after it: neither is waited for
  const bool stamp = rank == 0 && tid == 0;
  auto now = [&]() { return stamp ? globaltimer_ns() : 0ull; };
  auto step_done = [&](int step, u64 t) {
    if (stamp) st->t_step[step] = t;
  };
  u64 t = now();
  step_done(kStepStart, t);
  if (rank == 0) {
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
  for (unsigned v = gid; v < (unsigned)n; v += stride) {
    g.parent[v] = (int)v;
    g.minv[v] = kNoEdge;
    const int b = __ldg(g.nindex + v), e = __ldg(g.nindex + v + 1);
    bad |= b < 0 || e < b || e > m;
  }
  if (gid == 0) bad |= __ldg(g.nindex) != 0 || __ldg(g.nindex + n) != m;
  if (bad) atomicOr(&st->error, kErrFormat);
  t = now();
  if (!sy.sync()) return false;
  step_done(kStepPrep, t);
  if (ld_volatile(&st->error) & kErrFormat) return true;  // only set before the barrier: the whole group
  group_scan<kLight>(g, rank, ctas, sm);
  if (!sy.sync()) return false;
  const int filtered = st->filtered;
  if (!group_rounds(g, 0, -1, sy, sm)) return false;
  if (!filtered) return true;
  // parent[v] = root(v), and the tree most entries point into (a vote of 32)
  for (unsigned v = gid; v < (unsigned)n; v += stride) {
    const int p = __ldcg(g.parent + v);
    int r = p;
    for (int x = ld_ca(g.parent + r); x != r; x = ld_ca(g.parent + r)) r = x;
    if (r != p) __stcg(g.parent + v, r);
  }
  if (gid < 32) {
    int v = __ldg(g.nlist + (unsigned)(((u64)uf_prio((int)gid + 1) * (u64)m) >> 32));
    v = (unsigned)v < (unsigned)n ? v : 0;
    const int r = find_ro(v, g.parent);
    const unsigned same = __popc(__match_any_sync(0xffffffffu, r));
    if (same == __reduce_max_sync(0xffffffffu, same)) st->giant = r;  // any of the largest groups
  }
  t = now();
  if (!sy.sync()) return false;
  step_done(kStepFlatten, t);
  const int giant = (int)ld_volatile((const unsigned*)&st->giant);
  group_scan<kHeavy>(g, rank, ctas, sm);
  if (!sy.sync()) return false;
  return group_rounds(g, 1, giant, sy, sm);
}

__global__ void __launch_bounds__(kGroupThreads, kGroupBlocks) k_group(GroupArgs g) {
  __shared__ GroupSmem sm;
  GridSync sy;
  sy.init(g.st, g.st->bar, blockIdx.x, gridDim.x);
  group_solve(g, sy, sm);
}

// ------------------------------------------------------------------ batch
// A batch's mid-size graphs (too large for a cluster) by teams of CTAs side by
// side in one launch. A round on such a graph is bound by latency, not by the
// chip's width, so more graphs in flight on fewer CTAs each is what fills the
// chip; and a graph costs two team barriers instead of a chain of launches that
// wait for one another's SMs. 53 graphs of 0.1M to 2M entries: 3.6 ms on eight
// teams against 5.5 on eight streams. Teams and their graphs are planned on the
// host (plan_teams); a team's CTAs are its share of the entries.
constexpr int kMaxTeams = 48;

struct Team {
  u64* slots;     // min slots, root lists and parents, laid out per graph
  int4* wl0;      // for its largest graph
  int4* wl1;
  unsigned wl_cap;
  int first_graph;
  int first_cta;
};
struct TeamWords {  // zero when the launch starts
  unsigned bar[4];  // as DevState::bar
};

struct TeamArgs {
  const GraphDesc* graphs;      // by team
  const LearnedChoice* choice;  // learned mode: by graph, for graphs of learned_min entries or more
  int teams, learned_min;
  Team team[kMaxTeams + 1];     // the last one holds the ends of the lists
  DevState* states;             // by team
  TeamWords* words;
  const int* nindex;
  const int* nlist;
  const int* eweight;
  unsigned char* inMST;
  DevState* st;                 // the batch's error word and atomics counter
  int mode, explicit_thr, split;
  float quantile;
  unsigned solo;
  int min_tiles;
  int count_atomics;
};

__global__ void __launch_bounds__(kGroupThreads, kGroupBlocks) k_batch_group(__grid_constant__ const TeamArgs b) {
  __shared__ GroupSmem sm;
  __shared__ GroupArgs g;
  int t = 0;
  while (t + 1 < b.teams && (int)blockIdx.x >= b.team[t + 1].first_cta) t++;
  const Team& team = b.team[t];
  DevState* st = b.states + t;
  const unsigned ctas = (unsigned)(b.team[t + 1].first_cta - team.first_cta);
  GridSync sy;
  sy.init(st, b.words[t].bar, blockIdx.x - (unsigned)team.first_cta, ctas);
  bool ok = true;
  const int last = b.team[t + 1].first_graph;
  for (int i = team.first_graph; i < last; i++) {
    if (threadIdx.x == 0) {
      const GraphDesc d = b.graphs[i];
      g.nodes = d.nodes;
      g.edges = d.edges;
      g.nindex = b.nindex + d.nindex_off;
      g.nlist = b.nlist + d.edge_off;
      g.eweight = b.eweight + d.edge_off;
      g.inMST = b.inMST + d.edge_off;
      g.minv = team.slots;
      g.roots0 = reinterpret_cast<int*>(team.slots + d.nodes);
      g.roots1 = g.roots0 + d.nodes;
      g.parent = g.roots1 + d.nodes;
      g.wl0 = team.wl0;
      g.wl1 = team.wl1;
      g.wl_cap = team.wl_cap;
      g.chunk = min(256u, (team.wl_cap - (unsigned)d.edges) / ctas);
      if (g.chunk < 128) g.chunk = 0;  // a warp may append 128 entries at once
      g.st = st;
      g.mode = b.mode == ECL_THRESH_LEARNED && d.edges < b.learned_min ? (int)ECL_THRESH_HEURISTIC : b.mode;
      g.explicit_thr = b.explicit_thr;
      g.split = b.split;
      g.quantile = b.quantile;
      g.solo = b.solo;
      g.min_tiles = b.min_tiles;
      g.count_atomics = b.count_atomics;
    }
    if (sy.rank == 0) {  // a clear control block
      for (int k = threadIdx.x; k < (int)(sizeof(DevState) / sizeof(unsigned)); k += kGroupThreads)
        reinterpret_cast<unsigned*>(st)[k] = 0;
      __syncthreads();
      if (threadIdx.x == 0 && g.mode == ECL_THRESH_LEARNED) {
        const LearnedChoice c = b.choice[i];
        st->threshold = c.threshold;
        st->filtered = c.filtered;
      }
    }
    if (!(ok = sy.sync())) break;
    if (!(ok = group_solve(g, sy, sm) && sy.sync())) break;
    if (sy.rank == 0 && threadIdx.x == 0) {
      if (st->error) atomicOr(&b.st->error, st->error);
      if (b.count_atomics && st->atomics) atomicAdd(&b.st->atomics, st->atomics);
    }
    __syncthreads();  // before the control block is cleared again
  }
  if (!ok && threadIdx.x == 0) atomicOr(&b.st->error, kErrTimeout);
}

}  // namespace ecl
