// Kernels of the single-graph B200 ECL-MST engine.
//
// Replaces gpuMST<filter>'s kernels (ECL-MST/ECL_MST.cu): initPM (:147-154),
// initWL<first> (:157-207), kernel1 (:210-226), kernel2 (:229-240),
// kernel3 (:243-251), find (:127-134), join (:137-144). The answer is the
// reference's: the unique minimum spanning forest under the strict order
// (uint32 weight, CSR index j) over the one-direction entries nlist[j] > v,
// built in a light phase (w <= threshold, signed compare as at :172) and a
// heavy phase (w > threshold). Launch sequence of one solve:
//
//   k_prep        initPM + CSR checks + threshold choice + the task->row table
//                 of the scans
//   k_scan, light  initWL<true> (scan_device.cuh). Also zeroes inMST
//   k_round       the phase's Boruvka rounds in one cooperative launch
//                 (rounds_device.cuh: kernel1, kernel2, kernel3 per round,
//                 bounded grid barriers, no host round trip per round), and
//   k_round_tail  its last rounds on one thread-block cluster. The ablation
//                 switches run the variants in k_rounds instead.
//   k_flatten     parent[v] = root(v) once after the light phase, and a bit per
//                 vertex of its largest tree
//   k_scan, heavy  initWL<false>: keeps heavy entries across light trees
//   k_round, k_round_tail   heavy phase
#pragma once
#include <cuda_pipeline.h>
#include <cuda_runtime.h>
#include <climits>
#include <stdint.h>

#include "ecl_mst.h"
#include "internal.h"
#include "mst_kernels.cuh"

namespace ecl {

constexpr int kThreads = 512;          // threads of the prep and flatten kernels
constexpr int kGran = 512;             // entries of a scan task, and per step of the task->row table
// Round CTAs of 1024 threads, two per SM (measured on RMAT-22: 2.4 % faster
// with the learned schedule and 4.6 % with the heuristic one than 512 x 4;
// 256 x 8 was 11-15 % slower)
#ifndef ECL_ROUND_THREADS
#define ECL_ROUND_THREADS 1024
#endif
#ifndef ECL_ROUND_MIN_BLOCKS
#define ECL_ROUND_MIN_BLOCKS 2
#endif
#ifndef ECL_FIND_LOG
#define ECL_FIND_LOG 10
#endif
#ifndef ECL_PAIR_LOG
#define ECL_PAIR_LOG 10
#endif
constexpr int kRoundThreads = ECL_ROUND_THREADS;  // threads of a round CTA (one worklist entry each per tile)
#ifndef ECL_ROUND_EPT
#define ECL_ROUND_EPT 1
#endif
constexpr int kEPT = ECL_ROUND_EPT;    // worklist entries per thread in a round tile
constexpr int kHotLog = 9;             // hot representative table: 512 slots
constexpr int kHotSlots = 1 << kHotLog;
constexpr int kFindLog = ECL_FIND_LOG; // find cache
constexpr int kFindSlots = 1 << kFindLog;
constexpr int kPairLog = ECL_PAIR_LOG; // parallel-edge table
constexpr int kPairSlots = 1 << kPairLog;
constexpr u64 kNoPair = ~0ull;
constexpr int kSplitAfter = 8;         // find steps before path splitting starts
// Rounds whose worklist holds at least ECL_FLAT_ROUNDS x n entries first
// point every vertex at its root, so their finds are single loads (RMAT-22:
// 11 % faster with the reference heuristic's schedule, 1 % with the learned
// one; flattening from W >= n already was slower than from W >= 2n)
#ifndef ECL_FLAT_ROUNDS
#define ECL_FLAT_ROUNDS 2
#endif
constexpr unsigned long long kBarrierTimeoutNs = 5ull * 1000 * 1000 * 1000;

struct PrepArgs {
  int nodes, edges;
  const int* nindex;
  const int* eweight;
  int* parent;
  u64* minv0;
  u64* minv1;
  int* first_v;  // [tiles + 1]: row holding entry t * kGran; last = nodes - 1
  int tiles;     // ceil(edges / kGran)
  int mode, explicit_thr, split;
  float quantile;
  int use_lists;   // the light and heavy entries may be split into several lists
  int both_slots;  // minv1 is a min array too (the ablation variants)
  DevState* st;
  FeatAcc* feat;  // learned schedule: degree statistics gathered here, else null
};

struct ScanArgs {
  int nodes, edges;
  const int* nindex;
  const int* nlist;
  const int* eweight;
  const int* first_v;
  int tiles;
  int* parent;
  const unsigned* tree_bits;  // bit v: v lies in the light phase's largest tree
  int4* wl0;
  int4* wl1;
  unsigned wl_cap;
  unsigned char* inMST;
  int zero_vec;  // inMST 16-byte aligned
  unsigned chunk;     // worklist slots a CTA reserves at once (set at launch)
  int ids;            // 1 = append CSR indices (int) instead of tuples (kAblNoTuples)
  DevState* st;
};

struct RoundArgs {
  int phase;
  int nodes;
  int4* wl0;
  int4* wl1;
  unsigned wl_cap;
  int* parent;
  u64* minv0;
  u64* minv1;
  unsigned char* inMST;
  DevState* st;
  unsigned small_tail;
  int count_atomics;
  unsigned abl;  // kAbl* bits: techniques switched off to measure what they buy
  int min_tiles;  // keep one CTA per this many tiles of a round (0 = every CTA)
  // kAblNoTuples: the CSR and the vertex of every entry
  const int* nlist;
  const int* eweight;
  const int* slist;
};

// Ablation switches of the round kernel (mst_opts flags ECL_FLAG_NO_*).
enum : unsigned {
  kAblNoGuards = 1u,     // atomicMin without first reading the slot (ECL_MST.cu:222-223)
  kAblNoCoop = 2u,       // no warp reduction or CTA table for shared reps
  kDedup = 4u,           // parallel-edge elimination on (opt-in: measured slower on RMAT)
  kAblNoFindCache = 8u,  // no per-CTA root cache in the finds
  // The reference's later deoptimization steps, restated so that the forest
  // stays the reference's (one direction is kept):
  kAblNoIPC = 16u,     // NoImplicitPathCompression: compacted entries keep their
                       // endpoints, finds split paths from the first step and
                       // the mark pass finds again
                       // (ECL_MST_..._NoImplicitPathCompression.cu:121-133, 193-216)
  kAblNoTuples = 32u,  // NoTuples: worklists hold CSR indices; endpoints and
                       // weight are gathered every round (..._NoTuples.cu)
  kAblNoDD = 64u,      // NoDataDriven: every round reads the phase's whole list
                       // and nothing is compacted; the rounds end when no entry
                       // joins two trees (..._NoDataDriven.cu:166-180, 263-270)
  kAblBase = 128u,     // nothing off: what the others are compared with
};
// Switches under which worklist entries keep their endpoints (no rewrite to reps)
constexpr unsigned kAblKeepEnds = kAblNoIPC | kAblNoTuples | kAblNoDD;

// ------------------------------------------------------------------ prep
// Threshold rule, by mode (run by one CTA). HEURISTIC restates main's rule
// (ECL_MST.cu:408,432-440); QUANTILE takes a quantile of a 4096-entry hashed
// sample; LEARNED leaves the threshold, filter flag and split to the MLP
// kernel (k_mlp_apply, which runs beside this kernel on another stream and
// takes them from its own sorted sample).
__device__ void choose_threshold(const PrepArgs& a, int* samp) {
  DevState* st = a.st;
  const int tid = threadIdx.x;
  int mode = a.mode, split = a.split;
  float quantile = a.quantile;
  if (mode == ECL_THRESH_LEARNED) return;
  const int nodes = a.nodes, edges = a.edges;
  if (tid == 0) st->split = split;
  if (mode == ECL_THRESH_NONE || (mode == ECL_THRESH_QUANTILE && !(quantile < 1.0f))) {
    if (tid == 0) {
      st->filtered = 0;
      st->threshold = INT_MAX;
    }
    return;
  }
  if (mode == ECL_THRESH_EXPLICIT) {
    if (tid == 0) {
      st->filtered = 1;
      st->threshold = a.explicit_thr;
    }
    return;
  }
  if (mode == ECL_THRESH_HEURISTIC) {
    if (tid < 32) {  // one warp: a lane per sample, its rank by counting
      const int ns = edges < 20 ? edges : 20;
      unsigned val = (unsigned)tid;
      val = ((val >> 16) ^ val) * 0x45d9f3bu;
      val = ((val >> 16) ^ val) * 0x45d9f3bu;
      val = (val >> 16) ^ val;
      const bool filter = edges / nodes >= 4;
      const int x = filter && tid < ns ? a.eweight[val % (unsigned)edges] : INT_MAX;
      int rank = 0;
      for (int i = 0; i < ns; i++) {
        const int y = __shfl_sync(0xffffffffu, x, i);
        rank += y < x || (y == x && i < tid);
      }
      if (!filter) {
        if (tid == 0) {
          st->filtered = 0;
          st->threshold = INT_MAX;
        }
      } else if (tid < ns && rank == min(19, (int)(3.0 * nodes * ns / edges))) {
        st->filtered = 1;
        st->threshold = x;
      }
    }
    return;
  }
  const int S = 4096;
  for (int i = tid; i < S; i += blockDim.x) {
    const uint64_t r = ecl_mix64(0x5EED0000ull + (uint64_t)i);
    samp[i] = a.eweight[(unsigned)(r % (uint64_t)(unsigned)edges)];
  }
  __syncthreads();
  for (int k = 2; k <= S; k <<= 1) {  // bitonic sort in shared memory
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = tid; i < S; i += blockDim.x) {
        const int ixj = i ^ j;
        if (ixj > i) {
          const int x = samp[i], y = samp[ixj];
          if ((x > y) == ((i & k) == 0)) {
            samp[i] = y;
            samp[ixj] = x;
          }
        }
      }
      __syncthreads();
    }
  }
  if (tid == 0) {
    const float q = quantile < 0.f ? 0.f : quantile;
    int idx = (int)(q * (float)(S - 1));
    idx = idx < 0 ? 0 : (idx > S - 1 ? S - 1 : idx);
    st->filtered = 1;
    st->threshold = samp[idx];
  }
}

// The lists' split weights from k_prep's own sample of kThreads weights (one CTA): the sample
// of a wanted rank is the one with that many below it.
__device__ void choose_lists(const PrepArgs& a, int* samp) {
  DevState* st = a.st;
  const int tid = threadIdx.x;
  __syncthreads();
  const int thr = st->threshold, filtered = st->filtered;
  const uint64_t h = ecl_mix64(0xC1A55000ull + (uint64_t)tid);
  const int w = a.eweight[(unsigned)(h % (uint64_t)(unsigned)a.edges)];
  samp[tid] = w;
  const int light = __syncthreads_count(w <= thr);
  float r0, r1;
  split_ranks(a.nodes, a.edges, filtered, (float)light / kThreads, &r0, &r1);
  int below = 0;
  for (int i = 0; i < kThreads; i++) below += (unsigned)samp[i] < (unsigned)w || (samp[i] == w && i < tid);
  if (below == (int)(r0 * kThreads)) st->split_light = (unsigned)w;
  if (below == (int)(r1 * kThreads)) {
    st->split_heavy = (unsigned)w;
    st->mid = 1;
  }
  if (tid == 0 && r0 >= 1.f) st->split_light = 0xffffffffu;
}

__global__ void __launch_bounds__(kThreads) k_prep(PrepArgs a) {
  __shared__ int samp[4096];
  DevState* st = a.st;
  if (blockIdx.x == 0) {
    choose_threshold(a, samp);
    if (a.mode != ECL_THRESH_LEARNED) {
      if (a.use_lists) choose_lists(a, samp);
      else if (threadIdx.x == 0) st->split_light = 0xffffffffu;
    }
  }
  const int n = a.nodes, m = a.edges;
  const int gid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  bool bad = false;
  FeatPart fp;  // degree statistics (learned schedule)
  const int lane = threadIdx.x & 31;
  for (long long first = gid - lane; first < n; first += stride) {
    const int base = (int)first;
    const int v = first + lane < n ? base + lane : n;
    unsigned t0 = 0, t1 = 0;  // the table steps that start inside row v
    if (v < n) {
      a.parent[v] = v;
      a.minv0[v] = kNoEdge;
      if (a.both_slots) a.minv1[v] = kNoEdge;
      const int b = __ldg(a.nindex + v), e = __ldg(a.nindex + v + 1);
      const bool row_bad = b < 0 || e < b || e > m;
      bad |= row_bad;
      if (a.feat) fp.add(e > b ? (unsigned)(e - b) : 0u);
      if (!row_bad) {
        t0 = ((unsigned)b + kGran - 1) / kGran;
        t1 = ((unsigned)e + kGran - 1) / kGran;
      }
    }
    // Task->row table: every row writes itself at the steps it holds, a long
    // row with the whole warp.
    if (t1 - t0 <= 4)
      for (unsigned t = t0; t < t1; t++) a.first_v[t] = v;
    for (unsigned longs = __ballot_sync(0xffffffffu, t1 - t0 > 4); longs; longs &= longs - 1) {
      const int src = __ffs(longs) - 1;
      const unsigned f = __shfl_sync(0xffffffffu, t0, src), l = __shfl_sync(0xffffffffu, t1, src);
      for (unsigned t = f + lane; t < l; t += 32) a.first_v[t] = base + src;
    }
  }
  if (gid == 0) {
    a.first_v[a.tiles] = n - 1;
    bad |= __ldg(a.nindex) != 0 || __ldg(a.nindex + n) != m;
  }
  if (bad) atomicOr(&st->error, kErrFormat);
  if (a.feat) fp.fold<kThreads>(a.feat);  // uniform across the grid
}

enum ScanKind { kLight = 0, kHeavy = 1 };

// parent[v] = root(v) for every vertex, before a list of unmapped vertices and
// before the heavy scan, and a bit per vertex of the largest tree so far (a
// word per warp and 32 vertices). Four walks per thread run in lock step,
// their loads in flight together; they read through L1, where the few vertices
// near a giant tree's root stay (a value from before another thread's store is
// a lower ancestor of the same root, so a stale line only lengthens a walk).
__global__ void __launch_bounds__(kThreads) k_flatten(int* parent, int n, const DevState* st, unsigned* tree_bits,
                                                      int list) {
  constexpr int U = 4;
  if (list == kListHeavy ? !st->filtered : !st->lists[list].slots) return;  // nothing follows that reads it
  if (ld_volatile(&st->error) & (kErrFormat | kErrTimeout)) return;
  const int giant = st->giant, lane = threadIdx.x & 31;
  const int warps = gridDim.x * (kThreads / 32), w0 = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  for (long long base = (long long)w0 * (32 * U); base < n; base += (long long)warps * (32 * U)) {
    int v[U], first[U], p[U];
    bool walk[U];
#pragma unroll
    for (int i = 0; i < U; i++) {
      v[i] = (int)base + i * 32 + lane;
      walk[i] = base + i * 32 + lane < n;
      first[i] = p[i] = walk[i] ? __ldcg(parent + v[i]) : -1;
      walk[i] = walk[i] && p[i] != v[i];
    }
    for (bool any = true; any;) {
      any = false;
      int gp[U];
#pragma unroll
      for (int i = 0; i < U; i++) gp[i] = walk[i] ? ld_ca(parent + p[i]) : 0;
#pragma unroll
      for (int i = 0; i < U; i++)
        if (walk[i]) {
          if (gp[i] == p[i]) walk[i] = false;
          else any = true;
          p[i] = gp[i];
        }
    }
#pragma unroll
    for (int i = 0; i < U; i++) {
      if (p[i] >= 0 && p[i] != first[i]) __stcg(parent + v[i], p[i]);
      const unsigned word = __ballot_sync(0xffffffffu, p[i] == giant);
      if (lane == 0 && base + i * 32 < n) tree_bits[(base >> 5) + i] = word;
    }
  }
}

// ----------------------------------------------------------------- rounds
// Per-CTA shared-memory state of the round kernel. Representatives shared by
// many worklist entries (a growing giant component) would otherwise put
// every entry's parent read, min-slot guard read, atomicMin and reset on one
// L2 address; these small direct-mapped tables absorb the repeats per CTA.
struct RoundSmem {
  unsigned warp_off[32][2];  // the CTA's warp totals
  unsigned cursor;           // entries this CTA kept so far in the current find/min pass
  int seg_n;                 // segments of the list the passes read (1 = dense from seg_off[0])
  unsigned seg_q[kMaxRoundCtas + 1];  // entries in the segments before b (seg_q[seg_n] = all)
  unsigned seg_off[kMaxRoundCtas];    // first position of segment b
  int hot_rep[kHotSlots];    // hot representative -> CTA-local partial minimum
  u64 hot_key[kHotSlots];
  int reset_seen[kHotSlots]; // previous-round slots this CTA already cleared
  u64 find_cache[kFindSlots];// (vertex << 32) | root, valid within one pass
  u64 pair_tag[kPairSlots];  // (lo rep << 32) | hi rep of a tile's cross entry
  u64 pair_min[kPairSlots];  // smallest key of that rep pair within the tile
};

__device__ __forceinline__ unsigned hot_slot(int r) { return ((unsigned)r * 0x9E3779B1u) >> (32 - kHotLog); }
__device__ __forceinline__ unsigned find_slot(int r) { return ((unsigned)r * 0x85EBCA6Bu) >> (32 - kFindLog); }

__device__ __forceinline__ void round_smem_clear(RoundSmem& s) {
  if (threadIdx.x == 0) s.cursor = 0;
  for (int i = threadIdx.x; i < kHotSlots; i += blockDim.x) {
    s.hot_rep[i] = -1;
    s.hot_key[i] = kNoEdge;
    s.reset_seen[i] = -1;
  }
  for (int i = threadIdx.x; i < kFindSlots; i += blockDim.x) s.find_cache[i] = kNoEdge;
  for (int i = threadIdx.x; i < kPairSlots; i += blockDim.x) {
    s.pair_tag[i] = kNoPair;
    s.pair_min[i] = kNoEdge;
  }
}

__device__ __forceinline__ unsigned pair_slot(u64 pk) {
  return (unsigned)((pk * 0x9E3779B97F4A7C15ull) >> (64 - kPairLog));
}

// ---- segmented round worklists
// A find/min pass compacts its kept entries without any global reservation:
// the CTA that runs tile share b of the pass (tiles b, b + stride, ...) owns
// the output positions [region_b, region_b + share_b), where share_b counts
// the logical input entries of its tiles, and its warps take positions from a
// shared-memory cursor. The pass's output is therefore one dense segment per
// CTA (seg_cnt[b] kept entries from region_b). The next passes address that
// list by logical index through a prefix table of the segment counts, so a
// pass needs neither a global atomic per tile nor a CTA barrier per tile.

// The list read next is dense: entries [0, count) from position 0.
__device__ __forceinline__ void seg_set_dense(RoundSmem& s, unsigned count) {
  if (threadIdx.x == 0) {
    s.seg_n = 1;
    s.seg_off[0] = 0;
    s.seg_q[0] = 0;
    s.seg_q[1] = count;
  }
}

// The list read next is the one the grid's find/min pass just wrote (`nseg`
// segments, published in the control block before the grid barrier). The
// whole CTA builds the prefix table: thread t loads kSegPer consecutive
// segment counts, one warp scan and one pass over the warp totals give the
// prefixes. Every thread of the CTA must call this; the caller synchronises
// the CTA before the table is used.
constexpr int kSegPer = (kMaxRoundCtas + kRoundThreads - 1) / kRoundThreads;
__device__ __forceinline__ void seg_load(RoundSmem& s, const DevState* st, int nseg) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int b0 = kSegPer * t;
  unsigned c[kSegPer], mine = 0;
#pragma unroll
  for (int k = 0; k < kSegPer; k++) {
    const int b = b0 + k;
    c[k] = b < nseg ? __ldcg(&st->seg_cnt[b]) : 0u;
    if (b < nseg) s.seg_off[b] = __ldcg(&st->seg_off[b]);
    mine += c[k];
  }
  unsigned incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) s.warp_off[warp][0] = incl;
  __syncthreads();
  unsigned q = incl - mine;
  for (int w = 0; w < warp; w++) q += s.warp_off[w][0];
#pragma unroll
  for (int k = 0; k < kSegPer; k++) {
    const int b = b0 + k;
    if (b < nseg) s.seg_q[b] = q;
    q += c[k];
    if (b == nseg - 1) s.seg_q[nseg] = q;  // the thread holding the last segment
  }
  if (t == 0) s.seg_n = nseg;
}

// Position of logical entry i of the list described by the prefix table.
__device__ __forceinline__ unsigned seg_at(const RoundSmem& s, unsigned i) {
  const int nseg = s.seg_n;
  if (nseg == 1) return s.seg_off[0] + i;
  int lo = 0, hi = nseg;  // largest b with seg_q[b] <= i (seg_q[nseg] > i)
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (s.seg_q[mid] <= i) lo = mid;
    else hi = mid;
  }
  return s.seg_off[lo] + (i - s.seg_q[lo]);
}

// First output position of tile share `b` of a pass over W logical entries
// in tiles of `tile`, shares strided by `stride`: the logical entries of the
// tiles of all shares before b (the last tile may be partial).
__device__ __forceinline__ unsigned share_region(unsigned W, unsigned tile, unsigned b, unsigned stride) {
  const unsigned ntiles = (W + tile - 1) / tile;
  const unsigned q = ntiles / stride, rr = ntiles % stride;
  const unsigned long long full = (unsigned long long)tile * ((unsigned long long)q * b + min(b, rr));
  const unsigned last_owner = ntiles ? (ntiles - 1) % stride : 0u;
  const unsigned short_by = (unsigned)((unsigned long long)ntiles * tile - W);
  return (unsigned)(full - (ntiles && b > last_owner ? short_by : 0u));
}

// Parallel-edge elimination within a tile (opt-in through ECL_FLAG_DEDUP).
// Entries of one tile that join the same two trees are parallel edges of the
// contracted graph; only the one with the smallest (weight, j) key can be a
// forest edge (any forest through a heavier one is heavier than the same
// forest through the lightest), so the others may be dropped for good. Warp
// groups with equal rep pairs reduce first; group minima meet in a per-tile
// shared table. Measured on RMAT scale 22 the elimination costs more (two CTA
// barriers and the table per tile) than the smaller worklists save, so it is
// off by default. keep[k] is narrowed to the survivors. Every thread of the
// CTA must call this (it synchronises the CTA).
template <int E>
__device__ __forceinline__ void drop_parallel(const int4 (&e)[E], bool (&keep)[E], RoundSmem& s) {
  const int lane = threadIdx.x & 31;
  u64 pk[E], gmin[E];
#pragma unroll
  for (int k = 0; k < E; k++) {
    const unsigned lo = (unsigned)min(e[k].x, e[k].y), hi = (unsigned)max(e[k].x, e[k].y);
    pk[k] = keep[k] ? (((u64)lo << 32) | hi) : (0xFFFFFFFF00000000ull | (threadIdx.x * E + k));
    const u64 key = edge_key(e[k].z, e[k].w);
    gmin[k] = key;
    const unsigned g = __match_any_sync(0xffffffffu, pk[k]);
    if (!keep[k]) continue;
    if (g & (g - 1)) {
      const unsigned khi = (unsigned)(key >> 32);
      const unsigned mhi = __reduce_min_sync(g, khi);
      const unsigned mlo = __reduce_min_sync(g, khi == mhi ? (unsigned)key : 0xffffffffu);
      gmin[k] = ((u64)mhi << 32) | mlo;
    }
    if (lane == __ffs(g) - 1) {
      const unsigned slot = pair_slot(pk[k]);
      u64 t = ((volatile u64*)s.pair_tag)[slot];
      if (t == kNoPair) {
        t = atomicCAS(&s.pair_tag[slot], kNoPair, pk[k]);
        if (t == kNoPair) t = pk[k];
      }
      if (t == pk[k] && ((volatile u64*)s.pair_min)[slot] > gmin[k]) atomicMin(&s.pair_min[slot], gmin[k]);
    }
  }
  __syncthreads();  // the tile's pair table is complete
#pragma unroll
  for (int k = 0; k < E; k++) {
    if (keep[k]) {
      const unsigned slot = pair_slot(pk[k]);
      const u64 key = edge_key(e[k].z, e[k].w);
      const u64 best = s.pair_tag[slot] == pk[k] ? s.pair_min[slot] : gmin[k];
      keep[k] = key == best;
    }
  }
  __syncthreads();  // every check done before the table is cleared
  for (int i = threadIdx.x; i < kPairSlots; i += blockDim.x) {
    s.pair_tag[i] = kNoPair;
    s.pair_min[i] = kNoEdge;
  }
}

// Output positions for this thread's kept entries: one shared-memory atomic
// per warp on the CTA's cursor, no barrier. Returns the position of the
// thread's first kept entry (the rest follow) inside the CTA's segment that
// starts at `region`. Every lane of the warp must call this.
template <int E>
__device__ __forceinline__ unsigned warp_reserve(const bool (&keep)[E], RoundSmem& s, unsigned region) {
  const int lane = threadIdx.x & 31;
  unsigned cnt = 0;
#pragma unroll
  for (int k = 0; k < E; k++) cnt += keep[k];
  unsigned excl, total;
  if (E == 1) {
    const unsigned mask = __ballot_sync(0xffffffffu, cnt != 0);
    excl = __popc(mask & ((1u << lane) - 1u));
    total = __popc(mask);
  } else {
    unsigned incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    excl = incl - cnt;
    total = __shfl_sync(0xffffffffu, incl, 31);
  }
  unsigned base = 0;
  if (lane == 0 && total) base = atomicAdd(&s.cursor, total);
  base = __shfl_sync(0xffffffffu, base, 0);
  return region + base + excl;
}

// Roots of the 2*kEPT endpoints a thread holds, all walks advanced in lock
// step so their loads are in flight together. A per-CTA cache of
// (vertex << 32 | root) is consulted at every step (roots do not change
// during the find/min pass): after a walk it holds the start vertex, its
// parent and the root, so the nodes near the top of a large tree, which
// every walk through that tree would otherwise read from the same L2 lines,
// are read once per CTA. Hooking by random priority keeps trees shallow, so
// a walk only starts path splitting (re-pointing each visited node to its
// grandparent, which stays inside the tree) once it is kSplitAfter steps
// deep: the writes bound pathological chains, while splitting every walk
// would have the many walkers that share a start vertex all store to the
// same parent entries.
__device__ __forceinline__ int find_cached(const RoundSmem& s, int x) {
  const u64 c = ((const volatile u64*)s.find_cache)[find_slot(x)];
  return (int)(c >> 32) == x ? (int)(unsigned)c : -1;  // -1: not cached (x >= 0)
}

template <int N>
__device__ __forceinline__ void multi_find(int (&v)[N], const bool (&valid)[N], int* parent,
                                           RoundSmem& s, bool use_cache = true,
                                           int split_after = kSplitAfter) {
  int par[N], orig[N], first[N];  // first: the start vertex's parent
  unsigned miss = 0;
#pragma unroll
  for (int i = 0; i < N; i++) {
    orig[i] = v[i];
    par[i] = v[i];
    first[i] = v[i];
    if (!valid[i]) continue;
    const int r = use_cache ? find_cached(s, v[i]) : -1;
    if (r >= 0) {
      v[i] = par[i] = r;
    } else {
      miss |= 1u << i;
      par[i] = first[i] = __ldcg(parent + v[i]);
    }
  }
  for (int step = 0;; step++) {
    int gp[N];
    bool any = false;
#pragma unroll
    for (int i = 0; i < N; i++) {
      gp[i] = par[i];
      if (par[i] != v[i]) {
        const int r = use_cache ? find_cached(s, par[i]) : -1;
        if (r >= 0) {  // the rest of the walk is known
          v[i] = par[i] = gp[i] = r;
          continue;
        }
        any = true;
        gp[i] = __ldcg(parent + par[i]);
      }
    }
    if (!any) break;
#pragma unroll
    for (int i = 0; i < N; i++) {
      if (par[i] != v[i]) {
        if (step >= split_after && gp[i] != par[i]) __stcg(parent + v[i], gp[i]);
        v[i] = par[i];
        par[i] = gp[i];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < N; i++)
    if (use_cache && (miss & (1u << i))) {
      volatile u64* fc = (volatile u64*)s.find_cache;
      const u64 root = (unsigned)v[i];
      fc[find_slot(orig[i])] = ((u64)(unsigned)orig[i] << 32) | root;
      if (first[i] != v[i]) fc[find_slot(first[i])] = ((u64)(unsigned)first[i] << 32) | root;
      if (orig[i] != v[i]) fc[find_slot(v[i])] = (root << 32) | root;
    }
}

// How a find/min pass clears the previous round's min slots: not at all
// (first round), slot by slot for its entries' reps (deduplicated per CTA),
// or the whole array with coalesced stores when the entries outnumber the
// vertices enough that the scattered stores would cost more.
enum : int { kResetNone = 0, kResetSparse = 1, kResetDense = 2 };

// Clear a previous-round min slot once per CTA.
__device__ __forceinline__ void reset_prev(int r, u64* mprev, RoundSmem& s) {
  const unsigned slot = hot_slot(r);
  if (((volatile int*)s.reset_seen)[slot] == r) return;
  ((volatile int*)s.reset_seen)[slot] = r;
  __stcg(mprev + r, kNoEdge);
}

// Offer each of a thread's N (rep, key) pairs to the rep's min slot: the
// guarded atomicMin of ECL_MST.cu:221-223. Lanes of a warp holding the same
// rep first reduce to the group minimum (warp-cooperative for high-degree
// representatives); a group leader then folds it into the CTA's hot table.
// A lone entry of a rep already in the table folds into it as well, so a
// giant component's rep costs no global traffic. The rest (lone entries of
// other reps, leaders whose table slot belongs to another rep) read the
// global slots together (one round trip for all pairs) and issue
// fire-and-forget atomicMin only where the guard shows an improvement.
// Every lane of the warp must call this.
template <int N>
__device__ __forceinline__ void offer_mins(const int (&rep)[N], const u64 (&key)[N],
                                           const bool (&valid)[N], u64* mcur, RoundSmem& s,
                                           unsigned long long& atomics, bool coop = true,
                                           bool guard = true) {
  const int lane = threadIdx.x & 31;
  bool cold[N];
  u64 val[N];
#pragma unroll
  for (int i = 0; i < N; i++) {
    cold[i] = valid[i];
    val[i] = key[i];
    if (!coop) continue;  // uniform: every valid pair goes straight to its global slot
    cold[i] = false;
    const unsigned g = __match_any_sync(0xffffffffu, valid[i] ? rep[i] : -2 - lane);
    if (!valid[i]) continue;
    if ((g & (g - 1)) == 0) {
      // a lone entry of a rep already in the hot table folds into it too
      const unsigned slot = hot_slot(rep[i]);
      if (((volatile int*)s.hot_rep)[slot] == rep[i]) {
        if (((volatile u64*)s.hot_key)[slot] > key[i]) atomicMin(&s.hot_key[slot], key[i]);
      } else {
        cold[i] = true;
      }
      continue;
    }
    const unsigned khi = (unsigned)(key[i] >> 32);
    const unsigned hi = __reduce_min_sync(g, khi);
    const unsigned lo = __reduce_min_sync(g, khi == hi ? (unsigned)key[i] : 0xffffffffu);
    if (lane != __ffs(g) - 1) continue;
    const u64 gm = ((u64)hi << 32) | lo;
    const unsigned slot = hot_slot(rep[i]);
    int cur = ((volatile int*)s.hot_rep)[slot];
    if (cur < 0) {
      cur = atomicCAS(&s.hot_rep[slot], -1, rep[i]);
      if (cur < 0) cur = rep[i];
    }
    if (cur == rep[i]) {
      if (((volatile u64*)s.hot_key)[slot] > gm) atomicMin(&s.hot_key[slot], gm);
    } else {
      cold[i] = true;
      val[i] = gm;
    }
  }
  u64 seen[N];
#pragma unroll
  for (int i = 0; i < N; i++) seen[i] = cold[i] && guard ? __ldcg(mcur + rep[i]) : kNoEdge;
#pragma unroll
  for (int i = 0; i < N; i++) {
    if (cold[i] && seen[i] > val[i]) {
      atomicMin(mcur + rep[i], val[i]);
      atomics++;
    }
  }
}

// Worklist entry at position `pos`: a tuple {rep a, rep b, w, j}, or under
// kAblNoTuples a CSR index whose endpoints and weight are gathered (x = -1
// marks a null entry either way).
__device__ __forceinline__ int4 load_entry(const RoundArgs& a, const int4* list, unsigned pos) {
  if (a.abl & kAblNoTuples) {
    const int j = __ldcg(reinterpret_cast<const int*>(list) + pos);
    if (j < 0) return make_int4(-1, -1, 0, 0);
    return make_int4(__ldg(a.slist + j), __ldg(a.nlist + j), __ldg(a.eweight + j), j);
  }
  return __ldcg(list + pos);
}

__device__ __forceinline__ void store_entry(const RoundArgs& a, int4* list, unsigned pos, const int4& e) {
  if (a.abl & kAblNoTuples) reinterpret_cast<int*>(list)[pos] = e.w;
  else list[pos] = e;
}

// kernel1 (ECL_MST.cu:210-226) plus kernel3 of the previous round (:243-251):
// each input entry clears its endpoints' slots in the previous round's min
// array, resolves its endpoints to reps, and if they differ is compacted into
// `out` with the reps (implicit path compression, :218-219) and offers its
// key to both reps' min slots. The input is the list the prefix table in `s`
// describes (W logical entries); the kept entries go to this CTA's segment of
// `out` (share `start` of `stride`), whose size is left in s.cursor and
// added to *out_ctr and *kept_ctr.
//
// `fresh` marks the first round of a phase: its entries come straight from
// the scan, so both endpoints are roots (parent[v] = v before the light
// phase, the flattened light-tree roots before the heavy one) and differ.
// That round needs no find and keeps every entry: it only offers keys, and
// the scan's list serves as its output unchanged (no copy).
__device__ __forceinline__ void round_find_min(const RoundArgs& a, const int4* in, unsigned W,
                                               int4* out, unsigned* out_ctr, unsigned* kept_ctr,
                                               u64* mcur, u64* mprev, int reset, bool fresh,
                                               unsigned start, unsigned stride, RoundSmem& s,
                                               bool flat = false) {
  constexpr int N = 2 * kEPT;
  const unsigned tile = blockDim.x * kEPT;
  const unsigned ntiles = (W + tile - 1) / tile;
  const unsigned region = share_region(W, tile, start, stride);
  const bool dedup = (a.abl & kDedup) != 0;
  const bool keep_ends = (a.abl & kAblKeepEnds) != 0;  // entries are not rewritten to reps
  const bool count_only = (a.abl & kAblNoDD) != 0;     // nothing is compacted
  unsigned long long atomics = 0;
  if (reset == kResetDense)  // every slot of the previous round's array, coalesced
    for (unsigned i = start * blockDim.x + threadIdx.x; i < (unsigned)a.nodes; i += stride * blockDim.x)
      __stcg(mprev + i, kNoEdge);
  for (unsigned t = start; t < ntiles; t += stride) {
    int4 e[kEPT];
    bool in_range[kEPT];
#pragma unroll
    for (int k = 0; k < kEPT; k++) {
      const unsigned idx = t * tile + k * blockDim.x + threadIdx.x;
      in_range[k] = idx < W;
      e[k] = in_range[k] ? load_entry(a, in, seg_at(s, idx)) : make_int4(0, 0, 0, 0);
      if (e[k].x < 0) in_range[k] = false;  // null entry (unused scan slot)
    }
    int4 orig[kEPT];
#pragma unroll
    for (int k = 0; k < kEPT; k++) orig[k] = e[k];
    int v[N];
    bool vv[N];
#pragma unroll
    for (int k = 0; k < kEPT; k++) {
      v[2 * k] = e[k].x;
      v[2 * k + 1] = e[k].y;
      vv[2 * k] = vv[2 * k + 1] = in_range[k];
      if (reset == kResetSparse && in_range[k]) {
        reset_prev(e[k].x, mprev, s);
        reset_prev(e[k].y, mprev, s);
      }
    }
    bool keep[kEPT];
    if (fresh) {
#pragma unroll
      for (int k = 0; k < kEPT; k++) keep[k] = in_range[k];
    } else {
      if (flat) {  // parent[] was just flattened: one load names the root
#pragma unroll
        for (int i = 0; i < N; i++) v[i] = vv[i] ? __ldcg(a.parent + v[i]) : v[i];
      } else {
        multi_find<N>(v, vv, a.parent, s, !(a.abl & kAblNoFindCache), keep_ends ? 0 : kSplitAfter);
      }
#pragma unroll
      for (int k = 0; k < kEPT; k++) {
        keep[k] = in_range[k] && v[2 * k] != v[2 * k + 1];
        e[k].x = v[2 * k];
        e[k].y = v[2 * k + 1];
      }
      if (dedup) drop_parallel<kEPT>(e, keep, s);  // uniform across the CTA
      unsigned pos = warp_reserve<kEPT>(keep, s, region);
      if (!count_only) {
#pragma unroll
        for (int k = 0; k < kEPT; k++) {
          if (keep[k]) {
            if (pos < a.wl_cap) store_entry(a, out, pos, keep_ends ? orig[k] : e[k]);
            else atomicOr(&a.st->error, kErrOverflow);
            pos++;
          }
        }
      }
    }
    u64 key[N];
    bool kv[N];
#pragma unroll
    for (int k = 0; k < kEPT; k++) {
      key[2 * k] = key[2 * k + 1] = edge_key(e[k].z, e[k].w);
      kv[2 * k] = kv[2 * k + 1] = keep[k];
    }
    offer_mins<N>(v, key, kv, mcur, s, atomics, !(a.abl & kAblNoCoop), !(a.abl & kAblNoGuards));
  }
  __syncthreads();
  if (threadIdx.x == 0 && s.cursor) {
    atomicAdd(out_ctr, s.cursor);
    atomicAdd(kept_ctr, s.cursor);
  }
  // flush the CTA's partial minima of hot representatives
  for (int i = threadIdx.x; i < kHotSlots; i += blockDim.x) {
    const int r = s.hot_rep[i];
    if (r >= 0) {
      const u64 k = s.hot_key[i];
      if ((a.abl & kAblNoGuards) || __ldcg(mcur + r) > k) {
        atomicMin(mcur + r, k);
        atomics++;
      }
    }
  }
  if (a.count_atomics && atomics) atomicAdd(&a.st->atomics, atomics);
}

// After the barrier: the hot table's reps now read their final minima.
__device__ __forceinline__ void hot_refresh(const u64* mcur, RoundSmem& s) {
  for (int i = threadIdx.x; i < kHotSlots; i += blockDim.x) {
    const int r = s.hot_rep[i];
    if (r >= 0) s.hot_key[i] = __ldcg(mcur + r);
  }
  __syncthreads();
}

// kernel2 (ECL_MST.cu:229-240): an entry whose key is the minimum of either
// endpoint's slot is a forest edge: union the trees and mark inMST[j]. The
// list is the one the prefix table in `s` describes (W logical entries).
__device__ __forceinline__ void round_mark(const RoundArgs& a, const int4* wl, unsigned W,
                                           const u64* mcur, unsigned start, unsigned stride,
                                           RoundSmem& s) {
  constexpr int N = 2 * kEPT;
  const unsigned tile = blockDim.x * kEPT;
  const unsigned ntiles = (W + tile - 1) / tile;
  const bool keep_ends = (a.abl & kAblKeepEnds) != 0;
  for (unsigned t = start; t < ntiles; t += stride) {
    int4 e[kEPT];
    bool in_range[kEPT];
#pragma unroll
    for (int k = 0; k < kEPT; k++) {
      const unsigned idx = t * tile + k * blockDim.x + threadIdx.x;
      in_range[k] = idx < W;
      e[k] = in_range[k] ? load_entry(a, wl, seg_at(s, idx)) : make_int4(0, 0, 0, 0);
      if (e[k].x < 0) in_range[k] = false;  // null entry (unused scan slot)
    }
    if (keep_ends) {
      // Entries hold their endpoints, not reps: find them again. Unions of
      // this pass may already have moved a root; a key then meets the slot of
      // the tree it joined, which can only defer an edge to a later round:
      // every edge marked is still the lightest edge leaving a tree of the
      // find/min pass (the reference's kernel2 finds the same way, :198-216).
      int v[N];
      bool vv[N];
#pragma unroll
      for (int k = 0; k < kEPT; k++) {
        v[2 * k] = e[k].x;
        v[2 * k + 1] = e[k].y;
        vv[2 * k] = vv[2 * k + 1] = in_range[k];
      }
      multi_find<N>(v, vv, a.parent, s, false, 0);
#pragma unroll
      for (int k = 0; k < kEPT; k++) {
        e[k].x = v[2 * k];
        e[k].y = v[2 * k + 1];
        if (e[k].x == e[k].y) in_range[k] = false;
      }
    }
    u64 mx[kEPT], my[kEPT];
#pragma unroll
    for (int k = 0; k < kEPT; k++) {
      mx[k] = my[k] = kNoEdge;
      if (!in_range[k]) continue;
      const unsigned sx = hot_slot(e[k].x), sy = hot_slot(e[k].y);
      mx[k] = s.hot_rep[sx] == e[k].x ? s.hot_key[sx] : __ldcg(mcur + e[k].x);
      my[k] = s.hot_rep[sy] == e[k].y ? s.hot_key[sy] : __ldcg(mcur + e[k].y);
    }
#pragma unroll
    for (int k = 0; k < kEPT; k++) {
      if (!in_range[k]) continue;
      const u64 key = edge_key(e[k].z, e[k].w);
      if (key == mx[k] || key == my[k]) {
        cas_union(e[k].x, e[k].y, a.parent);
        a.inMST[e[k].w] = 1;
      }
    }
  }
}

__global__ void __launch_bounds__(kRoundThreads, ECL_ROUND_MIN_BLOCKS) k_rounds(RoundArgs a) {
  __shared__ RoundSmem s;
  DevState* st = a.st;
  const int ph = a.phase;
  if (ph == 1 && !st->filtered) return;
  // Only bits no CTA of this kernel can set, so every CTA takes the same exit.
  if (ld_volatile(&st->error) & (kErrFormat | kErrTimeout)) return;
  round_smem_clear(s);
  seg_set_dense(s, 0);  // round 0 reads the scan's list as it is
  __syncthreads();
  unsigned active = gridDim.x;  // CTAs still in the launch
  bool tail = active == 1;      // one CTA: CTA barriers stand for the grid's
  int r = 0;
  const bool stamp = blockIdx.x == 0 && threadIdx.x == 0;
  // Round 0 offers straight from the scan's list, whose endpoints are roots
  // (not so under kAblNoTuples: those lists hold CSR indices, whose
  // endpoints are gathered as they are).
  const bool fresh0 = !(a.abl & kAblNoTuples);
  const bool ndd = (a.abl & kAblNoDD) != 0;
  const ListCount list = st->lists[ph == 0 ? kListLight0 : kListHeavy];
  const unsigned first = min(list.slots, a.wl_cap);
  if (stamp) {
    st->t_round_start[ph] = globaltimer_ns();
    st->wl_count[ph][0] = first;
    st->wl_kept[ph][0] = list.kept;
  }
  for (;;) {
    unsigned W = r == 0 ? first : min(ld_volatile(&st->wl_count[ph][r]), a.wl_cap);
    if (W == 0) break;  // (kAblNoDD: no entry joined two trees last round)
    if (ndd) W = first;  // the phase's whole list, every round
    if (r >= ECL_MAX_ROUNDS) {
      if (stamp) atomicOr(&st->error, kErrRounds);
      break;
    }
    // CTAs the round keeps: one per min_tiles tiles of its worklist (the
    // rest leave for good; worklists never grow), or one CTA alone at the
    // small tail, which then syncs with CTA barriers only
    unsigned want = active;
    if (a.min_tiles > 0) {
      const unsigned per = (unsigned)a.min_tiles * blockDim.x * kEPT;
      want = min(want, max(1u, (W + per - 1) / per));
    }
    if (W <= a.small_tail) want = 1;
    if (want < active) {
      active = want;
      if (blockIdx.x >= active) return;
      tail = active == 1;
    }
    const unsigned start = blockIdx.x, stride = active;
    // A fresh round 0 reads the scan's list (wl0) and keeps it as its
    // output; the compacting rounds after it alternate between the lists.
    // The min-slot arrays alternate per round.
    const bool fresh = fresh0 && r == 0;
    const int k = fresh0 ? r - 1 : r;  // index among the compacting rounds
    const bool in1 = !fresh && !ndd && (k & 1) != 0;
    const int4* in = in1 ? a.wl1 : a.wl0;
    int4* out = in1 ? a.wl0 : a.wl1;
    const bool odd = (r & 1) != 0;
    u64* mcur = odd ? a.minv1 : a.minv0;
    u64* mprev = odd ? a.minv0 : a.minv1;
    // entries that keep their endpoints cannot name the previous round's
    // reps: those rounds clear the whole previous array
    const bool dense = (a.abl & kAblKeepEnds) || (!tail && 4ull * W >= (unsigned long long)a.nodes);
    const int reset = r == 0 ? kResetNone : (dense ? kResetDense : kResetSparse);
    // A round whose entries outnumber the vertices ECL_FLAT_ROUNDS times first
    // points every vertex at its root (one grid-stride pass; roots do not
    // change between passes), so each of its finds is a single load.
    const bool flat = ECL_FLAT_ROUNDS > 0 && !fresh && !tail && !(a.abl & kAblKeepEnds) &&
                      (unsigned long long)W >= (unsigned long long)ECL_FLAT_ROUNDS * (unsigned)a.nodes;
    if (flat) {
      for (int v = (int)(start * blockDim.x + threadIdx.x); v < a.nodes; v += (int)(stride * blockDim.x)) {
        const int rt = find_ro(v, a.parent);
        if (rt != v) __stcg(a.parent + v, rt);
      }
      if (!grid_barrier(st, kBarrierTimeoutNs, active)) return;
    }
    round_find_min(a, in, W, out, &st->wl_count[ph][r + 1], &st->wl_kept[ph][r + 1], mcur, mprev, reset,
                   fresh, start, stride, s, flat);
    if (fresh && blockIdx.x == 0 && threadIdx.x == 0) {  // the scan's list is round 0's output
      st->wl_count[ph][1] = W;
      st->wl_kept[ph][1] = list.kept;
    }
    if (!fresh && !tail && !ndd && threadIdx.x == 0) {  // this CTA's segment of the output list
      st->seg_cnt[blockIdx.x] = s.cursor;
      st->seg_off[blockIdx.x] = share_region(W, blockDim.x * kEPT, start, stride);
    }
    if (tail) __syncthreads();
    else if (!grid_barrier(st, kBarrierTimeoutNs, active)) return;
    if (stamp) st->t_round[ph][2 * r] = globaltimer_ns();
    const unsigned W2 = min(ld_volatile(&st->wl_count[ph][r + 1]), a.wl_cap);
    r++;
    if (W2 == 0) break;
    // the list the mark pass and the next round read: the scan's list (round
    // 0), the tail CTA's single segment, or the grid's per-CTA segments
    if (!fresh && !ndd) {
      if (tail) seg_set_dense(s, s.cursor);
      else seg_load(s, st, (int)active);
    }
    hot_refresh(mcur, s);
    round_mark(a, fresh || ndd ? in : out, ndd ? W : W2, mcur, start, stride, s);
    __syncthreads();
    round_smem_clear(s);
    if (tail) __syncthreads();
    else if (!grid_barrier(st, kBarrierTimeoutNs, active)) return;
    if (stamp) st->t_round[ph][2 * r - 1] = globaltimer_ns();
  }
  if (stamp) st->rounds[ph] = r;
}

// ------------------------------------------------ reference ablation steps
// kAblNoTuples: the vertex of every CSR entry (the reference's NoTuples
// variant keeps such an slist, Deoptimizations/..._NoTuples.cu:163-169),
// filled entry-parallel: a binary search in nindex between the rows the
// scans' task->row table gives.
__global__ void __launch_bounds__(kThreads) k_slist(const int* nindex, const int* first_v, int* slist,
                                                    int edges, const DevState* st) {
  if (ld_volatile(&st->error) & kErrFormat) return;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < edges; j += gridDim.x * blockDim.x) {
    int lo = __ldg(first_v + j / kGran), hi = __ldg(first_v + j / kGran + 1);
    while (lo < hi) {  // the last row starting at or before j
      const int mid = lo + ((hi - lo + 1) >> 1);
      if (__ldg(nindex + mid) <= j) lo = mid;
      else hi = mid - 1;
    }
    slist[j] = lo;
  }
}

// NoEdgeBased (Deoptimizations/..._NoEdgeBased.cu:152-195): all Boruvka
// rounds of a phase as vertex-centric passes over the CSR, one thread per
// vertex walking its row, in one cooperative launch: (A) every one-direction
// entry of the phase's weight class whose endpoints lie in different trees
// offers its key to both roots, (B) an entry holding the minimum of either
// root's slot joins the trees and is marked, (C) the slots are cleared. The
// rounds end when pass A finds no entry across two trees (the reference's
// go_again). Pass B finds while other threads join; an entry it marks is
// still the lightest edge leaving a tree of pass A, so the forest is the
// reference's (an edge missed in one round is found in a later one).
__global__ void __launch_bounds__(kRoundThreads, ECL_ROUND_MIN_BLOCKS) k_rounds_vertex(RoundArgs a,
                                                                                       const int* nindex) {
  DevState* st = a.st;
  const int ph = a.phase;
  if (ph == 1 && !st->filtered) return;
  if (ld_volatile(&st->error) & (kErrFormat | kErrTimeout)) return;
  const int n = a.nodes, thr = st->threshold;
  const bool filtered = st->filtered != 0, guard = !(a.abl & kAblNoGuards);
  const int gid = blockIdx.x * blockDim.x + threadIdx.x, gstride = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  u64* mv = a.minv0;
  const bool stamp = blockIdx.x == 0 && threadIdx.x == 0;
  if (stamp) st->t_round_start[ph] = globaltimer_ns();
  auto in_phase = [&](int w) { return !filtered || (ph == 0 ? w <= thr : w > thr); };
  int r = 0;
  for (;; r++) {
    if (r >= ECL_MAX_ROUNDS) {
      if (stamp) atomicOr(&st->error, kErrRounds);
      break;
    }
    unsigned live = 0;
    for (int v = gid; v < n; v += gstride) {  // pass A
      const int beg = __ldg(nindex + v), end = __ldg(nindex + v + 1);
      int rv = -1;
      for (int j = beg; j < end; j++) {
        const int nb = __ldg(a.nlist + j);
        if (nb <= v) continue;  // one direction
        const int w = __ldg(a.eweight + j);
        if (!in_phase(w)) continue;
        if (rv < 0) rv = find_halve(v, a.parent);
        const int rn = find_halve(nb, a.parent);
        if (rv == rn) continue;
        live++;
        const u64 key = edge_key(w, j);
        if (!guard || __ldcg(mv + rv) > key) atomicMin(mv + rv, key);
        if (!guard || __ldcg(mv + rn) > key) atomicMin(mv + rn, key);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) live += __shfl_xor_sync(0xffffffffu, live, o);
    if (lane == 0 && live) atomicAdd(&st->wl_count[ph][r + 1], live);
    if (!grid_barrier(st, kBarrierTimeoutNs, gridDim.x)) return;
    if (stamp) st->t_round[ph][2 * r] = globaltimer_ns();
    if (ld_volatile(&st->wl_count[ph][r + 1]) == 0) break;
    for (int v = gid; v < n; v += gstride) {  // pass B
      const int beg = __ldg(nindex + v), end = __ldg(nindex + v + 1);
      for (int j = beg; j < end; j++) {
        const int nb = __ldg(a.nlist + j);
        if (nb <= v) continue;
        const int w = __ldg(a.eweight + j);
        if (!in_phase(w)) continue;
        const int rv = find_ro(v, a.parent), rn = find_ro(nb, a.parent);
        if (rv == rn) continue;
        const u64 key = edge_key(w, j);
        if (key == __ldcg(mv + rv) || key == __ldcg(mv + rn)) {
          cas_union(rv, rn, a.parent);
          a.inMST[j] = 1;
        }
      }
    }
    if (!grid_barrier(st, kBarrierTimeoutNs, gridDim.x)) return;
    for (int v = gid; v < n; v += gstride) __stcg(mv + v, kNoEdge);  // pass C
    if (!grid_barrier(st, kBarrierTimeoutNs, gridDim.x)) return;
    if (stamp) st->t_round[ph][2 * r + 1] = globaltimer_ns();
  }
  if (stamp) {
    st->rounds[ph] = r;
    st->wl_count[ph][0] = st->wl_count[ph][1];
  }
}

}  // namespace ecl
