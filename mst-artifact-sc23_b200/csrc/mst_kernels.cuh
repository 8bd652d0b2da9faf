// Device building blocks of the B200 ECL-MST engine: coherent loads, the
// bounded grid barrier, bulk copies, find with path halving and the CAS union.
// Shared by the single-graph engine (ecl_mst.cu) and the batched engine.
#pragma once
#include <cuda_runtime.h>
#include <climits>
#include <stdint.h>

#include "ecl_mst.h"

namespace ecl {

typedef unsigned long long u64;

// Device error word bits (DevState::error).
enum : unsigned {
  kErrFormat = 1u,    // nindex not monotone / out of range, or nlist id >= nodes
  kErrOverflow = 2u,  // a worklist or descriptor buffer ran out of room
  kErrTimeout = 4u,   // a grid barrier waited past its limit
  kErrRounds = 8u,    // more Boruvka rounds than ECL_MAX_ROUNDS
  kErrIds = 16u       // nlist id out of range, found by a group's scan (k_group): a bit of
                      // its own, as the group leaves together on kErrFormat
};

// Most CTAs a round-kernel launch may have: each CTA of a find/min pass
// writes its kept entries as one segment of the round's output list.
constexpr int kMaxRoundCtas = 1024;

constexpr u64 kNoEdge = ~0ull;

// Degree statistics of the learned schedule's features, summed over all
// vertices (row degree = nindex[v + 1] - nindex[v]).
struct FeatAcc {
  unsigned long long deg_sum, deg_sq, zero, low, high;  // sum d, sum d^2, #d = 0, #d < 4, #d >= 32
  unsigned max_deg;
};

// One thread's part of the degree statistics.
struct FeatPart {
  unsigned long long d1 = 0, d2 = 0, z = 0, lo = 0, hi = 0;
  unsigned mx = 0;
  __device__ __forceinline__ void add(unsigned d) {
    d1 += d;
    d2 += (unsigned long long)d * d;
    z += d == 0;
    lo += d < 4;
    hi += d >= 32;
    mx = max(mx, d);
  }
  // Fold the CTA's parts into `acc`: warp shuffles, one shared-memory pass,
  // one atomic per counter per CTA. Every thread of the CTA (kBlock threads)
  // must call this.
  template <int kBlock>
  __device__ __forceinline__ void fold(FeatAcc* acc) {
    __shared__ unsigned long long part[5][kBlock / 32];
    __shared__ unsigned pmax[kBlock / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      d1 += __shfl_down_sync(0xffffffffu, d1, o);
      d2 += __shfl_down_sync(0xffffffffu, d2, o);
      z += __shfl_down_sync(0xffffffffu, z, o);
      lo += __shfl_down_sync(0xffffffffu, lo, o);
      hi += __shfl_down_sync(0xffffffffu, hi, o);
      mx = max(mx, __shfl_down_sync(0xffffffffu, mx, o));
    }
    if (lane == 0) {
      part[0][w] = d1;
      part[1][w] = d2;
      part[2][w] = z;
      part[3][w] = lo;
      part[4][w] = hi;
      pmax[w] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int i = 1; i < kBlock / 32; i++) {
        for (int k = 0; k < 5; k++) part[k][0] += part[k][i];
        pmax[0] = max(pmax[0], pmax[i]);
      }
      atomicAdd(&acc->deg_sum, part[0][0]);
      atomicAdd(&acc->deg_sq, part[1][0]);
      atomicAdd(&acc->zero, part[2][0]);
      atomicAdd(&acc->low, part[3][0]);
      atomicAdd(&acc->high, part[4][0]);
      atomicMax(&acc->max_deg, pmax[0]);
    }
  }
};

// The state a phase's rounds are in at the top of a round (kept in the control
// block where the cluster kernel takes over from the grid).
struct BorState {
  unsigned W;  // entries of the list read next
  unsigned C;  // live roots (0 before the first roots pass)
  int r;       // round
  int k;       // compactions so far
  int nseg;    // segments of the list (0 = dense)
  int flips;   // roots passes so far
  int first;   // no offer pass yet
  int skip;    // the tree that offers nothing, -1 = none
};

// One graph of a batch: where its rows and entries start in the batch's arrays.
struct GraphDesc {
  long long nindex_off, edge_off;
  int nodes, edges;
};

// The learned schedule's choice for one graph of a batch.
struct LearnedChoice {
  int threshold, filtered;
};

// The worklists a solve's scans build, in the order their rounds run. The light
// phase's entries may be split by weight into two lists, and the light scan may
// set aside the lightest of the heavy phase's: rounds on a short list of the
// lightest entries first leave most of the later ones inside one tree. Each
// list holds the smaller weights of its phase as unsigned, so the forest is the
// phase's. Lists 1 and 2 grow down from the end of the two arrays, beside the
// space the rounds before them compact into:
//   wl0:  [light 0, then heavy ...      ... light 1]
//   wl1:  [                             ...     mid]
enum : int { kListLight0 = 0, kListLight1 = 1, kListMid = 2, kListHeavy = 3 };
struct ListCount {
  unsigned slots, kept;  // slots reserved (null padding included), entries
};

// Times (globaltimer) of a solve in one launch, which has no events between its
// steps: its start, and the ends of prep and flatten (the scans end where
// t_round_start is, the rounds with the last offer pass).
enum : int { kStepStart = 0, kStepPrep, kStepFlatten, kSteps };

// Control block of one solve, zeroed before every solve.
struct alignas(128) DevState {
  int threshold;       // light phase keeps w <= threshold
  int filtered;        // 1 = light + heavy phase, 0 = one unfiltered phase
  int split;           // degree split asked for or learned (only reported: the scans need none)
  unsigned error;      // kErr* bits
  unsigned bar_count;  // grid barrier: CTAs arrived in the current generation
  unsigned bar_gen;    // grid barrier: generation counter
  int rounds[2];       // Boruvka rounds per phase
  float quantile;      // learned / quantile modes: filter quantile in [0,1]
  u64 atomics;         // guarded atomicMin issued (stats mode)
  unsigned wl_count[2][ECL_MAX_ROUNDS + 1];  // [phase][r] = entries entering round r
  // globaltimer stamps taken by CTA 0 at phase boundaries (diagnostics):
  // [phase][2r] after round r's find/min pass, [phase][2r+1] after its mark pass
  u64 t_round_start[2];
  u64 t_round[2][2 * ECL_MAX_ROUNDS];
  u64 t_step[kSteps];  // solves in one launch: ends of their steps (kStepStart ...)
  u64 t_list[4];       // separate launches: start of a list's rounds (0 = none)
  int r_list[4];       // and the phase's round it is
  ListCount lists[4];
  unsigned split_light;  // light entries up to this weight (as unsigned) go to list light 0
  unsigned split_heavy;  // heavy entries up to this weight go to list mid, if
  int mid;               // that list is used
  int lists_bad;         // the lists of one array overlap (more entries than it holds)
  unsigned wl_kept[2][ECL_MAX_ROUNDS + 1];  // [phase][r] = entries entering round r (no padding)
  // The last find/min pass's output list, one segment per CTA: CTA b wrote
  // seg_cnt[b] entries from position seg_off[b] (written before the grid
  // barrier that ends the pass, read after it).
  unsigned seg_cnt[kMaxRoundCtas];
  unsigned seg_off[kMaxRoundCtas];
  unsigned root_cnt[4][3];  // [list][pass % 3] = live roots a roots pass kept
  BorState resume;          // where the cluster kernel goes on with the phase
  unsigned bar[4];          // GridSync: k_round's counters by list; k_group's counter and gate
  unsigned graph;           // batch: the graph the cluster works on
  int giant;                // the light phase's largest tree (by a vote of sampled vertices)
};

// Weights at which a solve's lists are split (kListLight0 ...), as the shares
// of the graph's entries at or below them (2 = no split).
//   Light entries: the first kSplitLight x n go to list light 0, the others to
// light 1, if these are half as many at least and all of them kSplitMin. The
// rounds on half an entry per vertex leave few trees for the others, which then
// drop out at their first look; but the short list's last rounds cost their
// latency, 100-150 us (ER 3M, 4.4M light entries: 0.99 ms against 1.06, 1.21 at
// 0.25 x n; RMAT-18 unfiltered, 3.8M: 0.38 against 0.50; ER 1.2M, 1.7M: 0.66
// against 0.57).
//   Beyond L2 (kMidNodes) an entry dropped early saves more: kSplitLightFar
// (ER 16M 7.21 ms against 7.68, RMAT-25 the same; in L2, RMAT-22 1.42 ms against
// 1.36).
//   Heavy entries: list mid takes them up to kSplitHeavy x n entries in all,
// where the slots and parents of the vertices outgrow L2, so that every entry
// the heavy scan keeps costs DRAM accesses (ER 16M 7.7 ms against 8.9, RMAT-25
// 10.8 against 11.7; RMAT-22, in L2, 1.55 against 1.52).
//   The line kMidNodes, times below and beyond it without and with what it
// switches on: random graphs gain on both sides (degree 16, 7M vertices at the
// 10 % quantile 2.94 and 2.22 ms, 9M 3.43 and 2.83, 12M 5.22 and 3.79, 16M 7.36 and
// 5.34; degree 32 2.83 and 2.83, 3.61 and 3.78, 5.10 and 4.82, 8.28 and 6.87), power-law
// graphs lose on both (RMAT-22 1.40 and 1.53, RMAT-23 2.52 and 3.00, RMAT-24 5.37 and
// 5.77, heuristic; learned the same within 1.3 %). It lies where 20 bytes per
// vertex pass L2's 126 MB.
constexpr float kSplitLight = 0.5f, kSplitLightFar = 0.8f, kSplitHeavy = 2.0f;
constexpr int kSplitMin = 3 << 20;
constexpr int kMidNodes = 1 << 23;
__device__ __forceinline__ void split_ranks(int n, int m, int filtered, float light_share, float* rank0, float* rank1) {
  const float half = 0.5f * (float)m;
  const float f0 = (n >= kMidNodes ? kSplitLightFar : kSplitLight) * (float)n / half;
  const float f1 = kSplitHeavy * (float)n / half;
  *rank0 = f0 * 1.5f < light_share && light_share * half >= (float)kSplitMin ? f0 : 2.f;
  *rank1 = filtered && n >= kMidNodes && f1 > 1.3f * light_share && f1 <= 0.4f ? f1 : 2.f;
}

__device__ __forceinline__ u64 globaltimer_ns() {
  u64 t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned ld_volatile(const unsigned* p) {
  return *(const volatile unsigned*)p;
}

// Grid-wide barrier for cooperative launches among the `expected` CTAs
// still in the launch (the others have left for good). Every wait is bounded
// by `timeout_ns`; on expiry the kErrTimeout bit is set and all later
// barriers return at once, so a stuck CTA turns into an error status instead
// of a hang. Returns false once the timeout bit is set.
__device__ __forceinline__ bool grid_barrier(DevState* st, u64 timeout_ns, unsigned expected) {
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned gen = ld_volatile(&st->bar_gen);
    __threadfence();
    const unsigned arrived = atomicAdd(&st->bar_count, 1u);
    if (arrived == expected - 1) {
      atomicExch(&st->bar_count, 0u);
      __threadfence();
      atomicAdd(&st->bar_gen, 1u);
    } else {
      const u64 t0 = globaltimer_ns();
      unsigned ns = 32;
      while (ld_volatile(&st->bar_gen) == gen) {
        if (ld_volatile(&st->error) & kErrTimeout) break;
        if (globaltimer_ns() - t0 > timeout_ns) {
          atomicOr(&st->error, kErrTimeout);
          break;
        }
        __nanosleep(ns);
        if (ns < 256) ns <<= 1;
      }
    }
    __threadfence();
  }
  __syncthreads();
  return (ld_volatile(&st->error) & kErrTimeout) == 0;
}

// 32-bit global load through L1, for data that no CTA writes between two
// barriers (or where an older value will do).
__device__ __forceinline__ int ld_ca(const int* p) {
  int v;
  asm volatile("ld.global.ca.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// The last of the rows lo .. hi that starts at or before entry j: first(r) is
// row r's first entry, and row lo does.
template <class First>
__device__ __forceinline__ int last_row(First first, int lo, int hi, int j) {
  while (lo < hi) {
    const int mid = lo + ((hi - lo + 1) >> 1);
    if (first(mid) <= j) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// On from row v, whose entries end at `end`, to the row of entry j, which is at
// most `top`. A few rows are looked at one by one. A longer run is one of empty
// rows, of any length, and is bisected (last(lo, hi)): a million isolated
// vertices between two entries of a thread, walked row by row, took 50 ms a scan.
constexpr int kRowSteps = 4;
template <class First, class Last>
__device__ __forceinline__ void row_on(First first, Last last, int top, int j, int& v, int& end) {
  for (int k = 0; j >= end && v < top; k++) {
    if (k == kRowSteps) v = last(v + 1, top) - 1;  // row v + 1 starts at `end`
    v++;
    end = v < top ? first(v + 1) : INT_MAX;
  }
}
// ---- mbarriers and bulk asynchronous copies (cp.async.bulk, no multicast)
__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(u64* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

// Makes barrier initialisation visible to the asynchronous copy unit.
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Arrive and add `bytes` to the transaction count the phase waits for.
__device__ __forceinline__ void mbar_arrive_tx(u64* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}

// Test for the phase's completion; if it is not complete the thread is
// suspended until it completes or about 20 us pass (no busy spinning).
__device__ __forceinline__ bool mbar_try_wait(u64* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity), "r"(20000u)
      : "memory");
  return ok != 0;
}

// Wait for the phase of the given parity to complete, for at most
// `timeout_ns`; false on expiry.
__device__ __forceinline__ bool mbar_wait(u64* bar, unsigned parity, u64 timeout_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const u64 t0 = globaltimer_ns();
  while (!mbar_try_wait(bar, parity))
    if (globaltimer_ns() - t0 > timeout_ns) return false;
  return true;
}

// Orders this thread's generic-proxy shared-memory accesses before later
// asynchronous-proxy (bulk copy) accesses.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---- L2 eviction priorities (createpolicy + .L2::cache_hint, sm_80 and
// later): the CSR, read once per scan, is marked evict-first, the small array
// every warp of the heavy scan gathers from (parent[]) evict-last.
__device__ __forceinline__ u64 l2_policy_evict_first() {
  u64 p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}

__device__ __forceinline__ u64 l2_policy_evict_last() {
  u64 p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// Global -> shared bulk copy of `bytes` (a multiple of 16, both addresses
// 16-byte aligned) with an L2 cache policy; completion is counted on `bar`.
__device__ __forceinline__ void bulk_g2s_hint(void* dst, const void* src, unsigned bytes, u64* bar, u64 policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar)), "l"(policy)
      : "memory");
}

// 32-bit global load through L2 (no L1 allocation) with an L2 cache policy.
__device__ __forceinline__ int ld_cg_hint(const int* p, u64 policy) {
  int v;
  asm volatile("ld.global.cg.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(policy));
  return v;
}

// Union-find order. A root is hooked under a root of higher priority, where
// the priority is a fixed bijective 32-bit mix of the vertex id (the
// MurmurHash3 finalizer): parent pointers therefore always lead to strictly
// higher priority, so every walk ends and no cycle can form, and because the
// priorities are a random permutation of the ids, the chains built when many
// components merge in one round stay short in expectation (hooking by id, as
// the reference join does with max -> min at ECL_MST.cu:137-144, builds a
// chain as long as any id-monotone path of merging components).
__device__ __forceinline__ unsigned uf_prio(int v) {
  unsigned h = (unsigned)v;
  h ^= h >> 16;
  h *= 0x85ebca6bu;
  h ^= h >> 13;
  h *= 0xc2b2ae35u;
  h ^= h >> 16;
  return h;
}

// Root of v. Path splitting (each visited node is re-pointed to its
// grandparent) is applied on the way: it only shortcuts inside one tree, so
// concurrent finds still reach the same root. Must not run concurrently with
// unions.
__device__ __forceinline__ int find_halve(int v, int* parent) {
  int p = __ldcg(parent + v);
  while (p != v) {
    const int gp = __ldcg(parent + p);
    if (gp != p) __stcg(parent + v, gp);
    v = p;
    p = gp;
  }
  return v;
}

// Read-only root walk (no writes); safe next to unions.
__device__ __forceinline__ int find_ro(int v, const int* parent) {
  int p = __ldcg(parent + v);
  while (p != v) {
    v = p;
    p = __ldcg(parent + v);
  }
  return v;
}

// Union of the trees holding a and b (ECL_MST.cu:137-144): CAS-hook the
// lower-priority node under the higher-priority one if it is still a root;
// a failed CAS returns its current parent, which has higher priority, so the
// lower priority of the pair strictly increases and the loop ends.
__device__ __forceinline__ void cas_union(int a, int b, int* parent) {
  while (a != b) {
    if (uf_prio(a) > uf_prio(b)) {
      const int t = a;
      a = b;
      b = t;
    }
    const int old = atomicCAS(parent + a, a, b);
    if (old == a) return;
    a = old;
  }
}

// Tuple key of an edge: (uint32 weight, edge index), as ((ull)w << 32) | j.
__device__ __forceinline__ u64 edge_key(int w, int j) {
  return ((u64)(unsigned)w << 32) | (u64)(unsigned)j;
}

}  // namespace ecl
