// Boruvka rounds of one phase over a worklist of {rep a, rep b, weight, CSR
// index} entries: kernel1, kernel2 and kernel3 of the reference
// (ECL-MST/ECL_MST.cu:210-251), re-split into three passes per round:
//
//   offer    every entry maps its endpoints through parent[] (one load each:
//            the previous round left every live root's entry flat), is dropped
//            if they agree, else compacted with the new reps, and offers its
//            key to both reps' min slots
//   mark     an entry that holds either rep's minimum is a forest edge: union
//   roots    every live root walks to its new root once, clears its min slot,
//            and stays in the root list if it is still a root
//
// The walk through this round's unions is thus paid once per live root and
// not once per entry, and the finds of the next offer pass are single
// loads. Data that a pass only reads (parent[] while offering, the min slots
// while marking) is loaded through L1, so the entries that share a growing
// tree's root hit in the SM instead of queueing on one L2 line; the barrier's
// acquire makes the pass before visible.
#pragma once
#include "mst_device.cuh"

namespace ecl {

// The grid-wide round kernel: 1024 threads, one worklist entry each, two CTAs
// per SM. What bounds a pass is the latency of its dependent L2 accesses
// (entry, parent, min slot, atomic), so the most threads in flight win:
// measured on Erdos-Renyi 3M / RMAT-22 / RMAT-25, 1.117 / 1.689 / 12.61 ms
// against 1.161 / 1.746 / 12.92 ms with 512 threads of two entries and 1.249 /
// 1.815 / 13.10 ms with 256 of four. 512 x 1 x 4 CTAs is as fast but puts twice
// the CTAs on the barrier.
constexpr int kBorThreads = 1024, kBorEpt = 1, kBorBlocks = 2;
// The cluster kernel that ends a phase, from kTailEntries entries on: its
// passes end in a hardware cluster barrier instead of a grid barrier through
// L2. 8192 to 65536 entries measured within 2 %, 131072 slower (RMAT-14 235
// against 190 us).
constexpr int kTailCtas = 8, kTailThreads = 1024, kTailEpt = 1;
constexpr unsigned kTailEntries = 32768;

struct BorArgs {
  int phase, nodes;
  int list;                // kList*: the entries the rounds start from
  int4* wl0;
  int4* wl1;
  unsigned wl_cap;
  int* parent;
  u64* minv;               // all kNoEdge between phases
  int* roots0;             // live roots, nodes entries each
  int* roots1;
  unsigned char* inMST;
  DevState* st;
  unsigned tail;           // entries at which the cluster kernel takes over
  unsigned solo;           // entries at which its first CTA goes on alone
  int min_tiles;           // keep one CTA per this many tiles of a round (0 = every CTA)
  int count_atomics;
};

// Slots for `total` entries of a list that a CTA's warps append to, out of the
// chunk they share (`word`: first slot << 32 | slots given out; more given out
// than the `chunk` slots it holds: a warp is fetching the next one). The first
// `avail` of them start at `pos`, the others at `fresh`. One thread of a warp
// calls this; total <= chunk. A chunk of 0 reserves exactly what is asked for
// (a list without room for padding): same-address atomics take about 1.8 ns
// each, which is what sharing saves.
__device__ __forceinline__ void chunk_take(u64* word, unsigned chunk, unsigned* ctr, unsigned total, unsigned& pos,
                                           unsigned& avail, unsigned& fresh, DevState* st, unsigned cap) {
  if (chunk == 0) {
    pos = atomicAdd(ctr, total);
    avail = total;
    return;
  }
  for (;;) {
    const u64 old = atomicAdd(word, (u64)total);
    const unsigned used = (unsigned)old;
    pos = (unsigned)(old >> 32) + used;
    if (used + total <= chunk) {
      avail = total;
      return;
    }
    if (used <= chunk) {  // the one that overruns the chunk fetches the next
      avail = chunk - used;
      fresh = atomicAdd(ctr, chunk);
      atomicExch(word, ((u64)fresh << 32) | (total - avail));
      return;
    }
    for (unsigned spin = 0; (unsigned)*(volatile u64*)word > chunk; spin++)
      if (spin > (1u << 24)) {  // seconds: the other warp is gone
        atomicOr(&st->error, kErrTimeout);
        avail = 0;
        fresh = cap;  // nothing is written there
        return;
      }
  }
}

struct BorSmem {
  unsigned cursor;                    // entries this CTA kept in the current offer pass
  int seg_n;                          // segments of the list read next (0 = dense)
  unsigned seg_q[kMaxRoundCtas + 1];  // entries in the segments before b
  unsigned seg_off[kMaxRoundCtas];    // first position of segment b
  int hot_rep[kHotSlots];             // representative -> this CTA's partial minimum
  u64 hot_key[kHotSlots];
  unsigned warp_cnt[2][32];
  unsigned base[2];
};

__device__ __forceinline__ u64 ld_ca64(const u64* p) {
  u64 v;
  asm volatile("ld.global.ca.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_add_release_gpu(unsigned* p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Barrier among the first `active` of the `ctas` CTAs of a cooperative launch,
// or of one of its teams: one release add per CTA to a counter that only
// grows, and an acquire poll of the same counter by one thread; the other
// threads are ordered through the CTA barriers on both sides. (A counter that
// the last CTA resets before it releases a generation word took 1.85 us on 32
// to 296 CTAs.) The wait is bounded (kErrTimeout, and every later barrier then
// returns false).
struct GridSync {
  static constexpr bool kGrid = true;
  DevState* st;
  unsigned* word;  // the counter; regroup: [1] the last gate opened, [2] the barrier count there; zero at first
  unsigned rank, ctas, active, target, gates;
  __device__ __forceinline__ void init(DevState* s, unsigned* words, unsigned r, unsigned n) {
    st = s;
    word = words;
    rank = r;
    active = ctas = n;
    target = gates = 0;
  }
  __device__ __forceinline__ bool poll(const unsigned* p, unsigned at_least, bool nap) {
    u64 t0 = 0;
    for (unsigned spin = 1; (int)(ld_acquire_gpu(p) - at_least) < 0; spin++) {
      if (nap) __nanosleep(100);
      if ((spin & 1023u) == 0) {  // the limit, checked now and then
        const u64 now = globaltimer_ns();
        if (!t0) t0 = now;
        if (now - t0 > kBarrierTimeoutNs) atomicOr(&st->error, kErrTimeout);
        if (ld_volatile(&st->error) & kErrTimeout) return false;
      }
    }
    return true;
  }
  __device__ __forceinline__ bool sync() {
    __syncthreads();
    if (active == 1) return true;
    target += active;
    bool ok = true;
    if (threadIdx.x == 0) {
      red_add_release_gpu(word, 1u);
      ok = poll(word, target, false);
    }
    return __syncthreads_and(ok);
  }
  // All CTAs again, after rounds some of them `left`: those wait until the
  // first CTA, done with the rounds, opens the next gate, and take over its
  // count of the barriers.
  __device__ __forceinline__ bool regroup(bool left) {
    bool ok = true;
    gates++;
    __syncthreads();
    if (threadIdx.x == 0) {
      if (rank == 0) {
        word[2] = target;
        st_release_gpu(word + 1, gates);
      } else if (left) {
        ok = poll(word + 1, gates, true);
      }
    }
    active = ctas;
    ok = __syncthreads_and(ok);
    if (left) target = ld_volatile(word + 2);
    return ok;
  }
};

// The same interface over one thread-block cluster (hardware barrier), or
// over its first CTA alone.
struct ClusterSync {
  static constexpr bool kGrid = false;
  unsigned rank, active, ctas;
  __device__ __forceinline__ void init(unsigned n) {
    active = ctas = n;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  }
  __device__ __forceinline__ bool sync() {
    if (active == 1) {
      __syncthreads();
    } else {
      asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    }
    return true;
  }
};

__device__ __forceinline__ void bor_smem_init(BorSmem& s) {
  if (threadIdx.x == 0) {
    s.cursor = 0;
    s.seg_n = 0;
  }
  for (int i = threadIdx.x; i < kHotSlots; i += blockDim.x) {
    s.hot_rep[i] = -1;
    s.hot_key[i] = kNoEdge;
  }
}

// Prefix table of the `nseg` segments the last offer pass wrote. Every thread
// of the CTA calls this; the caller synchronises before the table is used.
template <int T>
__device__ __forceinline__ void bor_seg_load(BorSmem& s, const DevState* st, int nseg) {
  constexpr int kPer = (kMaxRoundCtas + T - 1) / T;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  unsigned c[kPer], mine = 0;
#pragma unroll
  for (int k = 0; k < kPer; k++) {
    const int b = kPer * t + k;
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
  if (lane == 31) s.warp_cnt[0][warp] = incl;
  __syncthreads();
  unsigned wsum = lane < warp ? s.warp_cnt[0][lane] : 0u;  // warps before this one
  wsum = __reduce_add_sync(0xffffffffu, wsum);
  unsigned q = wsum + incl - mine;
#pragma unroll
  for (int k = 0; k < kPer; k++) {
    const int b = kPer * t + k;
    if (b < nseg) s.seg_q[b] = q;
    q += c[k];
    if (b == nseg - 1) s.seg_q[nseg] = q;
  }
  if (t == 0) s.seg_n = nseg;
}

__device__ __forceinline__ unsigned bor_seg_at(const BorSmem& s, unsigned i) {
  const int nseg = s.seg_n;
  if (nseg == 0) return i;
  int lo = 0, hi = nseg;  // largest b with seg_q[b] <= i (seg_q[nseg] > i)
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (s.seg_q[mid] <= i) lo = mid;
    else hi = mid;
  }
  return s.seg_off[lo] + (i - s.seg_q[lo]);
}

// Offer (rep, key) pairs to the reps' min slots, except to `skip`: the forest
// needs every tree but one to pick its lightest edge, so the phase's largest
// tree, whose slot nearly every entry would hit, picks none. A rep already in
// the CTA's hot table folds into it; where neighbouring lanes hold equal reps
// the warp reduces them first (__match_any_sync) and a group of four or more
// claims a table slot; the rest read their slots together and issue an
// atomicMin where that improves it (ECL_MST.cu:221-223). Every lane calls this.
template <int N>
__device__ __forceinline__ unsigned bor_offer(const int (&rep)[N], const u64 (&key)[N], const bool (&valid)[N],
                                              int skip, u64* minv, BorSmem& s) {
  const int lane = threadIdx.x & 31;
  bool cold[N];
  u64 val[N];
#pragma unroll
  for (int i = 0; i < N; i++) {
    val[i] = key[i];
    cold[i] = valid[i] && rep[i] != skip;
    const unsigned slot = hot_slot(rep[i]);
    if (cold[i] && ((volatile int*)s.hot_rep)[slot] == rep[i]) {
      if (((volatile u64*)s.hot_key)[slot] > key[i]) atomicMin(&s.hot_key[slot], key[i]);
      cold[i] = false;
    }
    const int mine = cold[i] ? rep[i] : -2 - lane;
    const int before = __shfl_up_sync(0xffffffffu, mine, 1);
    if (!__any_sync(0xffffffffu, lane > 0 && before == mine)) continue;
    const unsigned g = __match_any_sync(0xffffffffu, mine);
    if (!cold[i] || (g & (g - 1)) == 0) continue;
    const unsigned khi = (unsigned)(key[i] >> 32);
    const unsigned hi = __reduce_min_sync(g, khi);
    const unsigned lo = __reduce_min_sync(g, khi == hi ? (unsigned)key[i] : 0xffffffffu);
    cold[i] = lane == __ffs(g) - 1;
    if (!cold[i]) continue;
    val[i] = ((u64)hi << 32) | lo;
    if (__popc(g) < 4) continue;
    int cur = ((volatile int*)s.hot_rep)[slot];
    if (cur < 0) {
      cur = atomicCAS(&s.hot_rep[slot], -1, rep[i]);
      if (cur < 0) cur = rep[i];
    }
    if (cur == rep[i]) {
      if (((volatile u64*)s.hot_key)[slot] > val[i]) atomicMin(&s.hot_key[slot], val[i]);
      cold[i] = false;
    }
  }
  u64 seen[N];
#pragma unroll
  for (int i = 0; i < N; i++) seen[i] = cold[i] ? __ldcg(minv + rep[i]) : 0ull;
  unsigned n = 0;
#pragma unroll
  for (int i = 0; i < N; i++)
    if (seen[i] > val[i]) {
      atomicMin(minv + rep[i], val[i]);
      n++;
    }
  return n;
}

// One step of the roots pass for U vertices per thread: live roots (those
// offered an edge this round, and `skip`, which is offered none) clear their
// slot and walk to their new root; the ones still a root are appended to
// `out`. `dup`: a vertex may come up more than once (roots taken from the
// entries), so the slot is exchanged and only the thread that got the key
// goes on. Every thread of the CTA calls this (it synchronises the CTA);
// `flip` alternates the reservation buffers, so one step's use of them is
// over before the next but one.
template <int U>
__device__ __forceinline__ void bor_roots_step(const BorArgs& a, const int (&v)[U], const bool (&valid)[U], bool dup,
                                               int skip, int* out, unsigned* ctr, int flip, BorSmem& s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  u64 k[U];
#pragma unroll
  for (int i = 0; i < U; i++) k[i] = valid[i] && !dup ? __ldcg(a.minv + v[i]) : kNoEdge;
  if (dup) {
#pragma unroll
    for (int i = 0; i < U; i++)
      if (valid[i] && v[i] != skip) k[i] = atomicExch(a.minv + v[i], kNoEdge);
  }
  bool live[U];
  int p[U];
#pragma unroll
  for (int i = 0; i < U; i++) {
    live[i] = valid[i] && (k[i] != kNoEdge || (v[i] == skip && !dup));
    p[i] = live[i] ? ld_ca(a.parent + v[i]) : 0;
    if (live[i] && !dup && k[i] != kNoEdge) __stcg(a.minv + v[i], kNoEdge);
  }
  bool walk[U];
#pragma unroll
  for (int i = 0; i < U; i++) walk[i] = live[i] && p[i] != v[i];
  unsigned keep = 0;
#pragma unroll
  for (int i = 0; i < U; i++) keep |= (unsigned)(live[i] && p[i] == v[i]) << i;
  for (bool any = true; any;) {
    any = false;
    int gp[U];
#pragma unroll
    for (int i = 0; i < U; i++) gp[i] = walk[i] ? ld_ca(a.parent + p[i]) : 0;
#pragma unroll
    for (int i = 0; i < U; i++)
      if (walk[i]) {
        if (gp[i] == p[i]) {
          __stcg(a.parent + v[i], p[i]);
          walk[i] = false;
        } else {
          p[i] = gp[i];
          any = true;
        }
      }
  }
  if (!out) return;
  // CTA-wide reservation of the kept roots
  const unsigned cnt = __popc(keep);
  unsigned incl = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) s.warp_cnt[flip][warp] = incl;
  __syncthreads();
  const int nw = blockDim.x >> 5;
  const unsigned w = lane < nw ? s.warp_cnt[flip][lane] : 0u;
  const unsigned before = __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u);
  if (warp == 0) {
    const unsigned total = __reduce_add_sync(0xffffffffu, w);
    if (lane == 0) s.base[flip] = total ? atomicAdd(ctr, total) : 0u;
  }
  __syncthreads();
  unsigned pos = s.base[flip] + before + incl - cnt;
#pragma unroll
  for (int i = 0; i < U; i++)
    if (keep & (1u << i)) out[pos++] = v[i];
}

// Rounds from state `b` until the list is empty (true) or, grid-wide, until
// it is at most a.tail entries long (false: `b` is where to go on). The
// endpoints of the lists light 0 and heavy are roots that differ: their first
// round finds nothing and compacts nothing (without kLists there are no others).
// CTAs beyond what a round needs leave (`left`); their `b` is meaningless.
//
// Below some 10^5 entries a round is bound by its dependent L2 accesses (0.35
// us a load or atomic) and barriers, so the loads that do not depend on each
// other are issued together, the entries of a CTA with one tile stay in
// registers from the offer to the mark pass (kKeep: not in k_round, which
// spills 60 bytes of its 32 registers a thread as it is; 2 % slower on RMAT-22),
// and where the vertices are few for the threads at work the roots pass looks at
// all of them instead of keeping a list.
template <int T, int E, bool kKeep, bool kLists, class Sync>
__device__ __forceinline__ bool bor_rounds(const BorArgs& a, BorState& b, Sync& sy, BorSmem& s, bool& left) {
  constexpr int N = 2 * E;
  constexpr unsigned tile = T * E;
  DevState* st = a.st;
  const int ph = a.phase, tid = threadIdx.x;
  left = false;
  // The list, and the arrays the rounds compact into in turn: never the one
  // whose end still holds the list, or a later one that fits beside it.
  const bool fresh_list = !kLists || a.list == kListLight0 || a.list == kListHeavy;
  const bool mid = kLists && a.list == kListMid;
  int4* const out0 = mid ? a.wl0 : a.wl1;
  int4* const out1 = mid ? a.wl1 : a.wl0;
  const int4* first_list = fresh_list ? a.wl0 : out1 + (a.wl_cap - st->lists[a.list].slots);
  unsigned atomics = 0;
  const bool stamp = sy.rank == 0 && tid == 0;
  bool done = true;
  // CTAs that work on a round of W entries, of `active`
  auto wanted = [&](unsigned W, unsigned active) {
    unsigned want = active;
    if (Sync::kGrid && a.min_tiles > 0) want = min(want, max(1u, (W + a.min_tiles * tile - 1) / (a.min_tiles * tile)));
    if ((!Sync::kGrid || !a.tail) && W <= a.solo) want = 1;
    return want;
  };
  // whether a roots pass by `threads` threads looks at all vertices
  auto scan_roots = [&](unsigned threads) { return (u64)(unsigned)a.nodes <= 4ull * threads; };
  while (b.W) {
    if (b.r >= ECL_MAX_ROUNDS) {
      if (stamp) atomicOr(&st->error, kErrRounds);
      break;
    }
    if (Sync::kGrid && b.W <= a.tail) {
      done = false;
      break;
    }
    const unsigned want = wanted(b.W, sy.active);
    if (want < sy.active) {
      sy.active = want;
      if (sy.rank >= want) {
        left = true;
        break;
      }
    }
    const unsigned start = sy.rank, stride = sy.active;
    const bool fresh = b.first && fresh_list;
    const int4* in = b.k == 0 ? first_list : ((b.k & 1) ? out0 : out1);
    int4* out = (b.k & 1) ? out1 : out0;
    const unsigned W = b.W, ntiles = (W + tile - 1) / tile;
    const unsigned region = share_region(W, tile, start, stride);
    const bool one = kKeep && ntiles <= stride;  // no CTA has a second tile
    int4 e[E];
    bool ok[E];
#pragma unroll
    for (int i = 0; i < E; i++) ok[i] = false;
    // ---- offer
    for (unsigned t = start; t < ntiles; t += stride) {
#pragma unroll
      for (int i = 0; i < E; i++) {
        const unsigned idx = t * tile + i * T + tid;
        ok[i] = idx < W;
        e[i] = ok[i] ? __ldcg(in + bor_seg_at(s, idx)) : make_int4(-1, -1, 0, 0);
        ok[i] = e[i].x >= 0;  // null entries (unused scan slots)
      }
      if (!fresh) {
        int x[N];
#pragma unroll
        for (int i = 0; i < E; i++) {
          x[2 * i] = ok[i] ? ld_ca(a.parent + e[i].x) : 0;
          x[2 * i + 1] = ok[i] ? ld_ca(a.parent + e[i].y) : 0;
        }
        unsigned mask[E], total = 0;
#pragma unroll
        for (int i = 0; i < E; i++) {
          e[i].x = x[2 * i];
          e[i].y = x[2 * i + 1];
          ok[i] = ok[i] && e[i].x != e[i].y;
          mask[i] = __ballot_sync(0xffffffffu, ok[i]);
          total += __popc(mask[i]);
        }
        unsigned pos = 0;
        if ((tid & 31) == 0 && total) pos = atomicAdd(&s.cursor, total);
        pos = region + __shfl_sync(0xffffffffu, pos, 0);
#pragma unroll
        for (int i = 0; i < E; i++) {
          const unsigned p = pos + __popc(mask[i] & ((1u << (tid & 31)) - 1u));
          if (ok[i]) {
            if (p < a.wl_cap) __stcg(out + p, e[i]);
            else atomicOr(&st->error, kErrOverflow);
          }
          pos += __popc(mask[i]);
        }
      }
      int rep[N];
      u64 key[N];
      bool val[N];
#pragma unroll
      for (int i = 0; i < E; i++) {
        rep[2 * i] = e[i].x;
        rep[2 * i + 1] = e[i].y;
        key[2 * i] = key[2 * i + 1] = edge_key(e[i].z, e[i].w);
        val[2 * i] = val[2 * i + 1] = ok[i];
      }
      atomics += bor_offer<N>(rep, key, val, b.skip, a.minv, s);
    }
    __syncthreads();
    if (tid == 0 && !fresh) {
      st->seg_cnt[start] = s.cursor;
      st->seg_off[start] = region;
      if (s.cursor) {
        atomicAdd(&st->wl_count[ph][b.r + 1], s.cursor);
        atomicAdd(&st->wl_kept[ph][b.r + 1], s.cursor);
      }
    }
    if (stamp && fresh) {  // the scan's list is the first round's output
      st->wl_count[ph][b.r + 1] = W;
      st->wl_kept[ph][b.r + 1] = ld_volatile(&st->lists[a.list].kept);
    }
    for (int i = tid; i < kHotSlots; i += T) {  // flush the partial minima
      const int r = s.hot_rep[i];
      if (r >= 0) {
        const u64 k = s.hot_key[i];
        if (__ldcg(a.minv + r) > k) {
          atomicMin(a.minv + r, k);
          atomics++;
        }
        s.hot_rep[i] = -1;
        s.hot_key[i] = kNoEdge;
      }
    }
    if (!sy.sync()) break;
    if (stamp) st->t_round[ph][2 * b.r] = globaltimer_ns();
    u64 mx[E], my[E];
    auto minima = [&]() {
#pragma unroll
      for (int i = 0; i < E; i++) {
        mx[i] = ok[i] && e[i].x != b.skip ? ld_ca64(a.minv + e[i].x) : kNoEdge;
        my[i] = ok[i] && e[i].y != b.skip ? ld_ca64(a.minv + e[i].y) : kNoEdge;
      }
    };
    auto mark = [&]() {
#pragma unroll
      for (int i = 0; i < E; i++) {
        const u64 key = edge_key(e[i].z, e[i].w);
        if (ok[i] && (key == mx[i] || key == my[i])) {
          cas_union(e[i].x, e[i].y, a.parent);
          a.inMST[e[i].w] = 1;
        }
      }
    };
    if (one) minima();
    const unsigned W2 = ld_volatile(&st->wl_count[ph][b.r + 1]);
    b.r++;
    if (W2 == 0) {
      b.W = 0;
      break;
    }
    // The next round's segment table is read here, two barriers before any CTA
    // can be at the end of that round's offer pass and publish new segments.
    if (!fresh) {
      if (stride > 1) bor_seg_load<T>(s, st, (int)stride);
      else if (tid == 0) s.seg_n = 0;  // one segment, from position 0
    }
    // ---- mark: the first round's scan list, or this CTA's own segment
    if (one) {
      mark();
    } else {
      const unsigned cnt = fresh ? W : s.cursor;
      const unsigned step = fresh ? stride * tile : tile;
      const int4* src = fresh ? in : out + region;
      for (unsigned base = fresh ? start * tile : 0u; base < cnt; base += step) {
#pragma unroll
        for (int i = 0; i < E; i++) {
          const unsigned idx = base + i * T + tid;
          e[i] = idx < cnt ? __ldcg(src + idx) : make_int4(-1, -1, 0, 0);
          ok[i] = e[i].x >= 0;
        }
        minima();
        mark();
      }
    }
    if (!sy.sync()) break;
    // ---- roots
    const bool all = scan_roots(stride * T) || (b.first && 4ull * W2 >= (unsigned)a.nodes);
    // threads of the next roots pass, and whether it will want a list
    const unsigned ahead = Sync::kGrid && W2 <= a.tail ? (W2 <= a.solo ? 1u : (unsigned)kTailCtas) * kTailThreads
                                                       : wanted(W2, stride) * T;
    int* rout = scan_roots(ahead) ? nullptr : ((b.flips & 1) ? a.roots1 : a.roots0);
    const int* rin = (b.flips & 1) ? a.roots0 : a.roots1;
    unsigned* rctr = &st->root_cnt[a.list][b.flips % 3];
    int flip = 0;
    constexpr int U = E > 1 ? 4 : 2;
    if (b.first && !all) {  // few entries for the vertices: take the roots from this CTA's entries
      const unsigned cnt = fresh ? W : s.cursor;
      const unsigned step = fresh ? stride * T : T;
      const int4* src = fresh ? in : out + region;
      // every CTA thread takes every step (the step synchronises the CTA)
      for (unsigned base = fresh ? start * T : 0u; base < cnt; base += step, flip ^= 1) {
        const unsigned idx = base + tid;
        const int4 x = idx < cnt ? __ldcg(src + idx) : make_int4(-1, -1, 0, 0);
        const int v[2] = {x.x, x.y};
        const bool valid[2] = {x.x >= 0, x.x >= 0};
        bor_roots_step<2>(a, v, valid, true, b.skip, rout, rctr, flip, s);
      }
      if (b.skip >= 0 && start == 0) {  // `skip` is in no slot: carried by hand
        const int v[2] = {b.skip, 0};
        const bool valid[2] = {tid == 0, false};
        bor_roots_step<2>(a, v, valid, false, b.skip, rout, rctr, flip, s);
      }
      // Every warp has read the CTA's count of entries before it is cleared: the
      // steps' CTA barriers see to that, but steps without a list have none.
      __syncthreads();
    } else {
      const unsigned cnt = all ? (unsigned)a.nodes : b.C;
      for (unsigned base = start * T * U; base < cnt; base += stride * T * U, flip ^= 1) {
        int v[U];
        bool valid[U];
#pragma unroll
        for (int i = 0; i < U; i++) {
          const unsigned idx = base + i * T + tid;
          valid[i] = idx < cnt;
          v[i] = !valid[i] ? 0 : (all ? (int)idx : __ldcg(rin + idx));
        }
        bor_roots_step<U>(a, v, valid, false, b.skip, rout, rctr, flip, s);
      }
    }
    if (stamp) st->root_cnt[a.list][(b.flips + 1) % 3] = 0;  // the next roots pass's counter
    if (tid == 0) s.cursor = 0;
    if (!sy.sync()) break;
    if (stamp) st->t_round[ph][2 * b.r - 1] = globaltimer_ns();
    if (rout) b.C = ld_volatile(rctr);
    b.flips++;
    if (b.skip >= 0) b.skip = ld_ca(a.parent + b.skip);
    if (!fresh) {
      b.nseg = stride > 1 ? (int)stride : 0;
      b.k++;
    }
    b.first = 0;
    b.W = W2;
  }
  if (a.count_atomics && atomics) atomicAdd(&st->atomics, (u64)atomics);
  return done;
}

// The rounds of one phase, grid-wide: a cooperative launch that ends when the
// list is empty or short enough for one cluster (k_round_tail).
__global__ void __launch_bounds__(kBorThreads, kBorBlocks) k_round(BorArgs a) {
  __shared__ BorSmem s;
  DevState* st = a.st;
  if (a.phase == 1 && !st->filtered) return;
  if (ld_volatile(&st->error) & (kErrFormat | kErrTimeout)) return;  // bits no CTA of this kernel sets before a barrier
  // every CTA finds the same: the lists of one array must not meet
  const unsigned l0 = st->lists[kListLight0].slots, l1 = st->lists[kListLight1].slots, l2 = st->lists[kListMid].slots;
  const bool first = a.list == kListLight0;
  if (first ? (u64)l0 + l1 > a.wl_cap || (u64)max(l0, l1) + l2 > a.wl_cap : st->lists_bad != 0) {
    if (first && blockIdx.x == 0 && threadIdx.x == 0) {
      atomicOr(&st->error, kErrOverflow);
      st->lists_bad = 1;
      st->resume = BorState{};
    }
    return;
  }
  BorState b = {};
  b.W = min(st->lists[a.list].slots, a.wl_cap);
  b.r = st->rounds[a.phase];
  b.first = 1;
  b.skip = first ? -1 : st->giant;
  GridSync sy;
  sy.init(st, &st->bar[a.list], blockIdx.x, gridDim.x);
  bor_smem_init(s);
  __syncthreads();
  const bool stamp = sy.rank == 0 && threadIdx.x == 0;
  if (stamp) {
    if (b.r == 0) st->t_round_start[a.phase] = globaltimer_ns();
    if (b.W && b.r < ECL_MAX_ROUNDS) {
      st->t_list[a.list] = globaltimer_ns();
      st->r_list[a.list] = b.r;
      st->wl_count[a.phase][b.r] = b.W;
      st->wl_kept[a.phase][b.r] = st->lists[a.list].kept;
    }
  }
  bool left;
  const bool done = bor_rounds<kBorThreads, kBorEpt, false, true>(a, b, sy, s, left);
  if (stamp && !left) {
    st->rounds[a.phase] = b.r;
    if (done) b.W = 0;
    st->resume = b;
  }
}

// The end of a list on one cluster: goes on from where k_round stopped. Its
// first CTA then names the tree that holds most of the vertices (a vote of
// sampled vertices), which the next list's rounds leave out of their offers.
__global__ void __cluster_dims__(kTailCtas, 1, 1) __launch_bounds__(kTailThreads, 1) k_round_tail(BorArgs a) {
  __shared__ BorSmem s;
  DevState* st = a.st;
  if (!st->filtered && a.phase == 1) return;
  if (ld_volatile(&st->error) & (kErrFormat | kErrTimeout)) return;  // set before this launch
  BorState b = st->resume;
  ClusterSync sy;
  sy.init(kTailCtas);
  bor_smem_init(s);
  __syncthreads();
  bool left = false;
  if (b.W) {
    if (b.nseg) {
      bor_seg_load<kTailThreads>(s, st, b.nseg);
      sy.sync();  // a CTA without entries publishes its new segment at once: not before all have read the old ones
    }
    bor_rounds<kTailThreads, kTailEpt, true, true>(a, b, sy, s, left);
    if (sy.rank == 0 && threadIdx.x == 0 && !left) st->rounds[a.phase] = b.r;
  }
  const bool more = a.list == kListLight0 ? st->filtered || st->lists[kListLight1].slots
                                          : a.list != kListHeavy && st->lists[a.list].slots;
  if (more && sy.rank == 0) {
    __syncthreads();
    int* vote = reinterpret_cast<int*>(s.seg_q);
    const int v = (int)(uf_prio((int)threadIdx.x + 1) % (unsigned)a.nodes);
    const int root = find_ro(v, a.parent);
    vote[threadIdx.x] = root;
    if (threadIdx.x == 0) s.hot_key[0] = 0;
    __syncthreads();
    unsigned same = 0;
    for (int i = 0; i < kTailThreads; i++) same += vote[i] == root;
    atomicMax(&s.hot_key[0], ((u64)same << 32) | (unsigned)root);
    __syncthreads();
    if (threadIdx.x == 0) st->giant = (int)(unsigned)s.hot_key[0];
  }
}

}  // namespace ecl
