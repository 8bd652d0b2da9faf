// The two CSR scans that build the phases' worklists (initWL, ECL-MST/
// ECL_MST.cu:157-207). Each reads one of the two entry arrays whole and the
// other only where the first leaves an entry in question:
//
//   light  streams eweight; the neighbour id and the row of an entry are looked
//          up only if its weight passes the light test. Also zeroes inMST.
//   heavy  streams nlist; every light edge joined two trees by now, so an entry
//          whose ends lie in one tree is dropped by that alone, and the weight
//          is read only for the entries kept. Nearly all of them lie in the
//          light phase's largest tree, so the test is a bit per vertex
//          (k_flatten's tree_bits, n/8 bytes) before it is two gathers of
//          parent[].
//
// A warp takes tasks of kGran = 512 consecutive entries on its own: its lane 0
// brings the stream's slice to shared memory by bulk copies (cp.async.bulk),
// kStages tasks deep, and every lane tests 16 entries, which leaves a 16-bit
// mask. What the scans are bound by is instructions and, in the heavy one, the
// lines that a warp's scattered loads touch, so the entries in question are
// first gathered into a queue of the warp's own, and then worked off with full
// lanes, two to a lane: look up the row (a binary search in the task's slice of
// nindex, copied ahead to shared memory), test, append. The common entry costs
// three instructions and the rare one runs with full lanes, whatever its row's
// length (the reference's thread / warp degree split, :167/:185, is not
// needed). Worklist slots come from the list's counter in chunks that a CTA's
// warps share (chunk_take); the unused tail of a CTA's last chunk is filled
// with null entries (x = -1).
//
// Light and heavy scan, against tiles of both arrays staged for a whole CTA:
// RMAT-22 (128.3M entries, 1.9M and 11.3M kept) 215 and 380 us against 332 and
// 512; ER 16M (536.9M, 31.1M and 12.6M) 1373 and 1150 against 1270 and 2262.
// Streaming one array takes 79 and 332 us at the measured copy bandwidth.
#pragma once
#include "rounds_device.cuh"

namespace ecl {

constexpr int kScanThreads = 256;        // 8 warps, each on its own tasks
constexpr int kScanWarps = kScanThreads / 32;
constexpr int kScanBlocks = 3;           // resident CTAs per SM (4: 64 registers spill, RMAT-22 11 % slower)
constexpr int kScanStages = 2;           // tasks whose entries are in shared memory or on the way (3: 7 % slower)
constexpr int kScanItems = 2;            // entries in question a lane works off at once
constexpr int kScanSlice = 256;          // nindex entries staged per task (longer slices are searched in L1)
// Rows of a task looked at one by one (heavy). A task of more, such as RMAT's
// high vertices', has few entries to a row, and working off all of them costs
// less than the rows' starts: RMAT-22 1.38 ms against 1.39 with 512 rows, 1.42
// with 1024 and 1.48 with 4096; with 64 a task of a grid (128 rows) is 7 %
// slower.
constexpr int kScanMaxRows = 192;
static_assert(kScanMaxRows < kScanSlice && kScanMaxRows / 32 + 2 <= 32, "in shared memory, a word per lane");
constexpr unsigned kScanDense = 224;     // entries in question of a task's 512, see k_scan_light
constexpr unsigned kScanMaxChunk = 384;  // worklist slots a CTA reserves at once,
constexpr unsigned kScanMinChunk = 128;  // never less than one warp may append

template <bool LIGHT>
struct alignas(16) ScanWarpSmem {
  int data[kScanStages][kGran];  // the stream's entries
  int slice[2][kScanSlice];      // nindex of this task's rows and the next one's
  u64 full[kScanStages];         // copies landed
  unsigned rows_out[kGran / 32]; // heavy: entries of rows outside the tree, a bit each
  int ends[LIGHT ? kGran : 4];   // light: the neighbours of the queue's entries
  unsigned short queue[kGran];   // entries in question, by position in the task
};
template <bool LIGHT>
struct ScanSmem {
  ScanWarpSmem<LIGHT> warp[kScanWarps];
  u64 chunk[4];                  // per list: the CTA's current slots (chunk_take)
  unsigned kept[4];
};

// Slot `slot` of list `kind` (kListLight0 ...).
__device__ __forceinline__ int4* list_slot(const ScanArgs& a, int kind, unsigned slot) {
  int4* const wl = kind == kListMid ? a.wl1 : a.wl0;
  return wl + (kind == kListLight1 || kind == kListMid ? a.wl_cap - 1u - slot : slot);
}

// Append the lanes' entries (up to ITEMS each) to the lists: entry i goes
// to list (cls >> 4 * i & 15), none if that nibble is 15. Every lane of the
// warp calls this.
template <int ITEMS>
__device__ __forceinline__ void lists_append(const ScanArgs& a, u64* chunks, unsigned* kept, int first, int last,
                                             unsigned cls, const int4 (&e)[ITEMS]) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int k = first; k <= last; k++) {
    unsigned mask[ITEMS], total = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
      mask[i] = __ballot_sync(0xffffffffu, ((cls >> (4 * i)) & 15u) == (unsigned)k);
      total += __popc(mask[i]);
    }
    if (!total) continue;
    unsigned pos = 0, avail = 0, fresh = 0;
    if (lane == 0) {
      chunk_take(&chunks[k], a.chunk, &a.st->lists[k].slots, total, pos, avail, fresh, a.st, a.wl_cap);
      atomicAdd(&kept[k], total);
    }
    pos = __shfl_sync(0xffffffffu, pos, 0);
    avail = __shfl_sync(0xffffffffu, avail, 0);
    fresh = __shfl_sync(0xffffffffu, fresh, 0);
    unsigned rank = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
      const unsigned r = rank + __popc(mask[i] & ((1u << lane) - 1u));
      rank += __popc(mask[i]);
      if (((cls >> (4 * i)) & 15u) != (unsigned)k) continue;
      const unsigned slot = r < avail ? pos + r : fresh + (r - avail);
      if (slot >= a.wl_cap) atomicOr(&a.st->error, kErrOverflow);
      else if (a.ids) reinterpret_cast<int*>(a.wl0)[slot] = e[i].w;
      else __stcg(list_slot(a, k, slot), e[i]);
    }
  }
}

// Null entries in the slots of the CTA's last chunk that were not given out.
// Every thread of the CTA calls this, after its warps' last appends.
__device__ __forceinline__ void list_close(const ScanArgs& a, int kind, u64 word, unsigned kept) {
  const unsigned base = (unsigned)(word >> 32);
  for (unsigned p = (unsigned)word + threadIdx.x; p < a.chunk; p += kScanThreads)
    if (base + p < a.wl_cap) {
      if (a.ids) reinterpret_cast<int*>(a.wl0)[base + p] = -1;
      else *list_slot(a, kind, base + p) = make_int4(-1, -1, 0, 0);
    }
  if (threadIdx.x == 0 && kept) atomicAdd(&a.st->lists[kind].kept, kept);
}

// The rows lo .. hi that hold a task's entries.
struct TaskRows {
  int lo, hi;
};
__device__ __forceinline__ TaskRows task_rows(const ScanArgs& a, int t) {
  if (t >= a.tiles) return TaskRows{0, 0};
  return TaskRows{__ldg(a.first_v + t), __ldg(a.first_v + t + 1)};
}

// Starts the copy of nindex[lo .. hi] to shared memory, if it fits.
__device__ __forceinline__ void slice_start(const ScanArgs& a, const TaskRows& r, int* slice) {
  const int len = r.hi - r.lo + 1;
  if (len <= kScanSlice)
    for (int i = threadIdx.x & 31; i < len; i += 32)
      __pipeline_memcpy_async(slice + i, a.nindex + r.lo + i, sizeof(int));
  __pipeline_commit();
}

// nindex[lo + k] of a task.
__device__ __forceinline__ int slice_at(const ScanArgs& a, const TaskRows& r, const int* slice, int k) {
  return r.hi - r.lo < kScanSlice ? slice[k] : __ldg(a.nindex + r.lo + k);
}

// The rows holding entries e[].w of the task: the last v with nindex[v] <= j.
// All lanes search the same number of steps.
__device__ __forceinline__ void rows_of(const ScanArgs& a, const TaskRows& r, const int* slice,
                                        const int4 (&e)[kScanItems], int (&v)[kScanItems]) {
  const int len = r.hi - r.lo + 1;
  int at[kScanItems] = {};
#pragma unroll 1
  for (int step = len <= 1 ? 0 : 1 << (31 - __clz(len - 1)); step; step >>= 1) {
#pragma unroll
    for (int i = 0; i < kScanItems; i++) {
      const int k = min(at[i] + step, len - 1);  // a probe beyond the end repeats the last row
      if (slice_at(a, r, slice, k) <= e[i].w) at[i] = k;
    }
  }
#pragma unroll
  for (int i = 0; i < kScanItems; i++) v[i] = r.lo + at[i];
}

template <class Smem, class Warp>
__device__ __forceinline__ void scan_open(const ScanArgs& a, Smem& sm, Warp& ws) {
  if (threadIdx.x < 4) {
    sm.chunk[threadIdx.x] = a.chunk;
    sm.kept[threadIdx.x] = 0;
  }
  if ((threadIdx.x & 31) < kScanStages) mbar_init(&ws.full[threadIdx.x & 31], 1);
  mbar_fence_init();
  __syncthreads();
}

// Brings task t's entries to stage s: the 16-byte multiple by a bulk copy, the
// last task's ragged end (or all, unaligned) by the lanes.
template <bool VEC, class Warp>
__device__ __forceinline__ void scan_fill(const ScanArgs& a, Warp& ws, const int* stream, int t, int s, u64 policy) {
  if (t >= a.tiles) return;
  const int lane = threadIdx.x & 31, j0 = t * kGran, cnt = min(kGran, a.edges - j0), bulk = VEC ? cnt & ~3 : 0;
  for (int q = bulk + lane; q < cnt; q += 32) ws.data[s][q] = __ldg(stream + j0 + q);
  __syncwarp();
  if (lane == 0) {
    fence_proxy_async_smem();
    mbar_arrive_tx(&ws.full[s], 4u * (unsigned)bulk);
    if (bulk) bulk_g2s_hint(ws.data[s], stream + j0, 4u * (unsigned)bulk, &ws.full[s], policy);
  }
}

// Waits for stage s and for the slice copies started before.
template <class Warp>
__device__ __forceinline__ bool scan_wait(const ScanArgs& a, Warp& ws, int s, unsigned parity) {
  __pipeline_wait_prior(0);
  const bool ok = __all_sync(0xffffffffu, mbar_wait(&ws.full[s], parity, kBarrierTimeoutNs));
  if (!ok && (threadIdx.x & 31) == 0) atomicOr(&a.st->error, kErrTimeout);
  __syncwarp();
  return ok;
}

// Puts the positions of the lanes' entries in question into the queue; returns
// how many there are.
template <bool kStrided>
__device__ __forceinline__ int scan_gather(unsigned mask, unsigned short* queue) {
  const int lane = threadIdx.x & 31;
  const unsigned mine = __popc(mask);
  unsigned incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  unsigned short* q = queue + (incl - mine);
  for (; mask; mask &= mask - 1) {
    const int k = __ffs(mask) - 1;
    *q++ = (unsigned short)(kStrided ? 32 * k + lane : 128 * (k >> 2) + 4 * lane + (k & 3));
  }
  __syncwarp();
  return (int)__shfl_sync(0xffffffffu, incl, 31);
}

// initWL<true>; also zeroes inMST (:306). Where kScanDense or more of a task's
// entries are in question (no filter, or a high one) the detour through the
// queue costs more than it saves: then every lane looks up its entries in
// place, four neighbours a load.
template <bool VEC>
__global__ void __launch_bounds__(kScanThreads, kScanBlocks) k_scan_light(ScanArgs a) {
  extern __shared__ __align__(16) unsigned char scan_dyn[];
  ScanSmem<true>& sm = *reinterpret_cast<ScanSmem<true>*>(scan_dyn);
  DevState* st = a.st;
  if (ld_volatile(&st->error) & kErrFormat) return;  // set by k_prep only
  const int n = a.nodes, m = a.edges, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto& ws = sm.warp[warp];
  const int thr = st->threshold;
  const unsigned t0 = st->split_light, t1 = st->split_heavy;
  const bool mid = st->mid != 0, nlist_vec = (((uintptr_t)a.nlist) & 15) == 0;
  const int last = mid ? kListMid : (t0 != 0xffffffffu ? kListLight1 : kListLight0);
  // no entry above this weight goes to any list
  const int top = mid ? max(thr, (int)min(t1, (unsigned)INT_MAX)) : thr;
  const u64 stream_pol = l2_policy_evict_first();
  scan_open(a, sm, ws);
  const int stride = gridDim.x * kScanWarps;
  int t = blockIdx.x * kScanWarps + warp;
#pragma unroll
  for (int s = 0; s < kScanStages; s++) scan_fill<VEC>(a, ws, a.eweight, t + s * stride, s, stream_pol);
  TaskRows rows = task_rows(a, t), next = task_rows(a, t + stride);
  slice_start(a, rows, ws.slice[0]);
  bool bad = false;
  int s = 0, buf = 0;
  unsigned parity = 0;
  // list of an entry of weight w
  auto list_of = [&](int w) -> unsigned {
    return w <= thr ? ((unsigned)w <= t0 ? (unsigned)kListLight0 : (unsigned)kListLight1)
                    : (mid && (unsigned)w <= t1 ? (unsigned)kListMid : 15u);
  };
#pragma unroll 1
  for (; t < a.tiles; t += stride) {
    const int j0 = t * kGran, cnt = min(kGran, m - j0);
    if (!scan_wait(a, ws, s, parity)) break;
    const int* slice = ws.slice[buf];
    slice_start(a, next, ws.slice[buf ^ 1]);
    const TaskRows after = task_rows(a, t + 2 * stride);
    const int* data = ws.data[s];
    unsigned mask = 0;  // four entries at 128 * i + 4 * lane
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int4 y = *reinterpret_cast<const int4*>(data + 128 * i + 4 * lane);
      mask |= (unsigned)(y.x <= top) << (4 * i) | (unsigned)(y.y <= top) << (4 * i + 1) |
              (unsigned)(y.z <= top) << (4 * i + 2) | (unsigned)(y.w <= top) << (4 * i + 3);
    }
    if (cnt < kGran) {
#pragma unroll
      for (int i = 0; i < 16; i++)
        if (128 * (i >> 2) + 4 * lane + (i & 3) >= cnt) mask &= ~(1u << i);
    }
    if (a.zero_vec && cnt == kGran) {
      *reinterpret_cast<uint4*>(a.inMST + j0 + 16 * lane) = make_uint4(0u, 0u, 0u, 0u);
    } else {
      for (int q = lane; q < cnt; q += 32) a.inMST[j0 + q] = 0;
    }
    if (__reduce_add_sync(0xffffffffu, __popc(mask)) >= kScanDense) {
      int4 nb[4];
#pragma unroll
      for (int g = 0; g < 4; g++) {
        const int at = 128 * g + 4 * lane, *p = a.nlist + j0 + at;
        if (nlist_vec && at + 4 <= cnt) {
          nb[g] = __ldcs(reinterpret_cast<const int4*>(p));
        } else {
          nb[g].x = at < cnt ? __ldg(p) : 0;
          nb[g].y = at + 1 < cnt ? __ldg(p + 1) : 0;
          nb[g].z = at + 2 < cnt ? __ldg(p + 2) : 0;
          nb[g].w = at + 3 < cnt ? __ldg(p + 3) : 0;
        }
      }
#pragma unroll 1
      for (int g = 0; g < 4; g++) {
        const int at = 128 * g + 4 * lane;
        // the row of the first, then on along nindex
        int lo = 0, hi = rows.hi - rows.lo;
        while (lo < hi) {
          const int mid_row = lo + ((hi - lo + 1) >> 1);
          if (slice_at(a, rows, slice, mid_row) <= j0 + at) lo = mid_row;
          else hi = mid_row - 1;
        }
        auto first = [&](int r) { return slice_at(a, rows, slice, r); };
        const int top = rows.hi - rows.lo;
        int row = lo, end = row < top ? first(row + 1) : INT_MAX;
        const int4 y = g == 0 ? nb[0] : g == 1 ? nb[1] : g == 2 ? nb[2] : nb[3];
        const int ends[4] = {y.x, y.y, y.z, y.w};
        int4 e[4];
        unsigned cls = 0xffffu;
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int j = j0 + at + i;
          row_on(first, [&](int lo, int hi) { return last_row(first, lo, hi, j); }, top, j, row, end);
          const int v = rows.lo + row;
          e[i] = make_int4(v, ends[i], data[at + i], j0 + at + i);
          const bool on = (mask >> (4 * g + i)) & 1u;
          bad |= on && (unsigned)ends[i] >= (unsigned)n;
          // one direction with a valid id (v < nb < n) as one unsigned compare
          if (on && (unsigned)ends[i] - (unsigned)v - 1u < (unsigned)(n - v - 1))
            cls ^= (15u ^ list_of(e[i].z)) << (4 * i);
        }
        lists_append<4>(a, sm.chunk, sm.kept, kListLight0, last, cls, e);
      }
    } else {
      int total = scan_gather<false>(mask, ws.queue);
      // the neighbours of the entries in question; those not beyond the task's
      // first row are the other direction and leave the queue
      int kept = 0;
#pragma unroll 1
      for (int base = 0; base < total; base += 32 * kScanItems) {
        int k[kScanItems], nb[kScanItems];
#pragma unroll
        for (int i = 0; i < kScanItems; i++) {
          const bool on = base + 32 * i + lane < total;
          k[i] = on ? (int)ws.queue[base + 32 * i + lane] : 0;
          nb[i] = on ? __ldg(a.nlist + j0 + k[i]) : -1;
          bad |= on && (unsigned)nb[i] >= (unsigned)n;
        }
        __syncwarp();  // read before the queue is written (kept <= base)
#pragma unroll
        for (int i = 0; i < kScanItems; i++) {
          const bool fwd = nb[i] > rows.lo && nb[i] < n;
          const unsigned m32 = __ballot_sync(0xffffffffu, fwd);
          if (fwd) {
            const int at = kept + __popc(m32 & ((1u << lane) - 1u));
            ws.queue[at] = (unsigned short)k[i];
            ws.ends[at] = nb[i];
          }
          kept += __popc(m32);
        }
        __syncwarp();
      }
      total = kept;
      // and work them off
#pragma unroll 1
      for (int base = 0; base < total; base += 32 * kScanItems) {
        int v[kScanItems];
        int4 e[kScanItems];
        unsigned cls = 0xffu;  // no list
#pragma unroll
        for (int i = 0; i < kScanItems; i++) {
          const bool on = base + 32 * i + lane < total;
          const int k = on ? (int)ws.queue[base + 32 * i + lane] : 0;
          e[i] = make_int4(0, on ? ws.ends[base + 32 * i + lane] : -1, data[k], j0 + k);
        }
        rows_of(a, rows, slice, e, v);
#pragma unroll
        for (int i = 0; i < kScanItems; i++) {
          e[i].x = v[i];
          if (e[i].y > v[i]) cls ^= (15u ^ list_of(e[i].z)) << (4 * i);  // one direction
        }
        lists_append<kScanItems>(a, sm.chunk, sm.kept, kListLight0, last, cls, e);
      }
    }
    __syncwarp();  // the stage and the queue are free
    scan_fill<VEC>(a, ws, a.eweight, t + kScanStages * stride, s, stream_pol);
    if (++s == kScanStages) {
      s = 0;
      parity ^= 1u;
    }
    rows = next;
    next = after;
    buf ^= 1;
  }
  __pipeline_wait_prior(0);
  if (bad) atomicOr(&st->error, kErrFormat);  // a neighbour id outside [0, n)
  __syncthreads();
  for (int k = kListLight0; k <= last; k++) list_close(a, k, sm.chunk[k], sm.kept[k]);
}

// initWL<false>. In question: entries whose neighbour lies outside the largest
// tree, and all forward entries of the rows outside it (or of a task whose rows
// are more than kScanMaxRows, a run of empty ones too long to walk).
template <bool VEC>
__global__ void __launch_bounds__(kScanThreads, kScanBlocks) k_scan_heavy(ScanArgs a) {
  extern __shared__ __align__(16) unsigned char scan_dyn[];
  ScanSmem<false>& sm = *reinterpret_cast<ScanSmem<false>*>(scan_dyn);
  DevState* st = a.st;
  if (ld_volatile(&st->error) & kErrFormat) return;  // set by k_prep only
  if (!st->filtered) return;
  const int n = a.nodes, m = a.edges, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto& ws = sm.warp[warp];
  const unsigned* bits = a.tree_bits;
  const u64 stream_pol = l2_policy_evict_first(), keep_pol = l2_policy_evict_last();
  scan_open(a, sm, ws);
  const int stride = gridDim.x * kScanWarps;
  int t = blockIdx.x * kScanWarps + warp;
#pragma unroll
  for (int s = 0; s < kScanStages; s++) scan_fill<VEC>(a, ws, a.nlist, t + s * stride, s, stream_pol);
  TaskRows rows = task_rows(a, t), next = task_rows(a, t + stride);
  slice_start(a, rows, ws.slice[0]);
  bool bad = false;
  int s = 0, buf = 0;
  unsigned parity = 0;
#pragma unroll 1
  for (; t < a.tiles; t += stride) {
    const int j0 = t * kGran, cnt = min(kGran, m - j0);
    if (!scan_wait(a, ws, s, parity)) break;
    const int* slice = ws.slice[buf];
    slice_start(a, next, ws.slice[buf ^ 1]);
    const TaskRows after = task_rows(a, t + 2 * stride);
    const int* data = ws.data[s];
    int x[16];  // the entries at 32 * i + lane
#pragma unroll
    for (int i = 0; i < 16; i++) x[i] = data[32 * i + lane];
    if (cnt < kGran) {
#pragma unroll
      for (int i = 0; i < 16; i++)
        if (32 * i + lane >= cnt) x[i] = 0;  // never forward
    }
    const bool full = rows.hi - rows.lo > kScanMaxRows;
    // The task's rows start at rows.lo: ids up to it are the other direction.
    const unsigned low = (unsigned)rows.lo + 1u, span = (unsigned)n - low;
    unsigned most = 0, mask = 0;
#pragma unroll
    for (int h = 0; h < 16; h += 8) {
      unsigned w[8];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        most = max(most, (unsigned)x[h + i]);
        w[i] = ~0u;
        if ((unsigned)x[h + i] - low < span) w[i] = __ldg(bits + (x[h + i] >> 5));
      }
#pragma unroll
      for (int i = 0; i < 8; i++) mask |= (~__funnelshift_r(w[i], 0u, x[h + i]) & 1u) << (h + i);
    }
    bad |= most >= (unsigned)n;
    // entries of rows outside the tree, four words of rows at once
    bool any = full;
    if (!full) {
      const int first = rows.lo >> 5, words = (rows.hi >> 5) - first + 1;
      const unsigned mine = lane < words ? __ldg(bits + first + lane) : ~0u;
      unsigned some = __ballot_sync(0xffffffffu, mine != ~0u);
#pragma unroll 1
      while (some) {
        int b[4], e[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int k = some ? __ffs(some) - 1 : 0;
          const unsigned w = __shfl_sync(0xffffffffu, mine, k);
          const int v = 32 * (first + k) + lane;
          b[i] = e[i] = 0;
          if (some && v >= rows.lo && v <= rows.hi && !((w >> lane) & 1u)) {
            b[i] = max(slice[v - rows.lo] - j0, 0);
            e[i] = v < rows.hi ? min(slice[v + 1 - rows.lo] - j0, cnt) : cnt;
          }
          some &= some - 1;
        }
        if (!__any_sync(0xffffffffu, b[0] < e[0] || b[1] < e[1] || b[2] < e[2] || b[3] < e[3])) continue;
        if (!any) {
          if (lane < kGran / 32) ws.rows_out[lane] = 0;
          __syncwarp();
          any = true;
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
          for (int k = b[i] >> 5; b[i] < e[i] && k <= (e[i] - 1) >> 5; k++) {
            const unsigned from = k == b[i] >> 5 ? ~0u << (b[i] & 31) : ~0u;
            const unsigned to = k == (e[i] - 1) >> 5 ? ~0u >> (31 - ((e[i] - 1) & 31)) : ~0u;
            atomicOr(&ws.rows_out[k], from & to);
          }
      }
      __syncwarp();
    }
    if (any) {
      unsigned fwd = 0, out = full ? 0xffffu : 0u;
#pragma unroll
      for (int i = 0; i < 16; i++) fwd |= (unsigned)((unsigned)x[i] - low < span) << i;
      if (!full) {
#pragma unroll
        for (int i = 0; i < 16; i++) out |= ((ws.rows_out[i] >> lane) & 1u) << i;
      }
      mask |= fwd & out;
    }
    const int total = scan_gather<true>(mask, ws.queue);
#pragma unroll 1
    for (int base = 0; base < total; base += 32 * kScanItems) {
      int v[kScanItems];
      int4 e[kScanItems];
      unsigned cls = 0xffu;  // no list
#pragma unroll
      for (int i = 0; i < kScanItems; i++) {
        const bool on = base + 32 * i + lane < total;
        const int k = on ? (int)ws.queue[base + 32 * i + lane] : 0;
        const int y = on ? data[k] : -1;
        e[i] = make_int4(0, y, on ? ld_cg_hint(a.parent + y, keep_pol) : 0, j0 + k);
      }
      rows_of(a, rows, slice, e, v);
#pragma unroll
      for (int i = 0; i < kScanItems; i++)
        e[i].x = e[i].y > v[i] ? ld_cg_hint(a.parent + v[i], keep_pol) : e[i].z;
#pragma unroll
      for (int i = 0; i < kScanItems; i++) {
        e[i].y = e[i].z;  // the neighbour's tree
        if (e[i].x != e[i].y) {
          e[i].z = __ldg(a.eweight + e[i].w);
          cls ^= (15u ^ (unsigned)kListHeavy) << (4 * i);
        }
      }
      lists_append<kScanItems>(a, sm.chunk, sm.kept, kListHeavy, kListHeavy, cls, e);
    }
    __syncwarp();  // the stage and the queue are free
    scan_fill<VEC>(a, ws, a.nlist, t + kScanStages * stride, s, stream_pol);
    if (++s == kScanStages) {
      s = 0;
      parity ^= 1u;
    }
    rows = next;
    next = after;
    buf ^= 1;
  }
  __pipeline_wait_prior(0);
  if (bad) atomicOr(&st->error, kErrFormat);  // a neighbour id outside [0, n)
  __syncthreads();
  list_close(a, kListHeavy, sm.chunk[kListHeavy], sm.kept[kListHeavy]);
}

}  // namespace ecl
