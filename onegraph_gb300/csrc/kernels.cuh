// kernels.cuh — sm_103a kernels of the out-of-memory engine.
//
//  k_compact   frontier bitmap -> compacted vertex list + u64 degree prefix +
//              LBS tile map, one pass with a decoupled look-back scan.  Replaces
//              setStaticAndOverloadLabelBool / myReduction / myExclusive_scan /
//              setStaticActiveNodeArray / setOverloadNodePointerSwap and the
//              host degree scan (BFS/oneGraph_BFS/gpu_kernels.h:243-379,
//              CalculateOpt.h:78-124) and the Subway generator's
//              flag/scan/queue/pointer steps (PR/sbw/subgraph_generator.h:57-234).
//  k_lbs<Op>   edge-balanced ("load-balanced search") expansion: every CTA owns
//              2048 consecutive edge positions of the compacted list, whatever
//              the degrees; columns are read coalesced.  Op = BFS / SSSP / CC
//              relax (gpu_kernels.h:180-241, SSSP :106-203, CC :105-157) or
//              the dynamic-region gather from page-locked host memory
//              (GraphMeta.h:471-506 fillEdgeArrByMultiThread).
//  k_pr_*      PageRank pull sum with a deterministic segmented reduction
//              (PR/OneGraph/gpu_kernels.h:107-158) and the rank update with an
//              FP64 L1 reduction (gpu_kernels.h:295-319).
#pragma once
#include <cuda/atomic>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace og {

constexpr int kThreads = 256;
constexpr uint32_t kTile = 2048;             // LBS edge positions per CTA
constexpr uint32_t kItems = kTile / kThreads;  // 8
// largest compaction tile: 1024 bitmap words (32768 vertices); the planner and
// the bitmaps' padding are sized by it
constexpr uint32_t kWordsPerCompactTile = 1024;

// device error bits (OR-ed into the engine's error word)
constexpr uint32_t kErrLookback = 1u;    // look-back wait gave up
constexpr uint32_t kErrEdgeIndex = 2u;   // edge index outside the array
constexpr uint32_t kErrVertex = 4u;      // column >= V
constexpr uint32_t kErrTileMap = 8u;     // LBS tile map inconsistent

// Polls after which a wait within a launch gives up: 2^24 (several seconds) for
// waits on work of fixed size; between the phases of a whole query, which may
// read every edge, a poll more for every 64 edges (a phase that gets through 0.2 G
// edges a second still ends in time).
constexpr uint32_t kSpinLimit = 1u << 24;
inline uint32_t wait_limit(uint64_t E) {
  return (uint32_t)((kSpinLimit + E / 64) < (1ull << 31) ? kSpinLimit + E / 64 : 1ull << 31);
}
constexpr uint32_t kErrBarrier = 16u;  // a bounded wait within a launch gave up

// Nanosecond global timer (the same clock on every SM).
__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

struct Counts {
  uint32_t n;        // compacted vertices
  uint32_t far_min;  // near/far split: smallest value left for later rounds
  uint64_t total;    // sum of their degrees (edge positions)
};

// Look-back scratch: one 16-byte slot per compaction tile, written and read as
// a single 128-bit access, so a slot carries its own state, count and degree
// sum and no fence or second load is needed: x = (n << 32) | (epoch << 2) |
// state, y = degree sum; state 1 the tile's aggregate, 2 the inclusive prefix.
struct Lookback {
  ulonglong2 *slot;
  uint32_t *ticket;
};

struct CompactArgs {
  const uint32_t *bits;  // frontier bitmap
  uint32_t v_begin, v_end;
  uint32_t w_begin, w_end, ntiles;
  uint32_t tile_words;   // bitmap words per tile: 128, 256, 512 or 1024
  const uint64_t *off;   // CSR offsets (V+1) on the device
  uint32_t *list;
  uint64_t *pref;        // exclusive degree prefix, pref[n] = total
  uint32_t *tile_first;  // LBS tile -> list index of the vertex holding its first position
  Counts *counts;
  Lookback lb;
  uint32_t *err;
  uint64_t list_cap;     // entries of list (pref has list_cap + 1)
  uint64_t tile_cap;     // entries of tile_first
  // near/far split (SSSP): when split != 0 only vertices with value < thr
  // are listed; the others stay waiting: they are OR-ed into far_bits (when
  // not null) and the smallest of their values goes to *far_min.  Vertices
  // that leave the waiting state (value < thr) have their bit cleared in
  // clear_bits (when not null).  The value is read before the offsets, so a
  // waiting vertex costs 4 bytes.
  const uint32_t *value;
  uint32_t thr;
  uint32_t split;
  uint32_t *far_bits;
  // atomicMax of (epoch << 32) | ~value over the waiting vertices: a key of
  // an older epoch (or zeroed memory) is always smaller, and within an epoch
  // the largest ~value is the smallest value
  unsigned long long *far_key;
  uint32_t *clear_bits;
  // Launch epoch in [1, 2^30): status words of other epochs read as empty, so
  // the status array needs no clearing between launches.  The CTA that takes
  // the last ticket resets the ticket counter for the next launch.
  uint32_t epoch;
};

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
  return cuda::atomic_ref<const uint32_t, cuda::thread_scope_device>(*p).load(
      cuda::memory_order_acquire);
}
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *p) {
  return cuda::atomic_ref<const uint32_t, cuda::thread_scope_device>(*p).load(
      cuda::memory_order_relaxed);
}
__device__ __forceinline__ void st_release(uint32_t *p, uint32_t v) {
  cuda::atomic_ref<uint32_t, cuda::thread_scope_device>(*p).store(v, cuda::memory_order_release);
}

// Block-wide exclusive scan of (u32, u64) pairs; returns the block totals.
__device__ __forceinline__ void block_scan_pair(uint32_t cnt, uint64_t sum, uint32_t &ex_cnt,
                                                uint64_t &ex_sum, uint32_t &tot_cnt,
                                                uint64_t &tot_sum) {
  __shared__ uint32_t s_wc[kThreads / 32];
  __shared__ uint64_t s_ws[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t ic = cnt;
  uint64_t is = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t c = __shfl_up_sync(0xffffffffu, ic, d);
    const uint64_t s = __shfl_up_sync(0xffffffffu, is, d);
    if (lane >= d) {
      ic += c;
      is += s;
    }
  }
  if (lane == 31) {
    s_wc[warp] = ic;
    s_ws[warp] = is;
  }
  __syncthreads();
  if (warp == 0) {
    uint32_t wc = lane < kThreads / 32 ? s_wc[lane] : 0;
    uint64_t ws = lane < kThreads / 32 ? s_ws[lane] : 0;
#pragma unroll
    for (int d = 1; d < kThreads / 32; d <<= 1) {
      const uint32_t c = __shfl_up_sync(0xffffffffu, wc, d);
      const uint64_t s = __shfl_up_sync(0xffffffffu, ws, d);
      if (lane >= d) {
        wc += c;
        ws += s;
      }
    }
    if (lane < kThreads / 32) {
      s_wc[lane] = wc;  // inclusive warp prefixes
      s_ws[lane] = ws;
    }
  }
  __syncthreads();
  const uint32_t wpc = warp ? s_wc[warp - 1] : 0;
  const uint64_t wps = warp ? s_ws[warp - 1] : 0;
  ex_cnt = wpc + ic - cnt;
  ex_sum = wps + is - sum;
  tot_cnt = s_wc[kThreads / 32 - 1];
  tot_sum = s_ws[kThreads / 32 - 1];
  __syncthreads();  // shared arrays are reused by the next call
}

__device__ __forceinline__ ulonglong2 ld_slot(const ulonglong2 *p) {
  ulonglong2 r;
  asm volatile(
      "{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
      : "=l"(r.x), "=l"(r.y)
      : "l"(p)
      : "memory");
  return r;
}
__device__ __forceinline__ void st_slot(ulonglong2 *p, uint32_t epoch, uint32_t state, uint32_t n, uint64_t e) {
  const unsigned long long x = ((unsigned long long)n << 32) | (epoch << 2) | state;
  asm volatile(
      "{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
      "l"(x), "l"((unsigned long long)e)
      : "memory");
}

// Warp-wide decoupled look-back of compaction tile `tile` (called by all 32
// lanes of warp 0): publishes the tile's totals (tot_n, tot_e) and returns in
// (pn, pe) the exclusive prefix of the tiles before it.  Each pass reads the
// slots of the 32 nearest unaccounted predecessors at once, sums their
// aggregates up to the nearest one holding an inclusive prefix, and stops
// there; tiles before the first count as an inclusive prefix of 0.  Waits
// are bounded by `spin_limit` polls: a slot that never appears sets
// kErrLookback in *err and bad = 1 (the caller then writes nothing), and the
// tile still publishes an inclusive prefix so that successors never wait
// forever.
__device__ __forceinline__ void lookback_prefix(const Lookback &lb, uint32_t tile, uint32_t epoch,
                                                uint32_t tot_n, uint64_t tot_e, uint32_t *err,
                                                uint32_t &pn, uint64_t &pe, int &bad,
                                                uint32_t spin_limit = kSpinLimit) {
  const int lane = threadIdx.x & 31;
  pn = 0;
  pe = 0;
  bad = 0;
  if (tile == 0) {
    if (lane == 0) st_slot(lb.slot, epoch, 2u, tot_n, tot_e);
    return;
  }
  if (lane == 0) st_slot(lb.slot + tile, epoch, 1u, tot_n, tot_e);
  for (int p = (int)tile - 1;; p -= 32) {
    const int q = p - lane;  // lane 0: nearest predecessor of the window
    uint32_t st = 2u, vn = 0;
    uint64_t ve = 0;
    if (q >= 0) {
      uint32_t spins = 0;
      for (;;) {
        const ulonglong2 v = ld_slot(lb.slot + q);
        st = ((uint32_t)v.x >> 2) == epoch ? ((uint32_t)v.x & 3u) : 0u;
        vn = (uint32_t)(v.x >> 32);
        ve = v.y;
        if (st != 0u || ++spins > spin_limit) break;
        __nanosleep(32);
      }
    }
    __syncwarp();
    if (__any_sync(0xffffffffu, st == 0u)) {  // bounded wait expired: report, never hang
      if (lane == 0) atomicOr(err, kErrLookback);
      bad = 1;
      break;
    }
    const unsigned incl = __ballot_sync(0xffffffffu, st == 2u);
    const int k = incl ? __ffs(incl) - 1 : 32;
    if (q < 0 || lane > k) {
      vn = 0;
      ve = 0;
    }
    vn = __reduce_add_sync(0xffffffffu, vn);
#pragma unroll
    for (int o = 16; o; o >>= 1) ve += __shfl_xor_sync(0xffffffffu, ve, o);
    pn += vn;
    pe += ve;
    if (k < 32) break;
  }
  if (lane == 0) st_slot(lb.slot + tile, epoch, 2u, pn + tot_n, pe + tot_e);  // published even when bad
}

// Block-wide exclusive scan of u32 counts; returns the block total.  Callers
// put a barrier between two calls.
__device__ __forceinline__ uint32_t block_scan_u32(uint32_t cnt, uint32_t &ex) {
  __shared__ uint32_t s_w[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t ic = cnt;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t c = __shfl_up_sync(0xffffffffu, ic, d);
    if (lane >= d) ic += c;
  }
  if (lane == 31) s_w[warp] = ic;
  __syncthreads();
  uint32_t wp = 0, tot = 0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; w++) {
    const uint32_t x = s_w[w];
    wp += w < warp ? x : 0u;
    tot += x;
  }
  ex = wp + ic - cnt;
  return tot;
}

// ------------------------------------------------------------- compaction
//
// Frontier compaction of a vertex range: bitmap words -> vertex list in
// increasing id order, u64 degree prefix and LBS tile map, one pass with a
// decoupled look-back.  A CTA's tile is tile_words bitmap words.  The set
// bits are first listed in shared memory, kListPass at a time, and the list
// entries (not the words) are then spread over the threads, so that a dense
// frontier costs a thread eight independent vertices per pass instead of a
// serial walk of 128, and a sparse one keeps one load per lane in flight.
// Bound: the dependent chain words -> (value ->) offsets -> look-back when the
// frontier is sparse, the 16 B of offsets and 12 B of list per vertex when it
// is dense.  With four words walked by each thread (the earlier form) an
// 8-source SSSP pass over 2^20 vertices spent 0.4 ms per compaction on 32 CTAs;
// this form took the pass from 7.2 to 2.8 ms and a resident SSSP query of 0.3 M
// vertices (108 compactions) from 2.4 to 1.95 ms.  64 registers (4 CTAs per SM):
// left to itself the compiler takes 118, which halves the CTAs in flight and
// costs 5 % of an SSSP query over 2^24 vertices.  Sel says which vertices are
// listed:
//  pre(v)                 v's state
//  want(pre)              whether its degree matters
//  settle(v, pre, d, far, clr)  the degree d when v is listed, else 0; far /
//                         clr: v's bit belongs in the far / cleared words
//  flush(w, far, clr)     those words, once per bitmap word
//  finish(tid)            per-thread reductions (all threads, has barriers)
//  emit(v, pos)           v is list entry pos
constexpr uint32_t kListPass = 8 * kThreads;
constexpr uint16_t kDropped = 0xffffu;

struct CompactShared {
  uint32_t word[kWordsPerCompactTile];   // scanned bits, later the listed ones
  uint32_t far[kWordsPerCompactTile], clr[kWordsPerCompactTile];
  uint32_t drop[kWordsPerCompactTile];   // scanned but not listed (several passes)
  uint16_t wbase[kWordsPerCompactTile];  // set bits before each word
  uint16_t list[kListPass];              // tile-local vertex of each entry of the pass
  uint16_t rank[kListPass];              // its list rank within the pass, or kDropped
  uint64_t pref[kListPass + kThreads + 1];  // its degree, then the exclusive prefix (padded: at())
  uint32_t tile, excl_n;
  uint64_t excl_e;
  int bad;
  // eight consecutive entries per thread, one pad per eight: no bank conflicts
  __device__ __forceinline__ static uint32_t at(uint32_t i) { return i + (i >> 3); }
};

// Set-bit ranks of the tile's words: returns the total, own first rank in ex.
__device__ __forceinline__ uint32_t compact_ranks(CompactShared &sh, uint32_t wpt, uint32_t w0, uint32_t nw,
                                                  uint32_t &pc, uint32_t &ex) {
  pc = 0;
  for (uint32_t j = 0; j < wpt; j++)
    if (w0 + j < nw) pc += __popc(sh.word[w0 + j]);
  const uint32_t N = block_scan_u32(pc, ex);
  uint32_t r = ex;
  for (uint32_t j = 0; j < wpt; j++)
    if (w0 + j < nw) {
      sh.wbase[w0 + j] = (uint16_t)r;
      r += __popc(sh.word[w0 + j]);
    }
  __syncthreads();
  return N;
}

// Lists the set bits of ranks [p0, p0 + kListPass).  Dense words are listed
// a warp per word, sparse ones by the threads that own them.
__device__ __forceinline__ void compact_list(CompactShared &sh, uint32_t wpt, uint32_t w0, uint32_t nw, uint32_t N,
                                             uint32_t pc, uint32_t ex, uint32_t p0) {
  if (N > 4 * nw) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t w = threadIdx.x >> 5; w < nw; w += kThreads / 32) {
      const uint32_t r = sh.wbase[w];
      if (r >= p0 + kListPass || r + 32 <= p0) continue;
      const uint32_t m = sh.word[w];
      const uint32_t k = r + __popc(m & ((1u << lane) - 1u)) - p0;
      if (((m >> lane) & 1u) && k < kListPass) sh.list[k] = (uint16_t)(w * 32 + lane);
    }
  } else if (ex < p0 + kListPass && ex + pc > p0) {
    uint32_t k = ex - p0;
    for (uint32_t j = 0; j < wpt; j++)
      if (w0 + j < nw)
        for (uint32_t m = sh.word[w0 + j]; m; m &= m - 1, k++)
          if (k < kListPass) sh.list[k] = (uint16_t)((w0 + j) * 32 + __ffs(m) - 1);
  }
  __syncthreads();
}

// Degrees in sh.pref -> ranks and exclusive prefixes; returns the pass totals.
__device__ __forceinline__ void compact_scan(CompactShared &sh, uint32_t m, uint32_t &tn, uint64_t &te) {
  const uint32_t i0 = threadIdx.x * 8;
  uint64_t d[8];
  uint32_t cnt = 0;
  uint64_t sum = 0;
#pragma unroll
  for (uint32_t i = 0; i < 8; i++) {
    d[i] = i0 + i < m ? sh.pref[CompactShared::at(i0 + i)] : 0;
    cnt += d[i] ? 1u : 0u;
    sum += d[i];
  }
  uint32_t exn;
  uint64_t exe;
  block_scan_pair(cnt, sum, exn, exe, tn, te);
#pragma unroll
  for (uint32_t i = 0; i < 8; i++)
    if (i0 + i < m) {
      sh.rank[i0 + i] = d[i] ? (uint16_t)exn : kDropped;
      sh.pref[CompactShared::at(i0 + i)] = exe;
      exn += d[i] ? 1u : 0u;
      exe += d[i];
      if (i0 + i + 1 == m) sh.pref[CompactShared::at(m)] = exe;
    }
  __syncthreads();
}

// Writes the pass's listed entries at list position base_n, degree base_e.
template <class Args, class Sel>
__device__ __forceinline__ void compact_emit(const Args &a, Sel &sel, const CompactShared &sh, uint64_t vbase,
                                             uint32_t m, uint32_t base_n, uint64_t base_e) {
  for (uint32_t x = threadIdx.x; x < (m + 31) / 32 * 32; x += kThreads) {
    const bool on = x < m && sh.rank[x] != kDropped;
    uint32_t pos = 0;
    uint64_t t = 0, te = 0;  // tiles that start inside this vertex
    if (on) {
      const uint64_t v = vbase + sh.list[x];
      const uint64_t ep = base_e + sh.pref[CompactShared::at(x)];
      pos = base_n + sh.rank[x];
      a.list[pos] = (uint32_t)v;
      a.pref[pos] = ep;
      t = (ep + kTile - 1) / kTile;
      te = (base_e + sh.pref[CompactShared::at(x + 1)] + kTile - 1) / kTile;
      if (te > a.tile_cap) {
        atomicOr(a.err, kErrTileMap);
        te = a.tile_cap;
      }
      sel.emit(v, pos);
    }
    // a hub's tiles are written by the whole warp
    const uint32_t big = __ballot_sync(0xffffffffu, te > t + 8);
    if (te <= t + 8)
      for (; t < te; t++) a.tile_first[t] = pos;
    for (uint32_t b = big; b; b &= b - 1) {
      const int l = __ffs(b) - 1;
      const uint64_t ts = __shfl_sync(0xffffffffu, t, l), tend = __shfl_sync(0xffffffffu, te, l);
      const uint32_t p = __shfl_sync(0xffffffffu, pos, l);
      for (uint64_t q = ts + (threadIdx.x & 31); q < tend; q += 32) a.tile_first[q] = p;
    }
  }
}

template <class Args, class Sel>
__device__ __forceinline__ void compact_tile(const Args &a, Sel &sel, CompactShared &sh) {
  if (threadIdx.x == 0) {
    sh.tile = atomicAdd(a.lb.ticket, 1u);
    if (sh.tile == a.ntiles - 1) *a.lb.ticket = 0u;  // every CTA of this launch has its ticket
  }
  __syncthreads();
  const uint32_t tile = sh.tile;
  const uint32_t wpt = a.tile_words <= kThreads ? 1u : a.tile_words / kThreads;  // words per thread
  const uint32_t wt = a.w_begin + tile * a.tile_words;
  const uint32_t nw = min(a.tile_words, a.w_end - wt);
  const uint32_t w0 = threadIdx.x * wpt;
  const uint64_t vbase = (uint64_t)wt * 32;
  uint32_t wv[kWordsPerCompactTile / kThreads];  // all of a thread's words in flight together
#pragma unroll
  for (uint32_t j = 0; j < kWordsPerCompactTile / kThreads; j++) {
    const uint32_t l = j * kThreads + threadIdx.x;
    wv[j] = l < nw ? a.bits[wt + l] : 0u;
  }
  uint32_t any = 0;
#pragma unroll
  for (uint32_t j = 0; j < kWordsPerCompactTile / kThreads; j++) {
    const uint32_t l = j * kThreads + threadIdx.x;
    if (l >= nw) break;
    uint32_t word = wv[j];
    const uint64_t vb = vbase + 32ull * l;
    if (vb < a.v_begin) {
      const uint32_t s = a.v_begin - (uint32_t)vb;
      word = s >= 32 ? 0 : word & (0xffffffffu << s);
    }
    if (vb + 32 > a.v_end) {
      const uint64_t k = a.v_end > vb ? a.v_end - vb : 0;
      word = k >= 32 ? word : word & ((1u << k) - 1u);
    }
    sh.word[l] = word;
    sh.far[l] = 0;
    sh.clr[l] = 0;
    sh.drop[l] = 0;
    any |= word;
  }
  uint32_t pc, ex, N = 0;
  if (__syncthreads_or(any)) N = compact_ranks(sh, wpt, w0, nw, pc, ex);  // most tiles of a sparse frontier are empty
  uint32_t tot_n = 0;
  uint64_t tot_e = 0;
  for (uint32_t p0 = 0; p0 < N; p0 += kListPass) {
    const uint32_t m = min(kListPass, N - p0);
    compact_list(sh, wpt, w0, nw, N, pc, ex, p0);
    // three phases, so that a thread's eight state loads and then its eight
    // offset pairs are in flight together
    uint32_t lv[8];
    typename Sel::Pre pre[8];
    uint64_t d[8];
#pragma unroll
    for (uint32_t j = 0; j < 8; j++) {
      const uint32_t x = j * kThreads + threadIdx.x;
      lv[j] = x < m ? sh.list[x] : 0xffffffffu;
      if (x < m) pre[j] = sel.pre(vbase + lv[j]);
    }
#pragma unroll
    for (uint32_t j = 0; j < 8; j++) {
      d[j] = 0;
      if (lv[j] != 0xffffffffu && sel.want(pre[j])) d[j] = a.off[vbase + lv[j] + 1] - a.off[vbase + lv[j]];
    }
#pragma unroll
    for (uint32_t j = 0; j < 8; j++) {
      if (lv[j] == 0xffffffffu) break;
      bool far = false, clr = false;
      const uint32_t l = lv[j];
      sh.pref[CompactShared::at(j * kThreads + threadIdx.x)] = sel.settle(vbase + l, pre[j], d[j], far, clr);
      if (far) atomicOr(&sh.far[l >> 5], 1u << (l & 31));
      if (clr) atomicOr(&sh.clr[l >> 5], 1u << (l & 31));
    }
    __syncthreads();
    uint32_t tn;
    uint64_t te;
    compact_scan(sh, m, tn, te);
    tot_n += tn;
    tot_e += te;
    if (N > kListPass) {  // several passes: the listed bits are listed again below
      for (uint32_t x = threadIdx.x; x < m; x += kThreads)
        if (sh.rank[x] == kDropped) atomicOr(&sh.drop[sh.list[x] >> 5], 1u << (sh.list[x] & 31));
      __syncthreads();
    }
  }
  if (N) {
    for (uint32_t l = threadIdx.x; l < nw; l += kThreads)
      if (sh.far[l] | sh.clr[l]) sel.flush(wt + l, sh.far[l], sh.clr[l]);
    sel.finish();
  }
  if (threadIdx.x < 32) {
    uint32_t pn = 0;
    uint64_t pe = 0;
    int bad = 0;
    lookback_prefix(a.lb, tile, a.epoch, tot_n, tot_e, a.err, pn, pe, bad);
    if (threadIdx.x == 0) {
      if (!bad && (uint64_t)pn + tot_n > a.list_cap) {
        atomicOr(a.err, kErrTileMap);
        bad = 1;
      }
      sh.excl_n = pn;
      sh.excl_e = pe;
      sh.bad = bad;
      if (!bad && tile == a.ntiles - 1) {
        a.counts->n = pn + tot_n;
        a.counts->total = pe + tot_e;
        a.pref[pn + tot_n] = pe + tot_e;
      }
    }
  }
  __syncthreads();
  if (sh.bad || tot_n == 0) return;  // bad: positions unknown, write nothing
  uint32_t base_n = sh.excl_n;
  uint64_t base_e = sh.excl_e;
  if (N <= kListPass) {
    compact_emit(a, sel, sh, vbase, N, base_n, base_e);
    return;
  }
  for (uint32_t l = threadIdx.x; l < nw; l += kThreads) sh.word[l] &= ~sh.drop[l];
  __syncthreads();
  compact_ranks(sh, wpt, w0, nw, pc, ex);
  for (uint32_t p0 = 0; p0 < tot_n; p0 += kListPass) {
    const uint32_t m = min(kListPass, tot_n - p0);
    compact_list(sh, wpt, w0, nw, tot_n, pc, ex, p0);
#pragma unroll 4
    for (uint32_t x = threadIdx.x; x < m; x += kThreads) {
      const uint64_t v = vbase + sh.list[x];
      sh.pref[CompactShared::at(x)] = a.off[v + 1] - a.off[v];
    }
    __syncthreads();
    uint32_t tn;
    uint64_t te;
    compact_scan(sh, m, tn, te);
    compact_emit(a, sel, sh, vbase, m, base_n, base_e);
    base_n += tn;
    base_e += te;
    __syncthreads();  // the next pass rewrites the shared list
  }
}

// Smallest of a per-thread value over the CTA (the result is thread 0's).
__device__ __forceinline__ uint32_t block_min_u32(uint32_t x) {
  __shared__ uint32_t s_m[kThreads / 32];
  const uint32_t w = __reduce_min_sync(0xffffffffu, x);
  if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5] = w;
  __syncthreads();
  uint32_t m = 0xffffffffu;
  if (threadIdx.x == 0)
#pragma unroll
    for (int i = 0; i < kThreads / 32; i++) m = min(m, s_m[i]);
  return m;
}

struct CompactSel {
  const CompactArgs &a;
  uint32_t tmin;  // smallest waiting value of this thread
  using Pre = uint32_t;
  __device__ __forceinline__ Pre pre(uint64_t v) const { return a.split ? __ldcg(a.value + v) : 0u; }
  __device__ __forceinline__ bool want(Pre x) const { return !a.split || x < a.thr; }
  __device__ __forceinline__ uint64_t settle(uint64_t, Pre x, uint64_t d, bool &far, bool &clr) {
    if (a.split) {
      far = x >= a.thr;
      clr = !far;
      if (far) tmin = min(tmin, x);
    }
    return d;
  }
  __device__ __forceinline__ void flush(uint32_t w, uint32_t far, uint32_t clr) const {
    if (far && a.far_bits) atomicOr(a.far_bits + w, far);
    if (clr && a.clear_bits) atomicAnd(a.clear_bits + w, ~clr);
  }
  __device__ __forceinline__ void finish() const {  // one far-key atomic per CTA
    if (!a.split) return;
    const uint32_t m = block_min_u32(tmin);
    if (m != 0xffffffffu && a.far_key)
      atomicMax(a.far_key, ((unsigned long long)a.epoch << 32) | (~m & 0xffffffffu));
  }
  __device__ __forceinline__ void emit(uint64_t, uint32_t) const {}
};

// Both regions' compactions in one launch: the first r[0].ntiles CTAs take
// region 0's tiles, the others region 1's (ntiles = 0: the region is empty and
// its counts are cleared).  Two launches on two streams needed four event
// operations more a round (ten rounds of eight-source SSSP over 2^20
// vertices: 2.29 ms, 2.25 in one launch).
template <class Args>
struct CompactPair {
  Args r[2];
};
template <class Args>
__device__ __forceinline__ const Args &compact_region(const CompactPair<Args> &p) {
  if (blockIdx.x == 0 && threadIdx.x < 2 && p.r[threadIdx.x].ntiles == 0 && p.r[threadIdx.x].counts)
    *p.r[threadIdx.x].counts = Counts{0, 0, 0};
  return p.r[blockIdx.x >= p.r[0].ntiles];
}

__global__ void __launch_bounds__(kThreads, 4) k_compact(const __grid_constant__ CompactPair<CompactArgs> p) {
  __shared__ CompactShared sh;
  const CompactArgs &a = compact_region(p);
  CompactSel sel{a, 0xffffffffu};
  compact_tile(a, sel, sh);
}

// Copies n <= 32 16-byte words to page-locked host memory (seen by the host once
// the stream is waited for).  A copy-engine transfer of 80 bytes starts 5-11 us
// after the kernel before it and takes 1.5 (the same ten rounds: 2.25 ms with
// it, 2.20 so).
__global__ void k_publish(const uint4 *src, uint4 *host, uint32_t n) {
  if (threadIdx.x < n) host[threadIdx.x] = __ldcg(src + threadIdx.x);
}

// ------------------------------------------------------------------ LBS

struct LbsArgs {
  const uint32_t *list;
  const uint64_t *pref;
  const uint32_t *tile_first;
  uint32_t n;            // list length
  uint64_t total;        // pref[n]
  uint64_t pos_begin;    // multiple of kTile
  uint64_t pos_end;
  const uint64_t *off;   // CSR mode: edge index = off[v] - pref[i] + q
  uint64_t stage_base;   // staging mode (off == nullptr): index = q - stage_base
  uint64_t edge_bound;   // entries addressable through the edge pointer
  uint32_t *err;
};

// Edge sources.  Staging buffers hold unpacked edges: u32 columns plus, for
// weighted graphs, weights in the narrowest width that holds them (W =
// uint8_t / uint16_t / uint32_t).  The static region and the page-locked host
// copy hold bit-packed records (SrcP).  A source yields one edge as a u32
// column or a {column, weight} pair; BFS, CC and PageRank read columns only.
//
// The LBS tiles address a vertex's edges through a cursor: cur(e) is the
// cursor of edge index e, at(c, x) the edge x positions after cursor c.
// Unpacked sources use the edge index itself; packed records use the bit
// offset, so a position costs a 32-bit multiply and a 64-bit add instead of a
// 64-bit multiply.  Cursor arithmetic is modulo 2^64 (a vertex that starts
// after the tile's first position has a "negative" base).
struct SrcU {
  using Item = uint32_t;
  const uint32_t *col;
  __device__ __forceinline__ Item load(uint64_t i) const { return col[i]; }
  __device__ __forceinline__ uint64_t cur(uint64_t e) const { return e; }
  __device__ __forceinline__ Item at(uint64_t c, uint32_t x) const { return col[c + x]; }
};
template <class W>
struct SrcW {
  using Item = uint2;
  const uint32_t *col;
  const W *w;
  __device__ __forceinline__ Item load(uint64_t i) const { return make_uint2(col[i], (uint32_t)w[i]); }
  __device__ __forceinline__ uint64_t cur(uint64_t e) const { return e; }
  __device__ __forceinline__ Item at(uint64_t c, uint32_t x) const { return load(c + x); }
};
// Bit-packed records (the page-locked host copy and the static region):
// record i holds bits [i*bpe, (i+1)*bpe) of `words`, column in the low bc
// bits, weight - wmin above it.  A record spans at most two words when
// bpe <= 33, else three; arrays carry two padding words at the end, so the
// reads below stay inside the array for every i below the record count.
// Consecutive lanes read consecutive records: the two loads of a warp touch
// the same bpe*4 contiguous bytes.
template <bool kW>
struct SrcP {
  using Item = typename std::conditional<kW, uint2, uint32_t>::type;
  const uint32_t *words;
  uint32_t bpe, bc, wmin;
  __device__ __forceinline__ uint64_t bits(uint64_t i) const {
    const uint64_t b = i * bpe;
    const uint64_t q = b >> 5;
    const uint32_t r = (uint32_t)b & 31u;
    uint64_t x = (((uint64_t)words[q + 1] << 32) | words[q]) >> r;
    if (r + bpe > 64) x |= (uint64_t)words[q + 2] << (64 - r);
    return x;
  }
  __device__ __forceinline__ Item load(uint64_t i) const {
    const uint64_t x = bits(i);
    const uint32_t col = bc >= 32 ? (uint32_t)x : (uint32_t)x & ((1u << bc) - 1u);
    if constexpr (kW) {
      const uint32_t bw = bpe - bc;
      const uint64_t w = bw == 0 ? 0 : (x >> bc) & ((bw >= 32) ? 0xffffffffull : ((1ull << bw) - 1));
      return make_uint2(col, (uint32_t)w + wmin);
    } else {
      return col;
    }
  }
  __device__ __forceinline__ uint64_t cur(uint64_t e) const { return e * bpe; }
  // x below 2^26 / bpe (a tile's positions).  The column is the low bc <= 32
  // bits of the record, so two words and one funnel shift hold it whatever
  // bpe is; a weight above it may need a third word.
  __device__ __forceinline__ Item at(uint64_t c, uint32_t x) const {
    const uint64_t b = c + x * bpe;
    return decode(words + (b >> 5), (uint32_t)b & 31u);
  }
  // The record starting at bit r of w[0] (w[1], w[2] hold its rest).
  __device__ __forceinline__ Item decode(const uint32_t *w, uint32_t r) const {
    const uint32_t lo = w[0], hi = w[1];
    const uint32_t f = __funnelshift_r(lo, hi, r);
    const uint32_t col = bc >= 32 ? f : f & ((1u << bc) - 1u);
    if constexpr (kW) {
      const uint32_t bw = bpe - bc;
      uint64_t y = (((uint64_t)hi << 32) | lo) >> r;
      if (r + bpe > 64) y |= (uint64_t)w[2] << (64 - r);
      const uint64_t wt = bw == 0 ? 0 : (y >> bc) & ((bw >= 32) ? 0xffffffffull : ((1ull << bw) - 1));
      return make_uint2(col, (uint32_t)wt + wmin);
    } else {
      return col;
    }
  }
};

// The columns of up to four consecutive records from bit `b` of the stream on
// (bpe <= 32), for lanes that each read a list of their own: such reads cost
// the L1 one tag lookup a lane and load, so the records come as one or two
// aligned 16-byte loads instead of eight words, and are shifted out of a
// 128-bit window.  `n` (0 to 4) records are wanted; the second load is made
// only if they reach into it, and what lies beyond them is not used.  The
// arrays are readable to a 16-byte boundary.  Measured: level 4 of a resident
// 2^20-vertex R-MAT (1.8 M records) 16 -> 14 us, a 64-source batch over 2^23
// vertices 12.9 -> 11.0 ms.
__device__ __forceinline__ void records4(const uint32_t *words, uint64_t b, uint32_t n, uint32_t bpe, uint32_t mask,
                                         uint32_t u[4]) {
  const uint4 *q = reinterpret_cast<const uint4 *>(words) + (b >> 7);
  const uint32_t r = (uint32_t)b & 127u;
  uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
  if (n) lo = q[0];
  if (r + n * bpe > 128u && n) hi = q[1];
  // window of four words from word r / 32 on, then from bit r % 32 on
  const bool s1 = r & 32u, s2 = r & 64u;
  uint32_t w[6] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y}, x[5];
  const uint32_t w6 = hi.z, w7 = hi.w;
  if (s2) {
    w[0] = w[2];
    w[1] = w[3];
    w[2] = w[4];
    w[3] = w[5];
    w[4] = w6;
    w[5] = w7;
  }
#pragma unroll
  for (int i = 0; i < 5; i++) x[i] = s1 ? w[i + 1] : w[i];
  const uint32_t sh = r & 31u;
#pragma unroll
  for (int i = 0; i < 4; i++) x[i] = __funnelshift_r(x[i], x[i + 1], sh);
#pragma unroll
  for (int j = 0; j < 4; j++) {
    u[j] = x[0] & mask;
    // shift the window by bpe (funnel shifts clamp at 32)
    x[0] = __funnelshift_rc(x[0], x[1], bpe);
    x[1] = __funnelshift_rc(x[1], x[2], bpe);
    x[2] = __funnelshift_rc(x[2], x[3], bpe);
    x[3] = __funnelshift_rc(x[3], 0u, bpe);
  }
}

// Dynamic-region records with fragment slots (the static-region replacement
// the reference declares as bfs_kernelStaticSwap / recordFragmentVisit,
// BFS/oneGraph_BFS/gpu_kernels.h:46-66,153-176): the page-locked record
// stream is cut into fragments of 2^fs words, and slot_of[f] >= 0 names a
// device slot holding a copy of fragment f followed by the stream's next
// words (a slot is 2^fs + kFragPad words), so a record whose first word lies
// in the fragment is read whole from the slot.  Other records are read from
// the host stream, which holds every record: slots only redirect reads, and
// results never depend on which fragments hold one.  The tile setup picks
// each vertex's source once (cur_range); note() counts, per fragment, the
// records a tile lists (by their first word); the host's replacement policy
// reads the counts between rounds.  The slot table only changes between
// launches.
constexpr uint32_t kFragPad = 4;  // words after a fragment's copy (keeps slots 16-byte aligned)
template <bool kW>
struct SrcF : SrcP<kW> {
  using Item = typename SrcP<kW>::Item;
  const uint32_t *slots;
  const int32_t *slot_of;
  uint32_t *visits;
  unsigned long long *miss;  // records of fragments with a slot that were read from the host copy
  uint32_t fs;
  // Cursors are absolute bit addresses (byte address x 8 + bit), so a
  // vertex's cursor points into its fragment's slot or into the host copy
  // and a record read needs no table lookup.  Device and host-mapped
  // addresses stay below 2^61, and a slot starts 16-byte aligned, so a
  // record's bit within its word is the same in both.
  __device__ __forceinline__ uint64_t cur(uint64_t e) const {
    return ((uint64_t)reinterpret_cast<uintptr_t>(this->words) << 3) + e * this->bpe;
  }
  // The cursor of edge index e for a vertex whose records in this tile are
  // [first, last]: into the slot when they all start in one fragment that
  // has one, else into the host copy.
  __device__ __forceinline__ uint64_t cur_range(uint64_t e, uint64_t first, uint64_t last) const {
    const uint64_t f = (first * this->bpe) >> (5 + fs);
    if (((last * this->bpe) >> (5 + fs)) == f) {
      const int32_t s = __ldg(slot_of + f);
      if (s >= 0) {
        const uint32_t *base = slots + (uint64_t)s * ((1ull << fs) + kFragPad);
        return ((uint64_t)reinterpret_cast<uintptr_t>(base) << 3) - (f << (5 + fs)) + e * this->bpe;
      }
    }
    return cur(e);
  }
  __device__ __forceinline__ Item at(uint64_t c, uint32_t x) const {
    const uint64_t b = c + x * this->bpe;
    return this->decode(reinterpret_cast<const uint32_t *>((uintptr_t)((b >> 5) << 2)), (uint32_t)b & 31u);
  }
  // cnt records from edge index e on: one visit count per fragment they start
  // in; a range over two fragments was read from the host copy, and its
  // records in fragments that have a slot are counted in *miss as well.
  __device__ __forceinline__ void note(uint64_t e, uint32_t cnt) const {
    uint64_t b = e * this->bpe;
    const bool split = (b >> (5 + fs)) != (((e + cnt - 1) * this->bpe) >> (5 + fs));
    while (cnt) {
      const uint64_t f = b >> (5 + fs);
      const uint32_t left = (uint32_t)(((f + 1) << (5 + fs)) - b);  // bits to the next fragment, < 2^26
      const uint32_t n = min(cnt, (left + this->bpe - 1) / this->bpe);
      atomicAdd(visits + f, n);
      if (split && __ldg(slot_of + f) >= 0) atomicAdd(miss, (unsigned long long)n);
      cnt -= n;
      b += (uint64_t)n * this->bpe;
    }
  }
};

// Copies fragment pairs[i].x of the record stream `words` (nwords words,
// padding included) into slot pairs[i].y: one CTA per pair.
__global__ void __launch_bounds__(kThreads) k_frag_fill(const uint32_t *words, uint64_t nwords, uint32_t *slots,
                                                        const uint2 *pairs, uint32_t n, uint32_t fs) {
  if (blockIdx.x >= n) return;
  const uint2 p = pairs[blockIdx.x];
  const uint64_t q0 = (uint64_t)p.x << fs;
  const uint64_t len = min((uint64_t)(1ull << fs) + kFragPad, nwords - min(nwords, q0));
  uint32_t *dst = slots + (uint64_t)p.y * ((1ull << fs) + kFragPad);
  // fragment starts are multiples of 2^fs >= 256 words and slots are
  // 16-byte aligned: whole uint4s first, then the tail
  const uint64_t n4 = len / 4;
  const uint4 *s4 = reinterpret_cast<const uint4 *>(words + q0);
  uint4 *d4 = reinterpret_cast<uint4 *>(dst);
  for (uint64_t i = threadIdx.x; i < n4; i += kThreads) d4[i] = s4[i];
  for (uint64_t i = n4 * 4 + threadIdx.x; i < len; i += kThreads) dst[i] = words[q0 + i];
}

// Slot table update after k_frag_fill: pairs[i] = (fragment, slot), and
// evict[i] the fragment that slot held before (UINT32_MAX: none).
__global__ void k_frag_table(int32_t *slot_of, const uint2 *pairs, const uint32_t *evict, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  // a fragment is never both evicted and filled in one update
  if (evict[i] != 0xffffffffu) slot_of[evict[i]] = -1;
  slot_of[pairs[i].x] = (int32_t)pairs[i].y;
}

struct DstU {
  uint32_t *col;
  __device__ __forceinline__ void store(uint64_t i, uint32_t x) const { col[i] = x; }
};
template <class W>
struct DstW {
  uint32_t *col;
  W *w;
  __device__ __forceinline__ void store(uint64_t i, uint2 x) const {
    col[i] = x.x;
    w[i] = (W)x.y;
  }
};

// Per-tile tables.  Most tiles hold far fewer vertices than positions, so the
// cursor and value tables have kLocal entries, and a tile with more vertices
// is worked off in parts of kThreads positions (which hold at most kThreads
// vertices each, plus one).  With tables for 2048 vertices a CTA took 37 KB of shared
// memory: four CTAs per SM and little L1.  kVal = false (BFS reads no source
// value) drops the value table.
constexpr uint32_t kLocal = 512;
template <class Val, bool kVal = true>
struct LbsShared {
  unsigned long long cb[kLocal];  // source cursor of tile position 0 for the vertex
  Val val[kVal ? kLocal : 1];     // source value of each local vertex
  alignas(16) unsigned short map[kTile];  // tile position -> local vertex
};

// Optional op hooks, detected at compile time:
//  list_val(v, e)   the source value belongs to the list entry at address e
//                   (an array parallel to the compacted list) instead of
//                   src_val(v);
//  probe_v(e, val)  the probe also sees the source value;
// and source hooks (SrcF):
//  cur_range(e, first, last)  the cursor of a vertex whose records in the
//                             tile are [first, last];
//  note(e, n)                 the tile lists n records from edge index e on.
template <class T, class = void>
struct HasListVal : std::false_type {};
template <class T>
struct HasListVal<T, std::void_t<decltype(&T::list_val)>> : std::true_type {};
template <class T, class = void>
struct HasNote : std::false_type {};
template <class T>
struct HasNote<T, std::void_t<decltype(&T::note)>> : std::true_type {};
template <class T, class = void>
struct HasCurRange : std::false_type {};
template <class T>
struct HasCurRange<T, std::void_t<decltype(&T::cur_range)>> : std::true_type {};
template <class T, class = void>
struct HasProbeVal : std::false_type {};
template <class T>
struct HasProbeVal<T, std::void_t<decltype(T::kProbeVal)>> : std::true_type {};
template <class T, class = void>
struct HasCommit : std::false_type {};
template <class T>
struct HasCommit<T, std::void_t<decltype(&T::commit)>> : std::true_type {};

// Positions of a tile that a thread has in flight.
template <class Op>
struct OpGroup {
  static constexpr int value = kItems;
};

// Runs `body(lo, hi, j0)` over positions [plo, phi) of tile k: once, or in parts
// of kThreads positions when the tile holds more than kLocal vertices.  In
// the body, position x belongs to table entry map[x] - j0, and src.at(cb[entry],
// x) is its record (cb holds the source cursor, Src::cur, of tile position
// 0).  Every vertex's edge indices in the range are checked against edge_bound
// when its entry is made; one out of bounds sets kErrEdgeIndex and the range is
// skipped.  Sh is LbsShared<Val, *>.
template <bool kNeedVal, class Src, class Op, class Sh, class Body>
__device__ __forceinline__ void lbs_run(const LbsArgs &a, const Src &src, const Op &op, Sh &sh, uint64_t k,
                                        uint32_t plo, uint32_t phi, Body body) {
  __shared__ uint32_t s_bad;
  const uint64_t pos0 = k * kTile;
  const uint64_t ntiles_total = (a.total + kTile - 1) / kTile;
  const uint32_t i0 = a.tile_first[k];
  const uint32_t i1 = (k + 1 < ntiles_total) ? a.tile_first[k + 1] : a.n - 1;
  if (i1 < i0 || i1 - i0 > kTile || i1 >= a.n) {
    if (threadIdx.x == 0) atomicOr(a.err, kErrTileMap);
    return;
  }
  const uint32_t nl = i1 - i0 + 1;
  const bool parts = nl > kLocal;  // uniform
  if (threadIdx.x == 0) s_bad = 0;
  // zero the position map: 2048 u16 = one 16-byte store per thread
  static_assert(kTile * sizeof(unsigned short) == kThreads * sizeof(uint4), "map zeroing");
  reinterpret_cast<uint4 *>(sh.map)[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  // table entry x of local vertex j (list prefix p, start r), whose positions in [lo, hi) are used
  auto entry = [&](uint32_t x, uint32_t j, uint64_t p, uint32_t r, uint32_t lo, uint32_t hi) {
    const uint32_t i = i0 + j;
    const uint64_t pn = a.pref[i + 1];
    if (r >= hi || pn <= pos0 + lo) return;  // no position here
    const uint32_t v = a.list[i];
    const uint64_t e0 = (a.off ? a.off[v] - p : (0ull - a.stage_base)) + pos0;  // edge index of position 0
    const uint64_t first = e0 + max(r, lo), last = e0 + (min(pn, pos0 + hi) - pos0) - 1;
    uint64_t cb = src.cur(e0);
    if (pn < p || last < first || last >= a.edge_bound) {
      s_bad = 1;
      atomicOr(a.err, kErrEdgeIndex);
    } else if constexpr (HasCurRange<Src>::value) {
      cb = src.cur_range(e0, first, last);
      if constexpr (HasNote<Src>::value) src.note(first, (uint32_t)(last - first + 1));
    }
    sh.cb[x] = cb;
    if constexpr (HasListVal<Op>::value) sh.val[x] = op.list_val(v, a.list + i);
    else if constexpr (kNeedVal) sh.val[x] = op.src_val(v);
  };
#pragma unroll 1
  for (uint32_t j = threadIdx.x; j < nl; j += kThreads) {
    const uint64_t p = a.pref[i0 + j];
    const uint32_t r = p > pos0 ? (uint32_t)min(p - pos0, (uint64_t)kTile) : 0u;
    // head flag.  Compacted lists hold no zero-degree vertex, so for j >= 1
    // the starts are distinct and strictly increasing (the first is 0).
    if (j >= 1 && r < kTile) sh.map[r] = (unsigned short)1;
    if (!parts) entry(j, j, p, r, plo, phi);
  }
  __syncthreads();
  // inclusive scan of the head flags (blocked: thread t owns positions 8t..8t+7)
  {
    uint4 m = reinterpret_cast<const uint4 *>(sh.map)[threadIdx.x];
    uint32_t f[kItems] = {m.x & 0xffffu, m.x >> 16, m.y & 0xffffu, m.y >> 16,
                          m.z & 0xffffu, m.z >> 16, m.w & 0xffffu, m.w >> 16};
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < (int)kItems; i++) s += f[i];
    uint32_t run;
    block_scan_u32(s, run);
#pragma unroll
    for (int i = 0; i < (int)kItems; i++) {
      run += f[i];
      f[i] = run;
    }
    m = make_uint4(f[0] | (f[1] << 16), f[2] | (f[3] << 16), f[4] | (f[5] << 16), f[6] | (f[7] << 16));
    reinterpret_cast<uint4 *>(sh.map)[threadIdx.x] = m;
  }
  __syncthreads();
  const uint32_t step = parts ? kThreads : kTile;
#pragma unroll 1
  for (uint32_t lo = plo; lo < phi; lo += step) {
    const uint32_t hi = min(lo + step, phi);
    uint32_t j0 = 0;
    if (parts) {
      j0 = sh.map[lo];
      const uint32_t j1 = sh.map[hi - 1];
      if (lo != plo) __syncthreads();  // the part before has been read
      for (uint32_t j = j0 + threadIdx.x; j <= j1; j += kThreads) {
        const uint64_t p = a.pref[i0 + j];
        entry(j - j0, j, p, p > pos0 ? (uint32_t)min(p - pos0, (uint64_t)kTile) : 0u, lo, hi);
      }
      __syncthreads();
    }
    if (s_bad) return;  // uniform: written before a barrier, or a part later by nobody
    body(lo, hi, j0);
  }
}

// Shared tables of an LBS relax tile for Op.
template <class Op>
using LbsSh = LbsShared<typename Op::Val, Op::kNeedVal || HasListVal<Op>::value>;

// One LBS tile (kTile positions starting at tile k of the list) of a CTA, or
// part `part` of `parts` (1, 2, 4 or 8) equal ones.
template <class Src, class Op>
__device__ __forceinline__ void lbs_tile(const LbsArgs &a, const Src &src, const Op &op, LbsSh<Op> &sh,
                                         uint64_t k, uint32_t part = 0, uint32_t parts = 1) {
  const uint64_t pos0 = k * kTile;
  if (pos0 >= a.pos_end) return;
  const uint32_t plo = part * (kTile / parts);
  const uint32_t phi = min((uint32_t)min((uint64_t)kTile, a.pos_end - pos0), plo + kTile / parts);
  if (plo >= phi) return;  // uniform
  lbs_run<Op::kNeedVal>(a, src, op, sh, k, plo, phi, [&](uint32_t lo, uint32_t hi, uint32_t j0) {
    constexpr int G = OpGroup<Op>::value;
    // Positions x0, x0 + kThreads, ...: G of them.  All their loads are issued
    // before the first relax, so each thread keeps G edge reads in flight (the
    // host-link gather is latency bound).
    auto group = [&](uint32_t x0) {
      typename Src::Item ev[G];
      uint32_t lv[G];
#pragma unroll
      for (int it = 0; it < G; it++) {
        const uint32_t x = it * kThreads + x0;
        lv[it] = 0;
        if (x < hi) {
          const uint32_t l = sh.map[x] - j0;
          lv[it] = l;
          ev[it] = src.at(sh.cb[l], x);
        }
      }
      if constexpr (HasCommit<Op>::value)
        if (!op.commit()) return;
      // Probe phase: every target's current state is read before the first
      // atomic, so the random reads of a thread overlap (in program order
      // the compiler may not lift a load above an earlier atomic).  A probe is
      // only a filter: relax() acts through atomics, so a stale probe costs an
      // extra atomic, never a wrong result.
      typename Op::Probe pr[G];
#pragma unroll
      for (int it = 0; it < G; it++)
        if (it * kThreads + x0 < hi) {
          if constexpr (HasProbeVal<Op>::value) pr[it] = op.probe_v(ev[it], sh.val[lv[it]]);
          else pr[it] = op.probe(ev[it]);
        }
#pragma unroll
      for (int it = 0; it < G; it++) {
        if (it * kThreads + x0 < hi)
          op.relax(ev[it], Op::kNeedVal ? sh.val[lv[it]] : typename Op::Val{},
                   pos0 + it * kThreads + x0, pr[it]);
      }
    };
    if constexpr (G == kItems) {
      group(lo + threadIdx.x);
    } else {
#pragma unroll 1
      for (uint32_t x = lo; x < hi; x += G * kThreads) group(x + threadIdx.x);
    }
  });
}

template <class Src, class Op>
__global__ void __launch_bounds__(kThreads, 5) k_lbs(LbsArgs a, Src src, Op op) {
  __shared__ LbsSh<Op> sh;
  lbs_tile(a, src, op, sh, a.pos_begin / kTile + blockIdx.x);
}

// Both regions of a round in one launch: n0 tiles of list 0 (static region,
// read from HBM) and n1 tiles of list 1 (dynamic region, read over the host
// link), interleaved in CTA order in proportion to their counts, so that at
// any time about n0 / (n0 + n1) of the resident CTAs work from HBM while the
// rest keep the link busy.  CTA b is a static tile iff
// floor((b + 1) n0 / n) > floor(b n0 / n); its tile index is floor(b n0 / n),
// else b - floor((b + 1) n0 / n) among the dynamic tiles.
struct PairTile {
  unsigned long long t;  // tile index within its region
  uint32_t r;            // 0: static region, 1: dynamic region
};
__device__ __forceinline__ PairTile pair_split(uint64_t b, uint64_t n0, uint64_t n) {
  if (n0 == n) return PairTile{b, 0u};
  if (n0 == 0) return PairTile{b, 1u};
  const uint64_t lo = b * n0 / n, hi = (b + 1) * n0 / n;
  return hi > lo ? PairTile{lo, 0u} : PairTile{b - hi, 1u};
}
// The split of this CTA, computed once: a 64-bit division is a long
// instruction sequence, so thread 0 runs it and the CTA reads the result.
__device__ __forceinline__ PairTile pair_split_cta(uint64_t n0, uint64_t n) {
  __shared__ PairTile s_pt;
  if (threadIdx.x == 0) s_pt = pair_split(blockIdx.x, n0, n);
  __syncthreads();
  return s_pt;
}

template <class Src0, class Src1, class Op>
__global__ void __launch_bounds__(kThreads, 5) k_lbs_pair(LbsArgs a0, Src0 s0, LbsArgs a1, Src1 s1, Op op,
                                                       uint64_t n0, uint64_t n) {
  __shared__ LbsSh<Op> sh;
  const PairTile pt = pair_split_cta(n0, n);
  if (pt.r == 0) lbs_tile(a0, s0, op, sh, a0.pos_begin / kTile + pt.t);
  else lbs_tile(a1, s1, op, sh, a1.pos_begin / kTile + pt.t);
}

// A staged round in one launch.  The two staging buffers are a ring of tile
// slots: position tile t is gathered into slot t % slots and relaxed out of it,
// one CTA per step.  state[slot] counts the slot's steps: use u of a slot is
// gathered when it reads 2u and relaxed when it reads 2u + 1.  CTAs take their
// step from a ticket: first `lead` gathers, then gather t + lead and relax t in
// turn, so a step waits only for steps with earlier tickets, which running
// CTAs hold; the whole grid need not be resident.  With lead = slots / 2 both
// waits are `slots` steps back and rarely last (5/8 to 7/8 of slots measured the same).
// One launch per chunk (gather of chunk c beside the relax of c - 1) was bound
// by a wave's latency per chunk and the gap between launches: 15 + 3 us for
// 1.65 MB that the link moves in 8; delta PageRank of 777777 vertices took 4.24
// ms so and takes 3.31 now (a round of 18.4 MB: 127 us, of them 87 link), BFS
// of 2^20 vertices with chunks of 55296 edges 1.95 (8.5 with two streams and an
// event each way per chunk).  A grid of 2 to 6 CTAs per SM that loop over the
// tickets was slower (4.19 to 3.41 ms).
constexpr uint32_t kRingSlots = 2048;  // most slots in use: 4 M positions, more than are ever in flight
constexpr uint32_t kRingPad = 32;      // words before them: the ticket's cache line
// kLimit: polls of a wait for a slot (a constant: read from the arguments it cost
// delta PageRank of 777777 vertices 3.10 ms instead of 3.02).
template <uint32_t kLimit>
struct StageRingT {
  uint32_t *state, *ticket;  // zeroed before the launch
  uint32_t slots, half;      // half: slots of buffer 0
};
using StageRing = StageRingT<kSpinLimit>;
struct StageStep {
  uint64_t tile, base;  // base: position minus buffer entry (mod 2^64)
  uint32_t slot, want;  // want: the state this step waits for; odd: relax
  uint32_t buf, ready;
};
// This CTA's step, from the next ticket.
template <class Ring>
__device__ __forceinline__ void stage_take(const Ring &g, uint64_t ntiles, StageStep &step) {
  if (threadIdx.x == 0) {
    const uint64_t i = atomicAdd(g.ticket, 1u), lead = min((uint64_t)(g.slots / 2), ntiles);
    const uint64_t j = i - lead, pairs = ntiles - lead;  // j: valid for i >= lead
    StageStep x;
    bool relax = false;
    if (i < lead) {
      x.tile = i;
    } else if (j < 2 * pairs) {
      relax = j & 1u;
      x.tile = (j >> 1) + (relax ? 0 : lead);
    } else {
      relax = true;
      x.tile = j - pairs;
    }
    const uint32_t use = (uint32_t)x.tile / g.slots;
    x.slot = (uint32_t)x.tile - use * g.slots;
    x.want = 2 * use + relax;
    x.buf = x.slot >= g.half;
    x.base = (x.tile - (x.slot - x.buf * g.half)) * kTile;
    x.ready = 0;
    step = x;
  }
  __syncthreads();
}
// Thread 0: waits for the step's slot, a bounded number of polls (an expired
// wait sets kErrBarrier, which ends the waits of the others).  The polls are
// relaxed and one fence follows: it also drops lines of the slot's earlier
// use from L1.
template <uint32_t kLimit>
__device__ __forceinline__ void stage_wait(const StageRingT<kLimit> &g, StageStep &x, uint32_t *err) {
  for (uint32_t spins = 0; ld_relaxed(g.state + x.slot) != x.want;) {
    if (++spins > kLimit || ((spins & 255u) == 0 && (ld_relaxed(err) & kErrBarrier))) {
      atomicOr(err, kErrBarrier);
      return;
    }
    __nanosleep(spins < 256 ? 20 : 200);
  }
  __threadfence();
  x.ready = 1;
}
// All threads: waits for the slot; false: gave up.
template <class Ring>
__device__ __forceinline__ bool stage_ready(const Ring &g, StageStep &x, uint32_t *err) {
  if (threadIdx.x == 0 && !x.ready) stage_wait(g, x, err);
  __syncthreads();
  return x.ready != 0;
}
template <class Ring>
__device__ __forceinline__ void stage_post(const Ring &g, StageStep &x, uint32_t *err) {
  __syncthreads();
  if (threadIdx.x != 0) return;
  if (!x.ready) stage_wait(g, x, err);  // a gather that stopped before its stores
  if (x.ready) st_release(g.state + x.slot, x.want + 1);
}

// The gather of a staged round as an edge op: position pos goes to entry
// pos - base of a staging buffer.  The slot is waited for after the link reads
// have been issued, so a step holds it for its stores alone.
template <class Dst, class Ring>
struct GatherOp {
  using Val = uint32_t;
  static constexpr bool kNeedVal = false;
  Dst stage;
  uint64_t base;
  const Ring *ring;
  StageStep *step;  // shared memory
  uint32_t *err;
  __device__ __forceinline__ bool commit() const { return stage_ready(*ring, *step, err); }
  __device__ uint32_t src_val(uint32_t) const { return 0; }
  using Probe = uint32_t;
  template <class Edge>
  __device__ __forceinline__ Probe probe(Edge) const {
    return 0u;
  }
  template <class Edge>
  __device__ __forceinline__ void relax(Edge e, uint32_t, uint64_t pos, Probe) const {
    stage.store(pos - base, e);
  }
};

template <class PSrc, class Dst, class Src, class Op, class Ring>
__global__ void __launch_bounds__(kThreads, 5) k_stage_round(const __grid_constant__ LbsArgs a, PSrc ps, Dst d0, Dst d1,
                                                             Src s0, Src s1, uint64_t cap, Op op,
                                                             const __grid_constant__ Ring ring) {
  __shared__ union {
    LbsSh<GatherOp<Dst, Ring>> gather;
    LbsSh<Op> relax;
  } sh;
  __shared__ StageStep x;
  stage_take(ring, (a.total + kTile - 1) / kTile, x);
  if (x.want & 1u) {
    if (!stage_ready(ring, x, a.err)) return;
    LbsArgs r = a;  // positions of a staging buffer instead of CSR offsets
    r.off = nullptr;
    r.stage_base = x.base;
    r.edge_bound = cap;
    lbs_tile(r, x.buf ? s1 : s0, op, sh.relax, x.tile);
  } else {
    lbs_tile(a, ps, GatherOp<Dst, Ring>{x.buf ? d1 : d0, x.base, &ring, &x, a.err}, sh.gather, x.tile);
  }
  stage_post(ring, x, a.err);
}

template <int MULT>
constexpr size_t gather_smem_bytes() {
  return 8 * (MULT * kTile + 1) + 4 * (MULT * kTile + 2) + 2 * (MULT * kTile);
}

// Dynamic-region gather, specialised: MULT x 2048 positions per CTA (the
// per-tile setup is amortised over more edges) and no per-vertex value table.
// Positions of a vertex are contiguous both in the host CSR and in the staging
// buffer, so this is a segmented copy; reads are coalesced 8-byte (or 4-byte)
// loads over NVLink-C2C, all ITEMS of a thread issued before the first store.
template <class Src, class Dst, int MULT>
__global__ void __launch_bounds__(kThreads) k_gather(LbsArgs a, Src src, Dst stage) {
  constexpr uint32_t TILE = MULT * kTile;
  constexpr int ITEMS = TILE / kThreads;
  // dynamic shared memory (gather_smem_bytes<MULT>() bytes, above the static 48 KB)
  extern __shared__ __align__(16) unsigned char g_smem[];
  unsigned long long *cb = (unsigned long long *)g_smem;          // TILE + 1
  uint32_t *rs = (uint32_t *)(cb + TILE + 1);                      // TILE + 2
  unsigned short *map = (unsigned short *)(rs + TILE + 2);         // TILE
  const uint64_t pos0 = a.pos_begin + (uint64_t)blockIdx.x * TILE;
  if (pos0 >= a.pos_end) return;
  const uint64_t pend = min(pos0 + TILE, a.pos_end);
  const uint32_t i0 = a.tile_first[pos0 / kTile];
  const uint32_t i1 = pend < a.total ? a.tile_first[pend / kTile] : a.n - 1;
  if (i1 < i0 || i1 - i0 > TILE || i1 >= a.n) {
    if (threadIdx.x == 0) atomicOr(a.err, kErrTileMap);
    return;
  }
  const uint32_t nl = i1 - i0 + 1;
  for (uint32_t j = threadIdx.x; j < nl; j += kThreads) {
    const uint32_t v = a.list[i0 + j];
    const uint64_t p = a.pref[i0 + j];
    rs[j] = p > pos0 ? (uint32_t)min(p - pos0, (uint64_t)TILE) : 0u;
    cb[j] = a.off[v] - p + pos0;
  }
  for (uint32_t x = threadIdx.x; x < TILE; x += kThreads) map[x] = 0;
  __syncthreads();
  for (uint32_t j = 1 + threadIdx.x; j < nl; j += kThreads)
    if (rs[j] < TILE) map[rs[j]] = 1;
  __syncthreads();
  {
    uint32_t f[ITEMS], sacc = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
      f[i] = map[threadIdx.x * ITEMS + i];
      sacc += f[i];
    }
    uint32_t ex, tot;
    uint64_t ex64, tot64;
    block_scan_pair(sacc, 0, ex, ex64, tot, tot64);
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
      ex += f[i];
      map[threadIdx.x * ITEMS + i] = (unsigned short)ex;
    }
  }
  __syncthreads();
  const uint32_t tlen = (uint32_t)(pend - pos0);
  typename Src::Item ev[ITEMS];
  uint32_t okm = 0;
#pragma unroll
  for (int it = 0; it < ITEMS; it++) {
    const uint32_t x = it * kThreads + threadIdx.x;
    if (x < tlen) {
      const uint64_t idx = cb[map[x]] + x;
      if (idx < a.edge_bound) {
        ev[it] = src.load(idx);
        okm |= 1u << it;
      } else {
        atomicOr(a.err, kErrEdgeIndex);
      }
    }
  }
  const uint64_t base = pos0 - a.stage_base;
#pragma unroll
  for (int it = 0; it < ITEMS; it++)
    if (okm & (1u << it)) stage.store(base + it * kThreads + threadIdx.x, ev[it]);
}

// ------------------------------------------------------------------ ops

__device__ __forceinline__ uint32_t edge_dst(uint32_t e) { return e; }
__device__ __forceinline__ uint32_t edge_dst(uint2 e) { return e.x; }
__device__ __forceinline__ uint32_t edge_w(uint32_t) { return 1u; }
__device__ __forceinline__ uint32_t edge_w(uint2 e) { return e.y; }

// Level-synchronous BFS with a visited bitmap: every vertex is claimed once.
struct BfsOp {
  using Val = uint32_t;
  static constexpr bool kNeedVal = false;
  uint32_t *visited, *next, *depth, *err;
  uint32_t V, newdepth;
  __device__ uint32_t src_val(uint32_t) const { return 0; }
  // The target's visited word, read through L1: bits are only ever set
  // during a launch (and global data cached in L1 does not outlive the
  // launch), so a stale word lacks bits at most and costs an extra atomic,
  // never a wrong result.  Hub vertices' words are read over and over.
  using Probe = uint32_t;
  template <class Edge>
  __device__ __forceinline__ Probe probe(Edge e) const {
    const uint32_t v = edge_dst(e);
    return v < V ? visited[v >> 5] : 0u;
  }
  template <class Edge>
  __device__ __forceinline__ void relax(Edge e, uint32_t, uint64_t, Probe p) const {
    const uint32_t v = edge_dst(e);
    if (v >= V) {
      atomicOr(err, kErrVertex);
      return;
    }
    const uint32_t w = v >> 5, bit = 1u << (v & 31);
    if (p & bit) return;
    // The probe holds every bit set before this launch, so v is reached at
    // this level, by this thread or another one of the launch: every writer
    // stores the same depth and sets the same bits.  No atomic's old value
    // is needed, so none is waited for (the atomics compile to reductions).
    atomicOr(visited + w, bit);
    depth[v] = newdepth;
    atomicOr(next + w, bit);
  }
};

// atomicMin relax shared by SSSP (weighted) and CC (label push).
template <bool kWeighted>
struct MinOp {
  using Val = uint32_t;
  static constexpr bool kNeedVal = true;
  uint32_t *value, *next, *err;
  uint32_t V;
  __device__ uint32_t src_val(uint32_t v) const { return __ldcg(value + v); }
  // The target's current value, read through L1: values only decrease during
  // a launch, so a stale value is too large at most and costs an extra
  // atomicMin, never a wrong result.
  using Probe = uint32_t;
  template <class Edge>
  __device__ __forceinline__ Probe probe(Edge e) const {
    const uint32_t v = edge_dst(e);
    return v < V ? value[v] : 0u;
  }
  template <class Edge>
  __device__ __forceinline__ void relax(Edge e, uint32_t sv, uint64_t, Probe p) const {
    const uint32_t v = edge_dst(e);
    if (v >= V) {
      atomicOr(err, kErrVertex);
      return;
    }
    const uint32_t cand = kWeighted ? sv + edge_w(e) : sv;
    if (cand >= p) return;
    // cand < p: v's value drops in this launch, to cand here or lower by
    // another thread that marks v as well, so v is in the next frontier
    // either way.  The atomics' old values are not needed (reductions).
    atomicMin(value + v, cand);
    atomicOr(next + (v >> 5), 1u << (v & 31));
  }
};

// ------------------------------------------------------------------ batched BFS

// Up to 64 BFS sources share one pass: bit s of a vertex's masks belongs to
// source s.  visited = bits already reached, cur = bits first reached at the
// current level (frontier), next = bits first reached at the next level.
// Level-synchronous, so a bit's level is its BFS depth, exactly as a
// single-source run computes it.
struct BatchOp {
  using Val = unsigned long long;
  static constexpr bool kNeedVal = true;
  unsigned long long *visited, *cur, *next;
  uint32_t *next_any;  // bitmap of vertices with next != 0
  uint32_t *err;
  uint32_t V;
  __device__ Val src_val(uint32_t v) const { return __ldcg(cur + v); }
  using Probe = unsigned long long;  // the target's visited mask (through L1, as BfsOp)
  template <class Edge>
  __device__ __forceinline__ Probe probe(Edge e) const {
    const uint32_t v = edge_dst(e);
    return v < V ? visited[v] : ~0ull;
  }
  template <class Edge>
  __device__ __forceinline__ void relax(Edge e, Val m, uint64_t, Probe p) const {
    const uint32_t v = edge_dst(e);
    if (v >= V) {
      atomicOr(err, kErrVertex);
      return;
    }
    Val nb = m & ~p;
    if (!nb) return;
    nb &= ~atomicOr(visited + v, nb);
    if (!nb) return;
    if (atomicOr(next + v, nb) == 0ull) atomicOr(next_any + (v >> 5), 1u << (v & 31));
  }
};

// PageRank by push over an out-edge CSR: the listed vertex u adds its
// contribution (rank / out-degree, the LBS source value) to the sum of every
// out-neighbour with an FP32 atomicAdd.  Nothing to probe.
struct PushOp {
  using Val = float;
  static constexpr bool kNeedVal = true;
  const float *contrib;
  float *sum;
  uint32_t *err;
  uint32_t V;
  __device__ Val src_val(uint32_t u) const { return contrib[u]; }
  using Probe = uint32_t;
  template <class Edge>
  __device__ __forceinline__ Probe probe(Edge) const {
    return 0u;
  }
  template <class Edge>
  __device__ __forceinline__ void relax(Edge e, Val c, uint64_t, Probe) const {
    const uint32_t v = edge_dst(e);
    if (v >= V) {
      atomicOr(err, kErrVertex);
      return;
    }
    if (c != 0.f) atomicAdd(sum + v, c);
  }
};

// Seeds source i (bit slots[i], or bit i when slots is null) at depth 1.
__global__ void k_batch_init(const uint32_t *srcs, uint32_t n, unsigned long long *visited,
                             unsigned long long *cur, uint32_t *cur_any, uint32_t *depth,
                             uint64_t V, uint8_t *depth8 = nullptr, const uint32_t *slots = nullptr) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t v = srcs[i], b = slots ? slots[i] : i;
  atomicOr(visited + v, 1ull << b);
  atomicOr(cur + v, 1ull << b);
  atomicOr(cur_any + (v >> 5), 1u << (v & 31));
  if (depth) depth[(uint64_t)b * V + v] = 1u;
  if (depth8) depth8[(uint64_t)b * V + v] = 1u;
}

// Clears the bits `mask` of every vertex's mask (slots released for reuse).
__global__ void k_batch_clear_bits(unsigned long long *m, uint64_t n, unsigned long long mask) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
    if (m[v] & mask) m[v] &= ~mask;
}

// Per-source count of the vertices first reached at this level (hist[s]),
// and, when depth != nullptr, their depth for the n x V output: level, less
// doff[s] when doff is not null (a source that joined a pass in flight).
__global__ void __launch_bounds__(kThreads) k_batch_level(const uint32_t *next_any,
                                                          const unsigned long long *next,
                                                          uint64_t nwords, uint32_t n,
                                                          unsigned long long *hist,
                                                          uint32_t *depth, uint64_t V,
                                                          uint32_t level, const uint32_t *doff = nullptr) {
  __shared__ uint32_t s_cnt[64];
  if (threadIdx.x < 64) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nwords;
       w += (uint64_t)gridDim.x * blockDim.x) {
    for (uint32_t bits = next_any[w]; bits; bits &= bits - 1) {
      const uint64_t v = w * 32 + (__ffs(bits) - 1);
      if (v >= V) break;
      for (unsigned long long m = next[v]; m; m &= m - 1) {
        const uint32_t s = __ffsll((long long)m) - 1;
        if (s < n) {
          atomicAdd(&s_cnt[s], 1u);
          if (depth) depth[(uint64_t)s * V + v] = doff ? level - doff[s] : level;
        }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < 64 && s_cnt[threadIdx.x]) atomicAdd(hist + threadIdx.x, (unsigned long long)s_cnt[threadIdx.x]);
}

// ------------------------------------------------------------------ PageRank

constexpr uint32_t kNoCarry = 0xffffffffu;

struct PrArgs {
  const float *contrib;   // rank[u] / outdeg[u] (0 for dangling u)
  float *sum;             // pull sums, written for every listed vertex
  float *cont;            // per LBS tile: partial of a vertex that began in an earlier tile
  float *carry;           // per LBS tile: partial of a vertex that began here and continues
  uint32_t *carry_idx;    // per LBS tile: list index of that vertex, kNoCarry if none
  uint32_t V;
  // contiguous lists (every vertex of the region that has edges is listed, or
  // a staging buffer): position q is record base + q of the record stream,
  // which holds nwords words
  uint64_t base, nwords;
  // iterations launched ahead: when not null, nothing is done once *done is set
  const uint32_t *done;
  uint32_t link;  // the records are read over the host link
  // when not null, this iteration is timed: t[0] is when the one before ended;
  // k_pr_fixup, right behind the pull, adds the time since to t[1] (ns of the
  // GPU's global timer) and one to t[2].  Every kPrTimed-th iteration is: the
  // timer is slow to read (3 % of the iterations of a graph of 0.1 M vertices
  // when all were; a stamp in the pull itself cost 4 us of 590)
  unsigned long long *t;
};

// Pull sum sum[v] = sum over in-edges (u -> v) of contrib[u]
// (PR/OneGraph/gpu_kernels.h:107-158), deterministic: the order of the
// additions depends only on the tiling of the compacted list.
//
// What bounds it is the random read of contrib: one L1 tag lookup per edge,
// and an L2 sector for those that miss.  So everything else is kept off the
// L1/shared pipe.  A thread owns eight consecutive positions and adds them in
// registers; vertex starts are one byte flag per position, read as one 8-byte
// word; a single block scan carries both the thread's vertex index and the sum
// of its open segment.  On contiguous lists (kDense: every iteration of the
// L1 form, the first rounds of the delta form, staged chunks) the record of a
// position does not depend on the list, so the tile's words are fetched 16
// bytes a lane before anything else and the gather starts while the flags
// are still being built.  Other lists read each record through its vertex's
// cursor.  Over the host link a warp's lanes read consecutive positions and hand
// the columns to their owners through shared memory: with each lane on its own
// eight records a warp asks for every sector several times (direct delta PageRank of
// 4.2 M vertices, two fifths resident: 21.1 ms so, 12.5 now); from HBM the detour
// costs more than it gives (all resident: 7.0 ms without, 8.0 with).  Measured on 8.4 M vertices and 131 M edges: 1.09 ms an iteration with
// positions strided over the threads and staged twice through shared memory,
// 0.53 ms in this form (247 G edges/s; 65 M edges: L1 81 % busy, L2 65 %).
constexpr uint32_t pr_flag_bytes(bool dense) { return dense ? kTile : 2 * kTile; }
constexpr uint32_t pr_smem_bytes(bool dense, uint32_t bpe) {
  // flags (cursor form: later each position's vertex), then by phase the
  // tile's words / the cursors, the columns, and the sums
  const uint32_t words = (kTile * bpe / 32 + 10) * 4, tot = (kTile + 1) * 4, cur = (kTile + 1) * 8;
  return pr_flag_bytes(dense) + (dense ? (words > tot ? words : tot) : cur) + 16;
}

template <bool kDense, class Src>
__device__ __forceinline__ void pr_tile(const LbsArgs &a, const Src &src, const PrArgs &p, uint64_t k) {
  extern __shared__ __align__(16) unsigned char pr_smem[];
  unsigned char *flag = pr_smem;
  uint32_t *words = reinterpret_cast<uint32_t *>(pr_smem + pr_flag_bytes(kDense));
  // !kDense
  unsigned long long *cur = reinterpret_cast<unsigned long long *>(words);
  uint16_t *map = reinterpret_cast<uint16_t *>(pr_smem);
  float *tot = reinterpret_cast<float *>(words);  // once the records are in registers
  __shared__ uint32_t s_bad, s_edge;
  __shared__ float s_wv[kThreads / 32];
  __shared__ uint32_t s_wc[kThreads / 32];
  const uint64_t pos0 = k * kTile;
  if (pos0 >= a.pos_end || (p.done && *p.done)) return;
  const uint64_t pend = min(pos0 + kTile, a.pos_end);
  const uint32_t tlen = (uint32_t)(pend - pos0), tid = threadIdx.x, x0 = tid * kItems;
  // the tile's words, from the 16-byte boundary at or before its first record
  const uint64_t bit0 = (p.base + pos0) * src.bpe;
  const uint64_t q0 = (bit0 >> 5) & ~3ull;
  const uint32_t n4 = kDense ? (uint32_t)((((p.base + pend) * src.bpe + 31) / 32 - q0 + 3) / 4) : 0;
  uint4 wv[2];  // two cover every record of up to 32 bits; wider ones loop below
  auto load4 = [&](uint32_t i) {
    const uint64_t q = q0 + 4ull * i;
    uint4 w = make_uint4(0u, 0u, 0u, 0u);
    if (q + 4 <= p.nwords) {
      w = *reinterpret_cast<const uint4 *>(src.words + q);
    } else {
      if (q < p.nwords) w.x = src.words[q];
      if (q + 1 < p.nwords) w.y = src.words[q + 1];
      if (q + 2 < p.nwords) w.z = src.words[q + 2];
    }
    return w;
  };
  if constexpr (kDense) {
    if (p.base + pend > a.edge_bound) {
      if (tid == 0) {
        atomicOr(a.err, kErrEdgeIndex);
        p.carry_idx[k] = kNoCarry;
      }
      return;
    }
#pragma unroll
    for (int j = 0; j < 2; j++)
      if (j * kThreads + tid < n4) wv[j] = load4(j * kThreads + tid);
  }
  const uint64_t ntiles_total = (a.total + kTile - 1) / kTile;
  const uint32_t i0 = a.tile_first[k];
  const uint32_t i1 = (k + 1 < ntiles_total) ? a.tile_first[k + 1] : a.n - 1;
  if (i1 < i0 || i1 - i0 > kTile || i1 >= a.n) {
    if (tid == 0) {
      atomicOr(a.err, kErrTileMap);
      p.carry_idx[k] = kNoCarry;
    }
    return;
  }
  const uint32_t nl = i1 - i0 + 1;
  *reinterpret_cast<uint2 *>(flag + x0) = make_uint2(0u, 0u);
  if (tid == 0) s_bad = 0;
  __syncthreads();
  if constexpr (kDense) {
#pragma unroll
    for (int j = 0; j < 2; j++)
      if (j * kThreads + tid < n4) reinterpret_cast<uint4 *>(words)[j * kThreads + tid] = wv[j];
    for (uint32_t i = 2 * kThreads + tid; i < n4; i += kThreads) reinterpret_cast<uint4 *>(words)[i] = load4(i);
  }
  bool bad = false;
  for (uint32_t j = tid; j < nl; j += kThreads) {
    const uint32_t i = i0 + j;
    const uint64_t s = a.pref[i];
    const uint32_t r = s > pos0 ? (uint32_t)min(s - pos0, (uint64_t)kTile) : 0u;
    // compacted lists hold no zero-degree vertex: starts are strictly increasing
    if (j >= 1 && r < kTile) flag[r] = 1;
    if constexpr (!kDense) {
      const uint64_t e0 = a.off[a.list[i]] - s + pos0;  // record of position 0
      const uint64_t q1 = min(a.pref[i + 1], pend);
      if (q1 > pos0 + r && (a.pref[i + 1] < s || e0 + (q1 - pos0) > a.edge_bound || e0 + r >= a.edge_bound)) bad = true;
      cur[j] = src.cur(e0);
    }
    // the tile's first vertex may have begun earlier, its last may go on
    if (j == 0) s_edge = s < pos0 ? 1u : 0u;
  }
  if (bad) {
    s_bad = 1;
    atomicOr(a.err, kErrEdgeIndex);
  }
  __syncthreads();
  if (s_bad) {
    if (tid == 0) p.carry_idx[k] = kNoCarry;
    return;
  }
  const uint2 fw = *reinterpret_cast<const uint2 *>(flag + x0);
  // bit i: a vertex starts at position x0 + i (the tile's first one is not marked)
  uint32_t heads = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) heads |= ((fw.x >> (8 * i)) & 1u) << i | ((fw.y >> (8 * i)) & 1u) << (4 + i);
  // whether a vertex ends with this thread's last position; the cursor form reads it before the map takes the
  // flags' place, the other one where it is needed (a register more costs it 2 %)
  auto ends_here = [&]() { return x0 + kItems >= tlen || flag[x0 + kItems]; };
  bool last = false;
  if constexpr (!kDense) last = ends_here();
  const uint32_t lane = tid & 31, warp = tid >> 5;
  uint32_t u[kItems];
  if constexpr (kDense) {
    const uint32_t b0 = (uint32_t)(bit0 - (q0 << 5)) + x0 * src.bpe;
#pragma unroll
    for (int i = 0; i < (int)kItems; i++) {
      const uint32_t b = b0 + i * src.bpe;
      u[i] = 0xffffffffu;  // no edge at this position
      if (x0 + i < tlen) u[i] = src.decode(words + (b >> 5), b & 31u);
    }
  } else {
    uint32_t c = __popc(heads), ic = c;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, ic, d);
      if (lane >= d) ic += t;
    }
    if (lane == 31) s_wc[warp] = ic;
    __syncthreads();
    uint32_t l = ic - c;
    for (uint32_t w = 0; w < warp; w++) l += s_wc[w];
    if (!p.link) {  // uniform
#pragma unroll
      for (int i = 0; i < (int)kItems; i++) {
        l += (heads >> i) & 1u;
        u[i] = x0 + i < tlen ? src.at(cur[l], x0 + i) : 0xffffffffu;
      }
      __syncthreads();  // s_wc is written again below
    } else {
      uint32_t m[kItems / 2];
#pragma unroll
      for (int i = 0; i < (int)kItems; i += 2) {
        l += (heads >> i) & 1u;
        m[i / 2] = l;
        l += (heads >> (i + 1)) & 1u;
        m[i / 2] |= l << 16;
      }
      *reinterpret_cast<uint4 *>(map + x0) = make_uint4(m[0], m[1], m[2], m[3]);  // every flag has been read
      __syncthreads();
#pragma unroll
      for (int i = 0; i < (int)kItems; i++) {
        const uint32_t x = i * kThreads + tid;
        u[i] = x < tlen ? src.at(cur[map[x]], x) : 0xffffffffu;
      }
      __syncthreads();  // the cursors have been read: the columns take their place
#pragma unroll
      for (int i = 0; i < (int)kItems; i++) words[i * kThreads + tid] = u[i];
      __syncthreads();
#pragma unroll
      for (int i = 0; i < (int)kItems; i += 4) {
        const uint4 q = *reinterpret_cast<const uint4 *>(words + x0 + i);
        u[i] = q.x, u[i + 1] = q.y, u[i + 2] = q.z, u[i + 3] = q.w;
      }
    }
  }
  float c[kItems];
#pragma unroll
  for (int i = 0; i < (int)kItems; i++) {
    c[i] = 0.f;
    if (u[i] < p.V) c[i] = __ldg(p.contrib + u[i]);
    else if (u[i] != 0xffffffffu) atomicOr(a.err, kErrVertex);
  }
  // the thread's open segment: everything after its last vertex start
  float run = 0.f;
#pragma unroll
  for (int i = 0; i < (int)kItems; i++) run = ((heads >> i) & 1u) ? c[i] : run + c[i];
  // inclusive scan over the threads: vertex starts add, the open segment's
  // sum adds up to the nearest thread that holds a start
  float iv = run;
  uint32_t ic = __popc(heads);
#pragma unroll
  for (uint32_t d = 1; d < 32; d <<= 1) {
    const float v2 = __shfl_up_sync(0xffffffffu, iv, d);
    const uint32_t c2 = __shfl_up_sync(0xffffffffu, ic, d);
    if (lane >= d) {
      if (!ic) iv += v2;  // no start in the window so far: the segment extends to the left
      ic += c2;
    }
  }
  if (lane == 31) {
    s_wv[warp] = iv;
    s_wc[warp] = ic;
  }
  __syncthreads();
  float cv = 0.f;
  uint32_t l = 0;
#pragma unroll
  for (uint32_t w = 0; w < kThreads / 32; w++)
    if (w < warp) {
      cv = s_wc[w] ? s_wv[w] : cv + s_wv[w];
      l += s_wc[w];
    }
  const float lv = __shfl_up_sync(0xffffffffu, iv, 1);
  const uint32_t lc = __shfl_up_sync(0xffffffffu, ic, 1);
  if (lane > 0) {
    cv = lc ? lv : cv + lv;
    l += lc;
  }
  run = cv;  // the open segment's sum before this thread's first position
  // a vertex's total is written by the thread that adds its last position
#pragma unroll
  for (int i = 0; i < (int)kItems; i++) {
    if ((heads >> i) & 1u) {
      if (i > 0) tot[l] = run;
      l++;
      run = 0.f;
    }
    run += c[i];
  }
  if (x0 < tlen && (kDense ? ends_here() : last)) tot[l] = run;
  __syncthreads();
  for (uint32_t j = tid; j < nl; j += kThreads) {
    const uint32_t i = i0 + j;
    bool ends = true, here = true;  // v ends in this tile; v has positions in it
    if (j + 1 == nl) {
      here = j == 0 || a.pref[i] < pend;
      ends = a.pref[i + 1] <= pos0 + kTile;
      const bool carries = here && !ends && !(j == 0 && s_edge);
      p.carry_idx[k] = carries ? i : kNoCarry;
      if (carries) p.carry[k] = tot[j];
    }
    if (!here) continue;
    if (j == 0 && s_edge) p.cont[k] = tot[0];
    else if (ends) p.sum[a.list[i]] = tot[j];
  }
}

template <bool kDense, class Src>
__global__ void __launch_bounds__(kThreads, 6) k_pr_pull(LbsArgs a, Src src, PrArgs p) {
  pr_tile<kDense>(a, src, p, a.pos_begin / kTile + blockIdx.x);
}

// A staged PageRank round (see k_stage_round): the buffers hold columns as
// 32-bit records.
template <class PSrc, class Dst, class Src>
__global__ void __launch_bounds__(kThreads, 6) k_stage_round_pr(const __grid_constant__ LbsArgs a, PSrc ps, Dst d0,
                                                                Dst d1, Src s0, Src s1, uint64_t cap,
                                                                const __grid_constant__ PrArgs p,
                                                                const __grid_constant__ StageRing ring) {
  __shared__ LbsSh<GatherOp<Dst, StageRing>> sh;
  __shared__ StageStep x;
  stage_take(ring, (a.total + kTile - 1) / kTile, x);
  if (x.want & 1u) {
    if (!stage_ready(ring, x, a.err)) return;
    LbsArgs r = a;
    PrArgs q = p;
    r.edge_bound = cap;
    q.base = 0ull - x.base;
    q.nwords = cap;
    pr_tile<true>(r, x.buf ? s1 : s0, q, x.tile);
  } else {
    lbs_tile(a, ps, GatherOp<Dst, StageRing>{x.buf ? d1 : d0, x.base, &ring, &x, a.err}, sh, x.tile);
  }
  stage_post(ring, x, a.err);
}

// Both regions' pull sums in one launch, static and dynamic tiles interleaved
// in CTA order as in k_lbs_pair (each region keeps its own carry arrays, so
// the sums are the same as with two launches).
template <bool kDense, class Src>
__global__ void __launch_bounds__(kThreads, 6) k_pr_pull_pair(LbsArgs a0, Src s0, PrArgs p0, LbsArgs a1, Src s1,
                                                              PrArgs p1, uint64_t n0, uint64_t n) {
  const PairTile pt = pair_split_cta(n0, n);
  const bool st = pt.r == 0;  // one inlined tile body for both regions
  pr_tile<kDense>(st ? a0 : a1, st ? s0 : s1, st ? p0 : p1, (st ? a0.pos_begin : a1.pos_begin) / kTile + pt.t);
}

// Completes the sums of vertices split over several tiles, in tile order, for
// both regions: the first n0 threads take region 0's tiles, the next n1
// region 1's.
struct PrFixup {
  const uint32_t *list;
  const uint64_t *pref;
  uint32_t n;  // list length
  PrArgs p;
};
__global__ void k_pr_fixup(PrFixup f0, uint64_t n0, PrFixup f1, uint64_t n1) {
  const uint64_t x = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (x >= n0 + n1 || (f0.p.done && *f0.p.done)) return;
  if (f0.p.t && x == 0) {
    f0.p.t[1] += globaltimer_ns() - f0.p.t[0];
    f0.p.t[2]++;
  }
  const bool r0 = x < n0;
  const uint64_t k = r0 ? x : x - n0;
  const PrFixup &f = r0 ? f0 : f1;
  const uint32_t i = f.p.carry_idx[k];
  if (i >= f.n) return;  // kNoCarry
  float s = f.p.carry[k];
  const uint64_t end = f.pref[i + 1];
  for (uint64_t t = k + 1; t * kTile < end; t++) s += f.p.cont[t];
  f.p.sum[f.list[i]] = s;
}

// prKernel_Opt (PR/OneGraph/gpu_kernels.h:295-319): for every active vertex
// new = 0.15 + 0.85*sum; it stays active with the new rank iff |new-old| >
// thresh, otherwise it goes inactive keeping its rank.  One thread per bitmap
// word; writes the next active bitmap and counts the survivors.
__global__ void __launch_bounds__(kThreads) k_pr_update_delta(
    const uint32_t *cur, uint32_t *next, uint64_t nwords, float *rank, float *contrib,
    const float *sum, const uint32_t *outdeg, float thresh, uint32_t *active) {
  __shared__ uint32_t s_cnt;
  if (threadIdx.x == 0) s_cnt = 0;
  __syncthreads();
  uint32_t mine = 0;
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nwords;
       w += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t word = cur[w];
    uint32_t keep = 0;
    for (uint32_t m = word; m; m &= m - 1) {
      const uint32_t b = __ffs(m) - 1;
      const uint64_t v = w * 32 + b;
      const float nvv = 0.15f + 0.85f * sum[v];
      const float old = rank[v];
      const float diff = nvv > old ? nvv - old : old - nvv;
      if (diff > thresh) {
        rank[v] = nvv;
        const uint32_t od = outdeg[v];
        contrib[v] = od ? nvv / (float)od : 0.f;
        keep |= 1u << b;
      }
    }
    next[w] = keep;
    mine += __popc(keep);
  }
  atomicAdd(&s_cnt, mine);
  __syncthreads();
  if (threadIdx.x == 0 && s_cnt) atomicAdd(active, s_cnt);
}

// State of L1 iterations that are launched ahead of the host's checks.
struct PrLoop {
  double residual;  // of the last iteration
  uint32_t done;    // it was below the tolerance
  uint32_t iters;
  unsigned long long t[3];  // PrArgs::t
};
constexpr uint32_t kPrTimed = 8;

// Normalised update p' = teleport + damping*sum for every vertex, with the L1
// delta accumulated in FP64: per-thread, then a fixed-shape block tree, one
// partial per block (the grid size is fixed, so the order never changes).
// Bound by FP64 (few units on this part): 8.4 M vertices took 69 us with two
// conversions, a subtraction and an addition each.  new - old is first taken in
// FP32 together with its rounding error (Knuth's two-sum); where a warp's
// errors are all zero, as in most iterations but the first, the FP32
// difference is exact and costs one conversion and one addition, with the
// same bits.  Four vertices per thread and load; all four arrays are 16-byte
// aligned (their own allocations, or padded in the arena).
__global__ void __launch_bounds__(kThreads) k_pr_update_l1(uint64_t V, float *rank, float *contrib,
                                                           const float *sum, const uint32_t *outdeg,
                                                           float teleport, float damping,
                                                           double *part, const uint32_t *done) {
  __shared__ double s_d[kThreads];
  if (done && *done) return;
  double acc = 0.0;
  // one vertex's update; d = new - old in FP32, err its rounding error
  auto one = [&](float s, uint32_t od, float &r, float &c, float &old, float &d, float &err) {
    const float nvv = teleport + damping * s;
    old = r;
    d = __fsub_rn(nvv, r);
    const float t = __fsub_rn(d, nvv);
    err = __fsub_rn(__fsub_rn(nvv, __fsub_rn(d, t)), __fadd_rn(r, t));
    r = nvv;
    c = od ? nvv / (float)od : 0.f;
  };
  const uint64_t V4 = V / 4;
  for (uint64_t q = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; q < V4; q += (uint64_t)gridDim.x * blockDim.x) {
    const float4 s = reinterpret_cast<const float4 *>(sum)[q];
    const uint4 od = reinterpret_cast<const uint4 *>(outdeg)[q];
    float4 r = reinterpret_cast<float4 *>(rank)[q], c;
    float old[4], d[4], err[4];
    one(s.x, od.x, r.x, c.x, old[0], d[0], err[0]);
    one(s.y, od.y, r.y, c.y, old[1], d[1], err[1]);
    one(s.z, od.z, r.z, c.z, old[2], d[2], err[2]);
    one(s.w, od.w, r.w, c.w, old[3], d[3], err[3]);
    reinterpret_cast<float4 *>(rank)[q] = r;
    reinterpret_cast<float4 *>(contrib)[q] = c;
    const bool exact = err[0] == 0.f && err[1] == 0.f && err[2] == 0.f && err[3] == 0.f;
    if (__all_sync(__activemask(), exact)) {
#pragma unroll
      for (int i = 0; i < 4; i++) acc += (double)fabsf(d[i]);
    } else {
      acc += fabs((double)r.x - (double)old[0]);
      acc += fabs((double)r.y - (double)old[1]);
      acc += fabs((double)r.z - (double)old[2]);
      acc += fabs((double)r.w - (double)old[3]);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x < V - 4 * V4) {
    const uint64_t v = 4 * V4 + threadIdx.x;
    float old, d, err;
    one(sum[v], outdeg[v], rank[v], contrib[v], old, d, err);
    acc += fabs((double)rank[v] - (double)old);
  }
  s_d[threadIdx.x] = acc;
  __syncthreads();
  for (int s = kThreads / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) s_d[threadIdx.x] += s_d[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = s_d[0];
}

// Begins iterations: clears the state (first), or goes on with it after a wait.
__global__ void k_pr_begin(PrLoop *loop, int first) {
  if (first) *loop = PrLoop{};
  loop->t[0] = globaltimer_ns();
}

// Sum of the partials, and the end of the iteration.
__global__ void k_pr_finish(const double *part, uint32_t n, PrLoop *loop, double tol, int stamp) {
  __shared__ double s_d[kThreads];
  if (loop->done) return;
  double acc = 0.0;
  for (uint32_t i = threadIdx.x; i < n; i += kThreads) acc += part[i];
  s_d[threadIdx.x] = acc;
  __syncthreads();
  for (int s = kThreads / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) s_d[threadIdx.x] += s_d[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    loop->residual = s_d[0];
    loop->iters++;
    if (s_d[0] < tol) loop->done = 1;
    if (stamp) loop->t[0] = globaltimer_ns();  // the next iteration is timed
  }
}

__global__ void k_pr_init(uint64_t V, float *rank, float *contrib, float *sum, const uint32_t *outdeg,
                          float r0) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V;
       v += (uint64_t)gridDim.x * blockDim.x) {
    rank[v] = r0;
    const uint32_t od = outdeg[v];
    contrib[v] = od ? r0 / (float)od : 0.f;
    sum[v] = 0.f;
  }
}

__global__ void k_degree_from_offsets(uint64_t V, const uint64_t *off, uint32_t *deg) {
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V;
       v += (uint64_t)gridDim.x * blockDim.x)
    deg[v] = (uint32_t)(off[v + 1] - off[v]);
}

// ------------------------------------------------------------------ checksums

// Result checksum in a fixed reduction order (fixed grid, fixed trees):
// mode 0: {#v with value != unreached, sum of those values} (BFS, SSSP)
// mode 1: {#v with label == v (components), sum of labels}     (CC)
// mode 2: {#v, bits of the FP64 sum of the FP32 ranks}          (PR)
__global__ void __launch_bounds__(kThreads) k_checksum(const uint32_t *val, uint64_t V, int mode,
                                                       uint32_t unreached,
                                                       unsigned long long *part) {
  __shared__ unsigned long long s_c[kThreads], s_s[kThreads];
  __shared__ double s_d[kThreads];
  unsigned long long c = 0, sum = 0;
  double d = 0.0;
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V;
       v += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t x = val[v];
    if (mode == 0) {
      if (x != unreached) {
        c++;
        sum += x;
      }
    } else if (mode == 1) {
      c += (x == v) ? 1 : 0;
      sum += x;
    } else {
      c++;
      d += (double)__uint_as_float(x);
    }
  }
  s_c[threadIdx.x] = c;
  s_s[threadIdx.x] = sum;
  s_d[threadIdx.x] = d;
  __syncthreads();
  for (int k = kThreads / 2; k > 0; k >>= 1) {
    if ((int)threadIdx.x < k) {
      s_c[threadIdx.x] += s_c[threadIdx.x + k];
      s_s[threadIdx.x] += s_s[threadIdx.x + k];
      s_d[threadIdx.x] += s_d[threadIdx.x + k];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[3 * blockIdx.x] = s_c[0];
    part[3 * blockIdx.x + 1] = s_s[0];
    part[3 * blockIdx.x + 2] = __double_as_longlong(s_d[0]);
  }
}

// Sums the partials of the blocks.  The integer sums are exact in
// any order; the FP64 sum is added in block order by one thread, as it defines
// the checksum's bits, but out of shared memory (one dependent global load per
// block took 120 us).
constexpr uint32_t kChecksumBatch = 1024;
__global__ void __launch_bounds__(kThreads) k_checksum_final(const unsigned long long *part, uint32_t n, int mode,
                                                             unsigned long long *out) {
  __shared__ unsigned long long s_c, s_s;
  __shared__ double s_d[kChecksumBatch];
  if (threadIdx.x == 0) s_c = s_s = 0;
  __syncthreads();
  unsigned long long c = 0, sum = 0;
  for (uint32_t i = threadIdx.x; i < n; i += kThreads) {
    c += part[3 * i];
    sum += part[3 * i + 1];
  }
  atomicAdd(&s_c, c);
  atomicAdd(&s_s, sum);
  double d = 0.0;
  if (mode == 2)
    for (uint32_t i0 = 0; i0 < n; i0 += kChecksumBatch) {
      const uint32_t m = min(kChecksumBatch, n - i0);
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < m; i += kThreads) s_d[i] = __longlong_as_double(part[3 * (i0 + i) + 2]);
      __syncthreads();
      if (threadIdx.x == 0)
        for (uint32_t i = 0; i < m; i++) d += s_d[i];
    }
  __syncthreads();
  if (threadIdx.x == 0) {
    out[0] = s_c;
    out[1] = mode == 2 ? (unsigned long long)__double_as_longlong(d) : s_s;
  }
}

// ------------------------------------------------------------------ fills

__global__ void k_fill_u32(uint32_t *p, uint64_t n, uint32_t v) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

// Byte depths of one source (0 unreached, 1 the source, at most 254 here)
// as u32 depths with `unreached` for 0, written to dst (device memory, or
// page-locked host memory through its device pointer).  Four vertices per
// thread, one 4-byte load each, when b is 4-byte aligned (rows of a matrix
// with V not a multiple of 4 are not); else one vertex per thread.
__global__ void k_depth_expand(const uint8_t *b, uint64_t n, uint32_t unreached, uint32_t *dst) {
  if (reinterpret_cast<uintptr_t>(b) & 3u) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n;
         v += (uint64_t)gridDim.x * blockDim.x)
      dst[v] = b[v] ? b[v] : unreached;
    return;
  }
  const uint64_t n4 = n / 4;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n4;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uchar4 q = reinterpret_cast<const uchar4 *>(b)[i];
    dst[4 * i] = q.x ? q.x : unreached;
    dst[4 * i + 1] = q.y ? q.y : unreached;
    dst[4 * i + 2] = q.z ? q.z : unreached;
    dst[4 * i + 3] = q.w ? q.w : unreached;
  }
  if (blockIdx.x == 0 && threadIdx.x < n - 4 * n4) {
    const uint64_t v = 4 * n4 + threadIdx.x;
    dst[v] = b[v] ? b[v] : unreached;
  }
}

// ---------------------------------------------------------- bottom-up BFS
//
// One bottom-up level of a direction-optimizing BFS (Beamer et al., 2012)
// on a symmetric graph: every unvisited vertex scans its own neighbours, four
// records at a time, and stops at the first one in the current frontier; it
// then gets depth newdepth and joins the next frontier.  Valid because the
// graph is symmetric (a neighbour u of v has the edge u -> v).  The depths
// equal the top-down ones: a vertex is reached at level L + 1 exactly when
// one of its neighbours has depth L.  Warps cover 32 consecutive vertices
// (one bitmap word), so each word of next / visited has a single writer.
// cnt[0] += vertices reached, cnt[1] += their degrees, cnt[2] += records read
// from the host copy, cnt[3] += records read from the static region.
//
// Large levels are bound by the L1's tag lookups (every lane reads a list of its
// own), small ones by the chain visited word -> offsets -> records -> frontier
// words.  So records come through records4, frontier words two at a time, the
// next word's visited bits are fetched ahead, and the last two unfinished
// vertices of a word are scanned by the whole warp, 32 records a step (a lane
// alone on a list of 40 records kept a level waiting for 10 us).  The counts of
// records read are those of four-record steps in either form.
template <class PS>
__device__ __forceinline__ void bottom_up_words(const uint64_t *off, uint32_t V, uint32_t Vs, const PS &stat,
                                                const PS &host, const uint32_t *cur, uint32_t *visited,
                                                uint32_t *next, uint32_t *depth, uint32_t newdepth,
                                                unsigned long long *cnt, uint32_t *err) {
  __shared__ unsigned long long s_cnt[4];
  if (threadIdx.x < 4) s_cnt[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31;
  uint32_t nn = 0;
  unsigned long long nm = 0, nh = 0, ns = 0;
  const uint64_t words = ((uint64_t)V + 31) / 32, nw = (uint64_t)gridDim.x * (kThreads / 32);
  // consecutive words go to different CTAs
  uint64_t w = (uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  uint32_t vis_next = w < words ? visited[w] : 0u;
  const uint32_t cmask = stat.bc >= 32 ? 0xffffffffu : (1u << stat.bc) - 1u;
  for (; w < words; w += nw) {
    const uint32_t vis = vis_next;
    if (w + nw < words) vis_next = visited[w + nw];
    const uint64_t v = w * 32 + lane;
    const bool st = v < Vs;
    uint64_t e = 0, e1 = 0;  // this lane's unread records
    if (v < V && !((vis >> lane) & 1u)) {
      e = off[v];
      e1 = off[v + 1];
    }
    const uint64_t deg = e1 - e;
    bool found = false;
    for (uint32_t open = __ballot_sync(0xffffffffu, e < e1); open; open = __ballot_sync(0xffffffffu, e < e1)) {
      if (__popc(open) > 2) {
        const uint32_t left = (uint32_t)min((uint64_t)4, e1 - e);
        uint32_t u[4];
        const uint32_t *base = st ? stat.words : host.words;
        if (stat.bpe <= 32) {  // uniform
          records4(base, e * stat.bpe, left, stat.bpe, cmask, u);
        } else {
#pragma unroll
          for (uint32_t j = 0; j < 4; j++) {
            const uint64_t b = (e + j) * stat.bpe;
            u[j] = j < left ? stat.decode(base + (b >> 5), (uint32_t)b & 31u) : 0u;
          }
        }
        // two frontier words at a time: most vertices of a large level are
        // found by their first records
        bool hit = false;
#pragma unroll
        for (uint32_t h = 0; h < 4; h += 2) {
          uint32_t f[2] = {0u, 0u};
#pragma unroll
          for (uint32_t j = 0; j < 2; j++)
            if (h + j < left && !hit) {
              if (u[h + j] < V) f[j] = (cur[u[h + j] >> 5] >> (u[h + j] & 31)) & 1u;
              else atomicOr(err, kErrVertex);
            }
          hit |= (f[0] | f[1]) != 0u;
        }
        if (st) ns += left;
        else nh += left;
        found |= hit;
        e = hit ? e1 : e + left;
      } else {
        const int l = __ffs(open) - 1;
        const uint64_t eb = __shfl_sync(0xffffffffu, e, l), ee = __shfl_sync(0xffffffffu, e1, l);
        const uint32_t left = (uint32_t)min((uint64_t)32, ee - eb);
        bool hit = false;
        if (lane < left) {
          const uint64_t b = (eb + lane) * stat.bpe;
          const uint32_t u =
              stat.decode((w * 32 + l < Vs ? stat.words : host.words) + (b >> 5), (uint32_t)b & 31u);
          if (u < V) hit = (cur[u >> 5] >> (u & 31)) & 1u;
          else atomicOr(err, kErrVertex);
        }
        const uint32_t hb = __ballot_sync(0xffffffffu, hit);
        if ((int)lane == l) {
          const uint32_t got = hb ? min(left, ((uint32_t)(__ffs(hb) - 1) / 4 + 1) * 4) : left;
          if (st) ns += got;
          else nh += got;
          found |= hb != 0u;
          e = hb ? e1 : e + left;
        }
      }
    }
    const uint32_t ball = __ballot_sync(0xffffffffu, found);
    if (lane == 0) {
      next[w] = ball;
      if (ball) visited[w] = vis | ball;
    }
    if (found) {
      depth[v] = newdepth;
      nn++;
      nm += deg;
    }
  }
  nn = __reduce_add_sync(0xffffffffu, nn);
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    nm += __shfl_xor_sync(0xffffffffu, nm, o);
    nh += __shfl_xor_sync(0xffffffffu, nh, o);
    ns += __shfl_xor_sync(0xffffffffu, ns, o);
  }
  if (lane == 0) {  // one global atomic per CTA and counter
    if (nn) atomicAdd(&s_cnt[0], (unsigned long long)nn);
    if (nm) atomicAdd(&s_cnt[1], nm);
    if (nh) atomicAdd(&s_cnt[2], nh);
    if (ns) atomicAdd(&s_cnt[3], ns);
  }
  __syncthreads();
  if (threadIdx.x < 4 && s_cnt[threadIdx.x]) atomicAdd(cnt + threadIdx.x, s_cnt[threadIdx.x]);
}

template <class PS>
__global__ void __launch_bounds__(kThreads) k_bfs_bottom_up(const uint64_t *off, uint32_t V, uint32_t Vs, PS stat,
                                                            PS host, const uint32_t *cur, uint32_t *visited,
                                                            uint32_t *next, uint32_t *depth, uint32_t newdepth,
                                                            unsigned long long *cnt, uint32_t *err) {
  bottom_up_words(off, V, Vs, stat, host, cur, visited, next, depth, newdepth, cnt, err);
}

// ------------------------------------------------------------ union-find CC
//
// Connected components of a symmetric graph by sampling union-find (the
// Afforest scheme): hook every vertex with its first two neighbours, find the
// giant component, then expand only the edges of vertices outside it.  A
// root is hooked only under a smaller root (CAS on parent[hi] == hi), so
// parent[x] <= x holds at all times and the root of every tree is the
// smallest vertex id in it: after compression parent[] is exactly the
// reference's CC label (minimum id of the component) with no relabelling.
// Walks follow strictly decreasing ids, so they end within V steps; a broken
// invariant sets kErrVertex instead of looping.

// Parents are read through L1.  The giant component's root is read by every
// walk, and from the L2 those reads of one line run one after another (linking
// 8.4 M vertices: 0.95 ms so, 0.27 ms through L1); a stale parent is an older ancestor, so a walk only ends too early, at a vertex that
// is no root any more, and the compare-and-swap on it returns the newer one.
__device__ __forceinline__ uint32_t uf_find(uint32_t *par, uint32_t x, uint32_t V, uint32_t *err) {
  for (uint32_t steps = 0; steps <= V; steps++) {
    const uint32_t p = __ldca(par + x);
    if (p == x) return x;
    if (p > x) {
      atomicOr(err, kErrVertex);
      return x;
    }
    const uint32_t gp = __ldca(par + p);
    if (gp < p) __stcg(par + x, gp);  // path halving: gp is an ancestor of x
    x = gp;
  }
  atomicOr(err, kErrVertex);
  return x;
}

__device__ __forceinline__ void uf_link(uint32_t *par, uint32_t a, uint32_t b, uint32_t V, uint32_t *err) {
  for (uint32_t tries = 0; tries <= V; tries++) {
    a = uf_find(par, a, V, err);
    b = uf_find(par, b, V, err);
    if (a == b) return;
    const uint32_t hi = max(a, b), lo = min(a, b);
    const uint32_t old = atomicCAS(par + hi, hi, lo);
    if (old == hi) return;
    a = old;  // hi had a parent already: go on from it
    b = lo;
  }
  atomicOr(err, kErrVertex);
}

// First sampling pass: reads every vertex's first two records (one or two
// 16-byte loads, where the passes used to fetch the same link sector twice) and
// hooks v under its first neighbour when that is smaller: parents are smaller
// than their vertices from the start, so a plain store does it, where linking
// all first edges by compare-and-swap spent 0.8 ms of retries on 2^23
// vertices.  What is left of the two edges (a larger first neighbour, the
// second one) goes to pend for k_uf_link.
template <class PS>
__global__ void __launch_bounds__(kThreads) k_uf_init(const uint64_t *off, uint32_t V, uint64_t static_edges, PS stat,
                                                      PS host, uint32_t *par, uint2 *pend, unsigned long long *reads,
                                                      uint32_t *states, uint32_t nstate, uint32_t *err) {
  if (blockIdx.x == 0)  // the barrier states of the compressions to come
    for (uint32_t i = threadIdx.x; i < nstate; i += kThreads) states[i] = 0u;
  const uint32_t cmask = stat.bc >= 32 ? 0xffffffffu : (1u << stat.bc) - 1u;
  uint32_t nh = 0, ns = 0;  // records read from the host copy / the static region
  for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < V; v += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t o = off[v];
    const uint32_t n = (uint32_t)min((uint64_t)2, off[v + 1] - o);
    const bool st = o < static_edges;
    const uint32_t *base = st ? stat.words : host.words;
    uint32_t u[4] = {0u, 0u, 0u, 0u};
    if (n) {
      if (stat.bpe <= 32) {  // uniform
        records4(base, o * stat.bpe, n, stat.bpe, cmask, u);
      } else {
        for (uint32_t j = 0; j < n; j++) {
          const uint64_t b = (o + j) * stat.bpe;
          u[j] = stat.decode(base + (b >> 5), (uint32_t)b & 31u);
        }
      }
    }
    if (st) ns += n;
    else nh += n;
    uint32_t p = (uint32_t)v;
    uint2 rest = make_uint2(0xffffffffu, 0xffffffffu);
    if ((n > 0 && u[0] >= V) || (n > 1 && u[1] >= V)) {
      atomicOr(err, kErrVertex);
    } else {
      if (n > 0) {
        if (u[0] < p) p = u[0];
        else rest.x = u[0];
      }
      if (n > 1) rest.y = u[1];
    }
    par[v] = p;
    pend[v] = rest;
  }
  nh = __reduce_add_sync(0xffffffffu, nh);
  ns = __reduce_add_sync(0xffffffffu, ns);
  if ((threadIdx.x & 31) == 0) {  // reads[0]: host records, reads[1]: static records
    if (nh) atomicAdd(reads, (unsigned long long)nh);
    if (ns) atomicAdd(reads + 1, (unsigned long long)ns);
  }
}

// The sampled edges that k_uf_init left over.  On a graph with a giant component
// most of them join the same few roots at the same time, and compare-and-swaps
// on one address run one after another in the L2: the lanes of a warp that want
// to hook the same root send one (8.4 M vertices: 1.1 ms with a swap per lane).
__global__ void __launch_bounds__(kThreads) k_uf_link(const uint2 *pend, uint32_t V, uint32_t *par, uint32_t *err) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) & ~31ull; base < V; base += stride) {
    const uint64_t v = base + lane;
    const uint2 r = v < V ? pend[v] : make_uint2(0xffffffffu, 0xffffffffu);
#pragma unroll 1
    for (int k = 0; k < 2; k++) {
      uint32_t x = (uint32_t)v, y = k ? r.y : r.x;
      bool todo = y != 0xffffffffu;
      for (uint32_t tries = 0; __any_sync(0xffffffffu, todo); tries++) {
        if (tries > V) {  // a broken forest: report, never hang
          if (todo) atomicOr(err, kErrVertex);
          break;
        }
        if (todo) {
          x = uf_find(par, x, V, err);
          y = uf_find(par, y, V, err);
          todo = x != y;
        }
        __syncwarp();
        const uint32_t hi = max(x, y), lo = min(x, y);
        const uint32_t same = __match_any_sync(0xffffffffu, todo ? hi : 0xffffffffu);
        uint32_t old = hi;
        const int first = __ffs(same) - 1;
        const bool mine = todo && (int)lane == first;
        if (mine) old = atomicCAS(par + hi, hi, lo);
        if (mine && old == hi) todo = false;
        old = __shfl_sync(0xffffffffu, mine && old == hi ? lo : old, first);  // hi's parent now
        if (todo) {
          x = old;
          y = lo;
        }
        __syncwarp();
      }
    }
  }
}

// Roots of k pseudo-random vertices (after compression), for the host to
// pick the most frequent one as the giant component.
__global__ void k_uf_roots(const uint32_t *par, uint32_t V, uint32_t k, uint32_t *roots) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= k) return;
  uint64_t z = 0x9e3779b97f4a7c15ull * (i + 1);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  z ^= z >> 31;
  roots[i] = __ldcg(par + (uint32_t)(z % V));
}

// Frontier of the final pass: vertices of degree > 2 (their first two edges
// are already linked) outside component c.  A lane per vertex, a warp per
// bitmap word.
__global__ void __launch_bounds__(kThreads) k_uf_mark(const uint64_t *off, const uint32_t *par, uint32_t V,
                                                      uint32_t c, uint32_t *bits, uint64_t nwords) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t nw = (uint64_t)gridDim.x * (kThreads / 32);
  for (uint64_t w = (blockIdx.x * (uint64_t)kThreads + threadIdx.x) >> 5; w < nwords; w += nw) {
    const uint64_t v = w * 32 + lane;
    const bool on = v < V && par[v] != c && off[v + 1] - off[v] > 2;
    const uint32_t word = __ballot_sync(0xffffffffu, on);
    if (lane == 0) bits[w] = word;
  }
}

// LBS op of the final pass: link the source vertex with every neighbour.
struct UnionOp {
  using Val = uint32_t;
  static constexpr bool kNeedVal = true;
  uint32_t *par, *err;
  uint32_t V;
  __device__ uint32_t src_val(uint32_t v) const { return v; }
  using Probe = uint32_t;  // the neighbour's parent (read early; links re-read it)
  template <class Edge>
  __device__ __forceinline__ Probe probe(Edge e) const {
    const uint32_t v = edge_dst(e);
    return v < V ? __ldcg(par + v) : 0u;
  }
  template <class Edge>
  __device__ __forceinline__ void relax(Edge e, uint32_t sv, uint64_t, Probe) const {
    const uint32_t v = edge_dst(e);
    if (v >= V) {
      atomicOr(err, kErrVertex);
      return;
    }
    uf_link(par, sv, v, V, err);
  }
};

__global__ void k_iota_u32(uint32_t *p, uint64_t n) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    p[i] = (uint32_t)i;
}

// bits [0, V) set, the rest of the words cleared
__global__ void k_fill_bits(uint32_t *bits, uint64_t nwords, uint64_t V) {
  for (uint64_t w = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; w < nwords;
       w += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t b = w * 32;
    bits[w] = b + 32 <= V ? 0xffffffffu : (b >= V ? 0u : ((1u << (V - b)) - 1u));
  }
}

__global__ void k_set_source(uint32_t *value, uint32_t src, uint32_t val, uint32_t *bits_a,
                             uint32_t *bits_b) {
  value[src] = val;
  bits_a[src >> 5] |= 1u << (src & 31);
  if (bits_b) bits_b[src >> 5] |= 1u << (src & 31);
}

}  // namespace og
