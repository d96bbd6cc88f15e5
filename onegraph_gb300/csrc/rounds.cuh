// rounds.cuh — device-driven rounds of single-source BFS, SSSP and label
// propagation: one cooperative kernel runs a whole query.
//
// The host-driven loop (engine.cu run_frontier) waits for every round's
// counts before it launches the next kernels; replaying a captured graph of
// a round's kernels still pays seven to eleven launches and their gaps a round
// (28 us a level of a road-like BFS, 46 us a round of a resident SSSP, most of
// it with the GPU idle).  Here the CTAs stay resident and the phases of a
// round are separated by grid barriers:
//   scan   every warp takes groups of words of the frontier bitmap and appends
//          the vertices it lists, their degree prefix and tile map to one list
//          per region; a 64-bit atomic reserves list entries and edge positions
//          together, so the order of the appends does not matter
//   relax  edge-balanced tiles of both lists, interleaved (lbs_tile)
// Rounds of very many tiles are handed over: the kernel ends after the scan, the
// host launches the relax on its own and then this kernel again (kHandRelax).
// Small BFS frontiers are expanded by a kernel of one CTA out of shared memory,
// level after level.
//
// The control logic is the host loop's, step for step (direction-optimizing
// BFS of Beamer et al. 2012 on symmetric graphs, top-down otherwise; near/far
// SSSP), and every CTA computes it from the same counters.  Data that other
// CTAs wrote in an earlier phase is read with plain loads: the barrier's
// acquire orders them (and drops stale L1 lines).
#pragma once
#include <cstddef>
#include <type_traits>

#include "batch_persist.cuh"
#include "kernels.cuh"

namespace og {

// A list reservation packs both of its counters into 64 bits: vertices above,
// edge positions below, as many bits as the graph's edge count takes.  Graphs
// whose two counts do not fit take the host-driven loop (2^28 vertices go with
// up to 2^35 edges, 240 GB of records).
inline uint32_t append_shift(uint64_t E) {
  uint32_t b = 1;
  while (E >> b) b++;
  return b;
}
inline bool rounds_fit(uint64_t V, uint64_t E) { return append_shift(V) + append_shift(E) <= 64; }
__host__ __device__ __forceinline__ uint64_t append_edges(unsigned long long app, uint32_t shift) {
  return app & ((1ull << shift) - 1);
}

// Counters of one scan and the relax after it.  Four of them are used in turn:
// after the barrier that ends scan s, CTA 0 clears the one of scan s + 2, whose
// last readers passed an earlier barrier.
struct alignas(128) RoundSlot {
  unsigned long long app[2];  // list reservations of the two regions
  uint32_t tile_next;         // tile counter of the relax
  uint32_t far_min;           // smallest waiting value the scan saw
  uint32_t near;              // the relax lowered a value below the threshold
  uint32_t far_cand;          // smallest value at or above it that the relax wrote
  unsigned long long bu[4];   // bottom-up: reached, their degrees, host / static records
};

struct RoundsState {
  unsigned long long bar;  // grid barrier: arrivals so far (polled: on a line of its own)
  alignas(128) uint32_t err;
  uint32_t posted;  // in the host's copy: the rest of it is there (rounds_post)
  // results for the host
  unsigned long long iterations, frontier_sum, edges_static, edges_dynamic;
  unsigned long long ns_total, ns_relax;
  // BFS state handed from launch to launch
  unsigned long long unexplored, fn;
  uint32_t level, par, bottom, counted, done;
  uint32_t small, n0, n;  // the frontier is listed: n0 static vertices, n in all
  // round handed over to a launch of its own (kHand*), and what it needs
  uint32_t hand, thr, far_min, pad0;
  unsigned long long hx[2];   // list reservations of the two regions
  unsigned long long hbu[4];  // bottom-up counts, taken by that launch
  RoundSlot slot[4];
};

struct RoundsArgs {
  uint32_t V, Vs;
  uint64_t E, static_edges, nwords;
  const uint64_t *off;
  uint32_t *value;
  uint32_t *bm[3];  // frontier by parity; BFS visited / SSSP waiting
  uint32_t *list[2];
  uint64_t *pref[2];
  uint32_t *tile[2];
  uint64_t list_cap[2], tile_cap[2];
  RoundsState *st;
  RoundsState *post;  // the host's copy, page-locked
  uint32_t *result;   // when not null: page-locked, takes the values of a query that has ended
  uint32_t src, delta, split, dopt, timer;
  uint32_t shift;  // of the vertex counter in a list reservation
  uint32_t spin_limit;
  uint64_t hand_hbm, hand_link;  // rounds of more tiles are handed over (hands_over)
  uint32_t hand_bottom;          // bottom-up levels are
};

// A round of many tiles is faster as a launch of one CTA per tile: the tables of
// a CTA's next tile are then built while its neighbours' reads are under way,
// where a CTA of this kernel waits for all its warps between two tiles, with
// fewer CTAs on the SM.  The state is kept in RoundsState meanwhile.  The line
// between the limits is where the link takes as long as HBM: 42 G edges/s
// against 160 (top-down BFS, R-MAT 24).
constexpr uint32_t kHandRelax = 1, kHandBottomUp = 2;
__device__ __forceinline__ bool hands_over(const RoundsArgs &a, uint64_t n0, uint64_t n1) {
  return n0 + n1 > (4 * n1 > n0 ? a.hand_link : a.hand_hbm);
}

// Results of up to this many vertices are stored to page-locked memory by the
// kernel that ends the query and copied to the caller's array by the host: a
// copy-engine transfer takes 5-11 us to start, a pageable target as long again.
// BFS, stored / copied: 17 thousand vertices 88.4 / 91.2 us, 28 thousand 75.3 / 76.3,
// 40 thousand 80.2 / 78.4, 0.1 M 117 / 103.
constexpr uint32_t kPostedResult = 1u << 15;

// All CTAs, after the last value has been written.
__device__ __forceinline__ void rounds_result(const RoundsArgs &a) {
  if (!a.result) return;
  for (uint32_t v = blockIdx.x * kThreads + threadIdx.x; v < a.V; v += gridDim.x * kThreads)
    a.result[v] = __ldcg(a.value + v);
}

// One thread, as the last thing a launch does: the state for the host.
__device__ __forceinline__ void rounds_post(const RoundsArgs &a) {
  constexpr size_t n = (offsetof(RoundsState, slot) - offsetof(RoundsState, err)) / 16;
  const uint4 *s = reinterpret_cast<const uint4 *>(&a.st->err);
  uint4 *d = reinterpret_cast<uint4 *>(&a.post->err);
#pragma unroll
  for (size_t i = 0; i < n; i++) d[i] = __ldcg(s + i);  // posted among them: 0 on the device
  __threadfence_system();
  *const_cast<volatile uint32_t *>(&a.post->posted) = 1u;
}

__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long *p) {
  return cuda::atomic_ref<const unsigned long long, cuda::thread_scope_device>(*p).load(cuda::memory_order_relaxed);
}

// Grid barrier over one counter of arrivals: `target`, which thread 0 keeps, grows by
// the grid size with every barrier.  The polls are relaxed and one acquire fence follows
// them: an acquiring poll drops the SM's whole L1 each time, under the CTAs
// that still work (a round's relax, resident SSSP of 0.3 M vertices: 13-15 us
// on average so, 9 us now).  A wait longer than `limit` polls (wait_limit) sets
// kErrBarrier and returns false instead of hanging.
__device__ __forceinline__ bool rounds_sync(RoundsState *st, unsigned long long &target, uint32_t limit) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    target += gridDim.x;
    __threadfence();
    atomicAdd(&st->bar, 1ull);
    uint32_t spins = 0;
    while (ld_relaxed64(&st->bar) < target) {
      if (++spins > limit) {
        atomicOr(&st->err, kErrBarrier);
        ok = 0;
        break;
      }
      __nanosleep(spins < 256 ? 20 : 200);
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// Scan of a frontier, a warp per group of `gw` consecutive bitmap words (1 to
// 32, one per lane): no block barriers, so a warp's chain is words -> (value
// ->) offsets -> reservation -> list.  Set bits are listed in shared memory,
// kScanBatch at a time, and a batch's vertices spread over the lanes.
constexpr uint32_t kScanLane = 4, kScanBatch = 32 * kScanLane;
struct ScanWarp {
  uint16_t list[kScanBatch];
  uint32_t near[32], far[32];
};
struct ScanShared {
  ScanWarp w[kThreads / 32];
};

// Lists the set bits of `word` (lane l: word wt + l; bits of one region) that
// are near (value below thr, or any without kSplit) and have edges, in region
// r's list.  near / far bits are left in sh.near / sh.far; returns the lane's
// smallest far value.
template <bool kSplit>
__device__ __forceinline__ uint32_t scan_group(const RoundsArgs &a, ScanWarp &sh, uint64_t wt, uint32_t word, int r,
                                               uint32_t thr, unsigned long long *app) {
  const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u;
  const uint64_t vbase = wt * 32;
  uint32_t tmin = 0xffffffffu, ex = __popc(word);
  const uint32_t pc = ex;
#pragma unroll
  for (uint32_t d = 1; d < 32; d <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, ex, d);
    if (lane >= d) ex += x;
  }
  const uint32_t N = __shfl_sync(0xffffffffu, ex, 31);
  ex -= pc;
  const uint32_t nzw = __ballot_sync(0xffffffffu, word != 0u);
  const bool dense = N > 4 * __popc(nzw);
#pragma unroll 1
  for (uint32_t p0 = 0; p0 < N; p0 += kScanBatch) {
    const uint32_t m = min(kScanBatch, N - p0);
    __syncwarp();
    if (dense) {  // all lanes on one word after another
      for (uint32_t b = nzw; b; b &= b - 1) {
        const int l = __ffs(b) - 1;
        const uint32_t x = __shfl_sync(0xffffffffu, word, l);
        const uint32_t k = __shfl_sync(0xffffffffu, ex, l) + __popc(x & below) - p0;
        if (((x >> lane) & 1u) && k < kScanBatch) sh.list[k] = (uint16_t)(l * 32 + lane);
      }
    } else if (ex < p0 + kScanBatch && ex + pc > p0) {
      uint32_t k = ex - p0;
      for (uint32_t x = word; x; x &= x - 1, k++)
        if (k < kScanBatch) sh.list[k] = (uint16_t)(lane * 32 + __ffs(x) - 1);
    }
    __syncwarp();
    const uint32_t q = (m + 31) / 32, i0 = lane * q;  // lane's entries: [i0, i0 + q)
    uint32_t lv[kScanLane], val[kScanLane];
    uint64_t d[kScanLane];
#pragma unroll
    for (uint32_t j = 0; j < kScanLane; j++) {
      lv[j] = j < q && i0 + j < m ? sh.list[i0 + j] : 0xffffffffu;
      val[j] = kSplit && lv[j] != 0xffffffffu ? __ldcg(a.value + vbase + lv[j]) : 0u;
    }
#pragma unroll
    for (uint32_t j = 0; j < kScanLane; j++) {
      d[j] = 0;
      if (lv[j] != 0xffffffffu && (!kSplit || val[j] < thr))
        d[j] = a.off[vbase + lv[j] + 1] - a.off[vbase + lv[j]];
    }
    uint32_t cnt = 0;
    uint64_t sum = 0;
#pragma unroll
    for (uint32_t j = 0; j < kScanLane; j++) {
      if (kSplit && lv[j] != 0xffffffffu) {
        const uint32_t bit = 1u << (lv[j] & 31);
        if (val[j] < thr) {
          atomicOr(&sh.near[lv[j] >> 5], bit);
        } else {
          atomicOr(&sh.far[lv[j] >> 5], bit);
          tmin = min(tmin, val[j]);
        }
      }
      cnt += d[j] ? 1u : 0u;
      sum += d[j];
    }
    uint32_t ic = cnt;
    uint64_t is = sum;
#pragma unroll
    for (uint32_t s = 1; s < 32; s <<= 1) {
      const uint32_t xc = __shfl_up_sync(0xffffffffu, ic, s);
      const uint64_t xs = __shfl_up_sync(0xffffffffu, is, s);
      if (lane >= s) {
        ic += xc;
        is += xs;
      }
    }
    const uint32_t tn = __shfl_sync(0xffffffffu, ic, 31);
    if (tn == 0) continue;
    unsigned long long base = 0;
    if (lane == 31) base = atomicAdd(app, ((unsigned long long)tn << a.shift) | is);
    base = __shfl_sync(0xffffffffu, base, 31);
    const uint64_t te = __shfl_sync(0xffffffffu, is, 31);
    uint32_t pos = (uint32_t)(base >> a.shift);
    uint64_t ep = append_edges(base, a.shift);
    uint32_t *list = a.list[r], *tile = a.tile[r];
    uint64_t *pref = a.pref[r];
    if ((uint64_t)pos + tn > a.list_cap[r] || (ep + te + kTile - 1) / kTile > a.tile_cap[r]) {
      if (lane == 0) atomicOr(&a.st->err, kErrTileMap);
      continue;
    }
    // the entry after the batch's last: the next append writes the same value
    if (lane == 0) pref[pos + tn] = ep + te;
    pos += ic - cnt;
    ep += is - sum;
#pragma unroll
    for (uint32_t j = 0; j < kScanLane; j++) {
      uint64_t t = 0, tend = 0;  // tiles that start inside this vertex
      if (d[j]) {
        list[pos] = (uint32_t)(vbase + lv[j]);
        pref[pos] = ep;
        t = (ep + kTile - 1) / kTile;
        tend = (ep + d[j] + kTile - 1) / kTile;
      }
      const uint32_t big = __ballot_sync(0xffffffffu, tend > t + 8);
      if (tend <= t + 8)
        for (; t < tend; t++) tile[t] = pos;
      for (uint32_t b = big; b; b &= b - 1) {  // a hub's tiles: the whole warp
        const int l = __ffs(b) - 1;
        const uint64_t ts = __shfl_sync(0xffffffffu, t, l), te2 = __shfl_sync(0xffffffffu, tend, l);
        const uint32_t p = __shfl_sync(0xffffffffu, pos, l);
        for (uint64_t x = ts + lane; x < te2; x += 32) tile[x] = p;
      }
      pos += d[j] ? 1u : 0u;
      ep += d[j];
    }
  }
  return tmin;
}

// BFS (kSplit = false, kZeroCur = false): lists `cur` and clears `next`, whose
// bits are the level before.  SSSP / CC (kZeroCur): lists `cur`, which is
// cleared; with kSplit, far vertices join the waiting set and near ones leave
// it, and with `merge` the waiting set is scanned too.  A warp owns its
// group's words, so no bitmap update needs an atomic.  Small graphs get small
// groups, so that the frontier is spread over all warps.
// Not inlined, as the other phases: inlined, 300-460 B a thread were spilled.  What
// spills now is a few words around the calls (24-28 B a thread in k_min_rounds, 160
// in k_bfs_rounds) and in the scans (up to 76 B), not in the loops over tiles.
template <bool kSplit, bool kZeroCur>
__device__ __noinline__ void scan_frontier(const RoundsArgs &a, ScanShared &shared, uint32_t *cur, uint32_t *next,
                                           uint32_t *waiting, bool merge, uint32_t thr, RoundSlot *slot) {
  ScanWarp &sh = shared.w[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t words = ((uint64_t)a.V + 31) / 32, nwarps = (uint64_t)gridDim.x * (kThreads / 32);
  uint32_t gw = 1;
  while (gw < 32 && gw * nwarps < words) gw *= 2;
  uint32_t tmin = 0xffffffffu;
  // consecutive groups go to different CTAs
  const uint64_t warp = (uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  for (uint64_t wt = warp * gw; wt < words; wt += nwarps * gw) {
    const uint64_t w = wt + lane;
    const bool on = lane < gw && w < words;
    const uint32_t cw = on ? cur[w] : 0u;
    uint32_t ww = on && kSplit && merge ? waiting[w] : 0u;
    if (!kZeroCur && on) next[w] = 0u;
    const uint32_t word = cw | ww;
    if (!__any_sync(0xffffffffu, word != 0u)) continue;
    if (kSplit) {
      if (!merge && word) ww = waiting[w];
      sh.near[lane] = sh.far[lane] = 0u;
    }
    // static vertices first, then dynamic ones; one group at most holds both
    const uint64_t vb = w * 32;
    const uint32_t smask = vb + 32 <= a.Vs ? 0xffffffffu : (vb >= a.Vs ? 0u : (1u << (a.Vs - vb)) - 1u);
    if (wt * 32 < a.Vs) tmin = min(tmin, scan_group<kSplit>(a, sh, wt, word & smask, 0, thr, &slot->app[0]));
    if ((wt + gw) * 32 > a.Vs) tmin = min(tmin, scan_group<kSplit>(a, sh, wt, word & ~smask, 1, thr, &slot->app[1]));
    __syncwarp();
    if (kSplit && word) {
      const uint32_t wnew = (ww & ~sh.near[lane]) | sh.far[lane];
      if (wnew != ww) waiting[w] = wnew;
    }
    if (kZeroCur && cw) cur[w] = 0u;
    __syncwarp();
  }
  if (kSplit) {
    const uint32_t m = block_min_u32(tmin);
    if (threadIdx.x == 0 && m != 0xffffffffu) atomicMin(&slot->far_min, m);
  }
}

__device__ __forceinline__ uint64_t list_tiles(unsigned long long app, uint32_t shift) {
  return (append_edges(app, shift) + kTile - 1) / kTile;
}

__device__ __forceinline__ void slot_clear(RoundSlot *s) {
  s->app[0] = s->app[1] = 0;
  s->tile_next = 0;
  s->far_min = s->far_cand = 0xffffffffu;
  s->near = 0;
  s->bu[0] = s->bu[1] = s->bu[2] = s->bu[3] = 0;
}

// What a CTA's threads have in common lives in shared memory, and one tile body
// serves both regions: the regions' arguments kept in registers across the tile
// loop cost 98 registers per thread (2 CTAs per SM), and the op, the barrier's
// target and the timers as many spills.
template <class Src, class Op>
struct RelaxShared {
  LbsArgs a[2];
  Src s[2];
  PairTile pt[2];
  uint32_t b[2];
  Op op;
  unsigned long long target;
  uint32_t shift;
};

// Relax of both regions' lists.  A CTA's first tile is its index in the grid
// (a list with fewer tiles than CTAs is spread over all of them, whichever
// left the barrier first); the others are handed out by an atomic counter, so
// CTAs that got cheap tiles take more.  When there are fewer tiles than CTAs,
// each is split into up to eight parts of 256 positions: one SM takes 12 us
// over a full tile's 4096 atomics, and a round of three tiles used three SMs
// (resident SSSP of 0.3 M vertices: 1.12 ms with whole tiles, 0.86 with parts).
// The next ticket (and its region split, by thread 0) is fetched while the
// current tile runs.
template <class Src, class Op>
__device__ __noinline__ void relax_lists(RelaxShared<Src, Op> &rs, LbsSh<Op> &sh, RoundSlot *slot) {
  __builtin_assume(__isShared(&rs));  // shared, not generic, accesses
  __builtin_assume(__isShared(&sh));
  if (threadIdx.x == 0) {
    for (int r = 0; r < 2; r++) {
      const unsigned long long x = slot->app[r];
      LbsArgs &l = rs.a[r];
      l.n = (uint32_t)(x >> rs.shift);
      l.total = l.pos_end = append_edges(x, rs.shift);
    }
  }
  __syncthreads();
  const uint64_t n0 = (rs.a[0].total + kTile - 1) / kTile, n1 = (rs.a[1].total + kTile - 1) / kTile;
  uint32_t parts = 1;
  while (parts < kItems && (n0 + n1) * parts * 2 <= gridDim.x) parts *= 2;
  const uint64_t n = (n0 + n1) * parts;
  if (threadIdx.x == 0) {
    rs.b[0] = blockIdx.x;
    if (rs.b[0] < n) rs.pt[0] = pair_split(rs.b[0] / parts, n0, n0 + n1);
  }
  __syncthreads();
  for (int k = 0;; k ^= 1) {
    const uint32_t b = rs.b[k];
    if (b >= n) break;
    const PairTile pt = rs.pt[k];
    if (threadIdx.x == 0) {
      const uint32_t nb = gridDim.x + atomicAdd(&slot->tile_next, 1u);
      rs.b[k ^ 1] = nb;
      if (nb < n) rs.pt[k ^ 1] = pair_split(nb / parts, n0, n0 + n1);
    }
    lbs_tile(rs.a[pt.r], rs.s[pt.r], rs.op, sh, pt.t, b % parts, parts);
    __syncthreads();  // the tile tables are rebuilt and the next ticket is read after this
  }
}

template <class Src, class Op>
__device__ __forceinline__ void relax_setup(const RoundsArgs &a, RelaxShared<Src, Op> &rs, const Src &s0,
                                            const Src &s1) {
  if (threadIdx.x == 0) {
    for (int r = 0; r < 2; r++) {
      LbsArgs &l = rs.a[r];
      l.list = a.list[r];
      l.pref = a.pref[r];
      l.tile_first = a.tile[r];
      l.pos_begin = 0;
      l.off = a.off;
      l.stage_base = 0;
      l.edge_bound = r ? a.E : a.static_edges;
      l.err = &a.st->err;
    }
    rs.s[0] = s0;
    rs.s[1] = s1;
    rs.target = 0;
    rs.shift = a.shift;
  }
}

// ------------------------------------------------------------ SSSP and CC

// MinOp, in shared memory, that also notes whether the CTA lowered a value below
// the threshold and the smallest value at or above it that it wrote: the next
// round then needs no scan to learn that nothing near is left.
template <bool kWeighted>
struct MinRoundOp : MinOp<kWeighted> {
  uint32_t thr;
  mutable uint32_t near, far_cand;
  template <class Edge>
  __device__ __forceinline__ void relax(Edge e, uint32_t sv, uint64_t, uint32_t p) const {
    const uint32_t v = edge_dst(e);
    if (v >= this->V) {
      atomicOr(this->err, kErrVertex);
      return;
    }
    const uint32_t cand = kWeighted ? sv + edge_w(e) : sv;
    if (cand >= p) return;
    atomicMin(this->value + v, cand);
    atomicOr(this->next + (v >> 5), 1u << (v & 31));
    if constexpr (!kWeighted) return;  // no threshold
    if (cand < thr) near = 1u;
    else if (cand < far_cand) atomicMin(&far_cand, cand);  // seldom: the smallest so far is read first
  }
};

// Eight records at a time do not fit: the tile loop spills 160 B a thread for
// weighted ones (64 registers, four CTAs per SM) and 64 B for columns, 68 B and
// none with four.  Resident SSSP of 0.3 M vertices 874 us with eight, 856 with four;
// label propagation over the link, R-MAT 20, 1.02 ms and 0.98.
template <bool kWeighted>
struct OpGroup<MinRoundOp<kWeighted>> {
  static constexpr int value = 4;
};

// SSSP from a.src (kWeighted; a.split: near/far with width a.delta) or label
// propagation.  A round whose relax lowered nothing below the threshold is
// followed by one scan of frontier and waiting set together at the advanced
// threshold (the host loop scans the frontier, then the waiting set).
// CTAs per SM, measured: three for label propagation and BFS (80 registers,
// 23 M directed edges 529 us against 534-566 at four; resident BFS of 2^20 vertices
// 175 against 183), four for SSSP, whose host-link rounds want more reads in
// flight (2^24 vertices 12.66 ms against 12.74 at three and 12.71 at five; resident
// queries of 0.3 M vertices would rather have three: 0.78 ms against 0.86 and 0.94).
template <bool kWeighted>
__global__ void __launch_bounds__(kThreads, kWeighted ? 4 : 3) k_min_rounds(const __grid_constant__ RoundsArgs a,
                                                                           const __grid_constant__ SrcP<kWeighted> s0,
                                                                           const __grid_constant__ SrcP<kWeighted> s1) {
  using Op = MinRoundOp<kWeighted>;
  __shared__ union {
    LbsSh<Op> lbs;
    ScanShared scan;
  } sh;
  __shared__ RelaxShared<SrcP<kWeighted>, Op> rs;
  RoundsState *st = a.st;
  const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
  if (lead) st->ns_total -= globaltimer_ns();
  // initial values and frontier (SSSP/oneGraph/GraphMeta.h:376-381,
  // CC/onegraph/GraphMeta.h:341-345); the host cleared st
  const bool resume = st->hand != 0;  // behind the relax of a round handed over
  const uint64_t gid = blockIdx.x * (uint64_t)kThreads + threadIdx.x, gsz = (uint64_t)gridDim.x * kThreads;
  if (!resume) {
    for (uint64_t v = gid; v < a.V; v += gsz) a.value[v] = kWeighted ? (v == a.src ? 1u : 0xffffffffu) : (uint32_t)v;
    for (uint64_t w = gid; w < a.nwords; w += gsz) {
      const uint64_t b = w * 32;
      uint32_t x = 0;
      if (!kWeighted) x = b + 32 <= a.V ? 0xffffffffu : (b >= a.V ? 0u : (1u << (a.V - b)) - 1u);
      else if (w == a.src >> 5) x = 1u << (a.src & 31);
      a.bm[0][w] = x;
      a.bm[1][w] = 0u;
      if (a.split) a.bm[2][w] = 0u;
    }
  }
  relax_setup(a, rs, s0, s1);
  if (lead)
    for (int i = 0; i < 4; i++) slot_clear(st->slot + i);
  uint64_t t = 1ull + a.delta;
  uint32_t par = resume ? st->par : 0u, far_min = resume ? st->far_min : 0xffffffffu;
  uint32_t thr = resume ? st->thr : !a.split || t > 0xffffffffull ? 0xffffffffu : (uint32_t)t;
  if (!rounds_sync(st, rs.target, a.spin_limit)) return;

  bool merge = false, hand = false;
  for (uint32_t seq = 0;; seq++) {
    RoundSlot *slot = st->slot + (seq & 3u);
    if (a.split) scan_frontier<true, true>(a, sh.scan, a.bm[par], nullptr, a.bm[2], merge, thr, slot);
    else scan_frontier<false, true>(a, sh.scan, a.bm[par], nullptr, nullptr, false, 0u, slot);
    if (!rounds_sync(st, rs.target, a.spin_limit)) return;
    if (lead) slot_clear(st->slot + ((seq + 2) & 3u));
    const unsigned long long x0 = slot->app[0], x1 = slot->app[1];
    const uint64_t n = (x0 >> a.shift) + (x1 >> a.shift);
    if (a.split) far_min = merge ? slot->far_min : min(far_min, slot->far_min);
    if (n == 0) {
      if (!a.split || far_min == 0xffffffffu) break;
      t = (uint64_t)far_min + a.delta;
      thr = t > 0xffffffffull ? 0xffffffffu : (uint32_t)t;
      merge = true;
      continue;
    }
    if (lead) {
      st->iterations++;
      st->frontier_sum += n;
      st->edges_static += append_edges(x0, a.shift);
      st->edges_dynamic += append_edges(x1, a.shift);
    }
    if (hands_over(a, list_tiles(x0, a.shift), list_tiles(x1, a.shift))) {
      // the launch that relaxes them does not note what it lowers: the next
      // scan is one at the present threshold
      if (lead) {
        st->hx[0] = x0;
        st->hx[1] = x1;
        st->par = par ^ 1u;
        st->thr = thr;
        st->far_min = far_min;
      }
      hand = true;
      break;
    }
    if (threadIdx.x == 0) {
      rs.op.value = a.value;
      rs.op.next = a.bm[par ^ 1];
      rs.op.err = &st->err;
      rs.op.V = a.V;
      rs.op.thr = thr;
      rs.op.near = 0;
      rs.op.far_cand = 0xffffffffu;
    }
    if (lead && a.timer) st->ns_relax -= globaltimer_ns();
    relax_lists(rs, sh.lbs, slot);  // has a barrier before the first tile and after each
    if (a.split && threadIdx.x == 0) {
      if (rs.op.near) slot->near = 1u;
      if (rs.op.far_cand != 0xffffffffu) atomicMin(&slot->far_cand, rs.op.far_cand);
    }
    if (!rounds_sync(st, rs.target, a.spin_limit)) return;
    if (lead && a.timer) st->ns_relax += globaltimer_ns();
    par ^= 1u;
    merge = false;
    if (a.split && !slot->near) {
      const uint32_t f = min(far_min, slot->far_cand);
      if (f == 0xffffffffu) break;  // nothing lowered, nothing waiting
      t = (uint64_t)f + a.delta;
      thr = t > 0xffffffffull ? 0xffffffffu : (uint32_t)t;
      merge = true;
    }
  }
  if (!hand) rounds_result(a);
  if (lead) {
    st->hand = hand ? kHandRelax : 0u;
    st->done = !hand;
    st->ns_total += globaltimer_ns();
    rounds_post(a);
  }
}

// -------------------------------------------------------------------- BFS

constexpr uint64_t kBfsAlpha = 14, kBfsBeta = 24;
// Frontiers that one CTA expands alone (k_bfs_small): up to 4096 vertices and
// 16384 edges, about what it gets through in the time of the two grid
// barriers, the scan and the relax that a level over the whole grid costs.
constexpr uint32_t kSmallThreads = 1024, kSmallCap = 4 * kSmallThreads, kSmallEdges = 16384;
// The grid hands over to it after this many small top-down levels in a row:
// the last levels of a low-diameter graph are not worth a launch.
constexpr uint32_t kSmallStreak = 4;

struct SmallShared {
  uint64_t o[2][kSmallCap];
  uint32_t v[2][kSmallCap];
  uint32_t d[2][kSmallCap];  // degree (capped), then the exclusive prefix
  uint32_t cnt[2];
  uint32_t wsum[kSmallThreads / 32];
  uint32_t nz, es;
};

// Initial depths, bitmaps and state (BFS/oneGraph_BFS/GraphMeta.h:376-381).
__global__ void __launch_bounds__(kThreads) k_bfs_init(const __grid_constant__ RoundsArgs a) {
  const uint64_t gid = blockIdx.x * (uint64_t)kThreads + threadIdx.x, gsz = (uint64_t)gridDim.x * kThreads;
  for (uint64_t v = gid; v < a.V; v += gsz) a.value[v] = v == a.src ? 1u : a.V + 1;
  for (uint64_t w = gid; w < a.nwords; w += gsz) {
    const uint32_t x = w == a.src >> 5 ? 1u << (a.src & 31) : 0u;
    a.bm[0][w] = x;
    a.bm[1][w] = 0u;
    a.bm[2][w] = x;
  }
  if (gid == 0) {
    RoundsState *st = a.st;
    st->bar = 0;
    st->err = st->posted = st->hand = 0;
    st->iterations = st->frontier_sum = st->edges_static = st->edges_dynamic = 0;
    st->ns_total = st->ns_relax = 0;
    st->unexplored = a.E;
    st->fn = 0;
    st->level = 1;
    st->par = st->bottom = st->counted = st->done = 0;
    st->small = 1;  // the frontier to start from: entry 0 of the static list
    st->n0 = st->n = 1;
    a.list[0][0] = a.src;
  }
}

// Levels of small frontiers, one CTA: starts from the list that k_bfs_init or
// k_bfs_rounds left.  Every edge of a level takes one returning atomicOr on the
// visited bitmap, with the target's offsets loaded beside it, so a level is a
// chain of three memory round trips and a few block barriers.  Ends when the BFS
// has ended, or when the frontier is too large or goes bottom-up (its bits
// are then in bm[par ^ 1], and par flips).  A road-like BFS of 0.35 M vertices
// and 896 levels: 24-26 ms as replayed level graphs, 4.3 ms here.
__global__ void __launch_bounds__(kSmallThreads) k_bfs_small(const __grid_constant__ RoundsArgs a,
                                                             const __grid_constant__ SrcP<false> s0,
                                                             const __grid_constant__ SrcP<false> s1) {
  extern __shared__ __align__(16) unsigned char small_smem[];
  SmallShared &sm = *reinterpret_cast<SmallShared *>(small_smem);
  RoundsState *st = a.st;
  if (st->done || !st->small) return;
  const unsigned long long t0 = globaltimer_ns();
  uint32_t level = st->level, par = st->par, counted = st->counted;
  unsigned long long unexplored = st->unexplored;
  unsigned long long its = 0, fsum = 0, es = 0, ed = 0, fn = 0;
  uint32_t *over = a.bm[par ^ 1];  // all zero here; takes what the next queue cannot
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  {
    const uint32_t n0 = st->n0, n = st->n;
    for (uint32_t i = tid; i < n; i += kSmallThreads) {
      const uint32_t v = i < n0 ? a.list[0][i] : a.list[1][i - n0];
      const uint64_t o = a.off[v];
      sm.v[0][i] = v;
      sm.o[0][i] = o;
      sm.d[0][i] = (uint32_t)min(a.off[v + 1] - o, (uint64_t)(kSmallEdges + 1));
    }
    if (tid == 0) {
      sm.cnt[0] = n;
      sm.nz = sm.es = 0;
      st->bar = 0;  // the last k_bfs_rounds launch, if any, has ended: the next one's barriers start afresh
    }
  }
  __syncthreads();
  int c = 0;
  bool done = false, bottom = false;
  for (;;) {
    const uint32_t m = sm.cnt[c];
    if (m > kSmallCap) break;  // the overflow is in `over` already
    // exclusive prefix of the degrees; vertices with edges; static edges
    const uint32_t i0 = tid * 4;
    uint32_t dd[4], sum = 0, nz = 0, se = 0;
#pragma unroll
    for (uint32_t i = 0; i < 4; i++) {
      dd[i] = i0 + i < m ? sm.d[c][i0 + i] : 0u;
      sum += dd[i];
      nz += dd[i] ? 1u : 0u;
      if (i0 + i < m && sm.v[c][i0 + i] < a.Vs) se += dd[i];
    }
    uint32_t ic = sum;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, ic, s);
      if (lane >= s) ic += x;
    }
    nz = __reduce_add_sync(0xffffffffu, nz);
    se = __reduce_add_sync(0xffffffffu, se);
    if (lane == 31) sm.wsum[warp] = ic;
    if (lane == 0 && nz) {
      atomicAdd(&sm.nz, nz);
      if (se) atomicAdd(&sm.es, se);
    }
    if (tid == 0) sm.cnt[c ^ 1] = 0;
    __syncthreads();
    const uint32_t ws = sm.wsum[lane];
    const uint32_t total = __reduce_add_sync(0xffffffffu, ws);
    uint32_t ex = __reduce_add_sync(0xffffffffu, lane < warp ? ws : 0u) + ic - sum;
#pragma unroll
    for (uint32_t i = 0; i < 4; i++)
      if (i0 + i < m) {
        sm.d[c][i0 + i] = ex;
        ex += dd[i];
      }
    const uint32_t n = sm.nz, estat = sm.es;
    if (n == 0) {
      done = true;
      break;
    }
    if (total > kSmallEdges) break;
    if (!counted) unexplored -= min(unexplored, (unsigned long long)total);
    counted = 0;
    if (a.dopt && total > unexplored / kBfsAlpha) {
      bottom = true;
      fn = n;
      counted = 1;
      break;
    }
    its++;
    fsum += n;
    es += estat;
    ed += total - estat;
    __syncthreads();
    if (tid == 0) sm.nz = sm.es = 0;
    // no branches around the loads, so that a thread's searches, records and
    // targets overlap
    constexpr int U = 2;
    const uint32_t step0 = m > 1 ? 1u << (31 - __clz(m - 1)) : 0u;  // largest power of two below m
    for (uint32_t base = 0; base < total; base += U * kSmallThreads) {
      uint32_t lo[U], u[U];
      bool on[U];
#pragma unroll
      for (int j = 0; j < U; j++) lo[j] = 0;
      for (uint32_t step = step0; step; step >>= 1)  // last entry whose prefix is at most x
#pragma unroll
        for (int j = 0; j < U; j++) {
          const uint32_t x = base + j * kSmallThreads + tid, t = min(lo[j] + step, m - 1);
          lo[j] = sm.d[c][t] <= x ? t : lo[j];
        }
#pragma unroll
      for (int j = 0; j < U; j++) {
        const uint32_t x = base + j * kSmallThreads + tid;
        uint64_t e = sm.o[c][lo[j]] + (x - sm.d[c][lo[j]]);
        on[j] = x < total;
        if (on[j] && e >= a.E) atomicOr(&st->err, kErrEdgeIndex);
        on[j] = on[j] && e < a.E;
        e = on[j] ? e : 0ull;
        const uint64_t bit = e * s0.bpe;
        u[j] = s0.decode((e < a.static_edges ? s0.words : s1.words) + (bit >> 5), (uint32_t)bit & 31u);
      }
#pragma unroll
      for (int j = 0; j < U; j++) {
        if (on[j] && u[j] >= a.V) atomicOr(&st->err, kErrVertex);
        on[j] = on[j] && u[j] < a.V;
        u[j] = on[j] ? u[j] : 0u;
      }
      uint32_t old[U];
      uint64_t o0[U], o1[U];
#pragma unroll
      for (int j = 0; j < U; j++) {
        o0[j] = a.off[u[j]];
        o1[j] = a.off[u[j] + 1];
        old[j] = 0xffffffffu;
        if (on[j]) old[j] = atomicOr(a.bm[2] + (u[j] >> 5), 1u << (u[j] & 31));
      }
#pragma unroll
      for (int j = 0; j < U; j++) {
        const bool won = !((old[j] >> (u[j] & 31)) & 1u);
        const uint32_t ball = __ballot_sync(0xffffffffu, won);
        if (!ball) continue;
        uint32_t pos = 0;
        if (lane == 0) pos = atomicAdd(&sm.cnt[c ^ 1], __popc(ball));
        pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(ball & ((1u << lane) - 1u));
        if (won) {
          a.value[u[j]] = level + 1;
          if (pos < kSmallCap) {
            sm.v[c ^ 1][pos] = u[j];
            sm.o[c ^ 1][pos] = o0[j];
            sm.d[c ^ 1][pos] = (uint32_t)min(o1[j] - o0[j], (uint64_t)(kSmallEdges + 1));
          } else {
            atomicOr(over + (u[j] >> 5), 1u << (u[j] & 31));
          }
        }
      }
    }
    __syncthreads();
    level++;
    c ^= 1;
  }
  if (!done) {
    const uint32_t m = min(sm.cnt[c], kSmallCap);
    for (uint32_t i = tid; i < m; i += kSmallThreads) atomicOr(over + (sm.v[c][i] >> 5), 1u << (sm.v[c][i] & 31));
  }
  if (tid == 0) {
    st->iterations += its;
    st->frontier_sum += fsum;
    st->edges_static += es;
    st->edges_dynamic += ed;
    st->level = level;
    st->par = par ^ 1u;
    st->counted = counted;
    st->unexplored = unexplored;
    st->bottom = bottom;
    st->fn = fn;
    st->done = done;
    st->small = 0;
    const unsigned long long dt = globaltimer_ns() - t0;
    st->ns_total += dt;
    if (a.timer) st->ns_relax += dt;
  }
}

// One bottom-up level: every word of `next` is written.
__device__ __noinline__ void bfs_bottom_up_level(const RoundsArgs &a, const SrcP<false> stat, const SrcP<false> host,
                                                 const uint32_t *cur, uint32_t *next, uint32_t newdepth,
                                                 RoundSlot *slot) {
  bottom_up_words(a.off, a.V, a.Vs, stat, host, cur, a.bm[2], next, a.value, newdepth, slot->bu, &a.st->err);
}

__global__ void __launch_bounds__(kThreads, 3) k_bfs_rounds(const __grid_constant__ RoundsArgs a,
                                                            const __grid_constant__ SrcP<false> s0,
                                                            const __grid_constant__ SrcP<false> s1) {
  __shared__ union {
    LbsSh<BfsOp> lbs;
    ScanShared scan;
  } sh;
  __shared__ RelaxShared<SrcP<false>, BfsOp> rs;
  RoundsState *st = a.st;
  const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
  if (st->done) {  // set before this launch: every CTA reads the same
    rounds_result(a);
    if (lead) rounds_post(a);
    return;
  }
  if (lead) st->ns_total -= globaltimer_ns();
  relax_setup(a, rs, s0, s1);
  bool bottom = st->bottom, counted = st->counted, done = false;
  uint32_t level = st->level, par = st->par, streak = 0, hand = 0;
  uint64_t unexplored = st->unexplored, fn = st->fn;
  // After a bottom-up level: accounting and the direction of the next one; true
  // when it reached nothing.
  auto counted_bottom = [&](const unsigned long long *bu) {
    const uint64_t nn = bu[0];
    if (lead) {
      st->iterations++;
      st->frontier_sum += fn;
      st->edges_dynamic += bu[2];
      st->edges_static += bu[3];
    }
    unexplored -= min(unexplored, (uint64_t)bu[1]);
    if (nn == 0) return true;
    bottom = !(nn < a.V / kBfsBeta && nn < fn);  // small and shrinking: top-down again
    fn = nn;
    counted = true;
    level++;
    par ^= 1u;
    return false;
  };
  if (st->hand == kHandBottomUp) done = counted_bottom(st->hbu);
  if (lead)
    for (int i = 0; i < 4; i++) slot_clear(st->slot + i);
  if (!rounds_sync(st, rs.target, a.spin_limit)) return;  // every CTA has read the state that is rewritten at the end
  for (uint32_t seq = 0; !done; seq++) {
    uint32_t *cur = a.bm[par], *next = a.bm[par ^ 1];
    RoundSlot *slot = st->slot + (seq & 3u);
    if (!bottom) {
      scan_frontier<false, false>(a, sh.scan, cur, next, nullptr, false, 0u, slot);
      if (!rounds_sync(st, rs.target, a.spin_limit)) return;
      if (lead) slot_clear(st->slot + ((seq + 2) & 3u));
      const unsigned long long x0 = slot->app[0], x1 = slot->app[1];
      const uint64_t n0 = x0 >> a.shift, n = n0 + (x1 >> a.shift);
      const uint64_t m0 = append_edges(x0, a.shift), mf = m0 + append_edges(x1, a.shift);
      if (n == 0) {
        done = true;
        break;
      }
      streak = n <= kSmallCap && mf <= kSmallEdges ? streak + 1 : 0;
      if (streak > kSmallStreak) {  // accounting and direction choice are k_bfs_small's
        if (lead) {
          st->n0 = (uint32_t)n0;
          st->n = (uint32_t)n;
        }
        break;
      }
      if (!counted) unexplored -= min(unexplored, mf);
      counted = false;
      if (a.dopt && mf > unexplored / kBfsAlpha) {
        bottom = counted = true;
        fn = n;
      } else {
        if (lead) {
          st->iterations++;
          st->frontier_sum += n;
          st->edges_static += m0;
          st->edges_dynamic += mf - m0;
        }
        if (hands_over(a, list_tiles(x0, a.shift), list_tiles(x1, a.shift))) {
          if (lead) {
            st->hx[0] = x0;
            st->hx[1] = x1;
          }
          hand = kHandRelax;
          level++;
          par ^= 1u;
          break;
        }
        if (threadIdx.x == 0) rs.op = BfsOp{a.bm[2], next, a.value, &st->err, a.V, level + 1};
        if (lead && a.timer) st->ns_relax -= globaltimer_ns();
        relax_lists(rs, sh.lbs, slot);
        if (!rounds_sync(st, rs.target, a.spin_limit)) return;
        if (lead && a.timer) st->ns_relax += globaltimer_ns();
        level++;
        par ^= 1u;
        continue;
      }
    }
    streak = 0;
    if (a.hand_bottom) {
      hand = kHandBottomUp;
      break;
    }
    bfs_bottom_up_level(a, s0, s1, cur, next, level + 1, slot);
    if (!rounds_sync(st, rs.target, a.spin_limit)) return;
    if (lead) slot_clear(st->slot + ((seq + 2) & 3u));
    done = counted_bottom(slot->bu);
  }
  if (done) rounds_result(a);
  if (lead) {
    st->done = done;
    st->small = !done && !hand;
    st->hand = hand;
    st->level = level;
    st->par = par;
    st->counted = counted;
    st->bottom = hand == kHandBottomUp;
    st->fn = fn;
    st->hbu[0] = st->hbu[1] = st->hbu[2] = st->hbu[3] = 0;
    st->unexplored = unexplored;
    st->ns_total += globaltimer_ns();
    rounds_post(a);
  }
}

// ------------------------------------------------------------- union-find CC

// parent[v] = root of v for every vertex, by pointer jumping between grid
// barriers: a pass takes each vertex up to kJumpHops parents up, from where the
// pass before has taken them, until one leaves no vertex below its root.  A
// thread stores its own vertices only, and the barrier drops the parents that
// L1 holds, so chains shrink by the number of hops with every pass.  Bound by
// latency, a round trip per hop.  A kernel of whole walks per vertex kept each
// wave of threads waiting for its longest chain where first neighbours form
// chains: union-find CC of a 5000 x 4000 grid numbered by rows 2.72 ms with it,
// 0.87 now (4 hops 0.94, two walks a thread 0.88); R-MAT of 2^23 vertices, whose
// chains are shorter than a pass, 0.45 either way.
constexpr uint32_t kJumps = 3;  // compressions of a run
constexpr uint32_t kJumpHops = 8;
constexpr int kJumpWalks = 4;  // vertices a thread has in flight
__global__ void __launch_bounds__(kThreads) k_uf_jump(uint32_t *par, uint32_t V, RoundsState *st, uint32_t spin_limit,
                                                    uint32_t *err) {
  unsigned long long target = 0;
  const uint64_t first = blockIdx.x * (uint64_t)kThreads + threadIdx.x, stride = (uint64_t)gridDim.x * kThreads;
  for (uint32_t pass = 0;; pass++) {
    uint32_t open = 0;
    for (uint64_t v = first; v < V; v += kJumpWalks * stride) {
      uint32_t x[kJumpWalks], p[kJumpWalks], todo = 0;
#pragma unroll
      for (int j = 0; j < kJumpWalks; j++) {
        const bool on = v + j * stride < V;
        x[j] = p[j] = on ? (uint32_t)(v + j * stride) : 0u;
        todo |= (on ? 1u : 0u) << j;
      }
      const uint32_t mine = todo;
      uint32_t own[kJumpWalks];
#pragma unroll
      for (uint32_t h = 0; h <= kJumpHops; h++) {
        if (!todo) break;
#pragma unroll
        for (int j = 0; j < kJumpWalks; j++)
          if ((todo >> j) & 1u) p[j] = __ldca(par + x[j]);
#pragma unroll
        for (int j = 0; j < kJumpWalks; j++) {
          if (h == 0) own[j] = p[j];
          if (p[j] > x[j]) atomicOr(err, kErrVertex);
          if (p[j] >= x[j]) todo &= ~(1u << j);  // x is a root
          else x[j] = p[j];
        }
      }
      open |= todo;
#pragma unroll
      for (int j = 0; j < kJumpWalks; j++)
        if (((mine >> j) & 1u) && x[j] != own[j]) __stcg(par + v + j * stride, x[j]);
    }
    uint32_t *flag = &st->slot[pass & 3u].near;
    if (__syncthreads_or(open != 0u) && threadIdx.x == 0) *flag = 1u;
    if (blockIdx.x == 0 && threadIdx.x == 0) st->slot[(pass + 2) & 3u].near = 0u;  // last read before the barrier before
    if (!rounds_sync(st, target, spin_limit) || pass > 64) {
      if (threadIdx.x == 0) atomicOr(err, kErrBarrier);
      return;
    }
    if (!__ldcg(flag)) return;
  }
}

}  // namespace og
