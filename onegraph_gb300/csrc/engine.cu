// engine.cu — the out-of-memory engine behind og_engine_* / og_bfs / og_sssp /
// og_cc / og_pr (onegraph.h).
//
// One engine = one graph on one GB300, planned against a device budget:
//  * static region: vertices [0, Vs) whose whole adjacency lies in the edge
//    prefix [0, off[Vs]); that prefix is copied to HBM once
//    (GraphMeta.h:234-291 initGraphDevice, 300-360 getMaxPartitionSize);
//  * dynamic region: vertices [Vs, V); their edges stay in page-locked host
//    memory and every round the active ones are gathered by a kernel over the
//    host link into one of two device staging buffers (side stream), while the
//    previous buffer is relaxed and the static region is relaxed on the main
//    stream (CalculateOpt.h:75-188, GraphMeta.h:471-557).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>
#include <chrono>
#include <cstring>
#include <mutex>
#include <new>
#include <vector>

#include "batch_persist.cuh"
#include "kernels.cuh"
#include "og_internal.hpp"
#include "rounds.cuh"
#include "sssp_batch.cuh"

using namespace og;

#define CK(x)                                                                          \
  do {                                                                                 \
    cudaError_t e_ = (x);                                                              \
    if (e_ != cudaSuccess)                                                             \
      return og::fail(OG_E_CUDA, "%s: %s (%s:%d)", #x, cudaGetErrorString(e_), __FILE__, \
                      __LINE__);                                                       \
  } while (0)

#define RC(x)                    \
  do {                           \
    int r_ = (x);                \
    if (r_ != OG_OK) return r_;  \
  } while (0)

// Fragment slots of an OG_CFG_REPLACE engine (SrcF, kernels.cuh): the slot
// memory, the device slot table and its host mirror, and the policy state.
struct FragState {
  uint32_t fs = 0;          // log2 words per fragment
  uint64_t nfrag = 0;       // fragments of the packed record stream
  uint32_t nslots = 0;
  uint64_t bytes = 0;       // device bytes for slots, tables and update lists
  uint32_t *slots_d = nullptr;
  int32_t *slot_of_d = nullptr;
  uint32_t *visits_d = nullptr;  // records listed per fragment since the last step
  unsigned long long *miss_d = nullptr;  // of those, records of slotted fragments read from the host
  unsigned long long *miss_h = nullptr;  // page-locked
  uint2 *pairs_d = nullptr;      // one update: (fragment, slot)
  uint32_t *evict_d = nullptr;   // one update: the fragment each slot held before
  uint32_t max_pairs = 0;
  uint32_t *visits_h = nullptr;  // page-locked
  uint2 *pairs_h = nullptr;      // page-locked
  uint32_t *evict_h = nullptr;   // page-locked
  cudaEvent_t ev_ready = nullptr;  // slot updates done (the dynamic stream waits on it)
  std::vector<int32_t> slot_of;  // host mirror of slot_of_d
  std::vector<uint32_t> owner;   // fragment held by each slot (UINT32_MAX: none)
  std::vector<float> score;      // records listed per fragment, halved every step
  std::vector<void *> dallocs, hallocs;
  uint64_t dalloc_bytes = 0;
  bool broken = false;     // a layout failed: queries through the slots are refused
  uint64_t since = 0;      // dynamic records listed since the last policy step
  uint64_t step_min = 0;   // records between policy steps (as many as the slots hold)
  og_fragment_stats st{};
};

// Counts-sized (16-byte) parts of an engine's control block (og_engine::counts_d).
constexpr uint32_t kControlCounts = 5;

struct og_engine {
  og_graph *g = nullptr;
  og_config cfg{};
  og_plan plan{};
  int dev = 0;
  int sms = 0;
  bool pr_enabled = false;
  bool registered = false;
  uint32_t V = 0, Vs = 0;
  uint64_t nwords = 0;

  cudaStream_t s_main = nullptr, s_dyn = nullptr, s_gat = nullptr;
  cudaEvent_t ev_round = nullptr, ev_cd = nullptr, ev_dyn_done = nullptr;
  cudaEvent_t ev_gat[2] = {nullptr, nullptr}, ev_rel[2] = {nullptr, nullptr};
  cudaEvent_t t_s0 = nullptr, t_s1 = nullptr, t_d0 = nullptr;
  std::vector<cudaEvent_t> t_gat;  // start/end pairs around each gather launch

  uint64_t *off_d = nullptr;
  // edges as bit-packed records (host copy and static region) and as
  // unpacked u32 columns + weights of wbytes (1, 2, 4) in the staging buffers
  uint32_t *spk_d = nullptr;                 // static region records (HBM)
  uint32_t bpe = 0, bc = 0, wmin = 0;        // record layout
  uint32_t *stage_col[2] = {nullptr, nullptr};  // staging buffers (columns)
  void *stage_w[2] = {nullptr, nullptr};        // staging buffers (weights)
  const uint32_t *hpk_d = nullptr;           // page-locked host records, device view
  uint32_t wbytes = 0;
  uint32_t *value_d = nullptr;
  uint32_t *bm[3] = {nullptr, nullptr, nullptr};
  uint32_t *list_d[2] = {nullptr, nullptr};
  uint64_t *pref_d[2] = {nullptr, nullptr};
  uint32_t *tile_d[2] = {nullptr, nullptr};
  uint64_t list_cap[2] = {0, 0}, tile_cap[2] = {0, 0};
  Lookback lb[2]{};
  uint32_t lb_tiles = 0;
  // What the host reads after a compaction, in one copy: Counts[2], u64 far
  // key[2], 4 error words (err_d, active_d), 4 mask words (sb_masks).
  Counts *counts_d = nullptr, *counts_h = nullptr;
  uint32_t epoch = 0;  // look-back epoch of the last compaction launch
  uint32_t *err_d = nullptr, *err_h = nullptr;
  uint32_t *active_d = nullptr;

  // PageRank state
  float *contrib_d = nullptr, *sum_d = nullptr, *cont_d = nullptr, *carry_d = nullptr;
  uint32_t *outdeg_d = nullptr, *carry_idx_d = nullptr;
  double *part_d = nullptr;
  PrLoop *prl_d = nullptr, *prl_h = nullptr;  // L1 iterations: state and its page-locked mirror
  // iterations the last run of this damping and tolerance took (launched before
  // the first check)
  uint32_t pr_hint = 8;
  float pr_hint_damping = 0;
  double pr_hint_tol = -1;
  uint32_t part_n = 0;
  uint64_t pr_tiles = 0;

  // batched BFS state
  bool batch_enabled = false;
  unsigned long long *bmask[3] = {nullptr, nullptr, nullptr};  // visited, cur, next
  unsigned long long *hist_d = nullptr, *hist_h = nullptr;
  uint32_t *srcs_d = nullptr, *srcs_h = nullptr;
  // persistent kernel state
  uint32_t *ptile_d = nullptr;
  uint64_t ptile_cap = 0;
  uint32_t *cta_n = nullptr;
  unsigned long long *cta_e = nullptr;
  unsigned long long *smf_d = nullptr;  // batched BFS: per-source frontier degree sums
  uint32_t *bar_d = nullptr;   // [0..1] barrier, [2] error, [3] levels, [4..11] 4 x u64 stats
  uint32_t *pmisc_h = nullptr;  // host copy of bar_d
  int tuned = -1;               // index into kPersistConfigs chosen by the autotuner
  cudaGraphExec_t graph = nullptr;
  // device-driven rounds (rounds.cuh): state and its page-locked host mirror
  RoundsState *rounds_d = nullptr, *rounds_h = nullptr;
  uint32_t *ring_d = nullptr;  // staged rounds: ticket, then (kRingPad words on) the slot states
  uint32_t level_loop = 0;        // OG_LOOP_AUTO / OG_LOOP_HOST
  uint32_t relax_timer = 0;       // OG_PARAM_RELAX_TIMER
  void *out = nullptr;            // the running query's result array, null once it is delivered
  uint32_t graph_n = 0;
  int graph_cfg = -1;
  int graph_dopt = -1;
  bool graph_broken = false;

  // batched BFS depth matrix (n x V u32, outside the budget), kept between
  // calls that ask for depths; its byte form for og_bfs_batch_u8
  uint32_t *depth_d = nullptr;
  uint64_t depth_cap = 0;  // entries
  uint8_t *depth8_d = nullptr;
  uint64_t depth8_cap = 0;

  // multi-source SSSP (og_sssp_batch, sssp_batch.cuh): sb_k sources per pass
  // in rows of sb_ks slots; its rows, pending masks and near masks share
  // `arena` with the batched BFS masks
  uint32_t sb_k = 0, sb_ks = 0;
  unsigned char *arena = nullptr;
  uint32_t *sb_dist = nullptr, *sb_pend = nullptr, *sb_lmask = nullptr;
  uint32_t *sb_masks = nullptr;  // device: [0] pending slots seen, [1] waiting slots, [2..3] spare
  uint32_t *sb_io_h = nullptr;   // page-locked: sources [0, 32), slots [32, 64), masks [64, 68)
  uint32_t *sb_io_d = nullptr;
  unsigned long long *sb_ck_d = nullptr, *sb_ck_h = nullptr;  // per-slot checks (2 x 32)
  uint32_t sb_thr = 0, sb_far_min = 0;
  uint32_t sb_delta = 0;  // OG_PARAM_SSSP_BATCH_DELTA: near/far width of the batch (0: every round)
  bool sb_advance = false;
  uint32_t sb_dirty = 0;  // slots whose distances are not all unreached
  bool sb_session = false;  // a session is open: no other query ran since og_sssp_batch_begin

  // batched BFS level by level (og_bfs_batch_begin ... _fetch): up to 64
  // slots over the batch masks; a slot's depths are offset by the level it
  // joined at, and a finished slot's visited bits are cleared when it is
  // joined again
  uint32_t *bb_io_d = nullptr, *bb_io_h = nullptr;  // sources [0,64), slots [64,128), depth offsets [128,192)
  bool bb_session = false;  // no other query ran since og_bfs_batch_begin
  bool bb_record = false;   // depths recorded in depth_d (64 x V)
  uint32_t bb_level = 1;    // depth of the frontier the next step expands, for a source at depth 1 at begin
  uint32_t bb_par = 0;      // frontier parity: cur = bmask[1 + par], cur_any = bm[par]
  uint64_t bb_used = 0;     // slots joined and not finished
  uint64_t bb_dirty = 0;    // finished slots whose visited bits are still set
  uint32_t bb_off[64] = {};
  uint64_t bb_reached[64] = {}, bb_dsum[64] = {};

  FragState *frag = nullptr;  // OG_CFG_REPLACE: fragment slots of the dynamic region

  og_engine *parent = nullptr;  // set on clones: resident state belongs to the parent
  int clones = 0;               // live clones of this engine
  uint64_t resident_bytes = 0;  // device bytes of the shared resident state
  unsigned long long *sum64_d = nullptr;  // result checksum scratch

  uint32_t sssp_delta = 0;  // near/far split width (0: plain frontier relaxation)
  uint32_t cc_method = 0;   // OG_CC_AUTO / OG_CC_LABEL_PROPAGATION / OG_CC_UNION_FIND
  uint32_t bfs_direction = 0;  // OG_BFS_AUTO / OG_BFS_TOP_DOWN

  int last_algo = -1;
  uint64_t launches = 0;  // kernels launched since the query began
  std::vector<void *> dallocs;
  uint64_t dbytes = 0;
};

namespace {

constexpr int kGatherMult = 2;  // gather tiles of 4096 positions
constexpr uint32_t kMaxPersistCtas = 2048;

template <class T>
int dalloc(og_engine *e, T **p, uint64_t count) {
  const uint64_t bytes = std::max<uint64_t>(count * sizeof(T), 256);
  void *q = nullptr;
  cudaError_t err = cudaMalloc(&q, bytes);
  if (err != cudaSuccess)
    return fail(OG_E_CUDA, "cudaMalloc(%llu B) failed: %s (engine holds %llu B)",
                (unsigned long long)bytes, cudaGetErrorString(err), (unsigned long long)e->dbytes);
  e->dallocs.push_back(q);
  e->dbytes += bytes;
  *p = (T *)q;
  return OG_OK;
}

int grid_for(uint64_t n, int sms) {
  const uint64_t g = (n + kThreads - 1) / kThreads;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>(g, (uint64_t)sms * 8));
}

// ------------------------------------------------------- fragment slots
//
// Static-region replacement (OG_CFG_REPLACE).  The reference declares its
// pieces and never defines them: recordFragmentVisit (per-fragment visit
// records), setFragmentData / setStaticFragmentData (which static fragments
// may be swapped) and bfs_kernelStaticSwap (BFS/oneGraph_BFS/gpu_kernels.h:
// 46-66,153-176, FragmentData in globals.h:22-33).  Here the swappable part
// is a set of slots carved from the static region's bytes; the relax counts
// the records it lists per fragment (SrcF::note) and frag_step, after every
// round, moves the most-read fragments without a slot into the slots whose
// fragments were read least.

void frag_release(og_engine *e) {
  FragState &F = *e->frag;
  for (void *p : F.dallocs) cudaFree(p);
  for (void *p : F.hallocs) cudaFreeHost(p);
  F.dallocs.clear();
  F.hallocs.clear();
  e->dbytes -= F.dalloc_bytes;
  if (!e->parent) e->resident_bytes -= std::min(e->resident_bytes, F.dalloc_bytes);
  F.dalloc_bytes = 0;
  F.slots_d = nullptr;
  F.slot_of_d = nullptr;
  F.visits_d = nullptr;
  F.miss_d = nullptr;
  F.miss_h = nullptr;
  F.pairs_d = nullptr;
  F.evict_d = nullptr;
  F.visits_h = nullptr;
  F.pairs_h = nullptr;
  F.evict_h = nullptr;
}

template <class T>
int frag_dalloc(og_engine *e, T **p, uint64_t count) {
  const uint64_t bytes = std::max<uint64_t>(count * sizeof(T), 256);
  void *q = nullptr;
  CK(cudaMalloc(&q, bytes));
  e->frag->dallocs.push_back(q);
  e->frag->dalloc_bytes += bytes;
  e->dbytes += bytes;
  *p = (T *)q;
  return OG_OK;
}

template <class T>
int frag_halloc(og_engine *e, T **p, uint64_t count) {
  void *q = nullptr;
  CK(cudaHostAlloc(&q, std::max<uint64_t>(count * sizeof(T), 64), cudaHostAllocDefault));
  e->frag->hallocs.push_back(q);
  *p = (T *)q;
  return OG_OK;
}

// Default fragment size: the power of two nearest packed words / 4096,
// clamped to [2^8, 2^14] words.
uint32_t frag_default_shift(uint64_t packed_words) {
  const double x = std::log2(std::max<double>(1.0, (double)packed_words / 4096.0));
  return (uint32_t)std::min(14.0, std::max(8.0, std::floor(x + 0.5)));
}

// Lays out slots of 2^fs + kFragPad words, the slot table, the visit counts
// and the update lists inside F.bytes of device memory.
// Device bytes of the tables and update lists for fragments of 2^fs words,
// and the most pairs one step moves (a quarter of the slots, at most 4096).
uint64_t frag_fixed_bytes(const FragState &F, uint64_t nfrag, uint32_t fs, uint32_t *max_pairs) {
  const uint64_t slot_words = (1ull << fs) + kFragPad;
  *max_pairs = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(4096, F.bytes / (4 * slot_words) / 4));
  return nfrag * 8 + (uint64_t)*max_pairs * 12 + 5 * 256;
}

// 0 when slots of 2^fs words fit F.bytes (checked before anything is freed).
int frag_fits(const og_engine *e, uint32_t fs) {
  const FragState &F = *e->frag;
  const uint64_t nfrag = (e->g->packed_words + (1ull << fs) - 1) >> fs;
  uint32_t mp;
  const uint64_t slot_words = (1ull << fs) + kFragPad;
  if (F.bytes < frag_fixed_bytes(F, nfrag, fs, &mp) + 4 * slot_words)
    return fail(OG_E_BUDGET, "fragment slots: %llu B of static region cannot hold one %llu-word slot and the "
                "%llu-fragment tables", (unsigned long long)F.bytes, (unsigned long long)slot_words,
                (unsigned long long)nfrag);
  return OG_OK;
}

int frag_layout(og_engine *e, uint32_t fs) {
  FragState &F = *e->frag;
  RC(frag_fits(e, fs));
  frag_release(e);
  F.broken = true;  // until the layout below completes
  const og_graph *g = e->g;
  F.fs = fs;
  F.nfrag = (g->packed_words + (1ull << fs) - 1) >> fs;
  const uint64_t slot_words = (1ull << fs) + kFragPad;
  const uint64_t fixed = frag_fixed_bytes(F, F.nfrag, fs, &F.max_pairs);
  const uint64_t ns = std::min<uint64_t>((F.bytes - fixed) / (4 * slot_words), std::min<uint64_t>(F.nfrag, 0x7fffffffull));
  F.nslots = (uint32_t)ns;
  RC(frag_dalloc(e, &F.slots_d, ns * slot_words));
  RC(frag_dalloc(e, &F.slot_of_d, F.nfrag));
  RC(frag_dalloc(e, &F.visits_d, F.nfrag));
  RC(frag_dalloc(e, &F.miss_d, 1));
  RC(frag_dalloc(e, &F.pairs_d, F.max_pairs));
  RC(frag_dalloc(e, &F.evict_d, F.max_pairs));
  if (!e->parent) e->resident_bytes += F.dalloc_bytes;
  RC(frag_halloc(e, &F.visits_h, F.nfrag));
  RC(frag_halloc(e, &F.miss_h, 1));
  RC(frag_halloc(e, &F.pairs_h, F.max_pairs));
  RC(frag_halloc(e, &F.evict_h, F.max_pairs));
  F.slot_of.assign(F.nfrag, -1);
  F.owner.assign(F.nslots, 0xffffffffu);
  F.score.assign(F.nfrag, 0.0f);
  F.since = 0;
  F.step_min = (uint64_t)((double)F.nslots * (double)(1ull << fs) * 32.0 / e->bpe);
  F.st = og_fragment_stats{};
  F.st.fragments = F.nfrag;
  F.st.slots = F.nslots;
  F.st.fragment_words = 1u << fs;
  F.broken = false;
  return OG_OK;
}

// Copies n (fragment, slot) pairs from F.pairs_h / F.evict_h into the slots
// and the table on stream s.
int frag_apply(og_engine *e, uint32_t n, cudaStream_t s) {
  FragState &F = *e->frag;
  if (n == 0) return OG_OK;
  CK(cudaMemcpyAsync(F.pairs_d, F.pairs_h, 8ull * n, cudaMemcpyHostToDevice, s));
  CK(cudaMemcpyAsync(F.evict_d, F.evict_h, 4ull * n, cudaMemcpyHostToDevice, s));
  k_frag_fill<<<n, kThreads, 0, s>>>(e->hpk_d, e->g->packed_words, F.slots_d, F.pairs_d, n, F.fs);
  k_frag_table<<<(n + 255) / 256, 256, 0, s>>>(F.slot_of_d, F.pairs_d, F.evict_d, n);
  e->launches += 2;
  CK(cudaGetLastError());
  return OG_OK;
}

// Empties the slots, then fills them with the fragments that follow the
// static prefix (the records a larger static prefix would hold).
int frag_reset(og_engine *e) {
  FragState &F = *e->frag;
  cudaStream_t s = e->s_main;
  F.broken = true;  // until every fill below is queued
  CK(cudaMemsetAsync(F.slot_of_d, 0xff, 4 * F.nfrag, s));
  CK(cudaMemsetAsync(F.visits_d, 0, 4 * F.nfrag, s));
  CK(cudaMemsetAsync(F.miss_d, 0, 8, s));
  const uint64_t f0 = (e->plan.static_edges * e->bpe >> 5) >> F.fs;
  uint32_t filled = 0;
  while (filled < F.nslots && f0 + filled < F.nfrag) {
    uint32_t n = 0;
    for (; n < F.max_pairs && filled < F.nslots && f0 + filled < F.nfrag; n++, filled++) {
      const uint32_t f = (uint32_t)(f0 + filled);
      F.pairs_h[n] = make_uint2(f, filled);
      F.evict_h[n] = 0xffffffffu;
      F.slot_of[f] = (int32_t)filled;
      F.owner[filled] = f;
    }
    RC(frag_apply(e, n, s));
    CK(cudaStreamSynchronize(s));  // the page-locked lists are reused
  }
  if (!F.ev_ready) CK(cudaEventCreateWithFlags(&F.ev_ready, cudaEventDisableTiming));
  F.broken = false;
  return OG_OK;
}

// After a compaction (the previous round's relax has finished), once as many
// records as the slots hold have been listed since the last step, or when
// `force` (a compaction that lists nothing, e.g. the query's last): reads
// the visit counts, moves the records served from slots out of the
// host-link bytes, and replaces slots.  Ascetic's rule: fragments read in
// this round that have no slot take the slots of fragments that were read
// least; scores are records listed, halved every step; a fragment comes in
// only if its score is at least a quarter of its records and above twice the
// evicted one's; the copies of one step read at most a quarter of the
// round's host-link bytes.  The dynamic stream waits for the updates.
int frag_step(og_engine *e, og_stats &st, bool force) {
  FragState &F = *e->frag;
  if (!force && F.since < F.step_min) return OG_OK;  // counts keep adding up on the device
  F.since = 0;
  cudaStream_t s = e->s_main;
  CK(cudaMemcpyAsync(F.visits_h, F.visits_d, 4 * F.nfrag, cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(F.miss_h, F.miss_d, 8, cudaMemcpyDeviceToHost, s));
  CK(cudaMemsetAsync(F.visits_d, 0, 4 * F.nfrag, s));
  CK(cudaMemsetAsync(F.miss_d, 0, 8, s));
  CK(cudaStreamSynchronize(s));
  uint64_t in_slots = 0, in_host = 0;
  std::vector<uint32_t> cand;
  const float min_score = (float)((double)(1ull << F.fs) * 32.0 / e->bpe / 4.0);
  for (uint64_t f = 0; f < F.nfrag; f++) {
    const uint32_t v = F.visits_h[f];
    F.score[f] = 0.5f * F.score[f] + (float)v;
    if (!v) continue;
    if (F.slot_of[f] >= 0) {
      in_slots += v;
    } else {
      in_host += v;
      if (F.score[f] >= min_score) cand.push_back((uint32_t)f);
    }
  }
  // records of slotted fragments that a range over a fragment end read from the host
  const uint64_t miss = std::min<uint64_t>(*F.miss_h, in_slots);
  in_slots -= miss;
  in_host += miss;
  F.st.records_slots += in_slots;
  F.st.records_host += in_host;
  const uint64_t slot_link = (in_slots * e->bpe) / 8;
  st.link_bytes -= std::min(st.link_bytes, slot_link);
  const uint64_t frag_bytes = 4ull * ((1ull << F.fs) + kFragPad);
  const uint64_t cap = (in_host * e->bpe / 8) / 4 / frag_bytes;
  uint32_t n = (uint32_t)std::min<uint64_t>({cap, (uint64_t)F.max_pairs, (uint64_t)F.nslots, (uint64_t)cand.size()});
  if (n == 0) return OG_OK;
  auto hot = [&](uint32_t a, uint32_t b) { return F.score[a] > F.score[b] || (F.score[a] == F.score[b] && a < b); };
  std::partial_sort(cand.begin(), cand.begin() + n, cand.end(), hot);
  std::vector<uint32_t> vict(F.nslots);
  for (uint32_t i = 0; i < F.nslots; i++) vict[i] = i;
  auto vscore = [&](uint32_t sl) { return F.owner[sl] == 0xffffffffu ? -1.0f : F.score[F.owner[sl]]; };
  std::partial_sort(vict.begin(), vict.begin() + n, vict.end(), [&](uint32_t a, uint32_t b) {
    return vscore(a) < vscore(b) || (vscore(a) == vscore(b) && a < b);
  });
  uint32_t m = 0;
  for (uint32_t i = 0; i < n; i++) {
    const uint32_t f = cand[i], sl = vict[i];
    if (F.score[f] <= 2.0f * vscore(sl) + 1.0f) break;
    const uint32_t old = F.owner[sl];
    F.pairs_h[m] = make_uint2(f, sl);
    F.evict_h[m] = old;
    if (old != 0xffffffffu) F.slot_of[old] = -1;
    F.slot_of[f] = (int32_t)sl;
    F.owner[sl] = f;
    m++;
  }
  if (m == 0) return OG_OK;
  RC(frag_apply(e, m, s));
  CK(cudaEventRecord(F.ev_ready, s));
  CK(cudaStreamWaitEvent(e->s_dyn, F.ev_ready, 0));
  F.st.swaps += m;
  F.st.swap_bytes += m * frag_bytes;
  st.link_bytes += m * frag_bytes;
  return OG_OK;
}

void destroy(og_engine *e) {
  if (!e) return;
  cudaSetDevice(e->dev);
  if (e->s_main) cudaStreamSynchronize(e->s_main);
  if (e->s_dyn) cudaStreamSynchronize(e->s_dyn);
  if (e->s_gat) cudaStreamSynchronize(e->s_gat);
  if (e->frag) {
    frag_release(e);
    if (e->frag->ev_ready) cudaEventDestroy(e->frag->ev_ready);
    delete e->frag;
    e->frag = nullptr;
  }
  for (void *p : e->dallocs) cudaFree(p);
  if (e->depth_d) cudaFree(e->depth_d);
  if (e->depth8_d) cudaFree(e->depth8_d);
  if (e->counts_h) cudaFreeHost(e->counts_h);
  if (e->hist_h) cudaFreeHost(e->hist_h);
  if (e->srcs_h) cudaFreeHost(e->srcs_h);
  if (e->sb_io_h) cudaFreeHost(e->sb_io_h);
  if (e->bb_io_h) cudaFreeHost(e->bb_io_h);
  if (e->sb_ck_h) cudaFreeHost(e->sb_ck_h);
  if (e->pmisc_h) cudaFreeHost(e->pmisc_h);
  if (e->graph) cudaGraphExecDestroy(e->graph);
  if (e->rounds_h) cudaFreeHost(e->rounds_h);
  if (e->prl_h) cudaFreeHost(e->prl_h);
  cudaEvent_t evs[] = {e->ev_round, e->ev_cd, e->ev_dyn_done, e->ev_gat[0], e->ev_gat[1],
                       e->ev_rel[0], e->ev_rel[1], e->t_s0, e->t_s1, e->t_d0};
  for (auto ev : evs)
    if (ev) cudaEventDestroy(ev);
  for (auto ev : e->t_gat) cudaEventDestroy(ev);
  if (e->s_main) cudaStreamDestroy(e->s_main);
  if (e->s_dyn) cudaStreamDestroy(e->s_dyn);
  if (e->s_gat) cudaStreamDestroy(e->s_gat);
  if (e->registered && e->g) {
    if (--e->g->registered == 0) {
      cudaHostUnregister(e->g->packed);
    }
  }
  if (e->parent) e->parent->clones--;
  cudaGetLastError();  // a failure while tearing down is not the next call's error
  delete e;
}

// Per-query state: streams, events, frontier/list arrays, staging buffers and
// the PageRank / batched-BFS working arrays.  A parent engine and each of its
// clones own one set; the resident graph (offsets, static edges, out-degrees,
// page-locked host CSR) is shared.
int create_query_state(og_engine *e) {
  const og_plan &P = e->plan;
  const uint64_t V = e->V;
  // A fully resident graph's queries are short and HBM-bound; an
  // out-of-memory graph's kernels wait on the host link with many CTAs
  // resident.  When both share the GPU (several engines, the server), the
  // resident graph's streams get the highest priority so that the block
  // scheduler places its CTAs first as SMs free up, instead of behind a
  // link-bound grid of millions of CTAs.
  int prio_lo = 0, prio_hi = 0;
  CK(cudaDeviceGetStreamPriorityRange(&prio_lo, &prio_hi));
  const int prio = P.dynamic_edges == 0 ? prio_hi : prio_lo;
  CK(cudaStreamCreateWithPriority(&e->s_main, cudaStreamNonBlocking, prio));
  CK(cudaStreamCreateWithPriority(&e->s_dyn, cudaStreamNonBlocking, prio));
  CK(cudaStreamCreateWithPriority(&e->s_gat, cudaStreamNonBlocking, prio));
  cudaEvent_t *evs[] = {&e->ev_round, &e->ev_cd, &e->ev_dyn_done, &e->ev_gat[0],
                        &e->ev_gat[1], &e->ev_rel[0], &e->ev_rel[1], &e->t_s0, &e->t_s1, &e->t_d0};
  for (auto ev : evs) CK(cudaEventCreate(ev));
  RC(dalloc(e, &e->value_d, V + 1));
  for (int i = 0; i < 3; i++) RC(dalloc(e, &e->bm[i], e->nwords));
  e->list_cap[0] = std::max<uint64_t>(e->Vs, 1);
  e->list_cap[1] = std::max<uint64_t>(V - e->Vs, 1);
  e->tile_cap[0] = P.static_edges / kTile + 2;
  e->tile_cap[1] = P.dynamic_edges / kTile + 2;
  // one allocation per array, the dynamic region's part after the static one,
  // so the batched kernel can also use them as a single list over [0, V)
  RC(dalloc(e, &e->list_d[0], e->list_cap[0] + e->list_cap[1]));
  RC(dalloc(e, &e->pref_d[0], e->list_cap[0] + e->list_cap[1] + 2));
  RC(dalloc(e, &e->tile_d[0], e->tile_cap[0] + e->tile_cap[1]));
  e->list_d[1] = e->list_d[0] + e->list_cap[0];
  e->pref_d[1] = e->pref_d[0] + e->list_cap[0] + 1;
  e->tile_d[1] = e->tile_d[0] + e->tile_cap[0];
  // The planner counts 64 B of look-back scratch per 1024 bitmap words and
  // region pair, i.e. two 16-byte slots per region, and 64 KiB for the small
  // arrays, of which 2 x 256 slots (8 KiB) are used here.
  e->lb_tiles = 2 * (uint32_t)((e->nwords + kWordsPerCompactTile - 1) / kWordsPerCompactTile) + 256;
  for (int r = 0; r < 2; r++) {  // one slot more than tiles: the ticket counter
    RC(dalloc(e, &e->lb[r].slot, e->lb_tiles + 1));
    e->lb[r].ticket = (uint32_t *)(e->lb[r].slot + e->lb_tiles);
    // epochs start at 1: zeroed slots are "empty"
    CK(cudaMemsetAsync(e->lb[r].slot, 0, sizeof(ulonglong2) * (e->lb_tiles + 1), e->s_main));
  }
  RC(dalloc(e, &e->counts_d, 64));  // 1 KiB
  CK(cudaMemsetAsync(e->counts_d, 0, kControlCounts * sizeof(Counts), e->s_main));
  e->err_d = (uint32_t *)(e->counts_d + 3);
  e->active_d = e->err_d + 1;
  e->sb_masks = (uint32_t *)(e->counts_d + 4);
  RC(dalloc(e, &e->sum64_d, 3ull * e->sms * 8 + 4));
  CK(cudaMallocHost(&e->counts_h, kControlCounts * sizeof(Counts)));
  e->err_h = (uint32_t *)(e->counts_h + 3);
  RC(dalloc(e, (char **)&e->rounds_d, kJumps * sizeof(RoundsState)));
  CK(cudaMallocHost(&e->rounds_h, sizeof(RoundsState) + 4 * kPostedResult));  // the state, then a small result
  CK(cudaMallocHost(&e->prl_h, sizeof(PrLoop)));
  if (P.chunk_edges && !(e->cfg.flags & OG_CFG_DIRECT)) {
    for (int b = 0; b < 2; b++) {
      RC(dalloc(e, &e->stage_col[b], P.chunk_edges));
      if (e->wbytes) RC(dalloc(e, (char **)&e->stage_w[b], P.chunk_edges * e->wbytes));
    }
    RC(dalloc(e, &e->ring_d, kRingPad + kRingSlots));  // 8 KiB of the planner's 64 for small arrays
  }
  // PageRank's contributions and sums live in the batch arena when the
  // engine has one (a context runs one computation at a time)
  const bool arena = e->batch_enabled || e->sb_k;
  if (e->pr_enabled) {
    if (!arena) {
      RC(dalloc(e, &e->contrib_d, V + 1));
      RC(dalloc(e, &e->sum_d, V + 1));
    }
    e->pr_tiles = e->tile_cap[0] + e->tile_cap[1];
    RC(dalloc(e, &e->cont_d, e->pr_tiles));
    RC(dalloc(e, &e->carry_d, e->pr_tiles));
    RC(dalloc(e, &e->carry_idx_d, e->pr_tiles));
    e->part_n = (uint32_t)e->sms * 8;
    RC(dalloc(e, &e->part_d, e->part_n));
    RC(dalloc(e, &e->prl_d, 1));
  }
  if (arena) {
    // one arena for the batched BFS masks (24 B per vertex), the
    // multi-source SSSP rows (4 sb_ks + 8 B per vertex) and PageRank's
    // contributions and sums (8 B per vertex): a context runs one at a time
    uint64_t per = std::max<uint64_t>(e->batch_enabled ? 24 : 0, e->sb_k ? 4ull * e->sb_ks + 8 : 0);
    if (e->pr_enabled) per = std::max<uint64_t>(per, 8);
    RC(dalloc(e, &e->arena, per * (V + 1)));
    if (e->pr_enabled) {
      e->contrib_d = (float *)e->arena;
      e->sum_d = e->contrib_d + (V + 4) / 4 * 4;  // 16-byte aligned; 8 of at least 24 B per vertex
    }
    if (e->batch_enabled)
      for (int i = 0; i < 3; i++) e->bmask[i] = (unsigned long long *)e->arena + (uint64_t)i * (V + 1);
    if (e->sb_k) {
      e->sb_dist = (uint32_t *)e->arena;
      e->sb_pend = e->sb_dist + (V + 1) * e->sb_ks;
      e->sb_lmask = e->sb_pend + (V + 1);  // list_cap[0] + list_cap[1] <= V + 1 entries
      RC(dalloc(e, &e->sb_io_d, 128));
      RC(dalloc(e, &e->sb_ck_d, 2 * kSbMaxSources));
      CK(cudaMallocHost(&e->sb_io_h, 128 * sizeof(uint32_t)));
      CK(cudaMallocHost(&e->sb_ck_h, 2 * kSbMaxSources * sizeof(unsigned long long)));
    }
  }
  if (e->batch_enabled) {
    RC(dalloc(e, &e->hist_d, (uint64_t)kMaxBatchLevels * 64));
    RC(dalloc(e, &e->srcs_d, 64));
    RC(dalloc(e, &e->bb_io_d, 192));
    CK(cudaMallocHost(&e->bb_io_h, 192 * sizeof(uint32_t)));
    e->ptile_cap = e->g->E / 1024 + 8;
    RC(dalloc(e, &e->ptile_d, e->ptile_cap));
    RC(dalloc(e, &e->cta_n, kMaxPersistCtas));
    RC(dalloc(e, &e->cta_e, kMaxPersistCtas));
    RC(dalloc(e, &e->smf_d, 2 * 64));
    RC(dalloc(e, &e->bar_d, 16));  // barrier (2), error, levels, stats (6 u64)
    CK(cudaMallocHost(&e->hist_h, (size_t)kMaxBatchLevels * 64 * sizeof(unsigned long long)));
    CK(cudaMallocHost(&e->srcs_h, 64 * sizeof(uint32_t)));
    CK(cudaMallocHost(&e->pmisc_h, 16 * sizeof(uint32_t)));
  }
  CK(cudaMemsetAsync(e->err_d, 0, 16, e->s_main));
  CK(cudaStreamSynchronize(e->s_main));
  return OG_OK;
}

int create(og_graph *g, const og_config *cfg, og_engine *e) {
  e->g = g;
  e->cfg = *cfg;
  e->dev = cfg->device;
  e->V = g->V;
  e->pr_enabled = g->kind == OG_GRAPH_PR || (cfg->flags & OG_CFG_PR);
  e->batch_enabled = (cfg->flags & OG_CFG_BATCH) != 0;
  e->sb_k = sb_sources(cfg->flags);
  if (e->sb_k > kSbMaxSources) return fail(OG_E_ARG, "OG_CFG_SSSP_BATCH(%u): at most %u sources", e->sb_k, kSbMaxSources);
  if (e->sb_k && g->kind != OG_GRAPH_WEIGHTED) return fail(OG_E_UNSUPPORTED, "multi-source SSSP needs a weighted graph");
  e->sb_ks = e->sb_k ? sb_row_slots(e->sb_k) : 0;
  CK(cudaSetDevice(e->dev));
  CK(cudaDeviceGetAttribute(&e->sms, cudaDevAttrMultiProcessorCount, e->dev));
  RC(graph_prepare(g));
  // default near/far width: a sixteenth of the weight range's midpoint sum
  // (4 for weights in [1, 64]), at least 1
  e->sssp_delta = g->kind == OG_GRAPH_WEIGHTED ? std::max<uint32_t>(1, (uint32_t)(((uint64_t)g->wmin + g->wmax) / 16)) : 0;
  e->wbytes = g->wbytes;
  e->bpe = g->bpe;
  e->bc = g->bc;
  e->wmin = g->wmin;
  RC(plan_compute(g->V, g->E, g->off, g->kind, cfg->budget_bytes, cfg->advisek, cfg->flags, &e->plan,
                  g->bpe, 4 + g->wbytes));
  if (cfg->flags & OG_CFG_REPLACE) {
    // half of the static prefix's bytes become fragment slots (the same split
    // og_graph_plan reports)
    uint64_t slot_bytes = 0;
    RC(plan_replace_split(g, cfg->flags, &e->plan, &slot_bytes));
    e->frag = new FragState;
    e->frag->bytes = slot_bytes;
  }
  const og_plan &P = e->plan;
  size_t free_b = 0, total_b = 0;
  CK(cudaMemGetInfo(&free_b, &total_b));
  if (P.budget_bytes > free_b)
    return fail(OG_E_BUDGET, "budget %llu B exceeds free device memory %llu B",
                (unsigned long long)P.budget_bytes, (unsigned long long)free_b);
  e->Vs = P.static_vertices;
  e->nwords = ((uint64_t)g->V + 31) / 32 + 2 * kWordsPerCompactTile;

  // kernels with more than 48 KB of shared memory opt in once per process
  const int gsm = (int)gather_smem_bytes<kGatherMult>();
  CK(cudaFuncSetAttribute(k_gather<SrcP<false>, DstU, kGatherMult>,
                          cudaFuncAttributeMaxDynamicSharedMemorySize, gsm));
  CK(cudaFuncSetAttribute(k_gather<SrcP<true>, DstW<uint8_t>, kGatherMult>,
                          cudaFuncAttributeMaxDynamicSharedMemorySize, gsm));
  CK(cudaFuncSetAttribute(k_gather<SrcP<true>, DstW<uint16_t>, kGatherMult>,
                          cudaFuncAttributeMaxDynamicSharedMemorySize, gsm));
  CK(cudaFuncSetAttribute(k_gather<SrcP<true>, DstW<uint32_t>, kGatherMult>,
                          cudaFuncAttributeMaxDynamicSharedMemorySize, gsm));
  // The SSSP relax reads each packed record as two overlapping words; the
  // second mostly hits L1, so it runs best with a large L1: 58 % of the
  // unified L1/shared storage as shared memory (3 CTAs of 38 KB per SM,
  // ~124 KB of L1).  Measured on R-MAT 27: 9.55 queries/s with the CUDA driver's
  // choice, 9.85 at 58 %, 6.77 at 86 %, 8.06 at 30 %.
  CK(cudaFuncSetAttribute(k_lbs_pair<SrcP<true>, SrcP<true>, MinOp<true>>,
                          cudaFuncAttributePreferredSharedMemoryCarveout, 58));
  CK(cudaFuncSetAttribute(k_bfs_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallShared)));
  if (cfg->flags & OG_CFG_REPLACE) {  // the same relax reading fragment slots
    CK(cudaFuncSetAttribute(k_lbs_pair<SrcP<true>, SrcF<true>, MinOp<true>>,
                            cudaFuncAttributePreferredSharedMemoryCarveout, 58));
    CK(cudaFuncSetAttribute(k_lbs<SrcF<true>, MinOp<true>>, cudaFuncAttributePreferredSharedMemoryCarveout, 58));
  }
  // The cursor form of the PageRank pull (18 KB of tables a CTA): 58 %.  The
  // contiguous form (10 KB) runs within 1.5 % of its best at the CUDA driver's
  // choice (8.4 M vertices, 131 M edges, 49 iterations: 30.9 ms; 30.5 at 30 %,
  // 37.1 at 20 %, 33.5 at 70 %).
  CK(cudaFuncSetAttribute(k_pr_pull<false, SrcP<false>>, cudaFuncAttributePreferredSharedMemoryCarveout, 58));
  CK(cudaFuncSetAttribute(k_pr_pull_pair<false, SrcP<false>>, cudaFuncAttributePreferredSharedMemoryCarveout, 58));

  // host CSR: page-lock so kernels can gather from it over the link
  if (P.dynamic_edges > 0) {
    if (cfg->flags & OG_CFG_NO_PIN) {
      int pageable = 0;
      CK(cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, e->dev));
      if (!pageable) return fail(OG_E_UNSUPPORTED, "device cannot read pageable host memory");
      e->hpk_d = g->packed;
    } else {
      if (g->registered == 0) {
        int ro = 0;
        cudaDeviceGetAttribute(&ro, cudaDevAttrHostRegisterReadOnlySupported, e->dev);
        CK(cudaHostRegister(g->packed, g->packed_words * 4,
                            cudaHostRegisterMapped | (ro ? cudaHostRegisterReadOnly : 0)));
      }
      g->registered++;
      e->registered = true;
      void *dp = nullptr;
      CK(cudaHostGetDevicePointer(&dp, g->packed, 0));
      e->hpk_d = (const uint32_t *)dp;
    }
  }

  // resident graph state shared with clones
  const uint64_t V = g->V;
  RC(dalloc(e, &e->off_d, V + 1));
  if (P.static_edges) RC(dalloc(e, &e->spk_d, g->packed_words_for(P.static_edges) + 4));  // records4
  if (e->pr_enabled) RC(dalloc(e, &e->outdeg_d, V + 1));
  e->resident_bytes = e->dbytes;
  if (e->frag) RC(frag_layout(e, frag_default_shift(g->packed_words)));
  RC(create_query_state(e));
  if (e->dbytes > P.budget_bytes)
    return fail(OG_E_BUDGET, "engine allocated %llu B, above the %llu B budget",
                (unsigned long long)e->dbytes, (unsigned long long)P.budget_bytes);

  // initGraphDevice: offsets, the static edge prefix, PageRank out-degrees
  CK(cudaMemcpyAsync(e->off_d, g->off, 8 * (V + 1), cudaMemcpyHostToDevice, e->s_main));
  if (P.static_edges)
    CK(cudaMemcpyAsync(e->spk_d, g->packed, 4 * g->packed_words_for(P.static_edges),
                       cudaMemcpyHostToDevice, e->s_main));
  if (e->pr_enabled) {
    if (g->kind == OG_GRAPH_PR) {
      CK(cudaMemcpyAsync(e->outdeg_d, g->outdeg, 4 * V, cudaMemcpyHostToDevice, e->s_main));
    } else {
      k_degree_from_offsets<<<grid_for(V, e->sms), kThreads, 0, e->s_main>>>(V, e->off_d, e->outdeg_d);
      e->launches++;
    }
  }
  if (e->frag) RC(frag_reset(e));
  CK(cudaStreamSynchronize(e->s_main));
  CK(cudaGetLastError());
  return OG_OK;
}

// A query context on the parent's resident graph (nothing resident is copied).
int clone(og_engine *parent, og_engine *e) {
  e->parent = parent;
  e->g = parent->g;
  e->cfg = parent->cfg;
  e->plan = parent->plan;
  e->dev = parent->dev;
  e->sms = parent->sms;
  e->pr_enabled = parent->pr_enabled;
  e->batch_enabled = parent->batch_enabled;
  e->sb_k = parent->sb_k;
  e->sb_ks = parent->sb_ks;
  e->sb_delta = parent->sb_delta;
  e->V = parent->V;
  e->Vs = parent->Vs;
  e->nwords = parent->nwords;
  e->off_d = parent->off_d;
  e->spk_d = parent->spk_d;
  e->hpk_d = parent->hpk_d;
  e->bpe = parent->bpe;
  e->bc = parent->bc;
  e->wmin = parent->wmin;
  e->wbytes = parent->wbytes;
  e->outdeg_d = parent->outdeg_d;
  e->tuned = parent->tuned;
  e->sssp_delta = parent->sssp_delta;
  e->cc_method = parent->cc_method;
  e->bfs_direction = parent->bfs_direction;
  e->level_loop = parent->level_loop;
  e->relax_timer = parent->relax_timer;
  CK(cudaSetDevice(e->dev));
  RC(create_query_state(e));
  parent->clones++;
  return OG_OK;
}

// ------------------------------------------------------------------ rounds

// Near/far split (SplitArgs::on): list only vertices with value < thr; the
// waiting ones go to far_bits (when not null) and their minimum to the
// region's Counts::far_min; listed ones are cleared from clear_bits.
struct SplitArgs {
  bool on = false;
  uint32_t thr = 0;
  uint32_t *far_bits = nullptr;
  uint32_t *clear_bits = nullptr;
};

// Words per compaction tile: the smallest of 128, 256, 512 and 1024 that
// keeps the range within max_tiles tiles.  Small tiles spread a small graph
// over the SMs (2^20 vertices are 32 tiles of 1024 words but 256 of 128);
// beyond what is resident at once (four CTAs per SM) more tiles only add
// latency.
uint32_t compact_tile_words(uint32_t words, uint32_t max_tiles) {
  uint32_t tw = 128;
  while (tw < kWordsPerCompactTile && (words + tw - 1) / tw > max_tiles) tw *= 2;
  return tw;
}

CompactArgs compact_args(og_engine *e, int r, const uint32_t *bits, const SplitArgs &sp) {
  const uint32_t vb = r ? e->Vs : 0, ve = r ? e->V : e->Vs;
  CompactArgs a{};
  a.counts = e->counts_d + r;
  if (ve <= vb) return a;  // empty region
  a.bits = bits;
  a.v_begin = vb;
  a.v_end = ve;
  a.w_begin = vb / 32;
  a.w_end = (uint32_t)(((uint64_t)ve + 31) / 32);
  a.tile_words = compact_tile_words(a.w_end - a.w_begin, std::min(e->lb_tiles - 1, 4u * (uint32_t)e->sms));
  a.ntiles = (a.w_end - a.w_begin + a.tile_words - 1) / a.tile_words;
  a.off = e->off_d;
  a.list = e->list_d[r];
  a.pref = e->pref_d[r];
  a.tile_first = e->tile_d[r];
  a.lb = e->lb[r];
  a.err = e->err_d;
  a.list_cap = e->list_cap[r];
  a.tile_cap = e->tile_cap[r];
  a.value = e->value_d;
  a.thr = sp.thr;
  a.split = sp.on ? 1u : 0u;
  a.far_bits = sp.far_bits;
  a.far_key = (unsigned long long *)(e->counts_d + 2) + r;
  a.clear_bits = sp.clear_bits;
  a.epoch = e->epoch;
  return a;
}

// Both regions in one launch.
template <class Args, class Kernel>
int launch_compact(og_engine *e, const CompactPair<Args> &p, Kernel kernel) {
  const uint32_t n0 = p.r[0].ntiles, n1 = p.r[1].ntiles;
  if (std::max(n0, n1) + 1 > e->lb_tiles) return fail(OG_E_STATE, "compaction scratch too small");
  if (n0 + n1) {
    kernel<<<n0 + n1, kThreads, 0, e->s_main>>>(p);
    e->launches++;
  } else {
    CK(cudaMemsetAsync(e->counts_d, 0, 2 * sizeof(Counts), e->s_main));
  }
  return OG_OK;
}

// Waits for a compaction and what is enqueued before it; counts, error words
// and multi-source masks come to the host in one copy.
int compact_wait(og_engine *e) {
  static_assert(sizeof(Counts) == sizeof(uint4), "one word per entry");
  k_publish<<<1, 32, 0, e->s_main>>>((const uint4 *)e->counts_d, (uint4 *)e->counts_h, kControlCounts);
  e->launches++;
  CK(cudaStreamSynchronize(e->s_main));
  return OG_OK;
}

LbsArgs lbs_args(og_engine *e, int r, uint64_t pos_begin, uint64_t pos_end, bool csr,
                 uint64_t edge_bound) {
  LbsArgs a;
  a.list = e->list_d[r];
  a.pref = e->pref_d[r];
  a.tile_first = e->tile_d[r];
  a.n = e->counts_h[r].n;
  a.total = e->counts_h[r].total;
  a.pos_begin = pos_begin;
  a.pos_end = pos_end;
  a.off = csr ? e->off_d : nullptr;
  a.stage_base = pos_begin;
  a.edge_bound = edge_bound;
  a.err = e->err_d;
  return a;
}

unsigned lbs_grid(uint64_t pb, uint64_t pe) { return (unsigned)((pe - pb + kTile - 1) / kTile); }

int check_device_error(og_engine *e) {
  const uint32_t err = *e->err_h;
  if (!err) return OG_OK;
  if (err & kErrLookback) return fail(OG_E_TIMEOUT, "frontier compaction look-back wait gave up");
  if (err & kErrBarrier) return fail(OG_E_TIMEOUT, "a wait between thread blocks gave up");
  return fail(OG_E_DEVICE, "kernel reported an out-of-range index (flags 0x%x)", err);
}

// Edge views of an engine: EK<void> reads columns only (BFS, CC, PageRank,
// batched BFS), EK<W> columns and weights (SSSP, W = staging weight type).
// The static region and the host copy are packed records (PSrc); staging
// buffers hold unpacked edges (Src / Dst).
template <class W>
struct EK {
  static constexpr bool kFrag = false;
  using PSrc = SrcP<true>;
  using Src = SrcW<W>;
  using Dst = DstW<W>;
  static PSrc stat(const og_engine *e) { return PSrc{e->spk_d, e->bpe, e->bc, e->wmin}; }
  static PSrc host(const og_engine *e) { return PSrc{e->hpk_d, e->bpe, e->bc, e->wmin}; }
  static Src stage(const og_engine *e, int b) { return Src{e->stage_col[b], (const W *)e->stage_w[b]}; }
  static Dst stage_dst(const og_engine *e, int b) { return Dst{e->stage_col[b], (W *)e->stage_w[b]}; }
};
template <>
struct EK<void> {
  static constexpr bool kFrag = false;
  using PSrc = SrcP<false>;
  using Src = SrcU;
  using Dst = DstU;
  static PSrc stat(const og_engine *e) { return PSrc{e->spk_d, e->bpe, e->bc, e->wmin}; }
  static PSrc host(const og_engine *e) { return PSrc{e->hpk_d, e->bpe, e->bc, e->wmin}; }
  static Src stage(const og_engine *e, int b) { return Src{e->stage_col[b]}; }
  static Dst stage_dst(const og_engine *e, int b) { return Dst{e->stage_col[b]}; }
};
using EKU = EK<void>;
// An OG_CFG_REPLACE engine's views: the dynamic region is read through the
// fragment slots (direct mode only: there are no staging buffers).
template <class W>
struct EKF : EK<W> {
  static constexpr bool kFrag = true;
  using HSrc = SrcF<!std::is_void<W>::value>;
  static HSrc host(const og_engine *e) {
    HSrc h;
    h.words = e->hpk_d;
    h.bpe = e->bpe;
    h.bc = e->bc;
    h.wmin = e->wmin;
    h.slots = e->frag->slots_d;
    h.slot_of = e->frag->slot_of_d;
    h.visits = e->frag->visits_d;
    h.miss = e->frag->miss_d;
    h.fs = e->frag->fs;
    return h;
  }
};

// Relax op factory per algorithm; `level` is the BFS depth of the frontier.
struct RoundOps {
  int algo;
  uint32_t level;
};

template <class Src0, class Src1>
int launch_relax_pair(og_engine *e, const RoundOps &ro, const LbsArgs &a0, Src0 s0, const LbsArgs &a1,
                      Src1 s1, uint32_t *next, cudaStream_t s) {
  const uint64_t n0 = lbs_grid(a0.pos_begin, a0.pos_end), n1 = lbs_grid(a1.pos_begin, a1.pos_end);
  const uint64_t n = n0 + n1;
  if (n == 0) return OG_OK;
  if (n > 0x7fffffffull) return fail(OG_E_STATE, "relax grid of %llu tiles", (unsigned long long)n);
  if (ro.algo == OG_ALGO_BFS) {
    BfsOp op{e->bm[2], next, e->value_d, e->err_d, e->V, ro.level + 1};
    k_lbs_pair<Src0, Src1, BfsOp><<<(unsigned)n, kThreads, 0, s>>>(a0, s0, a1, s1, op, n0, n);
  } else if (ro.algo == OG_ALGO_SSSP) {
    MinOp<true> op{e->value_d, next, e->err_d, e->V};
    k_lbs_pair<Src0, Src1, MinOp<true>><<<(unsigned)n, kThreads, 0, s>>>(a0, s0, a1, s1, op, n0, n);
  } else {
    MinOp<false> op{e->value_d, next, e->err_d, e->V};
    k_lbs_pair<Src0, Src1, MinOp<false>><<<(unsigned)n, kThreads, 0, s>>>(a0, s0, a1, s1, op, n0, n);
  }
  e->launches++;
  return OG_OK;
}

template <class Src>
int launch_relax(og_engine *e, const RoundOps &ro, const LbsArgs &a, Src src, uint32_t *next,
                 cudaStream_t s) {
  const unsigned grid = lbs_grid(a.pos_begin, a.pos_end);
  if (grid == 0) return OG_OK;
  if (ro.algo == OG_ALGO_BFS) {
    BfsOp op{e->bm[2], next, e->value_d, e->err_d, e->V, ro.level + 1};
    k_lbs<Src, BfsOp><<<grid, kThreads, 0, s>>>(a, src, op);
  } else if (ro.algo == OG_ALGO_SSSP) {
    MinOp<true> op{e->value_d, next, e->err_d, e->V};
    k_lbs<Src, MinOp<true>><<<grid, kThreads, 0, s>>>(a, src, op);
  } else {
    MinOp<false> op{e->value_d, next, e->err_d, e->V};
    k_lbs<Src, MinOp<false>><<<grid, kThreads, 0, s>>>(a, src, op);
  }
  e->launches++;
  return OG_OK;
}

// The ring of a staged round (k_stage_round) over both staging buffers, cleared
// on `s`.
int stage_ring(og_engine *e, StageRing *g, cudaStream_t s) {
  const uint64_t half = e->plan.chunk_edges / kTile;
  g->state = e->ring_d + kRingPad;
  g->ticket = e->ring_d;
  g->slots = (uint32_t)std::min<uint64_t>(2 * half, kRingSlots);
  g->half = (uint32_t)std::min<uint64_t>(half, kRingSlots);
  CK(cudaMemsetAsync(e->ring_d, 0, 4ull * (kRingPad + g->slots), s));
  return OG_OK;
}

// A staged round of the dynamic list `a`.
template <class K>
int launch_stage_round(og_engine *e, const RoundOps &ro, const LbsArgs &a, uint32_t *next, cudaStream_t s) {
  StageRing ring;
  RC(stage_ring(e, &ring, s));
  const unsigned grid = 2 * lbs_grid(0, a.total);
  auto launch = [&](auto op) {
    k_stage_round<<<grid, kThreads, 0, s>>>(a, K::host(e), K::stage_dst(e, 0), K::stage_dst(e, 1), K::stage(e, 0),
                                            K::stage(e, 1), e->plan.chunk_edges, op, ring);
  };
  if constexpr (std::is_same<typename K::Src, SrcU>::value) {
    if (ro.algo == OG_ALGO_BFS) launch(BfsOp{e->bm[2], next, e->value_d, e->err_d, e->V, ro.level + 1});
    else launch(MinOp<false>{e->value_d, next, e->err_d, e->V});
  } else {
    launch(MinOp<true>{e->value_d, next, e->err_d, e->V});
  }
  e->launches++;
  return OG_OK;
}

template <class K>
int launch_gather(og_engine *e, const LbsArgs &a, int buf, cudaStream_t s) {
  constexpr uint64_t T = (uint64_t)kGatherMult * kTile;
  const unsigned grid = (unsigned)((a.pos_end - a.pos_begin + T - 1) / T);
  if (grid == 0) return OG_OK;
  k_gather<typename K::PSrc, typename K::Dst, kGatherMult>
      <<<grid, kThreads, gather_smem_bytes<kGatherMult>(), s>>>(a, K::host(e), K::stage_dst(e, buf));
  e->launches++;
  return OG_OK;
}

struct Timing {
  bool pend_s = false, pend_d = false;
  uint32_t pend_g = 0;  // gather launches whose event pair is still to be read
};

// Event pair g of the gather timing list, created on first use.
int gather_events(og_engine *e, uint32_t g, cudaEvent_t *b, cudaEvent_t *en) {
  while (e->t_gat.size() < 2ull * (g + 1)) {
    cudaEvent_t ev;
    CK(cudaEventCreate(&ev));
    e->t_gat.push_back(ev);
  }
  *b = e->t_gat[2 * g];
  *en = e->t_gat[2 * g + 1];
  return OG_OK;
}

void collect_timing(og_engine *e, Timing &t, og_stats *st) {
  float ms;
  if (t.pend_s && cudaEventElapsedTime(&ms, e->t_s0, e->t_s1) == cudaSuccess) st->ms_static += ms;
  if (t.pend_d && cudaEventElapsedTime(&ms, e->t_d0, e->ev_dyn_done) == cudaSuccess)
    st->ms_dynamic += ms;
  for (uint32_t g = 0; g < t.pend_g; g++)
    if (cudaEventElapsedTime(&ms, e->t_gat[2 * g], e->t_gat[2 * g + 1]) == cudaSuccess)
      st->ms_gather += ms;
  t.pend_s = t.pend_d = false;
  t.pend_g = 0;
}

struct NoPair {};
struct NoStage {};

// Whether the caller of run_regions has put work on s_main since the counts came
// back (push PageRank clears its sums there, the L1 pull updates the ranks): the
// dynamic region's own stream then waits for it, 2 us a round.
enum class MainStream { kIdle, kBusy };

// One round's region work given the compaction counts (already on the host).
// `static_fn(a)` / `dyn_fn(a, src, stream)` launch the per-region kernel;
// `pair_fn(a0, src0, a1, src1, stream)`, when given, launches both regions
// as one interleaved kernel (direct mode with both regions non-empty): the
// static tiles then overlap the link-bound dynamic ones instead of taking the
// SMs first.  Its time is counted as dynamic-region time.
// `stage_fn(a)`, when given, launches a staged round of the dynamic list a.
// `main`: see MainStream.
template <class K, class StaticFn, class DynFn, class PairFn = NoPair, class StageFn = NoStage>
int run_regions(og_engine *e, og_stats &st, Timing &tm, MainStream main, StaticFn static_fn, DynFn dyn_fn,
                PairFn pair_fn = PairFn(), StageFn stage_fn = StageFn()) {
  const Counts cs = e->counts_h[0], cd = e->counts_h[1];
  if constexpr (!std::is_same<PairFn, NoPair>::value) {
    if (cs.n && cd.n && (e->cfg.flags & OG_CFG_DIRECT)) {
      CK(cudaEventRecord(e->t_d0, e->s_main));
      RC(pair_fn(lbs_args(e, 0, 0, cs.total, true, e->plan.static_edges), K::stat(e),
                 lbs_args(e, 1, 0, cd.total, true, e->g->E), K::host(e), e->s_main));
      CK(cudaEventRecord(e->ev_dyn_done, e->s_main));
      tm.pend_d = true;
      st.chunks += 1;
      st.edges_static += cs.total;
      st.edges_dynamic += cd.total;
      st.link_bytes += (cd.total * e->bpe + 7) / 8;
      return OG_OK;
    }
  }
  if (cd.n && main == MainStream::kBusy) {
    CK(cudaEventRecord(e->ev_round, e->s_main));
    CK(cudaStreamWaitEvent(e->s_dyn, e->ev_round, 0));
  }
  if (cs.n) {
    CK(cudaEventRecord(e->t_s0, e->s_main));
    RC(static_fn(lbs_args(e, 0, 0, cs.total, true, e->plan.static_edges)));
    CK(cudaEventRecord(e->t_s1, e->s_main));
    tm.pend_s = true;
    st.edges_static += cs.total;
  }
  if (cd.n) {
    CK(cudaEventRecord(e->t_d0, e->s_dyn));
    if (K::kFrag || (e->cfg.flags & OG_CFG_DIRECT)) {
      RC(dyn_fn(lbs_args(e, 1, 0, cd.total, true, e->g->E), K::host(e), e->s_dyn));
      st.chunks += 1;
    } else if constexpr (!K::kFrag) {
      const uint64_t C = e->plan.chunk_edges;
      const uint64_t nch = (cd.total + C - 1) / C;
      if constexpr (!std::is_same<StageFn, NoStage>::value) {
        cudaEvent_t g0, g1;
        RC(gather_events(e, tm.pend_g, &g0, &g1));
        CK(cudaEventRecord(g0, e->s_dyn));
        RC(stage_fn(lbs_args(e, 1, 0, cd.total, true, e->g->E)));
        CK(cudaEventRecord(g1, e->s_dyn));
        tm.pend_g++;
      } else
      for (uint64_t c = 0; c < nch; c++) {
        const int buf = (int)(c & 1);
        const uint64_t b = c * C, en = std::min(b + C, cd.total);
        CK(cudaStreamWaitEvent(e->s_gat, e->ev_cd, 0));
        if (c >= 2) CK(cudaStreamWaitEvent(e->s_gat, e->ev_rel[buf], 0));
        cudaEvent_t g0, g1;
        RC(gather_events(e, tm.pend_g, &g0, &g1));
        CK(cudaEventRecord(g0, e->s_gat));
        RC(launch_gather<K>(e, lbs_args(e, 1, b, en, true, e->g->E), buf, e->s_gat));
        CK(cudaEventRecord(g1, e->s_gat));
        tm.pend_g++;
        CK(cudaEventRecord(e->ev_gat[buf], e->s_gat));
        CK(cudaStreamWaitEvent(e->s_dyn, e->ev_gat[buf], 0));
        RC(dyn_fn(lbs_args(e, 1, b, en, false, C), K::stage(e, buf), e->s_dyn));
        CK(cudaEventRecord(e->ev_rel[buf], e->s_dyn));
      }
      st.chunks += (uint32_t)nch;
    }
    CK(cudaEventRecord(e->ev_dyn_done, e->s_dyn));
    CK(cudaStreamWaitEvent(e->s_main, e->ev_dyn_done, 0));
    tm.pend_d = true;
    st.edges_dynamic += cd.total;
    st.link_bytes += (cd.total * e->bpe + 7) / 8;
  }
  return OG_OK;
}

// Compacts both regions of `cur` and brings the counts (and the error word) to
// the host.  Returns the number of listed vertices through *n.
// Smallest waiting value the last compaction of region r saw, or UINT32_MAX
// (its far key carries the launch epoch; another epoch means "none").
uint32_t far_of(const og_engine *e, int r) {
  const uint64_t key = ((const uint64_t *)(e->counts_h + 2))[r];
  return (uint32_t)(key >> 32) == e->epoch ? ~(uint32_t)key : 0xffffffffu;
}

int compact_round(og_engine *e, const uint32_t *cur, og_stats &st, Timing &tm, uint64_t *n,
                  const SplitArgs &sp = SplitArgs()) {
  if (++e->epoch >= (1u << 30)) {  // epoch wrap: clear the status words and far keys once
    for (int r = 0; r < 2; r++)
      CK(cudaMemsetAsync(e->lb[r].slot, 0, sizeof(ulonglong2) * e->lb_tiles, e->s_main));
    CK(cudaMemsetAsync(e->counts_d + 2, 0, sizeof(Counts), e->s_main));
    e->epoch = 1;
  }
  CK(cudaEventRecord(e->ev_round, e->s_main));
  const CompactPair<CompactArgs> p{{compact_args(e, 0, cur, sp), compact_args(e, 1, cur, sp)}};
  RC(launch_compact(e, p, k_compact));
  CK(cudaEventRecord(e->ev_cd, e->s_main));
  RC(compact_wait(e));
  collect_timing(e, tm, &st);
  float ms;
  if (cudaEventElapsedTime(&ms, e->ev_round, e->ev_cd) == cudaSuccess) st.ms_compact += ms;
  RC(check_device_error(e));
  *n = (uint64_t)e->counts_h[0].n + e->counts_h[1].n;
  return OG_OK;
}

template <class K>
int run_frontier(og_engine *e, int algo, uint32_t src, og_stats &st) {
  const uint64_t V = e->V;
  uint32_t *cur = e->bm[0], *next = e->bm[1];
  cudaStream_t s = e->s_main;
  const int g = grid_for(V, e->sms);
  CK(cudaMemsetAsync(e->err_d, 0, 16, s));
  CK(cudaMemsetAsync(cur, 0, 4 * e->nwords, s));
  CK(cudaMemsetAsync(next, 0, 4 * e->nwords, s));
  if (algo == OG_ALGO_BFS) {
    CK(cudaMemsetAsync(e->bm[2], 0, 4 * e->nwords, s));
    k_fill_u32<<<g, kThreads, 0, s>>>(e->value_d, V, (uint32_t)(V + 1));  // GraphMeta.h:378
    k_set_source<<<1, 1, 0, s>>>(e->value_d, src, 1u, cur, e->bm[2]);
    e->launches += 2;
  } else if (algo == OG_ALGO_SSSP) {
    if (e->sssp_delta > 0) CK(cudaMemsetAsync(e->bm[2], 0, 4 * e->nwords, s));  // waiting set
    CK(cudaMemsetAsync(e->counts_d + 2, 0, sizeof(Counts), s));  // far keys of earlier queries
    k_fill_u32<<<g, kThreads, 0, s>>>(e->value_d, V, 0xFFFFFFFFu);  // SSSP GraphMeta.h:377
    k_set_source<<<1, 1, 0, s>>>(e->value_d, src, 1u, cur, nullptr);
    e->launches += 2;
  } else {
    k_iota_u32<<<g, kThreads, 0, s>>>(e->value_d, V);  // CC GraphMeta.h:341-345
    k_fill_bits<<<g, kThreads, 0, s>>>(cur, e->nwords, V);
    e->launches += 2;
  }
  CK(cudaGetLastError());
  Timing tm;
  RoundOps ro{algo, 1};
  // SSSP near/far split (two-bucket delta stepping): a round expands only
  // frontier vertices closer than thr; the others move to the waiting set
  // (bm[2]) and are not looked at again until no near vertex is left.  Then
  // thr moves to the smallest waiting distance + delta and one scan of the
  // waiting set lists the vertices below it.  far_min is the minimum over
  // the waiting set as of the last scan, lowered by every insertion since; a
  // vertex listed from the frontier leaves the waiting set, so the minimum
  // may be stale-low, in which case the scan lists nothing and returns the
  // true minimum for the next try.
  const bool split = algo == OG_ALGO_SSSP && e->sssp_delta > 0;
  uint32_t *waiting = e->bm[2];
  uint64_t thr = 1ull + e->sssp_delta;
  uint32_t far_min = 0xffffffffu;
  bool advance = false;
  // Direction-optimizing BFS (symmetric graphs): a level is expanded bottom-up
  // when its frontier's edges exceed unexplored / kAlpha (unexplored = the
  // degrees of the vertices that have not been a frontier yet), and top-down
  // again once the frontier falls below V / kBeta while shrinking.
  constexpr uint64_t kAlpha = 14, kBeta = 24;
  const bool dopt = algo == OG_ALGO_BFS && e->bfs_direction == OG_BFS_AUTO && e->g->symmetric == 1;
  uint64_t unexplored = e->g->E;
  bool bottom = false, counted = false;
  uint64_t fn = 0;  // frontier size when it came from a bottom-up level
  for (;;) {
    uint64_t n = 0;
    if (dopt && bottom) {
      unsigned long long *cnt = e->sum64_d;  // reached, their degrees, host records, static records
      CK(cudaMemsetAsync(cnt, 0, 32, s));  // next is all zero here, as at every level start
      CK(cudaEventRecord(e->t_d0, s));
      k_bfs_bottom_up<EKU::PSrc><<<grid_for(V, e->sms), kThreads, 0, s>>>(
          e->off_d, (uint32_t)V, e->Vs, EKU::stat(e), EKU::host(e), cur, e->bm[2], next, e->value_d,
          ro.level + 1, cnt, e->err_d);
      e->launches++;
      CK(cudaEventRecord(e->ev_dyn_done, s));
      unsigned long long c4[4];
      CK(cudaMemcpyAsync(c4, cnt, 32, cudaMemcpyDeviceToHost, s));
      CK(cudaMemcpyAsync(e->err_h, e->err_d, 4, cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
      RC(check_device_error(e));
      float ms = 0;
      if (cudaEventElapsedTime(&ms, e->t_d0, e->ev_dyn_done) == cudaSuccess) st.ms_dynamic += ms;
      st.iterations++;
      st.frontier_sum += fn;
      st.edges_dynamic += c4[2];
      st.edges_static += c4[3];
      st.link_bytes += (c4[2] * e->bpe + 7) / 8;
      unexplored -= std::min<uint64_t>(unexplored, c4[1]);
      std::swap(cur, next);
      CK(cudaMemsetAsync(next, 0, 4 * e->nwords, s));  // the level just expanded
      ro.level++;
      if (c4[0] == 0) break;
      if (c4[0] < V / kBeta && c4[0] < fn) bottom = false;  // next level: compaction + top-down
      fn = c4[0];
      counted = true;
      continue;
    }
    SplitArgs sp;
    sp.on = split;
    sp.thr = (uint32_t)std::min<uint64_t>(thr, 0xffffffffull);
    sp.clear_bits = split ? waiting : nullptr;
    sp.far_bits = split && !advance ? waiting : nullptr;
    RC(compact_round(e, advance ? waiting : cur, st, tm, &n, sp));
    if constexpr (K::kFrag) RC(frag_step(e, st, n == 0));
    if (split) {
      const uint32_t fm = std::min(far_of(e, 0), far_of(e, 1));
      far_min = advance ? fm : std::min(far_min, fm);
    }
    if (n == 0) {
      if (!split || far_min == 0xffffffffu) break;
      thr = (uint64_t)far_min + e->sssp_delta;
      advance = true;
      continue;
    }
    advance = false;
    if (dopt) {
      const uint64_t mf = e->counts_h[0].total + e->counts_h[1].total;
      if (!counted) unexplored -= std::min(unexplored, mf);
      counted = false;
      if (mf > unexplored / kAlpha) {  // expand this frontier bottom-up
        bottom = true;
        fn = n;
        counted = true;
        continue;
      }
    }
    st.iterations++;
    st.frontier_sum += n;
    st.static_vertices += e->counts_h[0].n;
    auto sfn = [&](const LbsArgs &a) { return launch_relax(e, ro, a, K::stat(e), next, e->s_main); };
    auto dfn = [&](const LbsArgs &a, auto src, cudaStream_t ds) {
      return launch_relax(e, ro, a, src, next, ds);
    };
    auto pfn = [&](const LbsArgs &a0, auto s0, const LbsArgs &a1, auto s1, cudaStream_t ps) {
      return launch_relax_pair(e, ro, a0, s0, a1, s1, next, ps);
    };
    auto gfn = [&](const LbsArgs &a) {
      if constexpr (K::kFrag) return (int)OG_OK;  // direct mode only
      else return launch_stage_round<K>(e, ro, a, next, e->s_dyn);
    };
    RC((run_regions<K>(e, st, tm, MainStream::kIdle, sfn, dfn, pfn, gfn)));
    if constexpr (K::kFrag) e->frag->since += e->counts_h[1].total;
    CK(cudaMemsetAsync(cur, 0, 4 * e->nwords, e->s_main));
    std::swap(cur, next);
    ro.level++;
    CK(cudaGetLastError());
  }
  CK(cudaStreamSynchronize(e->s_main));
  CK(cudaMemcpy(e->err_h, e->err_d, 4, cudaMemcpyDeviceToHost));
  RC(check_device_error(e));
  e->last_algo = algo;
  return OG_OK;
}

// ---------------------------------------------------- device-driven rounds

// Whether a query runs in one cooperative kernel (rounds.cuh): direct mode or a
// fully resident graph (no staging pipeline to drive), and counters that fit
// its packed list reservations.
bool rounds_on_device(const og_engine *e) {
  return e->level_loop == OG_LOOP_AUTO && (e->plan.dynamic_edges == 0 || (e->cfg.flags & OG_CFG_DIRECT)) &&
         rounds_fit(e->V, e->g->E);
}

// Waits for the rounds kernel's state (rounds_post): it is in page-locked memory
// before the kernel has quite ended, so that the copy of the result can be
// enqueued meanwhile.  Returns as well when the stream is idle or failed, which
// is asked for rarely: the call takes the CUDA driver's locks.
int rounds_wait(og_engine *e) {
  const volatile uint32_t *posted = &e->rounds_h->posted;
  for (uint32_t i = 1; !*posted; i++) {
    if (i % 65536) continue;
    const cudaError_t q = cudaStreamQuery(e->s_main);
    if (q == cudaErrorNotReady) continue;
    CK(q);
    break;
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  return OG_OK;
}

// Tiles above which a round is relaxed by a launch of its own (hands_over), and
// vertices from which a bottom-up level is expanded by one.  A handover costs a
// wait and two launches, about 25 us.  In the rounds kernel / handed over, ms:
// resident rounds, label propagation on R-MAT 20 (16 thousand tiles a round) 0.82 /
// 0.50, 22 3.27 / 1.69, 24 13.6 / 6.8, at 4096 tiles about even; SSSP over
// the link, R-MAT 24 12.3 / 12.3, 26 54.1 / 47.5, 27 117 / 94.7; top-down BFS over
// the link, 24 8.73 / 8.96, 27 75.0 / 77.1: never handed over.  Bottom-up levels of
// BFS over the link, R-MAT 22 0.54 / 0.60, 23 0.92 / 0.92, 24 2.04 / 1.94, 27 14.2 /
// 12.6; resident 24 1.15 / 1.01.
constexpr uint64_t kHandHbm = 4096, kHandLink = 32768;
constexpr uint32_t kHandBottomVertices = 1u << 24;

// The relax of a round that the rounds kernel has handed over: its lists are in
// place, `op` acts on them as the kernel's would.
template <class Src, class Op>
int relax_handed(og_engine *e, const RoundsState &h, Src s0, Src s1, Op op) {
  LbsArgs a[2];
  uint64_t n[2];
  for (int r = 0; r < 2; r++) {
    Counts &c = e->counts_h[r];
    c.n = (uint32_t)(h.hx[r] >> append_shift(e->g->E));
    c.total = append_edges(h.hx[r], append_shift(e->g->E));
    a[r] = lbs_args(e, r, 0, c.total, true, r ? e->g->E : e->plan.static_edges);
    a[r].err = &e->rounds_d->err;
    n[r] = lbs_grid(0, c.total);
  }
  op.err = &e->rounds_d->err;
  if (n[0] && n[1])
    k_lbs_pair<Src, Src, Op><<<(unsigned)(n[0] + n[1]), kThreads, 0, e->s_main>>>(a[0], s0, a[1], s1, op, n[0],
                                                                                 n[0] + n[1]);
  else if (n[0])
    k_lbs<Src, Op><<<(unsigned)n[0], kThreads, 0, e->s_main>>>(a[0], s0, op);
  else
    k_lbs<Src, Op><<<(unsigned)n[1], kThreads, 0, e->s_main>>>(a[1], s1, op);
  e->launches++;
  return OG_OK;
}

// BFS, SSSP or label-propagation CC as one kernel.  The caller's array is written
// once, after the error word has been read: small results come with the state
// (RoundsArgs::result), larger ones by a copy.
int run_rounds(og_engine *e, int algo, uint32_t src, og_stats &st) {
  cudaStream_t s = e->s_main;
  RoundsArgs a{};
  a.V = e->V;
  a.Vs = e->Vs;
  a.E = e->g->E;
  a.static_edges = e->plan.static_edges;
  a.nwords = e->nwords;
  a.off = e->off_d;
  a.value = e->value_d;
  for (int i = 0; i < 3; i++) a.bm[i] = e->bm[i];
  for (int r = 0; r < 2; r++) {
    a.list[r] = e->list_d[r];
    a.pref[r] = e->pref_d[r];
    a.tile[r] = e->tile_d[r];
    a.list_cap[r] = e->list_cap[r];
    a.tile_cap[r] = e->tile_cap[r];
  }
  a.st = e->rounds_d;
  a.post = e->rounds_h;
  if (e->out && a.V <= kPostedResult) a.result = (uint32_t *)(e->rounds_h + 1);
  a.src = src;
  a.delta = algo == OG_ALGO_SSSP ? e->sssp_delta : 0;
  a.split = a.delta ? 1u : 0u;
  a.dopt = algo == OG_ALGO_BFS && e->bfs_direction == OG_BFS_AUTO && e->g->symmetric == 1;
  a.timer = e->relax_timer;
  a.shift = append_shift(a.E);
  a.spin_limit = wait_limit(a.E);
  a.hand_hbm = kHandHbm;
  a.hand_link = algo == OG_ALGO_BFS ? ~0ull : kHandLink;
  a.hand_bottom = a.V >= kHandBottomVertices;
  SrcP<false> u0 = EKU::stat(e), u1 = EKU::host(e);
  SrcP<true> w0{e->spk_d, e->bpe, e->bc, e->wmin}, w1{e->hpk_d, e->bpe, e->bc, e->wmin};
  const bool bfs = algo == OG_ALGO_BFS;
  const void *kern = bfs                    ? (const void *)k_bfs_rounds
                     : algo == OG_ALGO_SSSP ? (const void *)k_min_rounds<true>
                                            : (const void *)k_min_rounds<false>;
  int occ = 0;
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kThreads, 0));
  if (occ < 1) return fail(OG_E_UNSUPPORTED, "rounds kernel does not fit an SM");
  // all the CTAs that fit at once, or one per edge tile and per 1024 vertices
  // when the graph has fewer: a barrier over a few CTAs is cheaper
  const uint64_t work = std::max<uint64_t>(a.E / kTile, a.V / 1024) + 1;
  const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)occ * e->sms, work);
  void *args[3] = {&a, &u0, &u1};
  if (algo == OG_ALGO_SSSP) {
    args[1] = &w0;
    args[2] = &w1;
  }
  RoundsState &h = *e->rounds_h;
  if (bfs) {
    k_bfs_init<<<grid_for(std::max<uint64_t>(a.V, a.nwords), e->sms), kThreads, 0, s>>>(a);
    e->launches++;
  } else {
    CK(cudaMemsetAsync(e->rounds_d, 0, sizeof(RoundsState), s));
  }
  float ms_handed = 0, ms_handed_relax = 0;
  h.hand = 0;
  for (uint64_t pass = 0;; pass++) {
    h.posted = 0;
    const uint32_t handed = h.hand;
    if (handed) {
      CK(cudaEventRecord(e->t_d0, s));
      if (handed == kHandBottomUp) {
        k_bfs_bottom_up<EKU::PSrc><<<grid_for(a.V, e->sms), kThreads, 0, s>>>(
            e->off_d, a.V, a.Vs, u0, u1, a.bm[h.par], a.bm[2], a.bm[h.par ^ 1], e->value_d, h.level + 1,
            e->rounds_d->hbu, &e->rounds_d->err);
        e->launches++;
      } else if (bfs) {  // the state is already that of the next level
        RC(relax_handed(e, h, u0, u1, BfsOp{a.bm[2], a.bm[h.par], e->value_d, nullptr, a.V, h.level}));
      } else if (algo == OG_ALGO_SSSP) {
        RC(relax_handed(e, h, w0, w1, MinOp<true>{e->value_d, a.bm[h.par], nullptr, a.V}));
      } else {
        RC(relax_handed(e, h, u0, u1, MinOp<false>{e->value_d, a.bm[h.par], nullptr, a.V}));
      }
      CK(cudaEventRecord(e->ev_dyn_done, s));
      CK(cudaMemsetAsync(&e->rounds_d->bar, 0, sizeof e->rounds_d->bar, s));
    } else if (bfs) {
      k_bfs_small<<<1, kSmallThreads, sizeof(SmallShared), s>>>(a, u0, u1);
      e->launches++;
    }
    CK(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(kThreads), args, 0, s));
    e->launches++;
    RC(rounds_wait(e));
    if (!h.posted) {  // the kernel ended without its last stores: a barrier gave up
      CK(cudaMemcpyAsync(&h, e->rounds_d, sizeof h, cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
      if (!h.err) return fail(OG_E_STATE, "the rounds kernel ended early");
      break;
    }
    if (handed) {
      float ms = 0;
      CK(cudaEventElapsedTime(&ms, e->t_d0, e->ev_dyn_done));
      ms_handed += ms;
      if (handed == kHandRelax && a.timer) ms_handed_relax += ms;
    }
    if (h.done || h.err) break;
    if (pass > 2ull * a.V + 64) return fail(OG_E_STATE, "the rounds did not end");
  }
  if (h.err & kErrBarrier) return fail(OG_E_TIMEOUT, "grid barrier wait gave up");
  *e->err_h = h.err;
  RC(check_device_error(e));
  st.ms_dynamic += h.ns_total / 1e6 + ms_handed;
  st.ms_relax += h.ns_relax / 1e6 + ms_handed_relax;
  st.iterations += (uint32_t)h.iterations;
  st.frontier_sum += h.frontier_sum;
  st.edges_static += h.edges_static;
  st.edges_dynamic += h.edges_dynamic;
  st.link_bytes += (h.edges_dynamic * e->bpe + 7) / 8;
  st.chunks += (uint32_t)h.iterations;
  e->last_algo = algo;
  if (e->out && !a.result) return OG_OK;  // fetched by query_common
  CK(cudaStreamSynchronize(s));
  if (e->out) memcpy(e->out, a.result, 4ull * a.V);
  e->out = nullptr;
  return OG_OK;
}

// ------------------------------------------------------------------ batched BFS

// The n x V depth matrix (outside the budget), allocated on first use and
// kept for later calls; it grows when a call needs more sources.
int depth_matrix(og_engine *e, uint32_t n, uint32_t **out) {
  const uint64_t need = (uint64_t)n * e->V;
  if (need > e->depth_cap) {
    if (e->depth_d) cudaFree(e->depth_d);
    e->depth_d = nullptr;
    e->depth_cap = 0;
    CK(cudaMalloc(&e->depth_d, 4 * need));
    e->depth_cap = need;
  }
  *out = e->depth_d;
  return OG_OK;
}

int run_batch(og_engine *e, const uint32_t *srcs, uint32_t n, uint32_t *out, uint64_t *checks,
              og_stats &st) {
  const uint64_t V = e->V;
  uint32_t *cur_any = e->bm[0], *next_any = e->bm[1];
  unsigned long long *visited = e->bmask[0], *cur = e->bmask[1], *next = e->bmask[2];
  cudaStream_t s = e->s_main;
  uint32_t *depth_d = nullptr;
  if (out) {
    RC(depth_matrix(e, n, &depth_d));
    k_fill_u32<<<grid_for(n * V, e->sms), kThreads, 0, s>>>(depth_d, (uint64_t)n * V, (uint32_t)(V + 1));
    e->launches++;
  }
  std::vector<uint64_t> reached(n, 1), dsum(n, 1);  // each source: itself at depth 1
  CK(cudaMemsetAsync(e->err_d, 0, 16, s));
  CK(cudaMemsetAsync(cur_any, 0, 4 * e->nwords, s));
  CK(cudaMemsetAsync(next_any, 0, 4 * e->nwords, s));
  for (int i = 0; i < 3; i++) CK(cudaMemsetAsync(e->bmask[i], 0, 8 * (V + 1), s));
  CK(cudaMemcpyAsync(e->srcs_d, srcs, 4 * n, cudaMemcpyHostToDevice, s));
  k_batch_init<<<1, 64, 0, s>>>(e->srcs_d, n, visited, cur, cur_any, depth_d, V);
  e->launches++;
  CK(cudaGetLastError());
  Timing tm;
  for (uint32_t level = 1;; level++) {
    uint64_t nl = 0;
    RC(compact_round(e, cur_any, st, tm, &nl));
    if (nl == 0) break;
    st.iterations++;
    st.frontier_sum += nl;
    st.static_vertices += e->counts_h[0].n;
    BatchOp op{visited, cur, next, next_any, e->err_d, e->V};
    auto launch = [&](const LbsArgs &a, auto src, cudaStream_t ls) {
      const unsigned grid = lbs_grid(a.pos_begin, a.pos_end);
      if (grid) {
        k_lbs<decltype(src), BatchOp><<<grid, kThreads, 0, ls>>>(a, src, op);
        e->launches++;
      }
      return (int)OG_OK;
    };
    auto sfn = [&](const LbsArgs &a) { return launch(a, EKU::stat(e), e->s_main); };
    auto pfn = [&](const LbsArgs &a0, auto s0, const LbsArgs &a1, auto s1, cudaStream_t ps) {
      const uint64_t n0 = lbs_grid(a0.pos_begin, a0.pos_end), n1 = lbs_grid(a1.pos_begin, a1.pos_end);
      if (n0 + n1 > 0x7fffffffull) return fail(OG_E_STATE, "relax grid too large");
      k_lbs_pair<decltype(s0), decltype(s1), BatchOp><<<(unsigned)(n0 + n1), kThreads, 0, ps>>>(
          a0, s0, a1, s1, op, n0, n0 + n1);
      e->launches++;
      return (int)OG_OK;
    };
    RC((run_regions<EKU>(e, st, tm, MainStream::kIdle, sfn, launch, pfn)));
    CK(cudaMemsetAsync(e->hist_d, 0, 64 * 8, s));
    k_batch_level<<<grid_for(e->nwords, e->sms), kThreads, 0, s>>>(next_any, next, e->nwords, n,
                                                                 e->hist_d, depth_d, V, level + 1);
    e->launches++;
    CK(cudaMemcpyAsync(e->hist_h, e->hist_d, 64 * 8, cudaMemcpyDeviceToHost, s));
    CK(cudaMemsetAsync(cur_any, 0, 4 * e->nwords, s));
    CK(cudaMemsetAsync(cur, 0, 8 * (V + 1), s));
    CK(cudaStreamSynchronize(s));
    for (uint32_t i = 0; i < n; i++) {
      reached[i] += e->hist_h[i];
      dsum[i] += (uint64_t)(level + 1) * e->hist_h[i];
    }
    std::swap(cur_any, next_any);
    std::swap(cur, next);
    CK(cudaGetLastError());
  }
  CK(cudaMemcpy(e->err_h, e->err_d, 4, cudaMemcpyDeviceToHost));
  RC(check_device_error(e));
  if (out) CK(cudaMemcpy(out, depth_d, 4ull * n * V, cudaMemcpyDeviceToHost));
  if (checks)
    for (uint32_t i = 0; i < n; i++) {
      checks[2 * i] = reached[i];
      checks[2 * i + 1] = dsum[i];
    }
  e->last_algo = -1;  // the engine's value array holds no single result
  return OG_OK;
}

// ------------------------------------------------- batched BFS, level by level

// Opens a session: no slot in use, empty masks and frontier; with `record`
// the 64 x V depth matrix (outside the budget) is kept for og_bfs_batch_fetch.
int bb_begin_impl(og_engine *e, bool record) {
  const uint64_t V = e->V;
  cudaStream_t s = e->s_main;
  e->sb_session = false;  // the masks share the arena with the SSSP rows
  e->bb_session = false;
  CK(cudaMemsetAsync(e->err_d, 0, 16, s));
  CK(cudaMemsetAsync(e->bm[0], 0, 4 * e->nwords, s));
  CK(cudaMemsetAsync(e->bm[1], 0, 4 * e->nwords, s));
  for (int i = 0; i < 3; i++) CK(cudaMemsetAsync(e->bmask[i], 0, 8 * (V + 1), s));
  e->bb_record = record;
  if (record) {
    uint32_t *d = nullptr;
    RC(depth_matrix(e, 64, &d));
    k_fill_u32<<<grid_for(64 * V, e->sms), kThreads, 0, s>>>(d, 64 * V, (uint32_t)(V + 1));
    e->launches++;
  }
  CK(cudaStreamSynchronize(s));
  CK(cudaGetLastError());
  e->bb_level = 1;
  e->bb_par = 0;
  e->bb_used = e->bb_dirty = 0;
  e->bb_session = true;
  return OG_OK;
}

// Seeds slots[i] with srcs[i] at the current level boundary.
int bb_join_impl(og_engine *e, const uint32_t *srcs, const uint32_t *slots, uint32_t n) {
  if (n == 0) return OG_OK;
  if (n > 64) return fail(OG_E_ARG, "%u sources joined, a batch holds 64", n);
  uint64_t cols = 0;
  for (uint32_t i = 0; i < n; i++) {
    if (srcs[i] >= e->V) return fail(OG_E_ARG, "source %u >= V %u", srcs[i], e->V);
    if (slots[i] >= 64) return fail(OG_E_ARG, "slot %u >= 64", slots[i]);
    const uint64_t b = 1ull << slots[i];
    if (cols & b) return fail(OG_E_ARG, "slot %u joined twice", slots[i]);
    if (e->bb_used & b) return fail(OG_E_STATE, "slot %u is still in flight", slots[i]);
    cols |= b;
  }
  const uint64_t V = e->V;
  cudaStream_t s = e->s_main;
  if (cols & e->bb_dirty) {
    k_batch_clear_bits<<<grid_for(V + 1, e->sms), kThreads, 0, s>>>(e->bmask[0], V + 1, cols & e->bb_dirty);
    e->launches++;
    e->bb_dirty &= ~cols;
  }
  if (e->bb_record)
    for (uint32_t i = 0; i < n; i++) {
      k_fill_u32<<<grid_for(V, e->sms), kThreads, 0, s>>>(e->depth_d + (uint64_t)slots[i] * V, V,
                                                         (uint32_t)(V + 1));
      e->launches++;
    }
  for (uint32_t i = 0; i < n; i++) {
    e->bb_off[slots[i]] = e->bb_level - 1;
    e->bb_reached[slots[i]] = 1;  // the source itself, at depth 1
    e->bb_dsum[slots[i]] = 1;
  }
  CK(cudaStreamSynchronize(s));  // the page-locked buffer is rewritten only after the previous upload ran
  memcpy(e->bb_io_h, srcs, 4 * n);
  memcpy(e->bb_io_h + 64, slots, 4 * n);
  memcpy(e->bb_io_h + 128, e->bb_off, 4 * 64);
  CK(cudaMemcpyAsync(e->bb_io_d, e->bb_io_h, 192 * 4, cudaMemcpyHostToDevice, s));
  k_batch_init<<<1, 64, 0, s>>>(e->bb_io_d, n, e->bmask[0], e->bmask[1 + e->bb_par], e->bm[e->bb_par],
                                e->bb_record ? e->depth_d : nullptr, V, nullptr, e->bb_io_d + 64);
  e->launches++;
  CK(cudaGetLastError());
  e->bb_used |= cols;
  return OG_OK;
}

// One level: expands the frontier of every slot in flight.  A slot that
// reached no new vertex has finished: it leaves *pending, its checks are
// final and it may be joined again.
int bb_step_impl(og_engine *e, uint64_t *pending, bool *done, og_stats &st, Timing &tm) {
  const uint64_t V = e->V;
  cudaStream_t s = e->s_main;
  const uint32_t par = e->bb_par;
  uint32_t *cur_any = e->bm[par], *next_any = e->bm[1 - par];
  unsigned long long *visited = e->bmask[0], *cur = e->bmask[1 + par], *next = e->bmask[2 - par];
  uint64_t nl = 0;
  RC(compact_round(e, cur_any, st, tm, &nl));
  if (nl == 0) {  // nothing in flight
    e->bb_dirty |= e->bb_used;
    e->bb_used = 0;
    *pending = 0;
    *done = true;
    return OG_OK;
  }
  st.iterations++;
  st.frontier_sum += nl;
  st.static_vertices += e->counts_h[0].n;
  BatchOp op{visited, cur, next, next_any, e->err_d, e->V};
  auto launch = [&](const LbsArgs &a, auto src, cudaStream_t ls) {
    const unsigned grid = lbs_grid(a.pos_begin, a.pos_end);
    if (grid) {
      k_lbs<decltype(src), BatchOp><<<grid, kThreads, 0, ls>>>(a, src, op);
      e->launches++;
    }
    return (int)OG_OK;
  };
  auto sfn = [&](const LbsArgs &a) { return launch(a, EKU::stat(e), s); };
  auto pfn = [&](const LbsArgs &a0, auto s0, const LbsArgs &a1, auto s1, cudaStream_t ps) {
    const uint64_t n0 = lbs_grid(a0.pos_begin, a0.pos_end), n1 = lbs_grid(a1.pos_begin, a1.pos_end);
    if (n0 + n1 > 0x7fffffffull) return fail(OG_E_STATE, "relax grid too large");
    k_lbs_pair<decltype(s0), decltype(s1), BatchOp><<<(unsigned)(n0 + n1), kThreads, 0, ps>>>(
        a0, s0, a1, s1, op, n0, n0 + n1);
    e->launches++;
    return (int)OG_OK;
  };
  RC((run_regions<EKU>(e, st, tm, MainStream::kIdle, sfn, launch, pfn)));
  CK(cudaMemsetAsync(e->hist_d, 0, 64 * 8, s));
  const uint32_t depth = e->bb_level + 1;  // of the vertices this level reaches, for a source joined at begin
  k_batch_level<<<grid_for(e->nwords, e->sms), kThreads, 0, s>>>(next_any, next, e->nwords, 64, e->hist_d,
                                                               e->bb_record ? e->depth_d : nullptr, V, depth,
                                                               e->bb_io_d + 128);
  e->launches++;
  CK(cudaMemcpyAsync(e->hist_h, e->hist_d, 64 * 8, cudaMemcpyDeviceToHost, s));
  CK(cudaMemsetAsync(cur_any, 0, 4 * e->nwords, s));
  CK(cudaMemsetAsync(cur, 0, 8 * (V + 1), s));
  CK(cudaStreamSynchronize(s));
  CK(cudaGetLastError());
  for (uint32_t i = 0; i < 64; i++) {
    const uint64_t b = 1ull << i;
    if (!(e->bb_used & b)) continue;
    const uint64_t c = e->hist_h[i];
    if (c == 0) {
      e->bb_used &= ~b;
      e->bb_dirty |= b;
    } else {
      e->bb_reached[i] += c;
      e->bb_dsum[i] += (uint64_t)(depth - e->bb_off[i]) * c;
    }
  }
  e->bb_par ^= 1u;
  e->bb_level++;
  *pending = e->bb_used;
  *done = e->bb_used == 0;
  return OG_OK;
}

// ------------------------------------------------------- persistent batched BFS

struct PersistCfg {
  int block, items;
};
// candidate (CTA size, edge positions per thread); the tile is their product
constexpr PersistCfg kPersistConfigs[] = {{256, 8}, {128, 8}, {256, 4}, {512, 4}, {128, 16}};
constexpr int kNumPersistConfigs = 5;

// Bottom-up levels need the graph's reverse edges: only a symmetric graph has
// them in its own records.
uint32_t batch_dopt(const og_engine *e) {
  return e->bfs_direction == OG_BFS_AUTO && e->g->symmetric == 1 ? 1u : 0u;
}

// Configuration of an engine that has not been tuned.  512 x 4 keeps 32 warps
// on an SM where 256 x 8 keeps 16 (128 registers); on small graphs the latter's
// fewer CTAs make cheaper barriers.  64 sources, ms (512 x 4 / 256 x 8): 259 M
// edges 4.27 / 5.41, 31 M edges 0.85 / 0.92, 7.6 M 0.55 / 0.56, 3.7 M 0.49 / 0.48,
// 1.8 M 0.45 / 0.43.  Without bottom-up levels the pushes of every edge are
// most of the work, and the line lies lower: 8.0 M edges 0.64 / 0.79, 3.9 M 0.48 / 0.54,
// 1.0 M 0.35 / 0.37 (one source: 0.35 / 0.39, 0.28 / 0.30, 0.23 / 0.24).
int persist_default(const og_engine *e) { return e->g->E >= (batch_dopt(e) ? 8u << 20 : 1u << 20) ? 3 : 0; }

template <int B, int I>
int launch_persist_cfg(og_engine *e, const PersistArgs &a, cudaStream_t s) {
  auto kern = k_batch_persistent<B, I>;
  int occ = 0;
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, B, 0));
  if (occ < 1) return fail(OG_E_UNSUPPORTED, "persistent kernel does not fit an SM");
  const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)occ * e->sms, kMaxPersistCtas);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(B);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;  // all CTAs co-resident: the grid barriers rely on it
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  CK(cudaLaunchKernelEx(&cfg, kern, a));
  e->launches++;
  return OG_OK;
}

int launch_persist(og_engine *e, int ci, const PersistArgs &a, cudaStream_t s) {
  switch (ci) {
    case 0: return launch_persist_cfg<256, 8>(e, a, s);
    case 1: return launch_persist_cfg<128, 8>(e, a, s);
    case 2: return launch_persist_cfg<256, 4>(e, a, s);
    case 3: return launch_persist_cfg<512, 4>(e, a, s);
    default: return launch_persist_cfg<128, 16>(e, a, s);
  }
}

// Enqueues one whole batch on s_main: clear state, upload the sources from the
// page-locked buffer, seed, run every level in one cooperative kernel, copy
// the per-level counts and the status words back to page-locked memory.
int enqueue_persist(og_engine *e, uint32_t n, int ci, uint32_t *depth_d, uint8_t *depth8_d = nullptr) {
  const uint64_t V = e->V;
  cudaStream_t s = e->s_main;
  for (int i = 0; i < 3; i++) CK(cudaMemsetAsync(e->bmask[i], 0, 8 * (V + 1), s));
  CK(cudaMemsetAsync(e->bm[0], 0, 4 * e->nwords, s));
  CK(cudaMemsetAsync(e->bm[1], 0, 4 * e->nwords, s));
  CK(cudaMemsetAsync(e->bm[2], 0, 4 * e->nwords, s));  // deferred bottom-up vertices
  CK(cudaMemsetAsync(e->smf_d, 0, 8 * 2 * 64, s));
  CK(cudaMemsetAsync(e->hist_d, 0, 8ull * kMaxBatchLevels * 64, s));
  CK(cudaMemsetAsync(e->bar_d, 0, 64, s));
  CK(cudaMemcpyAsync(e->srcs_d, e->srcs_h, 4 * n, cudaMemcpyHostToDevice, s));
  k_batch_init<<<1, 64, 0, s>>>(e->srcs_d, n, e->bmask[0], e->bmask[1], e->bm[0], depth_d, V, depth8_d);
  e->launches++;
  PersistArgs a;
  a.V = e->V;
  a.nwords = e->nwords;
  a.off = e->off_d;
  a.ssrc = EKU::stat(e);
  a.hsrc = EKU::host(e);
  a.static_edges = e->plan.static_edges;
  a.E = e->g->E;
  a.visited = e->bmask[0];
  a.cur = e->bmask[1];
  a.next = e->bmask[2];
  a.cur_any = e->bm[0];
  a.next_any = e->bm[1];
  a.list = e->list_d[0];
  a.pref = e->pref_d[0];
  a.tile_first = e->ptile_d;
  a.list_cap = e->list_cap[0] + e->list_cap[1];
  a.tile_cap = e->ptile_cap;
  a.cta_n = e->cta_n;
  a.cta_e = e->cta_e;
  a.bar = e->bar_d;
  a.hist = e->hist_d;
  a.depth = depth_d;
  a.depth8 = depth8_d;
  a.n_src = n;
  a.err = e->bar_d + 2;
  a.levels = e->bar_d + 3;
  a.stat = (unsigned long long *)(e->bar_d + 4);
  a.smf = e->smf_d;
  a.defer = e->bm[2];
  a.Vs = e->Vs;
  a.dopt = batch_dopt(e);
  a.spin_limit = wait_limit(e->g->E);
  RC(launch_persist(e, ci, a, s));
  CK(cudaMemcpyAsync(e->hist_h, e->hist_d, 8ull * kMaxBatchLevels * 64, cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(e->pmisc_h, e->bar_d, 64, cudaMemcpyDeviceToHost, s));
  return OG_OK;
}

// Captures enqueue_persist for (n, config) as a CUDA graph once and replays it.
int run_persist_graph(og_engine *e, uint32_t n, int ci, bool *used_graph) {
  *used_graph = false;
  const int dopt = (int)batch_dopt(e);
  if (!e->graph_broken &&
      !(e->graph && e->graph_n == n && e->graph_cfg == ci && e->graph_dopt == dopt)) {
    if (e->graph) {
      cudaGraphExecDestroy(e->graph);
      e->graph = nullptr;
    }
    cudaGraph_t gr = nullptr;
    bool ok = cudaStreamBeginCapture(e->s_main, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
    const uint64_t before = e->launches;
    const int rc = ok ? enqueue_persist(e, n, ci, nullptr) : OG_E_CUDA;
    e->launches = before;  // captured, not launched
    if (ok) ok = cudaStreamEndCapture(e->s_main, &gr) == cudaSuccess && rc == OG_OK;
    if (ok) ok = cudaGraphInstantiate(&e->graph, gr, 0) == cudaSuccess;
    if (gr) cudaGraphDestroy(gr);
    if (!ok) {
      cudaGetLastError();
      e->graph = nullptr;
      e->graph_broken = true;  // fall back to direct launches from now on
    } else {
      e->graph_n = n;
      e->graph_cfg = ci;
      e->graph_dopt = dopt;
    }
  }
  if (e->graph) {
    CK(cudaGraphLaunch(e->graph, e->s_main));
    e->launches += 2;  // the seed kernel and the persistent kernel
    *used_graph = true;
    return OG_OK;
  }
  return enqueue_persist(e, n, ci, nullptr);
}

// out: V u32 depths per source (out_bytes 4) or byte depths (out_bytes 1).
// outs (og_bfs_batch_to): source i's V u32 depths go to outs[i] instead.
// The kernel then writes byte depths (an n x V byte matrix, a quarter of the
// u32 one) and each row is widened into its output; if some depth reaches
// 255, the outputs are filled by single-source runs instead.
int run_batch_persist(og_engine *e, const uint32_t *srcs, uint32_t n, void *out, int out_bytes,
                      uint64_t *clamped, uint64_t *checks, og_stats &st, int ci,
                      uint32_t *const *outs = nullptr) {
  const uint64_t V = e->V;
  memcpy(e->srcs_h, srcs, 4 * n);
  uint32_t *depth_d = nullptr;
  uint8_t *depth8_d = nullptr;
  bool graph = false;
  if (out && out_bytes == 4) {
    RC(depth_matrix(e, n, &depth_d));
    k_fill_u32<<<grid_for(n * V, e->sms), kThreads, 0, e->s_main>>>(depth_d, (uint64_t)n * V,
                                                                 (uint32_t)(V + 1));
    e->launches++;
  } else if (out || outs) {  // byte depths, written by the kernel itself (0 = unreached)
    const uint64_t need = (uint64_t)n * V;
    if (need > e->depth8_cap) {
      if (e->depth8_d) cudaFree(e->depth8_d);
      e->depth8_d = nullptr;
      e->depth8_cap = 0;
      CK(cudaMalloc(&e->depth8_d, need));
      e->depth8_cap = need;
    }
    depth8_d = e->depth8_d;
    CK(cudaMemsetAsync(depth8_d, 0, need, e->s_main));
  }
  // events outside any captured graph: they bracket the whole batch on s_main
  CK(cudaEventRecord(e->t_s0, e->s_main));
  if (out || outs) {
    RC(enqueue_persist(e, n, ci, depth_d, depth8_d));
  } else {
    RC(run_persist_graph(e, n, ci, &graph));
  }
  CK(cudaEventRecord(e->t_s1, e->s_main));
  CK(cudaStreamSynchronize(e->s_main));
  CK(cudaGetLastError());
  const uint32_t err = e->pmisc_h[2], levels = e->pmisc_h[3];
  const unsigned long long *stat = (const unsigned long long *)(e->pmisc_h + 4);
  if (err & kErrBarrier) return fail(OG_E_TIMEOUT, "batched BFS grid barrier wait gave up");
  if (err & kErrLevels) return fail(OG_E_STATE, "batched BFS needs more than %u levels", kMaxBatchLevels);
  if (err) return fail(OG_E_DEVICE, "batched BFS kernel reported an out-of-range index (0x%x)", err);
  float ms = 0;
  if (cudaEventElapsedTime(&ms, e->t_s0, e->t_s1) == cudaSuccess) st.ms_static += ms;
  st.iterations = levels;
  st.frontier_sum = stat[0];
  st.edges_static = stat[1] - stat[2];
  st.edges_dynamic = stat[2];
  st.link_bytes = (stat[2] * e->bpe + 7) / 8;  // packed records read over the link
  st.chunks = graph ? 1u : 0u;  // 1: replayed from the captured CUDA graph
  if (checks)
    for (uint32_t i = 0; i < n; i++) {
      uint64_t r = 1, d = 1;
      for (uint32_t L = 1; L <= levels && L < kMaxBatchLevels; L++) {
        const uint64_t c = e->hist_h[(uint64_t)L * 64 + i];
        r += c;
        d += (uint64_t)(L + 1) * c;
      }
      checks[2 * i] = r;
      checks[2 * i + 1] = d;
    }
  if (outs) {
    // entries at depth >= 255 do not fit a byte: single-source runs fill the
    // outputs (no n x V u32 matrix is needed for that)
    uint64_t c = 0;
    for (uint32_t L = 254; L <= levels && L < kMaxBatchLevels; L++)
      for (uint32_t i = 0; i < n; i++) c += e->hist_h[(uint64_t)L * 64 + i];
    if (c) {
      for (uint32_t i = 0; i < n; i++) {
        og_stats one;
        memset(&one, 0, sizeof one);
        RC(run_frontier<EKU>(e, OG_ALGO_BFS, srcs[i], one));
        CK(cudaMemcpyAsync(outs[i], e->value_d, 4ull * V, cudaMemcpyDeviceToHost, e->s_main));
        CK(cudaStreamSynchronize(e->s_main));
      }
      e->last_algo = -1;
      return OG_OK;
    }
    // widened into a V-entry device buffer, then one DMA copy per source
    // (kernel stores straight into page-locked memory measured several
    // times slower than the copy engine)
    uint32_t *stage = nullptr;
    RC(depth_matrix(e, 1, &stage));
    for (uint32_t i = 0; i < n; i++) {
      k_depth_expand<<<grid_for((V + 3) / 4, e->sms), kThreads, 0, e->s_main>>>(depth8_d + (uint64_t)i * V, V,
                                                                                (uint32_t)(V + 1), stage);
      e->launches++;
      CK(cudaMemcpyAsync(outs[i], stage, 4ull * V, cudaMemcpyDeviceToHost, e->s_main));
    }
    CK(cudaGetLastError());
  } else if (out && out_bytes == 4) {
    CK(cudaMemcpyAsync(out, depth_d, 4ull * n * V, cudaMemcpyDeviceToHost, e->s_main));
  } else if (out) {
    CK(cudaMemcpyAsync(out, depth8_d, (uint64_t)n * V, cudaMemcpyDeviceToHost, e->s_main));
    if (clamped) {  // entries at depth L + 1 >= 255, from the per-level counts
      uint64_t c = 0;
      for (uint32_t L = 254; L <= levels && L < kMaxBatchLevels; L++)
        for (uint32_t i = 0; i < n; i++) c += e->hist_h[(uint64_t)L * 64 + i];
      *clamped = c;
    }
  }
  CK(cudaStreamSynchronize(e->s_main));
  e->last_algo = -1;
  return OG_OK;
}

// ------------------------------------------------------------ multi-source SSSP

// k_compact_sb's arguments for region r over the active (scan_wait = false) or
// waiting bitmap.
SbCompactArgs compact_args_sb(og_engine *e, int r, uint32_t *bits, bool scan_wait) {
  const uint32_t vb = r ? e->Vs : 0, ve = r ? e->V : e->Vs;
  SbCompactArgs a{};
  a.counts = e->counts_d + r;
  if (ve <= vb) return a;  // empty region
  a.bits = bits;
  a.wait = e->bm[2];
  a.v_begin = vb;
  a.v_end = ve;
  a.w_begin = vb / 32;
  a.w_end = (uint32_t)(((uint64_t)ve + 31) / 32);
  a.tile_words = compact_tile_words(a.w_end - a.w_begin, std::min(e->lb_tiles - 1, 4u * (uint32_t)e->sms));
  a.ntiles = (a.w_end - a.w_begin + a.tile_words - 1) / a.tile_words;
  a.off = e->off_d;
  a.list = e->list_d[r];
  a.pref = e->pref_d[r];
  a.tile_first = e->tile_d[r];
  a.lmask = e->sb_lmask + (e->list_d[r] - e->list_d[0]);
  a.lb = e->lb[r];
  a.err = e->err_d;
  a.list_cap = e->list_cap[r];
  a.tile_cap = e->tile_cap[r];
  a.pend = e->sb_pend;
  a.dist = e->sb_dist;
  a.ks = e->sb_ks;
  a.thr = e->sb_thr;
  a.scan_wait = scan_wait ? 1u : 0u;
  a.far_key = (unsigned long long *)(e->counts_d + 2) + r;
  a.masks = e->sb_masks;
  a.epoch = e->epoch;
  return a;
}

// Clears the batch: no slot in use, no vertex active or waiting.
int sb_reset(og_engine *e) {
  if (!e->sb_k) return fail(OG_E_STATE, "engine created without OG_CFG_SSSP_BATCH");
  const uint64_t V = e->V;
  cudaStream_t s = e->s_main;
  CK(cudaMemsetAsync(e->err_d, 0, 16, s));
  CK(cudaMemsetAsync(e->bm[0], 0, 4 * e->nwords, s));  // active
  CK(cudaMemsetAsync(e->bm[2], 0, 4 * e->nwords, s));  // waiting
  CK(cudaMemsetAsync(e->sb_pend, 0, 4 * (V + 1), s));
  CK(cudaMemsetAsync(e->sb_masks, 0, 16, s));
  CK(cudaMemsetAsync(e->counts_d + 2, 0, sizeof(Counts), s));  // far keys of earlier queries
  k_fill_u32<<<grid_for((V + 1) * e->sb_ks, e->sms), kThreads, 0, s>>>(e->sb_dist, (V + 1) * e->sb_ks,
                                                                      0xffffffffu);
  e->launches++;
  const uint64_t thr = 1ull + e->sb_delta;
  e->sb_thr = e->sb_delta == 0 || thr > 0xffffffffull ? 0xffffffffu : (uint32_t)thr;
  e->sb_far_min = 0xffffffffu;
  e->sb_advance = false;
  e->sb_dirty = 0;
  e->sb_session = true;
  e->bb_session = false;  // the batch arena now holds SSSP rows
  CK(cudaGetLastError());
  return OG_OK;
}

// Seeds slots[i] with srcs[i] (their columns are reset first when a finished
// source left distances there).  A source may join while others are in
// flight: its distances start below any threshold, so it is expanded every
// round until it has caught up; the result is the same.
int sb_join_impl(og_engine *e, const uint32_t *srcs, const uint32_t *slots, uint32_t n) {
  if (n == 0) return OG_OK;
  if (n > e->sb_k) return fail(OG_E_ARG, "%u sources joined, the engine holds %u", n, e->sb_k);
  uint32_t cols = 0;
  for (uint32_t i = 0; i < n; i++) {
    if (srcs[i] >= e->V) return fail(OG_E_ARG, "source %u >= V %u", srcs[i], e->V);
    if (slots[i] >= e->sb_k) return fail(OG_E_ARG, "slot %u >= %u", slots[i], e->sb_k);
    if (cols & (1u << slots[i])) return fail(OG_E_ARG, "slot %u joined twice", slots[i]);
    cols |= 1u << slots[i];
  }
  cudaStream_t s = e->s_main;
  if (cols & e->sb_dirty) {
    k_sb_clear_cols<<<grid_for(e->V + 1, e->sms), kThreads, 0, s>>>(e->sb_dist, e->V + 1, e->sb_ks,
                                                                   cols & e->sb_dirty);
    e->launches++;
  }
  e->sb_dirty |= cols;
  // the page-locked buffer is rewritten only after the previous upload ran
  CK(cudaStreamSynchronize(s));
  memcpy(e->sb_io_h, srcs, 4 * n);
  memcpy(e->sb_io_h + 32, slots, 4 * n);
  CK(cudaMemcpyAsync(e->sb_io_d, e->sb_io_h, 256, cudaMemcpyHostToDevice, s));
  k_sb_seed<<<1, 32, 0, s>>>(e->sb_io_d, e->sb_io_d + 32, n, e->sb_dist, e->sb_ks, e->sb_pend, e->bm[0],
                             e->V, e->err_d);
  e->launches++;
  CK(cudaGetLastError());
  return OG_OK;
}

// One round: compaction of the active set (or of the waiting set after a
// threshold advance) in both regions, then the relax of the listed near
// pairs.  *pending receives the slots that still have work as of this
// round's compaction (a slot outside it has final distances); *done is set
// when nothing is active or waiting.
template <class K>
int sb_round(og_engine *e, og_stats &st, Timing &tm, uint32_t *pending, bool *done) {
  *done = false;
  if (++e->epoch >= (1u << 30)) {  // epoch wrap: clear the status words and far keys once
    for (int r = 0; r < 2; r++)
      CK(cudaMemsetAsync(e->lb[r].slot, 0, sizeof(ulonglong2) * e->lb_tiles, e->s_main));
    CK(cudaMemsetAsync(e->counts_d + 2, 0, sizeof(Counts), e->s_main));
    e->epoch = 1;
  }
  const bool adv = e->sb_advance;
  uint32_t *bits = adv ? e->bm[2] : e->bm[0];
  // masks[0] is per round; masks[1] (slots waiting) accumulates until the
  // waiting set is scanned again
  CK(cudaMemsetAsync(e->sb_masks, 0, adv ? 8 : 4, e->s_main));
  CK(cudaEventRecord(e->ev_round, e->s_main));
  const CompactPair<SbCompactArgs> p{{compact_args_sb(e, 0, bits, adv), compact_args_sb(e, 1, bits, adv)}};
  RC(launch_compact(e, p, k_compact_sb));
  CK(cudaEventRecord(e->ev_cd, e->s_main));
  RC(compact_wait(e));
  collect_timing(e, tm, &st);
  float ms;
  if (cudaEventElapsedTime(&ms, e->ev_round, e->ev_cd) == cudaSuccess) st.ms_compact += ms;
  RC(check_device_error(e));
  const uint32_t *masks = (const uint32_t *)(e->counts_h + 4);
  *pending = masks[0] | masks[1];
  const uint32_t fm = std::min(far_of(e, 0), far_of(e, 1));
  e->sb_far_min = adv ? fm : std::min(e->sb_far_min, fm);
  const uint64_t n = (uint64_t)e->counts_h[0].n + e->counts_h[1].n;
  if (n == 0) {
    if (e->sb_far_min == 0xffffffffu) {
      *done = true;
      *pending = 0;
      return OG_OK;
    }
    const uint64_t t = (uint64_t)e->sb_far_min + e->sb_delta;
    e->sb_thr = t > 0xffffffffull ? 0xffffffffu : (uint32_t)t;
    e->sb_advance = true;
    return OG_OK;
  }
  e->sb_advance = false;
  st.iterations++;
  st.frontier_sum += n;
  st.static_vertices += e->counts_h[0].n;
  SbOp op{e->list_d[0], e->sb_lmask, e->sb_dist, e->sb_pend, e->bm[0], e->err_d, e->V, e->sb_ks};
  auto launch = [&](const LbsArgs &a, auto src, cudaStream_t ls) {
    const unsigned grid = lbs_grid(a.pos_begin, a.pos_end);
    if (grid) {
      using S = decltype(src);
      if (e->sb_ks == 4) k_sb_relax<S, 4><<<grid, kThreads, 0, ls>>>(a, src, op);
      else if (e->sb_ks == 8) k_sb_relax<S, 8><<<grid, kThreads, 0, ls>>>(a, src, op);
      else if (e->sb_ks == 16) k_sb_relax<S, 16><<<grid, kThreads, 0, ls>>>(a, src, op);
      else k_sb_relax<S, 32><<<grid, kThreads, 0, ls>>>(a, src, op);
      e->launches++;
    }
    return (int)OG_OK;
  };
  auto sfn = [&](const LbsArgs &a) { return launch(a, K::stat(e), e->s_main); };
  auto pfn = [&](const LbsArgs &a0, auto s0, const LbsArgs &a1, auto s1, cudaStream_t ps) {
    const uint64_t n0 = lbs_grid(a0.pos_begin, a0.pos_end), n1 = lbs_grid(a1.pos_begin, a1.pos_end);
    if (n0 + n1 > 0x7fffffffull) return fail(OG_E_STATE, "relax grid too large");
    using S0 = decltype(s0);
    using S1 = decltype(s1);
    const unsigned grid = (unsigned)(n0 + n1);
    if (e->sb_ks == 4) k_sb_relax_pair<S0, S1, 4><<<grid, kThreads, 0, ps>>>(a0, s0, a1, s1, op, n0, n0 + n1);
    else if (e->sb_ks == 8) k_sb_relax_pair<S0, S1, 8><<<grid, kThreads, 0, ps>>>(a0, s0, a1, s1, op, n0, n0 + n1);
    else if (e->sb_ks == 16) k_sb_relax_pair<S0, S1, 16><<<grid, kThreads, 0, ps>>>(a0, s0, a1, s1, op, n0, n0 + n1);
    else k_sb_relax_pair<S0, S1, 32><<<grid, kThreads, 0, ps>>>(a0, s0, a1, s1, op, n0, n0 + n1);
    e->launches++;
    return (int)OG_OK;
  };
  RC((run_regions<K>(e, st, tm, MainStream::kIdle, sfn, launch, pfn)));
  CK(cudaGetLastError());
  return OG_OK;
}

int sb_round_any(og_engine *e, og_stats &st, Timing &tm, uint32_t *pending, bool *done) {
  if (e->wbytes == 1) return sb_round<EK<uint8_t>>(e, st, tm, pending, done);
  if (e->wbytes == 2) return sb_round<EK<uint16_t>>(e, st, tm, pending, done);
  return sb_round<EK<uint32_t>>(e, st, tm, pending, done);
}

// {reached, sum of distances} of every slot in cols, indexed by slot.
int sb_checks_impl(og_engine *e, uint32_t cols, uint64_t *out) {
  cudaStream_t s = e->s_main;
  CK(cudaMemsetAsync(e->sb_ck_d, 0, 16 * kSbMaxSources, s));
  k_sb_checks<<<(unsigned)e->sms * 4, kThreads, 0, s>>>(e->sb_dist, e->V, e->sb_ks, cols, e->sb_ck_d);
  e->launches++;
  CK(cudaMemcpyAsync(e->sb_ck_h, e->sb_ck_d, 16 * kSbMaxSources, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  for (uint32_t i = 0; i < 2 * kSbMaxSources; i++) out[i] = e->sb_ck_h[i];
  return OG_OK;
}

// Distances of slot `slot` into out (V entries of host memory), through the
// engine's value array.
int sb_fetch_impl(og_engine *e, uint32_t slot, uint32_t *out) {
  if (slot >= e->sb_k) return fail(OG_E_ARG, "slot %u >= %u", slot, e->sb_k);
  cudaStream_t s = e->s_main;
  k_sb_column<<<grid_for(e->V, e->sms), kThreads, 0, s>>>(e->sb_dist, e->V, e->sb_ks, slot, e->value_d);
  e->launches++;
  CK(cudaMemcpyAsync(out, e->value_d, 4ull * e->V, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  e->last_algo = -1;  // the value array holds no single-source result
  return OG_OK;
}

int run_sssp_batch(og_engine *e, const uint32_t *srcs, uint32_t n, uint32_t *out, uint64_t *checks,
                   og_stats &st) {
  RC(sb_reset(e));
  uint32_t slots[kSbMaxSources];
  for (uint32_t i = 0; i < n; i++) slots[i] = i;
  RC(sb_join_impl(e, srcs, slots, n));
  Timing tm;
  for (uint64_t r = 0;; r++) {
    uint32_t pending = 0;
    bool done = false;
    RC(sb_round_any(e, st, tm, &pending, &done));
    if (done) break;
    if (r > 16ull * e->V + 64) return fail(OG_E_STATE, "multi-source SSSP did not end after %llu rounds",
                                           (unsigned long long)r);
  }
  CK(cudaStreamSynchronize(e->s_main));
  collect_timing(e, tm, &st);
  CK(cudaMemcpy(e->err_h, e->err_d, 4, cudaMemcpyDeviceToHost));
  RC(check_device_error(e));
  if (checks) {
    uint64_t ck[2 * kSbMaxSources];
    RC(sb_checks_impl(e, (n >= 32 ? 0xffffffffu : (1u << n) - 1u), ck));
    for (uint32_t i = 0; i < 2 * n; i++) checks[i] = ck[i];
  }
  if (out)
    for (uint32_t i = 0; i < n; i++) RC(sb_fetch_impl(e, i, out + (uint64_t)i * e->V));
  e->last_algo = -1;
  return OG_OK;
}

// ------------------------------------------------------------------ PageRank

// Whether region r's compacted list holds every record of the region, so that
// list position q is record base + q.
bool pr_contiguous(const og_engine *e, int r) {
  return e->counts_h[r].total == (r == 0 ? e->plan.static_edges : e->g->E - e->plan.static_edges);
}

template <bool kDense>
int launch_pr_pull(og_engine *e, const LbsArgs &a, SrcP<false> src, const PrArgs &p, cudaStream_t s) {
  const unsigned grid = lbs_grid(a.pos_begin, a.pos_end);
  if (grid) {
    k_pr_pull<kDense><<<grid, kThreads, pr_smem_bytes(kDense, src.bpe), s>>>(a, src, p);
    e->launches++;
  }
  return OG_OK;
}

// Arguments of region r's pull; done: see PrArgs.
PrArgs pr_args(const og_engine *e, int r, const uint32_t *done) {
  PrArgs q{};
  const uint64_t toff = r ? e->tile_cap[0] : 0;  // the dynamic region's tiles follow the static ones
  q.contrib = e->contrib_d;
  q.sum = e->sum_d;
  q.V = e->V;
  q.cont = e->cont_d + toff;
  q.carry = e->carry_d + toff;
  q.carry_idx = e->carry_idx_d + toff;
  q.base = r ? e->plan.static_edges : 0;
  q.nwords = r ? e->g->packed_words : e->g->packed_words_for(e->plan.static_edges);
  q.done = done;
  q.link = (uint32_t)r;
  return q;
}

int launch_pr_pull_pair(og_engine *e, const LbsArgs &a0, SrcP<false> s0, const LbsArgs &a1, SrcP<false> s1,
                        const uint32_t *done, cudaStream_t ps) {
  const uint64_t n0 = lbs_grid(a0.pos_begin, a0.pos_end), n1 = lbs_grid(a1.pos_begin, a1.pos_end);
  if (n0 + n1 > 0x7fffffffull) return fail(OG_E_STATE, "pull grid too large");
  const unsigned n = (unsigned)(n0 + n1);
  if (pr_contiguous(e, 0) && pr_contiguous(e, 1))
    k_pr_pull_pair<true><<<n, kThreads, pr_smem_bytes(true, e->bpe), ps>>>(a0, s0, pr_args(e, 0, done), a1, s1,
                                                                           pr_args(e, 1, done), n0, n);
  else
    k_pr_pull_pair<false><<<n, kThreads, pr_smem_bytes(false, e->bpe), ps>>>(a0, s0, pr_args(e, 0, done), a1, s1,
                                                                             pr_args(e, 1, done), n0, n);
  e->launches++;
  return OG_OK;
}

int launch_pr_fixup(og_engine *e, const uint32_t *done, bool timed = false) {
  PrFixup f[2];
  uint64_t nt[2];
  for (int r = 0; r < 2; r++) {
    const Counts c = e->counts_h[r];
    f[r] = PrFixup{e->list_d[r], e->pref_d[r], c.n, pr_args(e, r, done)};
    f[r].p.t = timed ? e->prl_d->t : nullptr;
    nt[r] = c.n ? (c.total + kTile - 1) / kTile : 0;
  }
  if (nt[0] + nt[1]) {
    k_pr_fixup<<<(unsigned)((nt[0] + nt[1] + kThreads - 1) / kThreads), kThreads, 0, e->s_main>>>(f[0], nt[0], f[1],
                                                                                              nt[1]);
    e->launches++;
  }
  CK(cudaGetLastError());
  return OG_OK;
}

int pr_sums(og_engine *e, og_stats &st, Timing &tm, MainStream main) {
  auto sfn = [&](const LbsArgs &a) {
    return pr_contiguous(e, 0) ? launch_pr_pull<true>(e, a, EKU::stat(e), pr_args(e, 0, nullptr), e->s_main)
                               : launch_pr_pull<false>(e, a, EKU::stat(e), pr_args(e, 0, nullptr), e->s_main);
  };
  auto dfn = [&](const LbsArgs &a, auto src, cudaStream_t ds) {
    if constexpr (std::is_same<decltype(src), SrcU>::value) return (int)OG_OK;  // staged: gfn
    else
      return pr_contiguous(e, 1) ? launch_pr_pull<true>(e, a, src, pr_args(e, 1, nullptr), ds)
                                 : launch_pr_pull<false>(e, a, src, pr_args(e, 1, nullptr), ds);
  };
  auto gfn = [&](const LbsArgs &a) {
    StageRing ring;
    RC(stage_ring(e, &ring, e->s_dyn));
    auto buf = [&](int b) { return SrcP<false>{e->stage_col[b], 32u, 32u, 0u}; };
    k_stage_round_pr<<<2 * lbs_grid(0, a.total), kThreads, pr_smem_bytes(true, 32), e->s_dyn>>>(
        a, EKU::host(e), EKU::stage_dst(e, 0), EKU::stage_dst(e, 1), buf(0), buf(1), e->plan.chunk_edges,
        pr_args(e, 1, nullptr), ring);
    e->launches++;
    return (int)OG_OK;
  };
  auto pfn = [&](const LbsArgs &a0, auto s0, const LbsArgs &a1, auto s1, cudaStream_t ps) {
    return launch_pr_pull_pair(e, a0, s0, a1, s1, nullptr, ps);
  };
  RC((run_regions<EKU>(e, st, tm, main, sfn, dfn, pfn, gfn)));
  return launch_pr_fixup(e, nullptr);
}

int run_pr_delta(og_engine *e, float thresh, int max_rounds, og_stats &st) {
  const uint64_t V = e->V;
  uint32_t *cur = e->bm[0], *next = e->bm[1];
  cudaStream_t s = e->s_main;
  const int g = grid_for(V, e->sms);
  CK(cudaMemsetAsync(e->err_d, 0, 16, s));
  k_pr_init<<<g, kThreads, 0, s>>>(V, (float *)e->value_d, e->contrib_d, e->sum_d, e->outdeg_d,
                                   1.0f);  // PR/OneGraph/GraphMeta.h:354-357
  k_fill_bits<<<g, kThreads, 0, s>>>(cur, e->nwords, V);
  e->launches += 2;
  CK(cudaGetLastError());
  Timing tm;
  // The compaction of the next round is enqueued behind the update, and one wait
  // a round reads its counts and whether anything is active; a wait after
  // the update as well left the device idle twice a round (777777 vertices
  // staged, 17 rounds: 3.33 ms; 3.09 now).
  uint64_t n = 0;
  RC(compact_round(e, cur, st, tm, &n));
  for (int round = 1;; round++) {
    st.iterations++;
    st.frontier_sum += n;
    st.static_vertices += e->counts_h[0].n;
    RC(pr_sums(e, st, tm, MainStream::kIdle));  // the compaction was waited for
    CK(cudaMemsetAsync(e->active_d, 0, 4, s));
    k_pr_update_delta<<<grid_for(e->nwords, e->sms), kThreads, 0, s>>>(
        cur, next, e->nwords, (float *)e->value_d, e->contrib_d, e->sum_d, e->outdeg_d, thresh,
        e->active_d);
    e->launches++;
    if (round == max_rounds) {
      CK(cudaMemcpyAsync(e->err_h, e->err_d, 4, cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
      RC(check_device_error(e));
      break;
    }
    std::swap(cur, next);
    RC(compact_round(e, cur, st, tm, &n));
    if (e->err_h[1] == 0) break;
  }
  CK(cudaStreamSynchronize(s));
  collect_timing(e, tm, &st);
  e->last_algo = OG_ALGO_PR;
  return OG_OK;
}

// The update of every rank and the end of the iteration (k_pr_finish).
int launch_pr_update(og_engine *e, float teleport, float damping, double tol, const uint32_t *done, bool stamp = false) {
  k_pr_update_l1<<<e->part_n, kThreads, 0, e->s_main>>>(e->V, (float *)e->value_d, e->contrib_d, e->sum_d,
                                                        e->outdeg_d, teleport, damping, e->part_d, done);
  k_pr_finish<<<1, kThreads, 0, e->s_main>>>(e->part_d, e->part_n, e->prl_d, tol, stamp);
  e->launches += 2;
  return OG_OK;
}

// Reads the iterations' state back and waits.
int pr_check(og_engine *e, og_stats &st) {
  cudaStream_t s = e->s_main;
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(e->prl_h, e->prl_d, sizeof(PrLoop), cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(e->err_h, e->err_d, 4, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  RC(check_device_error(e));
  st.residual = e->prl_h->residual;
  return OG_OK;
}

int run_pr_l1(og_engine *e, float damping, double tol, int max_iter, og_stats &st) {
  const uint64_t V = e->V;
  uint32_t *cur = e->bm[0];
  cudaStream_t s = e->s_main;
  const int g = grid_for(V, e->sms);
  CK(cudaMemsetAsync(e->err_d, 0, 16, s));
  CK(cudaMemsetAsync(e->prl_d, 0, sizeof(PrLoop), s));
  k_pr_init<<<g, kThreads, 0, s>>>(V, (float *)e->value_d, e->contrib_d, e->sum_d, e->outdeg_d,
                                   (float)(1.0 / (double)V));
  e->launches++;
  k_fill_bits<<<g, kThreads, 0, s>>>(cur, e->nwords, V);
  e->launches++;
  CK(cudaGetLastError());
  Timing tm;
  uint64_t n = 0;
  RC(compact_round(e, cur, st, tm, &n));  // every vertex with in-edges, once
  const float teleport = (float)((1.0 - (double)damping) / (double)V);
  const Counts c0 = e->counts_h[0], c1 = e->counts_h[1];
  if (c1.n == 0 || (e->cfg.flags & OG_CFG_DIRECT)) {
    // Nothing to stage: iterations are launched ahead of the host's check, as
    // many as the last run took, then four at a time; those after the end
    // only read the done flag.  (A wait per iteration cost 25-35 us of each,
    // all of an iteration on a small graph.)
    const uint32_t *done = &e->prl_d->done;
    const LbsArgs a0 = lbs_args(e, 0, 0, c0.total, true, e->plan.static_edges);
    const LbsArgs a1 = lbs_args(e, 1, 0, c1.total, true, e->g->E);
    if (damping != e->pr_hint_damping || tol != e->pr_hint_tol) {
      e->pr_hint = 8;
      e->pr_hint_damping = damping;
      e->pr_hint_tol = tol;
    }
    uint32_t launched = 0, batch = std::max<uint32_t>(1, e->pr_hint);
    while (launched < (uint32_t)max_iter) {
      batch = std::min<uint32_t>(batch, (uint32_t)max_iter - launched);
      if (launched % kPrTimed == 0) {  // behind a wait: the first one is timed
        k_pr_begin<<<1, 1, 0, s>>>(e->prl_d, launched == 0);
        e->launches++;
      }
      for (uint32_t i = 0; i < batch; i++, launched++) {
        if (c0.n && c1.n) {
          RC(launch_pr_pull_pair(e, a0, EKU::stat(e), a1, EKU::host(e), done, s));
        } else if (c0.n || c1.n) {
          const int r = c0.n ? 0 : 1;
          RC((pr_contiguous(e, r)
                  ? launch_pr_pull<true>(e, r ? a1 : a0, r ? EKU::host(e) : EKU::stat(e), pr_args(e, r, done), s)
                  : launch_pr_pull<false>(e, r ? a1 : a0, r ? EKU::host(e) : EKU::stat(e), pr_args(e, r, done), s)));
        }
        RC(launch_pr_fixup(e, done, launched % kPrTimed == 0));
        RC(launch_pr_update(e, teleport, damping, tol, done, i + 1 < batch && (launched + 1) % kPrTimed == 0));
      }
      RC(pr_check(e, st));
      if (e->prl_h->done) break;
      batch = 4;
    }
    const uint64_t its = e->prl_h->iters;
    if (e->prl_h->t[2]) (c1.n ? st.ms_dynamic : st.ms_static) += e->prl_h->t[1] / 1e6 * its / e->prl_h->t[2];
    e->pr_hint = (uint32_t)its;
    st.iterations += (uint32_t)its;
    st.frontier_sum += n * its;
    st.static_vertices += c0.n * its;
    st.edges_static += c0.total * its;
    st.edges_dynamic += c1.total * its;
    st.link_bytes += (c1.total * e->bpe + 7) / 8 * its;
    if (c1.n) st.chunks += (uint32_t)its;
    e->last_algo = OG_ALGO_PR;
    return OG_OK;
  }
  for (int it = 0; it < max_iter; it++) {
    st.iterations++;
    st.frontier_sum += n;
    st.static_vertices += e->counts_h[0].n;
    RC(pr_sums(e, st, tm, MainStream::kBusy));
    RC(launch_pr_update(e, teleport, damping, tol, nullptr));
    RC(pr_check(e, st));
    collect_timing(e, tm, &st);
    if (e->prl_h->done) break;
  }
  e->last_algo = OG_ALGO_PR;
  return OG_OK;
}

// og_pr_l1_push: the graph holds out-edges; sums by scattered atomic adds.
int run_pr_l1_push(og_engine *e, float damping, double tol, int max_iter, og_stats &st) {
  const uint64_t V = e->V;
  uint32_t *cur = e->bm[0];
  cudaStream_t s = e->s_main;
  const int g = grid_for(V, e->sms);
  CK(cudaMemsetAsync(e->err_d, 0, 16, s));
  CK(cudaMemsetAsync(e->prl_d, 0, sizeof(PrLoop), s));
  k_pr_init<<<g, kThreads, 0, s>>>(V, (float *)e->value_d, e->contrib_d, e->sum_d, e->outdeg_d,
                                   (float)(1.0 / (double)V));
  e->launches++;
  k_fill_bits<<<g, kThreads, 0, s>>>(cur, e->nwords, V);
  e->launches++;
  CK(cudaGetLastError());
  Timing tm;
  uint64_t n = 0;
  RC(compact_round(e, cur, st, tm, &n));  // every vertex with out-edges, once
  const float teleport = (float)((1.0 - (double)damping) / (double)V);
  const PushOp op{e->contrib_d, e->sum_d, e->err_d, (uint32_t)V};
  auto launch = [&](const LbsArgs &a, auto src, cudaStream_t ls) {
    const unsigned grid = lbs_grid(a.pos_begin, a.pos_end);
    if (grid) {
      k_lbs<decltype(src), PushOp><<<grid, kThreads, 0, ls>>>(a, src, op);
      e->launches++;
    }
    return (int)OG_OK;
  };
  auto sfn = [&](const LbsArgs &a) { return launch(a, EKU::stat(e), e->s_main); };
  auto pfn = [&](const LbsArgs &a0, auto s0, const LbsArgs &a1, auto s1, cudaStream_t ps) {
    const uint64_t n0 = lbs_grid(a0.pos_begin, a0.pos_end), n1 = lbs_grid(a1.pos_begin, a1.pos_end);
    if (n0 + n1 > 0x7fffffffull) return fail(OG_E_STATE, "push grid too large");
    k_lbs_pair<decltype(s0), decltype(s1), PushOp><<<(unsigned)(n0 + n1), kThreads, 0, ps>>>(a0, s0, a1, s1, op,
                                                                                        n0, n0 + n1);
    e->launches++;
    return (int)OG_OK;
  };
  for (int it = 0; it < max_iter; it++) {
    st.iterations++;
    st.frontier_sum += n;
    st.static_vertices += e->counts_h[0].n;
    CK(cudaMemsetAsync(e->sum_d, 0, 4 * V, s));
    RC((run_regions<EKU>(e, st, tm, MainStream::kBusy, sfn, launch, pfn)));
    RC(launch_pr_update(e, teleport, damping, tol, nullptr));
    RC(pr_check(e, st));
    collect_timing(e, tm, &st);
    if (e->prl_h->done) break;
  }
  e->last_algo = OG_ALGO_PR;
  return OG_OK;
}

double now_ms() {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch())
      .count();
}

int fetch(og_engine *e, void *out) {
  CK(cudaSetDevice(e->dev));
  CK(cudaMemcpyAsync(out, e->value_d, 4ull * e->V, cudaMemcpyDeviceToHost, e->s_main));
  CK(cudaStreamSynchronize(e->s_main));
  return OG_OK;
}

template <class F>
int guarded(F f) {
  try {
    return f();
  } catch (const std::bad_alloc &) {
    return fail(OG_E_NOMEM, "host allocation failed");
  } catch (...) {
    return fail(OG_E_STATE, "unexpected exception");
  }
}

int query_common(og_engine *e, int algo, og_stats *st_out, void *out,
                 int (*body)(og_engine *, og_stats &, void *), void *ctx) {
  if (!e) return fail(OG_E_ARG, "null engine");
  return guarded([&]() -> int {
    clear_error();
    CK(cudaSetDevice(e->dev));
    cudaGetLastError();  // drop a stale error left by an unrelated earlier call
    og_stats st;
    memset(&st, 0, sizeof st);
    e->launches = 0;
    // every query reuses the frontier bitmaps, lists and arena of an open
    // multi-source SSSP or batched BFS session: the session ends here
    e->sb_session = false;
    e->bb_session = false;
    const double t0 = now_ms();
    e->out = out;
    const int rc = body(e, st, ctx);
    const bool left = e->out != nullptr;  // the body has not delivered the result
    e->out = nullptr;
    RC(rc);
    st.launches = e->launches;
    if (left) RC(fetch(e, out));
    st.ms_total = now_ms() - t0;
    if (st_out) *st_out = st;
    (void)algo;
    return OG_OK;
  });
}

}  // namespace

// ====================================================================== C ABI

extern "C" int og_engine_create(og_graph *g, const og_config *cfg, og_engine **out) {
  clear_error();
  if (!g || !out) return fail(OG_E_ARG, "og_engine_create: null argument");
  *out = nullptr;
  og_config c;
  memset(&c, 0, sizeof c);
  if (cfg) c = *cfg;
  return guarded([&]() -> int {
    og_engine *e = new og_engine;
    int rc = create(g, &c, e);
    if (rc != OG_OK) {
      std::string keep = og_last_error();
      destroy(e);
      return fail(rc, "%s", keep.c_str());
    }
    *out = e;
    return OG_OK;
  });
}

extern "C" int og_engine_clone(og_engine *parent, og_engine **out) {
  clear_error();
  if (!parent || !out) return fail(OG_E_ARG, "og_engine_clone: null argument");
  if (parent->parent) return fail(OG_E_ARG, "og_engine_clone: clone a parent engine, not a clone");
  if (parent->frag) return fail(OG_E_UNSUPPORTED, "og_engine_clone: an OG_CFG_REPLACE engine has no clones");
  *out = nullptr;
  return guarded([&]() -> int {
    og_engine *e = new og_engine;
    int rc = clone(parent, e);
    if (rc != OG_OK) {
      std::string keep = og_last_error();
      destroy(e);
      return fail(rc, "%s", keep.c_str());
    }
    *out = e;
    return OG_OK;
  });
}

extern "C" int og_engine_set_param(og_engine *e, int param, double value) {
  if (!e) return fail(OG_E_ARG, "og_engine_set_param: null engine");
  if (param == OG_PARAM_SSSP_DELTA) {
    if (value < 0 || value > 4294967295.0) return fail(OG_E_ARG, "delta out of range");
    e->sssp_delta = (uint32_t)value;
    return OG_OK;
  }
  if (param == OG_PARAM_CC_METHOD) {
    if (value != OG_CC_AUTO && value != OG_CC_LABEL_PROPAGATION && value != OG_CC_UNION_FIND)
      return fail(OG_E_ARG, "unknown CC method %g", value);
    e->cc_method = (uint32_t)value;
    return OG_OK;
  }
  if (param == OG_PARAM_BFS_DIRECTION) {
    if (value != OG_BFS_AUTO && value != OG_BFS_TOP_DOWN) return fail(OG_E_ARG, "unknown BFS direction %g", value);
    e->bfs_direction = (uint32_t)value;
    return OG_OK;
  }
  if (param == OG_PARAM_LEVEL_LOOP) {
    if (value != OG_LOOP_AUTO && value != OG_LOOP_HOST) return fail(OG_E_ARG, "unknown level loop %g", value);
    e->level_loop = (uint32_t)value;
    return OG_OK;
  }
  if (param == OG_PARAM_RELAX_TIMER) {
    if (value != 0 && value != 1) return fail(OG_E_ARG, "relax timer must be 0 or 1, not %g", value);
    e->relax_timer = (uint32_t)value;
    return OG_OK;
  }
  if (param == OG_PARAM_SSSP_BATCH_DELTA) {
    if (value < 0 || value > 4294967295.0) return fail(OG_E_ARG, "delta out of range");
    e->sb_delta = (uint32_t)value;
    return OG_OK;
  }
  if (param == OG_PARAM_FRAGMENT_WORDS) {
    if (!e->frag) return fail(OG_E_STATE, "fragment words: the engine was created without OG_CFG_REPLACE");
    uint32_t fs = 8;
    while (fs <= 20 && (double)(1u << fs) != value) fs++;
    if (fs > 20) return fail(OG_E_ARG, "fragment words must be a power of two in [2^8, 2^20], not %g", value);
    return guarded([&]() -> int {
      CK(cudaSetDevice(e->dev));
      CK(cudaStreamSynchronize(e->s_main));
      CK(cudaStreamSynchronize(e->s_dyn));
      RC(frag_layout(e, fs));  // checks the fit before releasing the old layout
      RC(frag_reset(e));
      CK(cudaStreamSynchronize(e->s_main));
      return (int)OG_OK;
    });
  }
  return fail(OG_E_ARG, "unknown parameter %d", param);
}

extern "C" int og_engine_get_param(const og_engine *e, int param, double *value) {
  if (!e || !value) return fail(OG_E_ARG, "og_engine_get_param: null argument");
  if (param == OG_PARAM_SSSP_DELTA) {
    *value = e->sssp_delta;
    return OG_OK;
  }
  if (param == OG_PARAM_CC_METHOD) {
    *value = e->cc_method;
    return OG_OK;
  }
  if (param == OG_PARAM_BFS_DIRECTION) {
    *value = e->bfs_direction;
    return OG_OK;
  }
  if (param == OG_PARAM_LEVEL_LOOP) {
    *value = e->level_loop;
    return OG_OK;
  }
  if (param == OG_PARAM_RELAX_TIMER) {
    *value = e->relax_timer;
    return OG_OK;
  }
  if (param == OG_PARAM_SSSP_BATCH_DELTA) {
    *value = e->sb_delta;
    return OG_OK;
  }
  if (param == OG_PARAM_FRAGMENT_WORDS) {
    if (!e->frag) return fail(OG_E_STATE, "fragment words: the engine was created without OG_CFG_REPLACE");
    *value = (double)(1u << e->frag->fs);
    return OG_OK;
  }
  return fail(OG_E_ARG, "unknown parameter %d", param);
}

extern "C" int og_engine_fragment_stats(const og_engine *e, og_fragment_stats *out) {
  if (!e || !out) return fail(OG_E_ARG, "og_engine_fragment_stats: null argument");
  if (!e->frag) return fail(OG_E_STATE, "the engine was created without OG_CFG_REPLACE");
  *out = e->frag->st;
  return OG_OK;
}

extern "C" int og_engine_bytes(const og_engine *e, uint64_t *resident, uint64_t *context) {
  if (!e) return fail(OG_E_ARG, "og_engine_bytes: null engine");
  if (resident) *resident = e->parent ? 0 : e->resident_bytes;
  if (context) *context = e->parent ? e->dbytes : e->dbytes - e->resident_bytes;
  return OG_OK;
}

extern "C" int og_engine_plan(const og_engine *e, og_plan *out) {
  if (!e || !out) return fail(OG_E_ARG, "og_engine_plan: null argument");
  *out = e->plan;
  return OG_OK;
}

extern "C" void og_engine_destroy(og_engine *e) { destroy(e); }

extern "C" int og_bfs(og_engine *e, uint32_t src, uint32_t *out_depth, og_stats *st) {
  if (e && src >= e->V) return fail(OG_E_ARG, "source %u >= V %u", src, e->V);
  return query_common(e, OG_ALGO_BFS, st, out_depth, [](og_engine *en, og_stats &s, void *c) {
    const uint32_t src_ = *(uint32_t *)c;
    if (en->frag && en->frag->broken)
      return fail(OG_E_STATE, "the fragment slots were not laid out (a failed OG_PARAM_FRAGMENT_WORDS change)");
    if (en->frag) return run_frontier<EKF<void>>(en, OG_ALGO_BFS, src_, s);
    return rounds_on_device(en) ? run_rounds(en, OG_ALGO_BFS, src_, s) : run_frontier<EKU>(en, OG_ALGO_BFS, src_, s);
  }, &src);
}

extern "C" int og_sssp(og_engine *e, uint32_t src, uint32_t *out_dist, og_stats *st) {
  if (e && src >= e->V) return fail(OG_E_ARG, "source %u >= V %u", src, e->V);
  if (e && e->g->kind != OG_GRAPH_WEIGHTED) return fail(OG_E_UNSUPPORTED, "SSSP needs a weighted graph");
  return query_common(e, OG_ALGO_SSSP, st, out_dist, [](og_engine *en, og_stats &s, void *c) {
    const uint32_t src_ = *(uint32_t *)c;
    if (en->frag && en->frag->broken)
      return fail(OG_E_STATE, "the fragment slots were not laid out (a failed OG_PARAM_FRAGMENT_WORDS change)");
    if (en->frag) return run_frontier<EKF<uint8_t>>(en, OG_ALGO_SSSP, src_, s);
    if (rounds_on_device(en)) return run_rounds(en, OG_ALGO_SSSP, src_, s);
    if (en->wbytes == 1) return run_frontier<EK<uint8_t>>(en, OG_ALGO_SSSP, src_, s);
    if (en->wbytes == 2) return run_frontier<EK<uint16_t>>(en, OG_ALGO_SSSP, src_, s);
    return run_frontier<EK<uint32_t>>(en, OG_ALGO_SSSP, src_, s);
  }, &src);
}

// ------------------------------------------------------------ union-find CC
//
// Symmetric graphs only (the result equals label propagation's there): two
// sampling passes over every vertex's first two edges (read once), compression, the giant
// component picked from 1024 sampled roots, then one edge-balanced pass over
// the edges of the vertices outside it (both regions, interleaved), and a
// final compression.  parent[] lives in value_d and ends as the labels.
int run_cc_uf(og_engine *e, og_stats &st) {
  const uint32_t V = e->V;
  cudaStream_t s = e->s_main;
  const int g = grid_for(V, e->sms);
  uint32_t *par = e->value_d;
  uint32_t jumps = 0;
  auto compress = [&]() -> int {  // every vertex right under its root
    int occ = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_uf_jump, kThreads, 0));
    const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)std::max(1, occ) * e->sms, V / 1024 + 1);
    uint32_t v = V, *p = par;
    RoundsState *state = e->rounds_d + jumps++;  // cleared by k_uf_init
    uint32_t limit = wait_limit(V);
    void *args[5] = {&p, &v, &state, &limit, &e->err_d};
    CK(cudaLaunchCooperativeKernel((const void *)k_uf_jump, dim3(grid), dim3(kThreads), args, 0, s));
    e->launches++;
    return OG_OK;
  };
  unsigned long long *reads = e->sum64_d;  // [0] host records, [1] static records
  uint32_t *roots_d = (uint32_t *)(e->sum64_d + 2);
  constexpr uint32_t kRoots = 1024;
  CK(cudaMemsetAsync(e->err_d, 0, 16, s));
  CK(cudaMemsetAsync(reads, 0, 16, s));
  cudaEvent_t t0 = e->t_d0, t1 = e->ev_dyn_done;
  CK(cudaEventRecord(t0, s));
  uint2 *pend = (uint2 *)e->pref_d[0];  // V + 2 entries of 8 bytes, not in use before the compaction
  k_uf_init<EKU::PSrc><<<g, kThreads, 0, s>>>(e->off_d, V, e->plan.static_edges, EKU::stat(e), EKU::host(e), par, pend,
                                              reads, (uint32_t *)e->rounds_d, kJumps * sizeof(RoundsState) / 4, e->err_d);
  RC(compress());
  k_uf_link<<<g, kThreads, 0, s>>>(pend, V, par, e->err_d);
  RC(compress());
  e->launches += 2;
  st.iterations += 2;
  k_uf_roots<<<(kRoots + kThreads - 1) / kThreads, kThreads, 0, s>>>(par, V, kRoots, roots_d);
  e->launches++;
  CK(cudaEventRecord(t1, s));
  std::vector<uint32_t> roots(kRoots);
  unsigned long long rd[2] = {0, 0};
  CK(cudaMemcpyAsync(roots.data(), roots_d, 4 * kRoots, cudaMemcpyDeviceToHost, s));
  CK(cudaMemcpyAsync(rd, reads, 16, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  float ms = 0;
  if (cudaEventElapsedTime(&ms, t0, t1) == cudaSuccess) st.ms_dynamic += ms;
  st.link_bytes += (rd[0] * e->bpe + 7) / 8;
  st.edges_dynamic += rd[0];
  st.edges_static += rd[1];
  std::sort(roots.begin(), roots.end());
  uint32_t c = roots[0], best = 0;
  for (uint32_t i = 0; i < kRoots;) {
    uint32_t j = i;
    while (j < kRoots && roots[j] == roots[i]) j++;
    if (j - i > best) {
      best = j - i;
      c = roots[i];
    }
    i = j;
  }
  // final pass over the vertices outside c
  uint32_t *cur = e->bm[0];
  k_uf_mark<<<grid_for(e->nwords * 32, e->sms), kThreads, 0, s>>>(e->off_d, par, V, c, cur, e->nwords);
  e->launches++;
  Timing tm;
  uint64_t n = 0;
  RC(compact_round(e, cur, st, tm, &n));
  if (n) {
    st.iterations++;
    st.frontier_sum += n;
    st.static_vertices += e->counts_h[0].n;
    UnionOp op{par, e->err_d, V};
    auto launch = [&](const LbsArgs &a, auto src, cudaStream_t ls) {
      const unsigned grid = lbs_grid(a.pos_begin, a.pos_end);
      if (grid) {
        k_lbs<decltype(src), UnionOp><<<grid, kThreads, 0, ls>>>(a, src, op);
        e->launches++;
      }
      return (int)OG_OK;
    };
    auto sfn = [&](const LbsArgs &a) { return launch(a, EKU::stat(e), e->s_main); };
    auto pfn = [&](const LbsArgs &a0, auto s0, const LbsArgs &a1, auto s1, cudaStream_t ps) {
      const uint64_t n0 = lbs_grid(a0.pos_begin, a0.pos_end), n1 = lbs_grid(a1.pos_begin, a1.pos_end);
      if (n0 + n1 > 0x7fffffffull) return fail(OG_E_STATE, "relax grid too large");
      k_lbs_pair<decltype(s0), decltype(s1), UnionOp><<<(unsigned)(n0 + n1), kThreads, 0, ps>>>(
          a0, s0, a1, s1, op, n0, n0 + n1);
      e->launches++;
      return (int)OG_OK;
    };
    RC((run_regions<EKU>(e, st, tm, MainStream::kIdle, sfn, launch, pfn)));
  }
  if (n) RC(compress());  // nothing was linked since the last compression otherwise
  CK(cudaStreamSynchronize(s));
  collect_timing(e, tm, &st);
  CK(cudaMemcpy(e->err_h, e->err_d, 4, cudaMemcpyDeviceToHost));
  RC(check_device_error(e));
  e->last_algo = OG_ALGO_CC;
  return OG_OK;
}

extern "C" int og_cc(og_engine *e, uint32_t *out_label, og_stats *st) {
  uint32_t dummy = 0;
  return query_common(e, OG_ALGO_CC, st, out_label, [](og_engine *en, og_stats &s, void *) {
    const bool uf = en->cc_method == OG_CC_UNION_FIND ||
                    (en->cc_method == OG_CC_AUTO && en->g->symmetric == 1);
    if (en->cc_method == OG_CC_UNION_FIND && en->g->symmetric != 1)
      return fail(OG_E_ARG, "union-find CC needs a graph known to be symmetric (og_graph_symmetric)");
    if (uf) return run_cc_uf(en, s);
    if (en->frag && en->frag->broken)
      return fail(OG_E_STATE, "the fragment slots were not laid out (a failed OG_PARAM_FRAGMENT_WORDS change)");
    if (en->frag) return run_frontier<EKF<void>>(en, OG_ALGO_CC, 0, s);
    if (rounds_on_device(en)) return run_rounds(en, OG_ALGO_CC, 0, s);
    return run_frontier<EKU>(en, OG_ALGO_CC, 0, s);
  }, &dummy);
}

namespace {
struct PrCtx {
  double a, b;
  int n;
};
}  // namespace

extern "C" int og_pr(og_engine *e, float *out_rank, double threshold, int max_rounds, og_stats *st) {
  if (e && !e->pr_enabled) return fail(OG_E_UNSUPPORTED, "engine has no PageRank state (OG_CFG_PR)");
  PrCtx c{threshold, 0, max_rounds};
  return query_common(e, OG_ALGO_PR, st, out_rank, [](og_engine *en, og_stats &s, void *cx) {
    const PrCtx &p = *(PrCtx *)cx;
    return run_pr_delta(en, (float)p.a, p.n, s);
  }, &c);
}

extern "C" int og_pr_l1(og_engine *e, float *out_rank, double damping, double tol, int max_iter,
                        og_stats *st) {
  if (e && !e->pr_enabled) return fail(OG_E_UNSUPPORTED, "engine has no PageRank state (OG_CFG_PR)");
  if (max_iter <= 0) return fail(OG_E_ARG, "max_iter must be positive");
  PrCtx c{damping, tol, max_iter};
  return query_common(e, OG_ALGO_PR, st, out_rank, [](og_engine *en, og_stats &s, void *cx) {
    const PrCtx &p = *(PrCtx *)cx;
    return run_pr_l1(en, (float)p.a, p.b, p.n, s);
  }, &c);
}

extern "C" int og_pr_l1_push(og_engine *e, float *out_rank, double damping, double tol, int max_iter,
                             og_stats *st) {
  if (e && !e->pr_enabled) return fail(OG_E_UNSUPPORTED, "engine has no PageRank state (OG_CFG_PR)");
  if (max_iter <= 0) return fail(OG_E_ARG, "max_iter must be positive");
  PrCtx c{damping, tol, max_iter};
  return query_common(e, OG_ALGO_PR, st, out_rank, [](og_engine *en, og_stats &s, void *cx) {
    const PrCtx &p = *(PrCtx *)cx;
    return run_pr_l1_push(en, (float)p.a, p.b, p.n, s);
  }, &c);
}

namespace {
struct BatchCtx {
  const uint32_t *srcs;
  uint32_t n;
  uint32_t *out;
  uint64_t *checks;
  int mode;  // 0 persistent (tuned configuration), 1 host-driven levels, 2+k persistent config k
  uint8_t *out8 = nullptr;  // og_bfs_batch_u8
  uint64_t *clamped = nullptr;
  uint32_t *const *outs = nullptr;  // og_bfs_batch_to
};

int batch_body(og_engine *en, og_stats &s, void *cx) {
  const BatchCtx &b = *(BatchCtx *)cx;
  if (b.mode == 1) return run_batch(en, b.srcs, b.n, b.out, b.checks, s);
  const int ci = b.mode >= 2 ? b.mode - 2 : (en->tuned >= 0 ? en->tuned : persist_default(en));
  if (b.out8) return run_batch_persist(en, b.srcs, b.n, b.out8, 1, b.clamped, b.checks, s, ci);
  return run_batch_persist(en, b.srcs, b.n, b.out, 4, nullptr, b.checks, s, ci, b.outs);
}

int batch_checks(og_engine *e, const uint32_t *srcs, int n) {
  if (!e || !srcs) return fail(OG_E_ARG, "og_bfs_batch: null argument");
  if (n < 1 || n > 64) return fail(OG_E_ARG, "og_bfs_batch: %d sources (1..64)", n);
  if (!e->batch_enabled) return fail(OG_E_UNSUPPORTED, "engine created without OG_CFG_BATCH");
  for (int i = 0; i < n; i++)
    if (srcs[i] >= e->V) return fail(OG_E_ARG, "source %u >= V %u", srcs[i], e->V);
  return OG_OK;
}
}  // namespace

extern "C" int og_bfs_batch(og_engine *e, const uint32_t *srcs, int n, uint32_t *out,
                            uint64_t *checks, og_stats *st) {
  RC(batch_checks(e, srcs, n));
  BatchCtx c{srcs, (uint32_t)n, out, checks, (e->cfg.flags & OG_CFG_BATCH_LEVELS) ? 1 : 0};
  return query_common(e, OG_ALGO_BFS, st, nullptr, batch_body, &c);
}

extern "C" int og_bfs_batch_to(og_engine *e, const uint32_t *srcs, int n, uint32_t *const *outs,
                               uint64_t *checks, og_stats *st) {
  RC(batch_checks(e, srcs, n));
  if (!outs) return fail(OG_E_ARG, "og_bfs_batch_to: null output list");
  for (int i = 0; i < n; i++)
    if (!outs[i]) return fail(OG_E_ARG, "og_bfs_batch_to: output %d is null", i);
  if (e->cfg.flags & OG_CFG_BATCH_LEVELS)
    return fail(OG_E_UNSUPPORTED, "og_bfs_batch_to runs the persistent kernel (engine has OG_CFG_BATCH_LEVELS)");
  BatchCtx c{srcs, (uint32_t)n, nullptr, checks, 0};
  c.outs = outs;
  return query_common(e, OG_ALGO_BFS, st, nullptr, batch_body, &c);
}

extern "C" int og_bfs_batch_u8(og_engine *e, const uint32_t *srcs, int n, uint8_t *out, uint64_t *clamped,
                               uint64_t *checks, og_stats *st) {
  RC(batch_checks(e, srcs, n));
  if (!out) return fail(OG_E_ARG, "og_bfs_batch_u8: null output");
  BatchCtx c{srcs, (uint32_t)n, nullptr, checks, 0, out, clamped};
  return query_common(e, OG_ALGO_BFS, st, nullptr, batch_body, &c);
}

extern "C" int og_host_alloc(uint64_t bytes, void **out) {
  clear_error();
  if (!out || bytes == 0) return fail(OG_E_ARG, "og_host_alloc: bad argument");
  *out = nullptr;
  CK(cudaHostAlloc(out, bytes, cudaHostAllocPortable));
  return OG_OK;
}

extern "C" void og_host_free(void *p) {
  if (p) cudaFreeHost(p);
}

extern "C" int og_bfs_batch_tune(og_engine *e, const uint32_t *srcs, int n, int reps,
                                 og_tune_result *res) {
  RC(batch_checks(e, srcs, n));
  if (reps < 1) reps = 1;
  og_tune_result r;
  memset(&r, 0, sizeof r);
  r.configs = kNumPersistConfigs;
  float best = 1e30f;
  for (int i = 0; i < kNumPersistConfigs; i++) {
    r.block[i] = kPersistConfigs[i].block;
    r.items[i] = kPersistConfigs[i].items;
    float tmin = 1e30f;
    for (int k = 0; k <= reps; k++) {  // the first run warms up
      og_stats st{};
      BatchCtx c{srcs, (uint32_t)n, nullptr, nullptr, 2 + i};
      RC(query_common(e, OG_ALGO_BFS, &st, nullptr, batch_body, &c));
      if (k > 0) tmin = std::min(tmin, (float)st.ms_static);
    }
    r.ms[i] = tmin;
    if (tmin < best) {
      best = tmin;
      r.best = i;
    }
  }
  e->tuned = r.best;
  if (res) *res = r;
  return OG_OK;
}

extern "C" int og_bfs_batch_set_config(og_engine *e, int config) {
  if (!e) return fail(OG_E_ARG, "null engine");
  if (config < -1 || config >= kNumPersistConfigs) return fail(OG_E_ARG, "config %d out of range", config);
  e->tuned = config;
  return OG_OK;
}

extern "C" int og_sssp_batch(og_engine *e, const uint32_t *srcs, int n, uint32_t *out, uint64_t *checks,
                             og_stats *st) {
  if (!e || !srcs) return fail(OG_E_ARG, "og_sssp_batch: null argument");
  if (e->g->kind != OG_GRAPH_WEIGHTED) return fail(OG_E_UNSUPPORTED, "SSSP needs a weighted graph");
  if (!e->sb_k) return fail(OG_E_STATE, "engine created without OG_CFG_SSSP_BATCH");
  if (n < 1 || n > (int)e->sb_k) return fail(OG_E_ARG, "n = %d, the engine holds 1..%u sources", n, e->sb_k);
  for (int i = 0; i < n; i++)
    if (srcs[i] >= e->V) return fail(OG_E_ARG, "source %u >= V %u", srcs[i], e->V);
  struct Ctx {
    const uint32_t *srcs;
    uint32_t n;
    uint32_t *out;
    uint64_t *checks;
  } c{srcs, (uint32_t)n, out, checks};
  return query_common(e, OG_ALGO_SSSP, st, nullptr, [](og_engine *en, og_stats &s, void *cx) {
    Ctx &q = *(Ctx *)cx;
    return run_sssp_batch(en, q.srcs, q.n, q.out, q.checks, s);
  }, &c);
}

extern "C" int og_sssp_batch_begin(og_engine *e) {
  if (!e) return fail(OG_E_ARG, "null engine");
  return guarded([&]() -> int {
    clear_error();
    CK(cudaSetDevice(e->dev));
    e->launches = 0;
    return sb_reset(e);
  });
}

extern "C" int og_sssp_batch_join(og_engine *e, const uint32_t *srcs, const uint32_t *slots, int n) {
  if (!e || n < 0 || (n && (!srcs || !slots))) return fail(OG_E_ARG, "og_sssp_batch_join: bad argument");
  if (!e->sb_k) return fail(OG_E_STATE, "engine created without OG_CFG_SSSP_BATCH");
  if (!e->sb_session)
    return fail(OG_E_STATE, "no open multi-source SSSP session: og_sssp_batch_begin first (any other query on "
                            "the engine ends a session)");
  return guarded([&]() -> int {
    clear_error();
    CK(cudaSetDevice(e->dev));
    return sb_join_impl(e, srcs, slots, (uint32_t)n);
  });
}

extern "C" int og_sssp_batch_step(og_engine *e, uint32_t *pending, int *done, og_stats *st) {
  if (!e || !pending || !done) return fail(OG_E_ARG, "og_sssp_batch_step: null argument");
  if (!e->sb_k) return fail(OG_E_STATE, "engine created without OG_CFG_SSSP_BATCH");
  if (!e->sb_session)
    return fail(OG_E_STATE, "no open multi-source SSSP session: og_sssp_batch_begin first (any other query on "
                            "the engine ends a session)");
  return guarded([&]() -> int {
    clear_error();
    CK(cudaSetDevice(e->dev));
    og_stats s;
    memset(&s, 0, sizeof s);
    const uint64_t l0 = e->launches;
    const double t0 = now_ms();
    Timing tm;
    bool d = false;
    RC(sb_round_any(e, s, tm, pending, &d));
    CK(cudaStreamSynchronize(e->s_main));
    collect_timing(e, tm, &s);
    CK(cudaMemcpy(e->err_h, e->err_d, 4, cudaMemcpyDeviceToHost));
    RC(check_device_error(e));
    s.launches = e->launches - l0;
    s.ms_total = now_ms() - t0;
    if (st) *st = s;
    *done = d ? 1 : 0;
    e->last_algo = -1;
    return OG_OK;
  });
}

extern "C" int og_sssp_batch_checks(og_engine *e, uint32_t slots, uint64_t *out) {
  if (!e || !out) return fail(OG_E_ARG, "og_sssp_batch_checks: null argument");
  if (!e->sb_k) return fail(OG_E_STATE, "engine created without OG_CFG_SSSP_BATCH");
  if (!e->sb_session)
    return fail(OG_E_STATE, "no open multi-source SSSP session: og_sssp_batch_begin first (any other query on "
                            "the engine ends a session)");
  return guarded([&]() -> int {
    clear_error();
    CK(cudaSetDevice(e->dev));
    return sb_checks_impl(e, slots, out);
  });
}

extern "C" int og_sssp_batch_fetch(og_engine *e, uint32_t slot, uint32_t *out) {
  if (!e || !out) return fail(OG_E_ARG, "og_sssp_batch_fetch: null argument");
  if (!e->sb_k) return fail(OG_E_STATE, "engine created without OG_CFG_SSSP_BATCH");
  if (!e->sb_session)
    return fail(OG_E_STATE, "no open multi-source SSSP session: og_sssp_batch_begin first (any other query on "
                            "the engine ends a session)");
  return guarded([&]() -> int {
    clear_error();
    CK(cudaSetDevice(e->dev));
    return sb_fetch_impl(e, slot, out);
  });
}

namespace {
int bb_session_ok(og_engine *e) {
  if (!e->batch_enabled) return fail(OG_E_UNSUPPORTED, "engine created without OG_CFG_BATCH");
  if (!e->bb_session)
    return fail(OG_E_STATE, "no open batched BFS session: og_bfs_batch_begin first (any other query on the "
                            "engine ends a session)");
  return OG_OK;
}
}  // namespace

extern "C" int og_bfs_batch_begin(og_engine *e, int record_depths) {
  if (!e) return fail(OG_E_ARG, "null engine");
  if (!e->batch_enabled) return fail(OG_E_UNSUPPORTED, "engine created without OG_CFG_BATCH");
  return guarded([&]() -> int {
    clear_error();
    CK(cudaSetDevice(e->dev));
    cudaGetLastError();
    e->launches = 0;
    e->last_algo = -1;
    return bb_begin_impl(e, record_depths != 0);
  });
}

extern "C" int og_bfs_batch_join(og_engine *e, const uint32_t *srcs, const uint32_t *slots, int n) {
  if (!e || n < 0 || (n && (!srcs || !slots))) return fail(OG_E_ARG, "og_bfs_batch_join: bad argument");
  RC(bb_session_ok(e));
  return guarded([&]() -> int {
    clear_error();
    CK(cudaSetDevice(e->dev));
    return bb_join_impl(e, srcs, slots, (uint32_t)n);
  });
}

extern "C" int og_bfs_batch_step(og_engine *e, uint64_t *pending, int *done, og_stats *st) {
  if (!e || !pending || !done) return fail(OG_E_ARG, "og_bfs_batch_step: null argument");
  RC(bb_session_ok(e));
  return guarded([&]() -> int {
    clear_error();
    CK(cudaSetDevice(e->dev));
    og_stats s;
    memset(&s, 0, sizeof s);
    const uint64_t l0 = e->launches;
    const double t0 = now_ms();
    Timing tm;
    bool d = false;
    RC(bb_step_impl(e, pending, &d, s, tm));
    collect_timing(e, tm, &s);
    CK(cudaMemcpy(e->err_h, e->err_d, 4, cudaMemcpyDeviceToHost));
    RC(check_device_error(e));
    s.launches = e->launches - l0;
    s.ms_total = now_ms() - t0;
    if (st) *st = s;
    *done = d ? 1 : 0;
    e->last_algo = -1;
    return OG_OK;
  });
}

extern "C" int og_bfs_batch_checks(og_engine *e, uint64_t slots, uint64_t *out) {
  if (!e || !out) return fail(OG_E_ARG, "og_bfs_batch_checks: null argument");
  RC(bb_session_ok(e));
  for (uint32_t i = 0; i < 64; i++) {
    const bool on = (slots >> i) & 1u;
    out[2 * i] = on ? e->bb_reached[i] : 0;
    out[2 * i + 1] = on ? e->bb_dsum[i] : 0;
  }
  return OG_OK;
}

extern "C" int og_bfs_batch_fetch(og_engine *e, uint32_t slot, uint32_t *out) {
  if (!e || !out) return fail(OG_E_ARG, "og_bfs_batch_fetch: null argument");
  RC(bb_session_ok(e));
  if (slot >= 64) return fail(OG_E_ARG, "slot %u >= 64", slot);
  if (!e->bb_record) return fail(OG_E_STATE, "the session was opened without depth recording");
  if ((e->bb_used >> slot) & 1u) return fail(OG_E_STATE, "slot %u is still in flight", slot);
  return guarded([&]() -> int {
    clear_error();
    CK(cudaSetDevice(e->dev));
    CK(cudaMemcpyAsync(out, e->depth_d + (uint64_t)slot * e->V, 4ull * e->V, cudaMemcpyDeviceToHost, e->s_main));
    CK(cudaStreamSynchronize(e->s_main));
    return OG_OK;
  });
}

extern "C" int og_result_checksum(og_engine *e, int algo, uint64_t *out) {
  if (!e || !out) return fail(OG_E_ARG, "og_result_checksum: null argument");
  if (e->last_algo != algo) return fail(OG_E_STATE, "no result of algorithm %d on the device", algo);
  return guarded([&]() -> int {
    CK(cudaSetDevice(e->dev));
    const int mode = algo == OG_ALGO_CC ? 1 : (algo == OG_ALGO_PR ? 2 : 0);
    const uint32_t unreached = algo == OG_ALGO_BFS ? e->V + 1 : 0xFFFFFFFFu;
    const uint32_t nb = (uint32_t)e->sms * 8;
    unsigned long long *fin = e->sum64_d + 3ull * nb;
    k_checksum<<<nb, kThreads, 0, e->s_main>>>(e->value_d, e->V, mode, unreached, e->sum64_d);
    k_checksum_final<<<1, kThreads, 0, e->s_main>>>(e->sum64_d, nb, mode, fin);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(e->counts_h, fin, 16, cudaMemcpyDeviceToHost, e->s_main));
    CK(cudaStreamSynchronize(e->s_main));
    memcpy(out, e->counts_h, 16);
    return OG_OK;
  });
}

extern "C" int og_result_fetch(og_engine *e, int algo, void *out) {
  if (!e || !out) return fail(OG_E_ARG, "og_result_fetch: null argument");
  if (e->last_algo != algo) return fail(OG_E_STATE, "no result of algorithm %d on the device", algo);
  return guarded([&]() { return fetch(e, out); });
}

// ------------------------------------------------------- kernel launchers

namespace {

uint32_t compact_tiles(uint32_t v_begin, uint32_t v_end) {
  const uint32_t wb = v_begin / 32, we = (uint32_t)(((uint64_t)v_end + 31) / 32);
  return (we - wb + kWordsPerCompactTile - 1) / kWordsPerCompactTile;
}

// Launches k_compact over [v_begin, v_end) with the given look-back scratch
// (already cleared) and error word.
void compact_launch(const uint32_t *bits, uint32_t v_begin, uint32_t v_end, const uint64_t *off,
                    uint32_t *list, uint64_t *pref, uint64_t list_cap, uint32_t *tile,
                    uint64_t tile_cap, Counts *counts, const Lookback &lb, uint32_t max_tiles, uint32_t *err,
                    cudaStream_t s) {
  CompactArgs a{};
  a.bits = bits;
  a.v_begin = v_begin;
  a.v_end = v_end;
  a.w_begin = v_begin / 32;
  a.w_end = (uint32_t)(((uint64_t)v_end + 31) / 32);
  a.tile_words = compact_tile_words(a.w_end - a.w_begin, max_tiles);
  a.ntiles = (a.w_end - a.w_begin + a.tile_words - 1) / a.tile_words;
  a.off = off;
  a.list = list;
  a.pref = pref;
  a.tile_first = tile;
  a.counts = counts;
  a.lb = lb;
  a.err = err;
  a.list_cap = list_cap;
  a.tile_cap = tile_cap;
  a.value = nullptr;
  a.thr = 0;
  a.split = 0;
  a.far_bits = nullptr;
  a.far_key = nullptr;
  a.clear_bits = nullptr;
  a.epoch = 1;  // the caller's scratch is zeroed before every launch
  k_compact<<<a.ntiles, kThreads, 0, s>>>(CompactPair<CompactArgs>{{a, CompactArgs{}}});
}

// Look-back scratch of `ntiles` tiles: a slot each, then the ticket.
uint64_t lookback_bytes(uint32_t ntiles) { return sizeof(ulonglong2) * (ntiles + 1ull); }

Lookback lookback_carve(void *base, uint32_t ntiles) {
  ulonglong2 *p = (ulonglong2 *)base;
  return Lookback{p, (uint32_t *)(p + ntiles)};
}

// Tiles a stand-alone compaction may use: those of 1024 words, and up to a few
// per SM of smaller ones.
uint32_t compact_max_tiles(uint32_t ntiles1024) { return std::max(ntiles1024, 1024u); }

int compact_args_ok(const uint32_t *bits, uint32_t v_begin, uint32_t v_end, const uint64_t *off,
                    uint32_t *out_list, uint64_t *out_pref, uint64_t list_cap, uint32_t *out_tile,
                    uint64_t tile_cap, og_counts *out_counts) {
  if (!bits || !off || !out_list || !out_pref || !out_tile || !out_counts)
    return fail(OG_E_ARG, "og_k_compact: null pointer");
  if (v_end < v_begin) return fail(OG_E_ARG, "og_k_compact: v_end < v_begin");
  if (list_cap == 0 || tile_cap == 0) return fail(OG_E_ARG, "og_k_compact: zero capacity");
  static_assert(sizeof(og_counts) == sizeof(Counts), "og_counts layout");
  static_assert(kCompactWords == kWordsPerCompactTile, "planner and kernel compaction tiles differ");
  return OG_OK;
}

int compact_status(uint32_t err) {
  if (!err) return OG_OK;
  if (err & kErrLookback) return fail(OG_E_TIMEOUT, "compaction look-back wait gave up");
  return fail(OG_E_DEVICE, "compaction output capacity too small (flags 0x%x)", err);
}

}  // namespace

extern "C" int og_k_compact(const uint32_t *bits, uint32_t v_begin, uint32_t v_end,
                            const uint64_t *off, uint32_t *out_list, uint64_t *out_pref,
                            uint64_t list_cap, uint32_t *out_tile, uint64_t tile_cap,
                            og_counts *out_counts, void *stream) {
  clear_error();
  RC(compact_args_ok(bits, v_begin, v_end, off, out_list, out_pref, list_cap, out_tile, tile_cap,
                     out_counts));
  cudaGetLastError();  // drop a stale error left by an unrelated earlier call
  cudaStream_t s = (cudaStream_t)stream;
  CK(cudaMemsetAsync(out_counts, 0, sizeof(og_counts), s));
  CK(cudaMemsetAsync(out_pref, 0, sizeof(uint64_t), s));
  if (v_end == v_begin) {
    CK(cudaStreamSynchronize(s));
    return OG_OK;
  }
  const uint32_t nt = compact_max_tiles(compact_tiles(v_begin, v_end));
  void *scratch = nullptr;
  CK(cudaMalloc(&scratch, lookback_bytes(nt) + 256));
  char *err_d = (char *)scratch + lookback_bytes(nt);
  Lookback lb = lookback_carve(scratch, nt);
  uint32_t err = 0;
  cudaError_t ce = cudaMemsetAsync(scratch, 0, lookback_bytes(nt) + 256, s);
  if (ce == cudaSuccess) {
    compact_launch(bits, v_begin, v_end, off, out_list, out_pref, list_cap, out_tile, tile_cap,
                   (Counts *)out_counts, lb, nt, (uint32_t *)err_d, s);
    ce = cudaGetLastError();
  }
  if (ce == cudaSuccess) ce = cudaMemcpyAsync(&err, err_d, 4, cudaMemcpyDeviceToHost, s);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
  cudaFree(scratch);
  if (ce != cudaSuccess) return fail(OG_E_CUDA, "og_k_compact: %s", cudaGetErrorString(ce));
  return compact_status(err);
}

// ------------------------------------------------ allocation-free variant
//
// og_k_compact_noalloc runs the same compaction with its look-back scratch in
// a fixed array that is part of the loaded library instead of memory it asks
// the CUDA runtime for.  Limit: kNoAllocTiles compaction tiles of 1024 bitmap
// words, counted from the word holding v_begin: 2^28 vertices when v_begin is
// a multiple of 32, 2^28 - 32 otherwise.  The array (229,700 bytes) lives on
// every device that loads the library, for as long as the process runs.

namespace {

constexpr uint32_t kNoAllocTiles = 8192;
constexpr uint64_t kNoAllocErrOffset = 4 * (kNoAllocTiles + 1ull) + 24ull * kNoAllocTiles + 64;
constexpr uint64_t kNoAllocBytes = kNoAllocErrOffset + 256;

static __device__ __align__(256) unsigned char g_compact_scratch[kNoAllocBytes];

constexpr int kMaxDevices = 64;
std::mutex g_scratch_mu;
void *g_scratch_addr[kMaxDevices] = {};

// Device address of g_compact_scratch on the current device.  Host code may
// not use the symbol itself: on the host it names a stand-in, not device
// memory.  Looked up once per device, the first time that device calls.
int scratch_address(void **out) {
  int dev = 0;
  CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail(OG_E_UNSUPPORTED, "device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (!g_scratch_addr[dev]) {
    void *p = nullptr;
    CK(cudaGetSymbolAddress(&p, g_compact_scratch));
    g_scratch_addr[dev] = p;
  }
  *out = g_scratch_addr[dev];
  return OG_OK;
}

}  // namespace

extern "C" int og_k_compact_noalloc(const uint32_t *bits, uint32_t v_begin, uint32_t v_end,
                                    const uint64_t *off, uint32_t *out_list, uint64_t *out_pref,
                                    uint64_t list_cap, uint32_t *out_tile, uint64_t tile_cap,
                                    og_counts *out_counts, void *stream) {
  clear_error();
  RC(compact_args_ok(bits, v_begin, v_end, off, out_list, out_pref, list_cap, out_tile, tile_cap,
                     out_counts));
  const uint32_t nt = v_end > v_begin ? compact_tiles(v_begin, v_end) : 0;
  if (nt > kNoAllocTiles)
    return fail(OG_E_ARG,
                "og_k_compact_noalloc: range of %u vertices needs %u scratch tiles, the fixed "
                "scratch holds %u (2^28 vertices per call from a multiple of 32)",
                v_end - v_begin, nt, kNoAllocTiles);
  void *base = nullptr;
  RC(scratch_address(&base));
  cudaGetLastError();  // drop a stale error left by an unrelated earlier call
  cudaStream_t s = (cudaStream_t)stream;
  CK(cudaMemsetAsync(out_counts, 0, sizeof(og_counts), s));
  CK(cudaMemsetAsync(out_pref, 0, sizeof(uint64_t), s));
  if (nt == 0) {
    CK(cudaStreamSynchronize(s));
    return OG_OK;
  }
  // the previous call's look-back state and error word must not leak in
  uint32_t *err_d = (uint32_t *)((char *)base + kNoAllocErrOffset);
  const uint32_t mt = compact_max_tiles(nt);
  CK(cudaMemsetAsync(base, 0, lookback_bytes(mt), s));
  CK(cudaMemsetAsync(err_d, 0, sizeof(uint32_t), s));
  compact_launch(bits, v_begin, v_end, off, out_list, out_pref, list_cap, out_tile, tile_cap,
                 (Counts *)out_counts, lookback_carve(base, mt), mt, err_d, s);
  CK(cudaGetLastError());
  uint32_t err = 0;
  CK(cudaMemcpyAsync(&err, err_d, sizeof err, cudaMemcpyDeviceToHost, s));
  CK(cudaStreamSynchronize(s));
  return compact_status(err);
}

extern "C" void og_graph_free(og_graph *g) {
  if (!g) return;
  if (g->registered) {
    cudaHostUnregister(g->packed);
  }
  og::graph_delete(g);
}

// Kernel-level launchers of include/onegraph_kernels.h (same translation unit).
#include "kernel_abi.cuh"
