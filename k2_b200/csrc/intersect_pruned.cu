// Pruned intersection of decoding graphs with a DenseFsaVec: a frame-synchronous
// beam search with a dynamic beam per sequence, followed window by window by a
// backward pass that applies the output beam.  Behaviour follows
// k2/csrc/intersect_dense_pruned.cu:41-1694 (MultiGraphDenseIntersectPruned with
// online_decoding == false) as its CPU build executes it:
//   - the states of frame t+1 are numbered in the order of the first arc of frame t
//     (in [state][arc] order) that reaches them above the cutoff; the reference
//     inserts into a hash sequentially on CPU, so the first arc wins (:1005-1028);
//   - the search beam per sequence moves towards `search_beam`, shrinks while more
//     than max_active states are alive and grows while fewer than min_active are,
//     in the reference's mixed float/double arithmetic (:687-767);
//   - every 20 frames the last 30 are pruned backwards (:164-199, :1373-1634); the
//     backward thread of the reference never changes what the forward pass reads,
//     so the windows are simply run in order.
//
// Sequences are independent, so one team of CTAs (a thread-block cluster of 1 to 16)
// owns one sequence from the first frame to the last: no host round trip per frame,
// no hash (a direct table per sequence, indexed by graph state, plays its role) and
// no kernel waits on another.  States and arcs of all frames of a sequence live in
// one arena, frame after frame, so the pruned result is already in lattice order and
// the output pass is a copy.
//
// A frame expands five to ten times the arcs that end in a state it creates, so the expanded
// arcs live in a scratch region at the far end of the arena and only those that enter a state
// are moved into the frame's part of it.  Every warp of the team owns a contiguous range of
// the frame's arcs: what it counts and lists stays in order, and one exchange of per-warp
// sums numbers a whole frame.
#include <algorithm>
#include <array>
#include <climits>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include <cooperative_groups.h>

#include "common.cuh"
#include "../../include/k2b200.h"

namespace cg = cooperative_groups;

namespace k2b {
namespace {

constexpr int kSearchThreads = 896;  // of 72 registers (with 1024 of 64: 1 to 3 % slower)
constexpr int kWindow = 30;       // frames pruned per backward phase (:171)
constexpr int kWindowShift = 20;  // frames between two phases (:172)

// order-preserving float <-> int (as k2/csrc/utils.h:406-414)
__device__ __forceinline__ int32_t OrderedInt(float f) {
  int32_t i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float OrderedFloat(int32_t i) {
  return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff);
}

struct SearchArgs {
  // graphs
  const int32_t *a_rs1, *a_rs2;
  const Arc *a_arcs;
  int32_t a_stride;  // 1: one graph per sequence, 0: one graph shared by all
  int32_t a_states;  // states of all graphs together
  // dense scores
  const float *scores;
  int32_t rows, cols;
  const int32_t *b_rs;
  int32_t num_seqs, T;  // T = rows of the longest sequence
  float search_beam, output_beam, min_active, max_active;
  int32_t allow_partial;
  // arenas, [num_seqs] slices of cap_s (+1) and cap_a elements
  int64_t cap_s, cap_a;
  int32_t *st_astate, *st_fwd, *st_arc0, *st_new, *st_cnt;
  float *st_bwd;
  int32_t *arc_aidx, *arc_dest;
  float *arc_ll, *arc_end;
  uint8_t *arc_deg;           // scratch: arcs leaving a new state, 255 for that many or more
  unsigned long long *winner;  // [num_seqs * a_states] (shared) or [a_states]
  int32_t *frame_s0, *frame_a0;  // [num_seqs][T + 2]
  int32_t *warp_first;         // [num_seqs][kTeamWarps]
  int32_t *seq_out;           // [num_seqs][kSeqOut]: states, arcs, extra final state, status,
                              // most states of a frame, most arcs leaving one
};

constexpr int kSeqOut = 6;
enum : int32_t { kSeqOk = 0, kSeqOverflow = 1, kSeqManyFinal = 2 };

// The CTAs that work on one sequence: a thread-block cluster (of one CTA when there are
// enough sequences to fill the GPU).  Arena data is exchanged through global memory,
// ordered by the cluster barrier; sums and maxima through distributed shared memory: a CTA
// writes its own to every CTA before the barrier and all are read locally behind it.  The CTAs
// of a cluster are always co-resident, so the barrier cannot wait for an unscheduled CTA.
constexpr int kMaxTeam = 16;
constexpr int kWarps = kSearchThreads / 32;
constexpr int kTeamWarps = kMaxTeam * kWarps;
// Slots of exchanged values.  A slot is written again only when another exchange, with its
// barrier, lies in between: the two slots of the thread scans alternate.
enum : int32_t { kSlotMax = 0, kSlotNew, kSlotKept, kSlotWindow, kSlotScan, kSlots = kSlotScan + 2 };
constexpr int kMaxRow = 8192;        // columns of a row of scores that are kept in shared memory
constexpr int kMarkWords = 8192;     // words of the set of new states: 2^18 graph states
struct Shared {
  unsigned long long cta_val[kSlots][kMaxTeam];
  unsigned long long warp_val[kWarps], warp_ex[kWarps];
  int4 rec[kWarps][32];                           // per warp: the states whose arcs it walks
  int32_t wbest[kWarps][32];
  uint32_t mark[kMarkWords];
  float row[kMaxRow];
  int32_t most_states, most_arcs;
};

struct Team {
  cg::cluster_group cluster;
  Shared *sh;
  int32_t rank, size;     // this CTA within the cluster
  int32_t tid, threads;   // this thread within the team
  int32_t warp, warps;    // this warp within the team
  mutable int32_t phase;

  __device__ Team(Shared *shared) : cluster(cg::this_cluster()), sh(shared), phase(0) {
    rank = (int32_t)cluster.block_rank();
    size = (int32_t)cluster.num_blocks();
    tid = rank * kSearchThreads + (int32_t)threadIdx.x;
    threads = size * kSearchThreads;
    warp = tid >> 5;
    warps = threads >> 5;
  }
  __device__ __forceinline__ void Sync() const {
    if (size == 1) __syncthreads(); else cluster.sync();
  }

  // Exclusive sum over the warps of the team of a value per warp (two counts packed into
  // it must not overflow); the barrier inside also orders the global writes made before.
  __device__ unsigned long long ScanWarps(int32_t slot, unsigned long long v,
                                          unsigned long long *total) const {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sh->warp_val[w] = v;
    __syncthreads();
    if (w == 0) {
      const unsigned long long x = lane < kWarps ? sh->warp_val[lane] : 0ull;
      unsigned long long inc = x;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long o = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += o;
      }
      if (lane < kWarps) sh->warp_ex[lane] = inc - x;
      const unsigned long long all = __shfl_sync(0xffffffffu, inc, 31);
      if (lane < size) *cluster.map_shared_rank(&sh->cta_val[slot][rank], lane) = all;
    }
    Sync();
    unsigned long long before = 0, sum = 0;
    for (int32_t r = 0; r < size; ++r) {
      const unsigned long long x = sh->cta_val[slot][r];
      sum += x;
      if (r < rank) before += x;
    }
    *total = sum;
    return before + sh->warp_ex[w];
  }

  // exclusive scan of one count per team thread; every thread gets the total
  __device__ int32_t Scan(int32_t v, int32_t *total) const {
    const int lane = threadIdx.x & 31;
    int32_t inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int32_t o = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += o;
    }
    unsigned long long all;
    const unsigned long long base = ScanWarps(
        kSlotScan + (phase++ & 1), (unsigned long long)__shfl_sync(0xffffffffu, inc, 31), &all);
    *total = (int32_t)all;
    return (int32_t)base + inc - v;
  }

  // largest value of the team; the barrier inside orders global writes likewise
  __device__ int32_t Max(int32_t v) const {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    v = __reduce_max_sync(0xffffffffu, v);
    if (lane == 0) sh->warp_val[w] = (unsigned long long)(uint32_t)v;
    __syncthreads();
    if (w == 0) {
      v = __reduce_max_sync(0xffffffffu, (int32_t)(uint32_t)sh->warp_val[lane < kWarps ? lane : 0]);
      if (lane < size)
        *cluster.map_shared_rank(&sh->cta_val[kSlotMax][rank], lane) = (unsigned long long)(uint32_t)v;
    }
    Sync();
    v = (int32_t)(uint32_t)sh->cta_val[kSlotMax][0];
    for (int32_t r = 1; r < size; ++r) v = max(v, (int32_t)(uint32_t)sh->cta_val[kSlotMax][r]);
    return v;
  }

  // true when `v` is non-zero on any thread of the team
  __device__ bool Any(int32_t v) const {
    int32_t total;
    Scan(v != 0, &total);
    return total != 0;
  }
};

// Views of one sequence's slices of the arenas.
struct SeqView {
  int32_t *st_astate, *st_fwd, *st_arc0, *st_new, *st_cnt;
  float *st_bwd;
  int32_t *arc_aidx, *arc_dest;
  float *arc_ll, *arc_end;
  uint8_t *arc_deg;
  unsigned long long *winner;
  int32_t *frame_s0, *frame_a0, *warp_first;
};

__device__ __forceinline__ SeqView ViewOf(const SearchArgs &g, int32_t seq) {
  SeqView v;
  const int64_t so = (int64_t)seq * (g.cap_s + 1), ao = (int64_t)seq * g.cap_a;
  v.st_astate = g.st_astate + so;
  v.st_fwd = g.st_fwd + so;
  v.st_arc0 = g.st_arc0 + so;
  v.st_new = g.st_new + so;
  v.st_cnt = g.st_cnt + so;
  v.st_bwd = g.st_bwd + so;
  v.arc_aidx = g.arc_aidx + ao;
  v.arc_dest = g.arc_dest + ao;
  v.arc_ll = g.arc_ll + ao;
  v.arc_end = g.arc_end + ao;
  v.arc_deg = g.arc_deg + ao;
  // the reference's hash key is dest_state_idx01 + seq * stride with the stride 0
  // for per-sequence graphs (:118-127): the same index works for a direct table
  v.winner = g.winner + (g.a_stride ? 0 : (int64_t)seq * g.a_states);
  v.frame_s0 = g.frame_s0 + (int64_t)seq * (g.T + 2);
  v.frame_a0 = g.frame_a0 + (int64_t)seq * (g.T + 2);
  v.warp_first = g.warp_first + (int64_t)seq * kTeamWarps;
  return v;
}

// The search beam and the cutoff of frame t (:718-766).  `dyn` is the beam carried
// from the previous frame; products with the literals 0.8, 0.2 and 1.25 are double
// products in the reference and are rounded to float on assignment.
__device__ float NextBeam(float dyn, float best, int32_t active, int32_t t, int32_t final_t,
                          const SearchArgs &g, float *cutoff) {
  const float default_beam = g.search_beam, max_active = g.max_active,
              min_active = g.min_active;
  float cur_min = min_active;
  if (t + 5 >= final_t) cur_min = fmaxf(min_active, max_active / 2);
  if ((float)active <= max_active) {
    if ((float)active >= cur_min || active == 0) {
      dyn = (float)(0.8 * (double)dyn + 0.2 * (double)default_beam);
    } else {
      if (dyn < default_beam) dyn = default_beam;
      dyn = (float)((double)dyn * 1.25);
    }
  } else if (t + 5 < final_t) {
    if (dyn > default_beam) dyn = default_beam;
    dyn = (float)((double)dyn * 0.8);
  }
  if (t == final_t - 1) dyn = 1.0e+10f;
  *cutoff = best - dyn;
  return dyn;
}

// Groups of 32 arcs whose loads a warp issues together.  A thread has 72 registers: four groups
// spill three times as much as two and gain nothing (54.1 and 54.8 ms for decoding 32 x 500 frames
// with output, best path and scores).
constexpr int kExpand = 2;

// Entries of the direct table that replaces the reference's hash: the frame in the
// high word, so that entries of earlier frames lose against any entry of this frame
// and the table never needs clearing; in the low word either an arc (a smaller arc
// index gives a larger value, so atomicMax keeps the first arc) or, with the top bit
// set, the number of the state that arc created.
__device__ __forceinline__ unsigned long long ArcEntry(int32_t t, int32_t q) {
  return ((unsigned long long)(uint32_t)(t + 1) << 32) | (uint32_t)(0x7fffffff - q);
}
__device__ __forceinline__ unsigned long long StateEntry(int32_t t, int32_t j) {
  return ((unsigned long long)(uint32_t)(t + 1) << 32) | 0x80000000u | (uint32_t)j;
}

// Arcs that a warp of the team owns of a frame that expands `na`: a multiple of 32.
__device__ __forceinline__ int32_t ArcsPerWarp(int32_t na, const Team &tm) {
  return ((na + tm.warps - 1) / tm.warps + 31) & ~31;
}
// State k expands arcs [f, f + deg): where a warp's range starts among them, the warp's walk
// over the states starts at k.
__device__ __forceinline__ void SetWarpFirst(const SeqView &v, int32_t per_warp, int32_t k,
                                             int32_t f, int32_t deg) {
  for (int32_t w = (f + per_warp - 1) / per_warp; w * per_warp < f + deg; ++w) v.warp_first[w] = k;
}

// A graph arc, read-only for the whole launch.
__device__ __forceinline__ Arc LoadArc(const Arc *p) {
  const int4 x = __ldg(reinterpret_cast<const int4 *>(p));
  Arc arc;
  arc.src = x.x;
  arc.dest = x.y;
  arc.label = x.z;
  arc.score = __int_as_float(x.w);
  return arc;
}

// The scores of a row of the dense matrix into shared memory, when they fit.
__device__ __forceinline__ void StageRow(const SearchArgs &g, const Team &tm, int32_t row) {
  if (g.cols > kMaxRow || row >= g.rows) return;
  const float *in = g.scores + (int64_t)row * g.cols;
  for (int32_t c = threadIdx.x; c < g.cols; c += kSearchThreads) tm.sh->row[c] = in[c];
}

// 32 states whose arcs a warp walks as one flat range: lane j has state j's first arc f
// (`end` where there is no state) and what goes with its arcs.  The records of the states
// that have arcs go to shared memory in order; the record of arc p is found by counting the
// states that start at or before it.
struct ArcWalk {
  const int4 *rec;
  int32_t f;
  bool nonempty;
  int32_t before;  // states with arcs that start before the next group

  __device__ __forceinline__ void Begin(int4 *recs, int32_t first, int32_t next, int4 mine,
                                        int32_t start) {
    const int lane = threadIdx.x & 31;
    f = first;
    nonempty = next > first;
    const uint32_t ne = __ballot_sync(0xffffffffu, nonempty);
    __syncwarp();  // the records before have been read
    if (nonempty) recs[__popc(ne & ((1u << lane) - 1u))] = mine;
    __syncwarp();
    rec = recs;
    before = __popc(__ballot_sync(0xffffffffu, nonempty && f < start));
  }
  // index of the record of arc pb + lane; groups of 32 arcs in order
  __device__ __forceinline__ int32_t Next(int32_t pb) {
    const int lane = threadIdx.x & 31;
    const uint32_t x = (uint32_t)(f - pb);
    const uint32_t starts =
        __reduce_or_sync(0xffffffffu, nonempty && x < 32u ? 1u << x : 0u);
    const int32_t r = before + __popc(starts & (0xffffffffu >> (31 - lane))) - 1;
    before += __popc(starts);
    return r;
  }
};

// One step of the search (GetArcs + PropagateForward, :778-1153): expands the na arcs leaving the
// ns states of frame t at [s0, s0 + ns) - where each state's arcs start among them (st_cnt)
// and where the warps start (warp_first) was laid out when the states were created - creates
// the states of frame t + 1 behind them, with the layout of their arcs, and appends the arcs
// that enter one of them to the arena at a0.  Returns false when an arena is full.
// *ns_next / *na_next: states of frame t + 1 and the arcs leaving them; *kept: arcs appended.
// beam: the search beam carried from frame to frame, the same in every thread.
//
// Bound by latency and by the rate of scattered accesses (about one per cycle and SM): the only
// ones left per expanded arc are its graph arc, which arrives with its neighbours', and its
// score, in shared memory; the table of states is looked at for the arcs above the cutoff, and
// for those whose destination is in the set of new states.
__device__ bool SearchStep(const SearchArgs &g, const SeqView &v, const Team &tm, int32_t seq,
                           int32_t t, int32_t final_t, int32_t row0, int32_t s0, int32_t ns,
                           int32_t a0, int32_t na, float *beam, int32_t *ns_next,
                           int32_t *na_next, int32_t *kept) {
  Shared *sh = tm.sh;
  constexpr unsigned kAll = 0xffffffffu;
  const float kNegInf = -INFINITY;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  *ns_next = *na_next = *kept = 0;
  if (na == 0) {  // no arc: the search of this sequence has ended, but for its beam
    float cutoff;
    *beam = NextBeam(*beam, kNegInf, ns, t, final_t, g, &cutoff);
    for (int32_t k = tm.tid; k < ns; k += tm.threads) v.st_arc0[s0 + k] = a0;
    __syncthreads();
    StageRow(g, tm, row0 + t + 1);
    tm.Sync();
    return true;
  }
  const int64_t raw = (g.cap_a - na) & ~(int64_t)31;  // the expanded arcs' place
  // (and as much again in front of it, for the warps' lists, until the arcs that are kept
  // go there)
  if (g.cap_a < na || raw - a0 < na) return false;
  int32_t *r_aidx = v.arc_aidx + raw, *r_dest = v.arc_dest + raw;
  float *r_ll = v.arc_ll + raw, *r_end = v.arc_end + raw;
  const int32_t per_warp = ArcsPerWarp(na, tm);
  const int32_t lo = (int32_t)min((int64_t)tm.warp * per_warp, (int64_t)na);
  const int32_t hi = min(lo + per_warp, na);
  int32_t *list = reinterpret_cast<int32_t *>(v.arc_end) + a0 + lo;
  int32_t *list_dest = v.arc_aidx + a0 + lo;  // until step 6
  uint8_t *list_deg = v.arc_deg + raw + lo;

  // graph of this sequence: its final state, for allow_partial (:861-871)
  const int32_t gi = seq * g.a_stride;
  const int32_t g_start = g.a_rs1[gi], g_final = g.a_rs1[gi + 1] - 1;
  bool redirect = false;
  if (g.allow_partial && t == final_t - 1) {
    // is there any arc with label -1 among the arcs expanded on this frame (:839-857)
    int32_t has = 0;
    for (int32_t k = tm.tid; k < ns; k += tm.threads) {
      const int32_t as = v.st_astate[s0 + k];
      for (int32_t a = g.a_rs2[as]; a < g.a_rs2[as + 1]; ++a) has |= (g.a_arcs[a].label == -1);
    }
    redirect = !tm.Any(has);
  }

  // ---- 1. arcs: scores, destination (as a graph state) and the best end score (:858-905).
  // (a row past the end is only asked for by a malformed graph whose arcs with
  // label -1 do not end in a state without arcs)
  const bool row_ok = row0 + t < g.rows;
  const bool staged = g.cols <= kMaxRow;
  const float *row = staged ? sh->row : g.scores + (int64_t)(row_ok ? row0 + t : 0) * g.cols;
  float best = kNegInf;
  const int32_t k_first = lo < hi ? v.warp_first[tm.warp] : ns;
  for (int32_t k0 = k_first; k0 < ns; k0 += 32) {
    const int32_t k = k0 + lane;
    int32_t f = na, fwd = 0, ga0 = 0;
    if (k < ns) {
      f = v.st_cnt[s0 + k];
      fwd = v.st_fwd[s0 + k];
      ga0 = __ldg(g.a_rs2 + v.st_astate[s0 + k]);
    }
    int32_t next = __shfl_down_sync(kAll, f, 1);
    if (lane == 31) next = k + 1 < ns ? v.st_cnt[s0 + k + 1] : na;
    const int32_t start = max(lo, __shfl_sync(kAll, f, 0));
    const int32_t chunk_end = __shfl_sync(kAll, next, 31), stop = min(hi, chunk_end);
    ArcWalk walk;
    walk.Begin(sh->rec[warp], f, next, make_int4(ga0 - f, fwd, 0, 0), start);
    for (int32_t pb = start; pb < stop; pb += 32 * kExpand) {
      int2 rec[kExpand];
      Arc arc[kExpand];
#pragma unroll
      for (int i = 0; i < kExpand; ++i) {
        const int32_t p = pb + 32 * i + lane, r = walk.Next(pb + 32 * i);
        if (p < stop) {
          rec[i] = *reinterpret_cast<const int2 *>(&sh->rec[warp][r]);
          arc[i] = LoadArc(g.a_arcs + (p + rec[i].x));
        }
      }
#pragma unroll
      for (int i = 0; i < kExpand; ++i) {
        const int32_t p = pb + 32 * i + lane;
        if (p < stop) {
          const uint32_t col = (uint32_t)(arc[i].label + 1);
          float acoustic = (row_ok && col < (uint32_t)g.cols) ? row[col] : kNegInf;
          int32_t dest = g_start + arc[i].dest;
          if (redirect) {
            dest = g_final;
            acoustic = 0.0f;
          }
          const float ll = acoustic + arc[i].score;
          const float end = OrderedFloat(rec[i].y) + ll;
          r_aidx[p] = p + rec[i].x;
          r_ll[p] = ll;
          r_dest[p] = dest;
          r_end[p] = end;
          best = fmaxf(best, end);  // (not a NaN)
        }
      }
    }
    if (chunk_end >= hi) break;
  }
  {
    float cutoff_f;
    *beam = NextBeam(*beam, OrderedFloat(tm.Max(OrderedInt(best))), ns, t, final_t, g, &cutoff_f);
    // ---- 2. first arc above the cutoff into every destination state (:1005-1028); the warp
    // lists those arcs and where they go.
    int32_t above = 0;
    for (int32_t pb = lo; pb < hi; pb += 32 * kExpand) {
      float end[kExpand];
      int32_t dest[kExpand];
#pragma unroll
      for (int i = 0; i < kExpand; ++i) {
        const int32_t p = pb + 32 * i + lane;
        end[i] = p < hi ? r_end[p] : kNegInf;
      }
#pragma unroll
      for (int i = 0; i < kExpand; ++i)
        dest[i] = end[i] > cutoff_f ? r_dest[pb + 32 * i + lane] : -1;
#pragma unroll
      for (int i = 0; i < kExpand; ++i) {
        const int32_t p = pb + 32 * i + lane;
        const bool in = dest[i] >= 0;
        const uint32_t m = __ballot_sync(kAll, in);
        if (in) {
          const int32_t at = above + __popc(m & ((1u << lane) - 1u));
          list[at] = p;
          list_dest[at] = dest[i];
          atomicMax(&v.winner[dest[i]], ArcEntry(t, p));
        }
        above += __popc(m);
      }
    }
    StageRow(g, tm, row0 + t + 1);  // this frame's has been used
    tm.Sync();
    // ---- 3. which of them created their destination state, and the arcs that leave it
    int32_t won = 0;
    uint32_t degs = 0;
    for (int32_t i0 = 0; i0 < above; i0 += 64) {
      int32_t p[2], d[2], deg[2];
      unsigned long long w[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int32_t at = i0 + 32 * i + lane;
        p[i] = at < above ? list[at] : 0;
        d[i] = at < above ? list_dest[at] : -1;
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        w[i] = 0;
        deg[i] = 0;
        if (d[i] >= 0) {
          w[i] = v.winner[d[i]];
          deg[i] = g.a_rs2[d[i] + 1] - g.a_rs2[d[i]];
        }
      }
      __syncwarp();  // the lists are rewritten from their start
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const bool in = d[i] >= 0 && w[i] == ArcEntry(t, p[i]);
        const uint32_t m = __ballot_sync(kAll, in);
        if (in) {
          const int32_t at = won + __popc(m & ((1u << lane) - 1u));
          list_dest[at] = d[i];
          list_deg[at] = (uint8_t)min(deg[i], 255);
          degs += (uint32_t)deg[i];
        }
        won += __popc(m);
      }
    }
    degs = __reduce_add_sync(kAll, degs);
    // ---- 4. the new states in the order of their arcs (:1031-1100), and the layout of the
    // arcs that will leave them
    const int32_t s1 = s0 + ns;
    unsigned long long total;
    const unsigned long long base = tm.ScanWarps(
        kSlotNew, (unsigned long long)(uint32_t)won | ((unsigned long long)degs << 32), &total);
    const int32_t nn = (int32_t)(total & 0xffffffffu), na1 = (int32_t)(total >> 32);
    if ((int64_t)s1 + nn > g.cap_s || na1 < 0) return false;
    const int32_t per_warp1 = max(ArcsPerWarp(na1, tm), 32);
    int32_t j = (int32_t)(base & 0xffffffffu), first = (int32_t)(base >> 32);
    for (int32_t i0 = 0; i0 < won; i0 += 32) {
      const bool in = i0 + lane < won;
      const int32_t d = in ? list_dest[i0 + lane] : 0;
      int32_t deg = in ? list_deg[i0 + lane] : 0;
      if (deg == 255) deg = g.a_rs2[d + 1] - g.a_rs2[d];
      int32_t inc = deg;
#pragma unroll
      for (int x = 1; x < 32; x <<= 1) {
        const int32_t o = __shfl_up_sync(kAll, inc, x);
        if (lane >= x) inc += o;
      }
      if (in) {
        const int32_t k = j + lane, f = first + inc - deg;
        v.st_astate[s1 + k] = d;
        v.st_fwd[s1 + k] = OrderedInt(kNegInf);
        v.st_cnt[s1 + k] = f;
        v.winner[d] = StateEntry(t, k);
        SetWarpFirst(v, per_warp1, k, f, deg);
      }
      j += 32;
      first += __shfl_sync(kAll, inc, 31);
    }
    for (int32_t x = threadIdx.x; x < kMarkWords; x += kSearchThreads) sh->mark[x] = 0u;
    tm.Sync();
    *ns_next = nn;
    *na_next = na1;
  }
  // ---- 5. the arcs that enter a new state, with its number, and the best score into every
  // new state; an arc below the cutoff still enters a state that another arc created
  // (:1103-1138).  The set of the new states (of all that share a bit of it, in graphs of
  // more than 2^18 states) keeps the others from looking at the table.
  const int32_t s1 = s0 + ns;
  for (int32_t k = threadIdx.x; k < *ns_next; k += kSearchThreads) {
    const uint32_t d = (uint32_t)v.st_astate[s1 + k] & (kMarkWords * 32 - 1);
    atomicOr(&sh->mark[d >> 5], 1u << (d & 31));
  }
  __syncthreads();
  int32_t entering = 0;
  for (int32_t pb = lo; pb < hi; pb += 32 * kExpand) {
    int32_t dest[kExpand];
    float end[kExpand];
    unsigned long long w[kExpand];
#pragma unroll
    for (int i = 0; i < kExpand; ++i) {
      const int32_t p = pb + 32 * i + lane;
      dest[i] = p < hi ? r_dest[p] : -1;
    }
#pragma unroll
    for (int i = 0; i < kExpand; ++i) {
      const uint32_t x = (uint32_t)dest[i] & (kMarkWords * 32 - 1);
      w[i] = 0ull;
      end[i] = 0.0f;
      if (dest[i] >= 0 && (sh->mark[x >> 5] >> (x & 31) & 1u)) {
        w[i] = v.winner[dest[i]];
        end[i] = r_end[pb + 32 * i + lane];
      }
    }
    __syncwarp();  // (the start of r_end takes the groups' masks, that of r_dest the numbers)
#pragma unroll
    for (int i = 0; i < kExpand; ++i) {
      const int32_t p = pb + 32 * i + lane;
      const bool in = (uint32_t)(w[i] >> 32) == (uint32_t)(t + 1) && (w[i] & 0x80000000u);
      const uint32_t m = __ballot_sync(kAll, in);
      if (in) {
        const int32_t idx1 = (int32_t)(w[i] & 0x7fffffffu);
        atomicMax(&v.st_fwd[s1 + idx1], OrderedInt(end[i]));
        const int32_t at = entering + __popc(m & ((1u << lane) - 1u));
        list[at] = p;
        r_dest[lo + at] = idx1;
      }
      if (lane == 0 && pb + 32 * i < hi && hi - lo > 1) {
        const int32_t group = (pb - lo) / 32 + i;
        r_end[lo + 2 * group] = __uint_as_float(m);
        r_end[lo + 2 * group + 1] = __int_as_float(entering);
      }
      entering += __popc(m);
    }
  }
  // ---- 6. these arcs go to the arena.  A state's first one is the first of its arcs' among
  // them: a warp sees to the states whose arcs start behind its own first arc, up to the
  // start of the next warp's (the first warp: also at its first arc).
  unsigned long long total;
  const int32_t base = a0 + (int32_t)tm.ScanWarps(kSlotKept, (unsigned long long)entering, &total);
  *kept = (int32_t)total;
  if (a0 + (int64_t)total > raw) return false;
  for (int32_t i0 = 0; i0 < entering; i0 += 64) {
    int32_t p[2], idx1[2], aidx[2];
    float ll[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int32_t at = i0 + 32 * i + lane;
      p[i] = at < entering ? list[at] : -1;
      idx1[i] = at < entering ? r_dest[lo + at] : 0;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (p[i] >= 0) {
        aidx[i] = r_aidx[p[i]];
        ll[i] = r_ll[p[i]];
      }
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (p[i] >= 0) {
        const int32_t at = base + i0 + 32 * i + lane;
        v.arc_aidx[at] = aidx[i];
        v.arc_ll[at] = ll[i];
        v.arc_dest[at] = idx1[i];
      }
  }
  if (lo < hi) {
    for (int32_t k0 = tm.warp == 0 ? 0 : k_first; k0 < ns; k0 += 32) {
      const int32_t k = k0 + lane;
      const int32_t f = k < ns ? v.st_cnt[s0 + k] : 0x7fffffff;
      if ((f > lo || tm.warp == 0) && f <= hi) {
        int32_t before = entering;
        if (f == lo) {
          before = 0;
        } else if (f < hi) {
          const int32_t group = (f - lo) >> 5;
          const uint32_t m = __float_as_uint(r_end[lo + 2 * group]);
          before = __float_as_int(r_end[lo + 2 * group + 1]) +
                   __popc(m & ((1u << ((f - lo) & 31)) - 1u));
        }
        v.st_arc0[s0 + k] = base + before;
      }
      if (__any_sync(kAll, f > hi)) break;
    }
  }
  tm.Sync();  // the scratch region is free again
  return true;
}

// Backward pass over frames [begin, end) with the output beam (PruneTimeRange,
// :1373-1634, with SetBackwardProbsFinal :1170-1193 and PropagateBackward
// :1239-1346), then compaction of those frames.  On entry the frames up to `end` are complete
// and frame `end` has its states and the layout of the arcs that will leave them, but no
// arcs; on return *s_top / *a_top are the ends of the arenas and the frame tables are
// updated.  Returns false when an arena has no room for the survivors twice.
//
// One barrier per frame for the backward pass, which leaves a record per 32 states of a frame (a
// unit): which survive and how many arcs, later the first of either.  One exchange of sums
// numbers the survivors of all frames; where a state goes follows from its unit's record.  They
// are gathered at the far end of the arenas and copied back.
__device__ bool PruneWindow(const SearchArgs &g, const SeqView &v, const Team &tm, int32_t seq,
                            int32_t begin, int32_t end, int32_t *s_top, int32_t *a_top,
                            bool keep_all_at_begin = true) {
  Shared *sh = tm.sh;
  constexpr unsigned kAll = 0xffffffffu;
  const float kNegInf = -INFINITY;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t gi = seq * g.a_stride;
  const int32_t g_final = g.a_rs1[gi + 1] - 1;  // last state of this sequence's graph
  const float beam = g.output_beam;
  tm.Sync();  // the frame tables
  const int32_t sb = v.frame_s0[begin], ab = v.frame_a0[begin];
  const int32_t se = v.frame_s0[end], ns_end = *s_top - se;

  // frame `end`: backward score = -forward score, whatever the state
  for (int32_t k = tm.tid; k < ns_end; k += tm.threads) {
    const float fwd = OrderedFloat(v.st_fwd[se + k]);
    v.st_bwd[se + k] = (fwd - fwd == 0.0f) ? -fwd : kNegInf;
  }
  tm.Sync();

  // the records of the units: a frame may leave one number unused behind its own, so that
  // unit 0 of a frame follows from its first state
  const int32_t num_units = (se - sb) / 32 + (end - begin);
  if (3 * (int64_t)num_units > g.cap_s) return false;
  int32_t *unit_mask = v.st_new, *unit_s = v.st_new + num_units, *unit_a = unit_s + num_units;
  auto unit0 = [&](int32_t t, int32_t s0) { return (s0 - sb) / 32 + (t - begin); };

  // ---- backwards: arc survival (the destination of another arc becomes -1) and the backward
  // score of every state
  {
    int32_t s0 = v.frame_s0[end], a1 = v.frame_a0[end];
    for (int32_t t = end - 1; t >= begin; --t) {
      const int32_t s_next = s0, a_next = a1;
      s0 = v.frame_s0[t];
      a1 = v.frame_a0[t];
      const int32_t ns = s_next - s0, u0 = unit0(t, s0), units = unit0(t + 1, s_next) - u0;
      const bool keep_all = t == begin && keep_all_at_begin;
      for (int32_t u = tm.warp; u < units; u += tm.warps) {
        const int32_t k = u * 32 + lane;
        int32_t f = a_next, fwd = 0, as = 0;
        if (k < ns) {
          f = v.st_arc0[s0 + k];
          fwd = v.st_fwd[s0 + k];
          as = v.st_astate[s0 + k];
        }
        int32_t next = __shfl_down_sync(kAll, f, 1);
        if (lane == 31) next = k + 1 < ns ? v.st_arc0[s0 + k + 1] : a_next;
        sh->wbest[warp][lane] = OrderedInt(kNegInf);
        const int32_t start = __shfl_sync(kAll, f, 0), stop = __shfl_sync(kAll, next, 31);
        int32_t arcs = 0;
        ArcWalk walk;
        walk.Begin(sh->rec[warp], f, next, make_int4(fwd, lane, 0, 0), start);
        for (int32_t pb = start; pb < stop; pb += 64) {
          int32_t d[2];
          float ll[2], nb[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int32_t p = pb + 32 * i + lane;
            d[i] = p < stop ? v.arc_dest[p] : -1;
            ll[i] = p < stop ? v.arc_ll[p] : 0.0f;
          }
#pragma unroll
          for (int i = 0; i < 2; ++i) nb[i] = d[i] >= 0 ? v.st_bwd[s_next + d[i]] : kNegInf;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int32_t p = pb + 32 * i + lane, r = walk.Next(pb + 32 * i);
            bool keep = false;
            if (p < stop) {
              const int2 rec = *reinterpret_cast<const int2 *>(&sh->rec[warp][r]);
              const float bl = ll[i] + nb[i];
              keep = d[i] >= 0 && bl + OrderedFloat(rec.x) >= -beam;
              if (keep) atomicMax(&sh->wbest[warp][rec.y], OrderedInt(bl));
              else v.arc_dest[p] = -1;
            }
            arcs += __popc(__ballot_sync(kAll, keep));
          }
        }
        __syncwarp();
        const float bwd =
            as == g_final ? -OrderedFloat(fwd) : OrderedFloat(sh->wbest[warp][lane]);
        if (k < ns) v.st_bwd[s0 + k] = bwd;
        const uint32_t kept = __ballot_sync(kAll, k < ns && (bwd != kNegInf || keep_all));
        if (lane == 0) {
          unit_mask[u0 + u] = (int32_t)kept;
          unit_a[u0 + u] = arcs;
        }
        __syncwarp();
      }
      tm.Sync();
    }
  }

  // ---- new numbers: the first surviving state and arc of every unit
  int32_t ks, ka;
  {
    const int32_t per_warp = (num_units + tm.warps - 1) / tm.warps;
    const int32_t lo = min(tm.warp * per_warp, num_units), hi = min(lo + per_warp, num_units);
    uint32_t states = 0, arcs = 0;
    for (int32_t i = lo + lane; i < hi; i += 32) {
      states += __popc(unit_mask[i]);
      arcs += (uint32_t)unit_a[i];
    }
    states = __reduce_add_sync(kAll, states);
    arcs = __reduce_add_sync(kAll, arcs);
    unsigned long long total;
    const unsigned long long base = tm.ScanWarps(
        kSlotWindow, (unsigned long long)states | ((unsigned long long)arcs << 32), &total);
    ks = (int32_t)(total & 0xffffffffu);
    ka = (int32_t)(total >> 32);
    int32_t j = sb + (int32_t)(base & 0xffffffffu), q = ab + (int32_t)(base >> 32);
    for (int32_t i0 = lo; i0 < hi; i0 += 32) {
      const bool in = i0 + lane < hi;
      const int32_t n = in ? __popc(unit_mask[i0 + lane]) : 0, a = in ? unit_a[i0 + lane] : 0;
      int32_t inc_s = n, inc_a = a;
#pragma unroll
      for (int x = 1; x < 32; x <<= 1) {
        const int32_t o = __shfl_up_sync(kAll, inc_s, x), p = __shfl_up_sync(kAll, inc_a, x);
        if (lane >= x) {
          inc_s += o;
          inc_a += p;
        }
      }
      if (in) {
        unit_s[i0 + lane] = j + inc_s - n;
        unit_a[i0 + lane] = q + inc_a - a;
      }
      j += __shfl_sync(kAll, inc_s, 31);
      q += __shfl_sync(kAll, inc_a, 31);
    }
  }
  // where the survivors are gathered: the states (and those of frame `end`) and the arcs
  const int64_t hold_s = g.cap_s - ks - ns_end, hold_a = g.cap_a - ka;
  if (hold_s < *s_top || hold_a < *a_top) return false;
  for (int32_t k = tm.tid; k < ns_end; k += tm.threads) {
    const int64_t h = hold_s + ks + k;
    v.st_astate[h] = v.st_astate[se + k];
    v.st_fwd[h] = v.st_fwd[se + k];
    v.st_cnt[h] = v.st_cnt[se + k];
  }
  tm.Sync();
  // ---- the survivors: the arcs of a unit are consecutive, and so are the places they go to
  {
    int32_t turn = 0;  // units so far, modulo the warps
    int32_t s1 = sb, a1 = ab;
    for (int32_t t = begin; t < end; ++t) {
      const int32_t s0 = s1;
      s1 = v.frame_s0[t + 1];
      a1 = v.frame_a0[t + 1];
      const int32_t ns = s1 - s0, u0 = unit0(t, s0), u1 = unit0(t + 1, s1), units = u1 - u0;
      const bool last = t + 1 == end;  // the states of frame `end` keep their numbers
      const int32_t new_s1 = last ? 0 : unit_s[u1];
      int32_t u = tm.warp - turn;
      if (u < 0) u += tm.warps;
      for (; u < units; u += tm.warps) {
        const int32_t k = u * 32 + lane;
        int32_t f = a1, as = 0, fwd = 0;
        if (k < ns) {
          f = v.st_arc0[s0 + k];
          as = v.st_astate[s0 + k];
          fwd = v.st_fwd[s0 + k];
        }
        const uint32_t kept = (uint32_t)unit_mask[u0 + u];
        const int32_t first_s = unit_s[u0 + u];
        int32_t q = unit_a[u0 + u];
        const int32_t start = __shfl_sync(kAll, f, 0);
        const int32_t stop = u * 32 + 32 < ns ? v.st_arc0[s0 + u * 32 + 32] : a1;
        int32_t my_q = q;
        for (int32_t pb = start; pb < stop; pb += 64) {
          int32_t d[2], aidx[2];
          float ll[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int32_t p = pb + 32 * i + lane;
            d[i] = p < stop ? v.arc_dest[p] : -1;
          }
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (d[i] >= 0) {
              aidx[i] = v.arc_aidx[pb + 32 * i + lane];
              ll[i] = v.arc_ll[pb + 32 * i + lane];
              if (!last) {
                const int32_t to = u1 + (d[i] >> 5);
                d[i] = unit_s[to] - new_s1 +
                       __popc((uint32_t)unit_mask[to] & ((1u << (d[i] & 31)) - 1u));
              }
            }
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint32_t m = __ballot_sync(kAll, d[i] >= 0);
            if (d[i] >= 0) {
              const int64_t at = hold_a + (q - ab) + __popc(m & ((1u << lane) - 1u));
              v.arc_aidx[at] = aidx[i];
              v.arc_ll[at] = ll[i];
              v.arc_dest[at] = d[i];
            }
            const uint32_t x = (uint32_t)(f - (pb + 32 * i));
            if (x < 32u) my_q = q + __popc(m & ((1u << x) - 1u));
            q += __popc(m);
          }
        }
        if (f >= stop) my_q = q;  // no arc at or behind its place
        if ((kept >> lane) & 1u) {
          const int64_t h = hold_s + (first_s - sb) + __popc(kept & ((1u << lane) - 1u));
          v.st_astate[h] = as;
          v.st_fwd[h] = fwd;
          v.st_arc0[h] = my_q;
        }
      }
      turn = (turn + units) % tm.warps;
    }
  }
  tm.Sync();
  // ---- back to their places
#pragma unroll 4
  for (int32_t k = tm.tid; k < ka; k += tm.threads) {
    v.arc_aidx[ab + k] = v.arc_aidx[hold_a + k];
    v.arc_ll[ab + k] = v.arc_ll[hold_a + k];
    v.arc_dest[ab + k] = v.arc_dest[hold_a + k];
  }
#pragma unroll 4
  for (int32_t k = tm.tid; k < ks + ns_end; k += tm.threads) {
    v.st_astate[sb + k] = v.st_astate[hold_s + k];
    v.st_fwd[sb + k] = v.st_fwd[hold_s + k];
    if (k < ks) v.st_arc0[sb + k] = v.st_arc0[hold_s + k];
    else v.st_cnt[sb + k] = v.st_cnt[hold_s + k];
  }
  // (a frame's first unit follows from its old first state, which nobody else reads now)
  for (int32_t t = begin + tm.tid; t <= end; t += tm.threads) {
    const int32_t u = t < end ? unit0(t, v.frame_s0[t]) : 0;
    v.frame_s0[t] = t < end ? unit_s[u] : sb + ks;
    v.frame_a0[t] = t < end ? unit_a[u] : ab + ka;
  }
  tm.Sync();
  *s_top = sb + ks + ns_end;
  *a_top = ab + ka;
  return true;
}

// Largest frame of the finished lattice of a sequence, in states and in arcs, over frames
// 0 .. frames - 1; by the first CTA of the team, its thread 0 has the result in sh.
__device__ void LargestFrame(const SeqView &v, const Team &tm, int32_t frames) {
  Shared *sh = tm.sh;
  if (tm.rank != 0) return;
  if (threadIdx.x == 0) sh->most_states = sh->most_arcs = 0;
  __syncthreads();
  int32_t ms = 0, ma = 0;
  for (int32_t t = threadIdx.x; t < frames; t += kSearchThreads) {
    ms = max(ms, v.frame_s0[t + 1] - v.frame_s0[t]);
    ma = max(ma, v.frame_a0[t + 1] - v.frame_a0[t]);
  }
  if (ms) atomicMax(&sh->most_states, ms);
  if (ma) atomicMax(&sh->most_arcs, ma);
  __syncthreads();
}

// One team per sequence: all frames of the search with the pruning windows in the
// reference's schedule (:164-199, :213-229).
__global__ void __launch_bounds__(kSearchThreads, 1) PrunedSearch(const SearchArgs g) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Shared &sh = *reinterpret_cast<Shared *>(smem_raw);
  const Team tm(&sh);
  const int32_t seq = blockIdx.x / tm.size;
  const SeqView v = ViewOf(g, seq);
  const int32_t row0 = g.b_rs[seq], final_t = g.b_rs[seq + 1] - row0;
  const int32_t T = g.T;
  const int32_t gi = seq * g.a_stride;
  const int32_t g_start = g.a_rs1[gi], g_states = g.a_rs1[gi + 1] - g_start;
  float beam = g.search_beam;

  // frame 0: the start state, if the graph has states (:435-472)
  int32_t s0 = 0, ns = g_states > 0 ? 1 : 0, a0 = 0;
  int32_t na = ns ? g.a_rs2[g_start + 1] - g.a_rs2[g_start] : 0;
  if (tm.tid == 0) {
    v.frame_s0[0] = 0;
    v.frame_a0[0] = 0;
    if (ns) {
      v.st_astate[0] = g_start;
      v.st_fwd[0] = OrderedInt(0.0f);
      v.st_cnt[0] = 0;
      if (na) SetWarpFirst(v, ArcsPerWarp(na, tm), 0, 0, na);
    }
  }
  StageRow(g, tm, row0);
  tm.Sync();
  int32_t s_top = ns, a_top = 0;
  int32_t status = kSeqOk;
  int32_t next_end = kWindowShift;  // end of the next pruning window
  for (int32_t t = 0; t < T; ++t) {
    int32_t nn, na1, kept;
    if (!SearchStep(g, v, tm, seq, t, final_t, row0, s0, ns, a0, na, &beam, &nn, &na1, &kept)) {
      status = kSeqOverflow;
      break;
    }
    s0 += ns;
    a0 += kept;
    ns = nn;
    na = na1;
    s_top = s0 + ns;
    a_top = a0;
    if (tm.tid == 0) {  // published by the next barrier
      v.frame_s0[t + 1] = s0;
      v.frame_a0[t + 1] = a0;
    }
    const int32_t this_end = next_end >= T ? T : next_end;
    if (t == this_end - 1) {
      const int32_t begin = max(0, next_end - kWindow);
      if (!PruneWindow(g, v, tm, seq, begin, this_end, &s_top, &a_top)) {
        status = kSeqOverflow;
        break;
      }
      s0 = s_top - ns;
      a0 = a_top;
      next_end += kWindowShift;
    }
  }
  if (status == kSeqOk) {  // the states of the last frame have no arcs in the lattice
    for (int32_t k = tm.tid; k < ns; k += tm.threads) v.st_arc0[s0 + k] = a_top;
  }
  if (status == kSeqOk) {
    if (tm.tid == 0) {
      v.frame_s0[T + 1] = s_top;  // frame T has no arcs
      v.frame_a0[T + 1] = a_top;
      v.st_arc0[s_top] = a_top;
    }
    tm.Sync();
    LargestFrame(v, tm, T + 1);
  }
  if (tm.tid == 0) {
    int32_t extra = 0;
    if (status == kSeqOk) {
      // a sequence whose final state did not survive still gets a final state, so
      // that the result is a valid FSA (:519-547)
      const int32_t at_final = v.frame_s0[final_t + 1] - v.frame_s0[final_t];
      if (at_final > 1) status = kSeqManyFinal;
      extra = (g_states > 0) * (1 - min(at_final, 1));
    }
    int32_t *o = g.seq_out + kSeqOut * seq;
    o[0] = s_top + extra;
    o[1] = a_top;
    o[2] = extra;
    o[3] = status;
    o[4] = sh.most_states;
    o[5] = sh.most_arcs;
  }
  tm.Sync();  // no CTA leaves while another may still read its shared memory
}

struct FormatArgs {
  SearchArgs g;
  const int32_t *out_rs1;   // [num_seqs + 1] first lattice state of every sequence
  const int32_t *arc_base;  // [num_seqs + 1] first lattice arc of every sequence
  int32_t *row_ids1, *row_splits2, *row_ids2;
  Arc *arcs;
  int32_t *arc_map_a, *arc_map_b;
  int32_t *level_offsets, *level_splits;
};

// Lattice of one (sequence, frame) (FormatOutput, :474-657): the arenas are already in
// [sequence][frame][state][arc] order.  gridDim.z CTAs share the states of a frame: with one
// of them the widest frame (10^4 states) took as long as all others together.
__global__ void FormatPruned(const FormatArgs f) {
  const SearchArgs &g = f.g;
  const int32_t seq = blockIdx.y, t = blockIdx.x;  // t in [0, T + 1]
  const SeqView v = ViewOf(g, seq);
  const int32_t row0 = g.b_rs[seq], final_t = g.b_rs[seq + 1] - row0;
  const int32_t sb = f.out_rs1[seq], ab = f.arc_base[seq];
  const int32_t s0 = v.frame_s0[t], s1 = v.frame_s0[t + 1];
  const bool first = blockIdx.z == 0;
  if (f.level_splits != nullptr && first && threadIdx.x == 0) {
    f.level_splits[(int64_t)seq * (g.T + 2) + t] = sb + s0;
    if (t == 0) f.level_offsets[seq] = seq * (g.T + 2);
    if (seq == g.num_seqs - 1 && t == g.T + 1) {
      f.level_offsets[g.num_seqs] = g.num_seqs * (g.T + 2);
      f.level_splits[(int64_t)g.num_seqs * (g.T + 2)] = f.out_rs1[g.num_seqs];
    }
  }
  if (t == g.T + 1) {
    // the extra final state, if any, and the end of the row_splits
    if (first && threadIdx.x == 0) {
      const int32_t extra = g.seq_out[kSeqOut * seq + 2];
      if (extra) {
        f.row_ids1[sb + s0] = seq;
        f.row_splits2[sb + s0] = ab + g.seq_out[kSeqOut * seq + 1];
      }
      if (seq == g.num_seqs - 1) f.row_splits2[f.out_rs1[g.num_seqs]] = f.arc_base[g.num_seqs];
    }
    return;
  }
  const int32_t next_s0 = s1;  // the states of frame t + 1 start where frame t ends
  for (int32_t k = s0 + blockIdx.z * blockDim.x + threadIdx.x; k < s1;
       k += gridDim.z * blockDim.x) {
    const int32_t p0 = v.st_arc0[k], p1 = v.st_arc0[k + 1];
    f.row_ids1[sb + k] = seq;
    f.row_splits2[sb + k] = ab + p0;
    for (int32_t p = p0; p < p1; ++p) {
      int32_t aidx = v.arc_aidx[p];
      const int32_t graph_label = g.a_arcs[aidx].label;
      Arc out;
      out.src = k;
      out.dest = next_s0 + v.arc_dest[p];
      out.label = graph_label;
      out.score = v.arc_ll[p];
      if (t == final_t - 1 && graph_label != -1) {  // allow_partial (:625-634)
        out.label = -1;
        aidx = -1;
      }
      f.arcs[ab + p] = out;
      f.row_ids2[ab + p] = sb + k;
      f.arc_map_a[ab + p] = aidx;
      f.arc_map_b[ab + p] = (row0 + t) * g.cols + graph_label + 1;
    }
  }
}


// CTAs per frame: about 16 per SM in all, however few the frames are.
unsigned FormatParts(int64_t frames, int64_t seqs) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(32, NumSms() * 16 / (frames * seqs)));
}

// ---------------------------------------------------------------------------
// Chunk-by-chunk decoding (OnlineDenseIntersecter, k2/csrc/intersect_dense_pruned.cu:
// 247-312 OnlineIntersect, :336-405 GetFinalFrame, :1739-1853 Decode).  Every stream
// brings the frames it has decoded so far (loaded into its arena slice before the
// launch); the kernel searches the frames of the chunk, prunes the last two frames of
// the history together with the chunk (:274-277), and closes the lattice with the final
// arcs that the extra row [0, -inf, ...] of the chunk allows.
// ---------------------------------------------------------------------------
struct OnlineArgs {
  SearchArgs g;            // g.T + 2 = capacity of the frame tables
  const int32_t *hist;     // [num_seqs] frames searched so far (index of the frontier)
  const float *beam_in;    // [num_seqs]
  float *beam_out;         // [num_seqs]
  int32_t chunk;           // frames in this chunk
  int32_t hist_max;        // longest history in the batch (the reference aligns streams
                           // at their ends, so the pruning window is counted from there)
};

// Layout of the arcs of a frame that are about to be expanded; returns their number.
__device__ int32_t LayoutFrame(const SearchArgs &g, const SeqView &v, const Team &tm, int32_t s0,
                               int32_t ns) {
  int32_t na = 0;
  for (int32_t base = 0; base < ns; base += tm.threads) {
    const int32_t k = base + tm.tid;
    int32_t deg = 0;
    if (k < ns) {
      const int32_t as = v.st_astate[s0 + k];
      deg = g.a_rs2[as + 1] - g.a_rs2[as];
    }
    int32_t tot;
    const int32_t ex = tm.Scan(deg, &tot);
    if (k < ns) v.st_cnt[s0 + k] = na + ex;
    na += tot;
  }
  tm.Sync();
  if (na > 0) {
    const int32_t per_warp = ArcsPerWarp(na, tm);
    for (int32_t k = tm.tid; k < ns; k += tm.threads) {
      const int32_t f = v.st_cnt[s0 + k];
      SetWarpFirst(v, per_warp, k, f, (k + 1 < ns ? v.st_cnt[s0 + k + 1] : na) - f);
    }
  }
  tm.Sync();
  return na;
}

// GetFinalFrame (:336-405): the arcs that leave the frontier on the extra row of the
// chunk; only those with a finite score stay (label -1, or every arc when
// allow_partial finds no final arc), all of them entering one final state.  Returns
// their number, or -1 when the arena is full.
__device__ int32_t FinalArcs(const SearchArgs &g, const SeqView &v, const Team &tm, int32_t seq,
                             int32_t row, int32_t s0, int32_t ns, int32_t a0) {
  const int32_t gi = seq * g.a_stride;
  (void)gi;
  const bool row_ok = row < g.rows;
  const float *r = g.scores + (int64_t)(row_ok ? row : 0) * g.cols;
  bool redirect = false;
  if (g.allow_partial) {
    int32_t has = 0;
    for (int32_t k = tm.tid; k < ns; k += tm.threads) {
      const int32_t as = v.st_astate[s0 + k];
      for (int32_t a = g.a_rs2[as]; a < g.a_rs2[as + 1]; ++a) has |= (g.a_arcs[a].label == -1);
    }
    redirect = !tm.Any(has);
  }
  int32_t na = 0;
  for (int32_t base = 0; base < ns; base += tm.threads) {
    const int32_t k = base + tm.tid;
    int32_t cnt = 0, as = 0;
    if (k < ns) {
      as = v.st_astate[s0 + k];
      for (int32_t a = g.a_rs2[as]; a < g.a_rs2[as + 1]; ++a) {
        const Arc arc = g.a_arcs[a];
        const uint32_t col = (uint32_t)(arc.label + 1);
        float acoustic = (row_ok && col < (uint32_t)g.cols) ? r[col] : -INFINITY;
        if (redirect) acoustic = 0.0f;
        const float ll = acoustic + arc.score;
        cnt += (ll - ll == 0.0f);
      }
    }
    int32_t tot;
    const int32_t ex = tm.Scan(cnt, &tot);
    const bool fits = (int64_t)a0 + na + tot <= g.cap_a;
    if (k < ns && fits) {
      int32_t p = a0 + na + ex;
      v.st_arc0[s0 + k] = p;
      for (int32_t a = g.a_rs2[as]; a < g.a_rs2[as + 1]; ++a) {
        const Arc arc = g.a_arcs[a];
        const uint32_t col = (uint32_t)(arc.label + 1);
        float acoustic = (row_ok && col < (uint32_t)g.cols) ? r[col] : -INFINITY;
        if (redirect) acoustic = 0.0f;
        const float ll = acoustic + arc.score;
        if (ll - ll == 0.0f) {
          v.arc_aidx[p] = a;
          v.arc_ll[p] = ll;
          v.arc_dest[p] = 0;
          ++p;
        }
      }
    }
    na += tot;
    if (!fits) return -1;
  }
  if (tm.tid == 0) v.st_arc0[s0 + ns] = a0 + na;
  tm.Sync();
  return na;
}

__global__ void __launch_bounds__(kSearchThreads, 1) OnlineChunk(const OnlineArgs o) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Shared &sh = *reinterpret_cast<Shared *>(smem_raw);
  const SearchArgs &g = o.g;
  const Team tm(&sh);
  const int32_t seq = blockIdx.x / tm.size;
  float beam = o.beam_in[seq];
  const SeqView v = ViewOf(g, seq);
  const int32_t row0 = g.b_rs[seq];
  const int32_t h = o.hist[seq];
  const int32_t kNoFinalFrame = 0x3fffffff;  // online: no end-of-sequence rules (:725-760)
  // the frontier: the states of frame h; what was kept of its arcs (the final arcs of
  // the previous chunk) is dropped and they are expanded again (:354-361)
  int32_t s0 = v.frame_s0[h], ns = v.frame_s0[h + 1] - s0, a0 = v.frame_a0[h];
  tm.Sync();  // the CTAs of the team have started: their shared memory can be written
  int32_t na = LayoutFrame(g, v, tm, s0, ns);
  StageRow(g, tm, row0);
  tm.Sync();
  int32_t s_top = s0 + ns, a_top = a0;
  int32_t status = kSeqOk;
  for (int32_t t = 0; t < o.chunk; ++t) {
    int32_t nn, na1, kept;
    if (!SearchStep(g, v, tm, seq, t, kNoFinalFrame, row0, s0, ns, a0, na, &beam, &nn, &na1,
                    &kept)) {
      status = kSeqOverflow;
      break;
    }
    s0 += ns;
    a0 += kept;
    ns = nn;
    na = na1;
    s_top = s0 + ns;
    a_top = a0;
    if (tm.tid == 0) {  // published by the next barrier
      v.frame_s0[h + t + 1] = s0;
      v.frame_a0[h + t + 1] = a0;
    }
  }
  const int32_t end = h + o.chunk;
  // PruneTimeRange(max(0, T_ - 2), T_ + chunk) in frames counted from the end of the
  // longest history: a stream with a shorter one starts inside the window, and then
  // its first frame is not the one whose states are all kept
  const int32_t begin_aligned = max(0, o.hist_max - 2) - (o.hist_max - h);
  if (status == kSeqOk &&
      !PruneWindow(g, v, tm, seq, max(begin_aligned, 0), end, &s_top, &a_top, begin_aligned >= 0))
    status = kSeqOverflow;
  if (status == kSeqOk) {
    s0 = s_top - ns;
    a0 = a_top;
    const int32_t nf = FinalArcs(g, v, tm, seq, row0 + o.chunk, s0, ns, a0);
    if (nf < 0) {
      status = kSeqOverflow;
    } else {
      a_top = a0 + nf;
      if (tm.tid == 0) {
        v.frame_s0[end + 1] = s_top;
        v.frame_a0[end + 1] = a_top;
        v.st_arc0[s_top] = a_top;
      }
    }
  }
  if (status == kSeqOk) {
    tm.Sync();
    LargestFrame(v, tm, end + 1);
  }
  if (tm.tid == 0) {
    int32_t *out = g.seq_out + kSeqOut * seq;
    out[0] = s_top;      // states without the final one
    out[1] = a_top;
    out[2] = end;        // frames: the frontier is frame `end`
    out[3] = status;
    out[4] = sh.most_states;
    out[5] = sh.most_arcs;
    o.beam_out[seq] = beam;
  }
  tm.Sync();
}

// Lattice of one (stream, frame) per CTA, all frames so far plus one final state that
// the final arcs enter (FormatOutput with online_decoding, :474-657; a stream without
// final arcs gets the state all the same, :519-547).  No arc_map_b.
__global__ void FormatOnline(const FormatArgs f, const int32_t *__restrict__ hist, int32_t chunk) {
  const SearchArgs &g = f.g;
  const int32_t seq = blockIdx.y, t = blockIdx.x;
  const SeqView v = ViewOf(g, seq);
  const int32_t end = hist[seq] + chunk;  // the frontier
  if (t > end + 1) return;
  const int32_t sb = f.out_rs1[seq], ab = f.arc_base[seq];
  const bool first = blockIdx.z == 0;
  if (f.level_splits != nullptr && first && threadIdx.x == 0) {
    // frames are layers; the final state is a layer of its own
    const int32_t lo = f.level_offsets[seq];
    f.level_splits[lo + t] = sb + v.frame_s0[t];
    if (seq == g.num_seqs - 1 && t == end + 1) f.level_splits[lo + t + 1] = f.out_rs1[g.num_seqs];
  }
  if (t == end + 1) {
    if (first && threadIdx.x == 0) {
      const int32_t s_top = v.frame_s0[end + 1];
      f.row_ids1[sb + s_top] = seq;
      f.row_splits2[sb + s_top] = ab + v.frame_a0[end + 1];
      if (seq == g.num_seqs - 1) f.row_splits2[f.out_rs1[g.num_seqs]] = f.arc_base[g.num_seqs];
    }
    return;
  }
  const int32_t s0 = v.frame_s0[t], s1 = v.frame_s0[t + 1];
  for (int32_t k = s0 + blockIdx.z * blockDim.x + threadIdx.x; k < s1;
       k += gridDim.z * blockDim.x) {
    const int32_t p0 = v.st_arc0[k], p1 = v.st_arc0[k + 1];
    f.row_ids1[sb + k] = seq;
    f.row_splits2[sb + k] = ab + p0;
    for (int32_t p = p0; p < p1; ++p) {
      int32_t aidx = v.arc_aidx[p];
      const int32_t graph_label = g.a_arcs[aidx].label;
      Arc out;
      out.src = k;
      out.dest = s1 + v.arc_dest[p];
      out.label = graph_label;
      out.score = v.arc_ll[p];
      if (t == end && graph_label != -1) {  // allow_partial (:625-634)
        out.label = -1;
        aidx = -1;
      }
      f.arcs[ab + p] = out;
      f.row_ids2[ab + p] = sb + k;
      f.arc_map_a[ab + p] = aidx;
    }
  }
}

// CTAs per sequence: the most with which the clusters of all n sequences are resident at once
// (a cluster lies within one group of SMs, so that is less than the number of SMs divided
// by n: 16 sequences of 8 CTAs fill groups of 18 SMs, an 18th would wait for one of them to
// end).  Sizes above 8 are not portable and are asked for.  One sequence of 150 frames on
// a graph of 20000 states: 8.3 ms with 8 CTAs, 6.1 with 16.
template <typename Kernel>
int32_t LaunchTeams(Kernel kernel, int32_t n, int32_t team, cudaStream_t stream,
                    const void *args) {
  static std::mutex mu;
  static std::map<int, std::array<int, kMaxTeam + 1>> resident;  // per device, by team size
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kSearchThreads);
  cfg.dynamicSmemBytes = sizeof(Shared);
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int dev = 0;
  K2B_CUDA_OK(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(mu);
    auto it = resident.find(dev);
    if (it == resident.end()) {
      K2B_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(Shared)));
      K2B_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
      std::array<int, kMaxTeam + 1> most = {};
      for (int32_t t = 2; t <= kMaxTeam; ++t) {
        cfg.gridDim = dim3(t);
        attr.val.clusterDim.x = t;
        if (cudaOccupancyMaxActiveClusters(&most[t], kernel, &cfg) != cudaSuccess) {
          most[t] = 0;
          cudaGetLastError();  // a size that this device does not take
        }
      }
      it = resident.emplace(dev, most).first;
    }
    if (team == 0) {
      team = kMaxTeam;
      while (team > 1 && it->second[team] < n) --team;
    }
  }
  cfg.gridDim = dim3(n * team);
  attr.val.clusterDim.x = team;
  void *params[] = {const_cast<void *>(args)};
  K2B_CUDA_OK(cudaLaunchKernelExC(&cfg, reinterpret_cast<const void *>(kernel), params));
  NoteLaunch();
  return kOk;
}

// Carves the workspace.  Everything is sized from the arguments alone, so the
// search and the output call agree on it.
struct PrunedLayout {
  SearchArgs g;
  int32_t *out_rs1, *arc_base;  // [num_seqs + 1] each
  size_t winner_bytes, bytes;
};

size_t Take(size_t *off, size_t n) {
  const size_t at = *off;
  *off += AlignUp(n);
  return at;
}

int32_t MakePrunedLayout(const k2b200_pruned_args *a, char *ws, PrunedLayout *L) {
  K2B_REQUIRE(a != nullptr, "NULL arguments");
  K2B_REQUIRE(a->search_beam > 0 && a->output_beam > 0, "search_beam and output_beam must be positive");
  K2B_REQUIRE(a->min_active_states >= 0 && a->max_active_states > a->min_active_states,
              "need 0 <= min_active_states < max_active_states");
  K2B_REQUIRE(a->num_seqs >= 1 && a->num_seqs <= 65535, "num_seqs must be in [1, 65535]");
  K2B_REQUIRE(a->num_fsas == a->num_seqs || a->num_fsas == 1,
              "a_fsas must hold one graph per sequence or a single shared graph (got %d graphs "
              "for %d sequences)", a->num_fsas, a->num_seqs);
  K2B_REQUIRE(a->h_b_row_splits != nullptr, "NULL h_b_row_splits");
  K2B_REQUIRE(a->max_states_per_seq >= 2 && a->max_arcs_per_seq >= 1 &&
                  a->max_states_per_seq < 0x7f000000 && a->max_arcs_per_seq < 0x7f000000,
              "arena capacities out of range");
  int32_t T = 0;
  for (int32_t i = 0; i < a->num_seqs; ++i) {
    const int32_t rows = a->h_b_row_splits[i + 1] - a->h_b_row_splits[i];
    K2B_REQUIRE(rows >= 1, "sequence %d has no rows", i);
    T = std::max(T, rows);
  }
  K2B_REQUIRE(a->h_b_row_splits[a->num_seqs] == a->rows, "b row_splits do not cover the scores");
  SearchArgs &g = L->g;
  g.a_rs1 = a->a_row_splits1;
  g.a_rs2 = a->a_row_splits2;
  g.a_arcs = reinterpret_cast<const Arc *>(a->a_arcs);
  g.a_stride = a->num_fsas == 1 && a->num_seqs > 1 ? 0 : 1;
  g.a_states = a->num_states;
  g.scores = a->scores;
  g.rows = a->rows;
  g.cols = a->cols;
  g.b_rs = a->b_row_splits;
  g.num_seqs = a->num_seqs;
  g.T = T;
  g.search_beam = a->search_beam;
  g.output_beam = a->output_beam;
  g.min_active = (float)a->min_active_states;
  g.max_active = (float)a->max_active_states;
  g.allow_partial = a->allow_partial;
  g.cap_s = a->max_states_per_seq;
  g.cap_a = a->max_arcs_per_seq;
  const size_t n = (size_t)a->num_seqs, ns = n * ((size_t)g.cap_s + 1), na = n * (size_t)g.cap_a;
  size_t off = 0;
  auto i32 = [&](size_t count) { return reinterpret_cast<int32_t *>(ws + Take(&off, 4 * count)); };
  auto f32 = [&](size_t count) { return reinterpret_cast<float *>(ws + Take(&off, 4 * count)); };
  g.st_astate = i32(ns);
  g.st_fwd = i32(ns);
  g.st_arc0 = i32(ns);
  g.st_new = i32(ns);
  g.st_cnt = i32(ns);
  g.st_bwd = f32(ns);
  g.arc_aidx = i32(na);
  g.arc_dest = i32(na);
  g.arc_ll = f32(na);
  g.arc_end = f32(na);
  g.arc_deg = reinterpret_cast<uint8_t *>(ws + Take(&off, na));
  L->winner_bytes = 8 * (g.a_stride ? (size_t)std::max(a->num_states, 1)
                                    : n * (size_t)std::max(a->num_states, 1));
  g.winner = reinterpret_cast<unsigned long long *>(ws + Take(&off, L->winner_bytes));
  g.frame_s0 = i32(n * ((size_t)T + 2));
  g.frame_a0 = i32(n * ((size_t)T + 2));
  g.warp_first = i32(n * kTeamWarps);
  g.seq_out = i32(kSeqOut * n);
  L->out_rs1 = i32(n + 1);
  L->arc_base = i32(n + 1);
  L->bytes = off;
  return kOk;
}


// Many device-to-device copies in one launch (the eight arrays of every stream): grid =
// (copies, parts of a copy), 4-byte elements.  A stream's history runs to millions of arcs;
// one CTA per copy took 400 us for the arrays of four streams.
struct CopyJob {
  const int32_t *src;
  int32_t *dst;
  int64_t count;
};
__global__ void CopyMany(const CopyJob *__restrict__ jobs) {
  const CopyJob j = jobs[blockIdx.x];
  const int64_t step = (int64_t)gridDim.y * blockDim.x;
  for (int64_t k = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; k < j.count; k += 4 * step) {
    int32_t x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k + u * step < j.count) x[u] = j.src[k + u * step];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k + u * step < j.count) j.dst[k + u * step] = x[u];
  }
}

// The online entry points share the arena layout of the batch search: the frame
// tables are sized for the longest history plus the chunk.
struct OnlineLayout {
  PrunedLayout base;
  int32_t *hist;
  float *beam_in, *beam_out;
  CopyJob *jobs;  // [8 * num_seqs]
  int32_t chunk, hist_max;
  size_t bytes;
};

int32_t MakeOnlineLayout(const k2b200_online_args *a, char *ws, OnlineLayout *L) {
  K2B_REQUIRE(a != nullptr && a->h_hist != nullptr && a->h_b_row_splits != nullptr,
              "NULL arguments");
  K2B_REQUIRE(a->num_seqs >= 1, "num_seqs must be positive");
  const int32_t rows0 = a->h_b_row_splits[1] - a->h_b_row_splits[0];
  int32_t hist_max = 0;
  for (int32_t i = 0; i < a->num_seqs; ++i) {
    K2B_REQUIRE(a->h_b_row_splits[i + 1] - a->h_b_row_splits[i] == rows0,
                "the streams of a chunk must all have the same number of frames");
    K2B_REQUIRE(a->h_hist[i] >= 0, "negative history length");
    hist_max = std::max(hist_max, a->h_hist[i]);
  }
  K2B_REQUIRE(rows0 >= 2, "a chunk needs at least one frame besides its final row");
  // a batch-mode argument block whose longest sequence has hist_max + chunk rows gives
  // frame tables of hist_max + chunk + 2 entries
  k2b200_pruned_args p = {};
  p.num_fsas = 1;
  p.num_states = a->num_states;
  p.num_arcs = a->num_arcs;
  p.a_row_splits1 = a->a_row_splits1;
  p.a_row_splits2 = a->a_row_splits2;
  p.a_arcs = a->a_arcs;
  p.scores = a->scores;
  p.rows = a->rows;
  p.cols = a->cols;
  p.num_seqs = a->num_seqs;
  p.b_row_splits = a->b_row_splits;
  p.search_beam = a->search_beam;
  p.output_beam = a->output_beam;
  p.min_active_states = a->min_active_states;
  p.max_active_states = a->max_active_states;
  p.allow_partial = a->allow_partial;
  p.max_states_per_seq = a->max_states_per_seq;
  p.max_arcs_per_seq = a->max_arcs_per_seq;
  std::vector<int32_t> fake(a->num_seqs + 1);
  for (int32_t i = 0; i <= a->num_seqs; ++i) fake[i] = i * (hist_max + rows0 - 1);
  p.h_b_row_splits = fake.data();
  p.rows = fake[a->num_seqs];
  K2B_FORWARD(MakePrunedLayout(&p, ws, &L->base));
  SearchArgs &g = L->base.g;
  g.rows = a->rows;
  g.a_stride = 0;  // one graph, a table per stream
  g.T = hist_max + rows0 - 1;
  // the winner table of the batch layout was sized for a shared graph only when there is
  // more than one sequence; make room for one table per stream in every case
  size_t off = L->base.bytes;
  L->base.winner_bytes = 8 * (size_t)a->num_seqs * (size_t)std::max(a->num_states, 1);
  g.winner = reinterpret_cast<unsigned long long *>(ws + Take(&off, L->base.winner_bytes));
  L->hist = reinterpret_cast<int32_t *>(ws + Take(&off, 4 * (size_t)a->num_seqs));
  L->beam_in = reinterpret_cast<float *>(ws + Take(&off, 4 * (size_t)a->num_seqs));
  L->beam_out = reinterpret_cast<float *>(ws + Take(&off, 4 * (size_t)a->num_seqs));
  L->jobs = reinterpret_cast<CopyJob *>(ws + Take(&off, sizeof(CopyJob) * 8 * (size_t)a->num_seqs));
  L->chunk = rows0 - 1;
  L->hist_max = hist_max;
  L->bytes = off;
  return kOk;
}

}  // namespace
}  // namespace k2b

using namespace k2b;  // NOLINT

extern "C" {

int32_t k2b200_intersect_dense_pruned_workspace_bytes(const k2b200_pruned_args *args,
                                                      size_t *bytes, int64_t *total_levels) {
  PrunedLayout L;
  K2B_FORWARD(MakePrunedLayout(args, nullptr, &L));
  K2B_REQUIRE(bytes != nullptr, "NULL bytes");
  *bytes = L.bytes;
  if (total_levels) *total_levels = (int64_t)args->num_seqs * (L.g.T + 2);
  return kOk;
}

int32_t k2b200_intersect_dense_pruned_search(const k2b200_pruned_args *args, void *workspace,
                                             size_t workspace_bytes, void *stream_v,
                                             int32_t *num_states_out, int32_t *num_arcs_out,
                                             int32_t *arena_full) {
  return k2b200_intersect_dense_pruned_search_bounds(args, workspace, workspace_bytes, stream_v,
                                                     num_states_out, num_arcs_out, arena_full,
                                                     nullptr);
}

int32_t k2b200_intersect_dense_pruned_search_bounds(
    const k2b200_pruned_args *args, void *workspace, size_t workspace_bytes, void *stream_v,
    int32_t *num_states_out, int32_t *num_arcs_out, int32_t *arena_full, int32_t *layer_bounds) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  PrunedLayout L;
  K2B_FORWARD(MakePrunedLayout(args, reinterpret_cast<char *>(workspace), &L));
  K2B_REQUIRE(workspace != nullptr && workspace_bytes >= L.bytes, "workspace too small");
  K2B_REQUIRE(num_states_out && num_arcs_out && arena_full, "NULL output pointer");
  K2B_REQUIRE(args->a_row_splits1 && args->a_row_splits2 && args->b_row_splits &&
                  (args->a_arcs || args->num_arcs == 0) && args->scores,
              "NULL input pointer");
  const int32_t n = args->num_seqs;
  K2B_CUDA_OK(cudaMemsetAsync(L.g.winner, 0, L.winner_bytes, stream));
  K2B_REQUIRE(args->team_ctas == 0 || args->team_ctas == 1 || args->team_ctas == 2 ||
                  args->team_ctas == 4 || args->team_ctas == 8,
              "team_ctas must be 1, 2, 4 or 8");
  K2B_FORWARD(LaunchTeams(PrunedSearch, n, args->team_ctas, stream, &L.g));
  K2B_CUDA_OK(cudaGetLastError());
  std::vector<int32_t> h(kSeqOut * (size_t)n);
  K2B_CUDA_OK(cudaMemcpyAsync(h.data(), L.g.seq_out, sizeof(int32_t) * h.size(),
                              cudaMemcpyDeviceToHost, stream));
  K2B_CUDA_OK(cudaStreamSynchronize(stream));
  std::vector<int32_t> bases(2 * ((size_t)n + 1));
  int32_t *srs = bases.data(), *ars = bases.data() + n + 1;
  int64_t ts = 0, ta = 0;
  *arena_full = 0;
  for (int32_t i = 0; i < n; ++i) {
    if (h[kSeqOut * i + 3] == kSeqOverflow) *arena_full = 1;
    K2B_REQUIRE(h[kSeqOut * i + 3] != kSeqManyFinal,
                "sequence %d reaches more than one state on its last frame: arcs with label -1 "
                "must enter the final state of their graph", i);
    srs[i] = (int32_t)ts;
    ars[i] = (int32_t)ta;
    ts += h[kSeqOut * i];
    ta += h[kSeqOut * i + 1];
  }
  srs[n] = (int32_t)ts;
  ars[n] = (int32_t)ta;
  *num_states_out = *num_arcs_out = 0;
  if (layer_bounds != nullptr) {
    layer_bounds[0] = layer_bounds[1] = 1;
    for (int32_t i = 0; i < n; ++i) {
      layer_bounds[0] = std::max(layer_bounds[0], h[kSeqOut * i + 4]);
      layer_bounds[1] = std::max(layer_bounds[1], h[kSeqOut * i + 5]);
    }
  }
  if (*arena_full) return kOk;
  K2B_REQUIRE(ts < INT_MAX && ta < INT_MAX, "the lattice has too many states or arcs for int32");
  // out_rs1 and arc_base are adjacent in the workspace only up to alignment: two uploads
  K2B_FORWARD(UploadInts(srs, n + 1, L.out_rs1, stream));
  K2B_FORWARD(UploadInts(ars, n + 1, L.arc_base, stream));
  *num_states_out = (int32_t)ts;
  *num_arcs_out = (int32_t)ta;
  return kOk;
}

int32_t k2b200_intersect_dense_pruned_emit(const k2b200_pruned_args *args, void *workspace,
                                           size_t workspace_bytes, void *stream_v,
                                           const k2b200_lattice_out *out) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  PrunedLayout L;
  K2B_FORWARD(MakePrunedLayout(args, reinterpret_cast<char *>(workspace), &L));
  K2B_REQUIRE(workspace != nullptr && workspace_bytes >= L.bytes, "workspace too small");
  K2B_REQUIRE(out && out->row_splits1 && out->row_ids1 && out->row_splits2 && out->row_ids2 &&
                  out->arcs && out->arc_map_a && out->arc_map_b,
              "NULL output pointer");
  K2B_REQUIRE((out->level_offsets == nullptr) == (out->level_splits == nullptr),
              "level_offsets and level_splits go together");
  FormatArgs f;
  f.g = L.g;
  f.out_rs1 = L.out_rs1;
  f.arc_base = L.arc_base;
  f.row_ids1 = out->row_ids1;
  f.row_splits2 = out->row_splits2;
  f.row_ids2 = out->row_ids2;
  f.arcs = reinterpret_cast<Arc *>(out->arcs);
  f.arc_map_a = out->arc_map_a;
  f.arc_map_b = out->arc_map_b;
  f.level_offsets = out->level_offsets;
  f.level_splits = out->level_splits;
  K2B_CUDA_OK(cudaMemcpyAsync(out->row_splits1, L.out_rs1, sizeof(int32_t) * (args->num_seqs + 1),
                              cudaMemcpyDeviceToDevice, stream));
  dim3 grid(L.g.T + 2, args->num_seqs, FormatParts(L.g.T + 2, args->num_seqs));
  { FormatPruned<<<grid, 128, 0, stream>>>(f); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}


int32_t k2b200_online_decode_workspace_bytes(const k2b200_online_args *args, size_t *bytes) {
  OnlineLayout L;
  K2B_FORWARD(MakeOnlineLayout(args, nullptr, &L));
  K2B_REQUIRE(bytes != nullptr, "NULL bytes");
  *bytes = L.bytes;
  return kOk;
}

// Copies what stream `seq` has decoded so far into its slice of the arenas.
int32_t k2b200_online_decode_load(const k2b200_online_args *args, void *workspace, int32_t seq,
                                  const k2b200_online_stream *st, void *stream_v) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  OnlineLayout L;
  K2B_FORWARD(MakeOnlineLayout(args, reinterpret_cast<char *>(workspace), &L));
  K2B_REQUIRE(st != nullptr && seq >= 0 && seq < args->num_seqs, "bad stream");
  const SearchArgs &g = L.base.g;
  const int32_t h = args->h_hist[seq];
  K2B_REQUIRE(st->num_states <= g.cap_s && st->num_arcs <= g.cap_a,
              "the arena is smaller than what stream %d already holds", seq);
  const int64_t so = (int64_t)seq * (g.cap_s + 1), ao = (int64_t)seq * g.cap_a,
                fo = (int64_t)seq * (g.T + 2);
  auto copy = [&](void *dst, const void *src, size_t n) {
    return n == 0 ? cudaSuccess
                  : cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToDevice, stream);
  };
  K2B_CUDA_OK(copy(g.st_astate + so, st->astate, 4 * (size_t)st->num_states));
  K2B_CUDA_OK(copy(g.st_fwd + so, st->forward, 4 * (size_t)st->num_states));
  K2B_CUDA_OK(copy(g.st_arc0 + so, st->arc0, 4 * ((size_t)st->num_states + 1)));
  K2B_CUDA_OK(copy(g.arc_aidx + ao, st->arc_graph, 4 * (size_t)st->num_arcs));
  K2B_CUDA_OK(copy(g.arc_ll + ao, st->arc_score, 4 * (size_t)st->num_arcs));
  K2B_CUDA_OK(copy(g.arc_dest + ao, st->arc_dest, 4 * (size_t)st->num_arcs));
  K2B_CUDA_OK(copy(g.frame_s0 + fo, st->frame_state0, 4 * ((size_t)h + 2)));
  K2B_CUDA_OK(copy(g.frame_a0 + fo, st->frame_arc0, 4 * ((size_t)h + 2)));
  return kOk;
}

int32_t k2b200_online_decode_run(const k2b200_online_args *args, void *workspace,
                                 size_t workspace_bytes, void *stream_v, const float *h_beams_in,
                                 float *h_beams_out, int32_t *h_counts, int32_t *num_states_out,
                                 int32_t *num_arcs_out, int32_t *arena_full) {
  return k2b200_online_decode_run_bounds(args, workspace, workspace_bytes, stream_v, h_beams_in,
                                         h_beams_out, h_counts, num_states_out, num_arcs_out,
                                         arena_full, nullptr);
}

int32_t k2b200_online_decode_run_bounds(const k2b200_online_args *args, void *workspace,
                                        size_t workspace_bytes, void *stream_v,
                                        const float *h_beams_in, float *h_beams_out,
                                        int32_t *h_counts, int32_t *num_states_out,
                                        int32_t *num_arcs_out, int32_t *arena_full,
                                        int32_t *layer_bounds) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  OnlineLayout L;
  K2B_FORWARD(MakeOnlineLayout(args, reinterpret_cast<char *>(workspace), &L));
  K2B_REQUIRE(workspace != nullptr && workspace_bytes >= L.bytes, "workspace too small");
  K2B_REQUIRE(h_beams_in && h_beams_out && h_counts && num_states_out && num_arcs_out &&
                  arena_full, "NULL pointer");
  const int32_t n = args->num_seqs;
  K2B_CUDA_OK(cudaMemsetAsync(L.base.g.winner, 0, L.base.winner_bytes, stream));
  K2B_FORWARD(UploadInts(args->h_hist, n, L.hist, stream));
  K2B_FORWARD(UploadInts(reinterpret_cast<const int32_t *>(h_beams_in), n,
                         reinterpret_cast<int32_t *>(L.beam_in), stream));
  OnlineArgs o;
  o.g = L.base.g;
  o.hist = L.hist;
  o.beam_in = L.beam_in;
  o.beam_out = L.beam_out;
  o.chunk = L.chunk;
  o.hist_max = L.hist_max;
  K2B_REQUIRE(args->team_ctas == 0 || args->team_ctas == 1 || args->team_ctas == 2 ||
                  args->team_ctas == 4 || args->team_ctas == 8,
              "team_ctas must be 1, 2, 4 or 8");
  K2B_FORWARD(LaunchTeams(OnlineChunk, n, args->team_ctas, stream, &o));
  std::vector<int32_t> h(kSeqOut * (size_t)n);
  K2B_CUDA_OK(cudaMemcpyAsync(h.data(), L.base.g.seq_out, sizeof(int32_t) * h.size(),
                              cudaMemcpyDeviceToHost, stream));
  K2B_CUDA_OK(cudaMemcpyAsync(h_beams_out, L.beam_out, sizeof(float) * n, cudaMemcpyDeviceToHost,
                              stream));
  K2B_CUDA_OK(cudaStreamSynchronize(stream));
  std::vector<int32_t> bases(2 * ((size_t)n + 1));
  int32_t *srs = bases.data(), *ars = bases.data() + n + 1;
  int64_t ts = 0, ta = 0;
  *arena_full = 0;
  for (int32_t i = 0; i < n; ++i) {
    if (h[kSeqOut * i + 3] == kSeqOverflow) *arena_full = 1;
    h_counts[2 * i] = h[kSeqOut * i];
    h_counts[2 * i + 1] = h[kSeqOut * i + 1];
    srs[i] = (int32_t)ts;
    ars[i] = (int32_t)ta;
    ts += h[kSeqOut * i] + 1;  // one final state per stream
    ta += h[kSeqOut * i + 1];
  }
  srs[n] = (int32_t)ts;
  ars[n] = (int32_t)ta;
  *num_states_out = *num_arcs_out = 0;
  if (layer_bounds != nullptr) {
    layer_bounds[0] = layer_bounds[1] = 1;
    for (int32_t i = 0; i < n; ++i) {
      layer_bounds[0] = std::max(layer_bounds[0], h[kSeqOut * i + 4]);
      layer_bounds[1] = std::max(layer_bounds[1], h[kSeqOut * i + 5]);
    }
  }
  if (*arena_full) return kOk;
  K2B_REQUIRE(ts < INT_MAX && ta < INT_MAX, "the lattice has too many states or arcs for int32");
  K2B_FORWARD(UploadInts(srs, n + 1, L.base.out_rs1, stream));
  K2B_FORWARD(UploadInts(ars, n + 1, L.base.arc_base, stream));
  *num_states_out = (int32_t)ts;
  *num_arcs_out = (int32_t)ta;
  return kOk;
}

int32_t k2b200_online_decode_emit(const k2b200_online_args *args, void *workspace,
                                  size_t workspace_bytes, void *stream_v,
                                  const k2b200_lattice_out *out) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  OnlineLayout L;
  K2B_FORWARD(MakeOnlineLayout(args, reinterpret_cast<char *>(workspace), &L));
  K2B_REQUIRE(workspace != nullptr && workspace_bytes >= L.bytes, "workspace too small");
  K2B_REQUIRE(out && out->row_splits1 && out->row_ids1 && out->row_splits2 && out->row_ids2 &&
                  out->arcs && out->arc_map_a, "NULL output pointer");
  FormatArgs f;
  f.g = L.base.g;
  f.out_rs1 = L.base.out_rs1;
  f.arc_base = L.base.arc_base;
  f.row_ids1 = out->row_ids1;
  f.row_splits2 = out->row_splits2;
  f.row_ids2 = out->row_ids2;
  f.arcs = reinterpret_cast<Arc *>(out->arcs);
  f.arc_map_a = out->arc_map_a;
  f.arc_map_b = nullptr;
  K2B_REQUIRE((out->level_offsets == nullptr) == (out->level_splits == nullptr),
              "level_offsets and level_splits go together");
  f.level_offsets = out->level_offsets;
  f.level_splits = out->level_splits;
  if (out->level_offsets != nullptr) {
    // stream i has (history + chunk + 2) layers: its frames and the final state
    std::vector<int32_t> lo(args->num_seqs + 1, 0);
    for (int32_t i = 0; i < args->num_seqs; ++i)
      lo[i + 1] = lo[i] + args->h_hist[i] + L.chunk + 2;
    K2B_FORWARD(UploadInts(lo.data(), args->num_seqs + 1, out->level_offsets, stream));
  }
  K2B_CUDA_OK(cudaMemcpyAsync(out->row_splits1, L.base.out_rs1,
                              sizeof(int32_t) * (args->num_seqs + 1), cudaMemcpyDeviceToDevice,
                              stream));
  dim3 grid(L.base.g.T + 2, args->num_seqs, FormatParts(L.base.g.T + 2, args->num_seqs));
  { FormatOnline<<<grid, 128, 0, stream>>>(f, L.hist, L.chunk); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

// Copies stream `seq` out of its arena slice: num_states / num_arcs as reported by
// k2b200_online_decode_run, frame tables of (history + chunk + 2) entries.
int32_t k2b200_online_decode_store(const k2b200_online_args *args, void *workspace, int32_t seq,
                                   const k2b200_online_stream *st, void *stream_v) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  OnlineLayout L;
  K2B_FORWARD(MakeOnlineLayout(args, reinterpret_cast<char *>(workspace), &L));
  K2B_REQUIRE(st != nullptr && seq >= 0 && seq < args->num_seqs, "bad stream");
  const SearchArgs &g = L.base.g;
  const int32_t h = args->h_hist[seq] + L.chunk;
  const int64_t so = (int64_t)seq * (g.cap_s + 1), ao = (int64_t)seq * g.cap_a,
                fo = (int64_t)seq * (g.T + 2);
  auto copy = [&](const void *dst, const void *src, size_t n) {
    return n == 0 ? cudaSuccess
                  : cudaMemcpyAsync(const_cast<void *>(dst), src, n, cudaMemcpyDeviceToDevice,
                                    stream);
  };
  K2B_CUDA_OK(copy(st->astate, g.st_astate + so, 4 * (size_t)st->num_states));
  K2B_CUDA_OK(copy(st->forward, g.st_fwd + so, 4 * (size_t)st->num_states));
  K2B_CUDA_OK(copy(st->arc0, g.st_arc0 + so, 4 * ((size_t)st->num_states + 1)));
  K2B_CUDA_OK(copy(st->arc_graph, g.arc_aidx + ao, 4 * (size_t)st->num_arcs));
  K2B_CUDA_OK(copy(st->arc_score, g.arc_ll + ao, 4 * (size_t)st->num_arcs));
  K2B_CUDA_OK(copy(st->arc_dest, g.arc_dest + ao, 4 * (size_t)st->num_arcs));
  K2B_CUDA_OK(copy(st->frame_state0, g.frame_s0 + fo, 4 * ((size_t)h + 2)));
  K2B_CUDA_OK(copy(st->frame_arc0, g.frame_a0 + fo, 4 * ((size_t)h + 2)));
  return kOk;
}


// All streams in one launch: `streams` is a HOST array of num_seqs descriptors.
static int32_t CopyStreams(const k2b200_online_args *args, void *workspace,
                           const k2b200_online_stream *streams, bool load, cudaStream_t stream) {
  OnlineLayout L;
  K2B_FORWARD(MakeOnlineLayout(args, reinterpret_cast<char *>(workspace), &L));
  K2B_REQUIRE(streams != nullptr, "NULL streams");
  const SearchArgs &g = L.base.g;
  const int32_t n = args->num_seqs;
  std::vector<CopyJob> jobs;
  jobs.reserve(8 * (size_t)n);
  for (int32_t i = 0; i < n; ++i) {
    const k2b200_online_stream &st = streams[i];
    K2B_REQUIRE(st.num_states <= g.cap_s && st.num_arcs <= g.cap_a,
                "the arena is smaller than what stream %d holds", i);
    const int64_t h = args->h_hist[i] + (load ? 0 : L.chunk);
    const int64_t so = (int64_t)i * (g.cap_s + 1), ao = (int64_t)i * g.cap_a,
                  fo = (int64_t)i * (g.T + 2);
    struct { int32_t *arena; void *mine; int64_t count; } parts[8] = {
        {g.st_astate + so, st.astate, st.num_states},
        {g.st_fwd + so, st.forward, st.num_states},
        {g.st_arc0 + so, st.arc0, (int64_t)st.num_states + 1},
        {g.arc_aidx + ao, st.arc_graph, st.num_arcs},
        {reinterpret_cast<int32_t *>(g.arc_ll + ao), st.arc_score, st.num_arcs},
        {g.arc_dest + ao, st.arc_dest, st.num_arcs},
        {g.frame_s0 + fo, st.frame_state0, h + 2},
        {g.frame_a0 + fo, st.frame_arc0, h + 2}};
    for (const auto &p : parts) {
      CopyJob j;
      j.src = load ? reinterpret_cast<const int32_t *>(p.mine) : p.arena;
      j.dst = load ? p.arena : reinterpret_cast<int32_t *>(p.mine);
      j.count = p.count;
      jobs.push_back(j);
    }
  }
  static_assert(sizeof(CopyJob) % 4 == 0, "jobs travel as 32-bit words");
  K2B_FORWARD(UploadInts(reinterpret_cast<const int32_t *>(jobs.data()),
                         (int64_t)(jobs.size() * sizeof(CopyJob) / 4),
                         reinterpret_cast<int32_t *>(L.jobs), stream));
  int64_t longest = 1;
  for (const CopyJob &j : jobs) longest = std::max(longest, j.count);
  // about 8 CTAs per SM when the copies are long
  const int32_t parts = (int32_t)std::max<int64_t>(
      1, std::min<int64_t>(CeilDiv(longest, 1024), NumSms() * 8 / (int64_t)jobs.size() + 1));
  { CopyMany<<<dim3((unsigned)jobs.size(), parts), 256, 0, stream>>>(L.jobs); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

int32_t k2b200_online_decode_load_all(const k2b200_online_args *args, void *workspace,
                                      const k2b200_online_stream *streams, void *stream_v) {
  return CopyStreams(args, workspace, streams, true, reinterpret_cast<cudaStream_t>(stream_v));
}

int32_t k2b200_online_decode_store_all(const k2b200_online_args *args, void *workspace,
                                       const k2b200_online_stream *streams, void *stream_v) {
  return CopyStreams(args, workspace, streams, false, reinterpret_cast<cudaStream_t>(stream_v));
}

}  // extern "C"
