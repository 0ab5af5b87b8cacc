// Lattice-free total scores and gradients for band graphs (CTC and alike): the path
//   lattice = intersect_dense(graphs, dense, beam)        k2/csrc/intersect_dense.cu:100-1073
//   tot     = lattice.get_tot_scores(log_semiring=True)   k2/csrc/fsa_utils.cu:1124-1454,1809-1837
//   backward through arc posteriors and both arc maps     k2/csrc/fsa_utils.cu:1839-1901,
//                                                         k2/python/k2/autograd.py:30-117,511-664
// for graphs in which
//   * every arc goes from state s to s, s+1 or s+2, at most one arc per (source, destination), and
//   * all arcs entering a state carry the same label
// (what k2.ctc_graph builds, standard and modified: k2/csrc/fsa_algo.cu:577-730).  Then a state
// needs ONE dense score per frame (that of its label), the recursion over the states of a graph
// has neighbours only, and the states that survive pruning on a frame are few (a few tens out of
// hundreds).  The kernels are built on that:
//
//   BandViterbi   one small CTA per (graph, direction) walks all frames: a thread owns four
//                 consecutive states in registers, neighbours come by shuffles (and a
//                 hand-over between warps every few frames), the log-prob row of the frame arrives in a
//                 shared-memory ring by one bulk copy (TMA, mbarrier) issued many frames ahead.
//                 Same fp32 expressions as the reference: (prev + arc.score) + dense, then max.
//   BandPrep      all (graph, frame) levels in parallel: the reference's keep tests
//                 (intersect_dense.cu:289-296, 430-471) on the two Viterbi grids, then per level
//                 the COMPACT list of surviving states with, per state and entering arc, the
//                 factor exp(arc score) * exp(dense score) if the arc survives and 0 otherwise,
//                 and the list positions of the states the arcs come from and go to.
//   BandChainLists  one CTA per (graph, direction) walks the levels over the lists only: a thread
//                 holds the value of one surviving state, an entry names the list positions of
//                 its neighbours on the previous level, whose values are in shared memory:
//                 three multiply-adds per state and level, no exp or log, no test.  The lists
//                 arrive by bulk copies.  Values of a level share a power-of-two scale that
//                 follows the data.
//   BandChainExact  the same recursion with a (mantissa, exponent) pair per state, by state
//                 number in shared memory, for the graphs whose scores leave what a double
//                 with a per-level scale can hold or whose levels are wider than the registers
//                 of a warp; it runs after BandChainLists and returns at once for every other
//                 graph.
//   BandGradRows  all levels in parallel: posterior of (level, state) = alpha * beta / Z is the
//                 gradient of that state's dense score; every row of the gradient is written
//                 whole.
//   BandGrad      the same added to rows that sequences share, and arc posteriors for the
//                 gradient of the graph's arc scores.
//
// Each of these kernels waits for the one before it and is set up while that one still runs
// (LaunchBehind): 5 to 8 us of a pass.  BandViterbi and BandChainLists, whose CTAs are all resident
// from the start, let the next one start at once, BandPrep does near its end.  BandGather and
// LogSoftmaxRows do not: BandViterbi's CTAs then took what room there was beside theirs, two to an
// SM (32 x 500 x 5000: 241 us a pass instead of 225).
//
// The dense scores are read straight from the log-prob tensor the DenseFsaVec was made from
// ([rows, C], any C): the [rows + N, C + 1] score matrix is not needed.  The extra
// final row of a sequence ([0, -inf, ...], k2/csrc/fsa.h:138-185) is implied: on the level after
// the last frame a state scores 0 if its label is -1 and -inf otherwise.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "../../include/k2b200.h"
#include "band_tables.cuh"
#include "common.cuh"
#include "cp_async.cuh"
#include "prob_math.cuh"

namespace k2b {

constexpr int kBandMaxStates = 1024;
constexpr int kVitK = 4;              // states per thread of BandViterbi
constexpr int kVitFramesByState = 8;  // frames between two exchanges of its warps, rows by state
constexpr int kPrepLevels = 16;       // levels per chunk: their lists share one padded size
constexpr int kGradLevels = 4;        // levels per warp of BandGrad
constexpr int kDrainPolls = 4000000;  // bounded wait for copies in flight when a kernel gives up

// bits of the status word
constexpr int32_t kStatusNotBand = 1, kStatusLate = 2;
// bits of unfit[i]: the lean recursion cannot represent this graph's numbers
constexpr int32_t kUnfitFactors = 1, kUnfitRange = 2;


// Per (graph, sequence) pair; built on the host, uploaded once per call.
struct BandInfo {
  int32_t state_off;   // first state (idx01) of the graph in a_fsas
  int32_t num_states;  // S
  int32_t pitch;       // 32 * (S / 32 + 1): row pitch of this pair's grids; a padded list fits
  int32_t frames;      // T
  int32_t lp_row;      // row of the log-prob matrix that holds frame 0
  int32_t level_off;   // sum over earlier pairs of (T + 2)
  int32_t zero_end;    // rows [lp_row + T, zero_end) belong to no sequence (dense gradient)
  int32_t pad;
  int64_t grid_off;    // sum over earlier pairs of (T + 2) * pitch
};

// Entry of a level's list of surviving states.
struct __align__(8) BandItem {
  int32_t label;  // of the arcs entering the state
  uint16_t s;     // the state
  uint8_t inb;    // bit d: the arc from state s - d of the level before survives
  uint8_t outb;   // bit d: the arc to state s + d of the next level survives
};
static_assert(sizeof(BandItem) == 8, "BandItem must be 8 bytes");
constexpr int kOutbByte = 7;
// What the recursions read per list entry (level l, state s):
//   pw[d]  = exp(score of the arc from state s - d) * exp(dense score of s's label on
//            frame l - 1) if that arc survives between levels l - 1 and l, else 0;
//   src[d] = position, in the list of level l - 1, of state s - d (0 when pw[d] is 0);
//   dst[d] = position, in the list of level l + 1, of state s + d if the arc to it
//            survives (whose factor is pw[d] of THAT entry), else kNoDst.
// The lists of the kPrepLevels levels of a chunk are padded to the same multiple of 32 entries,
// larger than the longest of them: a padding entry has pw = 0, src = 0 and dst = kNoDst, and
// kNoDst (lane 31 of the last register) always names a padding entry of the next level.
// A level of n entries is stored as n x 16 bytes {pw[0], pw[1]} followed by n x 16 bytes
// {pw[2], src, dst} (byte d = of d, the fourth unused), so that the lanes of a warp read
// consecutive 16 bytes of shared memory.
struct __align__(16) BandFactor {
  double pw[3];
  uint32_t src, dst;
};
static_assert(sizeof(BandFactor) == 32, "BandFactor must be 32 bytes");
constexpr uint32_t kNoDst = 255;
constexpr int kMaxRegs = 4;     // warps of the list recursion
constexpr int kChainThreads = 32 * kMaxRegs;
constexpr int kKeepThreads = 128;  // of BandChainLists: they look after what the others leave behind
constexpr int kMaxListed = 32 * kMaxRegs - 1;  // entries of a level that it handles (one is padding)
// alpha of the final state on the last level (= Z) of a graph, as m * 2^e
struct __align__(16) BandTotal {
  double m;
  int32_t e;
  int32_t pad;
};

__device__ __forceinline__ double Pow2Clamp(int32_t e) {
  if (e < -1000) return 0.0;
  e = e > 1000 ? 1000 : e;
  return __longlong_as_double((long long)(1023 + e) << 52);
}

// Polls an mbarrier at most `limit` times.
__device__ __forceinline__ bool WaitSlot(uint64_t *bar, unsigned parity, int32_t limit) {
  for (int32_t k = 0; k < limit; ++k)
    if (MbarTryWait(bar, parity)) return true;
  return false;
}

// Dense score of a state with `label` on dense row `row` of a sequence of T frames whose
// frame 0 is at lp0 (the row T is the implied final row).
__device__ __forceinline__ float BandDense(const float *lp0, int32_t C, int32_t T, int32_t row,
                                           int32_t label) {
  if (row < T) return (label >= 0 && label < C) ? lp0[(int64_t)row * C + label] : -INFINITY;
  return label == -1 ? 0.0f : -INFINITY;
}

// ---------------------------------------------------------------------------
// Tables of a band graph, and the check that it is one.  One thread per state.
// status bit 0 is set when some graph is not a band graph.
// ---------------------------------------------------------------------------
__global__ void BandTables(const int32_t *__restrict__ row_splits1, int32_t num_fsas,
                           const int32_t *__restrict__ row_splits2, const Arc *__restrict__ arcs,
                           int32_t num_states, BandState *__restrict__ tab,
                           BandArc *__restrict__ tabf, int32_t *__restrict__ status) {
  const int32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= num_states) return;
  int32_t lo = 0, hi = num_fsas;  // row_splits1[lo] <= idx < row_splits1[hi]
  while (lo + 1 < hi) {
    const int32_t mid = (lo + hi) >> 1;
    if (row_splits1[mid] <= idx) lo = mid; else hi = mid;
  }
  const int32_t s = idx - row_splits1[lo];
  bool bad = false;
  {  // the arcs leaving this state: at most three, to s, s + 1, s + 2, no destination twice
    const int32_t a0 = row_splits2[idx], a1 = row_splits2[idx + 1];
    bad = a1 - a0 > 3;
    uint32_t seen = 0;
    for (int32_t k = a0; k < a1 && k < a0 + 3; ++k) {
      const Arc arc = arcs[k];
      const int32_t d = arc.dest - arc.src;
      if (arc.src != s || d < 0 || d > 2 || (seen >> d) & 1u) bad = true;
      else seen |= 1u << d;
    }
  }
  BandState st;
  st.label = kNoLabel;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    st.w[d] = -INFINITY;
    BandArc fa;
    fa.f = 0.0;
    fa.k = kZeroExp;
    fa.arc = -1;
    if (s - d >= 0) {
      const int32_t a0 = row_splits2[idx - d], a1 = min(row_splits2[idx - d + 1], a0 + 3);
      for (int32_t k = a0; k < a1; ++k) {
        const Arc arc = arcs[k];
        if (arc.dest != s || fa.arc >= 0) continue;
        st.w[d] = arc.score;
        fa.arc = k;
        ExpToMantExp(arc.score, &fa.f, &fa.k);
        if (st.label == kNoLabel) st.label = arc.label;
        else if (st.label != arc.label) bad = true;
      }
    }
    tabf[(int64_t)idx * 3 + d] = fa;
  }
  tab[idx] = st;
  if (bad) atomicOr(status, kStatusNotBand);
}

// The incoming-arc index of band graphs, from their tables: of the arcs that leave the states
// before s all but those of s - 1 and s - 2 that pass s by or end there have ended before it,
// so where the arcs entering s begin follows from its neighbours - one launch of 3 us where
// counting, prefix sums, scattering and sorting took seven.
__global__ void BandIncoming(const BandState *__restrict__ tab, const BandArc *__restrict__ tabf,
                             const int32_t *__restrict__ row_splits2, int32_t num_states,
                             int32_t *__restrict__ in_splits, int32_t *__restrict__ in_arcs,
                             int32_t *__restrict__ in_src, float *__restrict__ in_score) {
  const int32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx > num_states) return;
  int32_t at = row_splits2[idx];
  if (idx < num_states) {
    const BandArc *mine = tabf + (int64_t)idx * 3;
    int32_t arc[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) arc[d] = mine[d].arc;
    const bool past = idx + 1 < num_states && mine[3 + 2].arc >= 0;
    at -= (arc[1] >= 0) + (arc[2] >= 0) + past;
    const BandState st = tab[idx];
    int32_t k = at;
#pragma unroll
    for (int d = 2; d >= 0; --d)  // arcs in increasing order: the earlier source first
      if (arc[d] >= 0) {
        in_arcs[k] = arc[d];
        in_src[k] = idx - d;
        in_score[k] = st.w[d];
        ++k;
      }
  }
  in_splits[idx] = at;
}

// ---------------------------------------------------------------------------
// Viterbi forward / backward.  grid = (2 directions, pairs).
// Level l (0 .. T + 1) of the forward grid: best score of any path from the start state
// at level 0 to the state at level l; of the backward grid: from the state at level l to
// the final state at level T + 1.  The step between levels l and l + 1 consumes dense row l
// (row T being the implied final row).
//
// A thread holds four consecutive states in registers.  A warp OWNS the states of its
// last 32 - H lanes and recomputes, in its first H lanes, the 4H states before them (the
// mirror image walking backward): a state depends on itself and its two predecessors, so
// what the warp computes for its own states stays exact for 2H frames without hearing
// from its neighbour.  Frames are therefore taken in batches of F = 2H: the log-prob rows
// of a batch are contiguous and arrive by ONE bulk copy (TMA, completion on an mbarrier)
// requested batches ahead, the warps exchange their boundary states through shared memory
// once per batch, and the frames of a batch run without any wait, barrier or
// shared-memory store.  Same fp32 expressions as the reference: (prev + arc.score) + dense, then
// max.  A warp of its own requests the rows and waits for them; the others learn of it by the
// barrier that they need anyway (a wait of theirs on the mbarrier cost a tenth of the kernel, the
// requests by a thread that walks more).
// A graph that alternates (VitForm) takes 17 instructions per frame and warp: three shared-memory
// reads, a shuffle (backward: two), ten adds and maxima, a 16-byte store; any other takes 45.
// Bound by the latency of a frame: 36 ns with the three warps of 240 states, 53 on average with the
// nine of 801, 62 with six and 64 x 1000 frames of 500 classes, whose 174 MB from DRAM and 86 MB to it
// are two thirds of what the memory does in that time.  Cells that no path can pass, a quarter of
// these grids, are neither stored nor read, and a warp without others sits out (67 and 99 us for
// 16 x 1500 frames with all of them; 86 and 124 with all arcs by the general expressions and rows
// requested and waited for by the warps that walk).  Two states per thread: slower; eight: 99 us.
// ---------------------------------------------------------------------------
// The largest of three, NaN apart like fmaxf: one instruction.
__device__ __forceinline__ float Max3(float a, float b, float c) {
  float m;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}

// Whether a graph alternates, like those of k2.ctc_graph: every state but the final one has a
// self-loop and an arc from the state before it, all arcs score zero, and the states of even
// number share one label and have no arc from two states before.  (prev + 0) + dense is
// prev + dense.
template <bool kAlternates>
struct VitForm {
  static constexpr bool value = kAlternates;
};

constexpr int kVitMaxBatches = 4;  // batches of rows in flight
constexpr int kVitMaxWarps = 12;

// K consecutive values, stored or read as one word.
template <int K>
struct VitPack;
template <>
struct VitPack<2> {
  using type = float2;
};
template <>
struct VitPack<4> {
  using type = float4;
};
template <int K>
__device__ __forceinline__ void VitStore(float *p, const float (&v)[K]) {
  typename VitPack<K>::type t;
  memcpy(&t, v, sizeof(t));
  *reinterpret_cast<typename VitPack<K>::type *>(p) = t;
}
template <int K>
__device__ __forceinline__ void VitLoad(const float *p, float (&v)[K]) {
  const typename VitPack<K>::type t = *reinterpret_cast<const typename VitPack<K>::type *>(p);
  memcpy(v, &t, sizeof(t));
}

// The log-probs of the states' labels, in the layout of the grids: row r of a sequence at row r of
// its grid, -inf for a label without a column.  Bound by the 32-byte sectors of the log-probs
// that it touches.
constexpr int kGatherRows = 16;  // per CTA: two per warp
__global__ void __launch_bounds__(256)
BandGather(const BandInfo *infos, const BandState *tab, const float *lp, int32_t C,
           float *__restrict__ by_state) {
  __shared__ int32_t label_sh[kBandMaxStates];
  WaitForPrevious();
  const BandInfo f = infos[blockIdx.y];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t r0 = blockIdx.x * kGatherRows, r1 = min(r0 + kGatherRows, f.frames), S = f.num_states;
  if (S == 0 || r0 >= r1) return;
  for (int32_t s = threadIdx.x; s < S; s += 256) label_sh[s] = tab[f.state_off + s].label;
  __syncthreads();
  for (int32_t r = r0 + warp; r < r1; r += 8) {
    const float *in = lp + (int64_t)(f.lp_row + r) * C;
    float *out = by_state + f.grid_off + (int64_t)r * f.pitch;
    for (int32_t s0 = lane; s0 < S; s0 += 256) {
      float x[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int32_t s = s0 + 32 * k, label = s < S ? label_sh[s] : -1;
        x[k] = label >= 0 && label < C ? in[label] : -INFINITY;
      }
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (s0 + 32 * k < S) out[s0 + 32 * k] = x[k];
    }
  }
}

// A batch of rows [off, end), in floats from the 16-byte boundary src.  Where the copy between
// boundaries would leave the matrix [first, last), up to three elements are copied one by one.
__device__ __forceinline__ void CopyAtEdge(const float *first, const float *last, const float *src,
                                        int32_t off, int32_t end, float *dst, uint64_t *bar) {
  int32_t from = 0, to = (end + 3) & ~3;
  if (src < first || src + to > last) {
    if (src < first) from = 4;
    if (src + to > last) to = max(to - 4, from);
    for (int32_t k = off; k < min(from, end); ++k) dst[k] = src[k];
    for (int32_t k = max(to, off); k < end; ++k) dst[k] = src[k];
    // (the slot's next batch overwrites them)
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  MbarArriveExpectTx(bar, (unsigned)(to - from) * 4u);
  if (to > from) BulkCopyG2S(dst + from, src + from, (unsigned)(to - from) * 4u, bar);
}

// The frames of a batch, from row `row` on: `step` consumes the scores that `load` reads, which are
// read four frames ahead of it.
template <int kX, typename Load, typename Step>
__device__ __forceinline__ void VitFrames(int32_t n, const float *row, int32_t width,
                                          const Load &load, const Step &step) {
  constexpr int kAhead = 4, kFull = 16;
  if (n == kFull) {
    float x[2][kAhead][kX];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) load(row + u * width, x[0][u]);
#pragma unroll
    for (int g = 0; g < kFull / kAhead; ++g) {
      row += kAhead * width;
      if (g + 1 < kFull / kAhead) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) load(row + u * width, x[(g + 1) & 1][u]);
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) step(x[g & 1][u]);
    }
  } else {
#pragma unroll 4
    for (int32_t r = 0; r < n; ++r, row += width) {
      float x[kX];
      load(row, x);
      step(x);
    }
  }
}

// kByState: `lp` holds scores by state (BandGather) in the layout of the grids instead of
// log-prob rows of C columns: a thread reads its states' scores in one word.  With 5000 columns
// the copies of whole rows bounded the kernel (170 us for 500 frames); by state it takes 43,
// and BandGather 36.
// kEdge: the matrix starts or ends between two 16-byte boundaries.  (An instance of its own: a test
// per batch in the other one took 5 us of 1000 frames.)
template <bool kByState, bool kEdge>
__global__ void __launch_bounds__(32 * (kVitMaxWarps + 1), 1)
BandViterbi(const BandInfo *infos, const BandState *tab, const float *lp, int64_t lp_rows,
            int32_t C, float *__restrict__ vf, float *__restrict__ vb, int32_t F, int32_t nbatch,
            int32_t slot_floats, int32_t xch_pad, int32_t wait_limit,
            int32_t *__restrict__ status) {
  constexpr int K = kVitK;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[kVitMaxBatches];
  __shared__ int32_t any_late;
  constexpr unsigned kAll = 0xffffffffu;
  const int dir = blockIdx.x;
  WaitForPrevious();
  LetNextStart();
  const BandInfo f = infos[blockIdx.y];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int32_t S = f.num_states, T = f.frames, pitch = f.pitch;
  if (S == 0) return;
  const int32_t H = 2 * F / K;      // lanes that recompute the neighbour's states
  const int32_t own = 32 - H;       // lanes whose states this warp owns
  const int32_t width = kByState ? pitch : C;              // floats of a row
  float *ring = reinterpret_cast<float *>(smem_raw);       // [nbatch][slot_floats]: F rows
  float *xch = ring + (size_t)nbatch * slot_floats;        // [2][xch_pad], state s at s + 2F
  if (tid == 0) {
    for (int st = 0; st < nbatch; ++st) MbarInit(&full[st], 1);
    MbarInitFence();
    any_late = 0;
  }
  for (int32_t k = tid; k < 2 * xch_pad; k += blockDim.x) xch[k] = -INFINITY;
  __syncthreads();
  const int32_t num_batches = (T + F - 1) / F;
  const float *lp0 = kByState ? lp + f.grid_off : lp + (int64_t)f.lp_row * C;
  // A row may start anywhere (C need not be a multiple of four): a batch is copied from the
  // 16-byte boundary at or before its first element to the one at or after its last (which kEdge
  // keeps inside the matrix).
  const uint32_t lp0_words = (uint32_t)(reinterpret_cast<uintptr_t>(lp0) >> 2);
  auto words_off = [&](int32_t r) {
    return kByState ? 0 : (int32_t)((lp0_words + (uint32_t)r * (uint32_t)width) & 3u);
  };
  int32_t issued = 0;
  int32_t next_slot = 0;
  auto issue = [&]() {  // one thread only: the rows of the next batch into the next slot
    if (issued >= num_batches) return;
    const int32_t q = issued;
    // batch q: forward rows [qF, min((q+1)F, T)); backward rows [max(T-(q+1)F, 0), T-qF)
    const int32_t r0 = dir == 0 ? q * F : max(T - (q + 1) * F, 0);
    const int32_t r1 = dir == 0 ? min((q + 1) * F, T) : T - q * F;
    const int32_t off = words_off(r0);
    const int32_t slot = next_slot;
    next_slot = slot + 1 == nbatch ? 0 : slot + 1;
    if (kEdge) {
      CopyAtEdge(lp, lp + lp_rows * width, lp0 + (int64_t)r0 * width - off, off,
                 (r1 - r0) * width + off, ring + (size_t)slot * slot_floats, &full[slot]);
    } else {
      const unsigned bytes = (((unsigned)(r1 - r0) * (unsigned)width + (unsigned)off + 3u) & ~3u) * 4u;
      MbarArriveExpectTx(&full[slot], bytes);
      BulkCopyG2S(ring + (size_t)slot * slot_floats, lp0 + (int64_t)r0 * width - off, bytes,
                  &full[slot]);
    }
    ++issued;
  };
  bool late = false;
  // The last warp requests the rows and waits for them on behalf of all: the barrier before batch q
  // says that its rows are there and that every warp has finished batch q - 1.
  const bool producer = warp == (int)(blockDim.x >> 5) - 1;
  if (producer) {
    if (lane == 0)
      for (int32_t q = 0; q < nbatch; ++q) issue();
    __syncthreads_and(1);
    int32_t slot = 0;
    unsigned parity = 0;
    for (int32_t q = 0; q < num_batches; ++q) {
      if (!late) late = !WaitSlot(&full[slot], parity, wait_limit);
      __syncthreads();
      if (q > 0 && lane == 0 && !late) issue();  // into the slot of batch q - 1
      if (++slot == nbatch) {
        slot = 0;
        parity ^= 1u;
      }
    }
    if (dir == 0) __syncthreads();
  } else {

  // first state of this lane: forward, the recomputed states come first; backward, last
  const int32_t s0 = warp * own * K + (dir == 0 ? (lane - H) * K : lane * K);
  const bool mine = dir == 0 ? lane >= H : lane < own;   // a lane that owns its states
  const bool stores = mine && s0 < pitch;
  float *grid = (dir == 0 ? vf : vb) + f.grid_off + s0;
  // What is stored: four states s0 .. s0 + 3 of level l of R = T + 1 where one of them can lie on a
  // path (arcs advance by at most two states: S - 1 - 2 (R - l) <= s <= 2 l).  BandPrep reads no
  // others.  `at` is s0 - 2 l less the least that it may be.
  const int32_t least = S - 1 - 2 * (T + 1) - (K - 1);
  int32_t at = s0 - least - (dir == 0 ? 0 : 2 * (T + 1));
  const uint32_t most = stores && least <= 0 ? (uint32_t)-least + 1u : 0u;
  // Whether a warp has such states on any of the levels l0 .. l1; if not it sits out: its scores
  // stay -inf, or nobody asks for them any more.
  const int32_t warp_s0 = s0 - lane * K;
  auto on_paths = [&](int32_t l0, int32_t l1) {
    return warp_s0 <= 2 * l1 && warp_s0 + 32 * K - 1 >= S - 1 - 2 * (T + 1 - l0);
  };
  float v[K];
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = 0.0f;
  // exchange of boundary states: owners publish, recomputing lanes pick up
  const int32_t lead = 2 * F;
  auto exchange = [&](int32_t which) {
    float *x = xch + (size_t)which * xch_pad + lead;
    if (mine && s0 < xch_pad - lead - (K - 1)) VitStore<K>(x + s0, v);
    __syncthreads();
    if (!mine && s0 + lead >= 0 && s0 < xch_pad - lead - (K - 1)) VitLoad<K>(x + s0, v);
  };
  // The values next to a lane's states come from its neighbour.  What lane 0 (forward) or 31
  // (backward) gets instead is not a neighbour's: either it recomputes another warp's states,
  // of which the outermost two are lost per frame, or there is no such state and every score
  // into it is -inf.
  if (dir == 0) {
    // ---- forward: state s from s, s - 1, s - 2 ----------------------------------
    float w0[K], w1[K], w2[K];     // on the frames; -inf for a state whose label has no column
    float f0[K], f1[K], f2[K];     // on the implied final row: only arcs labelled -1 score
    int32_t col[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int32_t s = s0 + k;
      w0[k] = w1[k] = w2[k] = f0[k] = f1[k] = f2[k] = -INFINITY;
      col[k] = 0;
      if (s >= 0 && s < S) {
        const BandState t = tab[f.state_off + s];
        if (t.label >= 0 && t.label < C) {
          col[k] = t.label;
          w0[k] = t.w[0];
          w1[k] = t.w[1];
          w2[k] = t.w[2];
        } else if (t.label == -1) {
          f0[k] = t.w[0];
          f1[k] = t.w[1];
          f2[k] = t.w[2];
        }
      }
      v[k] = s == 0 ? 0.0f : -INFINITY;
    }
    if ((uint32_t)at < most) VitStore<K>(grid, v);
    auto step = [&](auto alternates, const float (&a0)[K], const float (&a1)[K],
                    const float (&a2)[K], const float (&x)[K]) {
      const float h1 = __shfl_up_sync(kAll, v[K - 1], 1);
      float nv[K];
      if (alternates.value) {
#pragma unroll
        for (int k = 0; k < K; k += 2) {
          const float b = k ? v[k ? k - 1 : 0] : h1;  // of the state before these two
          nv[k] = __fadd_rn(fmaxf(v[k], b), x[k]);
          nv[k + 1] = __fadd_rn(Max3(v[k + 1], v[k], __fadd_rn(b, a2[k + 1])), x[k + 1]);
        }
      } else {
        const float h2 = __shfl_up_sync(kAll, v[K - 2], 1);
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const float a = v[k];
          const float b = k >= 1 ? v[k >= 1 ? k - 1 : 0] : h1;
          const float c = k >= 2 ? v[k >= 2 ? k - 2 : 0] : (k == 1 ? h1 : h2);
          nv[k] = __fadd_rn(
              Max3(__fadd_rn(a, a0[k]), __fadd_rn(b, a1[k]), __fadd_rn(c, a2[k])), x[k]);
        }
      }
#pragma unroll
      for (int k = 0; k < K; ++k) v[k] = nv[k];
      grid += pitch;
      at -= 2;
      if ((uint32_t)at < most) VitStore<K>(grid, v);
    };
    int32_t xpar = 0, slot = 0;
    auto walk = [&](auto alternates) {
      auto load = [&](const float *row, float (&x)[K]) {
        if (kByState) {
          VitLoad<K>(row + col[0], x);
        } else {
#pragma unroll
          for (int k = 0; k < K; ++k)
            x[k] = alternates.value && k >= 2 && k % 2 == 0 ? x[0] : row[col[k]];
        }
      };
      for (int32_t q = 0; q < num_batches; ++q) {
        exchange(xpar);
        xpar ^= 1;
        const int32_t nf = min(F, T - q * F);
        const float *rowbuf = ring + (size_t)slot * slot_floats + words_off(q * F);
        if (++slot == nbatch) slot = 0;
        if (!on_paths(q * F, q * F + nf)) {
          grid += (int64_t)nf * pitch;
          at -= 2 * nf;
          continue;
        }
        VitFrames<K>(nf, rowbuf, width, load,
                     [&](const float (&x)[K]) { step(alternates, w0, w1, w2, x); });
      }
    };
    // (what the final state of a graph that alternates is given on the frames, where no arc
    // enters it, goes to no other state, and the backward score that it is added to is -inf)
    bool alternates = true;
    const int32_t even_label = tab[f.state_off].label;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int32_t s = s0 + k;
      if (s < 0 || s >= S) continue;
      const bool last = s == S - 1 && w0[k] == -INFINITY && w1[k] == -INFINITY && w2[k] == -INFINITY;
      const bool plain = w0[k] == 0.0f && (s == 0 || w1[k] == 0.0f) &&
                         (w2[k] == -INFINITY || (k % 2 == 1 && w2[k] == 0.0f));
      alternates &= (last || plain) && (k % 2 == 1 || col[k] == even_label);
    }
    if (kByState) col[0] = min(max(s0, 0), pitch - K);
    if (__syncthreads_and(alternates)) walk(VitForm<true>{});
    else walk(VitForm<false>{});
    // the implied final row: level T + 1
    exchange(xpar);
    {
      float x[K];
#pragma unroll
      for (int k = 0; k < K; ++k) x[k] = 0.0f;
      step(VitForm<false>{}, f0, f1, f2, x);
    }
  } else {
    // ---- backward: state s to s, s + 1, s + 2 -----------------------------------
    float wo[K][3];   // score of the arc s -> s + d on the frames (-inf: its label has no column)
    float fo[K][3];   // on the implied final row
    int32_t col[K + 2];   // of states s0 .. s0 + K + 1
    float skip[K + 2];    // score of the arc that enters the state from two states before
    bool alternates = true;
    const int32_t even_label = tab[f.state_off].label;
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int d = 0; d < 3; ++d) wo[k][d] = fo[k][d] = -INFINITY;
#pragma unroll
    for (int k = 0; k < K + 2; ++k) {
      const int32_t s = s0 + k;
      col[k] = 0;
      BandState t;
      t.w[0] = t.w[1] = t.w[2] = -INFINITY;
      t.label = kNoLabel;
      if (s < S) t = tab[f.state_off + s];
      const bool frame_label = t.label >= 0 && t.label < C;
      if (frame_label) col[k] = t.label;
      skip[k] = frame_label ? t.w[2] : -INFINITY;
      if (s < S && (frame_label || s < S - 1))
        alternates &= frame_label && t.w[0] == 0.0f && (s == 0 || t.w[1] == 0.0f) &&
                      (t.w[2] == -INFINITY || (k % 2 == 1 && t.w[2] == 0.0f));
      if (s < S && k % 2 == 0) alternates &= frame_label && t.label == even_label;
#pragma unroll
      for (int d = 0; d < 3; ++d)
        if (k - d >= 0 && k - d < K) {
          if (frame_label) wo[k - d >= 0 ? k - d : 0][d] = t.w[d];
          else if (t.label == -1) fo[k - d >= 0 ? k - d : 0][d] = t.w[d];
        }
    }
    if (kByState) {  // (states at and behind S score -inf: any column of the row will do)
      col[0] = min(s0, pitch - K);
      col[1] = min(s0 + K, pitch - 2);
    }
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = (s0 + k == S - 1) ? 0.0f : -INFINITY;
    grid += (int64_t)(T + 1) * pitch;
    if ((uint32_t)at < most) VitStore<K>(grid, v);
    // A graph that alternates: what a state scores with its label's score is needed once, by it and
    // by its two predecessors, which get it by shuffles.
    auto short_step = [&](const float (&x)[K]) {
      float g[K + 2];
#pragma unroll
      for (int k = 0; k < K; ++k) g[k] = __fadd_rn(v[k], x[k]);
      g[K] = __shfl_down_sync(kAll, g[0], 1);
      g[K + 1] = __shfl_down_sync(kAll, g[1], 1);
#pragma unroll
      for (int k = 0; k < K; k += 2) {
        v[k] = fmaxf(g[k], g[k + 1]);
        v[k + 1] = Max3(g[k + 1], g[k + 2], __fadd_rn(g[k + 3], skip[k + 3]));
      }
      grid -= pitch;
      at += 2;
      if ((uint32_t)at < most) VitStore<K>(grid, v);
    };
    auto step = [&](const float (&w)[K][3], const float (&x)[K + 2]) {
      const float g1 = __shfl_down_sync(kAll, v[0], 1), g2 = __shfl_down_sync(kAll, v[1], 1);
      float nv[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const float a = v[k];
        const float b = k + 1 < K ? v[k + 1 < K ? k + 1 : 0] : g1;
        const float c = k + 2 < K ? v[k + 2 < K ? k + 2 : 0] : (k + 2 == K ? g1 : g2);
        nv[k] = Max3(__fadd_rn(__fadd_rn(a, w[k][0]), x[k]),
                     __fadd_rn(__fadd_rn(b, w[k][1]), x[k + 1]),
                     __fadd_rn(__fadd_rn(c, w[k][2]), x[k + 2]));
      }
#pragma unroll
      for (int k = 0; k < K; ++k) v[k] = nv[k];
      grid -= pitch;
      at += 2;
      if ((uint32_t)at < most) VitStore<K>(grid, v);
    };
    {  // level T from level T + 1 through the implied final row (nothing to exchange yet:
       // only the final state is not -inf, and every lane knows it)
      float x[K + 2];
#pragma unroll
      for (int k = 0; k < K + 2; ++k) x[k] = 0.0f;
      step(fo, x);
    }
    int32_t xpar = 0, slot = 0;
    auto walk = [&](auto alternates) {
      constexpr int kX = decltype(alternates)::value ? K : K + 2;
      auto load = [&](const float *row, float (&x)[kX]) {
        if (kByState) {
          float lo[K], hi[2];
          VitLoad<K>(row + col[0], lo);
#pragma unroll
          for (int k = 0; k < K; ++k) x[k] = lo[k];
          if (kX > K) {
            VitLoad<2>(row + col[1], hi);
            x[kX - 2] = hi[0];
            x[kX - 1] = hi[1];
          }
        } else {
#pragma unroll
          for (int k = 0; k < kX; ++k)
            x[k] = alternates.value && k >= 2 && k % 2 == 0 ? x[0] : row[col[k]];
        }
      };
      for (int32_t q = 0; q < num_batches; ++q) {
        exchange(xpar);
        xpar ^= 1;
        const int32_t r1 = T - q * F, r0 = max(T - (q + 1) * F, 0);
        const float *rowbuf =
            ring + (size_t)slot * slot_floats + words_off(r0) + (size_t)(r1 - 1 - r0) * width;
        if (++slot == nbatch) slot = 0;
        if (!on_paths(r0, r1)) {
          grid -= (int64_t)(r1 - r0) * pitch;
          at += 2 * (r1 - r0);
          continue;
        }
        VitFrames<kX>(r1 - r0, rowbuf, -width, load, [&](const float (&x)[kX]) {  // level r
          if constexpr (decltype(alternates)::value) short_step(x);         // from level r + 1
          else step(wo, x);
        });
      }
    };
    if (__syncthreads_and(alternates)) walk(VitForm<true>{});
    else walk(VitForm<false>{});
  }
  }  // not the producer
  if (late) any_late = 1;
  __syncthreads();
  if (any_late) {
    // A copy did not arrive in time: the grids hold garbage.  Say so, and let the copies
    // that are still in flight towards this CTA's shared memory land before it retires.
    if (producer && lane == 0) {
      atomicOr(status, kStatusLate);
      for (int32_t q = max(0, issued - nbatch); q < issued; ++q)
        WaitSlot(&full[q % nbatch], (unsigned)(q / nbatch) & 1u, kDrainPolls);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Delay penalty: what the score of an arc that survives gains on frame t.  flags[arc] says
// which arcs are penalised.  Pruning does not see it.
// A path that is n symbols ahead of another has gained n penalties; where posteriors are so flat
// that such paths share a level for long, the graph goes to the (mantissa, exponent) recursion.
// ---------------------------------------------------------------------------
struct DelaySpec {
  float penalty;
  const uint8_t *flags;  // [arcs]
  __device__ __forceinline__ float Of(int32_t t, int32_t frames) const {
    return -penalty * (float)(t - (frames >> 1));
  }
};

__global__ void PenaltyFlags(const BandState *__restrict__ tab, const BandArc *__restrict__ tabf,
                             int32_t num_states, const uint8_t *__restrict__ repeat,
                             const int32_t *__restrict__ aux, uint8_t *__restrict__ flags) {
  const int32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= num_states) return;
  const int32_t label = tab[idx].label;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int32_t arc = tabf[(int64_t)idx * 3 + d].arc;
    if (arc < 0) continue;
    const int32_t symbol = repeat != nullptr ? (repeat[arc] ? 0 : label) : aux[arc];
    flags[arc] = symbol != 0 && symbol != -1;
  }
}

// ---------------------------------------------------------------------------
// Keep tests and lists.  grid = (chunks of kPrepLevels levels, pairs), kPrepWarps warps per CTA,
// which looks at the chunk's levels and the level on either side of them:
//   1. a warp per level, four states per lane at a time: state s of level l survives iff
//      vf[l][s] + vb[l][s] > cutoff (intersect_dense.cu:289-296); none does where BandViterbi stored
//      nothing.  Shared memory keeps, per
//      four states, their keep bits and the number of surviving states before them (together:
//      the list position of a state), and the surviving states in order;
//   2. a warp per 32 entries of a level: the reference's arc tests (intersect_dense.cu:430-471)
//      against the states of the level before and the dense score of the state's label give
//      the entering-arc bits, the factors and where the sources are; also (bits only) for the
//      level behind the chunk;
//   3. likewise: where the destinations are; an arc leaving an entry is an entering arc of the
//      next level seen from its source.
// Per level the result is the compact list of surviving states: a BandItem (label, state,
// bits) and a BandFactor per entry.  The passes are a few independent loads deep and all of a
// CTA's levels are in flight together; what bounds them is the latency of those loads where
// the batch is small and the traffic (the two grids once, 32 + 8 bytes per padded entry)
// where it is large.  (A warp that went through eight levels one after the other, behind a
// separate kernel for the keep bits, took 103 + 38 us at 64 x 1000 frames of up to 501 states;
// this takes 80, 212 MB read and 52 MB written.)
// totals[0] += surviving states, totals[2] += the arcs leaving them (the
// sizes the beam reduction looks at, intersect_dense.cu:289-320).  unfit[i] is set when the
// list recursion cannot take graph i: a score outside its arithmetic, or a level with
// more than kMaxListed surviving states.
// ---------------------------------------------------------------------------
constexpr float kMinLeanDense = -60.0f;   // dense score of a surviving arc
constexpr int32_t kMaxLeanArcExp = 60, kMinLeanArcExp = -90;  // binary exponent of exp(arc score)
constexpr int kPrepWarps = 9;             // 18 levels: two each
constexpr int kPrepSpan = kPrepLevels + 2;

// states of a graph rounded up to whole groups of 128 (four per lane of a warp)
__host__ __device__ static inline int32_t PrepPad(int32_t states) { return (states + 127) & ~127; }
static size_t BandPrepSmem(int32_t max_states) {
  return (size_t)kPrepSpan * (PrepPad(max_states) / 4 * 2 + PrepPad(max_states) * 3);
}

template <bool kDelay>
__global__ void __launch_bounds__(32 * kPrepWarps, 3)
BandPrep(const BandInfo *infos, const int32_t *a_row_splits2, const BandState *tab,
         const BandArc *tabf, const float *lp, int32_t C, const float *by_state, const float *vf,
         const float *vb, float beam, BandItem *__restrict__ items,
         BandFactor *__restrict__ factors, int2 *__restrict__ lists,
         int32_t *__restrict__ chunk_r, unsigned long long *__restrict__ totals,
         int32_t *__restrict__ unfit, int32_t count_arcs, DelaySpec delay) {
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int32_t longest_sh, risky_sh;
  __shared__ uint32_t counts_sh[2];
  __shared__ int32_t n_sh[kPrepSpan];
  const int32_t i = blockIdx.y;
  WaitForPrevious();
  const BandInfo f = infos[i];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int32_t S = f.num_states, T = f.frames, pitch = f.pitch;
  const int32_t a = blockIdx.x * kPrepLevels;  // the chunk's levels: a .. b - 1
  if (S == 0 || a > T + 1) return;
  const int32_t b = min(a + kPrepLevels, T + 2);
  const int32_t P = PrepPad(S);
  // level l of the chunk is row l - a + 1
  uint16_t *cells = reinterpret_cast<uint16_t *>(smem_raw);            // [span][P / 4]
  uint16_t *list = cells + kPrepSpan * (P / 4);                        // [span][P]
  unsigned char *inbs = reinterpret_cast<unsigned char *>(list + kPrepSpan * P);  // likewise
  const float *fg = vf + f.grid_off, *bg = vb + f.grid_off;
  if (tid == 0) {
    longest_sh = risky_sh = 0;
    counts_sh[0] = counts_sh[1] = 0;
  }
  float cutoff;
  {
    // (without a path BandViterbi stored neither)
    const bool path = S - 1 <= 2 * (T + 1);
    const float start = path ? bg[0] : -INFINITY,
                end = path ? fg[(int64_t)(T + 1) * pitch + (S - 1)] : -INFINITY;
    cutoff = __fsub_rn(start < end ? start : end, beam);
  }
  __syncthreads();
  // ---- 1. surviving states ----------------------------------------------------------------
  uint32_t n_cand = 0;
  for (int32_t row = warp; row < kPrepSpan; row += kPrepWarps) {
    const int32_t l = a - 1 + row;
    const bool there = l >= 0 && l <= b && l <= T + 1;
    const float *fr = fg + (int64_t)l * pitch + 4 * lane, *br = bg + (int64_t)l * pitch + 4 * lane;
    // the states that BandViterbi stored
    const int32_t first = S - 1 - 2 * (T + 1 - l) - 3, last = min(2 * l, S - 1);
    int32_t n = 0;
    for (int32_t g0 = 0; g0 < P; g0 += 512) {  // up to four groups of 128 states
      float4 x[4], y[4];
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int32_t s = g0 + 128 * g + 4 * lane;
        const bool in = there && s >= first && s <= last;  // (pitch covers the four states)
        x[g] = y[g] = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        if (in) {
          x[g] = *reinterpret_cast<const float4 *>(fr + g0 + 128 * g);
          y[g] = *reinterpret_cast<const float4 *>(br + g0 + 128 * g);
        }
      }
      uint32_t bits = 0, counts = 0;  // byte g: the keep bits of group g, how many they are
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        uint32_t m = 0;
        if (__fadd_rn(x[g].x, y[g].x) > cutoff) m |= 1u;
        if (__fadd_rn(x[g].y, y[g].y) > cutoff) m |= 2u;
        if (__fadd_rn(x[g].z, y[g].z) > cutoff) m |= 4u;
        if (__fadd_rn(x[g].w, y[g].w) > cutoff) m |= 8u;
        bits |= m << (8 * g);
        counts |= __popc(m) << (8 * g);
      }
      uint32_t incl = counts;  // at most 128 in a byte
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(kAll, incl, d);
        if (lane >= d) incl += o;
      }
      const uint32_t sums = __shfl_sync(kAll, incl, 31);
      incl -= counts;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        if (g0 + 128 * g >= P) break;  // uniform
        const uint32_t m = (bits >> (8 * g)) & 15u;
        const int32_t at = n + (int32_t)((incl >> (8 * g)) & 0xffu);
        const int32_t s = g0 + 128 * g + 4 * lane;
        cells[(row * P + s) >> 2] = (uint16_t)(at << 4 | m);
        const int32_t total = (int32_t)((sums >> (8 * g)) & 0xffu);
        n += total;
        if (total == 0) continue;  // uniform
        uint16_t *out = list + row * P + at;
        if (m & 1u) *out++ = (uint16_t)s;
        if (m & 2u) *out++ = (uint16_t)(s + 1);
        if (m & 4u) *out++ = (uint16_t)(s + 2);
        if (m & 8u) *out++ = (uint16_t)(s + 3);
        if (count_arcs && l >= a && l < b) {
          for (uint32_t r = m; r; r &= r - 1) {
            const int32_t idx = f.state_off + s + __ffs(r) - 1;
            n_cand += a_row_splits2[idx + 1] - a_row_splits2[idx];
          }
        }
      }
    }
    if (lane == 0) {
      n_sh[row] = n;
      if (l >= a && l < b) {
        atomicMax(&longest_sh, n);
        atomicAdd(&counts_sh[0], (uint32_t)n);
      }
    }
  }
  if (count_arcs) {  // uniform; the host leaves it out when no count could reach max_arcs
    n_cand = __reduce_add_sync(kAll, n_cand);
    if (lane == 0) atomicAdd(&counts_sh[1], n_cand);
  }
  __syncthreads();
  // the longest list of the chunk's levels decides how many entries each of them gets
  // (pitch >= padded), they lie `padded` entries apart from the start of the chunk;
  // lists[level] = (start, size)
  const int32_t longest = longest_sh;
  const int32_t blocks = longest / 32 + 1, padded = 32 * blocks;
  if (tid == 0) {
    chunk_r[f.level_off + a] = blocks;
    if (counts_sh[0]) atomicAdd(&totals[0], (unsigned long long)counts_sh[0]);
    if (counts_sh[1]) atomicAdd(&totals[2], (unsigned long long)counts_sh[1]);
  }
  if (tid < b - a)
    lists[f.level_off + a + tid] = make_int2(a * pitch + tid * padded, n_sh[tid + 1]);
  // position of state s (in 0 .. P - 1) on the level of `row`, -1 if it does not survive there
  auto position = [&](int32_t row, int32_t s) {
    const uint32_t cell = cells[(row * P + s) >> 2], bit = 1u << (s & 3);
    return cell & bit ? (int32_t)((cell >> 4) + __popc(cell & (bit - 1u))) : -1;
  };
  // ---- 2. entering arcs -------------------------------------------------------------------
  const float *lp0 = lp + (int64_t)f.lp_row * C;
  bool risky = longest > kMaxListed;
  {
    // a warp's two levels together, 32 entries of each at a time, for their loads to overlap
    static_assert(2 * kPrepWarps >= kPrepLevels + 1, "two levels per warp");
    const float *xrow[2], *brow[2], *frow[2];
    char *level[2];
    int32_t n[2], row[2];
    bool own[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int32_t k = warp + u * kPrepWarps, l = a + k;
      row[u] = k + 1;
      own[u] = l < b;
      n[u] = k <= b - a && l <= T + 1 ? n_sh[row[u]] : 0;
      xrow[u] = nullptr;
      if (l >= 1 && l <= T)
        xrow[u] = by_state != nullptr ? by_state + f.grid_off + (int64_t)(l - 1) * pitch
                                      : lp0 + (int64_t)(l - 1) * C;
      brow[u] = bg + (int64_t)l * pitch;
      frow[u] = fg + (int64_t)(l - 1) * pitch;
      level[u] = reinterpret_cast<char *>(factors + f.grid_off + (int64_t)a * pitch + k * padded) +
                 lane * 16;
    }
    const BandState *tab_f = tab + f.state_off;
    // (the level behind the chunk may have more entries than the chunk's)
    const int32_t upto = max(own[0] ? padded : 0, max(own[1] ? padded : n[1], n[0]));
    for (int32_t j = lane; j - lane < upto; j += 32) {
      int32_t s[2];
      bool in[2];
      BandState st[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        in[u] = j < n[u];
        s[u] = in[u] ? list[row[u] * P + j] : 0;
        if (in[u]) st[u] = tab_f[s[u]];
      }
      float x[2], bc[2], sf[2][3];
      uint32_t src[2], kept[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        kept[u] = src[u] = 0;
        x[u] = bc[u] = 0.0f;
        if (in[u] && row[u] + a >= 2) {
          if (xrow[u] == nullptr)  // the implied final row
            x[u] = st[u].label == -1 ? 0.0f : -INFINITY;
          else if (by_state != nullptr)
            x[u] = xrow[u][s[u]];
          else
            x[u] = st[u].label >= 0 && st[u].label < C ? xrow[u][st[u].label] : -INFINITY;
          bc[u] = brow[u][s[u]];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            const int32_t at = s[u] >= d ? position(row[u] - 1, s[u] - d) : -1;
            sf[u][d] = -INFINITY;
            if (at >= 0) {
              kept[u] |= 1u << d;
              src[u] |= ((uint32_t)at & 0xffu) << (8 * d);
              sf[u][d] = frow[u][s[u] - d];
            }
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        double pw[3] = {0.0, 0.0, 0.0};
        uint32_t from = 0;
        if (in[u]) {
          uint32_t inb = 0;
#pragma unroll
          for (int d = 0; d < 3; ++d)
            if (((kept[u] >> d) & 1u) &&
                __fadd_rn(__fadd_rn(sf[u][d], __fadd_rn(st[u].w[d], x[u])), bc[u]) > cutoff)
              inb |= 1u << d;
          inbs[row[u] * P + j] = (unsigned char)inb;
          if (own[u] && inb) {
            const double p = exp((double)x[u]);
            // outside what doubles with a scale that follows the data every few
            // levels hold: such graphs go to the (mantissa, exponent) recursion
            if (!(x[u] >= kMinLeanDense)) risky = true;
#pragma unroll
            for (int d = 0; d < 3; ++d)
              if ((inb >> d) & 1u) {
                from |= src[u] & (0xffu << (8 * d));
                pw[d] = p;
                // (the factor of a score of zero is one)
                if (kDelay || st[u].w[d] != 0.0f) {
                  const BandArc arc = tabf[(int64_t)(f.state_off + s[u]) * 3 + d];
                  pw[d] = arc.f * Pow2Clamp(arc.k) * p;
                  if (arc.k > kMaxLeanArcExp || arc.k < kMinLeanArcExp) risky = true;
                  if (kDelay) {
                    // the score as the lattice has it, a float
                    const int32_t l = a + row[u] - 1;
                    float sc = __fadd_rn(st[u].w[d], x[u]);
                    if (delay.flags[arc.arc]) sc = __fadd_rn(sc, delay.Of(l - 1, T));
                    pw[d] = exp((double)sc);
                    // what the limits above leave of a factor
                    if (!(pw[d] > 1e-52 && pw[d] < 1e52)) risky = true;
                  }
                }
              }
          }
        }
        if (own[u] && j < padded) {
          *reinterpret_cast<double2 *>(level[u]) = make_double2(pw[0], pw[1]);
          *reinterpret_cast<double *>(level[u] + padded * 16) = pw[2];
          *reinterpret_cast<uint32_t *>(level[u] + padded * 16 + 8) = from;
        }
        level[u] += 32 * 16;
      }
    }
  }
  if (risky) risky_sh = 1;
  __syncthreads();
  LetNextStart();
  // ---- 3. leaving arcs --------------------------------------------------------------------
  for (int32_t k = warp; k < b - a; k += kPrepWarps) {
    const int32_t row = k + 1, n = n_sh[row];
    const int64_t at = f.grid_off + (int64_t)a * pitch + k * padded;
    char *level = reinterpret_cast<char *>(factors + at) + padded * 16 + 12;
    const bool leaving = a + k <= T;
#pragma unroll 2
    for (int32_t j = lane; j < padded; j += 32) {
      uint32_t dst = kNoDst * 0x010101u;
      if (j < n) {
        const int32_t s = list[row * P + j];
        BandItem it;
        it.label = tab[f.state_off + s].label;
        uint32_t outb = 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const int32_t to = leaving && s + d < P ? position(row + 1, s + d) : -1;
          if (to >= 0 && ((inbs[(row + 1) * P + to] >> d) & 1u)) {
            outb |= 1u << d;
            dst ^= (kNoDst ^ ((uint32_t)to & 0xffu)) << (8 * d);
          }
        }
        it.s = (uint16_t)s;
        it.inb = (uint8_t)inbs[row * P + j];
        it.outb = (uint8_t)outb;
        items[at + j] = it;
      }
      *reinterpret_cast<uint32_t *>(level + j * 16) = dst;
    }
  }
  if (tid == 0 && risky_sh) atomicOr(&unfit[i], kUnfitFactors);
}

// ---------------------------------------------------------------------------
// alpha (dir 0) and beta (dir 1) over the lists.  grid = (2, pairs), up to kMaxRegs warps of a CTA
// walk: thread j holds entry j of the current level's list, which says at which POSITIONS of the
// previous list its neighbours are:
//   alpha_l[j] = sum_d pw_l[j][d] * alpha_{l-1}[src_l[j][d]]
//   beta_l[j]  = sum_d (pw_{l+1}[.][d] * beta_{l+1}[.]) at position dst_l[j][d]
// What bounds it is the latency of a level, in which a warp issues in order: one gather of three
// values from shared memory, two dependent multiply-adds, a store and a barrier of the warps that
// the chunk's lists need (none, with lists of up to 31 entries).  So these warps do nothing else,
// and what is not needed for the next level's values (the store to memory, the offsets and
// factors of the entries to come) is issued while the three values arrive.  Four more warps, the
// keepers, request the chunks, wait for them on behalf of all, look at the range of the values
// and write the exponents, a chunk behind.  A level takes 100 cycles forward, 135 backward:
// 73 us for 64 x 1000 frames, 99 for 16 x 1500 (91 and 130 with all of that in the same warps).
// Every level of a chunk of kPrepLevels levels has the same padded number of entries, so inside a
// chunk addresses advance by a constant.  No test: an absent neighbour is a padding entry,
// whose value is 0.  The chunks arrive in a ring in shared memory by one bulk copy each,
// requested chunks ahead.
// The values of a level are stored divided by 2^K; K changes every kRescale levels by the
// exponent of the largest value of the last of them.  A value that is not zero and
// below 2^-900 (or a value above 2^900) marks the graph in `unfit` for BandChainExact,
// like the graphs BandPrep marked, which return at once here.
// Outputs: alpha / beta at the list positions, K per level, tot[i], total[i].
// ---------------------------------------------------------------------------
constexpr int kRescale = 8;                     // levels between changes of the shared scale
constexpr int kChainSlots = 3;                  // chunks in flight
constexpr int kFacSlot = kPrepLevels * 32 * kMaxRegs;  // BandFactor entries of a chunk's levels
constexpr int kChainMaxChunks = 4096;           // of a graph: 65534 frames
constexpr int kSlotItems = kPrepLevels * 128;   // BandItem entries likewise (BandChainExact)

// The ring of chunks: lane 0 requests, every lane waits.
template <typename Item, int kCap>
struct ChunkRing {
  uint64_t *full;          // [kChainSlots]
  Item *slots;             // [kChainSlots][kCap]
  const Item *items0;      // the pair's lists
  const int2 *lst;         // (start, size) of every level, in shared memory
  int32_t pitch, L, num_chunks, dir, issued;
  __device__ __forceinline__ int32_t ChunkOf(int32_t q) const {
    return dir == 0 ? q : num_chunks - 1 - q;
  }
  // entries of a chunk's lists (they are contiguous from the chunk's start)
  __device__ __forceinline__ int32_t ChunkItems(int32_t c) const {
    const int32_t l1 = min((c + 1) * kPrepLevels, L) - 1;
    return lst[l1].x + lst[l1].y - c * kPrepLevels * pitch;
  }
  __device__ __forceinline__ void Issue() {  // lane 0: the next chunk into the next slot
    if (issued >= num_chunks) return;
    const int32_t c = ChunkOf(issued), slot = issued % kChainSlots;
    // a multiple of 16 bytes, at least 16, so that the copy is legal and the slot's barrier
    // completes once per use (a chunk starts on a multiple of four entries and has room for
    // at least four)
    constexpr int32_t kPer16 = sizeof(Item) >= 16 ? 1 : 16 / sizeof(Item);
    const int32_t n = max((min(ChunkItems(c), kCap) + kPer16 - 1) / kPer16 * kPer16, kPer16);
    const unsigned bytes = (unsigned)n * (unsigned)sizeof(Item);
    MbarArriveExpectTx(&full[slot], bytes);
    BulkCopyG2S(slots + (size_t)slot * kCap, items0 + (int64_t)c * kPrepLevels * pitch, bytes,
                &full[slot]);
    ++issued;
  }
  __device__ __forceinline__ void Drain() {  // lane 0, after giving up
    for (int32_t k = max(0, issued - kChainSlots); k < issued; ++k)
      WaitSlot(&full[k % kChainSlots], (unsigned)(k / kChainSlots) & 1u, kDrainPolls);
  }
};

// What a thread reads of its entry.
struct ChainRec {
  double p0, p1, p2;
  uint32_t at;  // positions: of the sources (forward) / destinations (backward)
};
template <int DIR, int kPer>
__device__ __forceinline__ ChainRec LoadRec(const char *r) {
  const double2 p01 = *reinterpret_cast<const double2 *>(r);
  const int4 q = *reinterpret_cast<const int4 *>(r + 16 * kPer);
  ChainRec x;
  x.p0 = p01.x;
  x.p1 = p01.y;
  x.p2 = __hiloint2double(q.y, q.x);
  x.at = DIR == 0 ? (uint32_t)q.z : (uint32_t)q.w;
  return x;
}

// Values of two levels, by list position: forward alpha; backward the three products pw[d] *
// beta, which is what the entries of the level below add up.  Position kNoDst is always zero.
struct ChainValues {
  double v[2][3][256];
};

// One thread's state of the walk.
struct ChainState {
  double acc, scale;
  int32_t Ksh;      // the level's values are stored divided by 2^Ksh
  int32_t hm;       // largest high word when it was last asked for, of this warp's values
};

// Shared-memory offsets of the values that an entry adds up, in a ChainValues buffer.
struct ChainFrom {
  uint32_t at[3];
};
template <int DIR>
__device__ __forceinline__ ChainFrom FromOf(uint32_t at) {
  ChainFrom a;
  a.at[0] = (at << 3) & 0x7f8u;
  a.at[1] = ((at >> 5) & 0x7f8u) + (DIR == 0 ? 0 : 2048);
  a.at[2] = ((at >> 13) & 0x7f8u) + (DIR == 0 ? 0 : 4096);
  return a;
}

__device__ __forceinline__ double LoadValue(unsigned smem) {
  double x;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x) : "r"(smem) : "memory");
  return x;
}
__device__ __forceinline__ void StoreValue(unsigned smem, double x) {
  asm volatile("st.shared.f64 [%0], %1;" ::"r"(smem), "d"(x) : "memory");
}

// The scale that the values of the next group of levels are multiplied with.
__device__ __forceinline__ void ChainRescale(int32_t hm, ChainState &st) {
  const int32_t e = hm > 0 ? (hm >> 20) - 1023 : 0;
  st.Ksh += e;
  st.scale = __longlong_as_double((long long)(1023 - e) << 52);
}

template <int kBuf>
struct ChainBuf {
  static constexpr int value = kBuf;
};

template <int kWarps>
__device__ __forceinline__ void ChainSync() {
  if (kWarps == 1) __syncwarp();
  else asm volatile("bar.sync 1, %0;" ::"n"(32 * kWarps) : "memory");
}

// The nl levels of a chunk; by the kWarps warps that its lists need.  r = this thread's entry
// of the first level walked, out = where its results go, half_scale: the exponents of the values of
// either half of the chunk.
template <int DIR, int kWarps>
__device__ __forceinline__ void ChainChunk(const char *r, double *out, int32_t *half_scale,
                                           int32_t l, int32_t nl, bool first_chunk,
                                           unsigned vals, int32_t *hi_sh, int &group,
                                           ChainState &st) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kStep = DIR == 0 ? 1 : -1;
  constexpr int kPer = 32 * kWarps;
  constexpr unsigned kBufBytes = sizeof(double) * 3 * 256;
  // levels (mod kRescale) that change the scale / end a group / clear the old maximum
  constexpr int kScales = DIR == 0 ? 0 : kRescale - 1, kEnds = DIR == 0 ? kRescale - 1 : 0,
                kClears = DIR == 0 ? 2 : kRescale - 3;
  const int tid = threadIdx.x, lane = tid & 31;
  const unsigned own = vals + tid * 8;
  // the entry of the level at hand and of the next one
  ChainRec rec = LoadRec<DIR, kPer>(r), next = rec;
  ChainFrom from = FromOf<DIR>(rec.at);
  if (nl > 1) next = LoadRec<DIR, kPer>(r + kStep * kPer * 32);
  // One level.  What is not needed for the next level's values is seen to while these three arrive:
  // where the level before goes (`pending`), the record after next, the next offsets.
  // tail: the level after next is not of this chunk; half: which half of the chunk it is in.
  auto level = [&](auto buf, int32_t phase, bool first, bool pending, bool tail, int32_t j,
                   int32_t half, bool single, bool starts) {
    constexpr int kBuf = decltype(buf)::value;
    const unsigned prev = vals + (kBuf ^ 1) * kBufBytes;
    const double x0 = LoadValue(prev + from.at[0]), x1 = LoadValue(prev + from.at[1]),
                 x2 = LoadValue(prev + from.at[2]);
    const bool rescaled = phase == kScales && !first;
    if (pending) out[kStep * (j - 1) * kPer] = st.acc;
    from = FromOf<DIR>(next.at);
    const ChainRec after = tail ? next : LoadRec<DIR, kPer>(r + kStep * (j + 2) * kPer * 32);
    if (rescaled) {
      // (one warp knows the maximum of the group before, unless another walked the chunk before)
      ChainRescale(kWarps == 1 && !starts ? st.hm : *reinterpret_cast<volatile int32_t *>(&hi_sh[group]),
                   st);
      group ^= 1;
    }
    double acc = DIR == 0 ? fma(rec.p0, x0, fma(rec.p1, x1, rec.p2 * x2)) : (x0 + x1) + x2;
    if (rescaled) acc *= st.scale;
    // the first level holds one state, with the value 1: the start state walking forward, the
    // final state walking backward
    if (first) acc = tid == 0 ? 1.0 : 0.0;
    if (DIR == 0) {
      StoreValue(own + kBuf * kBufBytes, acc);
    } else {
      StoreValue(own + kBuf * kBufBytes, rec.p0 * acc);
      StoreValue(own + kBuf * kBufBytes + 2048, rec.p1 * acc);
      StoreValue(own + kBuf * kBufBytes + 4096, rec.p2 * acc);
    }
    st.acc = acc;
    if (phase == kEnds) {  // (values are not negative: their order is that of the high words)
      out[kStep * j * kPer] = acc;
      st.hm = __reduce_max_sync(kAll, __double2hiint(acc));
      if (kWarps > 1) {
        if (lane == 0) atomicMax(&hi_sh[group], st.hm);
      } else if (tid == 0) {
        hi_sh[group] = st.hm;
      }
    }
    if (tid == 0) {
      if (phase == kScales || single) half_scale[half] = st.Ksh;
      if (phase == kClears) hi_sh[group ^ 1] = 0;
    }
    rec = next;
    next = after;
    ChainSync<kWarps>();
  };
  // level l's values are in buffer l & 1
  if (!first_chunk && nl == kPrepLevels) {
#pragma unroll
    for (int32_t g = 0; g < kPrepLevels / kRescale; ++g) {
#pragma unroll
      for (int j = 0; j < kRescale; ++j) {
        const int phase = DIR == 0 ? j : kRescale - 1 - j;
        const bool pending = j > 0;  // (the last level of a group of kRescale leaves nothing)
        const bool tail = j >= kRescale - 2 && g == kPrepLevels / kRescale - 1;
        const int32_t half = DIR == 0 ? g : 1 - g;
        if (phase & 1) level(ChainBuf<1>{}, phase, false, pending, tail, j, half, false, g == 0);
        else level(ChainBuf<0>{}, phase, false, pending, tail, j, half, false, g == 0);
      }
      r += kStep * kRescale * kPer * 32;
      out += kStep * kRescale * kPer;
    }
  } else {
    for (int32_t k = 0; k < nl; ++k, l += kStep) {
      const int32_t phase = l & (kRescale - 1);
      const bool tail = k >= nl - 2;
      const int32_t half = (l / kRescale) & 1;
      if (l & 1) level(ChainBuf<1>{}, phase, first_chunk && k == 0, false, tail, 0, half, true, true);
      else level(ChainBuf<0>{}, phase, first_chunk && k == 0, false, tail, 0, half, true, true);
      if (phase != kEnds) *out = st.acc;
      r += kStep * kPer * 32;
      out += kStep * kPer;
    }
  }
}

template <int DIR>
__device__ __forceinline__ void ChainWalk(const BandInfo &f, int32_t i, BandFactor *ring,
                                          ChainValues &vals, unsigned char *crc, uint64_t *full,
                                          int32_t *hi_sh, const BandFactor *factors,
                                          const int32_t *chunk_r, double *om,
                                          int32_t *__restrict__ oscale, double *tot,
                                          BandTotal *__restrict__ total, int32_t *unfit,
                                          int32_t *status, int32_t wait_limit) {
  constexpr unsigned kAll = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int32_t T = f.frames, pitch = f.pitch, L = T + 2;
  const int32_t num_chunks = (L + kPrepLevels - 1) / kPrepLevels;
  for (int32_t c = tid; c < num_chunks; c += kChainThreads + kKeepThreads)
    crc[c] = (unsigned char)chunk_r[f.level_off + c * kPrepLevels];
  if (tid < 6) vals.v[tid / 3][tid % 3][kNoDst] = 0.0;
  if (tid == 0) {
    for (int st = 0; st < kChainSlots; ++st) MbarInit(&full[st], 1);
    MbarInitFence();
    hi_sh[0] = hi_sh[1] = hi_sh[2] = hi_sh[3] = 0;
  }
  __syncthreads();
  const BandFactor *fac0 = factors + f.grid_off;
  om += f.grid_off;
  oscale += f.level_off;
  int32_t issued = 0;
  // the issuer: the next chunk (in walking order) into the next slot; a chunk is
  // levels * 32 * (warps it needs) entries, a multiple of 1 KB
  auto issue = [&]() {
    if (issued >= num_chunks) return;
    const int32_t c = DIR == 0 ? issued : num_chunks - 1 - issued, slot = issued % kChainSlots;
    const int32_t nl = min((c + 1) * kPrepLevels, L) - c * kPrepLevels;
    const unsigned bytes = (unsigned)(nl * 32 * (int32_t)crc[c]) * (unsigned)sizeof(BandFactor);
    MbarArriveExpectTx(&full[slot], bytes);
    BulkCopyG2S(ring + (size_t)slot * kFacSlot, fac0 + (int64_t)c * kPrepLevels * pitch, bytes,
                &full[slot]);
    ++issued;
  };
  const bool keeper = tid >= kChainThreads, issuer = tid == kChainThreads;
  if (issuer)
    for (int32_t k = 0; k < kChainSlots; ++k) issue();
  ChainState st;
  st.acc = 0.0;
  st.scale = 1.0;
  st.Ksh = st.hm = 0;
  int32_t hi_max = 0;             // keepers: largest high word,
  uint32_t min_hi = 0xffffffffu;  // smallest (high word - 1), zeros apart
  // the keepers' share: what the walk of chunk q left in memory
  auto keep = [&](int32_t q) {
    const int32_t c = DIR == 0 ? q : num_chunks - 1 - q, a = c * kPrepLevels;
    const int32_t nl = min(kPrepLevels, L - a), me = tid - kChainThreads;
    const double *v = om + (int64_t)a * pitch;
    const int32_t n = nl * 32 * crc[c];
#pragma unroll 4
    for (int32_t k = me; k < n; k += kKeepThreads) {
      const int32_t hi = __double2hiint(v[k]);  // values are not negative
      hi_max = max(hi_max, hi);
      min_hi = min(min_hi, (uint32_t)hi - 1u);  // a zero does not count
    }
    if (me < nl) oscale[a + me] = hi_sh[4 + 2 * (q & 1) + me / kRescale];
  };
  int group = 0;
  bool late = false, idle = false;
  int32_t slot = 0;
  unsigned parity = 0;
  for (int32_t q = 0; q < num_chunks; ++q) {
    // the issuer's warp has seen chunk q arrive; the chunk before has been read, and its last
    // level's values are there.  (Whether to go on is part of the barrier: warps that disagreed
    // would wait for one another in the levels of the chunk.)
    late = __syncthreads_or(tid / 32 == kChainThreads / 32 &&
                            !WaitSlot(&full[slot], parity, wait_limit));
    if (late) break;
    const int32_t c = DIR == 0 ? q : num_chunks - 1 - q;
    const BandFactor *mine = ring + (size_t)slot * kFacSlot;
    if (++slot == kChainSlots) {
      slot = 0;
      parity ^= 1u;
    }
    if (keeper) {
      if (q > 0 && issuer) issue();  // into the slot of the chunk before
      if (q > 0) keep(q - 1);
      continue;
    }
    if (idle) {  // what the warps at work kept track of
      st.Ksh = hi_sh[2];
      group = hi_sh[3];
    }
    const int32_t l_lo = c * kPrepLevels, nl = min(l_lo + kPrepLevels, L) - l_lo;
    const int32_t rc = crc[c];
    const int32_t l = DIR == 0 ? l_lo : l_lo + nl - 1;
    idle = warp >= rc;
    if (!idle) {
      const int32_t at = (l - l_lo) * 32 * rc + tid;
      const char *r = reinterpret_cast<const char *>(mine + (l - l_lo) * 32 * rc) + tid * 16;
      double *out = om + (int64_t)l_lo * pitch + at;
      int32_t *half_scale = hi_sh + 4 + 2 * (q & 1);
      switch (rc) {
        case 1: ChainChunk<DIR, 1>(r, out, half_scale, l, nl, q == 0, SmemAddr(&vals), hi_sh, group, st); break;
        case 2: ChainChunk<DIR, 2>(r, out, half_scale, l, nl, q == 0, SmemAddr(&vals), hi_sh, group, st); break;
        case 3: ChainChunk<DIR, 3>(r, out, half_scale, l, nl, q == 0, SmemAddr(&vals), hi_sh, group, st); break;
        default: ChainChunk<DIR, 4>(r, out, half_scale, l, nl, q == 0, SmemAddr(&vals), hi_sh, group, st); break;
      }
    }
    if (tid == 0) {
      hi_sh[2] = st.Ksh;
      hi_sh[3] = group;
    }
  }
  if (late) {
    if (issuer) {
      atomicOr(status, kStatusLate);
      for (int32_t k = max(0, issued - kChainSlots); k < issued; ++k)
        WaitSlot(&full[k % kChainSlots], (unsigned)(k / kChainSlots) & 1u, kDrainPolls);
    }
  }
  __syncthreads();  // the last chunk's values
  if (keeper && !late) {
    keep(num_chunks - 1);
    // values that are not zero must have kept clear of the ends of a double's range
    const int32_t hm = __reduce_max_sync(kAll, hi_max);
    const uint32_t hn = __reduce_min_sync(kAll, min_hi);
    if ((hm >= ((1023 + 900) << 20) || hn < (uint32_t)(((1023 - 900) << 20) - 1)) && lane == 0)
      atomicOr(&unfit[i], kUnfitRange);
  }
  if (DIR == 0 && tid == 0) {
    // entry 0 of the last level is the final state
    if (*status & kStatusLate) {
      tot[i] = nan("");
    } else if (!late && st.acc > 0.0) {
      tot[i] = log(st.acc) + (double)st.Ksh * 0.69314718055994530942;
      BandTotal z;
      z.m = st.acc;
      z.e = st.Ksh;
      z.pad = 0;
      total[i] = z;
    }
  }
}

__global__ void __launch_bounds__(kChainThreads + kKeepThreads)
BandChainLists(const BandInfo *infos, const BandFactor *factors, const int32_t *chunk_r,
               double *am, double *bm, int32_t *__restrict__ a_scale,
               int32_t *__restrict__ b_scale, double *tot, BandTotal *__restrict__ total,
               int32_t *unfit, int32_t *status, int32_t wait_limit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[kChainSlots];
  __shared__ ChainValues vals;
  __shared__ int32_t hi_sh[8];
  __shared__ unsigned char crc[kChainMaxChunks];
  const int dir = blockIdx.x;
  const int32_t i = blockIdx.y;
  WaitForPrevious();
  LetNextStart();
  const BandInfo f = infos[i];
  if (dir == 0 && threadIdx.x == 0) {
    tot[i] = -INFINITY;
    BandTotal z;
    z.m = 0.0;
    z.e = 0;
    z.pad = 0;
    total[i] = z;
  }
  // BandChainExact takes the graphs BandPrep marked.  (The other direction's CTA may mark this one
  // at any time: one answer for all warps, which wait for one another in the levels.)
  if (f.num_states == 0 || __syncthreads_or(unfit[i] != 0)) return;
  BandFactor *ring = reinterpret_cast<BandFactor *>(smem_raw);  // [slots][kFacSlot]
  if (dir == 0)
    ChainWalk<0>(f, i, ring, vals, crc, full, hi_sh, factors, chunk_r, am, a_scale, tot, total, unfit, status,
                 wait_limit);
  else
    ChainWalk<1>(f, i, ring, vals, crc, full, hi_sh, factors, chunk_r, bm, b_scale, tot, total, unfit, status,
                 wait_limit);
}

constexpr int kExactThreads = 128;

// The same recursion with a (mantissa, exponent) pair per state, for the graphs marked in
// `unfit`; every other graph returns at once.  exp(dense score) is recomputed from the
// log-probs, the arc factors come from the graph's tables: no range limit.
__device__ void
ExactWalk(const BandInfo *infos, const BandArc *tabf, const float *lp, int32_t C,
          const BandItem *items, const int2 *lists, double *__restrict__ am,
          int32_t *__restrict__ ae, double *__restrict__ bm, int32_t *__restrict__ be,
          double *tot, BandTotal *__restrict__ total, const int32_t *unfit, int32_t *status,
          int32_t st_pad, int32_t lv_pad, int32_t wait_limit, const BandState *tab,
          const DelaySpec &delay) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[kChainSlots];
  const int dir = blockIdx.x;
  const int32_t i = blockIdx.y;
  const BandInfo f = infos[i];
  const int tid = threadIdx.x;
  const int32_t S = f.num_states, T = f.frames, pitch = f.pitch, L = T + 2;
  if (S == 0) return;
  BandItem *ring = reinterpret_cast<BandItem *>(smem_raw);
  int2 *lst = reinterpret_cast<int2 *>(ring + kChainSlots * kSlotItems);
  ProbState *vals = reinterpret_cast<ProbState *>(lst + lv_pad);  // [2][st_pad], state s at s + 2
  for (int32_t l = tid; l < L; l += kExactThreads) lst[l] = lists[f.level_off + l];
  for (int32_t k = tid; k < 2 * st_pad; k += kExactThreads) {
    ProbState z;
    z.m = 0.0;
    z.e = kZeroExp;
    z.pad = 0;
    vals[k] = z;
  }
  if (tid == 0) {
    for (int st = 0; st < kChainSlots; ++st) MbarInit(&full[st], 1);
    MbarInitFence();
  }
  __syncthreads();
  ChunkRing<BandItem, kSlotItems> rg;
  rg.full = full;
  rg.slots = ring;
  rg.items0 = items + f.grid_off;
  rg.lst = lst;
  rg.pitch = pitch;
  rg.L = L;
  rg.num_chunks = (L + kPrepLevels - 1) / kPrepLevels;
  rg.dir = dir;
  rg.issued = 0;
  if (tid == 0)
    for (int32_t k = 0; k < kChainSlots; ++k) rg.Issue();
  const float *lp0 = lp + (int64_t)f.lp_row * C;
  const BandArc *my_arcs = tabf + (int64_t)f.state_off * 3;
  double *om = (dir == 0 ? am : bm) + f.grid_off;
  int32_t *oe = (dir == 0 ? ae : be) + f.grid_off;
  bool late = false;
  int32_t step = 0;
  for (int32_t q = 0; q < rg.num_chunks; ++q) {
    const int32_t c = rg.ChunkOf(q), slot = q % kChainSlots;
    if (!late) late = !WaitSlot(&full[slot], (unsigned)(q / kChainSlots) & 1u, wait_limit);
    late = __syncthreads_or(late);
    if (late) break;
    const int32_t chunk_start = c * kPrepLevels * pitch;
    const int32_t l_lo = c * kPrepLevels, nl = min(l_lo + kPrepLevels, L) - l_lo;
    const bool fits = rg.ChunkItems(c) <= kSlotItems;
    const BandItem *src = fits ? ring + (size_t)slot * kSlotItems - chunk_start : rg.items0;
    for (int32_t k = 0; k < nl; ++k, ++step) {
      const int32_t l = dir == 0 ? l_lo + k : l_lo + nl - 1 - k;
      const int2 ls = lst[l];
      ProbState *cur = vals + (step & 1) * st_pad + 2;
      const ProbState *prv = vals + ((step & 1) ^ 1) * st_pad + 2;
      for (int32_t j = tid; j < ls.y; j += kExactThreads) {
        const BandItem it = src[ls.x + j];
        const int32_t s = it.s;
        // exp(dense score) of this state's label on frame l - 1
        double pm = 0.0;
        int32_t pe = kZeroExp;
        if (l >= 1) ExpToMantExp(BandDense(lp0, C, T, l - 1, it.label), &pm, &pe);
        double m;
        int32_t e;
        if (step == 0) {
          const bool one = s == (dir == 0 ? 0 : S - 1);
          m = one ? 1.0 : 0.0;
          e = one ? 0 : kZeroExp;
        } else {
          const uint32_t bits = dir == 0 ? it.inb : it.outb;
          double t[3];
          int32_t x[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            // forward: alpha of the source; backward: beta * p of the destination
            t[d] = 0.0;
            x[d] = kZeroExp;
            if ((bits >> d) & 1u) {  // the bit names an arc of this graph
              const ProbState qs = dir == 0 ? prv[s - d] : prv[s + d];
              const BandArc arc = dir == 0 ? my_arcs[3 * s + d] : my_arcs[3 * (s + d) + d];
              double am_arc = arc.f;
              int32_t ak = arc.k;
              if (delay.penalty != 0.0f && delay.flags[arc.arc]) {
                const int32_t t_arc = dir == 0 ? l - 1 : l;
                const float gain = delay.Of(t_arc, T);
                double pen;
                int32_t pen_k;
                ExpToMantExp(gain, &pen, &pen_k);
                // (and what rounding the score to a float, as the lattice has it, makes of it)
                const BandState to = tab[f.state_off + (dir == 0 ? s : s + d)];
                const float x_arc = BandDense(lp0, C, T, t_arc, to.label);
                const float sc = __fadd_rn(__fadd_rn(to.w[d], x_arc), gain);
                am_arc *= pen * exp((double)sc - (double)to.w[d] - (double)x_arc - (double)gain);
                ak += pen_k;
              }
              t[d] = qs.m * am_arc;
              if (t[d] != 0.0) x[d] = qs.e + ak;
            }
          }
          const int32_t E = max(x[0], max(x[1], x[2]));
          const double sum =
              ScaleDown(t[0], x[0] - E) + ScaleDown(t[1], x[1] - E) + ScaleDown(t[2], x[2] - E);
          e = E;
          if (dir == 0) {
            e += pe;
            m = Renorm(sum * pm, &e);
          } else {
            m = Renorm(sum, &e);
          }
        }
        om[ls.x + j] = m;
        oe[ls.x + j] = e;
        ProbState r;
        r.pad = 0;
        if (dir == 0) {
          r.m = m;
          r.e = e;
          if (l == T + 1 && s == S - 1) {
            tot[i] = m == 0.0 ? -INFINITY : log(m) + (double)e * 0.69314718055994530942;
            BandTotal z;
            z.m = m;
            z.e = e;
            z.pad = 0;
            total[i] = z;
          }
        } else {  // what the level below adds: beta * p
          r.e = e + pe;
          r.m = Renorm(m * pm, &r.e);
        }
        cur[s] = r;
      }
      __syncthreads();  // the level is complete
    }
    if (tid == 0) rg.Issue();
  }
  if (late) {
    if (tid == 0) {
      atomicOr(status, kStatusLate);
      rg.Drain();
    }
    __syncthreads();
  }
  if (dir == 0 && tid == 0 && (*status & kStatusLate)) tot[i] = nan("");
}

// What the caller makes of the totals (k2b200_band_reduce), done by the CTA that finishes
// last: three launches of elementwise and reduction kernels less.
struct LossSpec {
  int32_t mode;       // 0: nothing, 1: -sum, 2: mean of -tot / length; both of float32 values
  int32_t lens_type;  // of the lengths: 1 int32, 2 int64, 3 float32, 4 float64
  const void *lens;
  float *loss;
};
__device__ __forceinline__ double LengthOf(const void *lens, int32_t type, int32_t i) {
  switch (type) {
    case 1: return (double)reinterpret_cast<const int32_t *>(lens)[i];
    case 2: return (double)reinterpret_cast<const int64_t *>(lens)[i];
    case 3: return (double)reinterpret_cast<const float *>(lens)[i];
    default: return reinterpret_cast<const double *>(lens)[i];
  }
}

__global__ void __launch_bounds__(kExactThreads)
BandChainExact(const BandInfo *infos, const BandArc *tabf, const float *lp, int32_t C,
               const BandItem *items, const int2 *lists, double *__restrict__ am,
               int32_t *__restrict__ ae, double *__restrict__ bm, int32_t *__restrict__ be,
               double *tot, BandTotal *__restrict__ total, const int32_t *unfit, int32_t *status,
               int32_t st_pad, int32_t lv_pad, int32_t wait_limit, LossSpec spec,
               uint32_t *ticket, const BandState *tab, DelaySpec delay) {
  WaitForPrevious();
  if (unfit[blockIdx.y] != 0)
    ExactWalk(infos, tabf, lp, C, items, lists, am, ae, bm, be, tot, total, unfit, status, st_pad,
              lv_pad, wait_limit, tab, delay);
  if (spec.mode == 0) return;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  uint32_t t = 0;
  if (lane == 0) {
    __threadfence();
    t = atomicAdd(ticket, 1u);
  }
  if (__shfl_sync(0xffffffffu, t, 0) + 1 != 2 * gridDim.y) return;
  __threadfence();
  double sum = 0.0;
  for (int32_t i = lane; i < (int32_t)gridDim.y; i += 32) {
    const float x = -(float)__ldcg(tot + i);
    sum += spec.mode == 2 ? (double)(x / (float)LengthOf(spec.lens, spec.lens_type, i)) : (double)x;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
  if (lane == 0) *spec.loss = (float)(spec.mode == 2 ? sum / (double)gridDim.y : sum);
}

// ---------------------------------------------------------------------------
// Gradients.  grid = (level chunks, pairs), a warp per chunk of kGradLevels levels.
// posterior(l, s) = alpha_l[s] * beta_l[s] / Z is dL/d(dense score of state s's label on
// frame l - 1) up to dL/dtot; it is ADDED to grad_b[(grad_row0[i] + l - 1) * grad_pitch +
// label + grad_col_off] (skipped when label + grad_col_off < 0: the final symbol has no
// column in the log-prob layout).  With kArcs the posterior of every surviving arc,
// alpha_{l-1}[src] e^w p_l[dest] beta_l[dest] / Z, is added to grad_a[arc]; the warp keeps
// alpha of the level before by state number in shared memory for that.
// ---------------------------------------------------------------------------
// dL/dtot of a graph: what the caller's upstream gradient says (k2b200_band_upstream).
struct GradSpec {
  const void *grad;
  int32_t is_double, stride, negate;
  int32_t lens_type;  // != 0: the upstream value is divided by (length of the graph * graphs)
  const void *lens;
  int32_t n;
  __device__ __forceinline__ double Of(int32_t i) const {
    const int64_t at = (int64_t)i * stride;
    double g = is_double ? reinterpret_cast<const double *>(grad)[at]
                         : (double)reinterpret_cast<const float *>(grad)[at];
    if (lens_type) g /= LengthOf(lens, lens_type, i) * n;
    return negate ? -g : g;
  }
};

// A CTA sees to the `width` columns of the gradient from blockIdx.z * width on, as many as a row
// of sums per warp leaves room for (one range up to 12 800 columns, 8 640 with the arcs of graphs
// of 1024 states); the arcs' posteriors go with the first range.
template <bool kArcs>
__global__ void __launch_bounds__(128)
BandGrad(const BandInfo *__restrict__ infos, const BandArc *__restrict__ tabf,
         const float *__restrict__ lp, const BandItem *__restrict__ items,
         const int2 *__restrict__ lists, const double *__restrict__ am,
         const int32_t *__restrict__ ae, const double *__restrict__ bm,
         const int32_t *__restrict__ be, const int32_t *__restrict__ a_scale,
         const int32_t *__restrict__ b_scale, const BandTotal *__restrict__ total,
         const int32_t *__restrict__ unfit, const GradSpec upstream,
         float *__restrict__ grad_a, float *__restrict__ grad_b,
         const int32_t *__restrict__ grad_row0, int32_t grad_pitch, int32_t grad_col_off,
         int32_t C, int32_t width, int32_t st_pad) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int32_t i = blockIdx.y;
  const BandInfo f = infos[i];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t S = f.num_states, T = f.frames;
  if (S == 0) return;
  const int32_t a = 1 + (blockIdx.x * 4 + warp) * kGradLevels;  // levels a .. b - 1
  if (a > T + 1) return;
  const int32_t b = min(a + kGradLevels, T + 2);
  const BandTotal z = total[i];
  if (z.m == 0.0) return;  // no path survives: all gradients are zero
  const double zinv = 1.0 / z.m;
  const bool exact = unfit[i] != 0;  // per-state exponents instead of per-level scales
  const int2 *lst = lists + f.level_off;
  const BandItem *items0 = items + f.grid_off;
  const double *am0 = am + f.grid_off, *bm0 = bm + f.grid_off;
  const int32_t *ae0 = ae + f.grid_off, *be0 = be + f.grid_off;
  const int32_t *as0 = a_scale + f.level_off, *bs0 = b_scale + f.level_off;
  const double tg = upstream.Of(i);
  const int64_t row0 = grad_row0 != nullptr ? grad_row0[i] : f.lp_row;
  const float *lp0 = lp + (int64_t)f.lp_row * C;
  // this warp's row of sums, one per column of the gradient (all zero between levels)
  // (without a gradient for the dense scores only the arcs are wanted)
  const int32_t col0 = blockIdx.z * width;
  const int32_t cols = grad_b != nullptr ? min(width, C + grad_col_off - col0) : 0;
  const bool arcs = kArcs && blockIdx.z == 0;
  uint32_t *sums = reinterpret_cast<uint32_t *>(smem_raw) + (size_t)warp * width;
  for (int32_t k = lane; k < cols; k += 32) sums[k] = 0u;
  __syncwarp();
  ProbState *prev = nullptr;  // alpha of the level before, state s at s + 2
  auto stage_alpha = [&](int32_t l) {
    const int32_t n = lst[l].y;
    const int64_t row = lst[l].x;
    for (int32_t j = lane; j < n; j += 32) {
      ProbState q;
      q.m = am0[row + j];
      q.e = exact ? ae0[row + j] : as0[l];
      q.pad = 0;
      prev[items0[row + j].s] = q;
    }
  };
  if (arcs) {
    prev = reinterpret_cast<ProbState *>(
               smem_raw + (((size_t)4 * width * sizeof(uint32_t) + 15) & ~(size_t)15)) +
           (size_t)warp * st_pad + 2;
    stage_alpha(a - 1);
    __syncwarp();
  }
  // the first 32 entries of the chunk's levels are requested together, before any is used
  int2 ls4[kGradLevels];
  BandItem it4[kGradLevels];
  double al4[kGradLevels], be4[kGradLevels];
#pragma unroll
  for (int u = 0; u < kGradLevels; ++u) {
    ls4[u] = a + u < b ? lst[a + u] : make_int2(0, 0);
    al4[u] = be4[u] = 0.0;
    it4[u].s = 0;
  }
#pragma unroll
  for (int u = 0; u < kGradLevels; ++u)
    if (lane < ls4[u].y) {
      it4[u] = items0[ls4[u].x + lane];
      al4[u] = am0[ls4[u].x + lane];
      be4[u] = bm0[ls4[u].x + lane];
    }
#pragma unroll
  for (int u = 0; u < kGradLevels; ++u) {
    const int32_t l = a + u;
    if (l >= b) break;
    const int32_t n = ls4[u].y;
    const int64_t row = ls4[u].x;
    const int32_t ea_l = as0[l], eb_l = bs0[l];
    for (int32_t j0 = 0; j0 < n; j0 += 32) {
      const int32_t j = j0 + lane;
      float g = 0.0f;
      int32_t key = -1 - lane;  // lanes with nothing to add are groups of their own
      if (j < n) {
        const BandItem it = j0 == 0 ? it4[u] : items0[row + j];
        const double alm = j0 == 0 ? al4[u] : am0[row + j], bem = j0 == 0 ? be4[u] : bm0[row + j];
        if (alm != 0.0 && bem != 0.0) {
          const int32_t ale = exact ? ae0[row + j] : ea_l, bee = exact ? be0[row + j] : eb_l;
          const int32_t col = it.label + grad_col_off - col0;  // of this range
          if (it.label != kNoLabel && it.label < C && col >= 0 && col < cols) {
            g = (float)(alm * bem * zinv * Pow2Clamp(ale + bee - z.e));
            key = col;
          }
          if (arcs) {
            const int32_t s = it.s;
            double pm;
            int32_t pe;
            ExpToMantExp(BandDense(lp0, C, T, l - 1, it.label), &pm, &pe);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              if (!((it.inb >> d) & 1u)) continue;
              const ProbState q = prev[s - d];
              const BandArc arc = tabf[(int64_t)(f.state_off + s) * 3 + d];
              // two steps, so that no intermediate product leaves the range of a double
              const double post = (q.m * arc.f * pm) * (bem * zinv) *
                                  Pow2Clamp(q.e + arc.k + pe + bee - z.e);
              if (post != 0.0) atomicAdd(grad_a + arc.arc, (float)(tg * post));
            }
          }
        }
      }
      // States with the same label (the blank states of a CTC graph) add to the same
      // element.  Their posteriors are summed in this warp's row of shared memory, in fixed
      // point (2^-31 units: a sum of posteriors of one frame is at most 1) with integer
      // atomics - native in shared memory, and independent of the order of the additions -
      // then every lane takes the sum of its column out of the row, which leaves the row
      // zero again, and whoever got it adds it to the gradient.
      if (key >= 0) atomicAdd(&sums[key], __float2uint_rn(g * 2147483648.0f));
      __syncwarp();
      if (key >= 0) {
        const uint32_t fixed = atomicExch(&sums[key], 0u);
        if (fixed != 0u)
          atomicAdd(grad_b + (row0 + l - 1) * grad_pitch + col0 + key,
                    (float)tg * ((float)fixed * (1.0f / 2147483648.0f)));
      }
      __syncwarp();
    }
    if (arcs) {
      __syncwarp();  // the level before has been read
      stage_alpha(l);
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------------------
// The same gradient for log-probs (or logits) that no two sequences share, written whole:
// every element of the rows of a sequence and of the rows up to the next one is stored
// once, so the caller's buffer needs no clearing (at 128 MB of log-probs the clear and the
// scattered additions took 29 + 26 us of memory time, this takes 36).  A warp per DenseRows
// rows; the row's sums gather in shared memory in fixed point as in BandGrad.  A CTA sees to the
// `width` columns from blockIdx.z * width on.  kSoftmax: the rows are log_softmax of the tensor
// the gradient is for, d = g - softmax * sum(g).
// ---------------------------------------------------------------------------
// Rows whose entries a warp requests together: two, twelve CTAs to an SM, and one, sixteen, where a
// row is read as well.  Bound by the chain list -> entries -> sums -> row of a warp beside the
// stores (the rows alone would take 22 of the 36 us of 64 x 1000 frames, 50 of 62 of 32 x 500 x
// 5000), so more warps with less each: with four rows and eight CTAs 37, 65 us, and 27 instead of 20
// from the logits of 32 x 600 x 501.
__host__ __device__ constexpr int DenseRows(bool softmax) { return softmax ? 1 : 2; }
// Columns of a range.  A warp stores its range alone, so a wide one leaves an SM few warps: 60 000
// columns x 2400 rows took 288 us (logits 4625) in ranges of 51 200, what fits in shared memory,
// 139 (678) in ranges of 6400, 139 (320) in ranges of 1600; up to 6400 columns the gradient of
// log-probs only loses by a second range (5000 x 16 000 rows: 109 us, halved 115).
constexpr int kGradColumns = 6400;

template <bool kSoftmax>
__global__ void __launch_bounds__(128, kSoftmax ? 16 : 12)
BandGradRows(const BandInfo *infos, const float *lp, const BandItem *items, const int2 *lists,
             const double *am, const int32_t *ae, const double *bm, const int32_t *be,
             const int32_t *a_scale, const int32_t *b_scale, const BandTotal *total,
             const int32_t *unfit, const GradSpec upstream, float *__restrict__ grad, int32_t C,
             int32_t width) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kDenseRows = DenseRows(kSoftmax);
  const int32_t i = blockIdx.y;
  WaitForPrevious();
  const BandInfo f = infos[i];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t T = f.frames, rows = f.zero_end - f.lp_row;
  const int32_t r0 = (blockIdx.x * (blockDim.x >> 5) + warp) * kDenseRows;
  if (r0 >= rows) return;
  const int32_t r1 = min(r0 + kDenseRows, rows);
  const int32_t col0 = blockIdx.z * width, cols = min(width, C - col0);
  uint32_t *sums = reinterpret_cast<uint32_t *>(smem_raw) + (size_t)warp * width;
  for (int32_t k = lane; k < width; k += 32) sums[k] = 0u;
  const BandTotal z = total[i];
  const bool dead = z.m == 0.0 || f.num_states == 0;  // no path survives: all zero
  const double zinv = dead ? 0.0 : 1.0 / z.m;
  const bool exact = unfit[i] != 0;
  const double tg = dead ? 0.0 : upstream.Of(i);
  const int2 *lst = lists + f.level_off + 1;  // row r is level r + 1
  const BandItem *items0 = items + f.grid_off;
  const double *am0 = am + f.grid_off, *bm0 = bm + f.grid_off;
  const int32_t *ae0 = ae + f.grid_off, *be0 = be + f.grid_off;
  const int32_t *as0 = a_scale + f.level_off + 1, *bs0 = b_scale + f.level_off + 1;
  // the first 32 entries of the rows are requested together, before any is used
  int2 ls4[kDenseRows];
  BandItem it4[kDenseRows];
  double al4[kDenseRows], be4[kDenseRows];
#pragma unroll
  for (int u = 0; u < kDenseRows; ++u) {
    ls4[u] = !dead && r0 + u < min(r1, T) ? lst[r0 + u] : make_int2(0, 0);
    al4[u] = be4[u] = 0.0;
    it4[u].s = 0;
    it4[u].label = kNoLabel;
  }
#pragma unroll
  for (int u = 0; u < kDenseRows; ++u)
    if (lane < ls4[u].y) {
      it4[u] = items0[ls4[u].x + lane];
      al4[u] = am0[ls4[u].x + lane];
      be4[u] = bm0[ls4[u].x + lane];
    }
  __syncwarp();
#pragma unroll
  for (int u = 0; u < kDenseRows; ++u) {
    const int32_t r = r0 + u;
    if (r >= r1) break;
    const int32_t n = ls4[u].y;
    const int64_t row = ls4[u].x;
    uint32_t added = 0;
    if (n > 0) {
      const int32_t ea_l = as0[r], eb_l = bs0[r];
      for (int32_t j = lane; j < n; j += 32) {
        const bool first = j < 32;
        const BandItem it = first ? it4[u] : items0[row + j];
        const double alm = first ? al4[u] : am0[row + j], bem = first ? be4[u] : bm0[row + j];
        if (alm == 0.0 || bem == 0.0 || it.label < 0 || it.label >= C) continue;
        const int32_t ale = exact ? ae0[row + j] : ea_l, bee = exact ? be0[row + j] : eb_l;
        const float g = (float)(alm * bem * zinv * Pow2Clamp(ale + bee - z.e));
        const uint32_t fixed = __float2uint_rn(g * 2147483648.0f);
        added += fixed;
        const uint32_t col = (uint32_t)(it.label - col0);
        if (col < (uint32_t)cols) atomicAdd(&sums[col], fixed);
      }
    }
    __syncwarp();
    float *out = grad + (int64_t)(f.lp_row + r) * C + col0;
    const bool vec = (cols & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    if (n == 0 && !(kSoftmax && r < T)) {
      if (vec) {
        for (int32_t c = lane * 4; c < cols; c += 128)
          *reinterpret_cast<float4 *>(out + c) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      } else {
        for (int32_t c = lane; c < cols; c += 32) out[c] = 0.0f;
      }
      continue;
    }
    // (columns without a posterior are 0 whatever the upstream gradient, infinities and NaN too;
    // rows whose softmax is NaN give NaN even if no path survives)
    const float tgf = (float)tg;
    auto value = [&](uint32_t fixed) {
      return fixed ? tgf * ((float)fixed * (1.0f / 2147483648.0f)) : 0.0f;
    };
    if (!kSoftmax) {
      if (vec) {
#pragma unroll 4
        for (int32_t c = lane * 4; c < cols; c += 128) {
          const uint4 x = *reinterpret_cast<const uint4 *>(sums + c);
          if (x.x | x.y | x.z | x.w) *reinterpret_cast<uint4 *>(sums + c) = make_uint4(0, 0, 0, 0);
          *reinterpret_cast<float4 *>(out + c) =
              make_float4(value(x.x), value(x.y), value(x.z), value(x.w));
        }
      } else {
#pragma unroll 4
        for (int32_t c = lane; c < cols; c += 32) {
          const uint32_t x = sums[c];
          if (x) sums[c] = 0u;
          out[c] = value(x);
        }
      }
    } else {
      // (the sum of a row's posteriors is at most 1, its fixed-point value fits 32 bits)
      const float total_g = value(__reduce_add_sync(kAll, added));
      const float *x = lp + (int64_t)(f.lp_row + r) * C + col0;
      // (four loads together: the compiler does not move one past what is stored before it; without a
      // test each, which took 173 us of 57 x 439 x 2723 frames, 160 so)
      auto put = [&](int32_t c, float p) {
        const uint32_t y = sums[c];
        if (y) sums[c] = 0u;
        out[c] = value(y) - expf(p) * total_g;
      };
      int32_t c = lane;
      for (; c + 96 < cols; c += 128) {
        float p[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) p[k] = x[c + 32 * k];
#pragma unroll
        for (int k = 0; k < 4; ++k) put(c + 32 * k, p[k]);
      }
      for (; c < cols; c += 32) put(c, x[c]);
    }
    __syncwarp();  // the row of sums is zero again
  }
}

// log_probs rows of the sequences = log_softmax of the logits rows.  A warp per row; the same
// expressions as LogSoftmaxFill (dense.cu).  kPer: a row of at most 32 * kPer columns is read once and
// held in registers, 0: it is read three times, from L1 after the first.  Bound by the latency of a
// row's reads and reductions (32 x 600 x 501: 18 us reading three times, 13 once; 8 would be the
// memory's).
template <int kPer>
__global__ void __launch_bounds__(256)
LogSoftmaxRows(const BandInfo *infos, const float *logits, int32_t C,
               float *__restrict__ log_probs) {
  WaitForPrevious();
  const BandInfo f = infos[blockIdx.y];
  const int32_t r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= f.frames) return;
  const float *in = logits + (int64_t)(f.lp_row + r) * C;
  float *out = log_probs + (int64_t)(f.lp_row + r) * C;
  float x[kPer > 0 ? kPer : 1], mx = -INFINITY, sum = 0.0f;
  if (kPer > 0) {
#pragma unroll
    for (int k = 0; k < kPer; ++k) x[k] = lane + 32 * k < C ? in[lane + 32 * k] : -INFINITY;
#pragma unroll
    for (int k = 0; k < kPer; ++k) mx = fmaxf(mx, x[k]);
  } else {
#pragma unroll 4
    for (int32_t c = lane; c < C; c += 32) mx = fmaxf(mx, in[c]);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
  if (kPer > 0) {
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      if (lane + 32 * k < C) sum += expf(x[k] - mx);
  } else {
#pragma unroll 4
    for (int32_t c = lane; c < C; c += 32) sum += expf(in[c] - mx);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
  const float lse = logf(sum);
  if (kPer > 0) {
#pragma unroll
    for (int k = 0; k < kPer; ++k)
      if (lane + 32 * k < C) out[lane + 32 * k] = (x[k] - mx) - lse;
  } else {
    // (read together: a read behind a store waits for it otherwise.  57 x 439 x 2723: 146 us, 190)
    for (int32_t c = lane; c < C; c += 128) {
      float v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c + 32 * u < C) v[u] = in[c + 32 * u];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (c + 32 * u < C) out[c + 32 * u] = (v[u] - mx) - lse;
    }
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct BandLayout {
  std::vector<BandInfo> infos;
  int64_t grid_elems = 0, reachable_states = 0, levels = 0;
  long long arc_frames = 0;
  int32_t max_states = 0, max_frames = 0, max_rows = 0;
  int32_t vit_threads = 32, vit_frames = 0, vit_batches = 0, vit_slot = 0, xch_pad = 0;
  bool by_state = false;
  int32_t first_row = 0;
  int32_t st_pad = 0, lv_pad = 0;
  size_t chain_smem = 0, exact_smem = 0, viterbi_smem = 0, prep_smem = 0;
  size_t off_infos, off_vf, off_vb, off_by_state, off_items, off_factors, off_lists, off_chunk_r,
      off_am, off_ae, off_bm, off_be, off_penalty, off_a_scale, off_b_scale, off_total, off_unfit,
      off_totals, off_status, total_bytes;  // off_status = off_totals + 40
  bool ok = true;
  const char *why = "";
  bool exclusive_rows = true;  // no two graphs on one sequence (they would share gradient rows)
};

constexpr size_t kBandSmemBudget = 200 * 1024;

static int32_t MakeBandLayout(const k2b200_band_loss_args *a, BandLayout *L) {
  K2B_REQUIRE(a != nullptr, "args is NULL");
  K2B_REQUIRE(a->num_fsas > 0, "a_fsas must contain at least one FSA (got %d)", a->num_fsas);
  K2B_REQUIRE(a->output_beam > 0, "output_beam must be > 0 (got %f)", a->output_beam);
  K2B_REQUIRE(a->h_a_row_splits1 && a->h_a_arc_splits && a->h_first_row && a->h_frames,
              "host arrays of the batch description are required");
  K2B_REQUIRE(a->num_classes > 0, "empty log-prob matrix");
  L->infos.resize(a->num_fsas);
  int64_t grid = 0, levels = 0;
  for (int32_t i = 0; i < a->num_fsas; ++i) {
    BandInfo &f = L->infos[i];
    f.state_off = a->h_a_row_splits1[i];
    f.num_states = a->h_a_row_splits1[i + 1] - f.state_off;
    f.pitch = 32 * (f.num_states / 32 + 1);
    f.frames = a->h_frames[i];
    K2B_REQUIRE(f.frames >= 0, "sequence of graph %d has a negative number of frames", i);
    if (i > 0)
      K2B_REQUIRE(f.frames <= a->h_frames[i - 1],
                  "Sequences (DenseFsaVec) must be in sorted order from greatest to least "
                  "length; graph %d has %d frames after %d",
                  i, f.frames, a->h_frames[i - 1]);
    f.lp_row = a->h_first_row[i];
    K2B_REQUIRE(f.lp_row >= 0 && (int64_t)f.lp_row + f.frames <= a->log_prob_rows,
                "frames of graph %d lie outside the log-prob matrix", i);
    if (i > 0 && f.lp_row == a->h_first_row[i - 1]) L->exclusive_rows = false;
    f.level_off = (int32_t)levels;
    f.grid_off = grid;
    grid += (int64_t)(f.frames + 2) * f.pitch;
    {
      // States that can survive: level l (0 .. R = T + 1) holds state s only if the start
      // state reaches it (arcs advance by at most two states: s <= 2 l) and it reaches
      // the last state m = S - 1 at level R (m - s <= 2 (R - l)).  Summed over the
      // levels, with k = m / 2: the grid without two triangles of k (k + 1) states.
      const int64_t S = f.num_states, m = S - 1, R = (int64_t)f.frames + 1, k = m / 2;
      L->reachable_states += (S > 0 && 2 * R >= m) ? 2 * k * (k + 1) + (R - 2 * k - 1) * m + R + 1
                                              : (R + 1) * S;
    }
    levels += f.frames + 2;
    L->max_states = std::max(L->max_states, f.num_states);
    L->max_frames = std::max(L->max_frames, f.frames);
    L->arc_frames += (long long)(f.frames + 1) *
                     (a->h_a_arc_splits[i + 1] - a->h_a_arc_splits[i]);
  }
  if (levels >= ((int64_t)1 << 31)) {
    SetError("problem too large: %lld (fsa, frame) levels", (long long)levels);
    return kTooLarge;
  }
  L->grid_elems = grid;
  L->levels = levels;
  {
    // rows of the log-probs that no sequence covers, each given to the sequence before it
    std::vector<int32_t> order(a->num_fsas);
    for (int32_t i = 0; i < a->num_fsas; ++i) order[i] = i;
    std::sort(order.begin(), order.end(), [&](int32_t x, int32_t y) {
      return L->infos[x].lp_row < L->infos[y].lp_row;
    });
    for (int32_t k = 0; k < a->num_fsas; ++k) {
      BandInfo &f = L->infos[order[k]];
      const int64_t end = k + 1 < a->num_fsas ? L->infos[order[k + 1]].lp_row : a->log_prob_rows;
      f.zero_end = (int32_t)std::min<int64_t>(std::max<int64_t>(end, f.lp_row + f.frames), INT32_MAX);
      if (end < f.lp_row + f.frames) L->exclusive_rows = false;
      L->max_rows = std::max(L->max_rows, f.zero_end - f.lp_row);
      f.pad = 0;
    }
    L->first_row = L->infos[order[0]].lp_row;
    if (a->log_prob_rows >= INT32_MAX) L->exclusive_rows = false;
  }
  // BandViterbi: rows by state when the log-prob rows are much wider than the states of a
  // graph: a CTA takes in 60 bytes per ns, so beyond 1024 columns a row takes longer to arrive
  // than to walk, and a row by state is read twice instead of the row of the log-probs.  Also
  // where two batches of two rows do not fit.
  // Else frames per batch (even, at most 16) so that at least two batches of rows fit in
  // shared memory, up to three within ~100 KB so that two CTAs of up to eight warps share an SM.
  // (Of more warps one fills an SM's registers: 76, 128, 256 x 1000 frames of 802 states and 500
  // classes take 162, 183, 351 us, 223, 259, 461 with the general step in 80 registers.)
  {
    const size_t max_pitch = 32 * ((size_t)L->max_states / 32 + 1);
    const size_t C = (size_t)a->num_classes;
    L->by_state = (C > 1024 && C > 3 * max_pitch) ||
                  4 * C * sizeof(float) > kBandSmemBudget - 16384;
    int32_t F = L->by_state ? kVitFramesByState : 16;
    const size_t row_bytes = sizeof(float) * (L->by_state ? max_pitch : C);
    while (F > 2 && 2 * F * row_bytes > kBandSmemBudget - 16384) F >>= 1;
    L->vit_frames = F;
    L->vit_slot = (int32_t)((F * row_bytes / sizeof(float) + 6 + 3) & ~(size_t)3);
    L->vit_batches = (int32_t)std::max<size_t>(
        2, std::min<size_t>(3, (100 * 1024) / std::max<size_t>(F * row_bytes, 1)));
    const int32_t own_states = (32 - 2 * F / kVitK) * kVitK;
    const int32_t warps = std::max(1, CeilDiv(std::max(L->max_states, 1), own_states));
    L->vit_threads = 32 * (warps + 1);
    L->xch_pad = (warps * own_states + 8 * F + 3) & ~3;
    L->viterbi_smem = sizeof(float) * ((size_t)L->vit_batches * L->vit_slot + 2 * (size_t)L->xch_pad);
    if (warps > kVitMaxWarps) {
      L->ok = false;
      L->why = "too many states for the Viterbi kernel";
    }
  }
  L->st_pad = ((L->max_states + 4) + 15) & ~15;
  L->lv_pad = (L->max_frames + 2 + 3) & ~3;
  L->prep_smem = BandPrepSmem(L->max_states);
  L->exact_smem = sizeof(BandItem) * kChainSlots * kSlotItems + sizeof(int2) * (size_t)L->lv_pad +
                  sizeof(ProbState) * 2 * (size_t)L->st_pad;
  L->chain_smem = sizeof(BandFactor) * kChainSlots * kFacSlot;
  if (L->max_states > kBandMaxStates) {
    L->ok = false;
    L->why = "a graph has more than 1024 states";
  } else if (L->chain_smem > kBandSmemBudget || L->exact_smem > kBandSmemBudget) {
    L->ok = false;
    L->why = "too many frames or states for the shared memory of the recursions";
  } else if (L->max_frames + 2 > kChainMaxChunks * kPrepLevels) {
    L->ok = false;
    L->why = "a sequence has more than 65534 frames";
  } else if (a->num_fsas > 65535) {
    L->ok = false;
    L->why = "more than 65535 graphs";
  }
  size_t off = 0;
  auto take = [&](size_t bytes) {
    size_t o = off;
    off += AlignUp(bytes ? bytes : 1);
    return o;
  };
  L->off_infos = take(sizeof(BandInfo) * a->num_fsas);
  L->off_vf = take(sizeof(float) * (size_t)grid);
  L->off_vb = take(sizeof(float) * (size_t)grid);
  L->off_by_state = take(L->by_state ? sizeof(float) * (size_t)grid : 0);
  L->off_items = take(sizeof(BandItem) * (size_t)grid);
  L->off_lists = take(sizeof(int2) * (size_t)levels);
  L->off_chunk_r = take(sizeof(int32_t) * (size_t)levels);
  L->off_factors = take(sizeof(BandFactor) * (size_t)grid);
  L->off_am = take(sizeof(double) * (size_t)grid);
  L->off_ae = take(sizeof(int32_t) * (size_t)grid);
  L->off_bm = take(sizeof(double) * (size_t)grid);
  L->off_be = take(sizeof(int32_t) * (size_t)grid);
  L->off_a_scale = take(sizeof(int32_t) * (size_t)levels);
  L->off_b_scale = take(sizeof(int32_t) * (size_t)levels);
  L->off_total = take(sizeof(BandTotal) * a->num_fsas);
  L->off_penalty = take((size_t)std::max(a->h_a_arc_splits[a->num_fsas], 1));
  L->off_unfit = take(sizeof(int32_t) * a->num_fsas);
  L->off_totals = take(64);  // five 64-bit totals, the status word, the ticket (at 48)
  L->off_status = L->off_totals + 5 * sizeof(long long);
  L->total_bytes = off;
  return kOk;
}

static bool BandReduceBeam(const k2b200_band_loss_args *a, const long long *h_totals,
                           float *beam) {
  long long limit = 0, total = 0;
  if (h_totals[0] > a->max_states) {
    limit = a->max_states;
    total = h_totals[0];
  } else if (h_totals[2] > a->max_arcs) {
    limit = a->max_arcs;
    total = h_totals[2];
  } else {
    return false;
  }
  // the reference's rule, intersect_dense.cu:854-862
  float cur = *beam, next = cur * sqrt(limit * 1.0 / total);
  if (next < cur * 0.25) next = cur * 0.25;
  if (next > cur * 0.75) next = cur * 0.75;
  *beam = next;
  return true;
}

static int32_t LaunchBandChains(const BandLayout &L, const k2b200_band_loss_args *args, char *ws,
                                double *tot_scores, const LossSpec &spec, const DelaySpec &delay,
                                cudaStream_t stream) {
  K2B_CUDA_OK(cudaFuncSetAttribute(BandChainLists, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)L.chain_smem));
  K2B_CUDA_OK(cudaFuncSetAttribute(BandChainExact, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)L.exact_smem));
  dim3 grid(2, args->num_fsas);
  const BandInfo *infos = reinterpret_cast<const BandInfo *>(ws + L.off_infos);
  const BandItem *items = reinterpret_cast<const BandItem *>(ws + L.off_items);
  const int2 *lists = reinterpret_cast<const int2 *>(ws + L.off_lists);
  double *am = reinterpret_cast<double *>(ws + L.off_am), *bm = reinterpret_cast<double *>(ws + L.off_bm);
  BandTotal *total = reinterpret_cast<BandTotal *>(ws + L.off_total);
  int32_t *unfit = reinterpret_cast<int32_t *>(ws + L.off_unfit);
  int32_t *status = reinterpret_cast<int32_t *>(ws + L.off_status);
  { K2B_CUDA_OK(LaunchBehind(BandChainLists, grid, kChainThreads + kKeepThreads, L.chain_smem, stream,
      infos, reinterpret_cast<const BandFactor *>(ws + L.off_factors),
      reinterpret_cast<const int32_t *>(ws + L.off_chunk_r), am, bm,
      reinterpret_cast<int32_t *>(ws + L.off_a_scale),
      reinterpret_cast<int32_t *>(ws + L.off_b_scale), tot_scores, total, unfit, status,
      CopyWaitLimit())); NoteLaunch(); }
  { K2B_CUDA_OK(LaunchBehind(BandChainExact, grid, kExactThreads, L.exact_smem, stream,
      infos, reinterpret_cast<const BandArc *>(args->band_arcs), args->log_probs,
      args->num_classes, items, lists, am, reinterpret_cast<int32_t *>(ws + L.off_ae), bm,
      reinterpret_cast<int32_t *>(ws + L.off_be), tot_scores, total, unfit, status, L.st_pad,
      L.lv_pad, CopyWaitLimit(), spec, reinterpret_cast<uint32_t *>(ws + L.off_totals + 48),
      reinterpret_cast<const BandState *>(args->band_states), delay));
    NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

}  // namespace k2b

using namespace k2b;

extern "C" {

void k2b200_debug_set_copy_wait_limit(int32_t polls) { SetCopyWaitLimit(polls); }

int32_t k2b200_band_tables_bytes(int32_t num_states, size_t *states_bytes, size_t *arcs_bytes) {
  K2B_REQUIRE(states_bytes && arcs_bytes, "NULL output pointer");
  const size_t n = (size_t)std::max(num_states, 1);
  *states_bytes = sizeof(BandState) * n;
  *arcs_bytes = sizeof(BandArc) * 3 * n;
  return kOk;
}

int32_t k2b200_band_tables(const int32_t *row_splits1, int32_t num_fsas,
                           const int32_t *row_splits2, const void *arcs, int32_t num_states,
                           void *band_states, void *band_arcs, int32_t *status, void *stream_v) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  K2B_REQUIRE(row_splits1 && row_splits2 && band_states && band_arcs && status,
              "NULL device pointer");
  K2B_REQUIRE(num_fsas > 0, "a_fsas must contain at least one FSA (got %d)", num_fsas);
  K2B_CUDA_OK(cudaMemsetAsync(status, 0, sizeof(int32_t), stream));
  if (num_states > 0)
    { BandTables<<<CeilDiv(num_states, 128), 128, 0, stream>>>(
        row_splits1, num_fsas, row_splits2, reinterpret_cast<const Arc *>(arcs), num_states,
        reinterpret_cast<BandState *>(band_states), reinterpret_cast<BandArc *>(band_arcs),
        status); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

int32_t k2b200_band_incoming(const void *band_states, const void *band_arcs,
                             const int32_t *row_splits2, int32_t num_states, int32_t *in_splits,
                             int32_t *in_arcs, int32_t *in_src, float *in_score, void *stream_v) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  K2B_REQUIRE(band_states && band_arcs && row_splits2 && in_splits && in_arcs && in_src && in_score,
              "NULL device pointer");
  { BandIncoming<<<CeilDiv((int64_t)num_states + 1, 128), 128, 0, stream>>>(
      reinterpret_cast<const BandState *>(band_states),
      reinterpret_cast<const BandArc *>(band_arcs), row_splits2, num_states, in_splits, in_arcs,
      in_src, in_score); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

int32_t k2b200_band_loss_supported(const k2b200_band_loss_args *args, int32_t *supported) {
  K2B_REQUIRE(supported != nullptr, "NULL output pointer");
  BandLayout L;
  K2B_FORWARD(MakeBandLayout(args, &L));
  *supported = L.ok ? 1 : 0;
  if (!L.ok) SetError("band loss path not applicable: %s", L.why);
  return kOk;
}

int32_t k2b200_band_loss_workspace_bytes(const k2b200_band_loss_args *args, size_t *bytes) {
  K2B_REQUIRE(bytes != nullptr, "NULL output pointer");
  BandLayout L;
  K2B_FORWARD(MakeBandLayout(args, &L));
  *bytes = L.total_bytes;
  return kOk;
}

int32_t k2b200_band_loss_plan(const k2b200_band_loss_args *args, int32_t *supported,
                              int32_t *exclusive_rows, size_t *bytes) {
  K2B_REQUIRE(supported && exclusive_rows && bytes, "NULL output pointer");
  BandLayout L;
  K2B_FORWARD(MakeBandLayout(args, &L));
  *supported = L.ok ? 1 : 0;
  *exclusive_rows = L.exclusive_rows ? 1 : 0;
  *bytes = L.total_bytes;
  if (!L.ok) SetError("band loss path not applicable: %s", L.why);
  return kOk;
}

int32_t k2b200_band_loss_forward(const k2b200_band_loss_args *args, void *workspace,
                                 size_t workspace_bytes, void *stream_v, double *tot_scores,
                                 float *beam_used) {
  return k2b200_band_loss_forward_reduce(args, workspace, workspace_bytes, stream_v, tot_scores,
                                         beam_used, nullptr);
}

int32_t k2b200_band_loss_forward_reduce(const k2b200_band_loss_args *args, void *workspace,
                                        size_t workspace_bytes, void *stream_v, double *tot_scores,
                                        float *beam_used, const k2b200_band_reduce *reduce) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  BandLayout L;
  K2B_FORWARD(MakeBandLayout(args, &L));
  K2B_REQUIRE(L.ok, "band loss path not applicable: %s", L.why);
  if (workspace == nullptr || workspace_bytes < L.total_bytes) {
    SetError("workspace of %zu bytes is smaller than the %zu required", workspace_bytes,
             L.total_bytes);
    return kWorkspaceTooSmall;
  }
  K2B_REQUIRE(args->a_row_splits2 && args->band_states && args->band_arcs && args->log_probs &&
                  tot_scores,
              "NULL device pointer");
  char *ws = reinterpret_cast<char *>(workspace);
  static_assert(sizeof(BandInfo) % sizeof(int32_t) == 0, "BandInfo is uploaded as int32 words");
  LossSpec spec = {0, 0, nullptr, nullptr};
  DelaySpec delay = {0.0f, nullptr};
  const float *logits = nullptr;
  if (reduce != nullptr) {
    K2B_REQUIRE(reduce->mode >= 0 && reduce->mode <= 2, "bad reduction mode %d", reduce->mode);
    K2B_REQUIRE(reduce->mode == 0 || reduce->loss != nullptr, "NULL loss pointer");
    K2B_REQUIRE(reduce->mode != 2 || (reduce->lens != nullptr && reduce->lens_type >= 1 &&
                                      reduce->lens_type <= 4),
                "the mean needs lengths");
    spec.mode = reduce->mode;
    spec.lens = reduce->lens;
    spec.lens_type = reduce->lens_type;
    spec.loss = reduce->loss;
    logits = reduce->logits;
    if (reduce->delay_penalty != 0.0f) {
      K2B_REQUIRE(reduce->arc_repeat != nullptr || reduce->arc_aux != nullptr,
                  "a delay penalty needs to know the arcs it applies to");
      delay.penalty = reduce->delay_penalty;
      delay.flags = reinterpret_cast<const uint8_t *>(ws + L.off_penalty);
    }
  }
  // unfit words, totals, the status word and the ticket lie one after the other: one clear for
  // the first pass (a repeated pass clears them again but for the status of the Viterbi kernels)
  K2B_FORWARD(UploadIntsAndClear(reinterpret_cast<const int32_t *>(L.infos.data()),
                                 (int64_t)L.infos.size() * (sizeof(BandInfo) / sizeof(int32_t)),
                                 reinterpret_cast<int32_t *>(ws + L.off_infos),
                                 reinterpret_cast<int32_t *>(ws + L.off_unfit),
                                 (int64_t)(L.off_totals + 64 - L.off_unfit) / 4, stream));
  if (delay.penalty != 0.0f && args->num_states > 0)
    { PenaltyFlags<<<CeilDiv(args->num_states, 128), 128, 0, stream>>>(
        reinterpret_cast<const BandState *>(args->band_states),
        reinterpret_cast<const BandArc *>(args->band_arcs), args->num_states, reduce->arc_repeat,
        reduce->arc_aux, const_cast<uint8_t *>(delay.flags)); NoteLaunch(); }
  if (logits != nullptr && L.max_frames > 0) {
    PhaseTimer timer(kPhaseDense, stream);
    dim3 grid(CeilDiv(L.max_frames, 8), args->num_fsas);
    const int32_t C = args->num_classes;
    auto kernel = C <= 128    ? LogSoftmaxRows<4>
                  : C <= 256  ? LogSoftmaxRows<8>
                  : C <= 512  ? LogSoftmaxRows<16>
                  : C <= 1024 ? LogSoftmaxRows<32>
                              : LogSoftmaxRows<0>;
    { K2B_CUDA_OK(LaunchBehind(kernel, grid, 256, 0, stream,
        reinterpret_cast<const BandInfo *>(ws + L.off_infos), logits, args->num_classes,
        const_cast<float *>(args->log_probs))); NoteLaunch(); }
  }
  {
    PhaseTimer timer(kPhaseViterbi, stream);
    NotePhaseKernel(kPhaseViterbi, "BandViterbi");
    K2B_CUDA_OK(cudaFuncSetAttribute(delay.penalty != 0.0f ? BandPrep<true> : BandPrep<false>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)L.prep_smem));
    const BandInfo *infos = reinterpret_cast<const BandInfo *>(ws + L.off_infos);
    const BandState *tab = reinterpret_cast<const BandState *>(args->band_states);
    if (L.by_state && L.max_frames > 0) {
      dim3 grid(CeilDiv(L.max_frames, kGatherRows), args->num_fsas);
      { K2B_CUDA_OK(LaunchBehind(BandGather, grid, 256, 0, stream, infos, tab, args->log_probs, args->num_classes,
                                             reinterpret_cast<float *>(ws + L.off_by_state)));
        NoteLaunch(); }
    }
    const uintptr_t lp_begin = reinterpret_cast<uintptr_t>(args->log_probs),
                    lp_end = lp_begin + sizeof(float) * (size_t)args->log_prob_rows *
                                            (size_t)args->num_classes;
    auto kernel = L.by_state                  ? BandViterbi<true, false>
                  : ((lp_begin | lp_end) & 15) ? BandViterbi<false, true>
                                               : BandViterbi<false, false>;
    K2B_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)L.viterbi_smem));
    dim3 grid(2, args->num_fsas);
    { K2B_CUDA_OK(LaunchBehind(kernel, grid, L.vit_threads, L.viterbi_smem, stream,
        infos, tab,
        L.by_state ? reinterpret_cast<const float *>(ws + L.off_by_state) : args->log_probs,
        args->log_prob_rows, args->num_classes, reinterpret_cast<float *>(ws + L.off_vf),
        reinterpret_cast<float *>(ws + L.off_vb), L.vit_frames, L.vit_batches, L.vit_slot,
        L.xch_pad, CopyWaitLimit(), reinterpret_cast<int32_t *>(ws + L.off_status)));
      NoteLaunch(); }
    K2B_CUDA_OK(cudaGetLastError());
  }
  // The lattice is never built, but its size still decides the beam
  // (intersect_dense.cu:300-320).  The grid bounds it (for the states: the part of the grid
  // that lies both behind the start state and before the last one): the host reads the
  // counts only when that bound does not already satisfy the limits, and after it has
  // launched the recursions, which in the rare case of a reduction run again.
  const bool need_count = L.reachable_states > args->max_states || L.arc_frames > args->max_arcs;
  float beam = args->output_beam;
  bool join_side = false;
  struct JoinOnExit {  // also on error returns: the caller may free the buffer being cleared
    cudaStream_t main;
    bool *armed;
    ~JoinOnExit() { if (*armed) SideJoin(main); }
  } join_guard{stream, &join_side};
  for (int iter = 0;; ++iter) {
    SideReadBackScope readback;
    if (iter > 0) {
      K2B_CUDA_OK(cudaMemsetAsync(ws + L.off_totals, 0, 5 * sizeof(long long), stream));
      K2B_CUDA_OK(cudaMemsetAsync(ws + L.off_totals + 48, 0, sizeof(uint32_t), stream));
      K2B_CUDA_OK(cudaMemsetAsync(ws + L.off_unfit, 0, sizeof(int32_t) * args->num_fsas, stream));
    }
    cudaStream_t side = nullptr;
    {
      PhaseTimer timer(kPhasePrune, stream);
      NotePhaseKernel(kPhasePrune, "BandPrep");
      dim3 grid(CeilDiv(L.max_frames + 2, kPrepLevels), args->num_fsas);
      auto prep = delay.penalty != 0.0f ? BandPrep<true> : BandPrep<false>;
      { K2B_CUDA_OK(LaunchBehind(prep, grid, 32 * kPrepWarps, L.prep_smem, stream,
          reinterpret_cast<const BandInfo *>(ws + L.off_infos), args->a_row_splits2,
          reinterpret_cast<const BandState *>(args->band_states),
          reinterpret_cast<const BandArc *>(args->band_arcs), args->log_probs,
          args->num_classes,
          L.by_state ? reinterpret_cast<const float *>(ws + L.off_by_state) : nullptr,
          reinterpret_cast<const float *>(ws + L.off_vf),
          reinterpret_cast<const float *>(ws + L.off_vb), beam,
          reinterpret_cast<BandItem *>(ws + L.off_items),
          reinterpret_cast<BandFactor *>(ws + L.off_factors),
          reinterpret_cast<int2 *>(ws + L.off_lists),
          reinterpret_cast<int32_t *>(ws + L.off_chunk_r),
          reinterpret_cast<unsigned long long *>(ws + L.off_totals),
          reinterpret_cast<int32_t *>(ws + L.off_unfit),
          L.arc_frames > args->max_arcs ? 1 : 0, delay)); NoteLaunch(); }
      // the host reads the counts behind BandPrep, while what follows runs
      if (need_count) {
        K2B_FORWARD(SideFork(stream, &side));
        K2B_FORWARD(readback.Begin(ws + L.off_totals, sizeof(long long) * 6));
      }
      K2B_CUDA_OK(cudaGetLastError());
    }
    if (iter == 0 && args->zero_fill != nullptr && args->zero_fill_bytes > 0) {
      // behind BandPrep, beside the recursions (up to four warps per graph and direction: the
      // SMs are all but idle); joined below
      K2B_FORWARD(SideFork(stream, &side));
      K2B_CUDA_OK(cudaMemsetAsync(args->zero_fill, 0, args->zero_fill_bytes, side));
      join_side = true;
    }
    {
      PhaseTimer timer(kPhaseChain, stream);
      NotePhaseKernel(kPhaseChain, "BandChainLists");
      K2B_FORWARD(LaunchBandChains(L, args, ws, tot_scores, spec, delay, stream));
    }
    if (!need_count) break;
    long long h_totals[6];
    K2B_FORWARD(readback.End(h_totals));
    K2B_REQUIRE((h_totals[5] & kStatusLate) == 0,
                "a copy of log-prob rows into shared memory did not complete in time");
    const float beam_before = beam;
    if (!BandReduceBeam(args, h_totals, &beam)) break;
    K2B_LOG(kLogInfo, "band loss: %lld states / %lld arcs exceed max_states %d / max_arcs %d, "
            "output beam %g -> %g", h_totals[0], h_totals[2], args->max_states, args->max_arcs,
            (double)beam_before, (double)beam);
    K2B_REQUIRE(iter < 200, "output beam reduction did not converge");
  }
  if (beam_used) *beam_used = beam;
  return kOk;
}

// Columns that a CTA of a gradient kernel sees to: all of them where `most` allows, else equal
// ranges; a multiple of four.
static int32_t ColumnRange(int32_t cols, size_t most) {
  const int32_t ranges = std::max(1, CeilDiv(cols, (int64_t)(most & ~(size_t)3)));
  return (CeilDiv(cols, ranges) + 3) & ~3;
}

static int32_t BandArcsOrScatter(const BandLayout &L, const k2b200_band_loss_args *args, char *ws,
                                 const GradSpec &upstream, float *grad_a, float *grad_b,
                                 const int32_t *grad_row0, int32_t grad_pitch,
                                 int32_t grad_col_off, cudaStream_t stream) {
  // columns in ranges that four rows of sums have room for beside the states of the arcs
  const size_t arc_bytes = grad_a ? sizeof(ProbState) * 4 * (size_t)L.st_pad : 0;
  const int32_t cols = grad_b == nullptr ? 0 : args->num_classes + grad_col_off;
  const int32_t width = ColumnRange(cols, (kBandSmemBudget - arc_bytes) / (4 * sizeof(uint32_t)));
  const size_t smem = sizeof(uint32_t) * 4 * (size_t)width + arc_bytes;
  dim3 grid(CeilDiv(L.max_frames + 1, 4 * kGradLevels), args->num_fsas,
            cols > 0 ? CeilDiv(cols, width) : 1);
  auto kernel = grad_a != nullptr ? BandGrad<true> : BandGrad<false>;
  K2B_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kBandSmemBudget));
  { kernel<<<grid, 128, smem, stream>>>(
      reinterpret_cast<const BandInfo *>(ws + L.off_infos),
      reinterpret_cast<const BandArc *>(args->band_arcs), args->log_probs,
      reinterpret_cast<const BandItem *>(ws + L.off_items),
      reinterpret_cast<const int2 *>(ws + L.off_lists),
      reinterpret_cast<const double *>(ws + L.off_am),
      reinterpret_cast<const int32_t *>(ws + L.off_ae),
      reinterpret_cast<const double *>(ws + L.off_bm),
      reinterpret_cast<const int32_t *>(ws + L.off_be),
      reinterpret_cast<const int32_t *>(ws + L.off_a_scale),
      reinterpret_cast<const int32_t *>(ws + L.off_b_scale),
      reinterpret_cast<const BandTotal *>(ws + L.off_total),
      reinterpret_cast<const int32_t *>(ws + L.off_unfit), upstream, grad_a, grad_b, grad_row0,
      grad_pitch, grad_col_off, args->num_classes, width, L.st_pad); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

int32_t k2b200_band_loss_backward(const k2b200_band_loss_args *args, void *workspace,
                                  size_t workspace_bytes, const double *tot_grad,
                                  int32_t tot_grad_stride, float *grad_a, float *grad_b,
                                  const int32_t *grad_row0, int32_t grad_pitch,
                                  int32_t grad_col_off, void *stream_v) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  BandLayout L;
  K2B_FORWARD(MakeBandLayout(args, &L));
  K2B_REQUIRE(L.ok, "band loss path not applicable: %s", L.why);
  if (workspace == nullptr || workspace_bytes < L.total_bytes) {
    SetError("workspace of %zu bytes is smaller than the %zu required", workspace_bytes,
             L.total_bytes);
    return kWorkspaceTooSmall;
  }
  K2B_REQUIRE(tot_grad && grad_b, "NULL device pointer");
  K2B_REQUIRE(grad_col_off == 0 || grad_col_off == 1, "grad_col_off must be 0 or 1");
  PhaseTimer timer(kPhaseGrad, stream);
  NotePhaseKernel(kPhaseGrad, "BandGrad");
  const GradSpec upstream = {tot_grad, 1, tot_grad_stride, 0, 0, nullptr, args->num_fsas};
  return BandArcsOrScatter(L, args, reinterpret_cast<char *>(workspace), upstream, grad_a, grad_b,
                           grad_row0, grad_pitch, grad_col_off, stream);
}

int32_t k2b200_band_loss_backward_dense(const k2b200_band_loss_args *args, void *workspace,
                                        size_t workspace_bytes,
                                        const k2b200_band_upstream *upstream, float *grad_a,
                                        float *grad_log_probs, int32_t softmax, void *stream_v) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  BandLayout L;
  K2B_FORWARD(MakeBandLayout(args, &L));
  K2B_REQUIRE(L.ok, "band loss path not applicable: %s", L.why);
  K2B_REQUIRE(L.exclusive_rows, "sequences share rows of the log-probs");
  if (workspace == nullptr || workspace_bytes < L.total_bytes) {
    SetError("workspace of %zu bytes is smaller than the %zu required", workspace_bytes,
             L.total_bytes);
    return kWorkspaceTooSmall;
  }
  K2B_REQUIRE(upstream && upstream->grad, "NULL upstream gradient");
  char *ws = reinterpret_cast<char *>(workspace);
  PhaseTimer timer(kPhaseGrad, stream);
  NotePhaseKernel(kPhaseGrad, "BandGradRows");
  const GradSpec spec = {upstream->grad,      upstream->is_double, upstream->stride,
                         upstream->negate,    upstream->lens_type, upstream->lens,
                         args->num_fsas};
  if (grad_log_probs != nullptr) {
    const int32_t C = args->num_classes;
    const int32_t width = ColumnRange(C, kGradColumns);
    if (L.first_row > 0)  // rows before the first sequence
      K2B_CUDA_OK(cudaMemsetAsync(grad_log_probs, 0, sizeof(float) * (size_t)L.first_row * C, stream));
    const size_t row_bytes = sizeof(uint32_t) * (size_t)width;
    // a row of sums per warp in shared memory: fewer warps per CTA when rows are long, so
    // that a CTA does not hold the SM's memory for one slow warp
    const int32_t warps = row_bytes * 4 <= 16 * 1024 ? 4 : row_bytes <= 8 * 1024 ? 2 : 1;
    auto kernel = softmax ? BandGradRows<true> : BandGradRows<false>;
    K2B_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kBandSmemBudget));
    dim3 grid(CeilDiv(std::max(L.max_rows, 1), warps * DenseRows(softmax)), args->num_fsas,
              CeilDiv(C, width));
    { K2B_CUDA_OK(LaunchBehind(kernel, grid, 32 * warps, row_bytes * warps, stream,
        reinterpret_cast<const BandInfo *>(ws + L.off_infos), args->log_probs,
        reinterpret_cast<const BandItem *>(ws + L.off_items),
        reinterpret_cast<const int2 *>(ws + L.off_lists),
        reinterpret_cast<const double *>(ws + L.off_am),
        reinterpret_cast<const int32_t *>(ws + L.off_ae),
        reinterpret_cast<const double *>(ws + L.off_bm),
        reinterpret_cast<const int32_t *>(ws + L.off_be),
        reinterpret_cast<const int32_t *>(ws + L.off_a_scale),
        reinterpret_cast<const int32_t *>(ws + L.off_b_scale),
        reinterpret_cast<const BandTotal *>(ws + L.off_total),
        reinterpret_cast<const int32_t *>(ws + L.off_unfit), spec, grad_log_probs, C, width));
      NoteLaunch(); }
    K2B_CUDA_OK(cudaGetLastError());
  }
  if (grad_a != nullptr)
    K2B_FORWARD(BandArcsOrScatter(L, args, ws, spec, grad_a, nullptr, nullptr, 0, 0, stream));
  return kOk;
}

int32_t k2b200_band_loss_status(const k2b200_band_loss_args *args, void *workspace,
                                size_t workspace_bytes, void *stream_v, int32_t *status) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  K2B_REQUIRE(status != nullptr, "NULL output pointer");
  BandLayout L;
  K2B_FORWARD(MakeBandLayout(args, &L));
  K2B_REQUIRE(workspace != nullptr && workspace_bytes >= L.total_bytes, "workspace too small");
  K2B_CUDA_OK(cudaMemcpyAsync(status, reinterpret_cast<char *>(workspace) + L.off_status,
                              sizeof(int32_t), cudaMemcpyDeviceToHost, stream));
  K2B_CUDA_OK(cudaStreamSynchronize(stream));
  if (*status & kStatusLate)
    K2B_LOG(kLogWarning, "band loss: a bounded wait for a copy into shared memory gave up; the "
            "results of that call are invalid");
  return kOk;
}

}  // extern "C"
