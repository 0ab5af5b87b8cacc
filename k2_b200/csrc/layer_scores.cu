// Forward/backward scores of a strictly layered FsaVec: every arc goes from one layer
// to the next, as in the lattices that the dense intersections emit (frames are layers).
// Reference arithmetic: k2/csrc/fsa_utils.cu:1124-1278, :1345-1454.
//
// The recursion is a chain of T dependent layers, so what bounds it is the latency of one
// layer, and the rest of the work is moved off that chain:
//   * LayerIncoming builds the incoming-arc index layer by layer.  The arcs that enter a
//     layer are exactly those that leave the layer before, one contiguous range, so the
//     index is a stable counting sort of that range by destination: no global scan, no
//     atomics on global memory and one launch (lfmmi lattice of 6.7 M arcs: 283 us by
//     counting, scanning, filling and sorting the whole FsaVec).
//   * PackLayerArcs writes one 16-byte record per arc: exp(score) as a double for the log
//     semiring (the score itself for the tropical one), the state at the other end and the
//     arc's index.
//   * LayerChain, one CTA per (FSA, direction), then needs one multiply-add per arc: values
//     of a layer are plain doubles that share a power of two, which follows the largest of
//     them every kRescale layers.  What that cannot hold (arc scores beyond +-kMaxScore,
//     values more than 2^280 away from it) raises the status word, and the caller's general
//     kernel, launched behind and otherwise returning at once, redoes the call.
//   * FinishLayerScores takes the logarithms, all states in parallel.
// A state's arcs are taken by one lane, or by eight when states have many; the few states of
// many arcs that lattices of the first kind have (hub states of decoding graphs) by a warp.
// Layers come through a ring in shared memory: a slot holds as many consecutive layers as
// fit (their records and splits are contiguous), fetched by two bulk copies that one lane of
// an extra warp issues ahead of the chain.  Lattices with layers too wide for a slot
// (decoding: thousands of states per frame) go to LayerChainWide, a cluster of CTAs per chain.
#include <algorithm>

#include <cooperative_groups.h>

#include "../../include/k2b200.h"
#include "common.cuh"
#include "cp_async.cuh"
#include "scores_internal.cuh"

namespace k2b {

constexpr size_t kLayerSmemBudget = 200 * 1024;
constexpr int kLight = 4;             // arcs that one lane sums by itself
constexpr int kRescale = 4;           // layers between changes of the shared exponent
constexpr float kMaxScore = 300.0f;   // |arc score|: exp() within 2^+-433
constexpr int kRangeExp = 280;        // values that are not zero stay within 2^+-280, so that no
                                      // product of one with a factor and a scale underflows
constexpr int kMaxSlots = 8;
constexpr int kChunkLayers = 32;      // layers of one slot at most

struct __align__(16) LayerArc {
  double w;       // exp(score) (log semiring) or the score (tropical)
  int32_t other;  // state (idx01) the arc comes from (forward) / goes to (backward)
  int32_t arc;    // index of the arc
};
static_assert(sizeof(LayerArc) == 16, "LayerArc must be 16 bytes");

// ---------------------------------------------------------------------------
// Incoming-arc index of a strictly layered FsaVec.  kWarps == 1: a warp per layer, four
// layers per CTA; else kWarps warps per layer.  cnt[kWarps][maxw] in shared memory: first
// the arcs of every warp's section per destination, then the position its next one gets.
// ---------------------------------------------------------------------------
template <int kWarps>
__global__ void __launch_bounds__(128)
LayerIncoming(const int32_t *__restrict__ row_splits1, const int32_t *__restrict__ row_ids1,
              const int32_t *__restrict__ row_splits2, const Arc *__restrict__ arcs,
              const int32_t *__restrict__ level_offsets, const int32_t *__restrict__ level_splits,
              int32_t num_fsas, int32_t num_states, int32_t num_arcs, int32_t maxw,
              int32_t *__restrict__ in_splits, int32_t *__restrict__ in_arcs,
              int32_t *__restrict__ in_src, float *__restrict__ in_score) {
  extern __shared__ int32_t cnt_smem[];
  __shared__ int32_t scan_smem[8];
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t num_levels = level_offsets[num_fsas];
  if (blockIdx.x == 0 && threadIdx.x == 0) in_splits[num_states] = num_arcs;
  const int32_t lv = kWarps == 1 ? blockIdx.x * 4 + warp : blockIdx.x;
  if (lv >= num_levels) return;
  const int32_t b = level_splits[lv], w = level_splits[lv + 1] - b;
  if (w <= 0 || w > maxw) return;
  const int32_t fsa = row_ids1[b], s_begin = row_splits1[fsa];
  // the arcs that enter: all that leave the layer before (none enter an FSA's first layer)
  const int32_t pb = lv > level_offsets[fsa] ? level_splits[lv - 1] : b;
  const int32_t a0 = row_splits2[pb], a1 = pb < b ? row_splits2[b] : a0;
  int32_t *cnt = cnt_smem + (size_t)warp * maxw;  // this warp's counters
  int32_t *all = kWarps == 1 ? cnt : cnt_smem;
  const int tid = kWarps == 1 ? lane : threadIdx.x;
  constexpr int nt = 32 * kWarps;
  auto sync = [&]() { if (kWarps == 1) __syncwarp(); else __syncthreads(); };
  for (int32_t k = tid; k < w; k += nt)
#pragma unroll
    for (int u = 0; u < kWarps; ++u) all[(size_t)u * maxw + k] = 0;
  sync();
  // this warp's section of the arcs
  const int32_t per = ((a1 - a0 + nt - 1) / nt) * 32;
  const int32_t c0 = kWarps == 1 ? a0 : min(a0 + warp * per, a1);
  const int32_t c1 = kWarps == 1 ? a1 : min(c0 + per, a1);
  for (int32_t a = c0 + lane; a < c1; a += 32) {
    const int32_t d = s_begin + arcs[a].dest - b;
    if ((uint32_t)d < (uint32_t)w) atomicAdd(&cnt[d], 1);
  }
  sync();
  // first position of every destination (and of every warp's share of it)
  int32_t run = a0;
  for (int32_t k0 = 0; k0 < w; k0 += nt) {
    const int32_t k = k0 + tid;
    int32_t mine = 0;
    if (k < w)
#pragma unroll
      for (int u = 0; u < kWarps; ++u) mine += all[(size_t)u * maxw + k];
    int32_t inc = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int32_t o = __shfl_up_sync(kAll, inc, d);
      if (lane >= d) inc += o;
    }
    int32_t total = __shfl_sync(kAll, inc, 31);
    if (kWarps > 1) {
      if (lane == 31) scan_smem[warp] = inc;
      __syncthreads();
      total = 0;
#pragma unroll
      for (int u = 0; u < kWarps; ++u) {
        if (u < warp) inc += scan_smem[u];
        total += scan_smem[u];
      }
      __syncthreads();
    }
    if (k < w) {
      int32_t pos = run + inc - mine;
      in_splits[b + k] = pos;
#pragma unroll
      for (int u = 0; u < kWarps; ++u) {
        const int32_t n = all[(size_t)u * maxw + k];
        all[(size_t)u * maxw + k] = pos;
        pos += n;
      }
    }
    run += total;
  }
  sync();
  for (int32_t a = c0; a < c1; a += 32) {
    Arc arc;
    int32_t d = -1 - lane;  // lanes without an arc match nobody
    if (a + lane < c1) {
      arc = arcs[a + lane];
      const int32_t x = s_begin + arc.dest - b;
      if ((uint32_t)x < (uint32_t)w) d = x;
    }
    const unsigned same = __match_any_sync(kAll, d);
    const int32_t rank = __popc(same & ((1u << lane) - 1u));
    int32_t pos = 0;
    if (d >= 0) pos = cnt[d];
    __syncwarp();
    if (d >= 0) {
      pos += rank;
      if (lane == 31 - __clz(same)) cnt[d] = pos + 1;
      in_arcs[pos] = a + lane;
      in_src[pos] = s_begin + arc.src;
      in_score[pos] = arc.score;
    }
    __syncwarp();
  }
}

int32_t BuildLayerIncoming(const k2b200_fsa_view *v, int32_t *in_splits, int32_t *in_arcs,
                           int32_t *in_src, float *in_score, cudaStream_t stream, bool *done) {
  *done = false;
  const int32_t maxw = std::max(v->max_layer_states, 1);
  const int64_t levels = (int64_t)v->max_layers * v->num_fsas;  // at least the true number
  if (!v->strict_layers || levels <= 0 || levels >= ((int64_t)1 << 31)) return kOk;
  // a warp per layer while layers are small (there are many of them), else four; with fewer
  // for the widest layers (10^4 states, 4 10^4 arcs) sorting the whole FsaVec is faster
  const bool one = maxw <= 1024 && v->num_arcs / levels <= 1024;
  const size_t smem = sizeof(int32_t) * 4 * (size_t)maxw;
  if (smem > kLayerSmemBudget) return kOk;
  auto kernel = one ? LayerIncoming<1> : LayerIncoming<4>;
  K2B_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kLayerSmemBudget));
  { kernel<<<one ? CeilDiv(levels, 4) : (int)levels, 128, smem, stream>>>(
      v->row_splits1, v->row_ids1, v->row_splits2, reinterpret_cast<const Arc *>(v->arcs),
      v->level_offsets, v->level_splits, v->num_fsas, v->num_states, v->num_arcs, maxw, in_splits,
      in_arcs, in_src, in_score); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  *done = true;
  return kOk;
}

// ---------------------------------------------------------------------------
// records of the arcs, in incoming and / or leaving order
// ---------------------------------------------------------------------------
template <bool kLog>
__global__ void PackLayerArcs(k2b200_fsa_view v, LayerArc *__restrict__ fwd,
                              LayerArc *__restrict__ bwd, int32_t *__restrict__ status) {
  const int32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= v.num_arcs) return;
  auto pack = [&](float score, int32_t other, int32_t arc) {
    LayerArc r;
    r.w = kLog ? exp((double)score) : (double)score;
    r.other = other;
    r.arc = arc;
    if (kLog && score != -INFINITY && !(fabsf(score) <= kMaxScore)) atomicOr(status, 4);
    return r;
  };
  if (fwd) fwd[k] = pack(v.in_score[k], v.in_src[k], v.in_arcs[k]);
  if (bwd) {
    const Arc arc = reinterpret_cast<const Arc *>(v.arcs)[k];
    bwd[k] = pack(arc.score, v.row_ids2[k] - arc.src + arc.dest, k);
  }
}

struct ChainPlan {
  int32_t maxw, nl_cap, cap_arcs, splits_ints, slot_bytes, slots, warps, group_log2;
  int32_t wide, team;
  size_t bytes;
  bool ok;
};

static ChainPlan PlanChain(const k2b200_fsa_view *v, int32_t ndir) {
  ChainPlan p = {};
  if (!v->strict_layers || v->max_layer_states <= 0 || v->max_layer_arcs < 0 || v->max_layers <= 0)
    return p;
  p.maxw = (v->max_layer_states + 3) & ~3;
  p.nl_cap = v->max_layers;
  const size_t bounds = 2 * sizeof(int32_t) * (size_t)((p.nl_cap + 1 + 3) & ~3);
  const size_t fixed = bounds + 2 * sizeof(double) * (size_t)p.maxw;
  const int64_t layers = (int64_t)v->num_fsas * v->max_layers;
  const int32_t mean_w = (int32_t)((v->num_states + layers - 1) / layers),
                mean_a = (int32_t)((v->num_arcs + layers - 1) / layers);
  // Eight lanes per state when states have many arcs, else one.  A warp costs a layer some
  // hundred instructions whatever it does, and one that runs alone issues one in about five
  // cycles: as many warps as a mean layer fills, at most 16.
  p.group_log2 = mean_a >= 6 * (int64_t)mean_w ? 3 : 0;
  p.warps = std::max(1, std::min(16, CeilDiv((int64_t)mean_w << p.group_log2, 32)));
  p.cap_arcs = std::max(v->max_layer_arcs, 512);
  p.splits_ints = (std::max(p.maxw, 256) + kChunkLayers + 8 + 3) & ~3;
  p.slot_bytes = p.cap_arcs * (int32_t)sizeof(LayerArc) + p.splits_ints * (int32_t)sizeof(int32_t);
  // with more CTAs than SMs, two of them should share one
  const size_t budget =
      (int64_t)ndir * v->num_fsas > 148 ? kLayerSmemBudget / 2 : kLayerSmemBudget;
  for (size_t limit : {budget, kLayerSmemBudget}) {
    if (fixed + 3 * (size_t)p.slot_bytes <= limit) {
      p.slots = (int32_t)std::min<size_t>(4, (limit - fixed) / p.slot_bytes);
      p.bytes = fixed + (size_t)p.slots * p.slot_bytes;
      p.ok = true;
      return p;
    }
  }
  // Layers too wide for that are shared by a cluster of CTAs.
  p.wide = 1;
  p.warps = 16;
  p.team = 1;
  while (p.team < 8 && (int64_t)ndir * v->num_fsas * p.team * 2 <= 148 &&
         p.team * 32 * p.warps < v->max_layer_states)
    p.team *= 2;
  p.bytes = bounds;
  p.ok = p.bytes <= kLayerSmemBudget;
  return p;
}

// The sum over a state's arcs (log) or its best entering arc (tropical).
template <typename Val, bool kLog>
struct StateSum {
  Val acc;
  int32_t best;
  __device__ __forceinline__ void Clear() {
    acc = kLog ? (Val)0 : (Val)-INFINITY;
    best = -1;
  }
  // arcs of a lane come in increasing order; ties: the later arc wins (ragged_ops_inl.h:649-655)
  __device__ __forceinline__ void Add(const LayerArc &r, Val x) {
    if (kLog) {
      acc = (Val)fma(r.w, (double)x, (double)acc);
    } else {
      const Val y = x + (Val)r.w;
      if (y >= acc) {
        acc = y;
        best = r.arc;
      }
    }
  }
  __device__ __forceinline__ void Merge(const StateSum &o) {
    if (kLog) {
      acc += o.acc;
    } else if (o.acc > acc || (o.acc == acc && o.best > best)) {
      acc = o.acc;
      best = o.best;
    }
  }
  // the same result on all lanes of every aligned group of `lanes`
  __device__ __forceinline__ void Across(int lanes) {
    for (int d = lanes >> 1; d > 0; d >>= 1) {
      StateSum o;
      o.acc = __shfl_xor_sync(0xffffffffu, acc, d);
      o.best = kLog ? 0 : __shfl_xor_sync(0xffffffffu, best, d);
      Merge(o);
    }
  }
  // arcs k, k + step, ... below k1; rec(k) and val(record) fetch
  template <typename Rec, typename Value>
  __device__ __forceinline__ void Walk(int32_t k, int32_t k1, int32_t step, Rec rec, Value val) {
    for (; k + 3 * step < k1; k += 4 * step) {
      LayerArc r[4];
      Val x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) r[u] = rec(k + u * step);
#pragma unroll
      for (int u = 0; u < 4; ++u) x[u] = val(r[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) Add(r[u], x[u]);
    }
    for (; k < k1; k += step) {
      const LayerArc r = rec(k);
      Add(r, val(r));
    }
  }
  // The states of the lanes in `heavy` (their arcs k0 .. k1 - 1), the whole warp on one at a
  // time; a lane whose state is not among them keeps what it has.
  template <typename Rec, typename Value>
  __device__ __forceinline__ void Heavy(unsigned heavy, int lane, int32_t k0, int32_t k1, Rec rec,
                                        Value val) {
    for (; heavy; heavy &= heavy - 1) {  // uniform
      const int owner = __ffs(heavy) - 1;
      StateSum q;
      q.Clear();
      q.Walk(__shfl_sync(0xffffffffu, k0, owner) + lane, __shfl_sync(0xffffffffu, k1, owner), 32,
             rec, val);
      q.Across(32);
      if (lane == owner) *this = q;
    }
  }
};

// The shared power of two of the log semiring: 2^K, replaced every kRescale layers by the
// exponent of the largest value since.  hi_slots: two words that the CTAs of a chain share.
template <bool kLog>
struct ChainScale {
  double mul = 1.0;
  int32_t K = 0, hi_max = 0;
  uint32_t min_hi = 0xffffffffu;
  __device__ __forceinline__ void BeginLayer(int32_t step, int32_t *hi_slots, bool first_thread) {
    if (!kLog) return;
    mul = 1.0;
    const int at = (step / kRescale) & 1;
    if (step % kRescale == 0 && step > 0) {
      const int32_t hm = *reinterpret_cast<volatile int32_t *>(&hi_slots[at ^ 1]);
      const int32_t e = hm > 0 ? (hm >> 20) - 1023 : 0;
      K += e;
      mul = __longlong_as_double((long long)(1023 - e) << 52);
    }
    if (step % kRescale == 1 && first_thread)
      *reinterpret_cast<volatile int32_t *>(&hi_slots[at ^ 1]) = 0;
  }
  __device__ __forceinline__ void Note(double x) {  // x >= 0
    if (!kLog) return;
    const int32_t hi = __double2hiint(x);
    hi_max = max(hi_max, hi);
    min_hi = min(min_hi, (uint32_t)hi - 1u);  // a zero does not count
  }
  __device__ __forceinline__ void EndLayer(int32_t step, int32_t *hi_slots, int lane,
                                           int32_t *status) {
    if (!kLog || step % kRescale != kRescale - 1) return;
    const int32_t hm = __reduce_max_sync(0xffffffffu, hi_max);
    if (lane == 0 && hm > 0) atomicMax(&hi_slots[(step / kRescale) & 1], hm);
    if (hm >= (1023 + kRangeExp) << 20 && lane == 0) atomicOr(status, 4);
    hi_max = 0;
  }
  __device__ __forceinline__ void End(int lane, int32_t *status) {
    if (!kLog) return;
    const int32_t hm = __reduce_max_sync(0xffffffffu, hi_max);
    const uint32_t hn = __reduce_min_sync(0xffffffffu, min_hi);
    if (lane == 0 && (hm >= (1023 + kRangeExp) << 20 ||
                      hn < (uint32_t)(((1023 - kRangeExp) << 20) - 1)))
      atomicOr(status, 4);
  }
};

// grid = (directions, fsas).  val_fwd / val_bwd: values per state (log: doubles relative to
// 2^scale[(dir * num_fsas + i) * nl_cap + layer]).  kGroup lanes per state (1 or 8).
template <typename Val, bool kLog, int kGroup>
__global__ void __launch_bounds__(544, 1)
LayerChain(k2b200_fsa_view v, const LayerArc *__restrict__ fwd_arcs,
           const LayerArc *__restrict__ bwd_arcs, Val *__restrict__ val_fwd,
           Val *__restrict__ val_bwd, int32_t *__restrict__ entering, int32_t *__restrict__ scale,
           int32_t dir_base, int32_t fsa_base, ChainPlan p, int32_t *__restrict__ status) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  constexpr unsigned kAll = 0xffffffffu;
  const int32_t i = fsa_base + blockIdx.y, dir = blockIdx.x + dir_base;
  const int32_t s_begin = v.row_splits1[i], s_end = v.row_splits1[i + 1];
  if (s_end == s_begin) return;
  const int32_t lv0 = v.level_offsets[i], nl = v.level_offsets[i + 1] - lv0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nw = p.warps;
  Val *out = dir == 0 ? val_fwd : val_bwd;
  const int32_t lvl_ints = (p.nl_cap + 1 + 3) & ~3;
  // everything in shared memory is addressed by index, so that it stays in that space
  const LayerArc *recs = reinterpret_cast<const LayerArc *>(smem_raw);
  int32_t *ints = reinterpret_cast<int32_t *>(smem_raw);
  const size_t vals_at = (size_t)p.slots * p.slot_bytes;
  Val *vals = reinterpret_cast<Val *>(smem_raw + vals_at);  // [2][maxw]
  int32_t *lvl = reinterpret_cast<int32_t *>(smem_raw + vals_at + 16 * (size_t)p.maxw);
  int32_t *alvl = lvl + lvl_ints;
  const int32_t *gsplits = dir == 0 ? v.in_splits : v.row_splits2;
  const LayerArc *garcs = dir == 0 ? fwd_arcs : bwd_arcs;
  __shared__ __align__(8) uint64_t full[kMaxSlots], empty[kMaxSlots];
  __shared__ int32_t chunk_layers[kMaxSlots];
  __shared__ int32_t bad_shared, hi_shared[2];
  if (tid == 0) {
    bad_shared = nl > p.nl_cap;
    hi_shared[0] = hi_shared[1] = 0;
    for (int32_t s = 0; s < p.slots; ++s) {
      MbarInit(&full[s], 1);
      MbarInit(&empty[s], nw);  // one arrival per warp
    }
    MbarInitFence();
  }
  __syncthreads();
  if (!bad_shared)
    for (int32_t k = tid; k <= nl; k += blockDim.x) {
      const int32_t s = v.level_splits[lv0 + k];
      lvl[k] = s;
      alvl[k] = gsplits[s];
    }
  __syncthreads();
  if (!bad_shared) {
    bool bad = false;
    for (int32_t k = tid; k < nl; k += blockDim.x)
      bad |= lvl[k + 1] - lvl[k] > p.maxw || alvl[k + 1] - alvl[k] > p.cap_arcs;
    if (bad) bad_shared = 1;
  }
  __syncthreads();
  if (bad_shared) {  // the caller's bounds do not hold: the general kernel takes the call
    if (tid == 0) atomicOr(status, 1);
    return;
  }
  const int32_t slot_recs = p.slot_bytes >> 4, slot_ints = p.slot_bytes >> 2;
  if (warp == nw) {
    // ---- the producer: one lane keeps the ring full ---------------------------------
    if (lane != 0) return;
    const int32_t splits_end = (v.num_states + 1) & ~3;  // last multiple of 4 in the splits
    int32_t slot = 0, issued = 0;
    unsigned parity = 1;  // a fresh barrier counts as "previous phase complete"
    for (int32_t done = 0; done < nl;) {
      int32_t lo, hi;  // layers lo .. hi - 1
      if (dir == 0) {
        lo = done;
        hi = lo + 1;
        while (hi < nl && hi - lo < kChunkLayers && alvl[hi + 1] - alvl[lo] <= p.cap_arcs &&
               lvl[hi + 1] - lvl[lo] + 8 <= p.splits_ints)
          ++hi;
      } else {
        hi = nl - done;
        lo = hi - 1;
        while (lo > 0 && hi - lo < kChunkLayers && alvl[hi] - alvl[lo - 1] <= p.cap_arcs &&
               lvl[hi] - lvl[lo - 1] + 8 <= p.splits_ints)
          --lo;
      }
      done += hi - lo;
      if (!MbarWaitBounded(&empty[slot], parity)) {
        atomicOr(status, 2);
        break;
      }
      const int32_t b = lvl[lo], e = lvl[hi];
      int32_t *sp = ints + slot * slot_ints + p.cap_arcs * 4;
      const int32_t c0 = b & ~3, c1 = max(c0, min((e + 1 + 3) & ~3, splits_end));
      for (int32_t k = c1; k <= e; ++k) sp[k - c0] = gsplits[k];  // at most 3 trailing ints
      chunk_layers[slot] = hi - lo;
      const unsigned bytes_s = (unsigned)(c1 - c0) * 4u,
                     bytes_a = (unsigned)(alvl[hi] - alvl[lo]) * (unsigned)sizeof(LayerArc);
      MbarArriveExpectTx(&full[slot], bytes_s + bytes_a);
      if (bytes_s) BulkCopyG2S(sp, gsplits + c0, bytes_s, &full[slot]);
      if (bytes_a)
        BulkCopyG2S(smem_raw + (size_t)slot * p.slot_bytes, garcs + alvl[lo], bytes_a, &full[slot]);
      slot = slot + 1 == p.slots ? 0 : slot + 1;
      parity ^= (slot == 0);
      ++issued;
    }
    // no copy is in flight towards this CTA's shared memory when it retires
    for (int32_t k = max(0, issued - p.slots); k < issued; ++k)
      MbarWaitBounded(&full[k % p.slots], (unsigned)(k / p.slots) & 1u);
    return;
  }

  // ---- the chain -----------------------------------------------------------------------
  const int32_t root = dir == 0 ? s_begin : s_end - 1, nc = 32 * nw;
  const int32_t per_trip = nc / kGroup;  // states that one trip of all lanes takes
  int32_t *my_scale = kLog ? scale + ((int64_t)dir * v.num_fsas + i) * p.nl_cap : nullptr;
  ChainScale<kLog> sc;
  auto layer_sync = [&]() {
    if (nw == 1) __syncwarp();
    else asm volatile("bar.sync 1, %0;" ::"r"(nc) : "memory");
  };
  // the layer whose splits and first records are fetched, one layer ahead of the chain
  struct Ahead {
    int32_t b, e;         // its states
    int32_t body, splits; // where the records / splits of its chunk start in shared memory
    int32_t slot;         // >= 0: the chunk ends with this layer
    int32_t s, k0, k1;    // this lane's state and its arcs
    LayerArc r0;          // first of them
  };
  int32_t slot = p.slots - 1, left = 0, body = 0, splits = 0;
  unsigned parity = 1;
  bool opened = false;  // a chunk was waited for since the last barrier
  const int32_t mine_at = tid / kGroup;
  auto fetch = [&](int32_t step, Ahead &f) {
    const int32_t l = dir == 0 ? step : nl - 1 - step;
    f.b = lvl[l];
    f.e = lvl[l + 1];
    if (left == 0) {
      slot = slot + 1 == p.slots ? 0 : slot + 1;
      parity ^= (slot == 0);
      if (!MbarWaitBounded(&full[slot], parity)) {
        atomicOr(status, 2);
        *reinterpret_cast<volatile int32_t *>(&bad_shared) = 2;
      }
      opened = true;
      left = chunk_layers[slot];
      const int32_t lo = dir == 0 ? l : l - left + 1;
      body = slot * slot_recs - alvl[lo];
      splits = slot * slot_ints + p.cap_arcs * 4 - (lvl[lo] & ~3);
    }
    --left;
    f.slot = left == 0 ? slot : -1;
    f.body = body;
    f.splits = splits;
    f.s = f.b + mine_at;
    f.k0 = f.k1 = 0;
    if (f.s < f.e) {
      f.k0 = ints[splits + f.s];
      f.k1 = ints[splits + f.s + 1];
      if (kGroup == 1 && f.k0 < f.k1) f.r0 = recs[body + f.k0];
    }
  };
  int32_t prev_at = p.maxw, cur_at = 0, pb = 0;  // values of the layer before, of this layer
  auto layer = [&](int32_t step, Ahead &now, Ahead &next) -> bool {
    if (step + 1 < nl) fetch(step + 1, next);
    sc.BeginLayer(step, hi_shared, tid == 0);
    const int32_t prev = prev_at - pb, cur = cur_at - now.b;
    int32_t s = now.s, k0 = now.k0, k1 = now.k1;
    auto rec = [&](int32_t k) { return recs[now.body + k]; };
    auto val = [&](const LayerArc &r) { return vals[prev + r.other]; };
    for (int32_t s0 = now.b;;) {
      StateSum<Val, kLog> q;
      q.Clear();
      if (kGroup == 1) {
        const int32_t deg = k1 - k0;
        const unsigned heavy = __ballot_sync(kAll, deg > kLight);
        if (deg > 0 && deg <= kLight) {
          if (s0 == now.b) {
            q.Add(now.r0, val(now.r0));
            ++k0;
          }
          for (; k0 < k1; ++k0) {
            const LayerArc r = rec(k0);
            q.Add(r, val(r));
          }
        }
        if (heavy) q.Heavy(heavy, lane, k0, k1, rec, val);
      } else {
        q.Walk(k0 + (lane & (kGroup - 1)), k1, kGroup, rec, val);
        q.Across(kGroup);
      }
      if (s < now.e && (kGroup == 1 || (lane & (kGroup - 1)) == 0)) {
        if (kLog) {
          q.acc = q.acc * (Val)sc.mul;
          if (q.acc == (Val)0 && s == root) q.acc = (Val)1;
          sc.Note((double)q.acc);
        } else {
          if (q.acc == (Val)-INFINITY && s == root) q.acc = (Val)0;
          if (entering != nullptr && dir == 0) entering[s] = q.best;
        }
        vals[cur + s] = q.acc;
        out[s] = q.acc;
      }
      s0 += per_trip;
      if (s0 >= now.e) break;  // uniform
      s += per_trip;
      k0 = k1 = 0;
      if (s < now.e) {
        k0 = ints[now.splits + s];
        k1 = ints[now.splits + s + 1];
      }
    }
    sc.EndLayer(step, hi_shared, lane, status);
    if (kLog && tid == 0) my_scale[dir == 0 ? step : nl - 1 - step] = sc.K;
    if (now.slot >= 0) {  // this warp has read the chunk
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(SmemAddr(&empty[now.slot]))
                     : "memory");
    }
    pb = now.b;
    const int32_t t = prev_at;
    prev_at = cur_at;
    cur_at = t;
    layer_sync();
    if (opened) {
      if (*reinterpret_cast<volatile int32_t *>(&bad_shared)) return false;  // uniform
      opened = false;
    }
    return true;
  };
  Ahead f0, f1;
  fetch(0, f0);
  for (int32_t step = 0; step < nl; step += 2) {
    if (!layer(step, f0, f1)) break;
    if (step + 1 < nl && !layer(step + 1, f1, f0)) break;
  }
  sc.End(lane, status);
}

// The same for layers too wide for the ring: the CTAs of a cluster share a layer.  grid =
// (directions x team, fsas).  Splits, records and the values of the layer before come from
// L2; what does not depend on values is fetched a layer ahead, so that a layer costs one
// gather and one cluster barrier, a microsecond, whatever its width (up to team x 512 states
// a trip).
template <typename Val, bool kLog>
__global__ void __launch_bounds__(512, 1)
LayerChainWide(k2b200_fsa_view v, const LayerArc *__restrict__ fwd_arcs,
               const LayerArc *__restrict__ bwd_arcs, Val *val_fwd, Val *val_bwd,
               int32_t *__restrict__ entering, int32_t *__restrict__ scale, int32_t *hi_slots,
               int32_t dir_base, int32_t fsa_base, ChainPlan p, int32_t *__restrict__ status) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  constexpr unsigned kAll = 0xffffffffu;
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  const int32_t rank = (int32_t)cluster.block_rank(), team = p.team;
  const int32_t i = fsa_base + blockIdx.y, dir = (int32_t)blockIdx.x / team + dir_base;
  const int32_t s_begin = v.row_splits1[i], s_end = v.row_splits1[i + 1];
  const int32_t lv0 = v.level_offsets[i], nl = v.level_offsets[i + 1] - lv0;
  if (s_end == s_begin) return;  // uniform over the cluster, as is the next return
  const int tid = threadIdx.x, lane = tid & 31;
  Val *out = dir == 0 ? val_fwd : val_bwd;
  int32_t *lvl = reinterpret_cast<int32_t *>(smem_raw);
  const int32_t *gsplits = dir == 0 ? v.in_splits : v.row_splits2;
  const LayerArc *garcs = dir == 0 ? fwd_arcs : bwd_arcs;
  if (nl > p.nl_cap) {
    if (tid == 0) atomicOr(status, 1);
    return;
  }
  for (int32_t k = tid; k <= nl; k += blockDim.x) lvl[k] = v.level_splits[lv0 + k];
  int32_t *my_hi = hi_slots + 2 * ((int64_t)dir * v.num_fsas + i);
  __syncthreads();
  const int32_t root = dir == 0 ? s_begin : s_end - 1;
  const int32_t nt = team * 512, at = rank * 512 + tid;
  int32_t *my_scale = kLog ? scale + ((int64_t)dir * v.num_fsas + i) * p.nl_cap : nullptr;
  ChainScale<kLog> sc;
  auto layer_sync = [&]() {
    if (team == 1) __syncthreads(); else cluster.sync();
  };
  auto layer_of = [&](int32_t step) { return dir == 0 ? step : nl - 1 - step; };
  struct Ahead {
    int32_t k0, k1;
    LayerArc r0;
  };
  auto fetch_splits = [&](int32_t step, Ahead &f) {
    f.k0 = f.k1 = 0;
    if (step >= nl) return;
    const int32_t l = layer_of(step), s = lvl[l] + at;
    if (s < lvl[l + 1]) {
      f.k0 = __ldg(gsplits + s);
      f.k1 = __ldg(gsplits + s + 1);
    }
  };
  auto fetch_record = [&](Ahead &f) {
    if (f.k0 < f.k1) f.r0 = garcs[f.k0];
  };
  auto rec = [&](int32_t k) { return garcs[k]; };
  auto val = [&](const LayerArc &r) { return __ldcg(out + r.other); };
  Ahead now, next, after;
  fetch_splits(0, now);
  fetch_record(now);
  fetch_splits(1, next);
  for (int32_t step = 0; step < nl; ++step) {
    fetch_record(next);
    fetch_splits(step + 2, after);
    const int32_t l = layer_of(step), b = lvl[l], e = lvl[l + 1];
    sc.BeginLayer(step, my_hi, rank == 0 && tid == 0);
    for (int32_t s0 = b; s0 < e; s0 += nt) {
      const int32_t s = s0 + at;
      if (s0 > b) {
        now.k0 = now.k1 = 0;
        if (s < e) {
          now.k0 = __ldg(gsplits + s);
          now.k1 = __ldg(gsplits + s + 1);
        }
        fetch_record(now);
      }
      StateSum<Val, kLog> q;
      q.Clear();
      int32_t k0 = now.k0;
      const int32_t k1 = now.k1, deg = k1 - k0;
      const unsigned heavy = __ballot_sync(kAll, deg > kLight);
      if (deg > 0 && deg <= kLight) {
        q.Add(now.r0, val(now.r0));
        q.Walk(k0 + 1, k1, 1, rec, val);
      }
      if (heavy) q.Heavy(heavy, lane, k0, k1, rec, val);
      if (s < e) {
        if (kLog) {
          q.acc = q.acc * (Val)sc.mul;
          if (q.acc == (Val)0 && s == root) q.acc = (Val)1;
          sc.Note((double)q.acc);
        } else {
          if (q.acc == (Val)-INFINITY && s == root) q.acc = (Val)0;
          if (entering != nullptr && dir == 0) entering[s] = q.best;
        }
        __stcg(out + s, q.acc);
      }
    }
    sc.EndLayer(step, my_hi, lane, status);
    if (kLog && rank == 0 && tid == 0) my_scale[l] = sc.K;
    layer_sync();
    now = next;
    next = after;
  }
  sc.End(lane, status);
}

// out[s] = log(m[s]) + scale of its layer * ln 2.  grid = (layer tiles, fsas, parts of a
// layer), `lanes` threads (a power of two) on a part.  m and out may be the same array.
template <typename Real>
__global__ void __launch_bounds__(128)
FinishLayerScores(k2b200_fsa_view v, const double *m, const int32_t *__restrict__ scale,
                  int32_t nl_cap, int32_t fsa_base, int32_t lanes, Real *out) {
  const int32_t lane = threadIdx.x & (lanes - 1);
  const int32_t i = fsa_base + blockIdx.y,
                l = (blockIdx.x * blockDim.x + threadIdx.x) / (unsigned)lanes;
  const int32_t lv = v.level_offsets[i] + l;
  if (l >= nl_cap || lv >= v.level_offsets[i + 1]) return;
  const int32_t b = v.level_splits[lv], e = v.level_splits[lv + 1];
  const double shift = (double)scale[(int64_t)i * nl_cap + l] * 0.69314718055994530942;
  for (int32_t s = b + (int32_t)blockIdx.z * lanes + lane; s < e; s += (int32_t)gridDim.z * lanes) {
    const double x = m[s];
    out[s] = x == 0.0 ? (Real)-INFINITY : (Real)(log(x) + shift);
  }
}

namespace {
struct ChainScratch {
  LayerArc *fwd_arcs, *bwd_arcs;
  int32_t *scale, *status;  // status and the words of ChainScale are cleared together
  double *vals;  // [2][num_states], for results in float
  size_t clear_bytes, bytes;
};
}  // namespace

static ChainScratch CarveScratch(const k2b200_fsa_view *v, void *scratch) {
  ChainScratch c;
  char *base = reinterpret_cast<char *>(scratch);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off += AlignUp(std::max<size_t>(bytes, 1));
    return base + at;
  };
  const size_t na = (size_t)std::max(v->num_arcs, 1), ns = (size_t)std::max(v->num_states, 1);
  c.clear_bytes = sizeof(int32_t) * (4 + 4 * (size_t)v->num_fsas);
  c.status = reinterpret_cast<int32_t *>(take(c.clear_bytes));
  c.fwd_arcs = reinterpret_cast<LayerArc *>(take(sizeof(LayerArc) * na));
  c.bwd_arcs = reinterpret_cast<LayerArc *>(take(sizeof(LayerArc) * na));
  c.scale = reinterpret_cast<int32_t *>(
      take(sizeof(int32_t) * 2 * (size_t)v->num_fsas * (size_t)std::max(v->max_layers, 1)));
  c.vals = reinterpret_cast<double *>(take(sizeof(double) * 2 * ns));
  c.bytes = off;
  return c;
}

size_t LayerScratchBytes(const k2b200_fsa_view *v) { return CarveScratch(v, nullptr).bytes; }

int32_t *LayerStatusWord(const k2b200_fsa_view *v, void *scratch) {
  return CarveScratch(v, scratch).status;
}

template <typename Val, bool kLog>
static int32_t LaunchChain(const k2b200_fsa_view *v, const ChainScratch &c, const ChainPlan &p,
                           Val *val_fwd, Val *val_bwd, int32_t *entering, cudaStream_t stream) {
  const int32_t ndir = (val_fwd != nullptr) + (val_bwd != nullptr), dir_base = val_fwd ? 0 : 1;
  if (p.wide)
    K2B_CUDA_OK(cudaFuncSetAttribute(LayerChainWide<Val, kLog>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kLayerSmemBudget));
  auto kernel = p.group_log2 ? LayerChain<Val, kLog, 8> : LayerChain<Val, kLog, 1>;
  K2B_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kLayerSmemBudget));
  for (int32_t first = 0; first < v->num_fsas; first += 65535) {
    const int32_t n = std::min(v->num_fsas - first, 65535);
    if (!p.wide) {
      { kernel<<<dim3(ndir, n), 32 * (p.warps + 1), p.bytes, stream>>>(
          *v, c.fwd_arcs, c.bwd_arcs, val_fwd, val_bwd, entering, c.scale, dir_base, first, p,
          c.status); NoteLaunch(); }
      continue;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ndir * p.team, n);
    cfg.blockDim = dim3(32 * p.warps);
    cfg.dynamicSmemBytes = p.bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = p.team;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    K2B_CUDA_OK(cudaLaunchKernelEx(&cfg, LayerChainWide<Val, kLog>, *v,
                                   (const LayerArc *)c.fwd_arcs, (const LayerArc *)c.bwd_arcs,
                                   val_fwd, val_bwd, entering, c.scale, c.status + 4, dir_base,
                                   first, p, c.status));
    NoteLaunch();
  }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

template <typename Real>
int32_t LaunchLayerScores(const k2b200_fsa_view *v, int32_t log_semiring, Real *fwd, Real *bwd,
                          int32_t *entering, void *scratch, size_t scratch_bytes,
                          cudaStream_t stream, bool *launched) {
  *launched = false;
  if (scratch == nullptr || v->num_arcs == 0 || v->row_ids2 == nullptr) return kOk;
  if (fwd != nullptr && (v->in_src == nullptr || v->in_score == nullptr)) return kOk;
  const ChainPlan p = PlanChain(v, (fwd != nullptr) + (bwd != nullptr));
  const ChainScratch c = CarveScratch(v, scratch);
  if (!p.ok || scratch_bytes < c.bytes) return kOk;
  // bulk copies need 16-byte aligned sources
  auto aligned16 = [](const void *ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0; };
  if (!aligned16(scratch) || !aligned16(v->row_splits2) || (fwd && !aligned16(v->in_splits)))
    return kOk;
  K2B_CUDA_OK(cudaMemsetAsync(c.status, 0, c.clear_bytes, stream));
  auto pack = log_semiring ? PackLayerArcs<true> : PackLayerArcs<false>;
  { pack<<<CeilDiv(v->num_arcs, 256), 256, 0, stream>>>(*v, fwd ? c.fwd_arcs : nullptr,
                                                        bwd ? c.bwd_arcs : nullptr, c.status);
    NoteLaunch(); }
  if (log_semiring) {
    const bool in_place = sizeof(Real) == sizeof(double);
    double *vf = in_place ? reinterpret_cast<double *>(fwd) : c.vals,
           *vb = in_place ? reinterpret_cast<double *>(bwd) : c.vals + v->num_states;
    K2B_FORWARD((LaunchChain<double, true>(v, c, p, fwd ? vf : nullptr, bwd ? vb : nullptr,
                                           nullptr, stream)));
    for (int dir = 0; dir < 2; ++dir) {
      Real *out = dir == 0 ? fwd : bwd;
      if (out == nullptr) continue;
      for (int32_t first = 0; first < v->num_fsas; first += 65535) {
        // a few states per thread of a mean layer
        const int32_t mean_w =
            (int32_t)(v->num_states / std::max<int64_t>((int64_t)v->num_fsas * p.nl_cap, 1));
        int32_t lanes = 4;
        while (lanes < 128 && lanes < mean_w) lanes *= 2;
        dim3 grid(CeilDiv((int64_t)p.nl_cap * lanes, 128), std::min(v->num_fsas - first, 65535),
                  std::min(16, 1 + mean_w / 512));
        { FinishLayerScores<Real><<<grid, 128, 0, stream>>>(
            *v, dir == 0 ? vf : vb, c.scale + (int64_t)dir * v->num_fsas * p.nl_cap, p.nl_cap,
            first, lanes, out); NoteLaunch(); }
      }
    }
  } else {
    K2B_FORWARD((LaunchChain<Real, false>(v, c, p, fwd, bwd, entering, stream)));
  }
  K2B_CUDA_OK(cudaGetLastError());
  *launched = true;
  return kOk;
}

template int32_t LaunchLayerScores<float>(const k2b200_fsa_view *, int32_t, float *, float *,
                                          int32_t *, void *, size_t, cudaStream_t, bool *);
template int32_t LaunchLayerScores<double>(const k2b200_fsa_view *, int32_t, double *, double *,
                                           int32_t *, void *, size_t, cudaStream_t, bool *);

}  // namespace k2b
