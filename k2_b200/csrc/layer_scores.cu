// Forward/backward scores of a strictly layered FsaVec: every arc goes from one layer
// to the next, as in the lattices that the dense intersections emit (frames are layers).
// Reference arithmetic: k2/csrc/fsa_utils.cu:1124-1278, :1345-1454.
//
// The recursion is a chain of T dependent layers, so what bounds it is the latency of one
// layer, and the rest of the work is moved off that chain:
//   * SliceLayers lays the arcs of every layer out for the chain: one 16-byte record per arc
//     with exp(score) as a double for the log semiring (the score itself for the tropical
//     one), dealt out evenly to lanes and stored so that a warp reads a row of 32 records
//     without conflicts.  The arcs that enter a layer are exactly those that leave the layer
//     before, so no incoming-arc index of the FsaVec is needed.
//   * SliceChain, one CTA per (FSA, direction), then needs one multiply-add per arc: values
//     of a layer are plain doubles that share a power of two, which follows the largest of
//     them every kRescale layers.  What that cannot hold (arc scores beyond +-kMaxScore,
//     values more than 2^280 away from it) raises the status word, and ExactChain, launched
//     behind and otherwise returning at once, redoes the call.
//   * FinishLayerScores takes the logarithms, all states in parallel.
// Layers come through a ring in shared memory, many small ones per slot, each by a bulk copy
// that an extra warp issues ahead of the chain.  Lattices with layers too wide for a slot
// (decoding: thousands of states per frame) go to LayerChainWide, a cluster of CTAs per chain,
// which reads records in incoming / leaving order from L2 (LayerIncoming, PackLayerArcs).
#include <algorithm>

#include <cooperative_groups.h>

#include "../../include/k2b200.h"
#include "common.cuh"
#include "cp_async.cuh"
#include "prob_math.cuh"
#include "scores_internal.cuh"

namespace k2b {

constexpr size_t kLayerSmemBudget = 200 * 1024;
constexpr int kRescale = 4;           // layers between changes of the shared exponent
constexpr float kMaxScore = 300.0f;   // |arc score|: exp() within 2^+-433
constexpr int kRangeExp = 280;        // values that are not zero stay within 2^+-280, so that no
                                      // product of one with a factor and a scale underflows
constexpr int kMaxSlots = 8;
constexpr int kWideTeam = 8, kWideWarps = 16;  // CTAs that share a layer, warps of each
constexpr int kWideRecs = 2;                   // records of a lane ahead
constexpr int kDrainTests = 1 << 16;           // a millisecond, for stores that take microseconds
constexpr int kSliceMaxStates = 16384;  // states of a sliced layer

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
  int32_t maxw, nl_cap, warps;
  // sliced layers
  int32_t rows, slots, slot_bytes;
  // wide layers
  int32_t wide, team, cells;
  size_t bytes;
  bool ok;
};

static ChainPlan PlanChain(const k2b200_fsa_view *v, int32_t ndir, bool log_semiring) {
  ChainPlan p = {};
  if (!v->strict_layers || v->max_layer_states <= 0 || v->max_layer_arcs < 0 ||
      v->max_layers <= 0 || (int64_t)v->num_fsas * v->max_layers > INT32_MAX)
    return p;
  p.maxw = (v->max_layer_states + 3) & ~3;
  p.nl_cap = v->max_layers;
  const int64_t layers = (int64_t)v->num_fsas * v->max_layers;
  const int32_t mean_w = (int32_t)((v->num_states + layers - 1) / layers),
                mean_a = (int32_t)((v->num_arcs + layers - 1) / layers);
  // arcs per lane (rows of a block): what most states of a lattice have, or a share of it that
  // leaves the states of many arcs enough lanes.  From 1.2 to 1.6 arcs per state (alignments have 1.4,
  // at most three) three for small layers: then hardly a state has two lanes, and the tropical walk
  // of a single warp is the short one (SliceLayers + SliceChain, us, with two and three rows; 802
  // layers of 2 to 5 states 262 and 141, 402 of 10 states 169 and 132, of 48 192 and 189, 502 of 60 258
  // and 245; the log semiring 203 and 190, 229 and 229, 304 and 294).  Two beyond two blocks of lanes:
  // the regions take longer to write and to copy (402 of 64 states 206 and 207, of 256 364 and 417;
  // log 242 and 244, 424 and 462); and in the log semiring for layers of a few states, one lane each
  // or two (802 of 2 to 5: 685 and 704).
  const double mean_deg = (double)v->num_arcs / std::max(v->num_states, 1);
  const bool three = mean_deg >= 1.2 && mean_w <= 60 && (mean_w > 4 || !log_semiring);
  p.rows = mean_deg < 1.6 && !three ? 2 : mean_deg < 3.0 ? 3 : mean_deg < 6.0 ? 4 : 8;
  // Warps: a block of 32 lanes each, for a layer between the mean and the largest (a warp that
  // runs alone issues an instruction in about five cycles, so more warps than blocks only
  // add to the barrier).
  const int32_t blocks = CeilDiv(mean_w + mean_a / p.rows, 32),
                most = CeilDiv(p.maxw + v->max_layer_arcs / p.rows, 32);
  p.warps = std::max(1, std::min(16, std::min((blocks + most + 1) / 2, 2 * blocks)));
  const size_t vals = 2 * sizeof(double) * (size_t)p.maxw;
  // with more CTAs than SMs, two of them should share one
  const size_t budget =
      (int64_t)ndir * v->num_fsas > NumSms() ? kLayerSmemBudget / 2 : kLayerSmemBudget;
  // a slot takes the largest layer with a quarter of padding, or several small ones
  const size_t largest = (size_t)v->max_layer_arcs * 22 + (size_t)p.maxw * 16 + 4096;
  for (size_t limit : {budget, kLayerSmemBudget}) {
    if (vals + 2 * largest > limit || p.maxw > kSliceMaxStates) continue;
    p.slots = (int32_t)std::max<size_t>(2, std::min<size_t>(4, (limit - vals) / (24 * 1024)));
    while (p.slots > 2 && (limit - vals) / p.slots < largest) --p.slots;
    p.slot_bytes = (int32_t)(std::min<size_t>((limit - vals) / p.slots, 48 * 1024 + largest) & ~127);
    p.bytes = vals + (size_t)p.slots * p.slot_bytes;
    p.ok = true;
    return p;
  }
  // Layers too wide for that are shared by a cluster of CTAs.
  p.wide = 1;
  p.warps = kWideWarps;
  p.team = 1;
  while (p.team < kWideTeam && (int64_t)ndir * v->num_fsas * p.team * 2 <= NumSms() &&
         p.team * 32 * p.warps < v->max_layer_states)
    p.team *= 2;
  p.bytes = sizeof(int32_t) * (size_t)((p.nl_cap + 1 + 3) & ~3) +
            2 * sizeof(LayerArc) * kWideRecs * 32 * kWideWarps;
  p.ok = p.bytes <= kLayerSmemBudget;
  if (p.ok) {  // as many states of two layers as there is room for
    p.cells = (int32_t)std::min<int64_t>(
        p.maxw, (int64_t)(kLayerSmemBudget - p.bytes) / (2 * sizeof(double)) & ~1);
    p.bytes += 2 * sizeof(double) * (size_t)p.cells;
  }
  return p;
}

// ---------------------------------------------------------------------------
// Sliced layers: what the chain reads.  A layer's states are dealt out to lanes, a state of d
// arcs to n = 1, 2, 4 ... 32 of them so that a lane has at most K = ChainPlan::rows arcs, in
// order of falling n; 32 consecutive lanes are a block.  The r-th arc of a state goes to its
// lane r mod n, row r / n.  The K rows of a block hold a LayerArc per lane (weight 0 / NaN
// where there is no arc), so that the chain reads them without bank conflicts, without a
// search and without a test per arc.  A state of more than 32 K arcs has a block of its own
// with as many rows as it takes ("tall"), behind all others.
//   layer region: a word per lane of all blocks: state (index in its layer) | log2 n << 16 |
//     first lane of the state << 19; a word per tall block: first row | rows << 20; the rows
// Regions are handed out by an atomic counter; where a layer lies does not change results.
// ---------------------------------------------------------------------------
constexpr uint32_t kNoState = 0xffffu, kLaneHead = 1u << 19;
struct SliceDesc {
  uint32_t at;     // of the region, in units of 16 bytes
  int32_t size;    // likewise
  int32_t blocks;  // of K rows; -1: the pool was full, the arcs are read where they are
  int32_t tall;    // kSingle: none, and one block with a lane per state
};
constexpr int32_t kSingle = -1;
// Of a region in units of 16 bytes: where the rows start.
__device__ __forceinline__ constexpr int32_t SliceRowsAt(int32_t blocks, int32_t tall) {
  return (blocks + tall) * 8 + (tall + 3) / 4;
}

// Units of 16 bytes the pool needs: records for uneven lanes, two part-filled blocks per
// layer, lane words.  (A layer that finds the pool full is read the slow way; 2^32 - 1 units, what
// a SliceDesc can name, hold both directions of a lattice of 10^9 arcs.)
static int64_t SlicePoolUnits(const k2b200_fsa_view *v, const ChainPlan &p, int32_t ndir) {
  const int64_t layers = (int64_t)v->num_fsas * v->max_layers, arcs = v->num_arcs, k = p.rows;
  const int64_t units = arcs + arcs / 2 + (int64_t)v->num_states * (p.rows < 8 ? k - 1 : k / 2) +
                        layers * (40 * k + 16) + 1024;
  return std::min<int64_t>(units * ndir, UINT32_MAX);
}

// Layer `lv` of direction blockIdx.y + dir_base per team of kWarps warps (kWarps == 1: four
// layers per CTA).  A region of at most buf_units is put together in shared memory (scattered
// 16-byte stores to global memory took twice as long).  Bound by the latency of its phases at
// the few CTAs that the buffers leave room for; eight warps instead of four to a layer of 1 100
// arcs: 340 -> 294 us for 10 M arcs both ways (573 MB moved; sixteen warps: 440, barriers).
template <bool kLog, int kWarps>
__global__ void __launch_bounds__(kWarps == 1 ? 128 : 32 * kWarps)
SliceLayers(k2b200_fsa_view v, int32_t dir_base, int32_t K, int32_t maxw, int32_t maxa,
            int32_t buf_units, int32_t nl_total, int64_t pool_units,
            unsigned long long *__restrict__ pool_used, uint4 *__restrict__ pool,
            SliceDesc *__restrict__ descs, int32_t *__restrict__ status) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int nt = 32 * kWarps;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tid = kWarps == 1 ? lane : threadIdx.x;
  const int dir = blockIdx.y + dir_base;
  const int32_t lv = kWarps == 1 ? blockIdx.x * 4 + warp : blockIdx.x;
  if (lv >= v.level_offsets[v.num_fsas]) return;
  auto sync = [&]() { if (kWarps == 1) __syncwarp(); else __syncthreads(); };
  SliceDesc *desc = descs + (int64_t)dir * nl_total + lv;
  const int32_t b = v.level_splits[lv], w = v.level_splits[lv + 1] - b;
  if (w <= 0 || w > maxw) {
    if (tid == 0) {
      SliceDesc d = {0, 0, w <= 0 ? 0 : -1, 0};
      *desc = d;
      if (w > maxw) atomicOr(status, 1);  // the caller's bounds do not hold
    }
    return;
  }
  const Arc *arcs = reinterpret_cast<const Arc *>(v.arcs);
  const int32_t fsa = v.row_ids1[b], s_begin = v.row_splits1[fsa];
  // the arcs: those that leave the layer before (forward) or this layer (backward), and the
  // first state of the layer at their other end
  int32_t a0, a1, ob;
  if (dir == 0) {
    ob = lv > v.level_offsets[fsa] ? v.level_splits[lv - 1] : b;
    a0 = v.row_splits2[ob];
    a1 = ob < b ? v.row_splits2[b] : a0;
  } else {
    ob = b + w;
    a0 = v.row_splits2[b];
    a1 = v.row_splits2[b + w];
  }
  if (a1 - a0 > maxa) {
    if (tid == 0) {
      SliceDesc d = {0, 0, -1, 0};
      *desc = d;
      atomicOr(status, 1);
    }
    return;
  }
  // per team: the region, counters of every warp per state, lanes of every state
  unsigned char *team = smem_raw + (kWarps == 1 ? warp : 0) *
                                       ((size_t)buf_units * 16 + 4 * (2 * (size_t)maxw + 32));
  uint4 *buf = reinterpret_cast<uint4 *>(team);
  int32_t *cnt = reinterpret_cast<int32_t *>(buf + buf_units);  // [kWarps][maxw]
  int32_t *place = cnt + kWarps * maxw;                         // [maxw] first lane | log2 n << 24
  int32_t *head = place + maxw;                                 // [32] buckets and the like
  for (int32_t k = tid; k < w; k += nt)
#pragma unroll
    for (int u = 0; u < kWarps; ++u) cnt[u * maxw + k] = 0;
  if (tid < 32) head[tid] = 0;
  sync();
  const int32_t per = ((a1 - a0 + nt - 1) / nt) * 32;
  const int32_t c0 = kWarps == 1 ? a0 : min(a0 + warp * per, a1);
  const int32_t c1 = kWarps == 1 ? a1 : min(c0 + per, a1);
  int32_t *mine = cnt + (kWarps == 1 ? 0 : warp) * maxw;
  if (dir == 0) {
#pragma unroll 4
    for (int32_t a = c0 + lane; a < c1; a += 32) {
      const int32_t d = s_begin + arcs[a].dest - b;
      if ((uint32_t)d < (uint32_t)w) atomicAdd(&mine[d], 1);
    }
    sync();
  }
  // ---- lanes of every state: buckets 0 .. 5 are n = 32 .. 1, 6 the tall states ----------
  auto degree = [&](int32_t j) {
    if (dir != 0) return v.row_splits2[b + j + 1] - v.row_splits2[b + j];
    int32_t d = 0;
#pragma unroll
    for (int u = 0; u < kWarps; ++u) d += cnt[u * maxw + j];
    return d;
  };
  auto bucket_of = [&](int32_t d) {
    if (d > 32 * K) return 6;
    int n = 0;
    while (K << n < d) ++n;
    return 5 - n;
  };
  for (int32_t j = tid; j < w; j += nt) {
    const int32_t d = degree(j), bk = bucket_of(d);
    const int32_t rows = bk == 6 ? (d + 31) >> 5 : 0;
    atomicAdd(&head[bk], bk == 6 ? 32 : 32 >> bk);
    if (bk == 6) atomicAdd(&head[16], rows);
    place[j] = d;
  }
  sync();
  int32_t lanes = 0;
  for (int u = 0; u < 6; ++u) lanes += head[u];
  const int32_t blocks = (lanes + 31) >> 5, tall = head[6] >> 5;
  const int32_t rows_at = SliceRowsAt(blocks, tall);
  const int32_t units = rows_at + (blocks * K + head[16]) * 32;
  sync();
  if (tid == 0) {
    int32_t run = 0;
    for (int u = 0; u < 6; ++u) {
      head[8 + u] = run;  // first lane of the bucket
      run += head[u];
    }
    head[14] = blocks * 32;  // ... of the tall states
    head[17] = blocks * K;   // ... and their first row
    const unsigned long long at = atomicAdd(pool_used, (unsigned long long)units);
    SliceDesc d = {(uint32_t)at, units, blocks, head[5] == w && blocks == 1 ? kSingle : tall};
    // (a tall block's word has 12 bits for its rows, 20 for the first of them)
    if (at + units > (unsigned long long)pool_units || head[16] >= 4096 ||
        blocks * K + head[16] >= (1 << 20)) {
      d = SliceDesc{0, 0, -1, 0};
    }
    *desc = d;
    head[20] = d.blocks;
    head[21] = (int32_t)d.at;
  }
  sync();
  if (head[20] < 0) return;
  uint4 *const final_region = pool + (uint32_t)head[21];
  const bool staged = units <= buf_units;
  uint4 *region = staged ? buf : final_region;
  uint32_t *words = reinterpret_cast<uint32_t *>(region);
  LayerArc *recs = reinterpret_cast<LayerArc *>(region + rows_at);
  for (int32_t k = lanes + tid; k < blocks * 32; k += nt) words[k] = kNoState;
  {
    LayerArc none;
    none.w = kLog ? 0.0 : nan("");  // (never the larger one)
    none.other = 0;
    none.arc = -1;
    for (int32_t k = tid; k < units - rows_at; k += nt) recs[k] = none;
  }
  // every state's lanes, every warp's first arc of it
  for (int32_t j = tid; j < w; j += nt) {
    const int32_t d = place[j], bk = bucket_of(d);
    const int32_t nl = bk == 6 ? 5 : 5 - bk;
    const int32_t at = atomicAdd(&head[8 + bk], 1 << nl);
    // the row of its first arc times 32, plus its first lane of the block
    int32_t first = (at >> 5) * K * 32 + (at & 31);
    if (bk == 6) {
      const int32_t rows = (d + 31) >> 5, row = atomicAdd(&head[17], rows);
      words[(blocks + tall) * 32 + ((at >> 5) - blocks)] = (uint32_t)row | (uint32_t)rows << 20;
      first = row * 32;
    }
    place[j] = first | nl << 27;
    for (int32_t u = 0; u < 1 << nl; ++u)
      words[at + u] = (uint32_t)j | (uint32_t)nl << 16 | (u == 0 ? kLaneHead : 0u);
    if (dir == 0) {
      int32_t r = 0;
#pragma unroll
      for (int u = 0; u < kWarps; ++u) {
        const int32_t n = cnt[u * maxw + j];
        cnt[u * maxw + j] = r;
        r += n;
      }
    }
  }
  sync();  // (also: the records' padding is written before any arc)
  auto put = [&](const Arc &arc, int32_t a, int32_t j, int32_t rank, int32_t other) {
    const int32_t at = place[j] & 0x7ffffff, nl = (int32_t)((uint32_t)place[j] >> 27);
    LayerArc r;
    r.w = kLog ? exp((double)arc.score) : (double)arc.score;
    r.other = other;
    r.arc = a;
    recs[at + (rank & ((1 << nl) - 1)) + (rank >> nl) * 32] = r;
    if (kLog && arc.score != -INFINITY && !(fabsf(arc.score) <= kMaxScore)) atomicOr(status, 4);
  };
  if (dir != 0) {
#pragma unroll 2
    for (int32_t a = c0 + lane; a < c1; a += 32) {
      const Arc arc = arcs[a];
      const int32_t j = s_begin + arc.src - b;
      put(arc, a, j, a - v.row_splits2[b + j], s_begin + arc.dest - ob);
    }
  } else {
    // two batches of 32 arcs at a time, so that their loads are in flight together
    for (int32_t a = c0; a < c1; a += 64) {
      Arc arc[2];
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (a + 32 * u + lane < c1) arc[u] = arcs[a + 32 * u + lane];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (a + 32 * u >= c1) break;  // uniform
        int32_t j = -1 - lane;  // lanes without an arc match nobody
        if (a + 32 * u + lane < c1) {
          const int32_t x = s_begin + arc[u].dest - b;
          if ((uint32_t)x < (uint32_t)w) j = x;
        }
        const unsigned same = __match_any_sync(kAll, j);
        int32_t rank = 0;
        if (j >= 0) rank = mine[j] + __popc(same & ((1u << lane) - 1u));
        __syncwarp();
        if (j >= 0 && lane == 31 - __clz(same)) mine[j] = rank + 1;
        __syncwarp();
        if (j >= 0) put(arc[u], a + 32 * u + lane, j, rank, s_begin + arc[u].src - ob);
      }
    }
  }
  if (staged) {
    sync();
    for (int32_t k = tid; k < units; k += nt) final_region[k] = buf[k];
  }
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
#pragma unroll 1
    for (; k < k1; k += 4 * step) {
      LayerArc r[4];
      Val x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k + u * step < k1) r[u] = rec(k + u * step);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k + u * step < k1) x[u] = val(r[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k + u * step < k1) Add(r[u], x[u]);
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
// exponent of the largest value since.  hi_slots: two words that the warps of a CTA share.
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
      Rescale(*reinterpret_cast<volatile int32_t *>(&hi_slots[at ^ 1]));
    }
    if (step % kRescale == 1 && first_thread)
      *reinterpret_cast<volatile int32_t *>(&hi_slots[at ^ 1]) = 0;
  }
  __device__ __forceinline__ void Rescale(int32_t hm) {
    const int32_t e = hm > 0 ? (hm >> 20) - 1023 : 0;
    K += e;
    mul = __longlong_as_double((long long)(1023 - e) << 52);
  }
  // the largest of a warp's values since the last change, and 0 again
  __device__ __forceinline__ int32_t TakeMax(int lane, int32_t *status) {
    const int32_t hm = __reduce_max_sync(0xffffffffu, hi_max);
    if (hm >= (1023 + kRangeExp) << 20 && lane == 0) atomicOr(status, 4);
    hi_max = 0;
    return hm;
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
    const int32_t hm = TakeMax(lane, status);
    if (lane == 0 && hm > 0) atomicMax(&hi_slots[(step / kRescale) & 1], hm);
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

// The sum of state s (layer l of FSA i) when the layer was not sliced: all arcs of the layer
// are looked through.
template <typename Val, bool kLog>
__device__ __noinline__ StateSum<Val, kLog> SumUnsliced(const k2b200_fsa_view &v, int32_t i,
                                                        int32_t dir, int32_t l, int32_t s,
                                                        const Val *prev) {
  const int32_t lv = v.level_offsets[i] + l, s_begin = v.row_splits1[i];
  const int32_t b = v.level_splits[lv], e = v.level_splits[lv + 1];
  const Arc *arcs = reinterpret_cast<const Arc *>(v.arcs);
  const int32_t ob = dir != 0 ? e : l > 0 ? v.level_splits[lv - 1] : b;
  StateSum<Val, kLog> q;
  q.Clear();
  const int32_t a0 = v.row_splits2[dir == 0 ? ob : s],
                a1 = dir == 0 ? (ob < b ? v.row_splits2[b] : a0) : v.row_splits2[s + 1];
  for (int32_t a = a0; a < a1; ++a) {
    const Arc arc = arcs[a];
    if (dir == 0 && s_begin + arc.dest != s) continue;
    LayerArc r;
    r.w = kLog ? exp((double)arc.score) : (double)arc.score;
    r.other = s_begin + (dir == 0 ? arc.src : arc.dest) - ob;
    r.arc = a;
    q.Add(r, prev[r.other]);
  }
  return q;
}

// The walk over sliced layers.  grid = (directions, fsas).  val_fwd / val_bwd: values per
// state (log: doubles relative to 2^scale[(dir * num_fsas + i) * nl_cap + layer]).  The last
// warp feeds the ring: its lanes look at the next 32 layers, those that fit a slot go there
// with a bulk copy each.  A warp sums the blocks b = warp, warp + warps, ... of a layer.
struct __align__(16) SliceEntry {  // of a layer in a slot
  int32_t at;  // of the region in shared memory, in units of 16 bytes; -1: read from L2
  int32_t blocks, tall, first_state;
};

// kOne: one such warp, which has the short walk below (in the loop of several it cost 7 %).
template <typename Val, bool kLog, int K, bool kOne>
__global__ void __launch_bounds__(kOne ? 64 : 544, 1)
SliceChain(k2b200_fsa_view v, const uint4 *__restrict__ pool, const SliceDesc *__restrict__ descs,
           Val *__restrict__ val_fwd, Val *__restrict__ val_bwd, int32_t *__restrict__ entering,
           int32_t *__restrict__ scale, int32_t dir_base, int32_t fsa_base, int32_t nl_total,
           ChainPlan p, int32_t *__restrict__ status) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full[kMaxSlots], empty[kMaxSlots];
  __shared__ SliceEntry entries[kMaxSlots][32];
  __shared__ int32_t slot_layers[kMaxSlots], hi_shared[2];
  constexpr unsigned kAll = 0xffffffffu;
  const int32_t i = fsa_base + blockIdx.y, dir = blockIdx.x + dir_base;
  const int32_t s_begin = v.row_splits1[i], s_end = v.row_splits1[i + 1];
  if (s_end == s_begin) return;
  const int32_t lv0 = v.level_offsets[i], nl = v.level_offsets[i + 1] - lv0;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nw = kOne ? 1 : p.warps;
  Val *out = dir == 0 ? val_fwd : val_bwd;
  const uint32_t *shared_words = reinterpret_cast<const uint32_t *>(smem_raw);
  const LayerArc *shared_recs = reinterpret_cast<const LayerArc *>(smem_raw);
  Val *vals = reinterpret_cast<Val *>(smem_raw + (size_t)p.slots * p.slot_bytes);  // [2][maxw]
  if (tid == 0) {
    hi_shared[0] = hi_shared[1] = 0;
    for (int32_t s = 0; s < p.slots; ++s) {
      MbarInit(&full[s], 1);
      MbarInit(&empty[s], nw);  // one arrival per warp
    }
    MbarInitFence();
  }
  // (padding multiplies a value by zero: it has to be one)
  for (int32_t k = tid; k < 2 * p.maxw; k += blockDim.x) vals[k] = (Val)0;
  __syncthreads();
  if (nl > p.nl_cap) {  // the caller's bounds do not hold: the exact kernel takes the call
    if (tid == 0) atomicOr(status, 1);
    return;
  }
  if (warp == nw) {
    int32_t slot = 0, issued = 0;
    unsigned parity = 1;  // a fresh barrier counts as "previous phase complete"
    const int32_t cap = p.slot_bytes >> 4;
    for (int32_t done = 0; done < nl;) {
      const int32_t step = done + lane, l = dir == 0 ? step : nl - 1 - step;
      SliceDesc d = {0, 0, 0, 0};
      int32_t first = 0;
      if (step < nl) {
        d = descs[(int64_t)dir * nl_total + lv0 + l];
        first = v.level_splits[lv0 + l];
      }
      const int32_t size = d.size <= cap && d.blocks >= 0 ? d.size : 0;
      int32_t inc = size;
#pragma unroll
      for (int k = 1; k < 32; k <<= 1) {
        const int32_t o = __shfl_up_sync(kAll, inc, k);
        if (lane >= k) inc += o;
      }
      // (monotone, so the layers that fit are the first ones)
      const int32_t m = __popc(__ballot_sync(kAll, step < nl && inc <= cap));
      const int32_t total = __shfl_sync(kAll, inc, m - 1);
      if (!__all_sync(kAll, MbarWaitBounded(&empty[slot], parity))) {
        if (lane == 0) atomicOr(status, 2);
        break;
      }
      if (lane < m) {
        SliceEntry e = {d.size > 0 && size == 0 ? -1 : slot * cap + inc - size, d.blocks, d.tall,
                        first};
        entries[slot][lane] = e;
      }
      if (lane == 0) slot_layers[slot] = m;
      __syncwarp();
      if (lane == 0) MbarArriveExpectTx(&full[slot], (unsigned)total * 16u);
      __syncwarp();
      if (lane < m && size > 0)
        BulkCopyG2S(smem_raw + (size_t)(slot * cap + inc - size) * 16, pool + d.at,
                    (unsigned)size * 16u, &full[slot]);
      done += m;
      slot = slot + 1 == p.slots ? 0 : slot + 1;
      parity ^= (slot == 0);
      ++issued;
    }
    // no copy is in flight towards this CTA's shared memory when it retires
    for (int32_t k = max(0, issued - p.slots); k < issued; ++k)
      MbarWaitBounded(&full[k % p.slots], (unsigned)(k / p.slots) & 1u);
    return;
  }

  const int32_t root = dir == 0 ? s_begin : s_end - 1, nc = 32 * nw;
  int32_t *my_scale = kLog ? scale + ((int64_t)dir * v.num_fsas + i) * p.nl_cap : nullptr;
  auto layer_sync = [&]() {
    if (nw == 1) __syncwarp();
    else asm volatile("bar.sync 1, %0;" ::"r"(nc) : "memory");
  };
  ChainScale<kLog> sc;
  int32_t slot = p.slots - 1, k = 0, m = 0;
  unsigned parity = 1;
  int32_t prev = p.maxw, cur = 0;
  // A layer of one block with a lane per state (alignments), of the tropical semiring, in `now`; the
  // records of the layer behind it, if it is of the same kind and slot, go to `next` meanwhile.
  // What a warp that runs alone issues per layer bounds such a walk: 290 cycles, against 590 of the
  // general loop below.
  // (Its region then lies right behind: it is read before it is known whether it is of that kind.)
  // The first layer with states has the one that scores 0 without an arc: it takes the general loop.
  constexpr int32_t kSingleUnits = SliceRowsAt(1, 0) + K * 32;
  struct Single {
    uint32_t word;
    int32_t first_state;
    LayerArc x[K];
  };
  const int32_t last_single = p.slots * (p.slot_bytes >> 4) - kSingleUnits;
  auto read_single = [&](int32_t at, Single &l) {
    l.word = shared_words[at * 4 + lane];
    const LayerArc *r = shared_recs + at + SliceRowsAt(1, 0) + lane;
#pragma unroll
    for (int u = 0; u < K; ++u) l.x[u] = r[u * 32];
  };
  auto single = [&](const Single &now, Single &next, int32_t &at) {
    Val y[K];
#pragma unroll
    for (int u = 0; u < K; ++u) y[u] = vals[prev + now.x[u].other];
    bool more = false;
    at += kSingleUnits;
    if (k < m && at <= last_single) {
      read_single(at, next);
      const SliceEntry e = entries[slot][k];
      next.first_state = e.first_state;
      more = e.tall == kSingle && e.at == at;
    }
    StateSum<Val, kLog> q;
    q.Clear();
#pragma unroll
    for (int u = 0; u < K; ++u) q.Add(now.x[u], y[u]);
    if (now.word & kLaneHead) {
      const int32_t j = (int32_t)(now.word & kNoState), s = now.first_state + j;
      vals[cur + j] = q.acc;
      out[s] = q.acc;
      if (entering != nullptr && dir == 0) entering[s] = q.best;
    }
    const int32_t t = prev;
    prev = cur;
    cur = t;
    __syncwarp();
    return more;
  };
  bool begun = false;
  for (int32_t step = 0; step < nl; ++step) {
    if (k == m) {  // the next slot
      slot = slot + 1 == p.slots ? 0 : slot + 1;
      parity ^= (slot == 0);
      if (!__all_sync(kAll, MbarWaitBounded(&full[slot], parity))) {  // the whole warp, or none
        // nothing that the slot holds is looked at; the other warps still need the barriers
        atomicOr(status, 2);
        for (; step < nl; ++step) layer_sync();
        break;
      }
      k = 0;
      m = slot_layers[slot];
    }
    SliceEntry e = entries[slot][k++];
    if (e.tall == kSingle) {
      e.tall = 0;
      if (kOne && !kLog && e.at >= 0 && begun) {
        Single a, b;
        int32_t at = e.at;
        read_single(at, a);
        a.first_state = e.first_state;
        while (single(a, b, at)) {
          ++step;
          ++k;
          if (!single(b, a, at)) break;
          ++step;
          ++k;
        }
        if (k == m && lane == 0)  // this warp has read the slot
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(SmemAddr(&empty[slot]))
                       : "memory");
        continue;
      }
    }
    begun |= e.blocks != 0;
    sc.BeginLayer(step, hi_shared, tid == 0);
    auto finish = [&](int32_t j, StateSum<Val, kLog> &q) {
      const int32_t s = e.first_state + j;
      if (kLog) {
        q.acc = q.acc * (Val)sc.mul;
        if (q.acc == (Val)0 && s == root) q.acc = (Val)1;
        sc.Note((double)q.acc);
      } else {
        if (s == root && q.acc == (Val)-INFINITY) q.acc = (Val)0;
        if (entering != nullptr && dir == 0) entering[s] = q.best;
      }
      vals[cur + j] = q.acc;
      out[s] = q.acc;
    };
    // the lanes of a state bring their sums together
    auto across = [&](uint32_t word, StateSum<Val, kLog> &q) {
      const int32_t nlog = (int32_t)(word >> 16) & 7;
      const int32_t most = __reduce_max_sync(kAll, nlog);
      for (int32_t d = 0; d < most; ++d) {  // uniform
        StateSum<Val, kLog> o;
        o.acc = __shfl_xor_sync(kAll, q.acc, 1 << d);
        o.best = kLog ? 0 : __shfl_xor_sync(kAll, q.best, 1 << d);
        if (d < nlog) q.Merge(o);
      }
    };
    if (e.at >= 0) {
      const int32_t rows_at = e.at + SliceRowsAt(e.blocks, e.tall);
      for (int32_t blk = warp; blk < e.blocks; blk += nw) {
        const uint32_t word = shared_words[e.at * 4 + blk * 32 + lane];
        const LayerArc *r = shared_recs + rows_at + blk * (K * 32) + lane;
        LayerArc x[K];
        Val y[K];
#pragma unroll
        for (int u = 0; u < K; ++u) x[u] = r[u * 32];
#pragma unroll
        for (int u = 0; u < K; ++u) y[u] = vals[prev + x[u].other];
        StateSum<Val, kLog> q;
        q.Clear();
#pragma unroll
        for (int u = 0; u < K; ++u) q.Add(x[u], y[u]);
        if (__any_sync(kAll, word & (7u << 16))) across(word, q);
        if (word & kLaneHead) finish((int32_t)(word & kNoState), q);
      }
      for (int32_t t = warp; t < e.tall; t += nw) {
        const int32_t blk = e.blocks + t;
        const uint32_t word = shared_words[e.at * 4 + blk * 32 + lane],
                       tw = shared_words[(e.at + (e.blocks + e.tall) * 8) * 4 + t];
        const LayerArc *r = shared_recs + rows_at + (int32_t)(tw & 0xfffffu) * 32 + lane;
        StateSum<Val, kLog> q;
        q.Clear();
#pragma unroll 4
        for (int32_t u = 0; u < (int32_t)(tw >> 20); ++u) {
          const LayerArc x = r[u * 32];
          q.Add(x, vals[prev + x.other]);
        }
        across(word, q);
        if (word & kLaneHead) finish((int32_t)(word & kNoState), q);
      }
    } else if (e.blocks >= 0) {  // too large for a slot: from L2
      const int32_t l = dir == 0 ? step : nl - 1 - step;
      const uint4 *region = pool + descs[(int64_t)dir * nl_total + lv0 + l].at;
      const int32_t rows_at = SliceRowsAt(e.blocks, e.tall);
      for (int32_t blk = warp; blk < e.blocks + e.tall; blk += nw) {
        const uint32_t word = reinterpret_cast<const uint32_t *>(region)[blk * 32 + lane];
        int32_t row = blk * K, rows = K;
        if (blk >= e.blocks) {
          const uint32_t tw = reinterpret_cast<const uint32_t *>(
              region)[(e.blocks + e.tall) * 32 + blk - e.blocks];
          row = (int32_t)(tw & 0xfffffu);
          rows = (int32_t)(tw >> 20);
        }
        const LayerArc *r = reinterpret_cast<const LayerArc *>(region + rows_at) + row * 32 + lane;
        StateSum<Val, kLog> q;
        q.Clear();
#pragma unroll 4
        for (int32_t u = 0; u < rows; ++u) {
          const LayerArc x = r[u * 32];
          q.Add(x, vals[prev + x.other]);
        }
        across(word, q);
        if (word & kLaneHead) finish((int32_t)(word & kNoState), q);
      }
    } else {
      const int32_t l = dir == 0 ? step : nl - 1 - step;
      const int32_t w = v.level_splits[lv0 + l + 1] - e.first_state;
      for (int32_t j = tid; j < w && j < p.maxw; j += nc) {
        StateSum<Val, kLog> q =
            SumUnsliced<Val, kLog>(v, i, dir, l, e.first_state + j, vals + prev);
        finish(j, q);
      }
    }
    sc.EndLayer(step, hi_shared, lane, status);
    if (kLog && tid == 0) my_scale[dir == 0 ? step : nl - 1 - step] = sc.K;
    if (k == m) {  // this warp has read the slot
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(SmemAddr(&empty[slot]))
                     : "memory");
    }
    const int32_t t = prev;
    prev = cur;
    cur = t;
    layer_sync();
  }
  sc.End(lane, status);
}

// The same recursion for whatever left the range of SliceChain, or lost a copy: returns at
// once unless *status is set.  Log values are (mantissa, exponent) pairs and the factors come
// from the arcs' scores, so there is no range; everything is read from L2.
template <typename Real, bool kLog>
struct ExactSum {
  double m = 0.0;
  int32_t e = kZeroExp, best = -1;
  Real top = -INFINITY;
  __device__ __forceinline__ void Merge(const ExactSum &o) {
    if (kLog) {
      const int32_t En = max(e, o.e);
      m = ScaleDown(m, e - En) + ScaleDown(o.m, o.e - En);
      e = En;
    } else if (o.top > top || (o.top == top && o.best > best)) {
      top = o.top;
      best = o.best;
    }
  }
  __device__ __forceinline__ void Across(int lanes_below) {  // over the lanes `lanes_below` off
    ExactSum o;
    o.m = __shfl_xor_sync(0xffffffffu, m, lanes_below);
    o.e = __shfl_xor_sync(0xffffffffu, e, lanes_below);
    o.best = __shfl_xor_sync(0xffffffffu, best, lanes_below);
    o.top = __shfl_xor_sync(0xffffffffu, top, lanes_below);
    Merge(o);
  }
};

template <typename Real, bool kLog>
__global__ void __launch_bounds__(256)
ExactChain(k2b200_fsa_view v, const uint4 *__restrict__ pool, const SliceDesc *__restrict__ descs,
           double *mant, int32_t *expo, Real *fwd, Real *bwd, int32_t *__restrict__ entering,
           int32_t dir_base, int32_t fsa_base, int32_t nl_total, int32_t K,
           const int32_t *__restrict__ status) {
  if (*status == 0) return;
  const int32_t i = fsa_base + blockIdx.y, dir = blockIdx.x + dir_base;
  const int32_t s_begin = v.row_splits1[i], s_end = v.row_splits1[i + 1];
  const int32_t lv0 = v.level_offsets[i], nl = v.level_offsets[i + 1] - lv0;
  const Arc *arcs = reinterpret_cast<const Arc *>(v.arcs);
  Real *out = dir == 0 ? fwd : bwd;
  double *m = mant + (int64_t)dir * v.num_states;
  int32_t *x = expo + (int64_t)dir * v.num_states;
  const int32_t root = dir == 0 ? s_begin : s_end - 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int32_t step = 0; step < nl; ++step) {
    const int32_t l = dir == 0 ? step : nl - 1 - step;
    const int32_t b = v.level_splits[lv0 + l], e = v.level_splits[lv0 + l + 1];
    auto add = [&](ExactSum<Real, kLog> &q, int32_t a) {
      const Arc arc = arcs[a];
      const int32_t other = s_begin + (dir == 0 ? arc.src : arc.dest);
      ExactSum<Real, kLog> o;
      if (kLog) {
        int32_t k;
        ExpToMantExp(arc.score, &o.m, &k);
        o.m *= m[other];
        o.e = o.m != 0.0 ? x[other] + k : kZeroExp;
      } else {
        o.top = out[other] + (Real)arc.score;
        o.best = a;
      }
      q.Merge(o);
    };
    auto finish = [&](int32_t s, const ExactSum<Real, kLog> &q) {
      if (kLog) {
        int32_t E = q.e;
        double mm = Renorm(q.m, &E);
        if (mm == 0.0 && s == root) {
          mm = 1.0;
          E = 0;
        }
        m[s] = mm;
        x[s] = E;
        out[s] = mm == 0.0 ? (Real)-INFINITY
                           : (Real)(log(mm) + (double)E * 0.69314718055994530942);
      } else {
        out[s] = q.top == (Real)-INFINITY && s == root ? (Real)0 : q.top;
        if (dir == 0 && entering != nullptr) entering[s] = q.best;
      }
    };
    SliceDesc d = descs[(int64_t)dir * nl_total + lv0 + l];
    if (d.tall == kSingle) d.tall = 0;
    if (d.blocks >= 0 && (*status & 1) == 0) {
      const uint4 *region = pool + d.at;
      const uint32_t *words = reinterpret_cast<const uint32_t *>(region);
      for (int32_t blk = warp; blk < d.blocks + d.tall; blk += nw) {
        const uint32_t word = words[blk * 32 + lane];
        int32_t row = blk * K, rows = K;
        if (blk >= d.blocks) {
          const uint32_t tw = words[(d.blocks + d.tall) * 32 + blk - d.blocks];
          row = (int32_t)(tw & 0xfffffu);
          rows = (int32_t)(tw >> 20);
        }
        const LayerArc *r =
            reinterpret_cast<const LayerArc *>(region + SliceRowsAt(d.blocks, d.tall)) + row * 32 +
            lane;
        ExactSum<Real, kLog> q;
        for (int32_t u = 0; u < rows; ++u)
          if (r[u * 32].arc >= 0) add(q, r[u * 32].arc);
        const int32_t nlog = (int32_t)(word >> 16) & 7;
        for (int32_t u = 0; u < 5; ++u) {
          ExactSum<Real, kLog> o = q;
          o.Across(1 << u);
          if (u < nlog) q = o;
        }
        if (word & kLaneHead) finish(b + (int32_t)(word & kNoState), q);
      }
    } else {  // a warp per state looks through the layer's arcs
      const int32_t ob = l > 0 ? v.level_splits[lv0 + l - 1] : b;
      const int32_t f0 = v.row_splits2[ob], f1 = ob < b ? v.row_splits2[b] : f0;
      for (int32_t s = b + warp; s < e; s += nw) {
        const int32_t a0 = dir == 0 ? f0 : v.row_splits2[s],
                      a1 = dir == 0 ? f1 : v.row_splits2[s + 1];
        ExactSum<Real, kLog> q;
        for (int32_t a = a0 + lane; a < a1; a += 32)
          if (dir != 0 || s_begin + arcs[a].dest == s) add(q, a);
        for (int u = 16; u > 0; u >>= 1) q.Across(u);
        if (lane == 0) finish(s, q);
      }
    }
    __syncthreads();
  }
}

// What the CTAs of a chain hand one another: stores into another CTA's shared memory that count
// as bytes on its barrier, so that nothing is fenced and nobody waits but the reader.  Addresses
// are those of the cluster's window.
__device__ __forceinline__ uint32_t InRank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void StoreAsync(uint32_t addr, int32_t x, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(
                   addr),
               "r"(x), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void StoreAsync(uint32_t addr, float x, uint32_t bar) {
  StoreAsync(addr, __float_as_int(x), bar);
}
__device__ __forceinline__ void StoreAsync(uint32_t addr, double x, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                   addr),
               "l"(__double_as_longlong(x)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void ClusterSync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The same for layers too wide for the ring: the CTAs of a cluster share a layer.  grid =
// (directions x team, fsas).  A state has 1, 2, 4 or 8 lanes, as many as the width of the layer
// leaves it, so that few states have more arcs than the records, up to two per lane, that are
// copied to shared memory two layers ahead (as many again are brought to L1).
//
// Every CTA has the values of the last two layers in its shared memory: a lane that has a value
// stores it into all of them, and every warp a word beside it (the largest value it has seen),
// each layer.  A layer is complete where all its bytes have come, and then everybody is past
// the layer before, whose place the next one takes.  All else (global stores, records, splits)
// is between a warp's stores and its wait.  Layers of more than `p.cells` states go through L2, with
// a barrier of the cluster.
//
// Bound by what arrives: about 1.5 cycles per value and CTA, and a microsecond per layer besides.
// 153 layers of 1 200 states, forward: 341 -> 235 us with the layer before in L2 and a barrier of the
// cluster per layer (its release alone was 700 cycles); 58 layers of 3 000: 220 -> 190.  Slower:
// the values where they were made and read from there (281; the barrier again), a bulk copy per
// CTA pair (300), two states per store (263), teams of four (269; 261 for the 3 000), four
// records per lane (252).
template <typename Val, bool kLog>
__global__ void __launch_bounds__(32 * kWideWarps, 1)
LayerChainWide(k2b200_fsa_view v, const LayerArc *__restrict__ fwd_arcs,
               const LayerArc *__restrict__ bwd_arcs, Val *val_fwd, Val *val_bwd,
               int32_t *__restrict__ entering, int32_t *__restrict__ scale, int32_t dir_base,
               int32_t fsa_base, ChainPlan p, int32_t wait_limit, int32_t *__restrict__ status) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[2];
  __shared__ int32_t words[2][kWideTeam * kWideWarps];
  constexpr unsigned kAll = 0xffffffffu;
  namespace cg = cooperative_groups;
  const int32_t rank = (int32_t)cg::this_cluster().block_rank(), team = p.team;
  const int32_t i = fsa_base + blockIdx.y, dir = (int32_t)blockIdx.x / team + dir_base;
  const int32_t s_begin = v.row_splits1[i], s_end = v.row_splits1[i + 1];
  const int32_t lv0 = v.level_offsets[i], nl = v.level_offsets[i + 1] - lv0;
  if (s_end == s_begin) return;  // uniform over the cluster, as is the next return
  const int tid = threadIdx.x, lane = tid & 31;
  Val *out = dir == 0 ? val_fwd : val_bwd;
  Val *vals = reinterpret_cast<Val *>(smem_raw);  // [2][p.cells]
  constexpr int kRecs = kWideRecs, nc = 32 * kWideWarps;
  LayerArc *recs = reinterpret_cast<LayerArc *>(smem_raw + 2 * sizeof(double) * (size_t)p.cells) +
                   tid;  // [2][kRecs][threads]
  int32_t *lvl = reinterpret_cast<int32_t *>(recs - tid + 2 * kRecs * nc);
  const int32_t *gsplits = dir == 0 ? v.in_splits : v.row_splits2;
  const LayerArc *garcs = dir == 0 ? fwd_arcs : bwd_arcs;
  if (nl > p.nl_cap) {
    if (tid == 0) atomicOr(status, 1);
    return;
  }
  for (int32_t k = tid; k <= nl; k += blockDim.x) lvl[k] = v.level_splits[lv0 + k];
  if (tid == 0) {
    MbarInit(&bars[0], 1);
    MbarInit(&bars[1], 1);
    MbarInitFence();
  }
  __syncthreads();
  ClusterSync();
  const int32_t root = dir == 0 ? s_begin : s_end - 1;
  const int32_t nt = team * nc, at = rank * nc + tid;
  int32_t *my_scale = kLog ? scale + ((int64_t)dir * v.num_fsas + i) * p.nl_cap : nullptr;
  ChainScale<kLog> sc;
  auto layer_of = [&](int32_t step) { return dir == 0 ? step : nl - 1 - step; };
  struct Splits {
    int32_t k0, k1, log_lanes;  // of the lane's state; log2 of the lanes of a state
  };
  // lanes per state in a layer of `width` states
  auto log_lanes_of = [&](int32_t width) {
    return (width << 1 <= nt) + (width << 2 <= nt) + (width << 3 <= nt);
  };
  auto splits_of = [&](int32_t step) {
    Splits f = {0, 0, 0};
    if (step >= nl) return f;
    const int32_t l = layer_of(step), b = lvl[l], e = lvl[l + 1];
    f.log_lanes = log_lanes_of(e - b);
    const int32_t s = b + (at >> f.log_lanes);
    if (s < e) {
      f.k0 = __ldg(gsplits + s);
      f.k1 = __ldg(gsplits + s + 1);
    }
    return f;
  };
  auto fetch_records = [&](int32_t step, const Splits &f) {
    const int32_t lanes = 1 << f.log_lanes, k = f.k0 + (lane & (lanes - 1));
    LayerArc *to = recs + (step & 1) * (kRecs * nc);
#pragma unroll
    for (int u = 0; u < kRecs; ++u)
      if (k + u * lanes < f.k1) CpAsync16(to + u * nc, garcs + k + u * lanes);
    CpAsyncCommit();
    if (k + kRecs * lanes < f.k1) {
#pragma unroll 1
      for (int32_t t = k + kRecs * lanes; t < min(f.k1, k + 2 * kRecs * lanes); t += lanes) {
        int32_t unused;
        asm volatile("ld.global.ca.s32 %0, [%1];" : "=r"(unused) : "l"(&garcs[t].arc));
      }
    }
  };
  auto rec = [&](int32_t k) { return garcs[k]; };
  // The layer before: its values in shared memory (or not), its first state, its last one's number.
  const uint32_t vals0 = SmemAddr(vals), bars0 = SmemAddr(bars);
  uint32_t was_vals = vals0;
  int32_t was_b = 0, was_last = 0;
  bool was_far = false;
  auto find = [&](int32_t other) {  // where the value is: an address, or the state itself
    return was_far ? other
                   : (int32_t)(was_vals + min((uint32_t)(other - was_b), (uint32_t)was_last) *
                                              (uint32_t)sizeof(Val));
  };
  auto found = [&](int32_t where) {
    if (was_far) return __ldcg(out + where);
    return *reinterpret_cast<const Val *>(__cvta_shared_to_generic((uint32_t)where));
  };
  auto val = [&](const LayerArc &r) { return found(find(r.other)); };
  Splits now = splits_of(0), next = splits_of(1), after = splits_of(2);
  LayerArc r[kRecs];
  // the records of the lane's state, `other` replaced by where the value is
  auto take_records = [&](int32_t step) {
    const int32_t lanes = 1 << now.log_lanes, k = now.k0 + (lane & (lanes - 1));
    const LayerArc *from = recs + (step & 1) * (kRecs * nc);
    CpAsyncWait<0>();
#pragma unroll
    for (int u = 0; u < kRecs; ++u)
      if (k + u * lanes < now.k1) {
        r[u] = from[u * nc];
        r[u].other = find(r[u].other);
      }
  };
  fetch_records(0, now);
  take_records(0);
  fetch_records(1, next);
  int32_t b, e;  // the layer's states
  auto begin = [&](int32_t step) {
    const int32_t l = layer_of(step);
    b = lvl[l];
    e = lvl[l + 1];
    if (tid == 0)
      MbarArriveExpectTx(&bars[step & 1],
                         (unsigned)(team * kWideWarps * 4 +
                                    (e - b > p.cells ? 0 : (e - b) * (int)sizeof(Val))));
  };
  begin(0);
  bool ok = true;
  int32_t last_step = 0;
  for (int32_t step = 0; step < nl && ok; ++step) {
    const int32_t log_lanes = now.log_lanes, lanes = 1 << log_lanes, g = lane & (lanes - 1);
    const bool far = e - b > p.cells;
    const uint32_t to = (uint32_t)((step & 1) * p.cells) * (uint32_t)sizeof(Val),
                   to_bar = bars0 - vals0 + 8u * (step & 1);
    sc.mul = 1.0;
    if (kLog && step % kRescale == 0 && step > 0) {
      int32_t hm = 0;
      for (int32_t k = lane; k < team * kWideWarps; k += 32) hm = max(hm, words[(step - 1) & 1][k]);
      sc.Rescale(__reduce_max_sync(kAll, hm));
    }
    StateSum<Val, kLog> q;
    auto store = [&](int32_t s) {  // what global memory gets
      if (!kLog && entering != nullptr && dir == 0) entering[s] = q.best;
      __stcg(out + s, q.acc);
    };
    q.Clear();
    const int32_t last = b + (max(e - b - 1, 0) & -nt);  // (nt: a power of two)
    // warps beyond the layer's last state have nothing to add
    const int32_t end = e - ((at & ~31) >> log_lanes);
    for (int32_t s0 = b; s0 < end; s0 += nt) {  // (more than once only with a lane per state)
      const int32_t s = s0 + (at >> log_lanes);
      if (s0 > b) {
        now.k0 = now.k1 = 0;
        if (s < e) {
          now.k0 = __ldg(gsplits + s);
          now.k1 = __ldg(gsplits + s + 1);
        }
#pragma unroll
        for (int u = 0; u < kRecs; ++u)
          if (now.k0 + u < now.k1) {
            r[u] = garcs[now.k0 + u];
            r[u].other = find(r[u].other);
          }
      }
      q.Clear();
      const int32_t k0 = now.k0, k1 = now.k1;
      // states of many arcs are left to the whole warp
      const bool many = k1 - k0 > 4 * kRecs * lanes;
      if (!many) {
        Val x[kRecs];
#pragma unroll
        for (int u = 0; u < kRecs; ++u)
          if (k0 + g + u * lanes < k1) x[u] = found(r[u].other);
#pragma unroll
        for (int u = 0; u < kRecs; ++u)
          if (k0 + g + u * lanes < k1) q.Add(r[u], x[u]);
        q.Walk(k0 + g + kRecs * lanes, k1, lanes, rec, val);
      }
      const unsigned heavy = __ballot_sync(kAll, many && g == 0);
      if (heavy) q.Heavy(heavy, lane, k0, k1, rec, val);
      q.Across(lanes);
      if (s < e) {
        if (kLog) {
          q.acc = q.acc * (Val)sc.mul;
          if (q.acc == (Val)0 && s == root) q.acc = (Val)1;
          sc.Note((double)q.acc);
        } else if (q.acc == (Val)-INFINITY && s == root) {
          q.acc = (Val)0;
        }
        // the state's lanes share the CTAs out among them
        if (!far) {
          const uint32_t cell = to + (uint32_t)(s - b) * (uint32_t)sizeof(Val);
          for (int32_t r = g; r < team; r += lanes) {
            const uint32_t there = InRank(vals0, r);
            StoreAsync(there + cell, q.acc, there + to_bar);
          }
        }
        if (g == 0 && s0 < last) store(s);
      }
    }
    const int32_t s = last + (at >> log_lanes);
    if (far && s < e && g == 0) store(s);
    const int32_t word = kLog && step % kRescale == kRescale - 1 ? sc.TakeMax(lane, status) : 0;
    __syncwarp();
    if (lane < team)
      StoreAsync(InRank(SmemAddr(&words[step & 1][at >> 5]), lane), word,
                 InRank(vals0, lane) + to_bar);
    if (!far && s < e && g == 0) store(s);
    if (kLog && rank == 0 && tid == 0) my_scale[layer_of(step)] = sc.K;
    was_far = far;
    was_vals = vals0 + to;
    was_b = b;
    was_last = max(e - b, 1) - 1;
    now = next;
    next = after;
    take_records(step + 1);
    fetch_records(step + 2, next);
    after = splits_of(step + 3);
    if (step + 1 < nl) begin(step + 1);
    if (far) ClusterSync();
    ok = __all_sync(kAll,
                    MbarWaitBounded(&bars[step & 1], (unsigned)(step >> 1) & 1u, wait_limit));
    last_step = step;
  }
  if (!ok) {
    if (lane == 0) atomicOr(status, 2);
    // the others still meet at the barriers of the layers that go through L2
    for (int32_t step = last_step + 1; step < nl; ++step)
      if (lvl[layer_of(step) + 1] - lvl[layer_of(step)] > p.cells) ClusterSync();
  }
  sc.End(lane, status);
  CpAsyncWait<0>();
  // No CTA leaves while another may store into it: behind this barrier nobody does any more, and what
  // is still on its way where a wait gave up is of that layer or the next one (nobody gets further
  // without this CTA's words).  The bytes of the next one may never be complete.
  ClusterSync();
  if (!ok && tid == 0)
    for (int32_t step = last_step; step < min(last_step + 2, nl); ++step)
      for (int k = 0; k < kDrainTests; ++k)
        if (MbarTestWait(&bars[step & 1], (unsigned)(step >> 1) & 1u)) break;
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
  // cleared together: status, the slice pool's counter
  int32_t *status;
  unsigned long long *pool_used;
  uint4 *pool;        // sliced layers
  SliceDesc *descs;   // [2][layers]
  LayerArc *fwd_arcs, *bwd_arcs;  // wide layers
  int32_t *scale, *expo;
  double *vals;  // [2][num_states]
  int64_t pool_units;
  size_t clear_bytes, bytes;
};

ChainScratch CarveScratch(const k2b200_fsa_view *v, const ChainPlan &p, int32_t ndir,
                          void *scratch) {
  ChainScratch c = {};
  char *base = reinterpret_cast<char *>(scratch);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off += AlignUp(std::max<size_t>(bytes, 1));
    return base + at;
  };
  const size_t na = (size_t)std::max(v->num_arcs, 1), ns = (size_t)std::max(v->num_states, 1);
  const size_t layers = (size_t)v->num_fsas * (size_t)std::max(v->max_layers, 1);
  c.clear_bytes = sizeof(int32_t) * 4;
  c.status = reinterpret_cast<int32_t *>(take(c.clear_bytes));
  c.pool_used = reinterpret_cast<unsigned long long *>(c.status + 2);
  if (p.wide) {
    c.fwd_arcs = reinterpret_cast<LayerArc *>(take(sizeof(LayerArc) * na));
    c.bwd_arcs = reinterpret_cast<LayerArc *>(take(sizeof(LayerArc) * na));
  } else if (p.ok) {
    c.pool_units = SlicePoolUnits(v, p, ndir);
    c.pool = reinterpret_cast<uint4 *>(take(sizeof(uint4) * (size_t)c.pool_units));
    c.descs = reinterpret_cast<SliceDesc *>(take(sizeof(SliceDesc) * 2 * layers));
  }
  c.scale = reinterpret_cast<int32_t *>(take(sizeof(int32_t) * 2 * layers));
  c.expo = reinterpret_cast<int32_t *>(take(sizeof(int32_t) * 2 * ns));
  c.vals = reinterpret_cast<double *>(take(sizeof(double) * 2 * ns));
  c.bytes = off;
  return c;
}
}  // namespace

size_t LayerScratchBytes(const k2b200_fsa_view *v, int32_t ndir) {
  // (the caller does not say in which semiring it will ask)
  return std::max(CarveScratch(v, PlanChain(v, ndir, false), ndir, nullptr).bytes,
                  CarveScratch(v, PlanChain(v, ndir, true), ndir, nullptr).bytes);
}

bool LayerScoresNeedIncoming(const k2b200_fsa_view *v, int32_t ndir) {
  const ChainPlan p = PlanChain(v, ndir, true);  // (as in the other semiring)
  return !p.ok || p.wide || v->num_arcs == 0;
}

template <typename Val, bool kLog>
static int32_t LaunchChain(const k2b200_fsa_view *v, const ChainScratch &c, const ChainPlan &p,
                           Val *val_fwd, Val *val_bwd, int32_t *entering, cudaStream_t stream) {
  const int32_t ndir = (val_fwd != nullptr) + (val_bwd != nullptr), dir_base = val_fwd ? 0 : 1;
  const int32_t layers = v->num_fsas * v->max_layers;
  if (!p.wide) {
    // a warp per layer while layers are small (there are many of them)
    const bool one = p.maxw <= 512 && v->num_arcs / std::max(layers, 1) <= 256;
    // (the counters of eight warps for wider layers would leave an SM a single CTA)
    const int32_t warps = one ? 1 : p.maxw <= 1024 ? 8 : 4;
    const size_t fixed = sizeof(int32_t) * ((warps + 1) * (size_t)p.maxw + 32);
    // room for a layer well above the mean, with several CTAs per SM
    const int64_t mean = (SlicePoolUnits(v, p, 1) - 1024) / std::max(layers, 1);
    int32_t buf = (int32_t)std::min<int64_t>(2 * mean, one ? 512 : 3072);
    if (!one) buf = (int32_t)std::min<int64_t>(buf, (int64_t)(kLayerSmemBudget - fixed) / 16);
    const size_t smem = (one ? 4 : 1) * (fixed + 16 * (size_t)buf);
    auto slice = one          ? SliceLayers<kLog, 1>
                 : warps == 8 ? SliceLayers<kLog, 8>
                              : SliceLayers<kLog, 4>;
    K2B_CUDA_OK(cudaFuncSetAttribute(slice, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kLayerSmemBudget));
    { slice<<<dim3(one ? CeilDiv(layers, 4) : layers, ndir), one ? 128 : 32 * warps, smem, stream>>>(
        *v, dir_base, p.rows, p.maxw, v->max_layer_arcs, buf, layers, c.pool_units, c.pool_used,
        c.pool, c.descs, c.status); NoteLaunch(); }
    constexpr bool kOne = !kLog;
    auto chain = p.rows == 2   ? SliceChain<Val, kLog, 2, false>
                 : p.rows == 3 ? SliceChain<Val, kLog, 3, false>
                 : p.rows == 4 ? SliceChain<Val, kLog, 4, false>
                               : SliceChain<Val, kLog, 8, false>;
    if (kOne && p.warps == 1)
      chain = p.rows == 2   ? SliceChain<Val, kLog, 2, kOne>
              : p.rows == 3 ? SliceChain<Val, kLog, 3, kOne>
              : p.rows == 4 ? SliceChain<Val, kLog, 4, kOne>
                            : SliceChain<Val, kLog, 8, kOne>;
    K2B_CUDA_OK(cudaFuncSetAttribute(chain, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kLayerSmemBudget));
    for (int32_t first = 0; first < v->num_fsas; first += 65535) {
      const int32_t n = std::min(v->num_fsas - first, 65535);
      { chain<<<dim3(ndir, n), 32 * (p.warps + 1), p.bytes, stream>>>(
          *v, c.pool, c.descs, val_fwd, val_bwd, entering, c.scale, dir_base, first, layers, p,
          c.status); NoteLaunch(); }
    }
    K2B_CUDA_OK(cudaGetLastError());
    return kOk;
  }
  auto pack = kLog ? PackLayerArcs<true> : PackLayerArcs<false>;
  { pack<<<CeilDiv(v->num_arcs, 256), 256, 0, stream>>>(*v, val_fwd ? c.fwd_arcs : nullptr,
                                                        val_bwd ? c.bwd_arcs : nullptr, c.status);
    NoteLaunch(); }
  K2B_CUDA_OK(cudaFuncSetAttribute(LayerChainWide<Val, kLog>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)kLayerSmemBudget));
  for (int32_t first = 0; first < v->num_fsas; first += 65535) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ndir * p.team, std::min(v->num_fsas - first, 65535));
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
                                   val_fwd, val_bwd, entering, c.scale, dir_base, first, p,
                                   CopyWaitLimit(), c.status));
    NoteLaunch();
  }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

template <typename Real>
int32_t LaunchLayerScores(const k2b200_fsa_view *v, int32_t log_semiring, Real *fwd, Real *bwd,
                          int32_t *entering, void *scratch, size_t scratch_bytes,
                          cudaStream_t stream, bool *launched, const int32_t **redo_if) {
  *launched = false;
  *redo_if = nullptr;
  if (scratch == nullptr || v->num_arcs == 0 || v->row_ids1 == nullptr || v->row_ids2 == nullptr)
    return kOk;
  const int32_t ndir = (fwd != nullptr) + (bwd != nullptr), dir_base = fwd ? 0 : 1;
  const ChainPlan p = PlanChain(v, ndir, log_semiring != 0);
  const ChainScratch c = CarveScratch(v, p, ndir, scratch);
  if (!p.ok || scratch_bytes < c.bytes || (reinterpret_cast<uintptr_t>(scratch) & 15)) return kOk;
  if (p.wide && fwd != nullptr && (v->in_src == nullptr || v->in_score == nullptr)) return kOk;
  K2B_CUDA_OK(cudaMemsetAsync(c.status, 0, c.clear_bytes, stream));
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
  if (p.wide) {
    *redo_if = c.status;
  } else {
    auto exact = log_semiring ? ExactChain<Real, true> : ExactChain<Real, false>;
    for (int32_t first = 0; first < v->num_fsas; first += 65535) {
      { exact<<<dim3(ndir, std::min(v->num_fsas - first, 65535)), 256, 0, stream>>>(
          *v, c.pool, c.descs, c.vals, c.expo, fwd, bwd, entering, dir_base, first,
          v->num_fsas * v->max_layers, p.rows, c.status); NoteLaunch(); }
    }
  }
  K2B_CUDA_OK(cudaGetLastError());
  *launched = true;
  return kOk;
}

template int32_t LaunchLayerScores<float>(const k2b200_fsa_view *, int32_t, float *, float *,
                                          int32_t *, void *, size_t, cudaStream_t, bool *,
                                          const int32_t **);
template int32_t LaunchLayerScores<double>(const k2b200_fsa_view *, int32_t, double *, double *,
                                           int32_t *, void *, size_t, cudaStream_t, bool *,
                                           const int32_t **);

}  // namespace k2b
