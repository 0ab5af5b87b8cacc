// Persistent frame-synchronous Viterbi kernel for graphs that fit in shared memory.
//
// One CTA per (graph/sequence pair, direction) walks all frames in-kernel: the
// graph's arcs (in incoming order for the forward direction, leaving order for
// the backward one) and the two ping-pong score vectors live in shared memory,
// the dense rows are prefetched into a shared-memory ring with cp.async several
// frames ahead of the recursion, and one __syncthreads per frame is the only
// synchronisation.  Each frame's state scores are also written to the global
// (t, state) grids that the pruning pass reads.
//
// Same arithmetic as the per-frame launch path (and as the reference's DoStep,
// k2/csrc/intersect_dense.cu:778-847): (prev + arc.score) + dense, then max.
#include <algorithm>
#include <vector>

#include <type_traits>

#include "cp_async.cuh"
#include "intersect_internal.cuh"

namespace k2b {

constexpr size_t kSmemBudget = 200 * 1024;  // of the 227 KB a CTA may use
constexpr int kMaxStages = 8;

struct SmemPlan {
  int32_t s_pad, a_pad, row_pad, stages;
  size_t bytes;
};

static SmemPlan PlanSmem(int32_t max_states, int32_t max_arcs, int32_t cols) {
  SmemPlan p;
  p.s_pad = (max_states + 1 + 3) & ~3;
  p.a_pad = (max_arcs + 3) & ~3;
  p.row_pad = (cols + 1 + 3) & ~3;  // +1: a -inf slot for out-of-range labels
  size_t fixed = sizeof(float) * 2 * p.s_pad      // score ping-pong
                 + sizeof(int32_t) * p.s_pad      // splits
                 + (size_t)12 * p.a_pad;          // other-end state, column slot, score
  size_t row = sizeof(float) * p.row_pad;
  int32_t stages = 0;
  if (fixed < kSmemBudget) stages = (int32_t)std::min<size_t>(kMaxStages, (kSmemBudget - fixed) / row);
  p.stages = stages;
  p.bytes = fixed + row * std::max(stages, 0);
  return p;
}

bool PersistentViterbiFits(const Layout &L, const k2b200_intersect_args *a) {
  SmemPlan p = PlanSmem(L.max_states, L.max_arcs, a->cols);
  return p.stages >= 2 && a->num_fsas <= 65535;
}

// grid = (2 directions, pairs); dynamic shared memory per PlanSmem.
__global__ void __launch_bounds__(1024)
PersistentViterbi(const FsaInfo *__restrict__ infos, const Arc *__restrict__ arcs,
                  const int32_t *__restrict__ a_row_splits2,
                  const int32_t *__restrict__ in_splits, const int32_t *__restrict__ in_arcs,
                  const float *__restrict__ scores, int32_t cols, float *__restrict__ fwd,
                  float *__restrict__ bwd, int32_t s_pad, int32_t a_pad, int32_t row_pad,
                  int32_t stages, int32_t lanes_log2, const int32_t *__restrict__ only_unfit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (only_unfit != nullptr && !only_unfit[blockIdx.y]) return;
  const FsaInfo f = infos[blockIdx.y];
  const int dir = blockIdx.x;  // 0 forward, 1 backward
  const int32_t S = f.num_states, A = f.num_arcs, Tk = f.tk;
  if (S == 0) return;
  float *score_buf = reinterpret_cast<float *>(smem_raw);           // [2][s_pad]
  int32_t *splits = reinterpret_cast<int32_t *>(score_buf + 2 * s_pad);  // [s_pad]
  int32_t *arc_state = splits + s_pad;                              // [a_pad]
  int32_t *arc_col = arc_state + a_pad;                             // [a_pad]
  float *arc_score = reinterpret_cast<float *>(arc_col + a_pad);   // [a_pad]
  float *ring = arc_score + a_pad;                                  // [stages][row_pad]

  const int tid = threadIdx.x, nt = blockDim.x;
  // ---- stage the graph --------------------------------------------------
  const int32_t *gsplits = (dir == 0 ? in_splits : a_row_splits2) + f.state_off;
  for (int32_t s = tid; s <= S; s += nt) splits[s] = gsplits[s] - f.arc_off;
  for (int32_t k = tid; k < A; k += nt) {
    Arc arc = arcs[dir == 0 ? in_arcs[f.arc_off + k] : f.arc_off + k];
    arc_state[k] = dir == 0 ? arc.src : arc.dest;
    int32_t c = arc.label + 1;
    arc_col[k] = (c >= 0 && c < cols) ? c : cols;  // slot `cols` holds -inf
    arc_score[k] = arc.score;
  }
  for (int32_t st = tid; st < stages; st += nt) ring[(size_t)st * row_pad + cols] = -INFINITY;
  // ---- initial scores -----------------------------------------------------
  float *grid = (dir == 0 ? fwd : bwd) + f.grid_off;
  for (int32_t s = tid; s < S; s += nt) {
    float v = (dir == 0 ? (s == 0) : (s == S - 1)) ? 0.0f : -INFINITY;
    score_buf[s] = v;
    grid[(int64_t)(dir == 0 ? 0 : Tk) * S + s] = v;
  }
  // ---- prefetch the first stages-1 rows -----------------------------------
  // step t (1..Tk) consumes dense row t-1 (forward) or Tk-t (backward)
  auto issue_row = [&](int32_t step) {
    if (step <= Tk) {
      const int64_t row = (int64_t)f.row0 + (dir == 0 ? step - 1 : Tk - step);
      const float *src = scores + row * cols;
      float *dst = ring + (size_t)((step - 1) % stages) * row_pad;
      for (int32_t c = tid; c < cols; c += nt) CpAsync4(dst + c, src + c);
    }
    CpAsyncCommit();  // always commit so the group count stays uniform
  };
  for (int32_t step = 1; step < stages; ++step) issue_row(step);

  const int32_t G = 1 << lanes_log2, g = tid & (G - 1);
  const int32_t states_per_pass = nt >> lanes_log2;
  for (int32_t t = 1; t <= Tk; ++t) {
    CpAsyncWaitDyn(stages - 2);  // this thread's copies of row for step t have landed
    __syncthreads();             // ... everyone's have; previous frame's scores are complete
    issue_row(t + stages - 1);   // refills the slot consumed by step t-1
    const float *cur = score_buf + ((t - 1) & 1) * s_pad;
    float *nxt = score_buf + (t & 1) * s_pad;
    const float *row = ring + (size_t)((t - 1) % stages) * row_pad;
    float *gout = grid + (int64_t)(dir == 0 ? t : Tk - t) * S;
    for (int32_t s0 = 0; s0 < S; s0 += states_per_pass) {
      const int32_t s = s0 + (tid >> lanes_log2);
      float best = -INFINITY;
      if (s < S) {
        for (int32_t k = splits[s] + g; k < splits[s + 1]; k += G) {
          float v = __fadd_rn(__fadd_rn(cur[arc_state[k]], arc_score[k]), row[arc_col[k]]);
          best = v > best ? v : best;
        }
      }
      for (int32_t d = G >> 1; d > 0; d >>= 1) {
        float o = __shfl_xor_sync(0xffffffffu, best, d);
        best = o > best ? o : best;
      }
      if (s < S && g == 0) {
        nxt[s] = best;
        gout[s] = best;
      }
    }
  }
  CpAsyncWait<0>();
}

// ---------------------------------------------------------------------------
// Register variant for graphs whose states have at most kMaxDeg arcs in each
// direction (CTC graphs have 3) and at most 1024 states: one thread per state keeps
// its arcs in registers and fetches the dense scores of its own arcs straight from
// global memory kPrefetch frames ahead, so a frame costs one __syncthreads, kMaxDeg
// shared-memory reads of the previous frame's scores and a few adds.  Unused arc
// slots carry a score of -inf and never win the max.
//
// Bound by the gathers of dense scores, a sector each: three per state and frame took 175 us for
// 32 x 800 frames of up to 402 states.  Where all arcs that enter a state carry one label, as in
// CTC graphs, one is enough: walking forward it is added after the max (rounding is monotonic, so
// max_j fl(y_j + x) = fl(max_j y_j + x), bit for bit); walking backward, if moreover all arcs
// score zero, (score of the destination + 0) + x is the same for all arcs into that state, which
// leaves it behind with its x added: 107 us.
// ---------------------------------------------------------------------------
constexpr int kRegMaxDeg = 4;  // largest degree any instantiation handles

bool RegisterViterbiFits(const Layout &L, const k2b200_intersect_args *a) {
  return a->a_max_degree > 0 && a->a_max_degree <= kRegMaxDeg && L.max_states <= 1024 &&
         a->num_fsas <= 65535;
}

template <int kMaxThreads, int kDeg, int kRegPrefetch>
__global__ void __launch_bounds__(kMaxThreads)
RegisterViterbi(const FsaInfo *__restrict__ infos, const Arc *__restrict__ arcs,
                const int32_t *__restrict__ a_row_splits2, const int32_t *__restrict__ in_splits,
                const int32_t *__restrict__ in_arcs, const float *__restrict__ scores,
                int32_t cols, float *__restrict__ fwd, float *__restrict__ bwd) {
  __shared__ float buf[2][1024];
  const FsaInfo f = infos[blockIdx.y];
  const int dir = blockIdx.x;
  const int32_t S = f.num_states, Tk = f.tk;
  if (S == 0) return;
  const int32_t s = threadIdx.x;
  const bool active = s < S;

  int32_t other[kDeg], col[kDeg];
  float w[kDeg];
#pragma unroll
  for (int j = 0; j < kDeg; ++j) {
    other[j] = 0;
    col[j] = 0;
    w[j] = -INFINITY;
  }
  if (active) {
    const int32_t *splits = dir == 0 ? in_splits : a_row_splits2;
    const int32_t a0 = splits[f.state_off + s], n = splits[f.state_off + s + 1] - a0;
#pragma unroll
    for (int j = 0; j < kDeg; ++j) {
      if (j < n) {
        const Arc arc = arcs[dir == 0 ? in_arcs[a0 + j] : a0 + j];
        other[j] = dir == 0 ? arc.src : arc.dest;
        const int32_t c = arc.label + 1;
        if (c >= 0 && c < cols) {
          col[j] = c;
          w[j] = arc.score;
        }
      }
    }
  }
  // step t (1..Tk) consumes dense row t-1 (forward) or Tk-t (backward)
  const float *base = scores + (int64_t)f.row0 * cols;
  auto row_of = [&](int32_t step) {
    step = step > Tk ? Tk : step;
    return dir == 0 ? step - 1 : Tk - step;
  };
  float *grid = (dir == 0 ? fwd : bwd) + f.grid_off;
  const float first = (dir == 0 ? (s == 0) : (s == S - 1)) ? 0.0f : -INFINITY;
  if (active) grid[(int64_t)(dir == 0 ? 0 : Tk) * S + s] = first;
  // the column of the arcs that enter this state, and whether they and (walking backward) the
  // scores of the leaving arcs allow one gather per state
  int32_t my_col = 0;
  bool one = true;
  if (active) {
    bool any = false;
    const int32_t a0 = in_splits[f.state_off + s], a1 = in_splits[f.state_off + s + 1];
    for (int32_t k = a0; k < a1; ++k) {
      const int32_t c = arcs[in_arcs[k]].label + 1;
      if (c < 0 || c >= cols) continue;  // never scores
      if (any && c != my_col) one = false;
      my_col = c;
      any = true;
    }
    if (dir == 1)
#pragma unroll
      for (int j = 0; j < kDeg; ++j) one &= w[j] == 0.0f || w[j] == -INFINITY;
  }
  if (__syncthreads_and(one)) {
    // x[u]: of step t0 + u, walking backward of the step after it; rows past the end are the last
    const float *row = base + (int64_t)row_of(dir == 0 ? 1 : 2) * cols + my_col;
    const float *const end = base + (int64_t)row_of(Tk) * cols + my_col;
    const int64_t row_step = dir == 0 ? cols : -(int64_t)cols;
    auto next = [&]() {
      const float v = __ldg(row);
      if (row != end) row += row_step;
      return v;
    };
    float x[kRegPrefetch];
#pragma unroll
    for (int d = 0; d < kRegPrefetch; ++d) x[d] = next();
    buf[0][s] = dir == 0 ? first : __fadd_rn(first, __ldg(base + row_of(1) * cols + my_col));
    float *out = grid + (int64_t)(dir == 0 ? 1 : Tk - 1) * S + s;
    const int64_t out_step = dir == 0 ? S : -(int64_t)S;
    for (int32_t t0 = 1; t0 <= Tk; t0 += kRegPrefetch) {
#pragma unroll
      for (int u = 0; u < kRegPrefetch; ++u) {
        const int32_t t = t0 + u;
        if (t > Tk) break;
        __syncthreads();
        const float *cur = buf[(t - 1) & 1];
        float best = -INFINITY;
#pragma unroll
        for (int j = 0; j < kDeg; ++j) best = fmaxf(best, __fadd_rn(cur[other[j]], w[j]));
        // (a score that is not a number never wins)
        const float plus = fmaxf(__fadd_rn(best, x[u]), -INFINITY);
        x[u] = next();
        buf[t & 1][s] = plus;
        if (active) *out = dir == 0 ? plus : best;
        out += out_step;
      }
    }
    return;
  }
  float x[kDeg][kRegPrefetch];
#pragma unroll
  for (int d = 0; d < kRegPrefetch; ++d) {
    const int32_t r = row_of(1 + d) * cols;
#pragma unroll
    for (int j = 0; j < kDeg; ++j) x[j][d] = __ldg(base + r + col[j]);
  }
  buf[0][s] = first;
  for (int32_t t0 = 1; t0 <= Tk; t0 += kRegPrefetch) {
#pragma unroll
    for (int u = 0; u < kRegPrefetch; ++u) {
      const int32_t t = t0 + u;
      if (t > Tk) break;
      __syncthreads();
      const float *cur = buf[(t - 1) & 1];
      float best = -INFINITY;
#pragma unroll
      for (int j = 0; j < kDeg; ++j) {
        const float v = __fadd_rn(__fadd_rn(cur[other[j]], w[j]), x[j][u]);
        best = v > best ? v : best;
      }
      const int32_t r = row_of(t + kRegPrefetch) * cols;
#pragma unroll
      for (int j = 0; j < kDeg; ++j) x[j][u] = __ldg(base + r + col[j]);
      buf[t & 1][s] = best;
      if (active) grid[(int64_t)(dir == 0 ? t : Tk - t) * S + s] = best;
    }
  }
}

// ---------------------------------------------------------------------------
// Lane plans.  The recursion kernel keeps the arcs of state s in the registers of
// G(s) = ceil(degree(s) / kDeg) lanes of one warp, so that a frame costs every lane
// the same few arcs whatever the degree distribution of the graph is.  PlanLanes
// lays the lane groups of one graph and direction out over the threads of a CTA: groups
// sorted by size, largest first (states in increasing order within a size), packed
// next-fit into warps - a group never straddles two warps.
//   plan[(dir * n + i) * kLaneThreads + thread] = state | lane << 16 | G << 24, or -1
// bit 0 of unfit[i] is set when graph i needs more lanes than a CTA has (or has more than
// 32 * kDeg arcs on a state); the shared-memory kernels below take those graphs.
// Graphs whose largest degree is at most kDeg need no plan: thread s owns state s.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
PlanLanes(const FsaInfo *__restrict__ infos, int32_t n,
          const int32_t *__restrict__ a_row_splits2, const int32_t *__restrict__ in_splits,
          int32_t k_deg, int32_t threads, int32_t *__restrict__ plan, int32_t *__restrict__ unfit) {
  // per group size G = 1..32: number of states, lanes left in the warp where the
  // size class starts, first lane of that start, first lane of the following warps
  __shared__ int32_t count[33], head_room[33], head_pos[33], body_pos[33];
  __shared__ int32_t bad;
  const int32_t i = blockIdx.y, dir = blockIdx.x;
  const FsaInfo f = infos[i];
  const int32_t S = f.num_states;
  const int tid = threadIdx.x, nt = blockDim.x;
  int32_t *out = plan + ((int64_t)dir * n + i) * kLaneThreads;
  for (int32_t t = tid; t < kLaneThreads; t += nt) out[t] = -1;
  if (tid < 33) count[tid] = 0;
  if (tid == 0) bad = S > threads;
  __syncthreads();
  const int32_t *splits = (dir == 0 ? in_splits : a_row_splits2) + f.state_off;
  auto lanes_of = [&](int32_t s) {
    const int32_t deg = splits[s + 1] - splits[s];
    return deg <= k_deg ? 1 : (deg + k_deg - 1) / k_deg;
  };
  if (S <= threads)
    for (int32_t s = tid; s < S; s += nt) {
      const int32_t G = lanes_of(s);
      if (G > 32) bad = 1; else atomicAdd(&count[G], 1);
    }
  __syncthreads();
  if (tid == 0 && !bad) {
    int32_t pos = 0;
    for (int G = 32; G >= 1; --G) {
      const int32_t c = count[G];
      if (c == 0) continue;
      const int32_t room = (32 - (pos & 31)) / G;  // groups that still fit in this warp
      const int32_t per_warp = 32 / G;
      head_room[G] = room;
      head_pos[G] = pos;
      if (c <= room) {
        pos += c * G;
      } else {
        const int32_t rest = c - room;
        const int32_t body = (pos + room * G + 31) & ~31;
        body_pos[G] = body;
        pos = body + (rest / per_warp) * 32 + (rest % per_warp) * G;
      }
      if (pos > threads) bad = 1;
    }
    if (!bad && (pos > 768 || S > 768)) atomicOr(&unfit[n + i], 1);
  }
  __syncthreads();
  if (bad) {
    if (tid == 0) atomicOr(&unfit[i], 1);
    return;
  }
  // warp w places the size classes w, w + 8, ...: ordered compaction by ballot
  const int warp = tid >> 5, lane = tid & 31;
  for (int G = 1 + warp; G <= 32; G += nt >> 5) {
    if (count[G] == 0) continue;
    const int32_t per_warp = 32 / G, room = head_room[G];
    int32_t seen = 0;
    for (int32_t s0 = 0; s0 < S; s0 += 32) {
      const int32_t s = s0 + lane;
      const bool in = s < S && lanes_of(s) == G;
      const uint32_t m = __ballot_sync(0xffffffffu, in);
      if (in) {
        const int32_t j = seen + __popc(m & ((1u << lane) - 1u));
        int32_t p0;
        if (j < room) {
          p0 = head_pos[G] + j * G;
        } else {
          const int32_t r = j - room;
          p0 = body_pos[G] + (r / per_warp) * 32 + (r % per_warp) * G;
        }
        for (int32_t g = 0; g < G; ++g) out[p0 + g] = s | (g << 16) | (G << 24);
      }
      seen += __popc(m);
    }
  }
}


int32_t LaneThreads(const Layout &L) {
  return L.max_states + L.max_arcs / kLaneDeg <= kLaneRoom768 ? 768 : 1024;
}

constexpr int kVitRing = 4;   // slots of LanesViterbi's row ring = frames per unrolled group
constexpr size_t kVitRingBytes = 200 * 1024;

bool LanePlanApplies(const Layout &L, const k2b200_intersect_args *a) {
  const bool register_fit = a->a_max_degree > 0 && a->a_max_degree <= 4 && L.max_states <= 1024;
  return !register_fit && L.max_states <= kLaneThreads && a->num_fsas <= 65535 &&
         sizeof(float) * kVitRing * ((size_t)a->cols + 3) <= kVitRingBytes &&
         PersistentViterbiFits(L, a);
}

int32_t LaunchPlanLanes(const Layout &L, const k2b200_intersect_args *a, char *ws,
                        cudaStream_t stream) {
  int32_t *unfit = reinterpret_cast<int32_t *>(ws + L.off_unfit);
  K2B_CUDA_OK(cudaMemsetAsync(unfit, 0, sizeof(int32_t) * 2 * a->num_fsas, stream));
  if (!L.lane_plan) return kOk;
  { PlanLanes<<<dim3(2, a->num_fsas), 256, 0, stream>>>(
      reinterpret_cast<const FsaInfo *>(ws + L.off_infos), a->num_fsas, a->a_row_splits2,
      a->a_in_splits, kLaneDeg, L.lane_threads, reinterpret_cast<int32_t *>(ws + L.off_plan),
      unfit);
    NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

// ---------------------------------------------------------------------------
// Viterbi recursion with planned lanes: as RegisterViterbi, but the arcs of a state
// are spread over the G(s) lanes its plan gives it, which take the max by shuffles.
// The rows of dense scores arrive in a ring in shared memory by 4-byte cp.async, kVitAhead
// frames ahead (rows of C + 1 floats are not 16-byte aligned).  The frame loop is unrolled
// over the ring, so a frame costs a lane, per arc, a load of the neighbour's score and of
// the dense score at constant offsets, two additions and a max.  When all arcs of a warp's
// lanes carry the label of their state (walking forward in a graph where every state has
// one entering label) the dense score is added once per state, after the max: rounding is
// monotonic, so max_j fl(y_j + x) = fl(max_j y_j + x), bit for bit.
// Graphs marked unfit are skipped (PersistentViterbi handles them).
// ---------------------------------------------------------------------------
constexpr int kVitAhead = 3;  // rows requested ahead of the frame that uses them

// kPitch: floats of a ring slot, 0: cols_pad of them.  With a constant pitch every access of the
// frame loop has its slot in the instruction's offset.
// Bound by the latency of a frame and by the issue of its instructions: one max instead of a
// comparison and a selection, constant slot offsets, and copies by the warps that hold a
// column only took 500 frames of 4627 arcs from 246 to 215 us per round of CTAs (one CTA per
// SM).  40 registers, for two CTAs per SM, leave no room to request a lane's eight scores
// together: 256 CTAs took 460 us, and 431 with up to 80 (421 with the additions in pairs).
template <int kDeg, int kPitch, int kThreads>
__global__ void __launch_bounds__(kThreads, 1)
LanesViterbi(const FsaInfo *__restrict__ infos, int32_t n, const Arc *__restrict__ arcs,
             const int32_t *__restrict__ a_row_splits2, const int32_t *__restrict__ in_splits,
             const int32_t *__restrict__ in_arcs, const float *__restrict__ scores,
             int32_t cols, int32_t cols_pad, float *__restrict__ fwd, float *__restrict__ bwd,
             const int32_t *__restrict__ plan, const int32_t *__restrict__ unfit,
             ChainShare share) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float buf[2][kThreads];
  int32_t after;  // the step before the first one
  const int32_t chain = ChainOf(share, blockIdx.x, 2 * n, &after), i = chain >> 1;
  if ((unfit[i] & 1) || unfit[n + i] != LaneClass(kThreads)) return;
  const int dir = chain & 1;
  const int32_t S = infos[i].num_states, Tk = infos[i].tk;
  const int32_t end = share.part == 1 ? min(share.cut, Tk) : Tk;  // the last step
  if (S == 0 || (after > 0 && after >= end)) return;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int32_t pitch = kPitch ? kPitch : cols_pad;
  float *ring = reinterpret_cast<float *>(smem_raw);  // [kVitRing][pitch]
  int32_t s = -1, g = 0, G = 1, col0 = -1;
  {
    const int32_t code = plan[((int64_t)dir * n + i) * kLaneThreads + tid];
    if (code >= 0) {
      s = code & 0xffff;
      g = (code >> 16) & 0xff;
      G = code >> 24;
    }
  }
  // byte offsets of an arc's other end in a buffer and of its column in a row
  uint32_t other[kDeg], col[kDeg];
  float w[kDeg];
  bool same = true;
#pragma unroll
  for (int j = 0; j < kDeg; ++j) {
    other[j] = 0;
    col[j] = 0;
    w[j] = -INFINITY;
  }
  if (s >= 0) {
    const int32_t state_off = infos[i].state_off;
    const int32_t *splits = dir == 0 ? in_splits : a_row_splits2;
    const int32_t a0 = splits[state_off + s], a1 = splits[state_off + s + 1];
#pragma unroll
    for (int j = 0; j < kDeg; ++j) {
      const int32_t k = a0 + g + j * G;
      if (k < a1) {
        const Arc arc = arcs[dir == 0 ? in_arcs[k] : k];
        other[j] = 4u * (uint32_t)(dir == 0 ? arc.src : arc.dest);
        const int32_t c = arc.label + 1;
        if (c >= 0 && c < cols) {
          col[j] = 4u * (uint32_t)c;
          w[j] = arc.score;
          if (col0 < 0) col0 = c;
          else if (c != col0) same = false;
        }
      }
    }
  }
  const uint32_t col0_off = 4u * (uint32_t)max(col0, 0);
  const int32_t g_max = __reduce_max_sync(0xffffffffu, G);  // widest lane group of this warp
  const bool hoist = __syncthreads_and(same);  // uniform over the CTA
  // step t (1..Tk) consumes dense row t-1 (forward) or Tk-t (backward).  The warps that hold
  // a column copy it; the others neither copy nor wait.
  const bool copies = (tid & ~31) < cols;
  const float *src = scores + ((int64_t)infos[i].row0 + (dir == 0 ? after : Tk - 1 - after)) * cols;
  const int64_t src_step = dir == 0 ? cols : -(int64_t)cols;
  auto issue_row = [&](bool there, int32_t slot) {
    if (there)
      for (int32_t c = tid; c < cols; c += nt) CpAsync4(ring + slot * pitch + c, src + c);
    CpAsyncCommit();
    src += src_step;
  };
  if (copies)
    for (int32_t step = 1; step <= kVitAhead; ++step)
      issue_row(after + step <= end, (step - 1) % kVitRing);
  const int64_t stride = dir == 0 ? (int64_t)S : -(int64_t)S;
  const bool store = s >= 0 && g == 0;
  float *gout;
  {
    float *grid = (dir == 0 ? fwd : bwd) + infos[i].grid_off;
    float *first = grid + (int64_t)(dir == 0 ? after : Tk - after) * S;
    for (int32_t q = tid; q < S; q += nt) {
      float v0 = (dir == 0 ? (q == 0) : (q == S - 1)) ? 0.0f : -INFINITY;
      if (after > 0) v0 = first[q];
      else first[q] = v0;
      buf[0][q] = v0;
    }
    gout = first + stride + max(s, 0);
  }
  // the frame loop once per kind of CTA, so that the unrolled code of only one is fetched
  auto frames = [&](auto hoist_tag) {
    constexpr bool kHoist = decltype(hoist_tag)::value;
    for (int32_t t0 = after + 1; t0 <= end; t0 += kVitRing) {
#pragma unroll
      for (int u = 0; u < kVitRing; ++u) {
        const int32_t t = t0 + u;
        if (t > end) break;
        if (copies) CpAsyncWait<kVitAhead - 1>();  // this thread's part of row t has landed
        __syncthreads();  // ... everyone's has; the scores of step t - 1 are complete
        if (copies) issue_row(t + kVitAhead <= end, (u + kVitAhead) % kVitRing);
        // t0 is odd: (t - 1) & 1 == u & 1
        const char *cur = reinterpret_cast<const char *>(buf[u & 1]);
        const char *row = reinterpret_cast<const char *>(ring + u * pitch);
        auto at = [](const char *base, uint32_t off) {
          return *reinterpret_cast<const float *>(base + off);
        };
        // (a max of two chains: NaN never wins, as in the reference's comparisons)
        float best = -INFINITY, best1 = -INFINITY;
#pragma unroll
        for (int j = 0; j < kDeg; j += 2) {
          float2 x = AddPair(make_float2(at(cur, other[j]), at(cur, other[j + 1])),
                             make_float2(w[j], w[j + 1]));
          if (!kHoist) x = AddPair(x, make_float2(at(row, col[j]), at(row, col[j + 1])));
          best = fmaxf(best, x.x);
          best1 = fmaxf(best1, x.y);
        }
        best = fmaxf(best, best1);
#pragma unroll
        for (int32_t d = 16; d > 0; d >>= 1) {
          if (d < g_max) {  // warp-uniform
            const float o = __shfl_down_sync(0xffffffffu, best, d);
            if (g + d < G) best = fmaxf(best, o);
          }
        }
        if (store) {
          if (kHoist) best = __fadd_rn(best, at(row, col0_off));
          buf[(u + 1) & 1][s] = best;
          *gout = best;
        }
        gout += stride;
      }
    }
  };
  if (hoist) frames(std::true_type{}); else frames(std::false_type{});
  CpAsyncWait<0>();
}

int32_t LaunchLanesViterbi(const Layout &L, const k2b200_intersect_args *a,
                           const FsaInfo *d_infos, float *fwd, float *bwd, const int32_t *plan,
                           const int32_t *unfit, cudaStream_t stream) {
  static_assert(kLaneDeg % 2 == 0, "arcs are taken in pairs");
  ChainShare share = ShareChains(L);
  const int32_t cols_pad = (a->cols + 3) & ~3;
  auto launch = [&](auto kernel, int32_t threads, int32_t pitch) -> int32_t {
    const size_t smem = sizeof(float) * kVitRing * (size_t)pitch;
    K2B_REQUIRE(smem <= kVitRingBytes, "too many columns for the lane Viterbi kernel");
    K2B_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
    for (share.part = share.early > 0 ? 1 : 0; share.part <= (share.early > 0 ? 2 : 0);
         ++share.part) {
      kernel<<<share.part == 1 ? share.early : 2 * a->num_fsas, threads, smem, stream>>>(
          d_infos, a->num_fsas, reinterpret_cast<const Arc *>(a->a_arcs), a->a_row_splits2,
          a->a_in_splits, a->a_in_arcs, a->scores, a->cols, cols_pad, fwd, bwd, plan, unfit, share);
      NoteLaunch();
    }
    return kOk;
  };
  // graphs over phones have rows of up to 128 columns
#define K2B_LANES_VITERBI(THREADS)                                                           \
  {                                                                                          \
    if (a->cols <= 128) K2B_FORWARD(launch(LanesViterbi<kLaneDeg, 128, THREADS>, THREADS, 128)); \
    else K2B_FORWARD(launch(LanesViterbi<kLaneDeg, 0, THREADS>, THREADS, cols_pad)); \
  }
  K2B_LANE_THREADS(L.lane_threads, K2B_LANES_VITERBI);
#undef K2B_LANES_VITERBI
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

int32_t LaunchRegisterViterbi(const Layout &L, const k2b200_intersect_args *a,
                              const FsaInfo *d_infos, float *fwd, float *bwd,
                              cudaStream_t stream) {
  int32_t threads = std::max(32, (L.max_states + 31) / 32 * 32);
  dim3 grid(2, a->num_fsas);
  const Arc *arcs = reinterpret_cast<const Arc *>(a->a_arcs);
#define K2B_LAUNCH_REG(MAXT, DEG, PF)                                                      \
  { RegisterViterbi<MAXT, DEG, PF><<<grid, threads, 0, stream>>>(                         \
        d_infos, arcs, a->a_row_splits2, a->a_in_splits, a->a_in_arcs, a->scores, a->cols, \
        fwd, bwd); NoteLaunch(); }
  if (threads <= 512) {
    if (a->a_max_degree <= 3) K2B_LAUNCH_REG(512, 3, 12) else K2B_LAUNCH_REG(512, 4, 8)
  } else {
    if (a->a_max_degree <= 3) K2B_LAUNCH_REG(1024, 3, 8) else K2B_LAUNCH_REG(1024, 4, 6)
  }
#undef K2B_LAUNCH_REG
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

int32_t LaunchPersistentViterbi(const Layout &L, const k2b200_intersect_args *a,
                                const FsaInfo *d_infos, float *fwd, float *bwd,
                                cudaStream_t stream, const int32_t *only_unfit) {
  SmemPlan p = PlanSmem(L.max_states, L.max_arcs, a->cols);
  K2B_CUDA_OK(cudaFuncSetAttribute(PersistentViterbi, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)p.bytes));
  // lanes per state: about half the mean degree, so every lane loops ~2 arcs
  int32_t mean_deg = a->num_states > 0 ? (a->num_arcs + a->num_states - 1) / a->num_states : 1;
  int32_t lanes_log2 = 0;
  while ((2 << lanes_log2) <= mean_deg / 2 && lanes_log2 < 5) ++lanes_log2;
  int64_t lanes = (int64_t)L.max_states << lanes_log2;
  int32_t threads = (int32_t)std::min<int64_t>(1024, std::max<int64_t>(128, (lanes + 31) / 32 * 32));
  dim3 grid(2, a->num_fsas);
  { PersistentViterbi<<<grid, threads, p.bytes, stream>>>(
      d_infos, reinterpret_cast<const Arc *>(a->a_arcs), a->a_row_splits2, a->a_in_splits,
      a->a_in_arcs, a->scores, a->cols, fwd, bwd, p.s_pad, p.a_pad, p.row_pad, p.stages,
      lanes_log2, only_unfit); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

}  // namespace k2b
