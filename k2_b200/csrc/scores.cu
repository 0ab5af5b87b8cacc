// Forward/backward scores, total scores, arc posteriors and their gradients over a
// layered (top-sorted, acyclic) FsaVec, plus the small gather/scatter, best-path and
// property kernels that sit on the same path.
//
// Follows the arithmetic of the reference (k2/csrc/fsa_utils.cu:1124-1278
// GetForwardScores, :1345-1454 GetBackwardScores, :1809-1837 GetTotScores,
// :1839-1901 GetArcPost; k2/python/csrc/torch/fsa.cu:493-592 the backward of
// tot_scores; k2/csrc/tensor_ops.cu:304-334 IndexAdd; k2/csrc/fsa_algo.cu:869-1144
// ShortestPath; k2/csrc/fsa.cu:54-217 properties) but walks the layers inside one
// persistent kernel per (FSA, direction) instead of launching per state batch.
#include <algorithm>
#include <cmath>

#include "scores_internal.cuh"

namespace k2b {

// grid = (directions, fsas).  dir = blockIdx.x + dir_base: 0 forward, 1 backward.
template <typename Real, bool kLog>
__global__ void __launch_bounds__(256)
LayeredScores(k2b200_fsa_view v, Real *forward, Real *backward, int32_t *entering_arcs,
              int32_t dir_base, int32_t fsa_base, const int32_t *run_if) {
  // run_if (optional): only do the work when the word it points to is non-zero
  if (run_if != nullptr && *run_if == 0) return;
  LayeredScoresDevice<Real, kLog>(v, fsa_base + blockIdx.y, blockIdx.x + dir_base, forward,
                                  backward, entering_arcs);
}

template <typename Real>
__global__ void TotScores(const int32_t *__restrict__ row_splits1, int32_t num_fsas,
                          const Real *__restrict__ forward, Real *__restrict__ tot) {
  int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= num_fsas) return;
  int32_t b = row_splits1[i], e = row_splits1[i + 1];
  tot[i] = e > b ? forward[e - 1] : (Real)-INFINITY;
}

template <typename Real>
__device__ __forceinline__ Real PostOf(const int32_t *__restrict__ row_splits1, int32_t fsa,
                                       int32_t src01, const Arc &arc,
                                       const Real *__restrict__ forward,
                                       const Real *__restrict__ backward) {
  const int32_t b = row_splits1[fsa], e = row_splits1[fsa + 1];
  const Real kNegInf = -INFINITY;
  Real tot = (Real)0.5 * (forward[e - 1] + backward[b]);
  Real neg = tot != kNegInf ? -tot : kNegInf;
  return (Real)arc.score + forward[src01] + backward[b + arc.dest] + neg;
}

template <typename Real>
__global__ void ArcPost(const int32_t *__restrict__ row_splits1,
                        const int32_t *__restrict__ row_ids1,
                        const int32_t *__restrict__ row_ids2, const Arc *__restrict__ arcs,
                        int32_t num_arcs, const Real *__restrict__ forward,
                        const Real *__restrict__ backward, Real *__restrict__ post) {
  int32_t a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= num_arcs) return;
  const int32_t src01 = row_ids2[a];
  post[a] = PostOf(row_splits1, row_ids1[src01], src01, arcs[a], forward, backward);
}

template <typename Real>
__global__ void LogBackward(const int32_t *__restrict__ row_ids1,
                            const int32_t *__restrict__ row_ids2, int32_t num_arcs,
                            const Real *__restrict__ post, const Real *__restrict__ tot_grad,
                            int64_t stride, float *__restrict__ grad) {
  int32_t a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= num_arcs) return;
  int32_t fsa = row_ids1[row_ids2[a]];
  grad[a] = (float)(ExpReal<Real>(post[a]) * tot_grad[fsa * stride]);
}

// ArcPost and LogBackward in one pass, where nobody else wants the posteriors: 16 bytes of the arc
// and three gathers in, 4 bytes out, instead of 8 more each way.  Bound by latency and the
// exponential: 3.3 M arcs 46 + 34 -> 50 us.
template <typename Real>
__global__ void LogBackwardScores(const int32_t *__restrict__ row_splits1,
                                  const int32_t *__restrict__ row_ids1,
                                  const int32_t *__restrict__ row_ids2,
                                  const Arc *__restrict__ arcs, int32_t num_arcs,
                                  const Real *__restrict__ forward,
                                  const Real *__restrict__ backward,
                                  const Real *__restrict__ tot_grad, int64_t stride,
                                  float *__restrict__ grad) {
  const int32_t a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= num_arcs) return;
  const int32_t src01 = row_ids2[a], fsa = row_ids1[src01];
  const Real post = PostOf(row_splits1, fsa, src01, arcs[a], forward, backward);
  grad[a] = (float)(ExpReal<Real>(post) * tot_grad[fsa * stride]);
}

template <typename Real>
__global__ void TropicalBackward(const int32_t *__restrict__ row_ids1,
                                 const int32_t *__restrict__ row_ids2,
                                 const int32_t *__restrict__ best_arcs, int32_t num_best,
                                 const Real *__restrict__ tot_grad, int64_t stride,
                                 float *__restrict__ grad) {
  int32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= num_best) return;
  int32_t a = best_arcs[k];
  grad[a] = (float)tot_grad[row_ids1[row_ids2[a]] * stride];
}

__global__ void IndexAdd(const int32_t *__restrict__ index, const float *__restrict__ value,
                         int32_t n, float *__restrict__ in_out, int64_t size) {
  int32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  int32_t j = index[k];
  if (j >= 0 && j < size) atomicAdd(in_out + j, value[k]);
}

__global__ void IndexSelectI32(const int32_t *__restrict__ src, int64_t size,
                               const int32_t *__restrict__ index, int32_t n,
                               int32_t *__restrict__ out) {
  int32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  int32_t j = index[k];
  out[k] = (j >= 0 && j < size) ? src[j] : 0;
}

// Length of the best path of every FSA (0 when the trace does not reach the
// start state).  One thread per FSA; the walk is bounded by the FSA's state count.
__global__ void PathLengths(const int32_t *__restrict__ row_splits1, const Arc *__restrict__ arcs,
                            const int32_t *__restrict__ entering, int32_t num_fsas,
                            int32_t *__restrict__ lengths) {
  int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= num_fsas) return;
  int32_t b = row_splits1[i], e = row_splits1[i + 1], len = 0;
  if (e > b) {
    int32_t cur = e - 1, idx = entering[cur];
    while (idx != -1 && len <= e - b) {
      ++len;
      cur = b + arcs[idx].src;
      idx = entering[cur];
    }
    if (cur != b || len > e - b) len = 0;
  }
  lengths[i] = len;
}

__global__ void PathFill(const int32_t *__restrict__ row_splits1, const Arc *__restrict__ arcs,
                         const int32_t *__restrict__ entering, int32_t num_fsas,
                         const int32_t *__restrict__ path_splits, int32_t *__restrict__ best) {
  int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= num_fsas) return;
  int32_t p0 = path_splits[i], len = path_splits[i + 1] - p0;
  if (len == 0) return;
  int32_t b = row_splits1[i], cur = row_splits1[i + 1] - 1;
  for (int32_t k = len - 1; k >= 0; --k) {
    int32_t idx = entering[cur];
    best[p0 + k] = idx;
    cur = b + arcs[idx].src;
  }
}

// ---------------------------------------------------------------------------
// Best paths of a layered FsaVec (arcs go from one layer to a later one, as in lattices).  The
// trace back is a chain of dependent loads; read from global memory a step costs two of them,
// about half a microsecond (800 frames: 430 us, and as much again to fill the paths in once
// their lengths are known).  Here Predecessors looks up where the best arc of every state comes
// from, on all SMs; a CTA per FSA brings those of a run of layers into shared memory with all its
// threads, one thread follows the path through them, and all of them write the arcs that it
// took: best[i * max_layers + k] is the k-th last arc.  A step is a load and a
// store: 22 ns.  (The look-up within the one CTA, runs of 8192 states and tests at every step: 800
// layers of 13 states 42 us, now 18 + 2; 150 of 1 200: 87 -> 28 + 2; 32 FSAs of 100 000 states: 271 ->
// 28 + 18.)
// ---------------------------------------------------------------------------
constexpr int kTraceStates = 48 * 1024;  // predecessors in shared memory, at most (TraceRoom)
constexpr int kTraceLayers = 512;        // layers of a run at most, one per thread and trip
constexpr int kTraceFew = 8;             // runs of fewer layers are followed in global memory: to
                                         // fetch a run takes as long as some seven steps there

constexpr int kTraceSteps = 8;           // between looks at whether the run is left

// pred[s]: the state (of its FSA) that the best arc into s comes from, -1: none enters.
__global__ void __launch_bounds__(256)
Predecessors(const Arc *__restrict__ arcs, const int32_t *__restrict__ entering,
             int32_t num_states, int32_t *__restrict__ pred) {
  const int32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= num_states) return;
  const int32_t a = entering[s];
  pred[s] = a >= 0 ? arcs[a].src : -1;
}

// kRoom: the room that a run has, 0: `any_room`.  (Large lattices, of several runs, want the number in
// the code: 4 FSAs of up to 96 layers of 3 000 states 32 us, 42 without; 150 layers of 1 200 27, 37.)
template <int32_t kRoom>
__global__ void __launch_bounds__(512)
TraceLayers(k2b200_fsa_view v, const int32_t *__restrict__ entering,
            const int32_t *__restrict__ all_pred, int32_t any_room, int32_t *__restrict__ best,
            int32_t *__restrict__ lengths) {
  // A run's predecessors, from a multiple of four states on, as offsets in this array of `room`; one
  // outside the run, or none, is kOut, where kOut itself stands: a step then needs no test.
  extern __shared__ int4 pred4[];
  __shared__ int32_t path[kTraceLayers + kTraceSteps], cur_sh, steps_sh;
  const int32_t room = kRoom > 0 ? kRoom : any_room, kOut = 4 * room;
  const char *pred = reinterpret_cast<const char *>(pred4);
  const int32_t i = blockIdx.x;
  const int tid = threadIdx.x;
  const int32_t s_begin = v.row_splits1[i], s_end = v.row_splits1[i + 1];
  int32_t *out = best + (int64_t)i * v.max_layers;
  if (tid == 0) pred4[room / 4] = make_int4(kOut, kOut, kOut, kOut);
  int32_t len = 0, cur = s_end - 1, hi = v.level_offsets[i + 1];
  const int32_t lv0 = v.level_offsets[i];
  bool alive = s_end > s_begin;
  while (alive && hi > lv0 && len <= v.max_layers) {
    // as many layers below `hi` as fit
    const int32_t top = v.level_splits[hi];
    const int32_t l = hi - 1 - tid;
    const int32_t n =
        __syncthreads_count(l >= lv0 && top - (v.level_splits[l] & ~3) <= room);
    const int32_t lo = hi - max(n, 1), base = v.level_splits[lo], base4 = base & ~3;
    const bool staged = n >= min(kTraceFew, hi - lv0);
    if (staged) {  // (what is read beyond `top` is within the array's last four)
      const int4 *from = reinterpret_cast<const int4 *>(all_pred + base4);
      const int32_t lowest = base - base4, to_here = s_begin - base4;
      auto offset = [&](int32_t p) {
        const int32_t j = p + to_here;
        return p >= 0 && (uint32_t)(j - lowest) < (uint32_t)(top - base) ? 4 * j : kOut;
      };
#pragma unroll 4
      for (int32_t k = tid; k < (top - base4 + 3) >> 2; k += 512) {
        const int4 p = from[k];
        pred4[k] = make_int4(offset(p.x), offset(p.y), offset(p.z), offset(p.w));
      }
    }
    __syncthreads();
    if (tid == 0) {
      const int32_t limit = min(kTraceLayers, v.max_layers - len);
      int32_t k = 0;
      if (staged && cur >= base && cur < top) {
        int32_t c = 4 * (cur - base4);
        while (c != kOut && k < limit) {
#pragma unroll
          for (int u = 0; u < kTraceSteps; ++u) {
            path[k + u] = c;
            c = *reinterpret_cast<const int32_t *>(pred + c);
          }
          k += kTraceSteps;
        }
        if (c == kOut) {  // to the last state of the run, and on from it
          while (path[k - 1] == kOut) --k;
          const int32_t last = base4 + (path[k - 1] >> 2), from = all_pred[last];
          if (from < 0) --k;  // the path begins at this state
          cur = from < 0 ? -1 - last : s_begin + from;
        }
        if (k > limit || c != kOut) {
          cur = k > limit ? base4 + (path[limit] >> 2) : base4 + (c >> 2);
          k = limit;
        }
      } else if (!staged) {
        while (cur >= base && cur < top && k < limit) {
          const int32_t from = all_pred[cur];
          if (from < 0) {
            cur = -1 - cur;
            break;
          }
          path[k++] = 4 * (cur - base4);
          cur = s_begin + from;
        }
      }
      cur_sh = cur;
      steps_sh = k;
    }
    __syncthreads();
    for (int32_t k = tid; k < steps_sh; k += blockDim.x)
      out[len + k] = entering[base4 + (path[k] >> 2)];
    cur = cur_sh;
    len += steps_sh;
    alive = cur >= 0;
    hi = lo;
    __syncthreads();
  }
  // (a path ends where no arc enters: only at the start state is it complete)
  if (tid == 0) lengths[i] = cur == -1 - s_begin && s_end > s_begin ? len : 0;
}

// States of a run: no more than an FSA can have, and where there are more FSAs than SMs no more
// than lets two, three or four CTAs (its threads allow no more) share one.  512 alignments of up to
// 100 layers: 14.0 us with the most for all, 5.4 so; 600 of 300: 28.3 and 9.9; 2000 of 50: 38.7 and
// 13.1; 32 of 800: 17.2 both.
static int32_t TraceRoom(const k2b200_fsa_view *v) {
  const int32_t ctas = std::max(1, std::min(4, CeilDiv(v->num_fsas, NumSms())));
  int64_t states = v->num_states;
  if (v->max_layer_states > 0)
    states = std::min(states, (int64_t)v->max_layers * v->max_layer_states);
  // (a run begins at a multiple of four states)
  return (int32_t)std::min<int64_t>((states + 3 + 3) & ~(int64_t)3, kTraceStates / ctas);
}

// The paths as linear FSAs: arcs (states renumbered, labels and scores kept), the lattice arc
// of each, the row splits.  One CTA per FSA.
__global__ void __launch_bounds__(128)
WritePaths(const Arc *__restrict__ arcs, const int32_t *__restrict__ traced,
           const int32_t *__restrict__ lengths, int32_t num_fsas, int32_t max_layers,
           int32_t *__restrict__ path_splits, int32_t *__restrict__ row_splits1,
           int32_t *__restrict__ row_splits2, Arc *__restrict__ out, int32_t *__restrict__ best) {
  __shared__ int32_t arcs_before, paths_before;
  const int32_t i = blockIdx.x;
  if (threadIdx.x == 0) arcs_before = paths_before = 0;
  __syncthreads();
  int32_t na = 0, np = 0;
  for (int32_t j = threadIdx.x; j < i; j += blockDim.x) {
    na += lengths[j];
    np += lengths[j] > 0;
  }
  if (na) {
    atomicAdd(&arcs_before, na);
    atomicAdd(&paths_before, np);
  }
  __syncthreads();
  const int32_t p0 = arcs_before, s0 = p0 + paths_before, len = lengths[i];
  for (int32_t k = threadIdx.x; k < len; k += blockDim.x) {
    const int32_t a = traced[(int64_t)i * max_layers + (len - 1 - k)];
    Arc arc = arcs[a];
    arc.src = k;
    arc.dest = k + 1;
    out[p0 + k] = arc;
    best[p0 + k] = a;
    row_splits2[s0 + k] = p0 + k;
  }
  if (threadIdx.x == 0) {
    path_splits[i] = p0;
    row_splits1[i] = s0;
    if (len > 0) row_splits2[s0 + len] = p0 + len;
    if (i == num_fsas - 1) {
      const int32_t s1 = s0 + (len > 0 ? len + 1 : 0);
      path_splits[num_fsas] = p0 + len;
      row_splits1[num_fsas] = s1;
      row_splits2[s1] = p0 + len;
    }
  }
}

constexpr int32_t kAllProps = 0x1FF;

__global__ void PropsInit(int32_t *props, int32_t n_plus_one, char *reach, int64_t nreach) {
  int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n_plus_one) props[k] = kAllProps;
  if (k < nreach) reach[k] = 0;
}

__global__ void PropsArcs(const int32_t *__restrict__ row_splits1,
                          const int32_t *__restrict__ row_ids1,
                          const int32_t *__restrict__ row_splits2,
                          const int32_t *__restrict__ row_ids2, const Arc *__restrict__ arcs,
                          int32_t num_states, int32_t num_arcs, int32_t *props, char *reach) {
  int32_t a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= num_arcs) return;
  Arc arc = arcs[a];
  const int32_t idx01 = row_ids2[a], idx2 = a - row_splits2[idx01], idx0 = row_ids1[idx01],
                idx0x = row_splits1[idx0], idx0x_next = row_splits1[idx0 + 1],
                idx1 = idx01 - idx0x, idx0xx = row_splits2[idx0x], n = idx0x_next - idx0x;
  int32_t neg = 0;
  if (arc.src != idx1) neg |= 0x01;
  if (arc.dest <= arc.src) {
    neg |= 0x08;
    if (arc.dest < arc.src) neg |= 0x04;
  }
  if (arc.label == 0) neg |= 0x40;
  if (arc.label < 0) {
    if (arc.label != -1) neg |= 0x01;
    else if (arc.dest != n - 1) neg |= 0x01;
  }
  if (arc.label != -1 && arc.dest == n - 1) neg |= 0x01;
  if (arc.dest < 0 || arc.dest >= n) neg |= 0x01;
  else if (arc.dest != arc.src) reach[idx0x + arc.dest] = 1;
  if (idx0xx == a) {
    reach[idx0x] = 1;
    reach[num_states + idx0x_next - 1] = 1;
  }
  if (arc.dest != arc.src) reach[num_states + idx01] = 1;
  if (idx2 != 0) {
    Arc p = arcs[a - 1];
    if ((uint32_t)arc.label <= (uint32_t)p.label) neg |= 0x20;
    if ((uint32_t)arc.label < (uint32_t)p.label) neg |= 0x10;
    if (arc.label == p.label && arc.dest < p.dest) neg |= 0x10;
  }
  if (neg) atomicAnd(&props[idx0], ~neg);
}

__global__ void PropsStates(const int32_t *__restrict__ row_ids1, int32_t num_states,
                            const char *__restrict__ reach, int32_t *props) {
  int32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= num_states) return;
  int32_t neg = (reach[s] ? 0 : 0x80) | (reach[num_states + s] ? 0 : 0x100);
  if (neg) atomicAnd(&props[row_ids1[s]], ~neg);
}

__global__ void PropsFinish(const int32_t *__restrict__ row_splits1,
                            const int32_t *__restrict__ row_splits2, int32_t num_fsas,
                            int32_t *props) {
  int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= num_fsas) return;
  if (row_splits2[row_splits1[i]] == row_splits2[row_splits1[i + 1]]) atomicAnd(&props[i], ~0x02);
  __threadfence();
  atomicAnd(&props[num_fsas], props[i] & kAllProps);
}

}  // namespace k2b

using namespace k2b;

#define STREAM(s) reinterpret_cast<cudaStream_t>(s)

template <typename Real>
static int32_t LaunchGeneric(const k2b200_fsa_view *v, int32_t log_semiring, Real *fwd, Real *bwd,
                             int32_t *entering, const int32_t *run_if, cudaStream_t stream) {
  int32_t ndir = (fwd != nullptr) + (bwd != nullptr), dir_base = fwd ? 0 : 1;
  for (int32_t first = 0; first < v->num_fsas; first += 65535) {
    int32_t n = v->num_fsas - first < 65535 ? v->num_fsas - first : 65535;
    dim3 grid(ndir, n);
    if (log_semiring)
      { LayeredScores<Real, true><<<grid, 256, 0, stream>>>(*v, fwd, bwd, nullptr, dir_base,
                                                            first, run_if); NoteLaunch(); }
    else
      { LayeredScores<Real, false><<<grid, 256, 0, stream>>>(*v, fwd, bwd, entering, dir_base,
                                                             first, run_if); NoteLaunch(); }
  }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

template <typename Real>
static int32_t LaunchScores(const k2b200_fsa_view *v, int32_t log_semiring, Real *fwd, Real *bwd,
                            int32_t *entering, void *scratch, size_t scratch_bytes,
                            cudaStream_t stream) {
  int32_t ndir = (fwd != nullptr) + (bwd != nullptr);
  if (ndir == 0 || v->num_fsas == 0) return kOk;
  PhaseTimer timer(kPhaseScores, stream);
  bool launched = false;
  const int32_t *redo_if = nullptr;
  K2B_FORWARD(LaunchLayerScores<Real>(v, log_semiring, fwd, bwd, entering, scratch, scratch_bytes,
                                      stream, &launched, &redo_if));
  if (launched && redo_if == nullptr) return kOk;
  K2B_REQUIRE(fwd == nullptr || v->num_arcs == 0 || (v->in_splits && v->in_arcs && v->row_ids2),
              "forward scores need the incoming-arc index and row_ids2");
  // if the layer bounds were violated, or values out of range, everything is redone
  if (launched)
    return LaunchGeneric<Real>(v, log_semiring, fwd, bwd, entering, redo_if, stream);
  return LaunchGeneric<Real>(v, log_semiring, fwd, bwd, entering, nullptr, stream);
}

extern "C" {

const char *k2b200_last_error(void) { return LastError(); }
int32_t k2b200_abi_version(void) { return 5; }
int64_t k2b200_kernel_launch_count(void) { return LaunchCount(); }
void k2b200_profile_enable(int32_t on) { SetProfiling(on != 0); }
const char *k2b200_profile_kernel(int32_t phase) { return PhaseKernel(phase); }
double k2b200_profile_read_ms(int32_t phase, int64_t *intervals) {
  long long n = 0;
  double ms = (phase >= 0 && phase < kNumPhases) ? ReadPhase(phase, &n) : 0.0;
  if (intervals) *intervals = n;
  return ms;
}

int32_t k2b200_row_splits_to_row_ids(const int32_t *row_splits, int32_t num_rows,
                                     int32_t *row_ids, int32_t num_elems, void *stream) {
  return RowSplitsToRowIds(row_splits, num_rows, row_ids, num_elems, STREAM(stream));
}

int32_t k2b200_upload_i32(const int32_t *host_values, int64_t n, int32_t *device_out,
                          void *stream) {
  K2B_REQUIRE(n >= 0, "negative length");
  K2B_REQUIRE(n == 0 || (host_values != nullptr && device_out != nullptr), "NULL pointer");
  return UploadInts(host_values, n, device_out, STREAM(stream));
}

size_t k2b200_exclusive_sum_tmp_bytes(int64_t n) { return sizeof(int32_t) * ScanTmpInts(n); }
int32_t k2b200_exclusive_sum(const int32_t *in, int32_t *out, int64_t n, void *tmp,
                             void *stream) {
  return ExclusiveSum(in, out, n, reinterpret_cast<int32_t *>(tmp), STREAM(stream));
}

int64_t k2b200_exclusive_sum_static_max_len(void) { return ExclusiveSumStaticMaxLen(); }
int32_t k2b200_exclusive_sum_static(const int32_t *in, int32_t *out, int64_t n, void *stream) {
  K2B_REQUIRE(n == 0 || (in != nullptr && out != nullptr), "NULL pointer");
  K2B_REQUIRE(out != nullptr, "NULL output pointer");
  return ExclusiveSumStatic(in, out, n, STREAM(stream));
}

size_t k2b200_fsa_incoming_tmp_bytes(int32_t num_states, int32_t num_arcs) {
  return IncomingTmpBytes(num_states, num_arcs);
}
int32_t k2b200_fsa_incoming(const int32_t *row_splits1, const int32_t *row_ids1,
                            const int32_t *row_ids2, const void *arcs, int32_t num_fsas,
                            int32_t num_states, int32_t num_arcs, int32_t *in_splits,
                            int32_t *in_arcs, int32_t *in_src, float *in_score, void *tmp,
                            void *stream) {
  K2B_REQUIRE(num_fsas >= 0 && num_states >= 0 && num_arcs >= 0, "negative size");
  K2B_REQUIRE(in_splits && tmp, "NULL pointer");
  PhaseTimer timer(kPhaseIncoming, STREAM(stream));
  return BuildIncoming(row_splits1, row_ids1, row_ids2, reinterpret_cast<const Arc *>(arcs),
                       num_fsas, num_states, num_arcs, in_splits, in_arcs, in_src, in_score, tmp,
                       STREAM(stream));
}

int32_t k2b200_fsa_incoming_layers(const k2b200_fsa_view *v, int32_t *in_splits,
                                   int32_t *in_arcs, int32_t *in_src, float *in_score,
                                   int32_t *done, void *stream) {
  K2B_REQUIRE(v && in_splits && in_arcs && in_src && in_score && done, "NULL pointer");
  K2B_REQUIRE(v->row_splits1 && v->row_ids1 && v->row_splits2 && v->level_offsets &&
                  v->level_splits,
              "NULL pointer in the FsaVec view");
  PhaseTimer timer(kPhaseIncoming, STREAM(stream));
  bool ok = false;
  K2B_FORWARD(BuildLayerIncoming(v, in_splits, in_arcs, in_src, in_score, STREAM(stream), &ok));
  *done = ok ? 1 : 0;
  return kOk;
}

size_t k2b200_fsa_scores_scratch_bytes(const k2b200_fsa_view *v) {
  // (two directions need at least what one does)
  return v ? std::max(LayerScratchBytes(v, 1), LayerScratchBytes(v, 2)) : 0;
}
size_t k2b200_fsa_scores_dir_scratch_bytes(const k2b200_fsa_view *v, int32_t directions,
                                           int32_t *needs_incoming) {
  if (v == nullptr) return 0;
  if (needs_incoming) *needs_incoming = LayerScoresNeedIncoming(v, directions) ? 1 : 0;
  return LayerScratchBytes(v, directions);
}

int32_t k2b200_fsa_scores(const k2b200_fsa_view *v, int32_t log_semiring, int32_t use_double,
                          void *forward, void *backward, int32_t *entering_arcs, void *scratch,
                          size_t scratch_bytes, void *stream) {
  K2B_REQUIRE(v != nullptr, "NULL view");
  K2B_REQUIRE(v->row_splits1 && v->row_splits2 && v->level_offsets && v->level_splits,
              "NULL pointer in the FsaVec view");
  if (use_double)
    return LaunchScores<double>(v, log_semiring, reinterpret_cast<double *>(forward),
                                reinterpret_cast<double *>(backward), entering_arcs, scratch,
                                scratch_bytes, STREAM(stream));
  return LaunchScores<float>(v, log_semiring, reinterpret_cast<float *>(forward),
                             reinterpret_cast<float *>(backward), entering_arcs, scratch,
                             scratch_bytes, STREAM(stream));
}

int32_t k2b200_fsa_tot_scores(const int32_t *row_splits1, int32_t num_fsas, int32_t use_double,
                              const void *forward, void *tot_scores, void *stream) {
  if (num_fsas <= 0) return kOk;
  if (use_double)
    { TotScores<double><<<CeilDiv(num_fsas, 128), 128, 0, STREAM(stream)>>>(
        row_splits1, num_fsas, reinterpret_cast<const double *>(forward),
        reinterpret_cast<double *>(tot_scores)); NoteLaunch(); }
  else
    { TotScores<float><<<CeilDiv(num_fsas, 128), 128, 0, STREAM(stream)>>>(
        row_splits1, num_fsas, reinterpret_cast<const float *>(forward),
        reinterpret_cast<float *>(tot_scores)); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

int32_t k2b200_fsa_arc_post(const int32_t *row_splits1, const int32_t *row_ids1,
                            const int32_t *row_ids2, const void *arcs, int32_t num_fsas,
                            int32_t num_arcs, int32_t use_double, const void *forward,
                            const void *backward, void *arc_post, void *stream) {
  PhaseTimer timer(kPhasePost, STREAM(stream));
  (void)num_fsas;
  if (num_arcs <= 0) return kOk;
  const Arc *a = reinterpret_cast<const Arc *>(arcs);
  if (use_double)
    { ArcPost<double><<<CeilDiv(num_arcs, 256), 256, 0, STREAM(stream)>>>(
        row_splits1, row_ids1, row_ids2, a, num_arcs, reinterpret_cast<const double *>(forward),
        reinterpret_cast<const double *>(backward), reinterpret_cast<double *>(arc_post)); NoteLaunch(); }
  else
    { ArcPost<float><<<CeilDiv(num_arcs, 256), 256, 0, STREAM(stream)>>>(
        row_splits1, row_ids1, row_ids2, a, num_arcs, reinterpret_cast<const float *>(forward),
        reinterpret_cast<const float *>(backward), reinterpret_cast<float *>(arc_post)); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

int32_t k2b200_tot_scores_log_backward(const int32_t *row_ids1, const int32_t *row_ids2,
                                       int32_t num_arcs, int32_t use_double,
                                       const void *arc_post, const void *tot_scores_grad,
                                       int64_t grad_stride, float *arc_grad, void *stream) {
  PhaseTimer timer(kPhasePost, STREAM(stream));
  if (num_arcs <= 0) return kOk;
  if (use_double)
    { LogBackward<double><<<CeilDiv(num_arcs, 256), 256, 0, STREAM(stream)>>>(
        row_ids1, row_ids2, num_arcs, reinterpret_cast<const double *>(arc_post),
        reinterpret_cast<const double *>(tot_scores_grad), grad_stride, arc_grad); NoteLaunch(); }
  else
    { LogBackward<float><<<CeilDiv(num_arcs, 256), 256, 0, STREAM(stream)>>>(
        row_ids1, row_ids2, num_arcs, reinterpret_cast<const float *>(arc_post),
        reinterpret_cast<const float *>(tot_scores_grad), grad_stride, arc_grad); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

int32_t k2b200_tot_scores_log_backward_scores(const int32_t *row_splits1, const int32_t *row_ids1,
                                              const int32_t *row_ids2, const void *arcs,
                                              int32_t num_arcs, int32_t use_double,
                                              const void *forward, const void *backward,
                                              const void *tot_scores_grad, int64_t grad_stride,
                                              float *arc_grad, void *stream) {
  PhaseTimer timer(kPhasePost, STREAM(stream));
  if (num_arcs <= 0) return kOk;
  const Arc *a = reinterpret_cast<const Arc *>(arcs);
  if (use_double)
    { LogBackwardScores<double><<<CeilDiv(num_arcs, 256), 256, 0, STREAM(stream)>>>(
        row_splits1, row_ids1, row_ids2, a, num_arcs, reinterpret_cast<const double *>(forward),
        reinterpret_cast<const double *>(backward),
        reinterpret_cast<const double *>(tot_scores_grad), grad_stride, arc_grad); NoteLaunch(); }
  else
    { LogBackwardScores<float><<<CeilDiv(num_arcs, 256), 256, 0, STREAM(stream)>>>(
        row_splits1, row_ids1, row_ids2, a, num_arcs, reinterpret_cast<const float *>(forward),
        reinterpret_cast<const float *>(backward),
        reinterpret_cast<const float *>(tot_scores_grad), grad_stride, arc_grad); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

int32_t k2b200_tot_scores_tropical_backward(const int32_t *row_ids1, const int32_t *row_ids2,
                                            int32_t num_arcs, const int32_t *best_arcs,
                                            int32_t num_best_arcs, int32_t use_double,
                                            const void *tot_scores_grad, int64_t grad_stride,
                                            float *arc_grad, void *stream) {
  if (num_arcs <= 0) return kOk;
  K2B_CUDA_OK(cudaMemsetAsync(arc_grad, 0, sizeof(float) * (size_t)num_arcs, STREAM(stream)));
  if (num_best_arcs <= 0) return kOk;
  if (use_double)
    { TropicalBackward<double><<<CeilDiv(num_best_arcs, 256), 256, 0, STREAM(stream)>>>(
        row_ids1, row_ids2, best_arcs, num_best_arcs,
        reinterpret_cast<const double *>(tot_scores_grad), grad_stride, arc_grad); NoteLaunch(); }
  else
    { TropicalBackward<float><<<CeilDiv(num_best_arcs, 256), 256, 0, STREAM(stream)>>>(
        row_ids1, row_ids2, best_arcs, num_best_arcs,
        reinterpret_cast<const float *>(tot_scores_grad), grad_stride, arc_grad); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

int32_t k2b200_index_add(const int32_t *index, const float *value, int32_t n, float *in_out,
                         int64_t in_out_size, void *stream) {
  PhaseTimer timer(kPhasePost, STREAM(stream));
  if (n <= 0) return kOk;
  { IndexAdd<<<CeilDiv(n, 256), 256, 0, STREAM(stream)>>>(index, value, n, in_out, in_out_size); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

int32_t k2b200_index_select_i32(const int32_t *src, int64_t src_size, const int32_t *index,
                                int32_t n, int32_t *out, void *stream) {
  if (n <= 0) return kOk;
  { IndexSelectI32<<<CeilDiv(n, 256), 256, 0, STREAM(stream)>>>(src, src_size, index, n, out); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

size_t k2b200_shortest_path_tmp_bytes(int32_t num_fsas) {
  return AlignUp(sizeof(int32_t) * ((size_t)num_fsas + 1)) +
         AlignUp(sizeof(int32_t) * ScanTmpInts(num_fsas));
}

int32_t k2b200_shortest_path(const int32_t *row_splits1, const void *arcs,
                             const int32_t *entering_arcs, int32_t num_fsas,
                             int32_t *path_splits, int32_t *best_arcs, void *tmp, void *stream) {
  if (num_fsas <= 0) return kOk;
  K2B_REQUIRE(row_splits1 && entering_arcs && path_splits && best_arcs && tmp, "NULL pointer");
  char *p = reinterpret_cast<char *>(tmp);
  int32_t *lengths = reinterpret_cast<int32_t *>(p);
  int32_t *scan_tmp =
      reinterpret_cast<int32_t *>(p + AlignUp(sizeof(int32_t) * ((size_t)num_fsas + 1)));
  const Arc *a = reinterpret_cast<const Arc *>(arcs);
  { PathLengths<<<CeilDiv(num_fsas, 64), 64, 0, STREAM(stream)>>>(row_splits1, a, entering_arcs,
                                                               num_fsas, lengths); NoteLaunch(); }
  K2B_FORWARD(ExclusiveSum(lengths, path_splits, num_fsas, scan_tmp, STREAM(stream)));
  { PathFill<<<CeilDiv(num_fsas, 64), 64, 0, STREAM(stream)>>>(row_splits1, a, entering_arcs,
                                                            num_fsas, path_splits, best_arcs); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

size_t k2b200_best_paths_tmp_bytes(const k2b200_fsa_view *v) {
  if (v == nullptr) return 0;
  return AlignUp(sizeof(int32_t) * ((size_t)v->num_fsas + 1)) +
         AlignUp(sizeof(int32_t) * (size_t)v->num_fsas * (size_t)v->max_layers) +
         AlignUp(16 * ((size_t)std::max(v->num_states, 0) / 4 + 1) + 12);
}

int32_t k2b200_best_paths(const k2b200_fsa_view *v, const int32_t *entering_arcs,
                          int32_t *path_splits, int32_t *row_splits1, int32_t *row_splits2,
                          void *arcs, int32_t *best_arcs, void *tmp, void *stream) {
  K2B_REQUIRE(v && entering_arcs && path_splits && row_splits1 && row_splits2 && arcs &&
                  best_arcs && tmp,
              "NULL pointer");
  K2B_REQUIRE(v->row_splits1 && v->level_offsets && v->level_splits && v->max_layers > 0,
              "k2b200_best_paths needs a layered view");
  if (v->num_fsas <= 0) return kOk;
  int32_t *lengths = reinterpret_cast<int32_t *>(tmp);
  int32_t *traced = reinterpret_cast<int32_t *>(
      reinterpret_cast<char *>(tmp) + AlignUp(sizeof(int32_t) * ((size_t)v->num_fsas + 1)));
  // (read 16 bytes at a time, from a multiple of 16 bytes on, wherever `tmp` lies)
  int32_t *pred = reinterpret_cast<int32_t *>(
      (reinterpret_cast<uintptr_t>(traced) +
       AlignUp(sizeof(int32_t) * (size_t)v->num_fsas * (size_t)v->max_layers) + 15) &
      ~(uintptr_t)15);
  if (v->num_states > 0)
    { Predecessors<<<CeilDiv(v->num_states, 256), 256, 0, STREAM(stream)>>>(
        reinterpret_cast<const Arc *>(v->arcs), entering_arcs, v->num_states, pred); NoteLaunch(); }
  const int32_t room = TraceRoom(v);
  const int smem = (int)sizeof(int32_t) * (room + 4);
  auto trace = room == kTraceStates ? TraceLayers<kTraceStates> : TraceLayers<0>;
  K2B_CUDA_OK(cudaFuncSetAttribute(trace, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(int32_t) * (kTraceStates + 4)));
  { trace<<<v->num_fsas, 512, smem, STREAM(stream)>>>(*v, entering_arcs, pred, room, traced,
                                                            lengths);
    NoteLaunch(); }
  { WritePaths<<<v->num_fsas, 128, 0, STREAM(stream)>>>(
      reinterpret_cast<const Arc *>(v->arcs), traced, lengths, v->num_fsas, v->max_layers,
      path_splits, row_splits1, row_splits2, reinterpret_cast<Arc *>(arcs), best_arcs);
    NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

size_t k2b200_fsa_properties_tmp_bytes(int32_t num_fsas, int32_t num_states) {
  (void)num_fsas;
  return AlignUp(2 * (size_t)num_states + 2);
}

int32_t k2b200_fsa_properties(const int32_t *row_splits1, const int32_t *row_ids1,
                              const int32_t *row_splits2, const int32_t *row_ids2,
                              const void *arcs, int32_t num_fsas, int32_t num_states,
                              int32_t num_arcs, int32_t *properties, void *tmp, void *stream) {
  K2B_REQUIRE(properties && tmp, "NULL pointer");
  char *reach = reinterpret_cast<char *>(tmp);
  int64_t nreach = 2 * (int64_t)num_states;
  int64_t n0 = nreach > num_fsas + 1 ? nreach : num_fsas + 1;
  { PropsInit<<<CeilDiv(n0, 256), 256, 0, STREAM(stream)>>>(properties, num_fsas + 1, reach, nreach); NoteLaunch(); }
  if (num_arcs > 0)
    { PropsArcs<<<CeilDiv(num_arcs, 256), 256, 0, STREAM(stream)>>>(
        row_splits1, row_ids1, row_splits2, row_ids2, reinterpret_cast<const Arc *>(arcs),
        num_states, num_arcs, properties, reach); NoteLaunch(); }
  if (num_states > 0)
    { PropsStates<<<CeilDiv(num_states, 256), 256, 0, STREAM(stream)>>>(row_ids1, num_states, reach,
                                                                     properties); NoteLaunch(); }
  if (num_fsas > 0)
    { PropsFinish<<<CeilDiv(num_fsas, 128), 128, 0, STREAM(stream)>>>(row_splits1, row_splits2,
                                                                   num_fsas, properties); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

}  // extern "C"
