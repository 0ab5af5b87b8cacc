// CTC graphs of a batch of transcripts, built on the GPU.
//
// Same graphs, arc for arc, as k2::CtcGraphs (k2/csrc/fsa_algo.cu:577-730): a
// transcript of L symbols gives 2L+2 states - state 2k the blank state in front of
// symbol k (2L the trailing one), 2k+1 the state of symbol k, 2L+1 the final state.
// The reference launches one lambda per state and per arc around two ExclusiveSums;
// here one kernel sizes the per-symbol arc blocks, one exclusive sum places them and
// one kernel writes arcs, aux_labels and both row_splits.
#include <cstring>

#include "../../include/k2b200.h"
#include "band_tables.cuh"
#include "common.cuh"
#include "prob_math.cuh"

namespace k2b {

// Arcs contributed by symbol position k: blank state (2) + symbol state (2 or 3).
__global__ void CtcCountArcs(const int32_t *__restrict__ sym_row_splits,
                             const int32_t *__restrict__ sym_row_ids,
                             const int32_t *__restrict__ symbols, int32_t tot,
                             int32_t modified, int32_t *__restrict__ per_sym) {
  int32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= tot) return;
  const int32_t i = sym_row_ids[k];
  const bool last = k + 1 == sym_row_splits[i + 1];
  const int32_t next = last ? -1 : symbols[k + 1];
  per_sym[k] = 4 + ((modified || symbols[k] != next) ? 1 : 0);
}

__global__ void CtcWriteArcs(const int32_t *__restrict__ sym_row_splits,
                             const int32_t *__restrict__ sym_row_ids,
                             const int32_t *__restrict__ symbols, int32_t num_seqs, int32_t tot,
                             int32_t modified, const int32_t *__restrict__ sym_arc_off,
                             int32_t *__restrict__ row_splits1, int32_t *__restrict__ row_splits2,
                             Arc *__restrict__ arcs, int32_t *__restrict__ aux) {
  int32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  auto put = [&](int32_t pos, int32_t src, int32_t dest, int32_t label, int32_t a) {
    Arc arc;
    arc.src = src;
    arc.dest = dest;
    arc.label = label;
    arc.score = 0.0f;
    arcs[pos] = arc;
    aux[pos] = a;
  };
  if (k < tot) {
    const int32_t i = sym_row_ids[k], s0 = sym_row_splits[i];
    const int32_t pos_in = k - s0;                  // position in its transcript
    const int32_t state0 = 2 * s0 + 2 * i;          // first state (idx01) of FSA i
    const int32_t blk = sym_arc_off[k] + 2 * i;     // 2 tail arcs per earlier FSA
    const bool last = k + 1 == sym_row_splits[i + 1];
    const int32_t sym = symbols[k], next = last ? -1 : symbols[k + 1];
    const int32_t sb = 2 * pos_in, ss = sb + 1;
    put(blk + 0, sb, sb, 0, 0);
    put(blk + 1, sb, ss, sym, sym);
    put(blk + 2, ss, ss + 1, 0, 0);
    put(blk + 3, ss, ss, sym, 0);
    if (modified || sym != next) put(blk + 4, ss, ss + 2, next, next);
    row_splits2[state0 + sb] = blk;
    row_splits2[state0 + ss] = blk + 2;
  }
  if (k < num_seqs) {  // the trailing blank state and the final state of FSA k
    const int32_t s0 = sym_row_splits[k], s1 = sym_row_splits[k + 1], L = s1 - s0;
    const int32_t state0 = 2 * s0 + 2 * k;
    const int32_t tail = sym_arc_off[s1] + 2 * k;   // sym_arc_off has tot + 1 entries
    put(tail, 2 * L, 2 * L, 0, 0);
    put(tail + 1, 2 * L, 2 * L + 1, -1, -1);
    row_splits1[k] = state0;
    row_splits2[state0 + 2 * L] = tail;
    row_splits2[state0 + 2 * L + 1] = tail + 2;
    if (k == num_seqs - 1) {
      row_splits1[num_seqs] = state0 + 2 * L + 2;
      row_splits2[state0 + 2 * L + 2] = tail + 2;
    }
  }
}

// The same graphs and their band tables (band_loss.cu) from host transcripts, one CTA per graph:
// the host knows the arcs of every graph (it sizes the outputs), so a CTA places its own by a
// scan over its symbols, and nothing but the symbols is read.  meta: first symbol of every
// graph [n + 1], first arc of every graph [n + 1], symbols.  (Seven launches and a pass over
// the finished graph for the tables took 30 us of a small training step.)
__device__ __forceinline__ void CtcGraphBody(const int32_t *__restrict__ meta, int32_t n,
                                             int32_t modified, int32_t *__restrict__ row_splits1,
                                             int32_t *__restrict__ row_splits2,
                                             Arc *__restrict__ arcs, int32_t *__restrict__ aux,
                                             BandState *__restrict__ tab,
                                             BandArc *__restrict__ tabf) {
  __shared__ int32_t warp_sum[4];
  const int32_t i = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t y0 = meta[i], L = meta[i + 1] - y0;
  const int32_t *symbols = meta + 2 * (n + 1) + y0;
  const int32_t state0 = 2 * y0 + 2 * i;
  int32_t run = meta[n + 1 + i];  // first arc of the chunk's first symbol
  auto put = [&](int32_t pos, int32_t src, int32_t dest, int32_t label, int32_t a) {
    Arc arc;
    arc.src = src;
    arc.dest = dest;
    arc.label = label;
    arc.score = 0.0f;
    arcs[pos] = arc;
    aux[pos] = a;
  };
  // entering arcs of state s by distance (-1: none), all with score 0
  auto table = [&](int32_t s, int32_t label, int32_t a0, int32_t a1, int32_t a2) {
    const int32_t a[3] = {a0, a1, a2};
    BandState st;
    st.label = label;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      st.w[d] = a[d] >= 0 ? 0.0f : -INFINITY;
      BandArc f;
      f.f = a[d] >= 0 ? 1.0 : 0.0;
      f.k = a[d] >= 0 ? 0 : kZeroExp;
      f.arc = a[d];
      tabf[(int64_t)(state0 + s) * 3 + d] = f;
    }
    tab[state0 + s] = st;
  };
  for (int32_t base = 0; base <= L; base += blockDim.x) {
    const int32_t k = base + threadIdx.x;  // k == L: the trailing blank and the final state
    const int32_t sym = k < L ? symbols[k] : -1, next = k + 1 < L ? symbols[k + 1] : -1,
                  prev = k > 0 && k <= L ? symbols[k - 1] : -1;
    const bool third = k + 1 == L || modified || sym != next;
    const int32_t cnt = k < L ? 4 + third : k == L ? 2 : 0;
    int32_t inc = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int32_t o = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += o;
    }
    if (lane == 31) warp_sum[warp] = inc;
    __syncthreads();
    int32_t total = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (u < warp) inc += warp_sum[u];
      total += warp_sum[u];
    }
    const int32_t blk = run + inc - cnt;
    __syncthreads();
    run += total;
    if (k > L) continue;
    // arcs of the symbol before: it has the third one unless it is repeated
    const bool prev_third = k > 0 && (k == L || modified || prev != sym);
    const int32_t from_prev = k > 0 ? blk - (4 + prev_third) : -1;
    const int32_t sb = 2 * k, ss = sb + 1;
    row_splits2[state0 + sb] = blk;
    row_splits2[state0 + ss] = blk + 2;
    put(blk, sb, sb, 0, 0);
    table(sb, 0, blk, k > 0 ? from_prev + 2 : -1, -1);
    if (k < L) {
      put(blk + 1, sb, ss, sym, sym);
      put(blk + 2, ss, ss + 1, 0, 0);
      put(blk + 3, ss, ss, sym, 0);
      if (third) put(blk + 4, ss, ss + 2, next, next);
      table(ss, sym, blk + 3, blk + 1, prev_third ? from_prev + 4 : -1);
    } else {
      put(blk + 1, sb, ss, -1, -1);
      table(ss, -1, -1, blk + 1, prev_third ? from_prev + 4 : -1);
      row_splits1[i] = state0;
      if (i == n - 1) {
        row_splits1[n] = state0 + 2 * L + 2;
        row_splits2[state0 + 2 * L + 2] = blk + 2;
      }
    }
  }
}

constexpr int kCtcParamInts = 960;
__global__ void __launch_bounds__(128)
CtcGraphs(const int32_t *__restrict__ meta, int32_t n, int32_t modified, int32_t *row_splits1,
          int32_t *row_splits2, Arc *arcs, int32_t *aux, BandState *tab, BandArc *tabf) {
  CtcGraphBody(meta, n, modified, row_splits1, row_splits2, arcs, aux, tab, tabf);
}
__global__ void __launch_bounds__(128)
CtcGraphsSmall(const __grid_constant__ IntChunk<kCtcParamInts> meta, int32_t n, int32_t modified,
               int32_t *row_splits1, int32_t *row_splits2, Arc *arcs, int32_t *aux, BandState *tab,
               BandArc *tabf) {
  CtcGraphBody(meta.v, n, modified, row_splits1, row_splits2, arcs, aux, tab, tabf);
}

}  // namespace k2b

using namespace k2b;

extern "C" {

size_t k2b200_ctc_graph_tmp_bytes(int32_t num_symbols) {
  return AlignUp(sizeof(int32_t) * ((size_t)num_symbols + 1)) +
         AlignUp(sizeof(int32_t) * ((size_t)num_symbols + 1)) +
         AlignUp(sizeof(int32_t) * ScanTmpInts(num_symbols));
}

int32_t k2b200_ctc_graph(const int32_t *sym_row_splits, const int32_t *symbols, int32_t num_seqs,
                         int32_t num_symbols, int32_t modified, int32_t *row_splits1,
                         int32_t *row_splits2, void *arcs, int32_t *aux_labels, void *tmp,
                         void *stream_v) {
  K2B_REQUIRE(num_seqs > 0 && num_symbols >= 0, "need at least one transcript");
  K2B_REQUIRE(sym_row_splits && row_splits1 && row_splits2 && arcs && aux_labels && tmp,
              "NULL pointer");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  char *p = reinterpret_cast<char *>(tmp);
  int32_t *sym_row_ids = reinterpret_cast<int32_t *>(p);
  p += AlignUp(sizeof(int32_t) * ((size_t)num_symbols + 1));
  int32_t *per_sym = reinterpret_cast<int32_t *>(p);
  p += AlignUp(sizeof(int32_t) * ((size_t)num_symbols + 1));
  int32_t *scan_tmp = reinterpret_cast<int32_t *>(p);
  K2B_FORWARD(RowSplitsToRowIds(sym_row_splits, num_seqs, sym_row_ids, num_symbols, stream));
  if (num_symbols > 0)
    { CtcCountArcs<<<CeilDiv(num_symbols, 256), 256, 0, stream>>>(
        sym_row_splits, sym_row_ids, symbols, num_symbols, modified, per_sym); NoteLaunch(); }
  K2B_FORWARD(ExclusiveSum(per_sym, per_sym, num_symbols, scan_tmp, stream));
  int32_t n = num_symbols > num_seqs ? num_symbols : num_seqs;
  { CtcWriteArcs<<<CeilDiv(n, 256), 256, 0, stream>>>(
      sym_row_splits, sym_row_ids, symbols, num_seqs, num_symbols, modified, per_sym, row_splits1,
      row_splits2, reinterpret_cast<Arc *>(arcs), aux_labels); NoteLaunch(); }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

int32_t k2b200_ctc_graph_host(const int32_t *h_meta, int32_t num_seqs, int32_t num_symbols,
                              int32_t modified, int32_t *row_splits1, int32_t *row_splits2,
                              void *arcs, int32_t *aux_labels, void *band_states, void *band_arcs,
                              int32_t *meta_tmp, void *stream_v) {
  K2B_REQUIRE(num_seqs > 0 && num_symbols >= 0, "need at least one transcript");
  K2B_REQUIRE(h_meta && row_splits1 && row_splits2 && arcs && aux_labels && band_states &&
                  band_arcs && meta_tmp,
              "NULL pointer");
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  const int64_t ints = 2 * ((int64_t)num_seqs + 1) + num_symbols;
  Arc *out = reinterpret_cast<Arc *>(arcs);
  BandState *tab = reinterpret_cast<BandState *>(band_states);
  BandArc *tabf = reinterpret_cast<BandArc *>(band_arcs);
  if (ints <= kCtcParamInts) {  // short batches travel with the launch
    IntChunk<kCtcParamInts> c;
    memcpy(c.v, h_meta, sizeof(int32_t) * (size_t)ints);
    { CtcGraphsSmall<<<num_seqs, 128, 0, stream>>>(c, num_seqs, modified, row_splits1, row_splits2,
                                                 out, aux_labels, tab, tabf); NoteLaunch(); }
  } else {
    K2B_FORWARD(UploadInts(h_meta, ints, meta_tmp, stream));
    { CtcGraphs<<<num_seqs, 128, 0, stream>>>(meta_tmp, num_seqs, modified, row_splits1,
                                              row_splits2, out, aux_labels, tab, tabf);
      NoteLaunch(); }
  }
  K2B_CUDA_OK(cudaGetLastError());
  return kOk;
}

}  // extern "C"
