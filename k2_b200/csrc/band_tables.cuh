// Per-state tables of band graphs (band_loss.cu), which ctc_graph.cu writes along with the graphs.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace k2b {

constexpr int32_t kNoLabel = INT32_MIN;

// Per state (idx01): the arcs entering it.  w[d] = score of the arc from state s - d
// (-inf: no such arc); label = their common label (kNoLabel: no entering arc).
struct __align__(16) BandState {
  float w[3];
  int32_t label;
};
// Per (state, d): exp(w[d]) = f * 2^k and the arc's index (idx012), -1 if absent.
struct __align__(16) BandArc {
  double f;
  int32_t k;
  int32_t arc;
};

}  // namespace k2b
