// Kernels in which a warp walks the edges of its nodes on its own (tp_walk.cu), as the fused layer's entry points use them.
#pragma once

#include "common.cuh"

namespace eqt {

struct WalkArgs {
  const float* feat;        // (rows, DF, C), 16-byte aligned
  const int64_t* fidx;      // (E) feature row of each edge, or NULL (= e)
  const float* y;           // (Ey, DY); not read by the adjoint
  const int64_t* yidx;      // (E) row of y (of grad_y: the adjoint) of each edge, or NULL (= e)
  const int64_t* ptr;       // (N + 1) CSR of edges per node, or NULL (one edge per node)
  const float* scale;       // (T)
  const float* w;           // (P, C) weights: rows are mixed channel by channel instead of being written / read
  const float* g;           // adjoint: (N, R, C), with w (N, K, C)
  const float* x;           // (N, K, C) operand of the weight gradient, or NULL
  float* out;               // segment sum: (N, R, C), with w (N, K, C); adjoint: (Ey, DY)
  float* gw;                // (P, C) with x
  float* scratch;           // with x: walk_scratch_floats() of them
  int64_t n_out, n_edges;
  int C;
};

// Whether the kernels take a structure (key of its table, or of its table and weight step where w is given), and whether a table
// has the sizes of the structure that it names: the kernels read rows and entries by the structure's own.
bool walk_supported(uint64_t key, bool with_weights, bool adjoint, int channels);
bool walk_sizes(uint64_t key, bool with_weights, int entries, int rows, int d_feat, int d_y);
int64_t walk_scratch_floats(uint64_t mix_key, int64_t n_out, int channels);    // -1: not supported
int walk_segment_sum(uint64_t key, const WalkArgs& a, cudaStream_t s);
int walk_inner(uint64_t key, const WalkArgs& a, cudaStream_t s);

}  // namespace eqt
