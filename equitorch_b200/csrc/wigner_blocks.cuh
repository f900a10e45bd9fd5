// Float32 kernels for block-diagonal Wigner-D matrices (wigner_blocks.cu).  Each returns NOT_TAKEN where the
// irreps are outside what it handles; the general kernels of wigner.cu then run.
#pragma once

#include "common.cuh"

namespace eqt {

constexpr int NOT_TAKEN = -1;

int wigner_quads_forward(const eqt_wigner_table* t, const float* alpha, const float* beta, const float* gamma, float* d, int64_t n,
                         cudaStream_t st);
int wigner_quads_backward(const eqt_wigner_table* t, const float* alpha, const float* beta, const float* gamma, const float* grad_d,
                          float* ga, float* gb, float* gc, int64_t n, cudaStream_t st);

}  // namespace eqt
