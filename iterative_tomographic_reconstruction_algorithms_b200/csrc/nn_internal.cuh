// Internal declarations of libtomo_nn (the learned warm start's kernels).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/tomo_nn.h"

namespace tomo_nn {

constexpr int NN_OK = TOMO_NN_OK;
constexpr int NN_EINVAL = TOMO_NN_EINVAL;
constexpr int NN_ECUDA = TOMO_NN_ECUDA;

struct GemmArgs {
  const __nv_bfloat16 *A = nullptr;  // A[m*lda + k]
  int lda = 0;
  const __nv_bfloat16 *B = nullptr;  // B[n*ldb + k]
  int ldb = 0;
  int M = 0, N = 0, K = 0;
  float *Cf = nullptr;               // FP32 output ...
  __nv_bfloat16 *Cb = nullptr;       // ... or BF16 output
  int ldc = 0;
  const float *bias = nullptr;
  int relu = 0;
  unsigned *status = nullptr;        // bit 0 set if an MMA wait gave up
  int spins = 1 << 22;               // polls of a pipeline wait before it gives up
};

int gemm_launch(const GemmArgs &g, cudaStream_t s);

// 3x3 convolution, stride 1, zero padding 1, NHWC (nn_conv.cu).
int conv_launch(const __nv_bfloat16 *X, int batch, int H, int W, int Cin, const __nv_bfloat16 *Wt, int Cout, float *Yf,
                __nv_bfloat16 *Yb, const float *bias, int relu, const __nv_bfloat16 *mask, unsigned *status, int spins,
                cudaStream_t s);

// BF16 tensor map of `rank` dimensions (innermost first; strides in bytes from
// the second on) whose boxes have rows of rb = 16, 32, 64 or 128 bytes, stored
// with the swizzle of that width (none for 16); elements outside are zero.
int make_tensor_map(void *map, const void *base, int rank, const unsigned long long *dim,
                    const unsigned long long *stride, const unsigned *box, int rb);

// Weight and bias gradients of a 3x3 (taps 9) or 1x1 (taps 1) convolution
// (nn_wgrad.cu); work holds wgrad_workspace(...) bytes.
size_t wgrad_workspace(int batch, int H, int W, int Cin, int Cout, int taps);
int wgrad_launch(const __nv_bfloat16 *X, const __nv_bfloat16 *dY, int batch, int H, int W, int Cin, int Cout, int taps,
                 float *dW, float *db, void *work, unsigned *status, int spins, cudaStream_t s);

}  // namespace tomo_nn
