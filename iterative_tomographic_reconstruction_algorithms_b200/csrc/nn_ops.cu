// libtomo_nn: the C ABI of include/tomo_nn.h and the small kernels around the
// tensor-core ones (nn_gemm.cu, nn_conv.cu, nn_wgrad.cu): weight preparation, ReLU
// backward and Adam.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "nn_internal.cuh"

namespace tomo_nn {
namespace {

__device__ unsigned g_status;  // bit 0: a tensor-core wait gave up
std::atomic<int> g_wait_spins{1 << 22};

unsigned *status_ptr() {
  static std::mutex mu;
  static unsigned *ptr[64] = {nullptr};
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 0 || dev >= 64) return nullptr;
  if (!ptr[dev]) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_status) != cudaSuccess) return nullptr;
    ptr[dev] = (unsigned *)p;
  }
  return ptr[dev];
}

__global__ void prepare_weights_kernel(const float *__restrict__ W, int Cout, int Cin, int taps,
                                       __nv_bfloat16 *__restrict__ Wb, __nv_bfloat16 *__restrict__ Wd) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = (long long)Cout * taps * Cin;
  if (i >= n) return;
  const int ci = (int)(i % Cin), t = (int)((i / Cin) % taps), co = (int)(i / ((long long)Cin * taps));
  const __nv_bfloat16 v = __float2bfloat16_rn(W[i]);
  Wb[i] = v;
  if (Wd) Wd[((long long)ci * taps + (taps - 1 - t)) * Cout + co] = v;
}

__global__ void relu_bwd_kernel(const __nv_bfloat16 *__restrict__ Y, __nv_bfloat16 *__restrict__ dY, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
    if (!(__bfloat162float(Y[i]) > 0.0f)) dY[i] = __float2bfloat16_rn(0.0f);
}

__global__ void adam_kernel(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, size_t n, float lr, float b1, float b2, float eps, float c1,
                            float c2) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

}  // namespace

int make_tensor_map(void *map, const void *base, int rank, const unsigned long long *dim,
                    const unsigned long long *stride, const unsigned *box, int rb) {
  using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                              const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const Encode encode = [] {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess) fn = nullptr;
    return (Encode)fn;
  }();
  if (!encode) return NN_ECUDA;
  cuuint64_t d[5], s[4];
  cuuint32_t bx[5], es[5];
  for (int i = 0; i < rank; ++i) {
    d[i] = dim[i];
    bx[i] = box[i];
    es[i] = 1;
    if (i + 1 < rank) s[i] = stride[i];
  }
  const CUtensorMapSwizzle sw = rb == 128  ? CU_TENSOR_MAP_SWIZZLE_128B
                                : rb == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                : rb == 32 ? CU_TENSOR_MAP_SWIZZLE_32B
                                           : CU_TENSOR_MAP_SWIZZLE_NONE;
  return encode((CUtensorMap *)map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void *>(base), d, s, bx, es,
                CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? NN_OK
             : NN_ECUDA;
}

}  // namespace tomo_nn

using namespace tomo_nn;

extern "C" {

int tomo_nn_gemm(const void *A, int lda, const void *B, int ldb, int M, int N, int K, float *Cf, void *Cb,
                 int ldc, const float *bias, int relu, void *stream) {
  GemmArgs g;
  g.A = (const __nv_bfloat16 *)A;
  g.lda = lda;
  g.B = (const __nv_bfloat16 *)B;
  g.ldb = ldb;
  g.M = M;
  g.N = N;
  g.K = K;
  g.Cf = Cf;
  g.Cb = (__nv_bfloat16 *)Cb;
  g.ldc = ldc;
  g.bias = bias;
  g.relu = relu;
  g.status = status_ptr();
  g.spins = g_wait_spins.load();
  return gemm_launch(g, (cudaStream_t)stream);
}

int tomo_nn_conv3x3(const void *X, int batch, int H, int W, int Cin, const void *Wt, int Cout, float *Yf,
                    void *Yb, const float *bias, int relu, void *stream) {
  return conv_launch((const __nv_bfloat16 *)X, batch, H, W, Cin, (const __nv_bfloat16 *)Wt, Cout, Yf, (__nv_bfloat16 *)Yb,
                     bias, relu, nullptr, status_ptr(), g_wait_spins.load(), (cudaStream_t)stream);
}

int tomo_nn_conv3x3_masked(const void *X, int batch, int H, int W, int Cin, const void *Wt, int Cout, const void *mask,
                           void *Yb, void *stream) {
  if (!mask) return NN_EINVAL;
  return conv_launch((const __nv_bfloat16 *)X, batch, H, W, Cin, (const __nv_bfloat16 *)Wt, Cout, nullptr,
                     (__nv_bfloat16 *)Yb, nullptr, 0, (const __nv_bfloat16 *)mask, status_ptr(), g_wait_spins.load(),
                     (cudaStream_t)stream);
}

size_t tomo_nn_wgrad_workspace(int batch, int H, int W, int Cin, int Cout, int taps) {
  if ((taps != 9 && taps != 1) || Cin < 8 || Cout < 1 || batch < 1 || H < 1 || W < 1 ||
      (long long)H * W > 0x7fffffffLL / batch)
    return 256;  // tomo_nn_wgrad refuses these
  return wgrad_workspace(batch, H, W, Cin, Cout, taps);
}

int tomo_nn_wgrad(const void *X, const void *dY, int batch, int H, int W, int Cin, int Cout, int taps,
                  float *dW, float *db, void *work, size_t work_bytes, void *stream) {
  if ((taps != 9 && taps != 1) || Cin < 8 || Cin % 8 || Cout < 1 || batch < 1 || H < 1 || W < 1) return NN_EINVAL;
  const long long P = (long long)batch * H * W;
  if (P % 8 || P > 0x7fffffffLL) return NN_EINVAL;
  if (work_bytes < tomo_nn_wgrad_workspace(batch, H, W, Cin, Cout, taps)) return NN_EINVAL;
  return wgrad_launch((const __nv_bfloat16 *)X, (const __nv_bfloat16 *)dY, batch, H, W, Cin, Cout, taps, dW, db, work,
                      status_ptr(), g_wait_spins.load(), (cudaStream_t)stream);
}

int tomo_nn_prepare_weights(const float *W, int Cout, int Cin, int taps, void *Wb, void *Wd, void *stream) {
  const long long n = (long long)Cout * taps * Cin;
  if (n <= 0) return NN_EINVAL;
  prepare_weights_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      W, Cout, Cin, taps, (__nv_bfloat16 *)Wb, (__nv_bfloat16 *)Wd);
  return cudaGetLastError() == cudaSuccess ? NN_OK : NN_ECUDA;
}

int tomo_nn_relu_bwd(const void *Y, void *dY, size_t n, void *stream) {
  if (!n) return NN_OK;
  relu_bwd_kernel<<<(unsigned)std::min<size_t>((n + 255) / 256, 148 * 16), 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16 *)Y, (__nv_bfloat16 *)dY, n);
  return cudaGetLastError() == cudaSuccess ? NN_OK : NN_ECUDA;
}

int tomo_nn_adam(float *p, const float *g, float *m, float *v, size_t n, float lr, float beta1, float beta2,
                 float eps, int step, void *stream) {
  if (!n || step < 1) return NN_EINVAL;
  const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
  adam_kernel<<<(unsigned)std::min<size_t>((n + 255) / 256, 148 * 16), 256, 0, (cudaStream_t)stream>>>(
      p, g, m, v, n, lr, beta1, beta2, eps, c1, c2);
  return cudaGetLastError() == cudaSuccess ? NN_OK : NN_ECUDA;
}

int tomo_nn_set_wait_limit(int spins) {
  tomo_nn::g_wait_spins.store(spins < 0 ? (1 << 22) : spins);
  return NN_OK;
}

int tomo_nn_status(unsigned *flags) {
  unsigned *d = status_ptr();
  if (!d) return NN_ECUDA;
  unsigned h = 0;
  if (cudaDeviceSynchronize() != cudaSuccess) return NN_ECUDA;
  if (cudaMemcpy(&h, d, sizeof(unsigned), cudaMemcpyDeviceToHost) != cudaSuccess) return NN_ECUDA;
  const unsigned zero = 0;
  if (cudaMemcpy(d, &zero, sizeof(unsigned), cudaMemcpyHostToDevice) != cudaSuccess) return NN_ECUDA;
  if (flags) *flags = h;
  return NN_OK;
}

}  // extern "C"
