// The U-Net's passes between convolutions: 2x2 max-pooling, nearest upsampling
// with the skip's concatenation, their backwards, and the 1x1 head's backward.
// All are bound by memory, so each reads and writes its tensors once, 16 bytes
// (8 channels) per access, and the backwards also apply the ReLU of the
// convolution that they hand their gradient to (its output is what they read for
// the pooling's argmax, or the upsampled input).  As chains of library passes
// (upsample, cat, copies, pooling backward, add, ReLU) these were 6.9 of the 12.9
// ms of a training step at 4 x 768^2, 32 channels, 4 levels; now 0.66.
//
// Layouts: BF16, NHWC, channel counts multiples of 8, pointers 16-byte aligned.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "nn_internal.cuh"

namespace tomo_nn {
namespace {

constexpr int kThreads = 256;

struct Vec {  // 8 channels
  float f[8];
};
__device__ __forceinline__ Vec load8(const __nv_bfloat16 *p) {
  const uint4 u = __ldg((const uint4 *)p);
  const unsigned w[4] = {u.x, u.y, u.z, u.w};
  Vec v;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v.f[2 * i] = __uint_as_float(w[i] << 16);
    v.f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
  return v;
}
__device__ __forceinline__ void store8(__nv_bfloat16 *p, const Vec &v) {
  unsigned w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v.f[2 * i], v.f[2 * i + 1]);
    w[i] = *(const unsigned *)&h;
  }
  *(uint4 *)p = make_uint4(w[0], w[1], w[2], w[3]);
}

// A thread takes one vector of one row of the smaller image: block = row x part of it.
struct Place {
  long long row;  // image * h + y
  int x, c;       // pixel, first channel
  bool in;
};
__device__ __forceinline__ Place place(int bpr, int w, int C) {
  Place p;
  p.row = blockIdx.x / (unsigned)bpr;
  const unsigned i = (blockIdx.x % (unsigned)bpr) * kThreads + threadIdx.x, nc = (unsigned)C >> 3;
  p.x = (int)(i / nc);
  p.c = (int)(i - p.x * nc) * 8;
  p.in = p.x < w;
  return p;
}

// The larger of four in row-major order, the first among equals, a NaN over all
// before it (the library's rule).
__device__ __forceinline__ void argmax4(const float (&v)[4], float &m, int &at) {
  m = v[0];
  at = 0;
#pragma unroll
  for (int q = 1; q < 4; ++q)
    if (v[q] > m || v[q] != v[q]) {
      m = v[q];
      at = q;
    }
}

__global__ void __launch_bounds__(kThreads) pool_kernel(const __nv_bfloat16 *__restrict__ X, int bpr, int h, int w, int C,
                                                        __nv_bfloat16 *__restrict__ Y) {
  const Place p = place(bpr, w, C);
  if (!p.in) return;
  const size_t rs = (size_t)2 * w * C;  // a row of X
  const __nv_bfloat16 *s = X + (size_t)(2 * p.row) * rs + (size_t)2 * p.x * C + p.c;
  const Vec v[4] = {load8(s), load8(s + C), load8(s + rs), load8(s + rs + C)};
  Vec o;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float f[4] = {v[0].f[i], v[1].f[i], v[2].f[i], v[3].f[i]};
    int at;
    argmax4(f, o.f[i], at);
  }
  store8(Y + ((size_t)p.row * w + p.x) * C + p.c, o);
}

// dZ = (dS + dP at the window's maximum) where X > 0, else 0; dS has lds channels per pixel.
__global__ void __launch_bounds__(kThreads) pool_bwd_kernel(const __nv_bfloat16 *__restrict__ X,
                                                            const __nv_bfloat16 *__restrict__ dP,
                                                            const __nv_bfloat16 *__restrict__ dS, int lds, int bpr, int h,
                                                            int w, int C, __nv_bfloat16 *__restrict__ dZ) {
  const Place p = place(bpr, w, C);
  if (!p.in) return;
  const size_t px = (size_t)(2 * p.row) * 2 * w + 2 * p.x, at[4] = {px, px + 1, px + 2 * w, px + 2 * w + 1};
  Vec v[4], d[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    v[q] = load8(X + at[q] * C + p.c);
    d[q] = load8(dS + at[q] * lds + p.c);
  }
  const Vec g = load8(dP + ((size_t)p.row * w + p.x) * C + p.c);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float f[4] = {v[0].f[i], v[1].f[i], v[2].f[i], v[3].f[i]};
    float m;
    int a;
    argmax4(f, m, a);
#pragma unroll
    for (int q = 0; q < 4; ++q) d[q].f[i] = f[q] > 0.0f ? d[q].f[i] + (q == a ? g.f[i] : 0.0f) : 0.0f;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) store8(dZ + at[q] * C + p.c, d[q]);
}

// Y [2h][2w][Cu + Cs] = X [h][w][Cu], each pixel four times, beside S [2h][2w][Cs].
__global__ void __launch_bounds__(kThreads) upcat_kernel(const __nv_bfloat16 *__restrict__ X,
                                                         const __nv_bfloat16 *__restrict__ S, int bpr, int h, int w, int Cu,
                                                         int Cs, __nv_bfloat16 *__restrict__ Y) {
  const int C = Cu + Cs;
  const Place p = place(bpr, w, C);
  if (!p.in) return;
  const size_t px = (size_t)(2 * p.row) * 2 * w + 2 * p.x, at[4] = {px, px + 1, px + 2 * w, px + 2 * w + 1};
  uint4 u[4];
  if (p.c < Cu) {
    u[0] = u[1] = u[2] = u[3] = __ldg((const uint4 *)(X + ((size_t)p.row * w + p.x) * Cu + p.c));
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) u[q] = __ldg((const uint4 *)(S + at[q] * Cs + (p.c - Cu)));
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) *(uint4 *)(Y + at[q] * C + p.c) = u[q];
}

// dX = the sum of a pixel's four gradients (ldy channels per pixel of dY) where X > 0, else 0.
__global__ void __launch_bounds__(kThreads) up_bwd_kernel(const __nv_bfloat16 *__restrict__ dY, int ldy,
                                                          const __nv_bfloat16 *__restrict__ X, int bpr, int h, int w, int C,
                                                          __nv_bfloat16 *__restrict__ dX) {
  const Place p = place(bpr, w, C);
  if (!p.in) return;
  const __nv_bfloat16 *s = dY + ((size_t)(2 * p.row) * 2 * w + 2 * p.x) * ldy + p.c;
  const size_t rs = (size_t)2 * w * ldy, o = ((size_t)p.row * w + p.x) * C + p.c;
  const Vec d[4] = {load8(s), load8(s + ldy), load8(s + rs), load8(s + rs + ldy)}, x = load8(X + o);
  Vec r;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    r.f[i] = x.f[i] > 0.0f ? ((d[0].f[i] + d[1].f[i]) + d[2].f[i]) + d[3].f[i] : 0.0f;
  store8(dX + o, r);
}

// dZ [P][8] = {bf16(dY[p]), 0, ..}: the gradient of the head's one used output.
__global__ void __launch_bounds__(kThreads) pad8_kernel(const float *__restrict__ dY, long long P,
                                                        __nv_bfloat16 *__restrict__ dZ) {
  const long long p = (long long)blockIdx.x * kThreads + threadIdx.x;
  if (p >= P) return;
  const Vec v = {{__ldg(dY + p), 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f}};
  store8(dZ + p * 8, v);
}

// dX [P][C] = dZ [P][8] . Wt [C][8]^T where X > 0, else 0: too few terms for the
// tensor cores to matter.
__global__ void __launch_bounds__(kThreads) head_bwd_kernel(const __nv_bfloat16 *__restrict__ dZ,
                                                            const __nv_bfloat16 *__restrict__ Wt,
                                                            const __nv_bfloat16 *__restrict__ X, long long nv, int C,
                                                            __nv_bfloat16 *__restrict__ dX) {
  extern __shared__ float sw[];  // [8][C]
  for (int i = threadIdx.x; i < 8 * C; i += kThreads) sw[(i & 7) * C + (i >> 3)] = __bfloat162float(Wt[i]);
  __syncthreads();
  const int nc = C >> 3;
  for (long long i = (long long)blockIdx.x * kThreads + threadIdx.x; i < nv; i += (long long)gridDim.x * kThreads) {
    const long long p = i / nc;
    const int c = (int)(i - p * nc) * 8;
    const Vec d = load8(dZ + p * 8), x = load8(X + i * 8);
    Vec r;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float a = 0.0f;
#pragma unroll
      for (int k = 0; k < 8; ++k) a = __fmaf_rn(d.f[k], sw[k * C + c + j], a);
      r.f[j] = x.f[j] > 0.0f ? a : 0.0f;
    }
    store8(dX + i * 8, r);
  }
}

// blocks per row of w pixels, and in all; false if they do not fit a grid
bool rows_grid(int batch, int h, int w, int C, int *bpr, unsigned *grid) {
  const long long v = (long long)w * (C >> 3), b = (v + kThreads - 1) / kThreads, g = b * batch * h;
  *bpr = (int)b;
  *grid = (unsigned)g;
  return v <= 0x7fffffffLL && g <= 0x7fffffffLL;
}
bool bad(int batch, int h, int w, int C) { return batch < 1 || h < 1 || w < 1 || C < 8 || C % 8; }
bool odd(const void *a, const void *b, const void *c, const void *d) {
  return (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d) & 15) != 0;
}
int launched() { return cudaGetLastError() == cudaSuccess ? NN_OK : NN_ECUDA; }

}  // namespace
}  // namespace tomo_nn

using namespace tomo_nn;
using bf16 = __nv_bfloat16;

extern "C" {

int tomo_nn_pool(const void *X, int batch, int h, int w, int C, void *Y, void *stream) {
  int bpr;
  unsigned grid;
  if (bad(batch, h, w, C) || odd(X, Y, X, Y) || !rows_grid(batch, h, w, C, &bpr, &grid)) return NN_EINVAL;
  pool_kernel<<<grid, kThreads, 0, (cudaStream_t)stream>>>((const bf16 *)X, bpr, h, w, C, (bf16 *)Y);
  return launched();
}

int tomo_nn_pool_bwd(const void *X, const void *dP, const void *dS, int lds, int batch, int h, int w, int C, void *dZ,
                     void *stream) {
  int bpr;
  unsigned grid;
  if (bad(batch, h, w, C) || odd(X, dP, dS, dZ) || lds < C || lds % 8 || !rows_grid(batch, h, w, C, &bpr, &grid))
    return NN_EINVAL;
  pool_bwd_kernel<<<grid, kThreads, 0, (cudaStream_t)stream>>>((const bf16 *)X, (const bf16 *)dP, (const bf16 *)dS, lds,
                                                               bpr, h, w, C, (bf16 *)dZ);
  return launched();
}

int tomo_nn_upcat(const void *X, const void *S, int batch, int h, int w, int Cu, int Cs, void *Y, void *stream) {
  int bpr;
  unsigned grid;
  if (bad(batch, h, w, Cu) || bad(batch, h, w, Cs) || odd(X, S, Y, Y) || !rows_grid(batch, h, w, Cu + Cs, &bpr, &grid))
    return NN_EINVAL;
  upcat_kernel<<<grid, kThreads, 0, (cudaStream_t)stream>>>((const bf16 *)X, (const bf16 *)S, bpr, h, w, Cu, Cs, (bf16 *)Y);
  return launched();
}

int tomo_nn_up_bwd(const void *dY, int ldy, const void *X, int batch, int h, int w, int C, void *dX, void *stream) {
  int bpr;
  unsigned grid;
  if (bad(batch, h, w, C) || odd(dY, X, dX, dX) || ldy < C || ldy % 8 || !rows_grid(batch, h, w, C, &bpr, &grid))
    return NN_EINVAL;
  up_bwd_kernel<<<grid, kThreads, 0, (cudaStream_t)stream>>>((const bf16 *)dY, ldy, (const bf16 *)X, bpr, h, w, C,
                                                             (bf16 *)dX);
  return launched();
}

int tomo_nn_pad8(const float *dY, long long P, void *dZ, void *stream) {
  if (P < 1 || P > 0x7fffffffLL * kThreads || odd(dZ, dZ, dZ, dZ)) return NN_EINVAL;
  pad8_kernel<<<(unsigned)((P + kThreads - 1) / kThreads), kThreads, 0, (cudaStream_t)stream>>>(dY, P, (bf16 *)dZ);
  return launched();
}

int tomo_nn_head_bwd(const void *dZ, const void *Wt, const void *X, long long P, int C, void *dX, void *stream) {
  if (P < 1 || C < 8 || C % 8 || C > 1024 || odd(dZ, Wt, X, dX)) return NN_EINVAL;
  const long long nv = P * (C >> 3), blocks = (nv + kThreads - 1) / kThreads;
  head_bwd_kernel<<<(unsigned)(blocks < 148 * 8 ? blocks : 148 * 8), kThreads, sizeof(float) * 8 * C,
                    (cudaStream_t)stream>>>((const bf16 *)dZ, (const bf16 *)Wt, (const bf16 *)X, nv, C, (bf16 *)dX);
  return launched();
}

}  // extern "C"
