// Weight and bias gradients of a convolution on the tensor cores (sm_100a):
//
//   dW[co][tap][ci] = sum over pixels p of dY[p][co] X[p + tap][ci],
//
// one GEMM per tap with M = output channels, N = input channels and K =
// pixels, read straight from the NHWC tensors.
//
// Both operands are MN-major: a 16-byte unit holds 8 channels of one pixel,
// which is how NHWC memory lies, so no transposed copy is made.  A stage holds
// 64 pixels (in image order) of the output gradient as [8-channel chunk][pixel]
// [16 bytes] and what their taps need of the input.  Where W is a multiple of
// 8 that is, per input row of the taps, a strip of 8 groups of 10 pixels (8
// and one on each side): a tap is then an offset of (row, dx) into the strip
// and the two K groups of an MMA lie 10 pixels apart, so one staged strip
// serves the three taps of its row.  Otherwise (W not a multiple of 8: a
// group would run over the end of a row; 1x1) the stage holds the shifted 64
// pixels of every tap.  Each tap accumulates in TMEM columns of its own.
//
// Bound: the copies from L2 (with 32 channels 3.75 x the input and 3 x the
// gradient instead of 9 x the input).  Eight producer warps issue zero-filled
// 16-byte cp.async copies several stages ahead of one MMA thread.  The kernel
// this one replaces wrote the im2col matrix (9 copies of X, transposed) to
// memory and read it back: at 4 x 192^2, 128 -> 128 channels the whole
// gradient took 1.28 ms, now 0.17 ms; at 4 x 768^2, 32 -> 32, 6.19, now 0.69.
//
// Work split: a CTA owns up to 128 output channels, a block of input channels
// and a group of taps (TMEM holds 512 FP32 columns = taps x channels), and one
// of S contiguous ranges of 64-pixel blocks; it writes its partial sums once
// and wgrad_reduce_kernel adds the S partials in order.  S depends on the
// layer's shape alone, and pixels are added 16 at a time in image order, so
// the result depends neither on the grouping of the taps nor on scheduling.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "nn_ptx.cuh"

namespace tomo_nn {
namespace {

constexpr int kKP = 64;            // pixels of a stage
constexpr int kProd = 256;         // producer threads (warps 0-7); warps 0-3 also run the epilogue
constexpr int kWgThreads = kProd + 32;
constexpr int kMaxStages = 8;
constexpr int kSms = 148;
constexpr int kSmemMax = 224 * 1024;
constexpr int kDrainSpins = 1 << 22;

struct WgradArgs {
  const __nv_bfloat16 *X, *dY;
  float *part;  // [S][Cout][taps][Cin]
  unsigned *status;
  int spins;
  int H, W, Cin, Cout, ldY, taps;  // ldY: channels per pixel of dY in memory (Cout rounded up to 8)
  int P, nkb;                      // pixels, 64-pixel blocks
  FastDiv fhw, fw;
  int S, G, ntap, NB, Nb, Mb;  // splits; tap groups and taps per group; input-channel blocks and their width; output rows staged
  int mrows;                   // rows of an MMA: 64 up to 64 output channels, else 128
  int strip, sxc, syc, stage_bytes, tail_bytes, nst, cols;
};

// LAG: copy groups a producer keeps in flight behind the one it just issued.
template <int LAG, bool STRIP>
__global__ void __launch_bounds__(kWgThreads) wgrad_tc_kernel(WgradArgs g) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint64_t full[kMaxStages], empty[kMaxStages], done;
  __shared__ uint32_t tmem_slot;
  __shared__ int gave_up;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // unit: (output-channel block, input-channel block, tap group)
  int u = blockIdx.x;
  const int tg = u % g.G;
  u /= g.G;
  const int n0 = (u % g.NB) * g.Nb, m0 = (u / g.NB) * 128;
  const int tap0 = tg * g.ntap, ntap = min(g.ntap, g.taps - tap0);
  const int t0 = (int)((long long)g.nkb * blockIdx.y / g.S), t1 = (int)((long long)g.nkb * (blockIdx.y + 1) / g.S);
  const int ncx = min(g.Nb, g.Cin - n0) >> 3;                 // 8-channel chunks of X staged
  const int ncy = (min(128, g.Cout - m0) + 7) >> 3;           // and of dY
  const int r0 = tap0 / 3, nrow = (tap0 + ntap - 1) / 3 - r0 + 1;  // STRIP: input rows of the taps

  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                 "r"(g.cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  if (tid == 0) {
    for (int s = 0; s < g.nst; ++s) {
      mbar_init(smem_u32(&full[s]), kProd);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    mbar_init(smem_u32(&done), 1);
    gave_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t base = smem_u32(smem);

  if (warp < 8) {  // producers
    // Warp w stages pixels 8w .. 8w+7 of the block: of X, per input row (STRIP)
    // their strip of 10, else per tap the 8 shifted pixels; consecutive lanes
    // take consecutive chunks.
    constexpr int kGrp = STRIP ? 10 : 8;
    const int nx = (STRIP ? nrow : ntap) * kGrp * ncx, ny = 8 * ncy;
    // a lane's copies are 32 apart: (position, chunk) advances by (q, r)
    const int qx = 32 / ncx, rx = 32 % ncx, px0 = lane / ncx, cx0 = lane % ncx;
    const int qy = 32 / ncy, ry = 32 % ncy, py0 = lane / ncy, cy0 = lane % ncy;
    const int hw = g.H * g.W;
    int pending = 0;  // stages issued and not yet announced
    bool ok = true;
    for (int t = t0; t < t1 && ok; ++t) {
      const int it = t - t0, s = it % g.nst;
      if (it >= g.nst) ok = mbar_wait(smem_u32(&empty[s]), ((it / g.nst) - 1) & 1, g.spins);
      if (!ok) break;
      const uint32_t sx = base + s * g.stage_bytes + warp * kGrp * 16;
      const uint32_t sy = base + s * g.stage_bytes + (g.Nb >> 3) * g.sxc + warp * 128;
      const int p = t * kKP + warp * 8;
      if (STRIP) {  // the 8 pixels lie in one image row
        const int b = fast_div(p, g.fhw), q = p - b * hw, yc = fast_div(q, g.fw), xc = q - yc * g.W - 1;
        const int ya = yc + r0 - 1;
        const bool live = p < g.P;
        // strip position 0 of row ya (may lie outside the image: never read then)
        const __nv_bfloat16 *Xb = g.X + ((long long)b * hw + (long long)ya * g.W + xc) * g.Cin + n0;
#pragma unroll 4
        for (int i = lane, pos = px0, c = cx0; i < nx; i += 32) {
          const int r = pos / 10, o = pos - 10 * r;
          const bool in = live && (unsigned)(ya + r) < (unsigned)g.H && (unsigned)(xc + o) < (unsigned)g.W;
          cp_async16(sx + c * g.sxc + (r * 80 + o) * 16, in ? Xb + (r * g.W + o) * g.Cin + c * 8 : g.X, in);
          pos += qx;
          c += rx;
          if (c >= ncx) c -= ncx, ++pos;
        }
      } else {
#pragma unroll 2
        for (int i = lane, pos = px0, c = cx0; i < nx; i += 32) {
          const int j = pos >> 3, o = pos & 7, tap = g.taps == 9 ? tap0 + j : 4;
          const int b = fast_div(p + o, g.fhw), q = p + o - b * hw, yc = fast_div(q, g.fw);
          const int y = yc + tap / 3 - 1, x = q - yc * g.W + tap % 3 - 1;
          const bool in = p + o < g.P && (unsigned)y < (unsigned)g.H && (unsigned)x < (unsigned)g.W;
          const __nv_bfloat16 *src = in ? g.X + (size_t)(b * hw + y * g.W + x) * g.Cin + n0 + c * 8 : g.X;
          cp_async16(sx + c * g.sxc + (j * kKP + o) * 16, src, in);
          pos += qx;
          c += rx;
          if (c >= ncx) c -= ncx, ++pos;
        }
      }
      const __nv_bfloat16 *Yb = g.dY + (size_t)p * g.ldY + m0;
#pragma unroll 2
      for (int i = lane, px = py0, c = cy0; i < ny; i += 32) {
        const bool in = p + px < g.P;
        cp_async16(sy + c * g.syc + px * 16, in ? Yb + px * g.ldY + c * 8 : g.dY, in);
        px += qy;
        c += ry;
        if (c >= ncy) c -= ncy, ++px;
      }
      cp_async_commit();
      if (++pending > LAG) {  // the oldest pending stage has landed
        cp_async_wait<LAG>();
        fence_proxy_async();
        mbar_arrive(smem_u32(&full[(it - LAG) % g.nst]));
        --pending;
      }
    }
    cp_async_wait<0>();
    fence_proxy_async();
    if (ok)
      for (int it = t1 - t0 - pending; it < t1 - t0; ++it) mbar_arrive(smem_u32(&full[it % g.nst]));
    else
      atomicOr(&gave_up, 1);
  } else if (lane == 0) {  // the MMA thread
    const uint32_t idesc = instr_desc_mn(g.Nb, g.mrows);
    constexpr uint32_t kgroup = STRIP ? 160 : 128;  // bytes between groups of 8 pixels
    // descriptors of stage 0; an address advances by its bytes / 16
    const uint64_t da0 = smem_desc(base + (g.Nb >> 3) * g.sxc, 128, g.syc), db0 = smem_desc(base, kgroup, g.sxc);
    bool ok = true;
    int last = -1;
    for (int t = t0; t < t1; ++t) {
      const int it = t - t0, s = it % g.nst;
      ok = mbar_wait(smem_u32(&full[s]), (it / g.nst) & 1, g.spins);
      if (!ok) break;
      tc_fence_after();
      const uint64_t da = da0 + (uint32_t)(s * g.stage_bytes >> 4), db = db0 + (uint32_t)(s * g.stage_bytes >> 4);
      const uint32_t more = it > 0;
      int r = 0, dx = tap0 - 3 * r0;
      for (int j = 0; j < ntap; ++j) {
        const uint64_t dbj = db + (uint32_t)(STRIP ? r * 80 + dx : j * kKP);
        const uint32_t d = tmem + j * g.Nb;
        mma_bf16(d, da, dbj, idesc, more);
#pragma unroll
        for (int k = 1; k < kKP / 16; ++k) mma_bf16(d, da + k * 16, dbj + k * (2 * kgroup / 16), idesc, 1u);
        if (++dx == 3) dx = 0, ++r;
      }
      mma_commit(smem_u32(&empty[s]));
      last = it;
    }
    if (!ok) atomicOr(&gave_up, 1);
    // every MMA issued so far, also on the way out of a wait that gave up
    if (last >= 0) {
      mma_commit(smem_u32(&done));
      if (!mbar_wait(smem_u32(&done), 0, kDrainSpins)) atomicOr(&gave_up, 1);
    }
  }
  __syncwarp();
  __syncthreads();
  tc_fence_after();
  const bool ok = gave_up == 0;
  if (!ok && tid == 0 && g.status) atomicOr(g.status, 1);
  if (ok && warp < 4) {
    // 64-row accumulators lie in lanes 0-15 of each warp's 32
    const int co = g.mrows == 64 ? (lane < 16 ? m0 + warp * 16 + lane : g.Cout) : m0 + warp * 32 + lane;
    float *dst = g.part + ((size_t)blockIdx.y * g.Cout + (co < g.Cout ? co : 0)) * g.taps * g.Cin;
    for (int j = 0; j < ntap; ++j)
#pragma unroll 1
      for (int c0 = 0; c0 < (ncx << 3); c0 += 16) {
        float v[16];
        tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(j * g.Nb + c0), v);
        if (t1 <= t0)
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = 0.0f;
        if (co < g.Cout) {
          float4 *o = (float4 *)(dst + (size_t)(tap0 + j) * g.Cin + n0 + c0);
          o[0] = make_float4(v[0], v[1], v[2], v[3]);
          o[1] = make_float4(v[4], v[5], v[6], v[7]);
          if (c0 + 8 < (ncx << 3)) {
            o[2] = make_float4(v[8], v[9], v[10], v[11]);
            o[3] = make_float4(v[12], v[13], v[14], v[15]);
          }
        }
      }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(g.cols));
}

// dW[i] = sum_s part[s][i], s ascending (part is [S][n]).
__global__ void wgrad_reduce_kernel(const float *__restrict__ part, int S, size_t n, float *__restrict__ dW) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float acc = 0.0f;
#pragma unroll 8
  for (int s = 0; s < S; ++s) acc += __ldg(part + (size_t)s * n + i);
  dW[i] = acc;
}

// Bias gradient: block b sums its range of pixels of dY [P][C] per channel.  A
// thread takes 8 channels of every (threads / (C/8))-th pixel, in double, so
// the sum's own rounding stays below the result's; the block's threads and
// then the blocks (colsum_final_kernel) are added in order.
constexpr int kColThreads = 256, kColBlocks = 592;

__global__ void __launch_bounds__(kColThreads) colsum_kernel(const __nv_bfloat16 *__restrict__ Y, long long P, int C,
                                                             double *__restrict__ part) {
  __shared__ double red[kColThreads][8];
  const int nc = C >> 3;
  const long long p0 = P * blockIdx.x / gridDim.x, p1 = P * (blockIdx.x + 1) / gridDim.x;
  for (int cb = 0; cb < nc; cb += kColThreads) {
    const int w = min(nc - cb, kColThreads), rows = kColThreads / w;
    const int c = threadIdx.x % w, r = threadIdx.x / w;
    double a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (r < rows) {
      for (long long p = p0 + r; p < p1; p += 16 * rows) {  // 16 pixels in float, then double
        float f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 4
        for (int k = 0; k < 16; ++k) {
          const long long q = p + (long long)k * rows;
          if (q < p1) {
            const uint4 v = __ldg((const uint4 *)(Y + q * C) + cb + c);
            const unsigned w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              f[2 * i] += __uint_as_float(w4[i] << 16);
              f[2 * i + 1] += __uint_as_float(w4[i] & 0xffff0000u);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] += (double)f[i];
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) red[threadIdx.x][i] = a[i];
    __syncthreads();
    for (int k = threadIdx.x; k < 8 * w; k += kColThreads) {
      double s = 0.0;
      for (int q = 0; q < rows; ++q) s += red[q * w + (k >> 3)][k & 7];
      part[(size_t)blockIdx.x * C + 8 * cb + k] = s;
    }
    __syncthreads();
  }
}

// db[c] = sum over blocks of part[b][c]: a warp per channel, lanes 32 blocks
// apart, then a fixed butterfly (one thread per channel was a chain of 592
// loads, 32 us).
__global__ void __launch_bounds__(128) colsum_final_kernel(const double *__restrict__ part, int nblk, int C, int ld,
                                                           float *__restrict__ db) {
  const int c = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (c >= C) return;  // warp-uniform
  double s = 0.0;
  for (int b = lane; b < nblk; b += 32) s += part[(size_t)b * ld + c];
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) db[c] = (float)s;
}

size_t align256(size_t b) { return (b + 255) / 256 * 256; }

// Ranges of 64-pixel blocks whose partial sums are added afterwards: a
// function of the layer's shape (128 x 256 tiles of its weight matrix), at
// least 4096 pixels each.
int wgrad_split(long long P, int M, int N) {
  const int bn = N <= 32 ? 32 : N <= 64 ? 64 : N <= 128 ? 128 : 256;
  const long long tiles = (long long)((M + 127) / 128) * ((N + bn - 1) / bn);
  long long s = std::max(1LL, 296 / tiles);
  s = std::min(s, std::max(1LL, P / 4096));
  return (int)std::min(s, 64LL);
}

// How a gradient is cut: TMEM's 512 columns hold ntap x Nb accumulators, so
// wide layers split their taps into groups (each stages its pixels again) and,
// above 256 input channels, the channels too.  Fewer groups stage less; more
// give more CTAs: the smallest count that fits TMEM and gives at least 90
// CTAs (192^2, 128 -> 128: 0.17 ms with 96 CTAs; with 160, a second wave).
WgradArgs wgrad_plan(int batch, int H, int W, int Cin, int Cout, int taps) {
  WgradArgs g{};
  g.H = H;
  g.W = W;
  g.Cin = Cin;
  g.Cout = Cout;
  g.ldY = (Cout + 7) / 8 * 8;
  g.taps = taps;
  g.P = batch * H * W;
  g.nkb = (g.P + kKP - 1) / kKP;
  g.fhw = make_div(H * W);
  g.fw = make_div(W);
  g.S = wgrad_split(g.P, taps * Cin, Cout);
  g.NB = (Cin + 255) / 256;
  g.Nb = ((Cin + g.NB - 1) / g.NB + 15) / 16 * 16;
  g.NB = (Cin + g.Nb - 1) / g.Nb;
  const int MB = (Cout + 127) / 128;
  g.Mb = std::min(Cout, 128);
  g.mrows = Cout <= 64 ? 64 : 128;
  g.strip = taps == 9 && W % 8 == 0;
  for (g.G = 1; g.G <= taps; ++g.G) {
    g.ntap = (taps + g.G - 1) / g.G;
    if (g.G > 1 && (taps + g.ntap - 1) / g.ntap != g.G) continue;  // a smaller count gives the same groups
    if (g.ntap * g.Nb <= 512 && (MB * g.NB * g.G * g.S >= 90 || g.G == taps)) break;
  }
  g.cols = 32;
  while (g.cols < g.ntap * g.Nb) g.cols *= 2;
  int rows = 0;  // most input rows of a group's taps
  for (int t = 0; t < taps; t += g.ntap) rows = std::max(rows, (std::min(t + g.ntap, taps) - 1) / 3 - t / 3 + 1);
  // one 16-byte unit of padding per chunk spreads the copies over the banks
  g.sxc = (g.strip ? rows * 80 : g.ntap * kKP) * 16 + 16;
  g.syc = kKP * 16 + 16;
  g.stage_bytes = (g.Nb / 8) * g.sxc + ((g.Mb + 7) / 8) * g.syc;
  g.tail_bytes = (g.mrows / 8 - (g.Mb + 7) / 8) * g.syc;
  // two CTAs to an SM when there are more than one for each
  int budget = MB * g.NB * g.G * g.S > kSms && 2 * g.cols <= 512 ? kSmemMax / 2 : kSmemMax;
  if (2 * g.stage_bytes + g.tail_bytes > budget) budget = kSmemMax;
  g.nst = std::min(kMaxStages, (budget - g.tail_bytes) / g.stage_bytes);
  return g;
}

// out[p][c] = Y[p][c], c < C, and 0 for the channels up to ld: the gradient
// kernel's form of a dY whose channel count or address rules out 16-byte
// copies (ld = C rounded up to 8).  Also copies a misaligned X (ld = C).
__global__ void repack_kernel(const __nv_bfloat16 *__restrict__ Y, long long P, int C, int ld,
                              __nv_bfloat16 *__restrict__ out) {
  const long long n = P * ld;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long p = i / ld;
    const int c = (int)(i - p * ld);
    out[i] = c < C ? Y[p * C + c] : __float2bfloat16_rn(0.0f);
  }
}

struct WgradWork {  // byte offsets in the workspace
  size_t colsum, xcopy, ycopy, total;
};
WgradWork wgrad_work(const WgradArgs &g, int batch) {
  const size_t P = (size_t)batch * g.H * g.W;
  WgradWork w;
  w.colsum = align256(sizeof(float) * (size_t)g.S * g.taps * g.Cin * g.Cout);
  w.xcopy = w.colsum + align256(sizeof(double) * (size_t)kColBlocks * g.ldY);
  w.ycopy = w.xcopy + align256(sizeof(__nv_bfloat16) * P * g.Cin);
  w.total = w.ycopy + align256(sizeof(__nv_bfloat16) * P * g.ldY);
  return w;
}

}  // namespace

size_t wgrad_workspace(int batch, int H, int W, int Cin, int Cout, int taps) {
  return wgrad_work(wgrad_plan(batch, H, W, Cin, Cout, taps), batch).total;
}

int wgrad_launch(const __nv_bfloat16 *X, const __nv_bfloat16 *dY, int batch, int H, int W, int Cin, int Cout, int taps,
                 float *dW, float *db, void *work, unsigned *status, int spins, cudaStream_t s) {
  if ((uintptr_t)work & 15) return NN_EINVAL;
  WgradArgs g = wgrad_plan(batch, H, W, Cin, Cout, taps);
  const WgradWork ww = wgrad_work(g, batch);
  const long long P = (long long)batch * H * W;
  char *w = (char *)work;
  if ((uintptr_t)X & 15) {
    repack_kernel<<<kSms * 8, 256, 0, s>>>(X, P, Cin, Cin, (__nv_bfloat16 *)(w + ww.xcopy));
    X = (const __nv_bfloat16 *)(w + ww.xcopy);
  }
  if (((uintptr_t)dY & 15) || g.ldY != Cout) {
    repack_kernel<<<kSms * 8, 256, 0, s>>>(dY, P, Cout, g.ldY, (__nv_bfloat16 *)(w + ww.ycopy));
    dY = (const __nv_bfloat16 *)(w + ww.ycopy);
  }
  g.X = X;
  g.dY = dY;
  g.part = (float *)work;
  g.status = status;
  g.spins = spins;
  // an MMA reads mrows rows of A and Nb of B whatever the channel counts: rows
  // behind the staged ones are other bytes of the allocation, and only feed
  // accumulators that nothing reads
  const size_t smem = (size_t)g.nst * g.stage_bytes + g.tail_bytes;
  const int lag = g.nst >= 7 ? 5 : g.nst >= 5 ? 3 : g.nst >= 3 ? 2 : 1;
  auto fn = g.strip ? (lag == 5   ? wgrad_tc_kernel<5, true>
                       : lag == 3 ? wgrad_tc_kernel<3, true>
                       : lag == 2 ? wgrad_tc_kernel<2, true>
                                  : wgrad_tc_kernel<1, true>)
                    : (lag == 5   ? wgrad_tc_kernel<5, false>
                       : lag == 3 ? wgrad_tc_kernel<3, false>
                       : lag == 2 ? wgrad_tc_kernel<2, false>
                                  : wgrad_tc_kernel<1, false>);
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return NN_ECUDA;
  const int units = (Cout + 127) / 128 * g.NB * g.G;
  fn<<<dim3(units, g.S), kWgThreads, smem, s>>>(g);
  const size_t nout = (size_t)taps * Cin * Cout;
  wgrad_reduce_kernel<<<(unsigned)((nout + 255) / 256), 256, 0, s>>>(g.part, g.S, nout, dW);
  if (db) {
    double *cp = (double *)(w + ww.colsum);
    const int nblk = (int)std::min<long long>(kColBlocks, std::max<long long>(1, P / 64));
    colsum_kernel<<<nblk, kColThreads, 0, s>>>(dY, P, g.ldY, cp);
    colsum_final_kernel<<<(Cout + 3) / 4, 128, 0, s>>>(cp, nblk, Cout, g.ldY, db);
  }
  return cudaGetLastError() == cudaSuccess ? NN_OK : NN_ECUDA;
}

}  // namespace tomo_nn
