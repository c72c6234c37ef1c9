// Weight and bias gradients of a convolution on the tensor cores (sm_100a):
//
//   dW[co][tap][ci] = sum over pixels p of dY[p][co] X[p + tap][ci],
//
// one GEMM per tap with M = output channels, N = input channels and K =
// pixels, read straight from the NHWC tensors.
//
// Both operands are MN-major: a pixel's channels are a row, which is how NHWC
// memory lies, so no transposed copy is made.  A stage holds 64 pixels (in
// image order) of the output gradient and what their taps need of the input.
//
// wgrad_tma_kernel (1x1, and 3x3 where W is a multiple of 8): TMA boxes of
// 128-byte (64, 32, 16) swizzled rows; of the input, per tap row dy and block
// of 64 (32, 16, 8) channels, strips of 64 (16, 8) pixels and one on each side,
// whose fill is the zero padding.  The taps dx = 0, 1, 2 of a row are one pixel
// apart, so ONE MMA takes all three: its N blocks, a descriptor's block stride
// apart, are the same block of channels one row of memory further on.  That
// matters with few channels, where an MMA takes its minimum of 50 cycles: at
// 32 -> 32 channels 64 pixels take 12 MMAs of N = 96, not 36 of N = 32.
//
// wgrad_gather_kernel (3x3, W not a multiple of 8: the pixels of a group would
// run over the end of a row): eight producer warps stage the shifted 64 pixels
// of every tap by zero-filled 16-byte cp.async.  TMA moves 50-60 bytes per
// clock and SM in 128-byte rows, those copies 15.
//
// Measured at 4 x 192^2, 128 -> 128 channels: 1.28 ms when the im2col matrix
// was written out, 0.17 with 16-byte copies, now 0.052; 4 x 768^2, 32 -> 32:
// 6.19, 0.69, 0.18; 4 x 192^2, 384 -> 128: 3.42, 0.86, 0.14.
//
// Work split: a CTA owns up to 128 output channels, some of the (tap row,
// channel block) units that fit its 512 TMEM columns, and one of S contiguous
// ranges of 64-pixel blocks; it writes its partial sums once and
// wgrad_reduce_kernel adds the S partials in order.  S depends on the layer's
// shape alone, and pixels are added 16 at a time in image order, so the result
// depends neither on the units' grouping nor on scheduling.
#include <cuda.h>
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
constexpr int kSmemMax = 225 * 1024;
constexpr int kDrainSpins = 1 << 22;

struct WgradArgs {
  const __nv_bfloat16 *X, *dY;
  float *part;  // [S][Cout][taps][Cin]
  unsigned *status;
  int spins;
  int H, W, Cin, Cout, ldY, taps;  // ldY: channels per pixel of dY in memory (Cout rounded up to 8)
  int P, nkb;                      // pixels, 64-pixel blocks
  FastDiv fhw, fw;
  int S, mrows;                    // splits; rows of an MMA: 64 up to 64 output channels, else 128
  int stage_bytes, tail_bytes, nst, cols;
  // wgrad_tma_kernel
  int U, G, upg;                   // units, groups of them, units of a group
  int rb, chb, nblk, ndx, nmma;    // bytes of X's rows, their channels, channel blocks; taps of an MMA and its N
  int gw, strip_bytes, unit_bytes; // pixels of a strip, bytes of a strip and of a unit's strips
  int seg;                         // 64 pixels may go over the end of a row: two strips
  int kpm, blk_bytes;              // 64-pixel blocks of a stage, bytes of one
  int rby, chby, nby, yblk;        // the same of dY: rows, channels, blocks of a CTA's output channels, bytes of one
  // wgrad_gather_kernel
  int ntap, NB, Nb, Mb, sxc, syc;  // taps per group; input-channel blocks and their width; output rows staged
};

// The partial sums of 16 accumulator columns: row co, `n` of them from column
// element e of part's [taps][Cin].
__device__ __forceinline__ void store_part(const WgradArgs &g, int co, size_t e, const float (&v)[16], int n) {
  if (co >= g.Cout) return;
  float4 *o = (float4 *)(g.part + ((size_t)blockIdx.y * g.Cout + co) * g.taps * g.Cin + e);
  o[0] = make_float4(v[0], v[1], v[2], v[3]);
  o[1] = make_float4(v[4], v[5], v[6], v[7]);
  if (n > 8) {
    o[2] = make_float4(v[8], v[9], v[10], v[11]);
    o[3] = make_float4(v[12], v[13], v[14], v[15]);
  }
}

// Warps by role.  A single warp gets an MMA out every 80 clocks and a TMA box
// every 250 here, and each stage's barriers cost it some 400, so the work is
// spread: up to four warps issue MMAs, each those of some units (their
// accumulators are apart), warps 4 and 6 load the input's even and odd units, warp
// 5 the output gradient, and a stage is up to 4 blocks of 64 pixels.
// 4 x 768^2, 32 -> 32 channels: 0.36 ms with one warp each and a block per stage,
// 0.18 now; 96 -> 32: 0.64 and 0.40.
// SEG: blocks of 64 pixels that may go over the end of a row, in two strips then.
template <bool SEG>
__global__ void __launch_bounds__(224) wgrad_tma_kernel(WgradArgs g, const __grid_constant__ CUtensorMap mx,
                                                        const __grid_constant__ CUtensorMap my) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t xfull[2][kMaxStages], yfull[kMaxStages], empty[kMaxStages], done[4];
  __shared__ uint32_t tmem_slot;
  __shared__ int gave_up;
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int tg = blockIdx.x % g.G, m0 = (blockIdx.x / g.G) * 128;
  const int u0 = tg * g.upg, nu = min(g.upg, g.U - u0), nissue = min(nu, 4);
  const int t0 = (int)((long long)g.nkb * blockIdx.y / g.S), t1 = (int)((long long)g.nkb * (blockIdx.y + 1) / g.S);
  const uint32_t base = (smem_u32(smem_raw) + 1023) & ~1023u;  // swizzle period

  if (warp == 5) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                 "r"(g.cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  if (tid == 0) {
    for (int s = 0; s < g.nst; ++s) {
      mbar_init(smem_u32(&xfull[0][s]), 1);
      mbar_init(smem_u32(&xfull[1][s]), 1);
      mbar_init(smem_u32(&yfull[s]), 1);
      mbar_init(smem_u32(&empty[s]), nissue);
    }
    for (int w = 0; w < 4; ++w) mbar_init(smem_u32(&done[w]), 1);
    gave_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t y_off = g.upg * g.unit_bytes;
  bool ok = true;

  if (warp >= 4) {  // loads, by one thread each, whose loops are kept short: coordinates are stepped, not divided out
    if (lane == 0) {
      uint64_t *full = warp == 5 ? yfull : xfull[warp == 6];
      const int nst = g.nst;
      Ring r;
      int it = 0;
      if (warp != 5) {  // units 0, 2, .. or 1, 3, ..
        const int half = warp == 6, mine = (nu + 1 - half) >> 1;
        const int halo = g.ndx >> 1, nstrip = kKP / g.gw, gw = g.gw, W = g.W, H = g.H, chb = g.chb;
        const int nblk = g.nblk, sb = g.strip_bytes, ub = 2 * g.unit_bytes;
        const uint32_t bytes = mine * (gw + 2 * halo) * g.rb;  // of a strip
        const int dyu = (u0 + half) / nblk, cu = (u0 + half - dyu * nblk) * chb, cend = nblk * chb;
        // the next strip's first pixel; from P on it lies in images that do not exist: zero
        int x = t0 * kKP, y = 0, b = 0;
        if (halo) {
          b = fast_div(x, g.fhw);
          x -= b * H * W;
          y = fast_div(x, g.fw);
          x -= y * W;
        }
        auto strips = [&](uint32_t dst, int xs, uint32_t bar) {
          int yy = y + dyu - halo, c = cu;
          dst += half * g.unit_bytes;
          for (int u = 0; u < mine; ++u, dst += ub) {
            tma_load4(dst, &mx, c, xs - halo, yy, b, bar);
            c += 2 * chb;
            while (c >= cend) c -= cend, ++yy;
          }
        };
        auto next_row = [&] {
          if (++y == H) y = 0, ++b;
        };
        for (int t = t0; t < t1; ++it, r.next(nst)) {
          if (it >= nst) ok = role_wait(&empty[r.s], r.ph ^ 1u, g.spins, &gave_up);
          if (!ok) break;
          const uint32_t bar = smem_u32(&full[r.s]);
          uint32_t st = base + r.s * g.stage_bytes;
          const int te = min(t + g.kpm, t1);
          if (SEG) {
            int count = te - t;
            for (int k = t, xx = x; k < te; ++k)
              if ((xx += kKP) >= W) xx -= W, count += xx > 0;
            mbar_expect(bar, count * bytes);
            for (; t < te; ++t, st += g.blk_bytes) {
              strips(st, x, bar);
              if ((x += kKP) >= W) {  // the rest, from the next row's first pixel
                x -= W;
                next_row();
                if (x > 0) strips(st + sb, 0, bar);
              }
            }
          } else {
            mbar_expect(bar, (te - t) * nstrip * bytes);
            for (; t < te; ++t, st += g.blk_bytes)
              for (int q = 0; q < nstrip; ++q) {
                strips(st + q * sb, x, bar);
                x += gw;
                if (halo && x >= W) {
                  x = 0;
                  next_row();
                }
              }
          }
        }
      } else {
        const int nby = min(g.nby, (g.ldY - m0 + g.chby - 1) / g.chby);
        const uint32_t bytes = nby * kKP * g.rby;
        for (int t = t0; t < t1; ++it, r.next(nst)) {
          if (it >= nst) ok = role_wait(&empty[r.s], r.ph ^ 1u, g.spins, &gave_up);
          if (!ok) break;
          const uint32_t bar = smem_u32(&full[r.s]);
          uint32_t st = base + r.s * g.stage_bytes + y_off;
          const int te = min(t + g.kpm, t1);
          mbar_expect(bar, (te - t) * bytes);
          for (; t < te; ++t, st += g.blk_bytes)
            for (int c = 0; c < nby; ++c) tma_load3(st + c * g.yblk, &my, m0 + c * g.chby, t * kKP, 0, bar);
        }
      }
      // copies still in flight (after a wait that gave up nobody else waits for them)
      for (int k = max(0, it - nst); k < it; ++k)
        if (!mbar_wait(smem_u32(&full[k % nst]), (k / nst) & 1, kDrainSpins)) ok = false;
    }
  } else if (warp < nissue) {  // MMAs of units warp, warp + 4, ...
    const uint32_t idesc = instr_desc_mn(g.nmma, g.mrows);
    // K groups of 8 pixels follow one another, or, in strips of 8, lie a strip
    // apart; N blocks (taps) one pixel apart
    const uint32_t kg = g.gw == 8 ? g.strip_bytes : 8 * g.rb;
    const uint64_t dx0 = g.rb == 16 ? smem_desc_rb(0, kg, 16, 16) : smem_desc_rb(0, g.rb, kg, g.rb);
    const uint64_t dy0 = g.rby == 16 ? smem_desc_rb(0, 128, g.yblk, 16) : smem_desc_rb(0, g.yblk, 8 * g.rby, g.rby);
    const uint32_t sa = g.rby, sb = g.gw == 64 ? g.rb : g.gw == 16 ? g.strip_bytes >> 4 : g.strip_bytes >> 3;  // 16 pixels on
    Ring r;
    bool issued = false;
    uint32_t more = 0;
    int x = SEG ? t0 * kKP - fast_div(t0 * kKP, g.fw) * g.W : 0;
    for (int t = t0; t < t1; r.next(g.nst)) {
      ok = warp_wait(&xfull[warp & 1][r.s], r.ph, g.spins, &gave_up) && warp_wait(&yfull[r.s], r.ph, g.spins, &gave_up);
      if (!ok) break;
      tc_fence_after();
      uint32_t st = base + r.s * g.stage_bytes;
      for (const int te = min(t + g.kpm, t1); t < te; ++t, st += g.blk_bytes) {
        const uint64_t da = dy0 + ((st + y_off) >> 4);
        const int c = SEG ? (g.W - x) >> 3 : 8;  // K groups up to the end of the row
        if (SEG && c < kKP / 8) {
          // the others lie in the second strip; the MMA across the end has its two a strip apart
          const uint32_t back = g.strip_bytes - c * kg;
          const uint32_t over = back + kg;
          const uint64_t dxo = g.rb == 16 ? smem_desc_rb(0, over, 16, 16) : smem_desc_rb(0, g.rb, over, g.rb);
          for (int u = warp; u < nu; u += 4)
            for (int j = 0; j < 4; ++j) {
              const uint32_t at = st + u * g.unit_bytes + 2 * j * kg + (2 * j >= c ? back : 0);
              mma_warp<1>(tmem + u * g.nmma, da + j * sa, (2 * j + 1 == c ? dxo : dx0) + (at >> 4), idesc,
                          more | (j > 0));
            }
        } else {
          for (int u = warp; u < nu; u += 4)
            mma_warp<4>(tmem + u * g.nmma, da, dx0 + ((st + u * g.unit_bytes) >> 4), idesc, more, sa, sb);
        }
        if (SEG && (x += kKP) >= g.W) x -= g.W;
        more = 1;
      }
      mma_commit_warp(smem_u32(&empty[r.s]));
      issued = true;
    }
    // every MMA issued so far, also on the way out of a wait that gave up
    if (issued) {
      mma_commit_warp(smem_u32(&done[warp]));
      if (!mbar_wait(smem_u32(&done[warp]), 0, kDrainSpins)) ok = false;
    }
  }
  if (!ok) atomicOr(&gave_up, 1);
  __syncwarp();
  __syncthreads();
  tc_fence_after();
  if (gave_up && tid == 0 && g.status) atomicOr(g.status, 1);
  if (!gave_up && warp < 4) {
    // 64-row accumulators lie in lanes 0-15 of each warp's 32
    const int co = g.mrows == 64 ? (lane < 16 ? m0 + warp * 16 + lane : g.Cout) : m0 + warp * 32 + lane;
    for (int u = 0; u < nu; ++u) {
      const int dy = (u0 + u) / g.nblk, c = (u0 + u) % g.nblk;
      for (int k = 0; k < g.ndx * g.chb; k += 16) {  // columns: dx, channel of the block
        float v[16];
        tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(u * g.nmma + k), v);
        if (t1 <= t0)
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = 0.0f;
        if (g.chb >= 16) {
          store_part(g, co, (size_t)(dy * 3 + k / g.chb) * g.Cin + c * g.chb + k % g.chb, v, 16);
        } else {  // 8 channels: two taps
          float w[16];
#pragma unroll
          for (int i = 0; i < 8; ++i) w[i] = v[i + 8];
          store_part(g, co, (size_t)(dy * 3 + k / 8) * g.Cin + c * 8, v, 8);
          if (k + 8 < g.ndx * 8) store_part(g, co, (size_t)(dy * 3 + k / 8 + 1) * g.Cin + c * 8, w, 8);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(g.cols));
}

// LAG: copy groups a producer keeps in flight behind the one it just issued.
template <int LAG>
__global__ void __launch_bounds__(kWgThreads) wgrad_gather_kernel(WgradArgs g) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint64_t full[kMaxStages], empty[kMaxStages], done;
  __shared__ uint32_t tmem_slot;
  __shared__ int gave_up;
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  // unit: (output-channel block, input-channel block, tap group)
  int u = blockIdx.x;
  const int tg = u % g.G;
  u /= g.G;
  const int n0 = (u % g.NB) * g.Nb, m0 = (u / g.NB) * 128;
  const int tap0 = tg * g.ntap, ntap = min(g.ntap, g.taps - tap0);
  const int t0 = (int)((long long)g.nkb * blockIdx.y / g.S), t1 = (int)((long long)g.nkb * (blockIdx.y + 1) / g.S);
  const int ncx = min(g.Nb, g.Cin - n0) >> 3;                 // 8-channel chunks of X staged
  const int ncy = (min(128, g.Cout - m0) + 7) >> 3;           // and of dY

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
  bool ok = true;

  if (warp < 8) {  // producers: warp w stages pixels 8w .. 8w+7 of the block, consecutive lanes consecutive chunks
    const int nx = ntap * 8 * ncx, ny = 8 * ncy;
    // a lane's copies are 32 apart: (position, chunk) advances by (q, r)
    const int qx = 32 / ncx, rx = 32 % ncx, px0 = lane / ncx, cx0 = lane % ncx;
    const int qy = 32 / ncy, ry = 32 % ncy, py0 = lane / ncy, cy0 = lane % ncy;
    const int hw = g.H * g.W;
    Ring r, a;        // the stage being filled, the oldest not yet announced
    int pending = 0;  // stages issued and not yet announced
    for (int t = t0; t < t1; ++t, r.next(g.nst)) {
      if (t - t0 >= g.nst) ok = role_wait(&empty[r.s], r.ph ^ 1u, g.spins, &gave_up);
      if (!ok) break;
      const uint32_t sx = base + r.s * g.stage_bytes + warp * 128;
      const uint32_t sy = sx + (g.Nb >> 3) * g.sxc;
      const int p = t * kKP + warp * 8;
#pragma unroll 2
      for (int i = lane, pos = px0, c = cx0; i < nx; i += 32) {
        const int j = pos >> 3, o = pos & 7, tap = tap0 + j;
        const int b = fast_div(p + o, g.fhw), q = p + o - b * hw, yc = fast_div(q, g.fw);
        const int y = yc + tap / 3 - 1, x = q - yc * g.W + tap % 3 - 1;
        const bool in = p + o < g.P && (unsigned)y < (unsigned)g.H && (unsigned)x < (unsigned)g.W;
        const __nv_bfloat16 *src = in ? g.X + (size_t)(b * hw + y * g.W + x) * g.Cin + n0 + c * 8 : g.X;
        cp_async16(sx + c * g.sxc + (j * kKP + o) * 16, src, in);
        pos += qx;
        c += rx;
        if (c >= ncx) c -= ncx, ++pos;
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
        mbar_arrive(smem_u32(&full[a.s]));
        a.next(g.nst);
        --pending;
      }
    }
    cp_async_wait<0>();
    fence_proxy_async();
    for (; ok && pending > 0; --pending, a.next(g.nst)) mbar_arrive(smem_u32(&full[a.s]));
  } else {  // MMAs
    const uint32_t idesc = instr_desc_mn(g.Nb, g.mrows);
    // descriptors of stage 0; an address advances by its bytes / 16
    const uint64_t da0 = smem_desc(base + (g.Nb >> 3) * g.sxc, 128, g.syc), db0 = smem_desc(base, 128, g.sxc);
    Ring r;
    bool issued = false;
    for (int t = t0; t < t1; ++t, r.next(g.nst)) {
      ok = warp_wait(&full[r.s], r.ph, g.spins, &gave_up);
      if (!ok) break;
      tc_fence_after();
      const uint32_t st = (uint32_t)(r.s * g.stage_bytes) >> 4;
      for (int j = 0; j < ntap; ++j)
        mma_warp<4>(tmem + j * g.Nb, da0 + st, db0 + (st + j * kKP), idesc, t > t0, 16, 16);
      mma_commit_warp(smem_u32(&empty[r.s]));
      issued = true;
    }
    // every MMA issued so far, also on the way out of a wait that gave up
    if (issued) {
      mma_commit_warp(smem_u32(&done));
      if (!mbar_wait(smem_u32(&done), 0, kDrainSpins)) ok = false;
    }
  }
  if (!ok) atomicOr(&gave_up, 1);
  __syncwarp();
  __syncthreads();
  tc_fence_after();
  if (gave_up && tid == 0 && g.status) atomicOr(g.status, 1);
  if (!gave_up && warp < 4) {
    const int co = g.mrows == 64 ? (lane < 16 ? m0 + warp * 16 + lane : g.Cout) : m0 + warp * 32 + lane;
    for (int j = 0; j < ntap; ++j)
#pragma unroll 1
      for (int c0 = 0; c0 < (ncx << 3); c0 += 16) {
        float v[16];
        tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(j * g.Nb + c0), v);
        if (t1 <= t0)
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = 0.0f;
        store_part(g, co, (size_t)(tap0 + j) * g.Cin + n0 + c0, v, (ncx << 3) - c0);
      }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(g.cols));
}

// Bias gradient: block b sums its range of pixels of dY [P][C] per channel.  A
// thread takes 8 channels of every (threads / (C/8))-th pixel, 16 of them in float
// (8 significant bits each) and those sums in double; the block's threads and
// then the blocks (wgrad_reduce_kernel) are added in order.
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
#pragma unroll 8
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

// dW[i] = sum_s part[s][i], s ascending (part is [S][n]), in the first nw blocks;
// the others take db[c] = sum over blocks b of cpart[b][c], a warp per channel,
// lanes 32 blocks apart, then a fixed butterfly (one thread per channel was a
// chain of 592 loads, 32 us).
__global__ void __launch_bounds__(256) wgrad_reduce_kernel(const float *__restrict__ part, int S, size_t n,
                                                           float *__restrict__ dW, int nw,
                                                           const double *__restrict__ cpart, int nblk, int C, int ld,
                                                           float *__restrict__ db) {
  if ((int)blockIdx.x < nw) {
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    float acc = 0.0f;
#pragma unroll 8
    for (int s = 0; s < S; ++s) acc += __ldg(part + (size_t)s * n + i);
    dW[i] = acc;
    return;
  }
  const int c = (blockIdx.x - nw) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (c >= C) return;  // warp-uniform
  double s = 0.0;
#pragma unroll 4
  for (int b = lane; b < nblk; b += 32) s += __ldg(cpart + (size_t)b * ld + c);
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

int row_bytes(int c) { return c % 64 == 0 ? 128 : c % 32 == 0 ? 64 : c % 16 == 0 ? 32 : 16; }

// What a CTA of either kernel accumulates is limited by TMEM's 512 columns;
// fewer units (taps) to a CTA stage less per MMA but give more CTAs: the most
// that fit, or as many fewer as it takes to have 90 CTAs (4 x 192^2, 128 ->
// 128: 96 CTAs in one wave took 0.17 ms with the gather kernel, 160 in two 0.21).
constexpr int kMinCtas = 90;

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
  g.mrows = Cout <= 64 ? 64 : 128;
  const int MB = (Cout + 127) / 128;
  g.cols = 32;
  if (taps == 1 || W % 8 == 0) {
    g.rb = row_bytes(Cin);
    g.chb = g.rb / 2;
    g.nblk = Cin / g.chb;
    g.ndx = taps == 9 ? 3 : 1;
    g.nmma = (g.ndx * g.chb + 15) / 16 * 16;
    g.U = g.ndx * g.nblk;
    g.upg = std::min(g.U, 512 / g.nmma);
    while (g.upg > 1 && MB * ((g.U + g.upg - 1) / g.upg) * g.S < kMinCtas) --g.upg;
    g.rby = row_bytes(g.ldY);
    g.chby = g.rby / 2;
    g.nby = (std::min(g.ldY, 128) + g.chby - 1) / g.chby;
    g.yblk = kKP * g.rby;
    const int halo = g.ndx >> 1;
    // a strip of 64 pixels, and a second one where a row ends among them; images
    // narrower than that take strips of 16 or 8 (a TMA box costs some 250 clocks,
    // whatever its rows: 4 x 760^2, 32 -> 32 in strips of 8 took 1.02 ms, now 0.24)
    g.gw = taps == 1 || W >= 64 ? 64 : W % 16 == 0 ? 16 : 8;
    g.seg = taps == 9 && W >= 64 && W % 64;
    g.strip_bytes = ((g.gw + 2 * halo) * g.rb + 1023) / 1024 * 1024;
    g.unit_bytes = (g.seg ? 2 : kKP / g.gw) * g.strip_bytes;
    for (;; --g.upg) {  // two stages at least
      g.stage_bytes = g.upg * g.unit_bytes + g.nby * g.yblk;
      // an MMA reads mrows rows of dY whatever Cout: blocks behind the staged
      // ones are other bytes of the allocation, and feed accumulator rows that
      // nothing reads
      g.tail_bytes = std::max(0, g.mrows / g.chby - g.nby) * g.yblk;
      if (2 * g.stage_bytes + g.tail_bytes <= kSmemMax || g.upg == 1) break;
    }
    g.G = (g.U + g.upg - 1) / g.upg;
    while (g.cols < g.upg * g.nmma) g.cols *= 2;
  } else {
    g.NB = (Cin + 255) / 256;
    g.Nb = ((Cin + g.NB - 1) / g.NB + 15) / 16 * 16;
    g.NB = (Cin + g.Nb - 1) / g.Nb;
    g.Mb = std::min(Cout, 128);
    g.ntap = std::min(taps, 512 / g.Nb);
    while (g.ntap > 1 && MB * g.NB * ((taps + g.ntap - 1) / g.ntap) * g.S < kMinCtas) --g.ntap;
    g.G = (taps + g.ntap - 1) / g.ntap;
    g.ntap = (taps + g.G - 1) / g.G;
    // one 16-byte unit of padding per chunk spreads the copies over the banks
    g.syc = kKP * 16 + 16;
    for (;; --g.ntap) {
      g.sxc = g.ntap * kKP * 16 + 16;
      g.stage_bytes = (g.Nb / 8) * g.sxc + ((g.Mb + 7) / 8) * g.syc;
      g.tail_bytes = (g.mrows / 8 - (g.Mb + 7) / 8) * g.syc;
      if (2 * g.stage_bytes + g.tail_bytes <= kSmemMax || g.ntap == 1) break;
    }
    g.G = (taps + g.ntap - 1) / g.ntap;
    while (g.cols < g.ntap * g.Nb) g.cols *= 2;
  }
  const int ctas = MB * (g.NB ? g.NB : 1) * g.G * g.S;
  // two CTAs to an SM when there are more than one for each
  int budget = ctas > kSms && 2 * g.cols <= 512 ? kSmemMax / 2 - 1024 : kSmemMax;
  if (3 * g.stage_bytes + g.tail_bytes > budget) budget = kSmemMax;
  // A stage of the TMA kernel is up to 4 blocks, as long as there are three
  // stages (32 -> 32 at 768^2: 331 us with one, 267 with two, 235 with four).
  g.blk_bytes = g.stage_bytes;
  g.kpm = 1;
  while (g.rb && g.kpm < 4 && 3 * 2 * g.kpm * g.blk_bytes + g.tail_bytes <= budget) g.kpm *= 2;
  g.stage_bytes = g.kpm * g.blk_bytes;
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
  const int smem = 1024 + g.nst * g.stage_bytes + g.tail_bytes, MB = (Cout + 127) / 128;
  if (g.rb) {
    CUtensorMap mx, my;
    const unsigned long long uc = Cin, up = P, ul = g.ldY;
    const unsigned long long dx[4] = {uc, taps == 9 ? (unsigned long long)W : up, taps == 9 ? (unsigned long long)H : 1ull,
                                      taps == 9 ? (unsigned long long)batch : 1ull};
    const unsigned long long sx[3] = {2 * uc, 2 * uc * dx[1], 2 * uc * dx[1] * dx[2]};
    const unsigned bx[4] = {(unsigned)g.chb, (unsigned)(g.gw + g.ndx - 1), 1, 1};
    if (int rc = make_tensor_map(&mx, X, 4, dx, sx, bx, g.rb)) return rc;
    const unsigned long long dy[3] = {ul, up, 1}, sy[2] = {2 * ul, 2 * ul * up};
    const unsigned by[3] = {(unsigned)g.chby, kKP, 1};
    if (int rc = make_tensor_map(&my, dY, 3, dy, sy, by, g.rby)) return rc;
    auto fn = g.seg ? wgrad_tma_kernel<true> : wgrad_tma_kernel<false>;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return NN_ECUDA;
    fn<<<dim3(MB * g.G, g.S), 224, smem, s>>>(g, mx, my);
  } else {
    const int lag = g.nst >= 7 ? 5 : g.nst >= 5 ? 3 : g.nst >= 3 ? 2 : 1;
    auto fn = lag == 5   ? wgrad_gather_kernel<5>
              : lag == 3 ? wgrad_gather_kernel<3>
              : lag == 2 ? wgrad_gather_kernel<2>
                         : wgrad_gather_kernel<1>;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return NN_ECUDA;
    fn<<<dim3(MB * g.NB * g.G, g.S), kWgThreads, smem, s>>>(g);
  }
  const size_t nout = (size_t)taps * Cin * Cout;
  double *cp = (double *)(w + ww.colsum);
  const int nblk = (int)std::min<long long>(kColBlocks, std::max<long long>(1, P / 64)), nw = (int)((nout + 255) / 256);
  if (db) colsum_kernel<<<nblk, kColThreads, 0, s>>>(dY, P, g.ldY, cp);
  wgrad_reduce_kernel<<<nw + (db ? (Cout + 7) / 8 : 0), 256, 0, s>>>(g.part, g.S, nout, dW, nw, cp, nblk, Cout, g.ldY, db);
  return cudaGetLastError() == cudaSuccess ? NN_OK : NN_ECUDA;
}

}  // namespace tomo_nn
