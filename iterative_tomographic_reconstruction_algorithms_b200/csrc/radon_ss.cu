// Slant-stacking projector pair (linear interpolation) for sm_100a.
//
// Reference: common/operators/radon_module/pymodule_radon_slant_stacking/
// radon_ss.c:93-196 (method 1) with ray_limits :43-88.  For each angle and
// detector offset t in [-nh, nh) the reference steps along the major axis of
// the ray -- y when |sin| <= sqrt(1/2), else x -- over the integer range
// [round(lim_lo), round(lim_hi)) that ray_limits returns, interpolates the
// image linearly across the minor axis and weights by 1/|cos| or 1/|sin|.
// The output row is na - 1 - v.
//
// Evaluation order of the compiled reference (-O3 -ffast-math, read from its
// x86-64 code): minor coordinate f = fma(-m, s, t) * (1/c) (or fma(-m, c, t) *
// (1/s)), weights w = f - floor(f) and (floor(f) + 1) - f, limits
// fma(nh, s, t) / c etc. sorted.  The loop bounds are precomputed per (angle,
// t) on the host in that exact arithmetic (ss_setup) and shared by both
// kernels.
//
// Rays that miss the square [-nh, nh-1]^2 (possible only within about 1/nh
// radian of 180 degrees) make the reference index outside the image; here
// those rows are skipped.
#include <algorithm>
#include <cmath>

#include "f32x2.cuh"
#include "tomo_internal.cuh"

namespace tomo {
namespace {

constexpr double kS45 = 0.70710678118654757;

constexpr float kSsMagic = 12582912.0f;  // 1.5 * 2^23
constexpr int kSsMagicBits = 0x4B400000;  // its bit pattern
constexpr int kSsFrame = 4;

// Framed copies of the image: rows[y][P + x] and cols[x][P + y], with P =
// kSsFrame zeros on either side of a line.
__global__ void __launch_bounds__(256) ss_frame_kernel(const float *__restrict__ img, float *__restrict__ rows,
                                                       float *__restrict__ cols, int n) {
  __shared__ float tile[32][33];
  const size_t z = blockIdx.z;
  const int w = n + 2 * kSsFrame;
  const float *src = img + z * (size_t)n * n;
  float *R = rows + z * (size_t)n * w, *C = cols + z * (size_t)n * w;
  const int x0 = blockIdx.x * 32 - kSsFrame, y0 = blockIdx.y * 32 - kSsFrame;  // tiles cover the frame too
  for (int dy = threadIdx.y; dy < 32; dy += 8) {
    const int y = y0 + dy, x = x0 + threadIdx.x;
    const float v = y >= 0 && y < n && x >= 0 && x < n ? __ldg(src + (size_t)y * n + x) : 0.0f;
    tile[dy][threadIdx.x] = v;
    if (y >= 0 && y < n && x < n + kSsFrame) R[(size_t)y * w + kSsFrame + x] = v;
  }
  __syncthreads();
  for (int dy = threadIdx.y; dy < 32; dy += 8) {
    const int x = x0 + dy, y = y0 + threadIdx.x;
    if (x >= 0 && x < n && y < n + kSsFrame) C[(size_t)x * w + kSsFrame + y] = tile[threadIdx.x][dy];
  }
}

// Forward: a lane owns a ray (t, angle, slice) and steps along its major axis;
// a step interpolates across the minor one (steep rays: in an image row, else
// in a column, i.e. a row of the transposed copy, so that neighbouring lanes
// read neighbouring words).  The frame stands in for bounds tests, the angle's
// factor wt is applied once.  SPLIT warps share a ray's steps and are added in
// order: small images have too few rays to hide a step's latency (256^2 x 200:
// 61 us unsplit, now 18; 768^2 x 720: 0.58 ms unsplit, 0.38 by two); the split
// depends on n alone (ss_fwd_split).  SPLIT = 0 is the solvers' form
// (epilogue.cuh): one chain, the weight wt w rounded before each product.
// 4 x 641^2 x 600: 1.28 ms with bounds tests and weights per step, now 0.78;
// 2048^2 x 1800: 9.6, now 6.3.
template <int SPLIT>
__global__ void __launch_bounds__(128) ss_forward_kernel(const float *__restrict__ rows, const float *__restrict__ cols,
                                                         float *__restrict__ sino, const SsAngle *__restrict__ tab,
                                                         const int2 *__restrict__ lim, int n, int nh, int na, FwdEpi ep) {
  __shared__ float part[SPLIT > 1 ? SPLIT : 1][128];
  constexpr int kParts = SPLIT > 1 ? SPLIT : 1, kRays = 128 / kParts;
  const int lane = threadIdx.x % kRays, q = threadIdx.x / kRays;  // kRays is a multiple of 32: q is warp-uniform
  const int kt = blockIdx.x * kRays + lane;  // t + nh
  const int v = blockIdx.y;
  const size_t z = blockIdx.z;
  const bool live = kt < n;  // kt == 2nh (odd n) is never reached by a ray: stays 0
  const SsAngle g = tab[v];
  const int2 L = kt < 2 * nh ? lim[(size_t)v * (2 * nh) + kt] : make_int2(0, 0);
  int m0 = max(L.x, -nh), m1 = min(L.y, n - nh);  // rays that miss the square may leave it
  if (SPLIT > 1) {
    const int len = max(0, m1 - m0), s0 = m0;
    m0 = s0 + len * q / kParts;
    m1 = s0 + len * (q + 1) / kParts;
  }
  const int w = n + 2 * kSsFrame;
  const float ft = (float)(kt - nh), lo = (float)(-nh) - 2.0f, hi = (float)(n - nh) + 1.0f;
  const float *row = (g.steep ? rows : cols) + z * (size_t)n * w + (ptrdiff_t)(m0 + nh) * w + kSsFrame + nh - kSsMagicBits;
  float nm = (float)(-m0), acc = 0.0f;
#pragma unroll 4
  for (int m = m0; m < m1; ++m, nm -= 1.0f, row += w) {
    const float f = fminf(fmaxf(__fmul_rn(__fmaf_rn(nm, g.a, ft), g.rb), lo), hi);
    const float fd = __fadd_rd(f, kSsMagic);  // floor(f), as a float among the integers and in its bits
    const float fl = __fsub_rn(fd, kSsMagic), wq = __fsub_rn(f, fl);
    const float *p = row + __float_as_int(fd);
    const float w1 = __fsub_rn(__fadd_rn(fl, 1.0f), f);  // not 1 - wq: that loses the last bits of |f| < 1
    acc = fmaf(SPLIT ? w1 : __fmul_rn(g.wt, w1), __ldg(p), acc);
    acc = fmaf(SPLIT ? wq : __fmul_rn(g.wt, wq), __ldg(p + 1), acc);
  }
  if (SPLIT > 1) {
    part[q][lane] = acc;
    __syncthreads();
    if (q > 0) return;  // warp-uniform
    for (int k = 1; k < SPLIT; ++k) acc += part[k][lane];
  }
  if (SPLIT) acc *= g.wt;
  double r2 = 0.0;
  const size_t e = z * (size_t)na * n + (size_t)g.out_row * n + kt;
  if (live) sino[e] = fwd_apply(ep, acc, e, r2);
  const size_t block = ((size_t)z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  fwd_resid_commit(ep, r2, block * (kRays / 32) + lane / 32);
}

// ms with 2, 4 warps: 256^2 x 300 0.040, 0.038; 448^2 x 450 0.108, 0.099; 640^2 x 600 0.235,
// 0.233; 768^2 x 720 0.374, 0.378; 2048^2 x 1800 6.18, 6.40; several slices want fewer (4 x 641^2
// x 600: 0.781, 0.851; 8 x 256^2 x 300: 0.149, 0.151), but a slice has the same bits in any
// call.
int ss_fwd_split(int n) { return n > 448 ? 2 : 4; }

// Sinogram rows as pairs in the order of the angles, entry e = t + nh + pads of
// angle v: wt {S_t, S_t+1}, 0 outside the rays.  A row where one of these is not
// finite keeps {S_t, S_t+1} and is marked in raw[z][v] (as all are: ordered).
__global__ void __launch_bounds__(256) ss_expand_kernel(const float *__restrict__ sino, float2 *__restrict__ out,
                                                        int *__restrict__ raw, const SsAngle *__restrict__ tab, int n, int nh,
                                                        int na, int pads, int w2, bool ordered) {
  const int v = blockIdx.x;
  const size_t z = blockIdx.y;
  const SsAngle g = tab[v];
  const float *src = sino + (z * na + g.out_row) * (size_t)n;
  float2 *dst = out + (z * na + v) * (size_t)w2;
  bool bad = ordered;
  for (int t = threadIdx.x; t < 2 * nh; t += blockDim.x) bad |= !(fabsf(g.wt * __ldg(src + t)) < INFINITY);
  bad = __syncthreads_or(bad);
  if (threadIdx.x == 0) raw[z * na + v] = bad;
  const float wt = bad ? 1.0f : g.wt;
  for (int e = threadIdx.x; e < w2; e += blockDim.x) {
    const int t = e - pads;
    dst[e] = make_float2(t >= 0 && t < 2 * nh ? wt * __ldg(src + t) : 0.0f,
                         t + 1 >= 0 && t + 1 < 2 * nh ? wt * __ldg(src + t + 1) : 0.0f);
  }
}

// Adjoint: a lane holds 4 x 4 pixels of a 32 x 16 tile; warp q of a block's Q
// sums every Q-th angle from q on (the costlier angles near an axis go to all),
// and the sums are added in order.  Q depends on n alone.  Q = 1 is the solvers'
// form (epilogue.cuh): one chain, the weight wt w rounded before each product.
//
// At a pixel's major coordinate m the rays' minor coordinates f(t) = fma(-m, a,
// t) * rb lie |rb| = 1 / |cb| >= 1 apart, so a ray within 1 of the pixel's minor
// coordinate c is within |cb| <= 1 of the crossing t* of c: it is floor(t*) or
// the next.  It reaches c if f is in [c - 1, c + 1), with the forward's weight wt (f
// - floor f) or wt (floor f + 1 - f), which are wt (1 - |f - c|) but for the bits that f
// has below those of c = +-1 (BOTH, ss_centre).  A rounding of t* across an integer loses
// nothing while |cb| < 1 by more than that rounding (below n 2^-22 in all); the few
// angles nearer to an axis (NEAR) look at the rays before and behind too.  The two
// rays come as one pair, evaluated as packed operations.
//
// For finite values a ray with weight 0 can be passed by, and wt be applied to the
// value; an infinite value makes NaN of a weight of 0, and wt S may overflow where
// wt w S does not.  The rows where that matters are marked (raw) and go through
// ss_adj_raw.
//
// The ray's own limits (EDGE) matter only next to the border: at a pixel 4 or
// more inside the square both rays are inside it.
//
// Bound by FP32 and issue.  Candidate rays checked one by one against their
// limits, each credited to 4 pixels by 8 tests, took 3.53 ms at 4 x 641^2 x
// 600 and 18.1 at 2048^2 x 1800; this takes 1.19 and 6.8 (with the reference's products
// throughout half as long again).

// Whether ray t passes major coordinate m (without branches: the loads of a
// block's rays overlap).
__device__ __forceinline__ bool ss_in_limits(const int2 *__restrict__ lrow, int t, int m, int nh) {
  const int2 l = __ldg(lrow + min(max(t, -nh), nh - 1) + nh);
  return (t >= -nh) & (t < nh) & (m >= l.x) & (m < l.y);
}

// o += wt w S for the ray at f and the pixel at c, if it reaches it and `in`, as the
// reference has it: wt w is rounded, and a weight of 0 counts.
__device__ __forceinline__ void ss_credit(float &o, float f, float c, float wt, float S, bool in) {
  const float u = __fsub_rn(f, c - 1.0f), v = __fsub_rn(c + 1.0f, f);
  if ((u >= 0.0f) & (v > 0.0f) & in) o = fmaf(__fmul_rn(wt, fminf(u, v)), S, o);
}

// o + a marked row's credits to pixel (R, C); row: its pair at t = -nh.
__device__ __noinline__ float ss_adj_raw(float o, const SsAngle *__restrict__ tab, const float2 *__restrict__ row,
                                         const int2 *__restrict__ lrow, int R, int C, int nh) {
  const SsAngle g = *tab;
  const int mi = (g.steep ? R : C) - nh, ci = (g.steep ? C : R) - nh;
  const float m = (float)mi, c = (float)ci, t0 = floorf(fmaf(c, 1.0f / g.rb, m * g.a));
#pragma unroll 1
  for (int k = -1; k <= 2; ++k) {
    const int t = (int)t0 + k;
    ss_credit(o, __fmul_rn(__fmaf_rn(-m, g.a, t0 + (float)k), g.rb), c, g.wt, __ldg(row + nh + t).x, ss_in_limits(lrow, t, mi, nh));
  }
  return o;
}

// What a row's credits to pixel (m, c), |c| = 1, lack: its rays' weights as f - floor f
// or floor f + 1 - f, less those that the main loop takes, times wt S.
__device__ __forceinline__ float ss_centre(const SsAngle &g, const float2 *__restrict__ row, const int2 *__restrict__ lrow,
                                           int mi, int ci, int nh, bool limits, bool near) {
  const float m = (float)mi, c = (float)ci, fm = __fadd_rd(fmaf(c, 1.0f / g.rb, m * g.a), kSsMagic), t0 = __fsub_rn(fm, kSsMagic);
  const int ti = __float_as_int(fm) - kSsMagicBits;
  float o = 0.0f;
  auto ray = [&](int k, float S) {
    const float f = __fmul_rn(__fmaf_rn(-m, g.a, t0 + (float)k), g.rb);
    const float h = fminf(__fsub_rn(f, c - 1.0f), __fsub_rn(c + 1.0f, f)), q = 1.0f - fabsf(__fsub_rn(f, c));
    if ((fmaxf(h, q) > 0.0f) & (!limits || ss_in_limits(lrow, ti + k, mi, nh))) o = fmaf(fmaxf(h, 0.0f) - fmaxf(q, 0.0f), S, o);
  };
  const float2 S = __ldg(row + nh + ti);
  ray(0, S.x);
  ray(1, S.y);
  if (near) {
    ray(-1, __ldg(row + nh + ti - 1).x);
    ray(2, __ldg(row + nh + ti + 1).y);
  }
  return o;
}

template <bool STEEP, bool EDGE, bool NEAR, bool ORD, bool BOTH>
__device__ __forceinline__ void ss_adj_angle(const SsAngle &g, const float2 *__restrict__ row, const int2 *__restrict__ lrow,
                                             int a0, int b0, int nh, float (&acc)[4][4]) {
  const int M0 = (STEEP ? a0 : b0) - nh, C0 = (STEEP ? b0 : a0) - nh;  // major and minor coordinates of the block
  const float cb = 1.0f / g.rb, wt = g.wt;
  const F2 rb = f2(g.rb), a = f2(g.a), step = f2(0.0f, 1.0f);
#pragma unroll
  for (int i = 0; i < 4; ++i) {  // along the major axis
    const float m = (float)(M0 + i), ma = m * g.a;
    const F2 nm = f2(-m);
#pragma unroll
    for (int j = 0; j < 4; ++j) {  // along the minor axis
      const float c = (float)(C0 + j);
      const float fm = __fadd_rd(fmaf(c, cb, ma), kSsMagic);  // first ray
      const float2 S = __ldg(row + __float_as_int(fm));
      const F2 t = add2(f2(__fsub_rn(fm, kSsMagic)), step);
      const float2 f = unpack(mul2(fma2(nm, a, t), rb));  // scalar from here: see f32x2.cuh
      const int ti = __float_as_int(fm) - kSsMagicBits;
      float &o = STEEP ? acc[i][j] : acc[j][i];
      // as the reference has it (ORD), or on finite rows that hold wt S
      auto credit = [&](float f, float S, bool in) {
        if (ORD) {
          ss_credit(o, f, c, wt, S, in);
        } else {
          const float h = BOTH ? fminf(__fsub_rn(f, c - 1.0f), __fsub_rn(c + 1.0f, f)) : 1.0f - fabsf(__fsub_rn(f, c));
          if ((h > 0.0f) & in) o = fmaf(h, S, o);
        }
      };
      auto before_or_behind = [&](int k) {
        const float f = __fmul_rn(__fmaf_rn(-m, g.a, __fsub_rn(fm, kSsMagic) + (float)k), g.rb);
        credit(f, k < 0 ? __ldg(row + __float_as_int(fm) - 1).x : __ldg(row + __float_as_int(fm) + 1).y,
               !EDGE || ss_in_limits(lrow, ti + k, M0 + i, nh));
      };
      if (NEAR) before_or_behind(-1);
      const bool in0 = EDGE ? ss_in_limits(lrow, ti, M0 + i, nh) : true, in1 = EDGE ? ss_in_limits(lrow, ti + 1, M0 + i, nh) : true;
      credit(f.x, S.x, in0);
      credit(f.y, S.y, in1);
      if (NEAR) before_or_behind(2);
    }
  }
}

// Q = 4: 28 warps per SM (72 registers) take 6.7 ms at 2048^2 x 1800, 32 (64, with 12
// bytes spilled) 6.8.
template <int Q, bool BOTH>
__global__ void __launch_bounds__(32 * Q, (Q == 1 ? 0 : Q == 4 ? 28 : 32) / Q) ss_adjoint_kernel(const float2 *__restrict__ pairs,
                                                            const int *__restrict__ raw, float *__restrict__ img,
                                                            const SsAngle *__restrict__ tab, const int2 *__restrict__ lim,
                                                            int n, int nh, int na, int pads, int w2, AdjEpi ep) {
  __shared__ float part[Q > 1 ? (Q - 1) * 16 : 1][32];
  __shared__ float centre[Q > 1 && !BOTH ? Q : 1][3][32];  // what the tile's pixels with |c| = 1 lack: two half columns, two rows
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
  // the tiles of the border take longest: both border rows of tiles first
  const int by = blockIdx.y == 0 ? 0 : blockIdx.y == 1 ? gridDim.y - 1 : blockIdx.y - 1;
  const int b0 = blockIdx.x * 32 + 4 * (lane & 7), a0 = by * 16 + 4 * (lane >> 3);
  const size_t z = blockIdx.z;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
  // the tile's pixels are all 4 or more inside the square [0, 2 nh - 1]
  const bool edge = blockIdx.x * 32 < 4 || by * 16 < 4 || blockIdx.x * 32 + 36 > 2 * nh || by * 16 + 20 > 2 * nh;
  const float near = 1.0f - (float)n * 0x1p-22f;
  bool marked = false;  // rows of this warp's share
  if (Q > 1) {
    for (int u = q + Q * lane; u < na; u += Q * 32) marked |= __ldg(raw + z * na + u) != 0;
    marked = __any_sync(0xffffffffu, marked);
  }
  if (a0 < n && b0 < n) {
    const float2 *row = pairs + (z * na + q) * (size_t)w2 + pads + nh - kSsMagicBits;
    const int2 *lrow = lim + (size_t)q * 2 * nh;
#pragma unroll 1
    for (int u = q; u < na; u += Q, row += (size_t)Q * w2, lrow += (size_t)Q * 2 * nh) {
      const SsAngle g = tab[u];
      const bool nr = fabsf(g.rb) * near < 1.0f;
      if (marked && __ldg(raw + z * na + u)) continue;
      if (nr) {
        if (g.steep) ss_adj_angle<true, true, true, Q == 1, BOTH>(g, row, lrow, a0, b0, nh, acc);
        else ss_adj_angle<false, true, true, Q == 1, BOTH>(g, row, lrow, a0, b0, nh, acc);
      } else if (edge) {
        if (g.steep) ss_adj_angle<true, true, false, Q == 1, BOTH>(g, row, lrow, a0, b0, nh, acc);
        else ss_adj_angle<false, true, false, Q == 1, BOTH>(g, row, lrow, a0, b0, nh, acc);
      } else {
        if (g.steep) ss_adj_angle<true, false, false, Q == 1, BOTH>(g, row, lrow, a0, b0, nh, acc);
        else ss_adj_angle<false, false, false, Q == 1, BOTH>(g, row, lrow, a0, b0, nh, acc);
      }
    }
    if (marked)
#pragma unroll 1
      for (int u = q; u < na; u += Q)
        if (__ldg(raw + z * na + u))
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
              acc[i][j] = ss_adj_raw(acc[i][j], tab + u, pairs + (z * na + u) * (size_t)w2 + pads, lim + (size_t)u * 2 * nh,
                                     a0 + i, b0 + j, nh);
  }
  // the columns nh - 1 and nh + 1 of the tile for steep angles, a pixel a lane; the
  // rows for the others
  const int X0 = blockIdx.x * 32, Y0 = by * 16;
  const bool midx = X0 <= nh + 1 && X0 + 31 >= nh - 1, midy = Y0 <= nh + 1 && Y0 + 15 >= nh - 1;
  if (Q > 1 && !BOTH && (midx || midy)) {
    float cc = 0.0f, r0 = 0.0f, r1 = 0.0f;
    const int R = Y0 + (lane & 15), side = lane < 16 ? -1 : 1, C = X0 + lane;
#pragma unroll 2
    for (int u = q; u < na; u += Q) {
      if (marked && __ldg(raw + z * na + u)) continue;
      const SsAngle g = tab[u];
      const float2 *row = pairs + (z * na + u) * (size_t)w2 + pads;
      const int2 *lrow = lim + (size_t)u * 2 * nh;
      const bool nr = fabsf(g.rb) * near < 1.0f, limits = edge || nr;
      if (g.steep) {
        if (midx) cc += ss_centre(g, row, lrow, R - nh, side, nh, limits, nr);
      } else if (midy) {
        r0 += ss_centre(g, row, lrow, C - nh, -1, nh, limits, nr);
        r1 += ss_centre(g, row, lrow, C - nh, 1, nh, limits, nr);
      }
    }
    centre[q][0][lane] = cc;
    centre[q][1][lane] = r0;
    centre[q][2][lane] = r1;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int x = b0 + j - nh, y = a0 + i - nh;
        if (x == -1 || x == 1) acc[i][j] += centre[q][0][(a0 + i - Y0) + (x > 0 ? 16 : 0)];
        if (y == -1 || y == 1) acc[i][j] += centre[q][y > 0 ? 2 : 1][b0 + j - X0];
      }
  }
  if (q > 0)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) part[(q - 1) * 16 + 4 * i + j][lane] = acc[i][j];
  __syncthreads();
  if (q > 0) return;
#pragma unroll
  for (int r = 0; r < Q - 1; ++r)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] += part[r * 16 + 4 * i + j][lane];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int R = a0 + i, C = b0 + j;
      const bool live = R < n && C < n;
      adj_store(ep, acc[i][j], live, z * (size_t)n * n + (live ? (size_t)R * n + C : 0), img);
    }
}

// Warps of an adjoint tile.  ms (without the centre's part) with 4, 8, 16: 256^2 x 300 0.118, 0.077, 0.058; 512^2 x 500
// 0.271, 0.255, 0.222; 768^2 x 720 0.558, 0.536, 0.486; 1280^2 x 1024 1.69, 1.66, 1.62; 1600^2 x
// 1400 3.32, 3.33, 3.30; 2048^2 x 1800 6.72, 6.78, 6.75; also for several slices (4 x 641^2 x
// 600: 1.23, 1.21, 1.16).
int ss_adj_warps(int n) { return n > 1800 ? 4 : 16; }

// Both forms of the weight in the main loop (BOTH) or the centre's columns and rows
// afterwards, whose few pixels in a row of angles make long chains in small images: ms
// 128^2 x 120 0.034, 0.036; 256^2 x 300 0.060, 0.069; 384^2 x 400 0.134, 0.142; 448^2 x 450 0.183,
// 0.173; 768^2 x 720 0.527, 0.499; 1280^2 x 1024 1.74, 1.61.
bool ss_adj_both(int n) { return n <= 384; }

struct SsState {
  float2 *pairs = nullptr;                 // [chunk][na][w2]
  int *raw = nullptr;                      // [chunk][na]
  float *rows = nullptr, *cols = nullptr;  // [chunk][n][n + 2 kSsFrame]
  int pads = 0, w2 = 0, chunk = 1;
};

void ss_state_free(void *q) {
  auto *st = (SsState *)q;
  cudaFree(st->pairs);
  delete st;
}

static void sort4(float *a) {
  for (int i = 1; i < 4; ++i)
    for (int j = i; j > 0 && a[j] < a[j - 1]; --j) std::swap(a[j], a[j - 1]);
}

}  // namespace

int ss_setup(Plan &p) {
  const int na = p.g.na, nh = p.nh, nt = 2 * nh;
  std::vector<SsAngle> tab(na);
  std::vector<int2> lim((size_t)na * nt);
  const float fnh = (float)nh, fnh1 = (float)(nh - 1);
  for (int v = 0; v < na; ++v) {
    float s, c;
    sincosf(p.angles[v], &s, &c);
    SsAngle a{};
    a.out_row = na - 1 - v;  // radon_ss.c:111
    a.steep = std::fabs((double)s) <= kS45 ? 1 : 0;
    // steep: f = fma(-y, s, t) * (1/c), weight 1/|c|; else f = fma(-x, c, t) * (1/s)
    a.a = a.steep ? s : c;
    a.rb = a.steep ? 1.0f / c : 1.0f / s;
    a.wt = (float)(1.0 / std::fabs((double)(a.steep ? c : s)));
    tab[v] = a;
    for (int kt = 0; kt < nt; ++kt) {
      const int t = kt - nh;
      const float ft = (float)t;
      float l0, l1, l2, l3;
      if (std::fabs((double)s) < 1e-5) {
        l0 = 0; l1 = 0; l2 = -fnh; l3 = fnh1;
      } else if (std::fabs((double)c) < 1e-5) {
        l0 = -fnh; l1 = fnh1; l2 = 0; l3 = 0;
      } else {
        float xa[4] = {std::fma(fnh, s, ft) / c, std::fma(-s, fnh1, ft) / c, -fnh, fnh1};
        float ya[4] = {std::fma(fnh, c, ft) / s, std::fma(-c, fnh1, ft) / s, -fnh, fnh1};
        sort4(xa);
        sort4(ya);
        l0 = xa[1]; l1 = xa[2]; l2 = ya[1]; l3 = ya[2];
      }
      const float lo = a.steep ? l2 : l0, hi = a.steep ? l3 : l1;
      lim[(size_t)v * nt + kt] = make_int2((int)std::round(lo), (int)std::round(hi));
    }
  }
  TOMO_CUDA(cudaMalloc(&p.d_angles, sizeof(SsAngle) * (size_t)na));
  TOMO_CUDA(cudaMemcpy(p.d_angles, tab.data(), sizeof(SsAngle) * (size_t)na, cudaMemcpyHostToDevice));
  TOMO_CUDA(cudaMalloc(&p.d_aux, sizeof(int2) * lim.size()));
  TOMO_CUDA(cudaMemcpy(p.d_aux, lim.data(), sizeof(int2) * lim.size(), cudaMemcpyHostToDevice));
  auto *st = new SsState();
  p.ext = st;
  p.ext_free = ss_state_free;
  // |t| at a pixel stays below sqrt(2) (nh + 1) + 2, also for the pixels of a
  // tile that lie up to 3 outside the image
  st->pads = (int)std::ceil((nh + 1) * 0.41422) + 14;
  st->w2 = 2 * nh + 2 * st->pads;
  // one workspace for a chunk of slices: the adjoint's pairs, the forward's framed
  // copies, the marked rows
  const int n = p.g.n;
  const size_t pairs1 = (size_t)na * st->w2, framed1 = (size_t)n * (n + 2 * kSsFrame);
  st->chunk = slice_chunk(p, sizeof(float2) * pairs1 + 2 * sizeof(float) * framed1 + sizeof(int) * na);
  const size_t pairs = st->chunk * pairs1, framed = st->chunk * framed1;
  TOMO_CUDA(cudaMalloc(&st->pairs, sizeof(float2) * pairs + 2 * sizeof(float) * framed + sizeof(int) * st->chunk * na));
  st->rows = (float *)(st->pairs + pairs);
  st->cols = st->rows + framed;
  st->raw = (int *)(st->cols + framed);
  // residual partials of the fused solvers: one per warp of the ordered forward
  p.fwd_warps = (size_t)((n + 127) / 128) * 4 * na * p.g.nz;
  return TOMO_OK;
}

int ss_forward(Plan &p, const float *d_img, float *d_sino, cudaStream_t s, const FwdEpi &ep) {
  const int n = p.g.n, na = p.g.na, nz = p.g.nz, nh = p.nh;
  SsState &st = *(SsState *)p.ext;
  const int tiles = (n + 2 * kSsFrame + 31) / 32;
  const int split = ep.ordered ? 0 : ss_fwd_split(n), rays = 128 / std::max(split, 1);
  auto fn = split == 4 ? ss_forward_kernel<4> : split == 2 ? ss_forward_kernel<2> : ss_forward_kernel<0>;
  const size_t per = (size_t)n * n, per_sino = (size_t)na * n, slots = p.fwd_warps / nz;
  for (int z0 = 0; z0 < nz; z0 += st.chunk) {
    const int zc = std::min(st.chunk, nz - z0);
    ss_frame_kernel<<<dim3(tiles, tiles, zc), dim3(32, 8), 0, s>>>(d_img + z0 * per, st.rows, st.cols, n);
    fn<<<dim3((n + rays - 1) / rays, na, zc), 128, 0, s>>>(st.rows, st.cols, d_sino + z0 * per_sino,
                                                           (const SsAngle *)p.d_angles, (const int2 *)p.d_aux, n, nh, na,
                                                           epi_from(ep, z0 * per_sino, z0 * slots));
  }
  TOMO_CUDA(cudaGetLastError());
  return TOMO_OK;
}

int ss_adjoint(Plan &p, const float *d_sino, float *d_img, cudaStream_t s, const AdjEpi &ep) {
  const int n = p.g.n, na = p.g.na, nz = p.g.nz;
  SsState &st = *(SsState *)p.ext;
  const int Q = ep.ordered ? 1 : ss_adj_warps(n);
  auto fn = Q == 1 ? ss_adjoint_kernel<1, false> : Q == 4 ? ss_adjoint_kernel<4, false>
            : ss_adj_both(n) ? ss_adjoint_kernel<16, true> : ss_adjoint_kernel<16, false>;
  const size_t per = (size_t)n * n, per_sino = (size_t)na * n;
  for (int z0 = 0; z0 < nz; z0 += st.chunk) {
    const int zc = std::min(st.chunk, nz - z0);
    ss_expand_kernel<<<dim3(na, zc), 256, 0, s>>>(d_sino + z0 * per_sino, st.pairs, st.raw, (const SsAngle *)p.d_angles, n,
                                                 p.nh, na, st.pads, st.w2, ep.ordered);
    fn<<<dim3((n + 31) / 32, (n + 15) / 16, zc), 32 * Q, 0, s>>>(st.pairs, st.raw, d_img + z0 * per,
                                                                 (const SsAngle *)p.d_angles, (const int2 *)p.d_aux, n, p.nh,
                                                                 na, st.pads, st.w2, epi_from(ep, z0 * per));
  }
  TOMO_CUDA(cudaGetLastError());
  return TOMO_OK;
}

}  // namespace tomo
