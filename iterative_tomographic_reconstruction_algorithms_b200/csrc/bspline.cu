// Generalised (B-spline) Radon projector pair for sm_100a.
//
// Reference: common/operators/bspline_module/pymodule_genradon/gen_forwproj.c
// :22-78 and gen_backproj.c:22-74.  For every angle (degrees, converted as
// theta = (float)(deg * pi/180)), pixel (ky_i, kx_i) with kx = kx_i - n/2 and
// ky = n/2 - ky_i, the projection ps = cos*kx + sin*ky (compiled as
// fma(kx, cos, sin*ky)) feeds 2*ds+1 detector taps s = -ds..ds:
//   bin  yi = trunc((double)((float)s + ps) + n/2)         (C truncation),
//   lut  li = trunc((yi - n/2 - ps) * lut_step) + lut_size/2,
// skipped unless 0 <= yi < n and 0 <= li < lut_size - 1; the weight is
// lut[angle][li].  ds = (int)(support/2 + 0.5), lut_step = (lut_size/2) /
// (support/2).  The table itself is built on the host (bspline_functions.py).
//
// Forward = gather per bin over image lines, adjoint = gather per pixel over
// angles, for tables of support 4 and power-of-two length; otherwise forward =
// per (angle, block of bins) a pass over the band of pixels whose taps can reach
// the bins, summed in fixed point, and adjoint = gather per pixel over angles
// and taps.  Output rows follow the angle order (no reversal).
#include <algorithm>
#include <cmath>

#include "f32x2.cuh"
#include "fixed_sum.cuh"
#include "tomo_internal.cuh"

namespace tomo {
namespace {

constexpr double kPi = 3.141592653589793;

struct BsConst {
  int n, na, lut_size, lut_half, lut_max, ds;
  float lut_step, fmid;
  double mid;
};

__device__ __forceinline__ int bs_bin(int s, float ps, double mid) {
  return (int)__dadd_rn((double)__fadd_rn((float)s, ps), mid);  // trunc toward zero
}


// Forward: a block owns kBsBins consecutive bins of one angle and slice.  Its
// warps walk the band of pixels whose taps can reach those bins (a line per
// warp, each pixel once) and add every tap's product lut * value, as the
// reference rounds it, into shared-memory bins summed in fixed point
// (fixed_sum.cuh): deterministic, each bin the sum of the reference's float
// products to within the fixed-point unit, rounded once.  At most 3 pixels per line and tap reach a bin
// (ps moves by at least 1/sqrt(2) per pixel), which bounds the sums.
constexpr int kBsBins = 128, kBsThreads = 256;


// LUT index trunc((yi - n/2 - ps) * lut_step) + lut_size/2 (gen_forwproj.c:61).
__device__ __forceinline__ int bs_lut(int yi, float ps, const BsConst &k) {
  const float y = __fsub_rn((float)yi, k.fmid);
  return (int)__fmul_rn(__fsub_rn(y, ps), k.lut_step) + k.lut_half;
}

// The same index with the truncation toward zero taken without the
// conversion pipe (the forward's inner loop is conversion-bound).
__device__ __forceinline__ int bs_lut_fast(int yi, float ps, const BsConst &k) {
  const float a = __fmul_rn(__fsub_rn(__fsub_rn((float)yi, k.fmid), ps), k.lut_step);
  float fl;
  const int t = floor_i(fabsf(a), fl);
  return (a < 0.0f ? -t : t) + k.lut_half;
}

// bs_bin for even n >= 4 without the conversion pipe: n/2 is an integer, so
// trunc((double)t + n/2) == floor(t) + n/2, except that t in (-n/2 - 1, -n/2)
// truncates to bin 0 and a tiny negative t may round up to n/2 in the double
// sum (t in (-1, 0) takes the double rule).  Odd n: the double rule.
__device__ __forceinline__ int bs_bin_fast(int s, float ps, const BsConst &k, bool even, int nh, float b0lo) {
  const float t = __fadd_rn((float)s, ps);
  if (even && !(t < 0.0f && t > -1.0f)) {
    float fl;
    int yi = floor_i(t, fl) + nh;
    if (yi == -1 && t > b0lo) yi = 0;
    return yi;
  }
  return bs_bin(s, ps, k.mid);
}


__global__ void __launch_bounds__(kBsThreads) bs_forward_kernel(
    const float *__restrict__ img, float *__restrict__ sino, const float2 *__restrict__ cs,
    const float *__restrict__ lut, const unsigned *__restrict__ vmax, float lutmax, BsConst k, FwdEpi ep) {
  extern __shared__ float slut[];  // this angle's lut row
  __shared__ unsigned long long acc[kBsBins];
  __shared__ unsigned flg[kBsBins];  // non-finite products per bin (fixed_sum.cuh)
  const int B0 = blockIdx.x * kBsBins, v = blockIdx.y;
  const size_t z = blockIdx.z;
  const int n = k.n;
  const float *L = lut + (size_t)v * k.lut_size;
  for (int i = threadIdx.x; i < k.lut_size; i += blockDim.x) slut[i] = __ldg(L + i);
  for (int i = threadIdx.x; i < kBsBins; i += blockDim.x) {
    acc[i] = 0ull;
    flg[i] = 0u;
  }
  // fixed-point unit: |bin| <= 3 n (2 ds + 1) max|lut| max|finite value|
  const float vm = __uint_as_float(vmax[z]);
  const FixedScale fs = fixed_scale(3.0 * n * (2.0 * k.ds + 1.0) * (double)lutmax * (double)vm);
  __syncthreads();
  const float C = cs[v].x, S = cs[v].y;
  const float *I = img + z * (size_t)n * n;
  const bool by_rows = fabsf(C) >= fabsf(S);  // along a row ps moves by C per pixel
  const int Bend = min(B0 + kBsBins, n);
  const float plo = (float)(B0 - k.ds - 2) - k.fmid, phi = (float)(Bend - 1 + k.ds + 2) - k.fmid;
  const bool even = (n & 1) == 0 && n >= 4;  // n = 2: the bin-0 boundary sits at 0, use the double rule
  const float b0lo = -k.fmid - 1.0f;
  const int nh = n / 2;
  // each warp takes every 8th line, its lanes the line's band of pixels
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int line = warp; line < n; line += kBsThreads / 32) {
    // by rows: ky fixed, ps = kx*C + S*ky; by columns: kx fixed, ps = ky*S + kx*C
    const float fixed = by_rows ? (float)(-line + k.mid) : (float)(line - k.mid);
    const float slope = by_rows ? C : S;
    const float base = by_rows ? S * fixed : C * fixed;
    float u0 = (plo - base) / slope, u1 = (phi - base) / slope;
    if (u0 > u1) { const float t = u0; u0 = u1; u1 = t; }
    int j0, j1;
    if (by_rows) {  // kx = kx_i - mid
      j0 = (int)floorf(u0 + k.fmid) - 1;
      j1 = (int)ceilf(u1 + k.fmid) + 1;
    } else {        // ky = mid - ky_i
      j0 = (int)floorf(k.fmid - u1) - 1;
      j1 = (int)ceilf(k.fmid - u0) + 1;
    }
    j0 = max(j0, 0);
    j1 = min(j1, n - 1);
    for (int j = j0 + lane; j <= j1; j += 32) {
      const int kyi = by_rows ? line : j, kxi = by_rows ? j : line;
      const float val = __ldg(I + (size_t)kyi * n + kxi);
      if (val == 0.0f) continue;  // adds exactly nothing
      const float ky = (float)(-kyi + k.mid), kx = (float)(kxi - k.mid);
      const float ps = __fmaf_rn(kx, C, __fmul_rn(S, ky));
      for (int s = -k.ds; s <= k.ds; ++s) {
        const int yi = bs_bin_fast(s, ps, k, even, nh, b0lo);
        if (yi < B0 || yi >= Bend) continue;
        const int li = bs_lut_fast(yi, ps, k);
        if (li >= k.lut_max || li < 0) continue;
        fixed_add_product(acc + (yi - B0), flg + (yi - B0), __fmul_rn(slut[li], val), fs);
      }
    }
  }
  __syncthreads();
  const int b = B0 + (int)threadIdx.x;
  const bool live = threadIdx.x < kBsBins && b < n;
  float out = 0.0f;
  if (live) out = flg[threadIdx.x] ? nonfinite_value(flg[threadIdx.x]) : fixed_to_float(acc[threadIdx.x], fs);
  fwd_store(ep, out, live, z * (size_t)k.na * n + (size_t)v * n + (live ? b : 0), sino);
}

constexpr int kBsChunk = 1024;

__global__ void __launch_bounds__(256) bs_adjoint_kernel(
    const float *__restrict__ sino, float *__restrict__ img, const float2 *__restrict__ cs,
    const float *__restrict__ lut, BsConst k, AdjEpi ep) {
  __shared__ float2 scs[kBsChunk];
  const int n = k.n;
  const int kxi = blockIdx.x * blockDim.x + threadIdx.x;
  const int kyi = blockIdx.y * blockDim.y + threadIdx.y;
  const size_t z = blockIdx.z;
  const bool live = kxi < n && kyi < n;
  const float *Sg = sino + z * (size_t)k.na * n;
  const int tid = threadIdx.y * blockDim.x + threadIdx.x, nthr = blockDim.x * blockDim.y;
  const float ky = (float)(-kyi + k.mid), kx = (float)(kxi - k.mid);
  const bool even = (n & 1) == 0 && n >= 4;
  const int nh = n / 2;
  float acc = 0.0f;
  for (int v0 = 0; v0 < k.na; v0 += kBsChunk) {
    const int cnt = min(kBsChunk, k.na - v0);
    __syncthreads();
    for (int t = tid; t < cnt; t += nthr) scs[t] = cs[v0 + t];
    __syncthreads();
    if (!live) continue;
    for (int u = 0; u < cnt; ++u) {
      const int v = v0 + u;
      const float ps = __fmaf_rn(kx, scs[u].x, __fmul_rn(scs[u].y, ky));
      const float *row = Sg + (size_t)v * n;
      const float *L = lut + (size_t)v * k.lut_size;
      float fl;
      const int base = floor_i(ps, fl);
      const float frac = __fsub_rn(ps, fl);
      if (even && frac >= 0x1p-12f && frac <= 1.0f - 0x1p-12f) {
        // ps is at least 2^-12 from an integer, so fl(s + ps) never rounds
        // across one: every tap's bin is floor(ps) + s + n/2, with the
        // reference's truncation folding -1 onto bin 0 (t in (-n/2 - 1, -n/2))
        for (int s = -k.ds; s <= k.ds; ++s) {
          int yi = base + s + nh;
          if (yi == -1) yi = 0;
          if (yi >= n || yi < 0) continue;
          const int li = bs_lut(yi, ps, k);
          if (li >= k.lut_max || li < 0) continue;
          acc = fmaf(__ldg(row + yi), __ldg(L + li), acc);
        }
        continue;
      }
      for (int s = -k.ds; s <= k.ds; ++s) {
        const int yi = bs_bin(s, ps, k.mid);
        if (yi >= n || yi < 0) continue;
        const int li = bs_lut(yi, ps, k);
        if (li >= k.lut_max || li < 0) continue;
        acc = fmaf(__ldg(row + yi), __ldg(L + li), acc);
      }
    }
  }
  adj_store(ep, acc, live, z * (size_t)n * n + (size_t)(live ? kyi : 0) * n + (live ? kxi : 0), img);
}

// ---------------------------------------------------------------------------
// Tables with support 4 and a power-of-two length (the class's default: 2048)
// ---------------------------------------------------------------------------
// The step of the table index is then a power of two, so (y - ps) * step is
// exact, and the index is a function of the exact distance d = y - ps.  fl(s +
// ps) is exact too unless |ps| < 4 or s carries |ps| across a power of two: a
// tap's bin is otherwise floor(s + ps) + n/2, every bin within reach gets one
// tap, and the index alone decides whether it counts.  What is left (pixels
// close to an integer there, and bin 0, onto which the truncation folds bin -1)
// goes through the reference's rule tap by tap (bs_bin).  Other tables, images above
// 4096^2 and the solvers (epilogue.cuh) take the general kernels above.
constexpr float kBsMagic = 12582912.0f;   // 1.5 * 2^23
constexpr int kBsMagicBits = 0x4B400000;  // its bit pattern
constexpr int kBsFrame = 8;

// Framed copies of the image: rows[ky_i][P + kx_i] and cols[kx_i][P + ky_i],
// P = kBsFrame zeros on either side.
__global__ void __launch_bounds__(256) bs_frame_kernel(const float *__restrict__ img, float *__restrict__ rows,
                                                       float *__restrict__ cols, int n) {
  __shared__ float tile[32][33];
  const size_t z = blockIdx.z;
  const int w = n + 2 * kBsFrame;
  const float *src = img + z * (size_t)n * n;
  float *R = rows + z * (size_t)n * w, *C = cols + z * (size_t)n * w;
  const int x0 = blockIdx.x * 32 - kBsFrame, y0 = blockIdx.y * 32 - kBsFrame;  // tiles cover the frame too
  for (int dy = threadIdx.y; dy < 32; dy += 8) {
    const int y = y0 + dy, x = x0 + threadIdx.x;
    const float v = y >= 0 && y < n && x >= 0 && x < n ? __ldg(src + (size_t)y * n + x) : 0.0f;
    tile[dy][threadIdx.x] = v;
    if (y >= 0 && y < n && x < n + kBsFrame) R[(size_t)y * w + kBsFrame + x] = v;
  }
  __syncthreads();
  for (int dy = threadIdx.y; dy < 32; dy += 8) {
    const int x = x0 + dy, y = y0 + threadIdx.x;
    if (x >= 0 && x < n && y < n + kBsFrame) C[(size_t)x * w + kBsFrame + y] = tile[threadIdx.x][dy];
  }
}

// Whether bin y (from the centre) is reached by pixels whose taps' bins may not
// be floor(s + ps): |ps| < 4, or |ps| within 2 below a power of two.
__device__ __forceinline__ bool bs_special(float y) {
  const float a = fabsf(y);
  if (a < 8.0f) return true;
  const float p = __int_as_float(__float_as_int(a) & 0x7f800000);  // 2^e <= a
  return a - p < 4.0f || 2.0f * p - a < 6.0f;
}

// Above the rounding of fl(s + ps), |ps| <= n/sqrt(2) + 2.
__device__ __forceinline__ float bs_near(int n) { return (float)(n + 8) * 0x1p-24f; }

// A lane's bin and angle, as it walks lines l (ROWS: ky, else kx).
template <bool ROWS, int DIR>
struct BsLine {
  float C, S, y, base, slope, lo, hi;
  __device__ __forceinline__ BsLine(float C_, float S_, int b, const BsConst &k) : C(C_), S(S_), y((float)b - k.fmid) {
    const float inv = 1.0f / (ROWS ? C : -S);  // 1 / (ps per pixel)
    // pixel at which ps = y - 2 - 1/64
    base = (y - 2.015625f) * inv + k.fmid;
    slope = -(ROWS ? S : C) * inv;
    lo = DIR > 0 ? -8.0f : -3.0f;
    hi = DIR > 0 ? (float)(k.n + 2) : (float)(k.n + 7);
  }
  __device__ __forceinline__ static float coordinate(int i, const BsConst &k) {
    return ROWS ? k.fmid - (float)i : (float)i - k.fmid;
  }
  // the first of the six pixels, in the magic form
  __device__ __forceinline__ float first(float l) const {
    const float pos = fminf(fmaxf(fmaf(slope, l, base), lo), hi);
    return DIR > 0 ? __fadd_ru(pos, kBsMagic) : __fadd_rd(pos, kBsMagic);
  }
};

// How many taps of a pixel at distance d, ps from the centre, the reference puts into
// bin b (0, 1 or 2).
__device__ __forceinline__ int bs_count(float d, float ps, int b, const BsConst &k) {
  const float s0 = rintf(d);  // a tap on the bin is within 1 of the distance
  int m = 0;
#pragma unroll
  for (int s = -1; s <= 1; ++s) {
    const float t = s0 + (float)s;
    m += (fabsf(t) <= 2.0f) & (bs_bin((int)t, ps, k.mid) == b);
  }
  return m;
}

struct BsSix {
  float x[6];
};
// The products of a line's six pixels, each as often as the reference counts it.
template <bool ROWS, int DIR>
__device__ __noinline__ double bs_fwd_taps(BsSix s, float u0, float l, float so, float C, float S, int b, const BsConst &k) {
  double p = 0.0;
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    const float u = u0 + (float)(q * DIR);
    const float ps = ROWS ? __fmaf_rn(u, C, so) : __fmaf_rn(l, C, __fmul_rn(S, -u));
    const int m = bs_count(__fsub_rn((float)b - k.fmid, ps), ps, b, k);
    const double x = m ? (double)s.x[q] : 0.0;
    p += x;
    if (m == 2) p += x;
  }
  return p;
}

// All lines of a bin as the reference has them.
template <bool ROWS, int DIR>
__device__ __noinline__ double bs_fwd_again(const float *__restrict__ I, const float *__restrict__ L, int w, float C, float S, int b,
                                            const BsConst &k, int i0, int i1) {
  const BsLine<ROWS, DIR> B(C, S, b, k);
  double acc = 0.0;
  for (int i = i0; i < i1; ++i) {
    const float l = BsLine<ROWS, DIR>::coordinate(i, k), fm = B.first(l);
    const float *v = I + (size_t)i * w + kBsFrame + (__float_as_int(fm) - kBsMagicBits);
#pragma unroll 1
    for (int q = 0; q < 6; ++q) {
      const float u = __fsub_rn(__fsub_rn(fm, kBsMagic), k.fmid) + (float)(q * DIR);
      const float ps = ROWS ? __fmaf_rn(u, C, __fmul_rn(S, l)) : __fmaf_rn(l, C, __fmul_rn(S, -u));
      const int li = bs_lut(b, ps, k), m = bs_count(__fsub_rn(B.y, ps), ps, b, k);
      if (m && li >= 0 && li < k.lut_max) acc += (double)m * (double)__fmul_rn(__ldg(L + li), __ldg(v + q * DIR));
    }
  }
  return acc;
}

// Forward: a lane owns a bin and walks the lines (ROWS: image rows, when ps
// moves faster along x; else columns).  Per line the pixels with |y - ps| < 2
// (+ 1 table step) are among six consecutive ones, sigma = max(|C|, |S|) in
// [0.707, 1] apart (a seventh would lie 6 x 0.707 > 4.03 behind the first).
// The angle's table is in shared memory by half steps of the distance, with the
// index's truncation toward zero applied and 0 where no tap counts: entry floor(a)
// + ceil(a), a = d * step, needs no conversion.  MODE 1: some of the warp's bins are
// special, 2: it holds bin 0, whose pixels count twice (the reference's truncation
// folds the tap on bin -1 onto it).  Products are rounded as the reference rounds
// them and added in double, rounded once.  A sum that is not finite, for which a
// pixel out of reach may be the cause, is done again tap by tap.
//
// Bound by shared memory (six reads at the lanes' own phases, about 3.5 bank
// conflicts each) and the conversions to double; two pixels at a time as packed
// pairs.  Adding every tap to 64-bit fixed-point sums by two shared-memory atomics
// took 2.15 ms at 768^2 x 720 and 31.7 at 2048^2 x 1800; this takes 1.48 and
// 22.6 (1.66 and 25.5 pixel by pixel with NaN for the missing taps).
template <bool ROWS, int DIR, int MODE>
__device__ __forceinline__ double bs_fwd_bin(const float *__restrict__ I, const float *tab, const float *__restrict__ L, int entries,
                                             int w, float C, float S, int b, const BsConst &k, int i0, int i1) {
  const BsLine<ROWS, DIR> B(C, S, b, k);
  const float y = B.y;
  const float *line = I + (size_t)i0 * w + kBsFrame - kBsMagicBits;
  const unsigned org = (unsigned)entries / 2u - 2u * (unsigned)kBsMagicBits;  // entry of distance 0
  float lc = BsLine<ROWS, DIR>::coordinate(i0, k);
  const float thr = bs_special(y) ? bs_near(k.n) : -1.0f;
  const F2 C2 = f2(C), S2 = f2(S), y2 = f2(y), step2 = f2(k.lut_step), magic = f2(kBsMagic);
  double acc = 0.0;
#pragma unroll 1
  for (int i = i0; i < i1; ++i, line += w, lc += ROWS ? -1.0f : 1.0f) {
    const float fm = B.first(lc);
    const float *v = line + __float_as_int(fm);
    const float u0 = __fsub_rn(__fsub_rn(fm, kBsMagic), k.fmid), so = ROWS ? __fmul_rn(S, lc) : 0.0f;
    BsSix s;  // the products
    float(&x)[6] = s.x, near = 1.0f;
    double again = 0.0;
#pragma unroll
    for (int q = 0; q < 6; q += 2) {
      F2 ps;
      if (ROWS) ps = fma2(add2(f2(u0), f2((float)(q * DIR), (float)((q + 1) * DIR))), C2, f2(so));
      else ps = fma2(f2(lc), C2, mul2(S2, add2(f2(-u0), f2((float)(-q * DIR), (float)(-(q + 1) * DIR)))));
      const F2 d2 = rsub2(ps, y2);
      const float2 d = unpack(d2), fl = unpack(fma2_rd(d2, step2, magic)), ce = unpack(fma2_ru(d2, step2, magic));
      const float wa = tab[min(__float_as_uint(fl.x) + __float_as_uint(ce.x) + org, (unsigned)entries)];
      const float wb = tab[min(__float_as_uint(fl.y) + __float_as_uint(ce.y) + org, (unsigned)entries)];
      x[q] = __fmul_rn(wa, __ldg(v + q * DIR));
      x[q + 1] = __fmul_rn(wb, __ldg(v + (q + 1) * DIR));
      if (MODE > 0) {
        auto off = [](float e) { return fabsf(__fsub_rn(e, __fsub_rn(__fadd_rn(e, kBsMagic), kBsMagic))); };
        const float ra = off(d.x), rb = off(d.y);
        near = fminf(near, fminf(ra, rb));
        if (MODE > 1 && b == 0 && d.x > -2.0f && ra > 0.0f) again += (double)x[q];
        if (MODE > 1 && b == 0 && d.y > -2.0f && rb > 0.0f) again += (double)x[q + 1];
      }
    }
    double p = (((double)x[0] + (double)x[1]) + ((double)x[2] + (double)x[3])) + ((double)x[4] + (double)x[5]);
    if (MODE > 1) p += again;
    if (MODE > 0 && near < thr) p = bs_fwd_taps<ROWS, DIR>(s, u0, lc, so, C, S, b, k);
    acc += p;
  }
  if (!(fabs(acc) < INFINITY)) acc = bs_fwd_again<ROWS, DIR>(I, L, w, C, S, b, k, i0, i1);
  return acc;
}

// A block takes 128 / SPLIT bins of an angle, SPLIT warps sharing each bin's
// lines (added in order): lines of very unequal number per bin then balance
// better (513^2 x 400: 0.75 ms unsplit, 0.43 by four; 2048^2 x 1800 the same by
// two).  The split is a function of n alone (bs_fwd_split).
template <int SPLIT>
__global__ void __launch_bounds__(128, 8) bs_forward_pow2_kernel(const float *__restrict__ rows, const float *__restrict__ cols,
                                                              float *__restrict__ sino, const float2 *__restrict__ cs,
                                                              const float *__restrict__ lut, int entries, BsConst k) {
  extern __shared__ float tab[];  // [entries] by half steps, distances within 2 (+ 2 steps); 0 where no tap counts
  __shared__ double part[SPLIT][128 / SPLIT];
  constexpr int kBins = 128 / SPLIT;
  const int lane = threadIdx.x % kBins, q = threadIdx.x / kBins;
  const int b = blockIdx.x * kBins + lane, v = blockIdx.y, n = k.n, w = n + 2 * kBsFrame;
  const size_t z = blockIdx.z;
  const float *Lv = lut + (size_t)v * k.lut_size;
  const int org = entries / 2;
  for (int e = threadIdx.x; e <= entries; e += 128) {
    const int i2 = e - org;                    // floor(a) + ceil(a)
    const int li = (i2 >= 0 ? i2 >> 1 : -(-i2 >> 1)) + k.lut_half;  // toward zero
    tab[e] = e < entries && li >= 0 && li < k.lut_max ? __ldg(Lv + li) : 0.0f;
  }
  __syncthreads();
  const float C = cs[v].x, S = cs[v].y;
  const bool by_rows = fabsf(C) >= fabsf(S);
  const int W0 = blockIdx.x * kBins + (lane & ~31);  // the warp's first bin
  // lines whose ps range, o l +- |K| (n/2 + 1), meets the warp's bins
  const float K = fabsf(by_rows ? C : S), o = by_rows ? S : C, half = K * (k.fmid + 2.0f);
  int i0 = 0, i1 = n;
  if (fabsf(o) > 1e-4f) {
    const float y0 = (float)W0 - k.fmid - 3.0f - half, y1 = (float)(W0 + 31) - k.fmid + 3.0f + half;
    const float l0 = fminf(y0 / o, y1 / o), l1 = fmaxf(y0 / o, y1 / o);
    const float j0 = by_rows ? k.fmid - l1 : l0 + k.fmid, j1 = by_rows ? k.fmid - l0 : l1 + k.fmid;
    i0 = (int)floorf(fminf(fmaxf(j0 - 2.0f, 0.0f), (float)n));
    i1 = (int)ceilf(fminf(fmaxf(j1 + 2.0f, 0.0f), (float)n));
  }
  if (SPLIT > 1) {
    const int len = max(0, i1 - i0);
    i1 = i0 + len * (q + 1) / SPLIT;
    i0 += len * q / SPLIT;
  }
  const float *L = (by_rows ? rows : cols) + z * (size_t)n * w;
  const bool spec = __any_sync(0xffffffffu, bs_special((float)b - k.fmid)), first = __any_sync(0xffffffffu, b == 0);
  double acc;
#define BS_BIN(R, D) (first  ? bs_fwd_bin<R, D, 2>(L, tab, Lv, entries, w, C, S, b, k, i0, i1) \
                      : spec ? bs_fwd_bin<R, D, 1>(L, tab, Lv, entries, w, C, S, b, k, i0, i1) \
                             : bs_fwd_bin<R, D, 0>(L, tab, Lv, entries, w, C, S, b, k, i0, i1))
  if (by_rows) acc = C > 0.0f ? BS_BIN(true, 1) : BS_BIN(true, -1);
  else acc = S < 0.0f ? BS_BIN(false, 1) : BS_BIN(false, -1);
#undef BS_BIN
  if (SPLIT > 1) {
    part[q][lane] = acc;
    __syncthreads();
    if (q > 0) return;  // warp-uniform
    for (int r = 1; r < SPLIT; ++r) acc += part[r][lane];
  }
  if (b < n) sino[z * (size_t)k.na * n + (size_t)v * n + b] = (float)acc;
}

int bs_fwd_split(int n) { return n > 1024 ? 2 : 4; }

// The adjoint's table of an angle, by half steps of the fraction of ps: entry
// floor(f) + ceil(f), f = (ps - floor ps) step in (0, step), holds the four taps'
// weights, distances k - f / step for k = -1 .. 2.
__global__ void bs_lut4_kernel(const float *__restrict__ lut, float4 *__restrict__ out, BsConst k) {
  const float *L = lut + (size_t)blockIdx.x * k.lut_size;
  const int step = (int)k.lut_step;
  for (int i = threadIdx.x; i < 2 * step; i += blockDim.x) {
    const int fl = i >> 1, ce = (i + 1) >> 1;
    const int li[4] = {step - fl, 2 * step - fl, 3 * step - ce, 4 * step - ce};
    float v[4];
    for (int t = 0; t < 4; ++t) v[t] = li[t] >= 0 && li[t] < k.lut_max ? L[li[t]] : 0.0f;
    out[(size_t)blockIdx.x * 2 * step + i] = make_float4(v[0], v[1], v[2], v[3]);
  }
}

// Sinogram rows as groups, entry e = m + pads: {S_m-1, S_m, S_m+1, S_m+2}, 0
// outside [0, n); bin 0 twice, for the tap on bin -1 that folds onto it with
// the same weight.  A row where that is not finite is marked.
__global__ void __launch_bounds__(256) bs_expand_kernel(const float *__restrict__ sino, float4 *__restrict__ out,
                                                        int *__restrict__ mark, int n, int pads, int w2) {
  const float *src = sino + (size_t)blockIdx.x * n;
  float4 *dst = out + (size_t)blockIdx.x * w2;
  if (threadIdx.x == 0) mark[blockIdx.x] = !(2.0f * fabsf(__ldg(src)) < INFINITY);
  for (int e = threadIdx.x; e < w2; e += blockDim.x) {
    float v[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int m = e - pads - 1 + t;
      v[t] = m >= 0 && m < n ? __ldg(src + m) : 0.0f;
      if (m == 0) v[t] *= 2.0f;
    }
    dst[e] = make_float4(v[0], v[1], v[2], v[3]);
  }
}

// One angle's taps of a pixel by the reference's rule.
__device__ __noinline__ float bs_adj_taps(float ps, const float *__restrict__ row, const float *__restrict__ L, const BsConst &k,
                                          float acc) {
  for (int s = -2; s <= 2; ++s) {
    const int yi = bs_bin(s, ps, k.mid);
    if (yi >= k.n || yi < 0) continue;
    const int li = bs_lut(yi, ps, k);
    if (li >= k.lut_max || li < 0) continue;
    acc = fmaf(__ldg(row + yi), __ldg(L + li), acc);
  }
  return acc;
}

__device__ __forceinline__ bool bs_near_step(float f) { return fabsf(f - rintf(f)) < 0x1p-12f; }

// Adjoint: a block holds a 64 x 32 pixel tile, 4 rows per lane, and goes
// through its share of the angles with the angle's table of four weights (16
// KB) in shared memory, the next one on its way in registers.  A pixel and
// angle: floor of ps, one 16-byte read of four bins, one of four weights.
// Q shares of the angles for small images, whose tiles alone
// do not fill the SMs, added in order by bs_adj_sum_kernel (Q depends on n).
//
// Bound by L1 / shared memory: the weight reads are at the lanes' own phases
// (about 11 wavefronts), the bins' about 5.  A thread per pixel with five table
// reads from L1, each at its own line, took 3.04 ms at 768^2 x 720 and 46.3 at
// 2048^2 x 1800; this 1.28 and 22.0.
constexpr int kBsTW = 64, kBsTH = 32, kBsThreads4 = 512;

template <bool ODD>
__global__ void __launch_bounds__(kBsThreads4) bs_adjoint_pow2_kernel(const float *__restrict__ sino, const float4 *__restrict__ S4,
                                                                      const float4 *__restrict__ lut4,
                                                                      const float *__restrict__ lut, float *__restrict__ img,
                                                                      const float2 *__restrict__ cs, BsConst k, int pads, int w2,
                                                                      int Q, float *__restrict__ partial) {
  extern __shared__ float4 tab4[];
  const int n = k.n, nh = n / 2, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t z = blockIdx.z;
  const int q = blockIdx.x % Q;
  const int b0 = blockIdx.x / Q * kBsTW + 32 * (warp & 1) + lane, a0 = blockIdx.y * kBsTH + 4 * (warp >> 1);
  const int u0 = (int)((long long)k.na * q / Q), u1 = (int)((long long)k.na * (q + 1) / Q);
  const int entries = 2 * (int)k.lut_step;
  const float step = k.lut_step, x0 = (float)b0 - k.fmid, y0 = k.fmid - (float)a0;
  const float edge = 1.0f / step;
  float acc[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] = 0.0f;
  const float near = bs_near(n);
  const bool inside = a0 < n && b0 < n;
  constexpr int kPer = 2;  // entries of a thread: tables of up to 1024 entries
  float4 next[kPer];
  auto fetch = [&](int u) {
#pragma unroll
    for (int r = 0; r < kPer; ++r)
      if (tid + r * kBsThreads4 < entries) next[r] = __ldg(lut4 + (size_t)u * entries + tid + r * kBsThreads4);
  };
  if (u0 < u1) fetch(u0);
#pragma unroll 1
  for (int u = u0; u < u1; ++u) {
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kPer; ++r)
      if (tid + r * kBsThreads4 < entries) tab4[tid + r * kBsThreads4] = next[r];
    __syncthreads();
    if (u + 1 < u1) fetch(u + 1);
    if (!inside) continue;
    const float2 g = __ldg(cs + u);
    const float L0 = __ldg(lut + (size_t)u * k.lut_size);
    const float *srow = sino + (z * k.na + u) * (size_t)n;
    const float4 *row = S4 + (z * k.na + u) * (size_t)w2 + pads + nh - kBsMagicBits;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float ps = __fmaf_rn(x0, g.x, __fmul_rn(g.y, y0 - (float)i));
      const float fd = __fadd_rd(ODD ? __fadd_rn(ps, 0.5f) : ps, kBsMagic);
      const float frac = __fsub_rn(ps, __fsub_rn(__fsub_rn(fd, kBsMagic), ODD ? 0.5f : 0.0f));
      const unsigned e = __float_as_uint(__fmaf_rd(frac, step, kBsMagic)) + __float_as_uint(__fmaf_ru(frac, step, kBsMagic)) -
                         2u * (unsigned)kBsMagicBits;
      const float4 *sp = row + __float_as_int(fd);
      const float4 s = __ldg(sp), w = tab4[min(e, (unsigned)entries - 1u)];
      float o = acc[i];
      if (frac < edge) {  // the tap at distance -2 counts too (on bin 0 once)
        const int m = __float_as_int(fd) - kBsMagicBits + nh - 2;
        if (m >= 0 && m < n) o = fmaf(__ldg(srow + m), L0, o);
      }
      o = fmaf(s.x, w.x, o);
      o = fmaf(s.y, w.y, o);
      o = fmaf(s.z, w.z, o);
      if (frac > edge) o = fmaf(s.w, w.w, o);  // else the table has ended
      // |ps| < 4, where y - ps rounds, next to a table step; next to an integer
      // where fl(s + ps) may round across it; an integral ps next to bin 0, onto
      // which nothing folds then
      if ((fabsf(ps) < 4.0f && bs_near_step(frac * step)) ||
          (fabsf(frac - 0.5f) > 0.5f - near && (bs_special(ps) || ps < 4.0f - k.fmid)))
        o = bs_adj_taps(ps, srow, lut + (size_t)u * k.lut_size, k, acc[i]);
      acc[i] = o;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int R = a0 + i;
    const bool live = R < n && b0 < n;
    const size_t p = z * (size_t)n * n + (live ? (size_t)R * n + b0 : 0);
    if (live) (Q > 1 ? partial + (size_t)q * gridDim.z * n * n : img)[p] = acc[i];
  }
}

// The shares of slice blockIdx.y added in order (Q = 1: nothing to add).  A slice with
// marked rows, which may lack finite values, is done again by the reference's rule.
__global__ void __launch_bounds__(256) bs_adj_sum_kernel(const float *__restrict__ partial, int Q, float *__restrict__ img,
                                                         const float *__restrict__ sino, const int *__restrict__ mark,
                                                         const float2 *__restrict__ cs, const float *__restrict__ lut, BsConst k) {
  const size_t z = blockIdx.y, per = (size_t)k.n * k.n, total = per * gridDim.y;
  bool marked = false;
  for (int u = threadIdx.x; u < k.na; u += 256) marked |= __ldg(mark + z * k.na + u) != 0;
  marked = __syncthreads_or(marked);
  const size_t p = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (p >= per || (Q == 1 && !marked)) return;
  float acc = 0.0f;
  if (marked) {
    const int R = (int)(p / k.n);
    const float x = (float)((int)p - R * k.n) - k.fmid, y = k.fmid - (float)R;
    for (int u = 0; u < k.na; ++u) {
      const float2 g = __ldg(cs + u);
      acc = bs_adj_taps(__fmaf_rn(x, g.x, __fmul_rn(g.y, y)), sino + (z * k.na + u) * (size_t)k.n, lut + (size_t)u * k.lut_size, k, acc);
    }
  } else {
    for (int q = 0; q < Q; ++q) acc += partial[(size_t)q * total + z * per + p];
  }
  img[z * per + p] = acc;
}

// Shares of the angles: blocks enough for four rounds of two to an SM, since
// those at the rim finish early (768^2 x 720: 1.90 ms with 288 blocks, 1.28 with
// 1152), at most 16.
int bs_adj_shares(int n) {
  const int tiles = ((n + kBsTW - 1) / kBsTW) * ((n + kBsTH - 1) / kBsTH);
  return std::max(1, std::min(16, 1184 / tiles));
}

BsConst make_const(const Plan &p) {
  BsConst k{};
  k.n = p.g.n;
  k.na = p.g.na;
  k.lut_size = p.g.lut_size;
  k.lut_half = p.g.lut_size / 2;
  k.lut_max = p.g.lut_size - 1;
  k.ds = (int)(0.5 * (double)p.g.support + 0.5);
  k.lut_step = (float)((p.g.lut_size * 0.5) / ((double)p.g.support * 0.5));
  k.mid = 0.5 * p.g.n;
  k.fmid = (float)k.mid;
  return k;
}

struct BsState {
  float lutmax = 0.0f;        // max |lut|
  unsigned *vmax = nullptr;   // per slice: max |image| as float bits (general kernels)
  bool pow2 = false;          // support 4, power-of-two table
  void *work = nullptr;       // one workspace for what follows
  float4 *lut4 = nullptr, *S4 = nullptr;
  float *rows = nullptr, *cols = nullptr, *partial = nullptr;
  int *mark = nullptr;  // [chunk][na]
  int pads = 0, w2 = 0, Q = 1, entries = 0, chunk = 1;
};

void bs_state_free(void *q) {
  auto *st = (BsState *)q;
  cudaFree(st->vmax);
  cudaFree(st->work);
  delete st;
}

}  // namespace

int bs_setup(Plan &p) {
  const int na = p.g.na;
  if (!p.g.lut || p.g.lut_size < 2)
    return fail(TOMO_EINVAL, "bspline: lut and lut_size >= 2 are required");
  if (!(p.g.support > 0.0f) || p.g.support > 64.0f)
    return fail(TOMO_EINVAL, "bspline: support must be in (0, 64]");
  std::vector<float2> tab(na);
  for (int v = 0; v < na; ++v) {
    const float theta = (float)((double)p.angles[v] * (kPi / 180.0));  // gen_forwproj.c:43
    float s, c;
    sincosf(theta, &s, &c);
    tab[v] = make_float2(c, s);
  }
  TOMO_CUDA(cudaMalloc(&p.d_angles, sizeof(float2) * (size_t)na));
  TOMO_CUDA(cudaMemcpy(p.d_angles, tab.data(), sizeof(float2) * (size_t)na, cudaMemcpyHostToDevice));
  const size_t lb = sizeof(float) * (size_t)na * p.g.lut_size;
  TOMO_CUDA(cudaMalloc(&p.d_aux, lb));
  TOMO_CUDA(cudaMemcpy(p.d_aux, p.g.lut, lb, cudaMemcpyHostToDevice));
  if (sizeof(float) * (size_t)p.g.lut_size > 200 * 1024)
    return fail(TOMO_EINVAL, "bspline: lut_size too large (one row must fit in shared memory)");
  auto *st = new BsState();
  p.ext = st;
  p.ext_free = bs_state_free;
  const BsConst k = make_const(p);
  const int n = p.g.n, L = p.g.lut_size;
  // (a table that is not finite would poison the pixels out of reach)
  bool finite = true;
  for (size_t i = 0; i < (size_t)na * L; ++i) {
    st->lutmax = std::max(st->lutmax, std::fabs(p.g.lut[i]));
    finite = finite && std::isfinite(p.g.lut[i]);
  }
  st->pow2 = finite && p.g.support == 4.0f && (L & (L - 1)) == 0 && L >= 64 && L <= 2048 && n >= 4 && n <= 4096;
  if (st->pow2) {
    // |ps| stays below sqrt(2) (n/2 + 1) + 4, also for a tile's pixels outside the image
    st->pads = (int)std::ceil((p.nh + 1) * 0.41422) + 64;
    st->w2 = n + 2 * st->pads;
    st->Q = bs_adj_shares(n);
    st->entries = 8 * (int)k.lut_step + 8;
    // the weights, and the rest for a chunk of slices
    const size_t lut4 = (size_t)na * 2 * (size_t)k.lut_step, s41 = (size_t)na * st->w2, framed1 = (size_t)n * (n + 2 * kBsFrame);
    const size_t part1 = st->Q > 1 ? (size_t)st->Q * n * n : 0;
    st->chunk = slice_chunk(p, sizeof(float4) * s41 + sizeof(float) * (2 * framed1 + part1) + sizeof(int) * na);
    const size_t nz = st->chunk, s4 = nz * s41, framed = nz * framed1, part = nz * part1;
    TOMO_CUDA(cudaMalloc(&st->work, sizeof(float4) * (lut4 + s4) + sizeof(float) * (2 * framed + part) + sizeof(int) * nz * na));
    st->lut4 = (float4 *)st->work;
    st->S4 = st->lut4 + lut4;
    st->rows = (float *)(st->S4 + s4);
    st->cols = st->rows + framed;
    st->partial = st->cols + framed;
    st->mark = (int *)(st->partial + part);
    bs_lut4_kernel<<<na, 256>>>((const float *)p.d_aux, st->lut4, k);
    TOMO_CUDA(cudaGetLastError());
    TOMO_CUDA(cudaStreamSynchronize(0));  // later calls may come on streams that do not wait for this one
  }
  TOMO_CUDA(cudaMalloc(&st->vmax, sizeof(unsigned) * (size_t)std::max(1, p.g.nz)));
  if (sizeof(float) * (size_t)L > 48 * 1024)
    TOMO_CUDA(cudaFuncSetAttribute(bs_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(float) * L)));
  // residual partials of the fused solvers: one per warp of the general forward
  p.fwd_warps = (size_t)((n + kBsBins - 1) / kBsBins) * (kBsThreads / 32) * na * p.g.nz;
  p.g.lut = nullptr;
  return TOMO_OK;
}

int bs_forward(Plan &p, const float *d_img, float *d_sino, cudaStream_t s, const FwdEpi &ep) {
  const BsConst k = make_const(p);
  BsState &st = *(BsState *)p.ext;
  if (st.pow2 && !ep.ordered) {
    const int n = k.n, tiles = (n + 2 * kBsFrame + 31) / 32, split = bs_fwd_split(n), bins = 128 / split;
    auto fn = split == 4 ? bs_forward_pow2_kernel<4> : bs_forward_pow2_kernel<2>;
    for (int z0 = 0; z0 < p.g.nz; z0 += st.chunk) {
      const int zc = std::min(st.chunk, p.g.nz - z0);
      bs_frame_kernel<<<dim3(tiles, tiles, zc), dim3(32, 8), 0, s>>>(d_img + (size_t)z0 * n * n, st.rows, st.cols, n);
      fn<<<dim3((n + bins - 1) / bins, k.na, zc), 128, sizeof(float) * (st.entries + 1), s>>>(
          st.rows, st.cols, d_sino + (size_t)z0 * k.na * n, (const float2 *)p.d_angles, (const float *)p.d_aux, st.entries, k);
    }
    TOMO_CUDA(cudaGetLastError());
    return TOMO_OK;
  }
  const size_t per = (size_t)k.n * k.n;
  TOMO_CUDA(cudaMemsetAsync(st.vmax, 0, sizeof(unsigned) * p.g.nz, s));
  fixed_finite_absmax_kernel<<<dim3((unsigned)std::min<size_t>((per + 255) / 256, 1184), p.g.nz), 256, 0, s>>>(d_img, per,
                                                                                                   st.vmax);
  dim3 fg((k.n + kBsBins - 1) / kBsBins, k.na, p.g.nz);
  bs_forward_kernel<<<fg, kBsThreads, sizeof(float) * k.lut_size, s>>>(
      d_img, d_sino, (const float2 *)p.d_angles, (const float *)p.d_aux, st.vmax, st.lutmax, k, ep);
  TOMO_CUDA(cudaGetLastError());
  return TOMO_OK;
}

int bs_adjoint(Plan &p, const float *d_sino, float *d_img, cudaStream_t s, const AdjEpi &ep) {
  const BsConst k = make_const(p);
  BsState &st = *(BsState *)p.ext;
  if (st.pow2 && !ep.ordered) {
    const int n = k.n, nz = p.g.nz;
    const size_t smem = sizeof(float4) * 2 * (size_t)k.lut_step;
    auto fn = (n & 1) ? bs_adjoint_pow2_kernel<true> : bs_adjoint_pow2_kernel<false>;
    for (int z0 = 0; z0 < nz; z0 += st.chunk) {
      const int zc = std::min(st.chunk, nz - z0);
      const float *sino = d_sino + (size_t)z0 * k.na * n;
      float *img = d_img + (size_t)z0 * n * n;
      bs_expand_kernel<<<k.na * zc, 256, 0, s>>>(sino, st.S4, st.mark, n, st.pads, st.w2);
      fn<<<dim3((n + kBsTW - 1) / kBsTW * st.Q, (n + kBsTH - 1) / kBsTH, zc), kBsThreads4, smem, s>>>(
          sino, st.S4, st.lut4, (const float *)p.d_aux, img, (const float2 *)p.d_angles, k, st.pads, st.w2, st.Q, st.partial);
      bs_adj_sum_kernel<<<dim3((unsigned)(((size_t)n * n + 255) / 256), zc), 256, 0, s>>>(
          st.partial, st.Q, img, sino, st.mark, (const float2 *)p.d_angles, (const float *)p.d_aux, k);
    }
    TOMO_CUDA(cudaGetLastError());
    return TOMO_OK;
  }
  dim3 ab(32, 8), ag((k.n + 31) / 32, (k.n + 7) / 8, p.g.nz);
  bs_adjoint_kernel<<<ag, ab, 0, s>>>(d_sino, d_img, (const float2 *)p.d_angles,
                                      (const float *)p.d_aux, k, ep);
  TOMO_CUDA(cudaGetLastError());
  return TOMO_OK;
}

}  // namespace tomo
