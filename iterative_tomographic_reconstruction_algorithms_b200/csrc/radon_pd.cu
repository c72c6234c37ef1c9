// Pixel-driven projector pair (linear interpolation, method 1) for sm_100a.
//
// Reference: common/operators/radon_module/pymodule_radon_pixel_driven/
// radon_pd.c:20-90.  Every pixel (i, j) -- stored at image row n-1-i
// (:61) -- is represented by four sub-samples; the reference offsets x and y by
// the SAME delta[2k+1] (:42-43), so the four are (-1/4,-1/4) twice and
// (+1/4,+1/4) twice.  A sub-sample lands at T = nh - t, t = +-|x s - y c| with
// the sign rule of :46-55, and is split linearly between bins floor(T) and
// ceil(T) with weights |ceil(T) - T| and |T - floor(T)|; bin 0 never receives
// (:74,76) and an integral T gets weight 0 in both.  Output row v follows the
// (fftshifted) angle order of the input.
//
// Evaluation order of the compiled reference (-O3 -ffast-math, read from its
// x86-64 code), reproduced exactly: t = |fma(-c, y, x*s)|, its sign for every angle
// that of pd_line, and the first weight is |(t + ceil(T)) - nh|.
//
// Forward = gather per bin over image lines; adjoint = gather per pixel over
// angles.  The duplicate sub-samples are evaluated once with weight 2 * 1/4.
#include <algorithm>
#include <cmath>

#include "f32x2.cuh"
#include "tomo_internal.cuh"

namespace tomo {
namespace {

constexpr float kPdMagic = 12582912.0f;  // 1.5 * 2^23
constexpr int kPdMagicBits = 0x4B400000;  // its bit pattern

// T = nh - t with t = fma(c', y, RN(x s')), (s', c') = (sigma sin, -sigma cos),
// sigma = -1 for cos >= 0, else +1: for every angle the sign rule (y > x s / c)
// picks t = sigma (x s - y c), and rounding is symmetric.  (Where the test and
// the product round differently, |t| is below the rounding of T.)
__device__ __forceinline__ float2 pd_line(const PdAngle &g) {
  const float sg = g.c >= 0.0f ? -1.0f : 1.0f;
  return make_float2(sg * g.s, -(sg * g.c));
}

// Framed copies of the image for the forward: rows[i][P + j] and
// cols[j][P + i] hold pixel (loop row i, column j), with P = kPdFrame zeros on
// either side of a line.
constexpr int kPdFrame = 4;

__global__ void __launch_bounds__(256) pd_frame_kernel(const float *__restrict__ img, float *__restrict__ rows,
                                                       float *__restrict__ cols, int n) {
  __shared__ float tile[32][33];
  const size_t z = blockIdx.z;
  const int w = n + 2 * kPdFrame;
  const float *src = img + z * (size_t)n * n;
  float *R = rows + z * (size_t)n * w, *C = cols + z * (size_t)n * w;
  const int j0 = blockIdx.x * 32 - kPdFrame, i0 = blockIdx.y * 32 - kPdFrame;  // tiles cover the frame too
  for (int dy = threadIdx.y; dy < 32; dy += 8) {
    const int i = i0 + dy, j = j0 + threadIdx.x;
    const float v = i >= 0 && i < n && j >= 0 && j < n ? __ldg(src + (size_t)(n - 1 - i) * n + j) : 0.0f;
    tile[dy][threadIdx.x] = v;
    if (i >= 0 && i < n && j < n + kPdFrame) R[(size_t)i * w + kPdFrame + j] = v;
  }
  __syncthreads();
  for (int dy = threadIdx.y; dy < 32; dy += 8) {
    const int j = j0 + dy, i = i0 + threadIdx.x;
    if (j >= 0 && j < n && i < n + kPdFrame) C[(size_t)j * w + kPdFrame + i] = tile[threadIdx.x][dy];
  }
}

// Forward: a lane owns a bin b of an angle and walks the lines (ROWS: image
// rows, when T moves faster along x; else columns).  On a line and for a
// sub-sample, T rises by sigma = max(|s|, |c|) in [0.707, 1] per pixel in
// direction DIR, so the pixels with T in (b - 1, b + 1) are among three
// consecutive ones, found from the line's crossing of b - 1 (0.05 early, far
// above its rounding: a fourth pixel would lie past b - 1.05 + 3 sigma > b + 1).
// Each is evaluated with the reference's arithmetic: the first lies below b
// (floor(T) = b - 1, weight T - floor(T)), the third above (floor(T) = b,
// weight (t + ceil(T)) - nh), the second on either side; an integral T puts |(t +
// T) - nh|, the rounding of t, and 0 into bin T.
//
// The products are added in double and rounded once: deterministic, and as close
// to their exact sum as the 64-bit fixed-point sums in shared memory that this
// replaces.  Those took two 32-bit atomics per product, and bounded the forward:
// 1.57 ms at 768^2 x 720, now 0.96 (2048^2 x 1800: 25.2, now 16.2).  Bound by
// issue and the FP32 pipe.  (Adding a line's products in float first takes a tenth
// less, but keeps 24 bits of the sum, and reaches infinity next to the largest float
// where the bin is finite.)

// A bin and its angle, as both loops use them.
template <bool ROWS, int DIR>
struct PdBin {
  float fnh, fb, bm, bp;
  F2 base2, slope2, ns, nc, nh2, nbm, nbp, off, dir;
  __device__ __forceinline__ PdBin(float s, float c, int b, int nh) {
    fnh = (float)nh;
    fb = (float)b;
    bm = fb - 1.0f;
    bp = fb + 1.0f;
    const float k = ROWS ? s : c, o = ROWS ? c : s;  // t along the line, across lines
    const float inv = 1.0f / k;
    // position (pixel index) at which T = b - 1: base + slope * (line coordinate)
    const float at = (fnh - bm) * inv + fnh - 0.5f;
    base2 = f2(at + 0.25f - DIR * 0.05f, at - 0.25f - DIR * 0.05f);
    slope2 = f2(-o * inv);
    ns = f2(-s);
    nc = f2(-c);
    nh2 = f2(fnh);
    nbm = f2(-bm);
    nbp = f2(-bp);
    off = f2(0.25f - fnh, 0.75f - fnh);
    dir = f2((float)DIR);
  }
  // -t of the three pixels from coordinate u0 (along the line) on
  __device__ __forceinline__ void nt(F2 l, F2 u0, F2 &t0, F2 &t1, F2 &t2) const {
    const F2 u1 = add2(u0, dir), u2 = add2(u1, dir);
    if (ROWS) {
      t0 = fma2(nc, l, mul2(u0, ns));
      t1 = fma2(nc, l, mul2(u1, ns));
      t2 = fma2(nc, l, mul2(u2, ns));
    } else {
      const F2 xs = mul2(l, ns);
      t0 = fma2(nc, u0, xs);
      t1 = fma2(nc, u1, xs);
      t2 = fma2(nc, u2, xs);
    }
  }
  // an integral T's weight |(t + T) - nh|
  __device__ __forceinline__ float on_bin(float nt) const { return fabsf(__fsub_rn(__fadd_rn(-nt, fb), fnh)); }
};

// Every product as the reference rounds it, added in double.
template <bool ROWS, int DIR>
__device__ __forceinline__ double pd_fwd_exact(const float *__restrict__ L, int w, float s, float c, int b, int n, int nh,
                                               int i0, int i1) {
  const PdBin<ROWS, DIR> B(s, c, b, nh);
  const float lo = DIR > 0 ? -4.0f : -2.0f, hi = DIR > 0 ? (float)(n + 1) : (float)(n + 3);
  const float *line = L + (size_t)i0 * w + kPdFrame - kPdMagicBits;
  float lc = (float)i0 - B.fnh + 0.5f;  // the line's own coordinate
  double acc = 0.0;
#pragma unroll 2
  for (int i = i0; i < i1; ++i, line += w, lc += 1.0f) {
    const F2 l = add2(f2(lc), f2(-0.25f, 0.25f));
    const float2 ps = unpack(fma2(B.slope2, l, B.base2));
    const F2 pos = f2(fminf(fmaxf(ps.x, lo), hi), fminf(fmaxf(ps.y, lo), hi));
    const F2 fm = DIR > 0 ? add2_ru(pos, f2(kPdMagic)) : add2_rd(pos, f2(kPdMagic));  // next pixels in DIR
    const float2 fs = unpack(fm);
    const float *va = line + __float_as_int(fs.x), *vb = line + __float_as_int(fs.y);
    F2 t0, t1, t2;
    B.nt(l, add2(add2(fm, f2(-kPdMagic)), B.off), t0, t1, t2);
    const float2 w0 = unpack(add2(add2(B.nh2, t0), B.nbm));
    const F2 T1 = add2(B.nh2, t1);
    const float2 Ts = unpack(T1), wa = unpack(add2(T1, B.nbm)), wb = unpack(add2(add2(t1, B.nbp), B.nh2));  // wb: -weight
    const float2 w2 = unpack(add2(add2(t2, B.nbp), B.nh2));                                                 // -weight
    const float2 n1 = unpack(t1), T2 = unpack(add2(B.nh2, t2));
    const float a0 = __ldg(va), a1 = __ldg(va + DIR), a2 = __ldg(va + 2 * DIR);
    const float b0 = __ldg(vb), b1 = __ldg(vb + DIR), b2 = __ldg(vb + 2 * DIR);
    // below b the first of wa, -wb is the smaller one, above the second
    float px = __fmul_rn(fminf(wa.x, -wb.x), a1), py = __fmul_rn(fminf(wa.y, -wb.y), b1);
    if (Ts.x == B.fb) px = __fmaf_rn(0.0f, a1, __fmul_rn(B.on_bin(n1.x), a1));
    if (Ts.y == B.fb) py = __fmaf_rn(0.0f, b1, __fmul_rn(B.on_bin(n1.y), b1));
    double r = 0.0, q = 0.0;
    if (w0.x > 0.0f) r += (double)__fmul_rn(w0.x, a0);
    r += (double)px;
    if (T2.x < B.bp) r += (double)__fmul_rn(fabsf(w2.x), a2);
    if (w0.y > 0.0f) q += (double)__fmul_rn(w0.y, b0);
    q += (double)py;
    if (T2.y < B.bp) q += (double)__fmul_rn(fabsf(w2.y), b2);
    acc += r + q;
  }
  return acc;
}

// Out of the register budget of the loop that falls back to it.
template <bool ROWS, int DIR>
__device__ __noinline__ double pd_fwd_again(const float *__restrict__ L, int w, float s, float c, int b, int n, int nh, int i0,
                                            int i1) {
  return pd_fwd_exact<ROWS, DIR>(L, w, s, c, b, n, nh, i0, i1);
}

// The same with the two sub-samples' weights of a pixel added first (both are
// multiples of the spacing of T, so their sum is exact for T >= 2): four pixels,
// products and conversions to double per line instead of six (1.35 ms at 768^2 x
// 720 with six).  A sum that is not finite, as one weight's zero or two weights'
// overflow can make it, is left to pd_fwd_exact.
template <bool ROWS, int DIR>
__device__ __forceinline__ double pd_fwd_bin(const float *__restrict__ L, int w, float s, float c, int b, int n, int nh,
                                             int i0, int i1) {
  const PdBin<ROWS, DIR> B(s, c, b, nh);
  // the four pixels from the next one on, or from the one above it, stay in the frame
  const float lo = DIR > 0 ? -4.0f : -1.0f, hi = DIR > 0 ? (float)n : (float)(n + 2);
  const float *line = L + (size_t)i0 * w + kPdFrame - kPdMagicBits;
  float lc = (float)i0 - B.fnh + 0.5f;
  double acc = 0.0;
#pragma unroll 2
  for (int i = i0; i < i1; ++i, line += w, lc += 1.0f) {
    const F2 l = add2(f2(lc), f2(-0.25f, 0.25f));
    const float2 ps = unpack(fma2(B.slope2, l, B.base2));
    const float pos = fminf(fmaxf(ps.y, lo), hi);
    const float fy = DIR > 0 ? __fadd_ru(pos, kPdMagic) : __fadd_rd(pos, kPdMagic);  // next pixel in DIR
    // The first sub-sample crosses 0 to 1 pixels above the second: its next
    // pixel is taken to be the same or the one above it (a rounding's pixel more
    // or less at the start is within the 0.05)
    const float iy = __fsub_rn(fy, kPdMagic), up = iy + 1.0f;
    const bool same = DIR > 0 ? ps.x <= iy : ps.x < up;
    const float *v = line + __float_as_int(fy) + (DIR < 0 && !same ? 1 : 0);
    const float v0 = __ldg(v), v1 = __ldg(v + DIR), v2 = __ldg(v + 2 * DIR), v3 = __ldg(v + 3 * DIR);
    F2 t0, t1, t2;
    B.nt(l, add2(f2(same ? iy : up, iy), B.off), t0, t1, t2);
    const float2 T0 = unpack(add2(B.nh2, t0)), T2 = unpack(add2(B.nh2, t2));
    const F2 T1 = add2(B.nh2, t1);
    const float2 Ts = unpack(T1), wa = unpack(add2(T1, B.nbm));
    // above b the weight of bin floor(T) is -((nt + ceil(T)) + nh)
    const F2 nce = f2(Ts.x == B.fb ? -B.fb : -B.bp, Ts.y == B.fb ? -B.fb : -B.bp);
    const float2 wb = unpack(add2(add2(t1, nce), B.nh2));
    // the first and the third weight are 0 for a pixel out of reach: a saturating
    // sum, and a test, for (t + ceil(T)) - nh is not 0 when T is b + 1
    const float x0 = __saturatef(__fsub_rn(T0.x, B.bm)), y0 = __saturatef(__fsub_rn(T0.y, B.bm));
    const float2 w2 = unpack(add2(add2(t2, B.nbp), B.nh2));  // -weight
    const float x2 = T2.x < B.bp ? -w2.x : 0.0f, y2 = T2.y < B.bp ? -w2.y : 0.0f;
    const float x1 = fminf(wa.x, fabsf(wb.x)), y1 = fminf(wa.y, fabsf(wb.y));
    // e: the sub-sample that starts first, g: the other
    const float e0 = DIR > 0 ? y0 : x0, e1 = DIR > 0 ? y1 : x1, e2 = DIR > 0 ? y2 : x2;
    const float g0 = DIR > 0 ? x0 : y0, g1 = DIR > 0 ? x1 : y1, g2 = DIR > 0 ? x2 : y2;
    const float p0 = __fmul_rn(e0 + (same ? g0 : 0.0f), v0), p1 = __fmul_rn(e1 + (same ? g1 : g0), v1);
    const float p2 = __fmul_rn(e2 + (same ? g2 : g1), v2), p3 = __fmul_rn(same ? 0.0f : g2, v3);
    acc += ((double)p0 + (double)p1) + ((double)p2 + (double)p3);
  }
  if (!(fabs(acc) < INFINITY)) acc = pd_fwd_again<ROWS, DIR>(L, w, s, c, b, n, nh, i0, i1);
  return acc;
}

// A block takes 32 bins of an angle, whose lines SPLIT warps share (their sums are
// added in order): bins alone are too few warps to hide a line's latency in small
// images, and few enough in large ones that the blocks' ends show.  The split
// depends on n alone (pd_fwd_split), so a plan for some of the angles or several
// slices gives the same bits.  SPLIT = 0 is the solvers' form (epilogue.cuh),
// pd_fwd_exact with a warp per bin, four angles to a block.
constexpr int kPdAng = 4;

template <int SPLIT>
__global__ void __launch_bounds__(32 * (SPLIT ? SPLIT : kPdAng), 32 / (SPLIT ? SPLIT : kPdAng)) pd_forward_kernel(
    const float *__restrict__ rows, const float *__restrict__ cols, float *__restrict__ sino, const PdAngle *__restrict__ tab,
    int n, int nh, int na, FwdEpi ep) {
  constexpr int kParts = SPLIT ? SPLIT : 1;
  __shared__ double part[kParts][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, v = SPLIT ? blockIdx.y : blockIdx.y * kPdAng + warp;
  const int B0 = blockIdx.x * 32, b = B0 + lane, w = n + 2 * kPdFrame;
  const size_t z = blockIdx.z;
  const bool live = v < na && b < n;
  double acc = 0.0;
  if (v < na) {  // warp-uniform
    const float2 g = pd_line(tab[v]);
    const float s = g.x, c = g.y, fnh = (float)nh;
    const bool by_rows = fabsf(s) >= fabsf(c);
    // lines whose T range, nh - o l +- |k| (nh + 2), meets (B0 - 1, B0 + 32)
    const float k = fabsf(by_rows ? s : c), o = by_rows ? c : s, half = k * (fnh + 2.0f);
    int i0 = 0, i1 = n;
    if (fabsf(o) > 1e-4f) {
      const float l0 = (fnh - half - (float)(B0 + 33)) / o, l1 = (fnh + half - (float)(B0 - 2)) / o;
      i0 = max(0, (int)floorf(fminf(fmaxf(fminf(l0, l1) + fnh - 2.0f, 0.0f), (float)n)));
      i1 = min(n, (int)ceilf(fminf(fmaxf(fmaxf(l0, l1) + fnh + 2.0f, 0.0f), (float)n)));
    }
    if (SPLIT) {
      const int len = max(0, i1 - i0);
      i1 = i0 + len * (warp + 1) / kParts;
      i0 += len * warp / kParts;
    }
    const float *L = (by_rows ? rows : cols) + z * (size_t)n * w;
#define PD_BIN(R, D) (SPLIT ? pd_fwd_bin<R, D>(L, w, s, c, b, n, nh, i0, i1) : pd_fwd_exact<R, D>(L, w, s, c, b, n, nh, i0, i1))
    if (by_rows) acc = s < 0.0f ? PD_BIN(true, 1) : PD_BIN(true, -1);
    else acc = c < 0.0f ? PD_BIN(false, 1) : PD_BIN(false, -1);
#undef PD_BIN
  }
  if (SPLIT) {
    part[warp][lane] = acc;
    __syncthreads();
    if (warp > 0) return;
    for (int q = 1; q < SPLIT; ++q) acc += part[q][lane];
  }
  // bin 0 never receives; 0.5: two coinciding quarter-weight sub-samples
  const float out = b >= 1 ? (float)(0.5 * acc) : 0.0f;
  double r2 = 0.0;
  const size_t e = z * (size_t)na * n + (size_t)v * n + b;
  if (live) sino[e] = fwd_apply(ep, out, e, r2);
  const size_t block = ((size_t)z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  fwd_resid_commit(ep, r2, SPLIT ? block : block * kPdAng + warp);
}

// ms with 1 (four angles to a block), 4, 8 warps: 200^2 x 200 0.046, 0.042, 0.038; 320^2
// x 320 0.114, 0.099, 0.097; 384^2 x 400 0.177, 0.159, 0.157; 512^2 x 500 0.353, 0.321, 0.319;
// 768^2 x 720 1.033, 0.962, 0.966; 2048^2 x 1800 16.4, 16.2, 16.2.  Several slices do with
// fewer (8 x 256^2 x 300: 0.402, 0.390, 0.401), but a slice has the same bits in any call.
int pd_fwd_split(int n) { return n > 320 ? 4 : 8; }

// Sinogram rows as pairs, entry e = l + pads of angle v: {S_l, S_l+1}, the two
// bins a sub-sample with floor(T) = l is split between; bin 0 and the bins
// outside [0, n) never receive and are 0 here, so the adjoint's loop tests no
// bounds.
__global__ void __launch_bounds__(256) pd_expand_kernel(const float *__restrict__ sino, float2 *__restrict__ out, int n,
                                                        int pads, int w2) {
  const size_t row = blockIdx.x;  // z * na + v
  const float *src = sino + row * n;
  float2 *dst = out + row * w2;
  for (int e = threadIdx.x; e < w2; e += blockDim.x) {
    const int l = e - pads;
    dst[e] = make_float2(l >= 1 && l < n ? __ldg(src + l) : 0.0f, l + 1 >= 1 && l + 1 < n ? __ldg(src + l + 1) : 0.0f);
  }
}

// Adjoint: a lane holds 4 x 4 pixels of a 32 x 16 tile; the Q warps of a block
// sum Q contiguous shares of the angles, added in order through shared memory
// (Q depends on n alone, so the result does not depend on the device).  Q = 1 is
// the solvers' form (epilogue.cuh), one chain in the reference's order, with a
// row of 4 pixels per lane (R = 1) for small images.
//
// Per sub-sample: t and T as the reference rounds them, the pair at floor(T)
// in one 8-byte read, and its two weights, which carry the factor 1/2 of the two
// coinciding quarter-weight sub-samples (scaling by it rounds nothing; without it
// the sums would reach infinity at half the largest float).  An integral T, where
// floor and ceil are one bin, is rare and takes the branch.
//
// Bound by L1 (70 % of its rate) and FP32 (65 %): 9 operations and 2 FMAs per
// sub-sample, whose table pairs hit L1.  The two sub-samples go as f32x2 pairs,
// which halves the instructions (scalar ones: 0.57 ms against 0.51).  A thread
// per pixel with four reads, bounds tests and the sign rule per sub-sample took
// 1.52 ms at 768^2 x 720 and 25.5 at 2048^2 x 1800; this one 0.49 and 8.0.
constexpr int kPdGrp = 2;  // pixels that share the test for an integral T
template <int Q, int R>
__global__ void __launch_bounds__(32 * Q) pd_adjoint_kernel(const float2 *__restrict__ pairs, float *__restrict__ img,
                                                            const PdAngle *__restrict__ tab, int n, int nh, int na, int pads,
                                                            int w2, AdjEpi ep) {
  __shared__ float part[Q > 1 ? (Q - 1) * 4 * R : 1][32];
  const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
  const int b0 = blockIdx.x * 32 + 4 * (lane & 7), a0 = blockIdx.y * 4 * R + R * (lane >> 3);
  const size_t z = blockIdx.z;
  const float fnh = (float)nh;
  float acc[R][4];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
  const int u0 = (int)((long long)na * q / Q), u1 = (int)((long long)na * (q + 1) / Q);
  if (a0 < n && b0 < n) {
    const float x0 = (float)b0 - fnh + 0.5f, y0 = (float)(n - 1 - a0) - fnh + 0.5f;  // rows go up in y
    const F2 nh2 = f2(fnh), magic = f2(kPdMagic), half = f2(0.5f), nhalf = f2(-0.5f), hnh = f2(0.5f * fnh);
    const F2 hm = f2(0.5f * kPdMagic), hm1 = f2(0.5f * (kPdMagic - 1.0f));
    // row base minus the bits of the magic floor
    const float2 *row = pairs + (z * na + u0) * (size_t)w2 + pads - kPdMagicBits;
#pragma unroll 1
    for (int u = u0; u < u1; ++u, row += w2) {
      const float2 g = pd_line(tab[u]);
      const float s = g.x, c = g.y;
      // both sub-samples as a pair; nt = -t
      const F2 ns = f2(-s), nc = f2(-c);
      F2 xs[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) xs[j] = mul2(f2(x0 + (float)j - 0.25f, x0 + (float)j + 0.25f), ns);
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const F2 y = f2(y0 - (float)i - 0.25f, y0 - (float)i + 0.25f);
#pragma unroll
        for (int j0 = 0; j0 < 4; j0 += kPdGrp) {
        float2 wu[kPdGrp], wl[kPdGrp], Sa[kPdGrp], Sb[kPdGrp];
        F2 nt[kPdGrp];
#pragma unroll
        for (int j = 0; j < kPdGrp; ++j) {
          nt[j] = fma2(nc, y, xs[j0 + j]);
          const F2 T = add2(nh2, nt[j]);
          // floor(T) without the conversion pipe: T + 1.5 * 2^23 rounded down
          // lies where floats are the integers (|T| < 2^22), and its bits give
          // the integer
          const F2 fd = add2_rd(T, magic);
          const float2 fs = unpack(fd);
          Sa[j] = __ldg(row + __float_as_int(fs.x));
          Sb[j] = __ldg(row + __float_as_int(fs.y));
          // halves of the reference's weights T - floor(T) and, negative, (t + ceil(T)) - nh
          wu[j] = unpack(fma2(T, half, fma2(fd, nhalf, hm)));
          wl[j] = unpack(add2(fma2(nt[j], half, fma2(fd, nhalf, hm1)), hnh));
        }
        float least = fminf(wu[0].x, wu[0].y);
#pragma unroll
        for (int j = 1; j < kPdGrp; ++j) least = fminf(least, fminf(wu[j].x, wu[j].y));
        if (least == 0.0f) {  // an integral T: floor and ceil are one bin
#pragma unroll
          for (int j = 0; j < kPdGrp; ++j) {
            const float2 t = unpack(nt[j]);
            if (wu[j].x == 0.0f) {
              wl[j].x = -0.5f * fabsf(__fsub_rn(__fadd_rn(-t.x, __fadd_rn(fnh, t.x)), fnh));
              Sa[j].y = Sa[j].x;
            }
            if (wu[j].y == 0.0f) {
              wl[j].y = -0.5f * fabsf(__fsub_rn(__fadd_rn(-t.y, __fadd_rn(fnh, t.y)), fnh));
              Sb[j].y = Sb[j].x;
            }
          }
        }
#pragma unroll
        for (int j = 0; j < kPdGrp; ++j) {
          acc[i][j0 + j] = __fmaf_rn(wu[j].x, Sa[j].y, __fmaf_rn(-wl[j].x, Sa[j].x, acc[i][j0 + j]));
          acc[i][j0 + j] = __fmaf_rn(wu[j].y, Sb[j].y, __fmaf_rn(-wl[j].y, Sb[j].x, acc[i][j0 + j]));
        }
        }
      }
    }
  }
  if (q > 0)
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) part[(q - 1) * 4 * R + 4 * i + j][lane] = acc[i][j];
  __syncthreads();
  if (q > 0) return;
#pragma unroll
  for (int r = 0; r < Q - 1; ++r)
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] += part[r * 4 * R + 4 * i + j][lane];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int y = a0 + i, x = b0 + j;
      const bool live = y < n && x < n;
      adj_store(ep, acc[i][j], live, z * (size_t)n * n + (live ? (size_t)y * n + x : 0), img);
    }
}

// What the pair owns beside the angle table.
struct PdState {
  float *rows = nullptr, *cols = nullptr;  // [chunk][n][n + 2 kPdFrame]
  float2 *pairs = nullptr;                 // [chunk][na][w2]
  int pads = 0, w2 = 0, chunk = 1;
};

void pd_state_free(void *q) {
  auto *st = (PdState *)q;
  cudaFree(st->pairs);
  delete st;
}

// Warps of an adjoint tile.  ms with 4, 8, 16: 256^2 x 300 0.079, 0.052, 0.040; 320^2 x
// 320 0.089, 0.071, 0.071; 512^2 x 500 0.196, 0.187, 0.192; 768^2 x 720 0.510, 0.491, 0.513;
// 2048^2 x 1800 8.03, 8.03, 8.51.  (8 x 256^2 x 300: 0.200, 0.192, 0.212.)
int pd_adj_warps(int n) { return n > 320 ? 8 : 16; }

}  // namespace

int pd_setup(Plan &p) {
  const int na = p.g.na;
  std::vector<PdAngle> tab(na);
  for (int v = 0; v < na; ++v) {
    float s, c;
    sincosf(p.angles[v], &s, &c);
    PdAngle a{};
    a.s = s;
    a.c = c;
    tab[v] = a;
  }
  TOMO_CUDA(cudaMalloc(&p.d_angles, sizeof(PdAngle) * (size_t)na));
  TOMO_CUDA(cudaMemcpy(p.d_angles, tab.data(), sizeof(PdAngle) * (size_t)na, cudaMemcpyHostToDevice));
  auto *st = new PdState();
  p.ext = st;
  p.ext_free = pd_state_free;
  // |t| stays below sqrt(2) (nh + 1), also for the pixels of a tile that lie
  // up to 3 outside the image
  st->pads = (int)std::ceil((p.nh + 1) * 0.41422) + 12;
  st->w2 = p.g.n + 2 * st->pads;
  // one workspace for a chunk of slices: the adjoint's pairs, then the forward's framed copies
  const size_t pairs1 = (size_t)na * st->w2, framed1 = (size_t)p.g.n * (p.g.n + 2 * kPdFrame);
  st->chunk = slice_chunk(p, sizeof(float2) * pairs1 + 2 * sizeof(float) * framed1);
  const size_t pairs = st->chunk * pairs1, framed = st->chunk * framed1;
  TOMO_CUDA(cudaMalloc(&st->pairs, sizeof(float2) * pairs + 2 * sizeof(float) * framed));
  st->rows = (float *)(st->pairs + pairs);
  st->cols = st->rows + framed;
  // residual partials of the fused solvers: one per warp of the forward launch
  p.fwd_warps = (size_t)((p.g.n + 31) / 32) * ((na + kPdAng - 1) / kPdAng) * kPdAng * p.g.nz;
  return TOMO_OK;
}

int pd_forward(Plan &p, const float *d_img, float *d_sino, cudaStream_t s, const FwdEpi &ep) {
  const int n = p.g.n, na = p.g.na, nz = p.g.nz;
  PdState &st = *(PdState *)p.ext;
  const int tiles = (n + 2 * kPdFrame + 31) / 32;
  const int split = ep.ordered ? 0 : pd_fwd_split(n), warps = split ? split : kPdAng;
  auto fn = split == 8 ? pd_forward_kernel<8> : split == 4 ? pd_forward_kernel<4> : pd_forward_kernel<0>;
  const size_t per = (size_t)n * n, per_sino = (size_t)na * n, slots = p.fwd_warps / nz;
  for (int z0 = 0; z0 < nz; z0 += st.chunk) {
    const int zc = std::min(st.chunk, nz - z0);
    pd_frame_kernel<<<dim3(tiles, tiles, zc), dim3(32, 8), 0, s>>>(d_img + z0 * per, st.rows, st.cols, n);
    fn<<<dim3((n + 31) / 32, split ? na : (na + kPdAng - 1) / kPdAng, zc), 32 * warps, 0, s>>>(
        st.rows, st.cols, d_sino + z0 * per_sino, (const PdAngle *)p.d_angles, n, p.nh, na,
        epi_from(ep, z0 * per_sino, z0 * slots));
  }
  TOMO_CUDA(cudaGetLastError());
  return TOMO_OK;
}

int pd_adjoint(Plan &p, const float *d_sino, float *d_img, cudaStream_t s, const AdjEpi &ep) {
  const int n = p.g.n, na = p.g.na, nz = p.g.nz;
  PdState &st = *(PdState *)p.ext;
  const int Q = ep.ordered ? 1 : pd_adj_warps(n), R = ep.ordered && n <= 1024 ? 1 : 4;
  auto fn = R == 1    ? pd_adjoint_kernel<1, 1>
            : Q == 1  ? pd_adjoint_kernel<1, 4>
            : Q == 8  ? pd_adjoint_kernel<8, 4>
                      : pd_adjoint_kernel<16, 4>;
  const size_t per = (size_t)n * n, per_sino = (size_t)na * n;
  for (int z0 = 0; z0 < nz; z0 += st.chunk) {
    const int zc = std::min(st.chunk, nz - z0);
    pd_expand_kernel<<<na * zc, 256, 0, s>>>(d_sino + z0 * per_sino, st.pairs, n, st.pads, st.w2);
    fn<<<dim3((n + 31) / 32, (n + 4 * R - 1) / (4 * R), zc), 32 * Q, 0, s>>>(
        st.pairs, d_img + z0 * per, (const PdAngle *)p.d_angles, n, p.nh, na, st.pads, st.w2, epi_from(ep, z0 * per));
  }
  TOMO_CUDA(cudaGetLastError());
  return TOMO_OK;
}

}  // namespace tomo
