// 3x3 convolution (stride 1, zero padding 1) on the tensor cores (sm_100a):
// one GEMM with M = output pixels, N = output channels, K = 9 x input channels.
//
// An M tile is 8 x 16 output pixels.  Its input patch (10 x 18 pixels) is
// staged once, by one TMA box per block of 64 channels (32, 16 or 8 where the
// channel count asks for it), a pixel to a swizzled row; TMA's fill gives the
// zero padding.  The im2col rows of tap (dy, dx) are the patch's rows shifted
// by 10 dy + dx, with 8-row groups one patch row apart, so nine descriptors
// read all nine taps from the one copy.
//
// A persistent CTA per SM, warps by role: one stages patches, one weights, one or
// two issue the MMAs, two sets of four run the epilogue, each out of its own one
// of two TMEM accumulator sets.  Weights that fit beside three patches stay in
// shared memory for all of a CTA's tiles; others stream through a ring, and
// then two M tiles share each stage where their patches fit: a 128-pixel tile
// alone asks for 64 bytes of weights per clock of MMA time, about what L2
// gives an SM (16-byte cp.async copies, as before, stopped at 15).
//
// K runs tap by tap, channels ascending, 16 per MMA, whatever the shape of the
// launch, so a layer's result does not depend on it (above 384 channels the
// channels are taken 384 at a time).
//
// Measured, 4 images: 32 -> 32 channels at 768^2 0.99 -> 0.132 ms, 128 -> 128
// at 192^2 0.45 -> 0.049 ms (895 TFLOP/s), 256 -> 256 at 96^2 0.32 -> 0.046 ms.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "nn_ptx.cuh"

namespace tomo_nn {
namespace {

constexpr int kTW = 8, kTH = 16;             // output pixels of an M tile
constexpr int kPW = kTW + 2, kPH = kTH + 2;  // its input patch
constexpr int kPatch = kPW * kPH;
constexpr int kEpiWarps = 8;                 // two sets of four
constexpr int kConvThreads = (kEpiWarps + 4) * 32;
constexpr int kMaxSlots = 8, kMaxW = 8;
constexpr int kMaxPass = 384;                // channels of a patch
constexpr int kSms = 148;
constexpr int kSmemMax = 225 * 1024;
constexpr int kDrainSpins = 1 << 22;

struct ConvArgs {
  const float *bias;
  const __nv_bfloat16 *mask;  // outputs stand where it is > 0 (0 elsewhere); laid out like Yb
  float *Yf;
  __nv_bfloat16 *Yb;
  unsigned *status;
  int spins;
  int H, W, Cin, Cout, relu;
  int ntiles, ngroups;
  FastDiv ftx, fty;         // tiles of a row, rows of tiles of an image
  int NB, BN;               // output-channel blocks and their width
  int T, NS, NW, resident;  // tiles per group, patch slots, weight stages
  int issuers;              // warps that issue MMAs
  int npass, cpp;           // channel passes, channels per pass
  int rb, chb, kch;         // bytes of a row, its channels, channels of a weight stage (chb, or 16 when rows hold 8)
  int nblk, wblks, kblk16;  // channel blocks of a pass, weight blocks of a stage, bytes / 16 from a stage's patch block to the next
  int pblk, slot_bytes;     // bytes of a patch's channel block, of a slot
  int wblk, stage_bytes;    // bytes of a weight block (chb channels), of a stage
  int w_off, zero_off, bias_off, cols;
  int vec;                  // the output can be stored 16 bytes at a time
};

// KS: K steps of a weight stage (rows of 128, 64, and 32 or 16 bytes: 4, 2, 1);
// RES: the weights stay in shared memory (then T = 1 and one channel pass).
template <int KS, bool RES>
__global__ void __launch_bounds__(kConvThreads, 1) conv_tc_kernel(ConvArgs g, const __grid_constant__ CUtensorMap mx,
                                                                  const __grid_constant__ CUtensorMap mw) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t pfull[kMaxSlots], pempty[kMaxSlots], wfull[kMaxW], wempty[kMaxW], afull[2], aempty[2], done[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int gave_up;
  unsigned char *smem = (unsigned char *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);  // swizzle period
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int n0 = (blockIdx.x % g.NB) * g.BN, nv = min(g.BN, g.Cout - n0);
  const int grp0 = blockIdx.x / g.NB, gstep = gridDim.x / g.NB;
  const uint32_t base = smem_u32(smem);
  float *sbias = (float *)(smem + g.bias_off);
  const int c16 = (g.Cin + 15) / 16 * 16;

  if (warp == kEpiWarps + 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                 "r"(g.cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  if (tid == 0) {
    for (int s = 0; s < g.NS; ++s) {
      mbar_init(smem_u32(&pfull[s]), 1);
      mbar_init(smem_u32(&pempty[s]), 1);
    }
    for (int s = 0; s < g.NW; ++s) {
      mbar_init(smem_u32(&wfull[s]), 1);
      mbar_init(smem_u32(&wempty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&afull[s]), 1);
      mbar_init(smem_u32(&aempty[s]), 128);
    }
    mbar_init(smem_u32(&done[0]), 1);
    mbar_init(smem_u32(&done[1]), 1);
    gave_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  for (int i = tid; i < g.BN; i += kConvThreads) sbias[i] = (g.bias && i < nv) ? g.bias[n0 + i] : 0.0f;
  if (g.Cin == 8) {  // zeros: the K half behind the last tap, of the patch and of the weights
    for (int i = tid; i < (kPatch + g.BN) * 4; i += kConvThreads) ((uint32_t *)(smem + g.zero_off))[i] = 0u;
    fence_proxy_async();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  bool ok = true;

  if (warp < kEpiWarps) {  // epilogue: a lane is a pixel, warp w of a set owns accumulator rows 32w .. 32w+31
    const int set = warp >> 2, w4 = warp & 3;
    int job = set;
    for (int grp = grp0 + set * gstep; grp < g.ngroups; grp += 2 * gstep, job += 2) {
      const int tc = min(g.T, g.ntiles - grp * g.T);
      ok = warp_wait(&afull[set], (job >> 1) & 1, g.spins, &gave_up);  // the loads below take the whole warp
      if (!ok) break;
      tc_fence_after();
      for (int t = 0; t < tc; ++t) {
        const int tile = grp * g.T + t, row = fast_div(tile, g.ftx), b = fast_div(row, g.fty);
        const int tx = tile - row * g.ftx.d, ty = row - b * g.fty.d;
        const int m = w4 * 32 + lane, y = ty * kTH + (m >> 3), x = tx * kTW + (m & 7);
        const bool in = y < g.H && x < g.W;
        const size_t o = in ? (((size_t)b * g.H + y) * g.W + x) * g.Cout + n0 : 0;
        for (int c0 = 0; c0 < nv; c0 += 16) {
          float v[16];
          __syncwarp();  // lanes outside the image skipped the stores
          tmem_ld16(tmem + ((uint32_t)(w4 * 32) << 16) + (uint32_t)((set * g.T + t) * g.BN + c0), v);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            v[i] += sbias[c0 + i];
            if (g.relu) v[i] = fmaxf(v[i], 0.0f);
          }
          if (!in) continue;
          if (g.Yb) {
            __nv_bfloat16 *d = g.Yb + o + c0;
            if (g.mask) {
              const __nv_bfloat16 *k = g.mask + o + c0;
              if (g.vec) {
                const uint4 a = __ldg((const uint4 *)k), b = c0 + 8 < nv ? __ldg((const uint4 *)(k + 8)) : a;
                const unsigned w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  if (!(__uint_as_float(w[i] << 16) > 0.0f)) v[2 * i] = 0.0f;
                  if (!(__uint_as_float(w[i] & 0xffff0000u) > 0.0f)) v[2 * i + 1] = 0.0f;
                }
              } else {
#pragma unroll
                for (int i = 0; i < 16; ++i)
                  if (c0 + i < nv && !(__bfloat162float(k[i]) > 0.0f)) v[i] = 0.0f;
              }
            }
            if (g.vec) {  // nv is a multiple of 8
              unsigned w[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
                w[i] = *(const unsigned *)&h;
              }
              *(uint4 *)d = make_uint4(w[0], w[1], w[2], w[3]);
              if (c0 + 8 < nv) *(uint4 *)(d + 8) = make_uint4(w[4], w[5], w[6], w[7]);
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (c0 + i < nv) d[i] = __float2bfloat16_rn(v[i]);
            }
          } else {
            float *d = g.Yf + o + c0;
            if (g.vec) {  // nv is a multiple of 4
#pragma unroll
              for (int i = 0; i < 16; i += 4)
                if (c0 + i < nv) *(float4 *)(d + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (c0 + i < nv) d[i] = v[i];
            }
          }
        }
      }
      tc_fence_before();
      mbar_arrive(smem_u32(&aempty[set]));
    }
  } else if (warp == kEpiWarps) {  // patches
    if (lane == 0) {
      Ring r;
      int it = 0;
      for (int grp = grp0; grp < g.ngroups && ok; grp += gstep) {
        const int tc = min(g.T, g.ntiles - grp * g.T);
        for (int k = 0; k < tc * g.npass; ++k, ++it, r.next(g.NS)) {  // npass > 1 only with T == 1
          const int tile = grp * g.T + (g.npass > 1 ? 0 : k), ch0 = g.npass > 1 ? k * g.cpp : 0;
          if (it >= g.NS) ok = role_wait(&pempty[r.s], r.ph ^ 1u, g.spins, &gave_up);
          if (!ok) break;
          const int row = fast_div(tile, g.ftx), b = fast_div(row, g.fty), tx = tile - row * g.ftx.d, ty = row - b * g.fty.d;
          const int nb = g.npass == 1 ? g.nblk : (min(g.cpp, c16 - ch0) + g.chb - 1) / g.chb;
          const uint32_t bar = smem_u32(&pfull[r.s]), dst = base + r.s * g.slot_bytes;
          mbar_expect(bar, nb * kPatch * g.rb);
          for (int c = 0; c < nb; ++c)
            tma_load4(dst + c * g.pblk, &mx, ch0 + c * g.chb, tx * kTW - 1, ty * kTH - 1, b, bar);
        }
      }
      // copies still in flight (after a wait that gave up nobody else waits for them)
      for (int k = max(0, it - g.NS); k < it; ++k)
        if (!mbar_wait(smem_u32(&pfull[k % g.NS]), (k / g.NS) & 1, kDrainSpins)) ok = false;
    }
  } else if (warp == kEpiWarps + 1) {  // weights
    if (lane == 0) {
      if (g.resident) {
        const uint32_t bar = smem_u32(&wfull[0]);
        const int per = g.Cin == 8 ? 1 : (g.cpp + g.kch - 1) / g.kch * g.wblks;  // blocks of a tap
        mbar_expect(bar, 9 * per * g.BN * g.rb);
        for (int tap = 0; tap < 9; ++tap)
          for (int c = 0; c < per; ++c) tma_load3(base + g.w_off + (tap * per + c) * g.wblk, &mw, c * g.chb, tap, n0, bar);
        if (!mbar_wait(bar, 0, kDrainSpins)) ok = false;
      } else {
        Ring r;
        int it = 0;
        for (int grp = grp0; grp < g.ngroups && ok; grp += gstep)
          for (int p = 0; p < g.npass && ok; ++p) {
            const int ch0 = p * g.cpp, chs = min(g.cpp, c16 - ch0);
            for (int tap = 0; tap < 9 && ok; ++tap)
              for (int c0 = 0; c0 < chs; c0 += g.kch, ++it, r.next(g.NW)) {
                if (it >= g.NW) ok = role_wait(&wempty[r.s], r.ph ^ 1u, g.spins, &gave_up);
                if (!ok) break;
                const uint32_t bar = smem_u32(&wfull[r.s]), dst = base + g.w_off + r.s * g.stage_bytes;
                mbar_expect(bar, g.wblks * g.BN * g.rb);
                for (int c = 0; c < g.wblks; ++c)
                  tma_load3(dst + c * g.wblk, &mw, ch0 + c0 + c * g.chb, tap, n0, bar);
              }
          }
        for (int k = max(0, it - g.NW); k < it; ++k)
          if (!mbar_wait(smem_u32(&wfull[k % g.NW]), (k / g.NW) & 1, kDrainSpins)) ok = false;
      }
    }
  } else if (warp - (kEpiWarps + 2) < g.issuers) {  // MMAs; of two warps each takes every other tile
    const int step = RES ? g.issuers : 1, me = warp - (kEpiWarps + 2);
    const uint32_t idesc = instr_desc(g.BN);
    // descriptors of address 0; rows of 16 bytes hold 8 k, and the other 8 of
    // an MMA lie in the next block
    const uint64_t dx0 = smem_desc_rb(0, g.rb == 16 ? g.pblk : 16, kPW * g.rb, g.rb);
    const uint64_t dw0 = smem_desc_rb(0, g.rb == 16 ? g.wblk : 16, 8 * g.rb, g.rb);
    Ring pr, wr, ar;  // patch slots, weight stages, accumulator sets
    bool issued = false;
    if (me == 1) {
      pr.next(g.NS);
      ar.next(2);
    }
    const int first = grp0 + me * gstep;
    for (int grp = first; grp < g.ngroups && ok; grp += step * gstep) {
      const int tc = min(g.T, g.ntiles - grp * g.T);
      if (grp >= grp0 + 2 * gstep) ok = warp_wait(&aempty[ar.s], ar.ph ^ 1u, g.spins, &gave_up);
      if (ok && g.resident && grp == first) ok = warp_wait(&wfull[0], 0, g.spins, &gave_up);
      const uint32_t acc = tmem + (uint32_t)(ar.s * g.T * g.BN);
      for (int p = 0; p < g.npass && ok; ++p) {
        Ring slot[2];
        slot[0] = pr;
        pr.next(g.NS);
        slot[1] = pr;
        if (tc > 1) pr.next(g.NS);
        ok = warp_wait(&pfull[slot[0].s], slot[0].ph, g.spins, &gave_up);
        if (ok && tc > 1) ok = warp_wait(&pfull[slot[1].s], slot[1].ph, g.spins, &gave_up);
        if (!ok) break;
        tc_fence_after();
        issued = true;
        const uint32_t pa[2] = {base + slot[0].s * g.slot_bytes, base + slot[1].s * g.slot_bytes};
        if (KS == 1 && RES && g.Cin == 8) {  // two taps to an MMA: their patch offsets differ by the K-group stride
          const uint32_t wb = base + g.w_off, zr = base + g.zero_off;
#pragma unroll
          for (int i = 0; i < 5; ++i) {
            const int ta = 2 * i, tb = 2 * i + 1;
            const uint32_t oa = pa[0] + ((ta / 3) * kPW + ta % 3) * 16;
            const uint32_t ob = tb < 9 ? pa[0] + ((tb / 3) * kPW + tb % 3) * 16 : zr;
            const uint32_t wa = wb + ta * g.wblk, wn = tb < 9 ? wa + g.wblk : zr + kPatch * 16;
            mma_warp<1>(acc, smem_desc(oa, ob - oa, kPW * 16), smem_desc(wa, wn - wa, 128), idesc, i > 0 ? 1u : 0u);
          }
        } else {
          const int nk = (min(g.cpp, c16 - p * g.cpp) + g.kch - 1) / g.kch;
          uint32_t more = p > 0, wb = (base + g.w_off) >> 4;  // RES: the stages follow one another
          uint32_t xa = pa[0] >> 4, xb = pa[1] >> 4;
          const uint32_t px16 = g.rb >> 4, st16 = g.stage_bytes >> 4;
          for (int dy = 0; dy < 3 && ok; ++dy) {
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
              if (!RES && !ok) break;
              uint64_t da = dx0 + xa, db = dx0 + xb;
              for (int c = 0; c < nk; ++c) {
                if (!RES) {
                  ok = warp_wait(&wfull[wr.s], wr.ph, g.spins, &gave_up);
                  if (!ok) break;
                  tc_fence_after();
                  wb = (base + g.w_off + wr.s * g.stage_bytes) >> 4;
                }
                const uint64_t dw = dw0 + wb;
                mma_warp<KS>(acc, da, dw, idesc, more);
                if (!RES && tc > 1) mma_warp<KS>(acc + g.BN, db, dw, idesc, more);
                more = 1;
                da += g.kblk16;
                db += g.kblk16;
                wb += st16;
                if (!RES) {
                  mma_commit_warp(smem_u32(&wempty[wr.s]));
                  wr.next(g.NW);
                }
              }
              xa += dx < 2 ? px16 : (kPW - 2) * px16;  // the next tap's first pixel
              xb += dx < 2 ? px16 : (kPW - 2) * px16;
            }
          }
          if (!ok) break;
        }
        mma_commit_warp(smem_u32(&pempty[slot[0].s]));
        if (tc > 1) mma_commit_warp(smem_u32(&pempty[slot[1].s]));
      }
      if (ok) mma_commit_warp(smem_u32(&afull[ar.s]));
      ar.next(2);
      if (step == 2) {  // the other warp's tile
        pr.next(g.NS);
        ar.next(2);
      }
    }
    // every MMA issued so far, also on the way out of a wait that gave up
    if (issued) {
      mma_commit_warp(smem_u32(&done[me]));
      if (!mbar_wait(smem_u32(&done[me]), 0, kDrainSpins)) ok = false;
    }
  }
  if (!ok) atomicOr(&gave_up, 1);
  __syncwarp();
  __syncthreads();
  tc_fence_after();
  if (gave_up && tid == 0 && g.status) atomicOr(g.status, 1);
  if (warp == kEpiWarps + 2)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(g.cols));
}

int up1k(int b) { return (b + 1023) / 1024 * 1024; }

}  // namespace

int conv_launch(const __nv_bfloat16 *X, int batch, int H, int W, int Cin, const __nv_bfloat16 *Wt, int Cout, float *Yf,
                __nv_bfloat16 *Yb, const float *bias, int relu, const __nv_bfloat16 *mask, unsigned *status, int spins, cudaStream_t s) {
  if (batch < 1 || H < 1 || W < 1 || Cin < 8 || Cin % 8 || Cout < 1) return NN_EINVAL;
  if ((long long)batch * H * W > 0x7fffffffLL) return NN_EINVAL;
  if ((Yf == nullptr) == (Yb == nullptr) || (mask && !Yb)) return NN_EINVAL;
  if (((uintptr_t)X | (uintptr_t)Wt) & 15) return NN_EINVAL;  // TMA sources
  ConvArgs g{};
  g.bias = bias;
  g.mask = mask;
  g.Yf = Yf;
  g.Yb = Yb;
  g.status = status;
  g.spins = spins;
  g.H = H;
  g.W = W;
  g.Cin = Cin;
  g.Cout = Cout;
  g.relu = relu;
  const int tilesX = (W + kTW - 1) / kTW, tilesY = (H + kTH - 1) / kTH;
  g.ftx = make_div(tilesX);
  g.fty = make_div(tilesY);
  g.ntiles = batch * tilesX * tilesY;
  g.NB = (Cout + 127) / 128;
  g.BN = ((Cout + g.NB - 1) / g.NB + 15) / 16 * 16;
  g.NB = (Cout + g.BN - 1) / g.BN;
  // the widest rows the channel count allows: TMA and the MMAs move 128-byte
  // rows at 50-60 bytes per clock and SM, 16-byte ones at 15
  g.rb = Cin % 64 == 0 ? 128 : Cin % 32 == 0 ? 64 : Cin % 16 == 0 ? 32 : 16;
  g.chb = g.rb / 2;
  g.kch = std::max(16, g.chb);
  const int c16 = (Cin + 15) / 16 * 16;
  g.cpp = std::min(c16, kMaxPass);
  g.npass = (c16 + g.cpp - 1) / g.cpp;
  g.pblk = up1k(kPatch * g.rb);
  g.nblk = Cin == 8 ? 1 : (g.cpp + g.chb - 1) / g.chb;
  g.slot_bytes = g.nblk * g.pblk;
  g.wblk = up1k(g.BN * g.rb);
  g.wblks = g.kch / g.chb;
  g.stage_bytes = g.wblks * g.wblk;
  g.kblk16 = g.wblks * g.pblk >> 4;
  const int extra = (int)sizeof(float) * g.BN + (Cin == 8 ? (kPatch + g.BN) * 16 : 0);
  const int budget = kSmemMax - extra;
  const int wres = Cin == 8 ? 9 * g.wblk : 9 * ((g.cpp + g.kch - 1) / g.kch) * g.stage_bytes;
  if (g.npass == 1 && (Cin == 8 || wres + 3 * g.slot_bytes <= budget)) {
    g.resident = 1;
    g.T = 1;
    g.NW = 1;
    g.NS = std::min(kMaxSlots, (budget - wres) / g.slot_bytes);
    // MMAs of 32 columns end faster than one warp issues them; wider ones lose by
    // being mixed (4 x 768^2, 32 -> 32: 148 us with one warp, 132 with two; 32 -> 96:
    // 182, 246; 8 -> 32: 83, 87)
    g.issuers = g.BN <= 32 && Cin > 8 ? 2 : 1;
  } else {
    g.issuers = 1;
    // two tiles to a weight stage, once there are two for every SM
    g.T = g.npass == 1 && 2 * g.slot_bytes + 2 * g.stage_bytes <= budget && (long long)g.ntiles * g.NB >= 2 * kSms ? 2 : 1;
    g.NS = std::min(2 * g.T, (budget - 2 * g.stage_bytes) / g.slot_bytes);
    g.NW = std::min(kMaxW, (budget - g.NS * g.slot_bytes) / g.stage_bytes);
  }
  g.w_off = g.NS * g.slot_bytes;
  g.zero_off = g.w_off + (g.resident ? wres : g.NW * g.stage_bytes);
  g.bias_off = g.zero_off + (Cin == 8 ? (kPatch + g.BN) * 16 : 0);
  g.cols = 32;
  while (g.cols < 2 * g.T * g.BN) g.cols *= 2;
  g.ngroups = (g.ntiles + g.T - 1) / g.T;
  g.vec = Yb ? Cout % 8 == 0 && (((uintptr_t)Yb | (uintptr_t)mask) & 15) == 0 : Cout % 4 == 0 && ((uintptr_t)Yf & 15) == 0;
  CUtensorMap mx, mw;
  {
    const unsigned long long d[4] = {(unsigned long long)Cin, (unsigned long long)W, (unsigned long long)H,
                                     (unsigned long long)batch};
    const unsigned long long st[3] = {2ull * Cin, 2ull * Cin * W, 2ull * Cin * W * H};
    const unsigned box[4] = {(unsigned)g.chb, kPW, kPH, 1};
    if (int rc = make_tensor_map(&mx, X, 4, d, st, box, g.rb)) return rc;
  }
  {
    const unsigned long long d[3] = {(unsigned long long)Cin, 9, (unsigned long long)Cout};
    const unsigned long long st[2] = {2ull * Cin, 18ull * Cin};
    const unsigned box[3] = {(unsigned)g.chb, 1, (unsigned)g.BN};
    if (int rc = make_tensor_map(&mw, Wt, 3, d, st, box, g.rb)) return rc;
  }
  const int smem = 1024 + g.bias_off + (int)sizeof(float) * g.BN;
  const int ks = g.kch / 16;
  auto fn = g.resident ? (ks == 4 ? conv_tc_kernel<4, true> : ks == 2 ? conv_tc_kernel<2, true> : conv_tc_kernel<1, true>)
                       : (ks == 4   ? conv_tc_kernel<4, false>
                          : ks == 2 ? conv_tc_kernel<2, false>
                                    : conv_tc_kernel<1, false>);
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return NN_ECUDA;
  const int per = std::min(std::max(1, kSms / g.NB), g.ngroups);
  fn<<<per * g.NB, kConvThreads, smem, s>>>(g, mx, mw);
  return cudaGetLastError() == cudaSuccess ? NN_OK : NN_ECUDA;
}

}  // namespace tomo_nn
