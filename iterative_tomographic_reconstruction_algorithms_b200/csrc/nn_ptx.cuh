// PTX wrappers shared by the tensor-core kernels (nn_gemm.cu, nn_conv.cu, nn_wgrad.cu):
// cp.async, TMA, mbarriers with bounded waits, tcgen05 descriptors, MMA, TMEM loads.
#pragma once

#include <cuda.h>
#include <stdint.h>

#include "nn_internal.cuh"

namespace tomo_nn {
namespace {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool valid) {
  const int n = valid ? 16 : 0;  // 0: zero-fill, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait for phase `parity` of the barrier: at most `spins` polls;
// false if it gave up (at once when spins is 0).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int spins) {
  for (int i = 0; i < spins; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}

// Shared-memory matrix descriptor, no swizzle (version 1): core matrices of 8
// rows of 16 bytes.  K-major: lbo is the stride between the two 8-element K
// groups, sbo between 8-row groups.  MN-major (a row is one k, holding 8
// consecutive m or n): lbo is the stride between 8-row K groups, sbo between
// groups of 8 m or n.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// The same for rows of rb = 128, 64 or 32 bytes stored with the TMA swizzle of
// that width, or of 16 bytes without one.  K-major: sbo is the stride between
// 8-row groups; a K step within the row adds its bytes to the address.
// MN-major: lbo is the stride between blocks of rb / 2 channels, sbo between
// 8-row K groups (rb = 16: the reverse, as above).  The swizzle is a function
// of the shared-memory address, so a descriptor may start at any row.
__device__ __forceinline__ uint64_t smem_desc_rb(uint32_t addr, uint32_t lbo, uint32_t sbo, int rb) {
  const uint64_t layout = rb == 128 ? 2 : rb == 64 ? 4 : rb == 32 ? 6 : 0;
  return smem_desc(addr, lbo, sbo) | (layout << 61);
}

// Instruction descriptor: D F32, A and B BF16, both K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t instr_desc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
// The same for M = m and A and B both MN-major (bits 15 and 16).
__host__ __device__ constexpr uint32_t instr_desc_mn(int n, int m) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
               : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
      "%13, %14, %15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
        "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// KS consecutive K steps of one accumulator for a whole converged warp, issued
// by one elected lane: descriptor a advances by sa, b by sb (bytes / 16) a
// step; `more` accumulates onto what is there from the first step.  Issuing is
// what bounds small MMAs, so the loop around it should be uniform (a warp index
// the compiler can see is one: warp_index) and free of divisions; issued from a
// branch on the lane, with a division per step, an MMA took 300 cycles, here 60.
template <int KS>
__device__ __forceinline__ void mma_warp(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t more, uint32_t sa = 2,
                                         uint32_t sb = 2) {
  if constexpr (KS == 4)
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 a1, a2, a3, b1, b2, b3, s, t;\n\t"
        "cvt.u64.u32 s, %5;\n\tcvt.u64.u32 t, %6;\n\t"
        "add.s64 a1, %1, s;\n\tadd.s64 a2, a1, s;\n\tadd.s64 a3, a2, s;\n\t"
        "add.s64 b1, %2, t;\n\tadd.s64 b2, b1, t;\n\tadd.s64 b3, b2, t;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, 1;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %3, 1;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, %3, 1;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(more), "r"(sa), "r"(sb)
        : "memory");
  else if constexpr (KS == 2)
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 a1, b1, s, t;\n\t"
        "cvt.u64.u32 s, %5;\n\tcvt.u64.u32 t, %6;\n\t"
        "add.s64 a1, %1, s;\n\tadd.s64 b1, %2, t;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, 1;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(more), "r"(sa), "r"(sb)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(more)
        : "memory");
}
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }
__device__ __forceinline__ void mma_commit_warp(uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar)
      : "memory");
}

__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load3(uint32_t dst, const CUtensorMap *m, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(dst),
      "l"(m), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_load4(uint32_t dst, const CUtensorMap *m, int x, int y, int z, int w, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(dst),
      "l"(m), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
      : "memory");
}

// A role's wait: like mbar_wait, and false too once another role gave up.
__device__ __forceinline__ bool role_wait(const uint64_t *bar, uint32_t parity, int spins, const volatile int *gave_up) {
  const uint32_t b = smem_u32(bar);
  for (int i = 0; i < spins; ++i) {
    if (mbar_try_wait(b, parity)) return true;
    if ((i & 255) == 255 && *gave_up) return false;
  }
  return false;
}

// The same for a converged warp: one answer for all its lanes.
__device__ __forceinline__ bool warp_wait(const uint64_t *bar, uint32_t parity, int spins, const volatile int *gave_up) {
  return __all_sync(0xffffffffu, role_wait(bar, parity, spins, gave_up));
}

// x / d for 0 <= x < 2^31 as umulhi(x, m) >> s (m = ceil(2^(31 + l) / d), 2^l >= d).
struct FastDiv {
  unsigned m;
  int s, d;
};
__device__ __forceinline__ int fast_div(int x, const FastDiv &f) {
  return f.d == 1 ? x : (int)(__umulhi((unsigned)x, f.m) >> f.s);
}
inline FastDiv make_div(int d) {
  int l = 0;
  while ((1ll << l) < d) ++l;
  return {(unsigned)(((1ull << (31 + l)) + d - 1) / d), l - 1, d};
}

// Place in a ring of n stages and the parity of its current round.  (A
// division of the running count by n costs the issuing warp more than an MMA.)
struct Ring {
  int s = 0;
  uint32_t ph = 0;
  __device__ __forceinline__ void next(int n) {
    if (++s == n) {
      s = 0;
      ph ^= 1u;
    }
  }
};

}  // namespace
}  // namespace tomo_nn
