/*
 * Device helpers shared by the kernel files: three-input logic, the
 * microcanonical update rule, the warp bit transpose, mbarriers.
 */
#ifndef MICSA_DEVICE_CUH
#define MICSA_DEVICE_CUH

#include <stdint.h>

namespace {

constexpr unsigned FULL = 0xffffffffu;

/* all-ones if bond bit d of the site's coupling byte is set (one signed
 * bit-field extract) */
__device__ __forceinline__ uint32_t jmask(uint32_t jb, int d) {
  uint32_t r;
  asm("bfe.s32 %0, %1, %2, 1;" : "=r"(r) : "r"(jb), "r"(d));
  return r;
}

/* three-input bitwise function by truth table (a = 0xF0, b = 0xCC, c = 0xAA) */
template <int LUT>
__device__ __forceinline__ uint32_t lop3(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(a), "r"(b), "r"(c), "n"(LUT));
  return d;
}
__device__ __forceinline__ uint32_t xor3(uint32_t a, uint32_t b, uint32_t c) { return lop3<0x96>(a, b, c); }
__device__ __forceinline__ uint32_t maj3(uint32_t a, uint32_t b, uint32_t c) { return lop3<0xe8>(a, b, c); }

/* 32x32 bit transpose across a warp: lane c returns the word whose bit i is
 * bit c of lane i's input. */
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t x, int lane) {
  uint32_t m = 0x0000FFFFu;
#pragma unroll
  for (int j = 16; j != 0; j >>= 1, m ^= m << j) {
    const uint32_t p = __shfl_xor_sync(FULL, x, j);
    if (lane & j)
      x ^= ((p >> j) ^ x) & m;
    else
      x ^= (((x >> j) ^ p) & m) << j;
  }
  return x;
}

/* Microcanonical update with demon D = D0 + 2*D1 and unsatisfied-bond
 * counts (j1 + 2*j2) + (j3 + 2*j4): accept iff 0 <= D + u - 3 <= 3, then
 * D <- D + u - 3 -- the function the reference's ISI boolean algebra
 * computes (main.cu:1037-1074), equal to it on all 64 inputs, in a
 * shorter circuit: T = D + u (0 ... 9) summed carry-save into bits s0 + 2 s1
 * + 4 s2 (+ 8); accepted iff 3 <= T <= 6, i.e. s2 ^ (s1 & s0), which is 0
 * for T = 8 and 9 as well (s2 = s1 = 0), so the eights are not formed; then
 * D0 = !s0 and D1 = s0 ^ s1. */
__device__ __forceinline__ uint32_t isi_update(uint32_t j1, uint32_t j2, uint32_t j3,
                                               uint32_t j4, uint32_t &D0, uint32_t &D1) {
  const uint32_t s0 = xor3(D0, j1, j3), c0 = maj3(D0, j1, j3);
  const uint32_t t = xor3(D1, j2, j4), cc = maj3(D1, j2, j4);
  const uint32_t s1 = t ^ c0, s2 = lop3<0x78>(cc, t, c0);
  const uint32_t flip = lop3<0x78>(s2, s1, s0);
  const uint32_t d1 = s0 ^ s1;
  D0 = lop3<0x3a>(flip, s0, D0); /* flip ? !s0 : D0 */
  D1 = lop3<0xca>(flip, d1, D1); /* flip ? d1 : D1 */
  return flip;
}

/* ----------------------------------------------------- mbarriers */
/* transaction barriers in shared memory, bulk tensor loads (sm_90+ PTX) */
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
               ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
} /* namespace */

#endif
