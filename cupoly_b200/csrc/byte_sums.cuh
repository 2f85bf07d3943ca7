// Reduction of byte-matrix products (tdgt.cu, hps.cu): 8 column sums to a residue.
#pragma once
#include <cstdint>

namespace cpoly {

__device__ __forceinline__ uint64_t mad_wide(uint32_t a, uint32_t b, uint64_t c) {
  uint64_t r;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t pack64(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}

__device__ __forceinline__ double u32_to_double(uint32_t x) {  // exact, FP64 pipe only
  return __hiloint2double(0x43300000, (int)x) - 4503599627370496.0;
}

// Per-prime constants of the epilogues.  The powers of two sit in registers: as immediates
// the compiler turns the multiply-adds into separate shifts and adds.
struct Red {
  uint64_t p;
  uint32_t c;    // 2^63 - p
  uint32_t k8, k16;  // 2^8, 2^16
};

// value of 8 column sums: sum_j s[j] 2^(8 j) < 2^80 mod p, left below 2^63 + 2^48.
// Every s[j] <= 256 * 255 * 255, so s[j] + 2^8 s[j + 1] <= 4278124800 leaves room for the 17
// bits added to its word below: no carry ever leaves a 32-bit word.
__device__ __forceinline__ uint64_t col_sum(uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3, uint32_t s4,
                                            uint32_t s5, uint32_t s6, uint32_t s7, const Red& r) {
  const uint32_t a0 = s1 * r.k8 + s0, a1 = s3 * r.k8 + s2;
  const uint32_t a2 = s5 * r.k8 + s4, a3 = s7 * r.k8 + s6;
  const uint64_t t = mad_wide(a1, r.k16, pack64(a0, a2));  // bits 0 .. 63
  const uint32_t t0 = (uint32_t)t, t1 = (uint32_t)(t >> 32);
  const uint64_t h = mad_wide(a3, r.k16, t1);              // bits 32 .. 80
  const uint32_t top = (uint32_t)(h >> 31);                // value >> 63
  return mad_wide(top, r.c, pack64(t0, (uint32_t)h & 0x7FFFFFFFu));
}
__device__ __forceinline__ uint64_t col_sum(const uint32_t* s, const Red& r) {
  return col_sum(s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7], r);
}

}  // namespace cpoly
