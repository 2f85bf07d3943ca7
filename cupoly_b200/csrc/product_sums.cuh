// Sums of 64 x 64-bit products modulo the primes p = 2^63 - c (pointwise products, dot products).
#pragma once
#include "byte_sums.cuh"
#include "modarith.cuh"

namespace cpoly {

// The products of equal halves (bits 0 and 64) and the cross products (bit 32) keep sums of their
// own, so that a product is four wide multiply-adds on aligned register pairs and three carries;
// the two sums meet once, in fold().  LONG: sums of more than 2^128 (at most 2^134).
template <bool LONG>
struct ProductSum {
  uint32_t e0 = 0, e1 = 0, e2 = 0, e3 = 0, e4 = 0, o0 = 0, o1 = 0, o2 = 0;

  __device__ __forceinline__ void mac(uint64_t a, uint64_t b) {
    asm("{\n\t.reg .u32 a0, a1, b0, b1;\n\tmov.b64 {a0, a1}, %8;\n\tmov.b64 {b0, b1}, %9;\n\t"
        "mad.lo.cc.u32 %0, a0, b0, %0;\n\tmadc.hi.cc.u32 %1, a0, b0, %1;\n\t"
        "madc.lo.cc.u32 %2, a1, b1, %2;\n\tmadc.hi.cc.u32 %3, a1, b1, %3;\n\taddc.u32 %4, %4, 0;\n\t"
        "mad.lo.cc.u32 %5, a0, b1, %5;\n\tmadc.hi.cc.u32 %6, a0, b1, %6;\n\taddc.u32 %7, %7, 0;\n\t"
        "mad.lo.cc.u32 %5, a1, b0, %5;\n\tmadc.hi.cc.u32 %6, a1, b0, %6;\n\taddc.u32 %7, %7, 0;\n\t}"
        : "+r"(e0), "+r"(e1), "+r"(e2), "+r"(e3), "+r"(e4), "+r"(o0), "+r"(o1), "+r"(o2)
        : "l"(a), "l"(b));
  }

  // the sum when it is below 2^128
  __device__ __forceinline__ void words(uint64_t& lo, uint64_t& hi) const {
    uint32_t r1, r2, r3;
    asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, %7;\n\taddc.u32 %2, %5, %8;"
        : "=&r"(r1), "=&r"(r2), "=&r"(r3)
        : "r"(e1), "r"(e2), "r"(e3), "r"(o0), "r"(o1), "r"(o2));
    lo = pack64(e0, r1);
    hi = pack64(r2, r3);
  }

  // the sum mod p, any representative below 2^64: folds by 2^64 = 2 c, the last one's carry again
  __device__ __forceinline__ uint64_t fold(uint32_t c) const {
    const uint32_t C = 2 * c;
    uint32_t r1, r2, r3, r4, t0, t1, t2, k;
    asm("add.cc.u32 %0, %4, %8;\n\taddc.cc.u32 %1, %5, %9;\n\taddc.cc.u32 %2, %6, %10;\n\taddc.u32 %3, %7, 0;"
        : "=&r"(r1), "=&r"(r2), "=&r"(r3), "=&r"(r4)
        : "r"(e1), "r"(e2), "r"(e3), "r"(e4), "r"(o0), "r"(o1), "r"(o2));
    asm("{\n\t.reg .u32 q0, q1, kk;\n\t"
        "mad.lo.cc.u32 %0, %5, %7, %3;\n\tmadc.hi.cc.u32 %1, %5, %7, %4;\n\taddc.u32 kk, 0, 0;\n\t"
        "mul.lo.u32 q0, %6, %7;\n\tmul.hi.u32 q1, %6, %7;\n\tadd.cc.u32 %1, %1, q0;\n\taddc.u32 %2, q1, kk;\n\t}"
        : "=&r"(t0), "=&r"(t1), "=&r"(t2)
        : "r"(e0), "r"(r1), "r"(r2), "r"(r3), "r"(C));
    if (LONG) {  // r4 < 2^6: one more word t3 above t2, then one above 2^64
      const uint64_t t23 = mad_wide(r4, C, t2), w = (uint64_t)(uint32_t)(t23 >> 32) * C;
      asm("{\n\t.reg .u32 u2;\n\t"
          "mad.lo.cc.u32 %0, %3, %4, %0;\n\tmadc.hi.cc.u32 %1, %3, %4, %1;\n\taddc.u32 u2, 0, 0;\n\t"
          "add.cc.u32 %1, %1, %5;\n\taddc.u32 u2, u2, %6;\n\t"
          "mad.lo.cc.u32 %0, u2, %4, %0;\n\tmadc.hi.cc.u32 %1, u2, %4, %1;\n\taddc.u32 %2, 0, 0;\n\t}"
          : "+&r"(t0), "+&r"(t1), "=&r"(k)
          : "r"((uint32_t)t23), "r"(C), "r"((uint32_t)w), "r"((uint32_t)(w >> 32)));
    } else {
      asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\tmadc.hi.cc.u32 %1, %3, %4, %1;\n\taddc.u32 %2, 0, 0;"
          : "+&r"(t0), "+&r"(t1), "=&r"(k)
          : "r"(t2), "r"(C));
    }
    return mad_wide(k, C, pack64(t0, t1));
  }
};

// any v < 2^64 to [0, p)
__device__ __forceinline__ uint64_t canon(uint64_t v, uint32_t c, uint64_t p) {
  return red2p((v & 0x7FFFFFFFFFFFFFFFull) + ((v >> 63) ? c : 0), p);
}

// x y mod p for canonical Gaussian x, y and p = 2^63 - c; canonical, as gi_mul.
__device__ __forceinline__ void gi_mul_pm(uint64_t& cr, uint64_t& ci, ulonglong2 x, ulonglong2 y, uint64_t p,
                                          uint32_t c) {
  ProductSum<false> re, im;
  re.mac(x.x, y.x);
  re.mac(x.y, p - y.y);
  im.mac(x.x, y.y);
  im.mac(x.y, y.x);
  cr = canon(re.fold(c), c, p);
  ci = canon(im.fold(c), c, p);
}

}  // namespace cpoly
