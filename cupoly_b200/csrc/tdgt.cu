// DGT on the tensor cores (tcgen05, kind::i8) for sm_100a.
//
// Replaces the same cuPoly kernels as dgt_kernels.cuh (hdgt_tr / hidgt / hidgt_tr / dgt /
// idgt, cuPoly src/cuda/dgt.cu:681-1067) with the same results: the transform of one residue
// of N = 2^LOGN Gaussian elements, LOGN = 10 .. 13, as three radix passes of 16, NM = N / 256
// and 16 points.
//
// Why matrix products.  A radix pass applies one constant linear map over Z_p to many short
// vectors of residues.  Written over bytes it is an integer matrix product: a residue x has 8
// bytes x_i, and x c = sum_i x_i (c 2^(8 i) mod p), so the map is an 8-bit matrix whose entry
// (byte j of an output, byte i of an input) is byte j of c 2^(8 i) mod p.  Accumulators stay
// below 256 * 255 * 255 < 2^24, and an output is sum_j acc_j 2^(8 j) < 2^80, reduced mod p by
// one multiply (every prime is 2^63 - c, c < 2^31).  The CUDA-core kernels spend 13.25
// constant products per element at N = 4096 and are bound by the integer multiply pipe; here
// the tensor cores do all butterflies and 4 products per element are left, the twiddles
// between the passes.
//
// Why the split form.  p = 1 mod 4, so Z_p[i] is Z_p x Z_p: an element a + b i is the pair
// u = a + s b, v = a - s b with s^2 = -1.  In it the Gaussian twist costs nothing extra (it
// is part of the first twiddle), a twiddle is two products, and the first and last pass's
// matrices (32 x 32 residues) convert between the forms.
//
// Measured on B200, forward / inverse of 201 MB of residues (3072 at N = 4096, 62 us of traffic):
// N = 1024 160 / 163 us, 2048 160 / 152, 4096 172 / 181, 8192 221 / 214 us; the CUDA-core kernels
// 260 / 263, 267 / 274, 318 / 314, 332 / 345 us.  What bounds it: a unit's passes depend on each
// other, so its products (57 us at N = 4096) and its arithmetic (82 us of issue slots) overlap only
// across the two tiles of a pass.  Two units in flight on pairs of CTAs (cta_group::2, half of the
// matrices in each) were slower, 219 / 265 us: the hand-over between the CTAs on every pass costs
// more than the overlap gives.
//
// One persistent CTA per SM walks units of 4096 elements (8192 for N = 8192; 4096 / N
// residues of one prime for the smaller sizes) ordered by prime, so the matrices stay in
// shared memory.  The unit's 64 KB (128 KB) of shared memory hold the operand of each pass
// in the layout the tensor core reads; passes work in place, tile by tile (see the address
// functions).  16 warps read accumulators from tensor memory (two buffers of 256 columns),
// reduce, multiply by the twiddle and write the next pass's operand; one thread issues the
// products and the bulk copies.
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "byte_sums.cuh"
#include "dgt_kernels.cuh"
#include "launch.cuh"
#include "tdgt.cuh"
#include "umma.cuh"

namespace cpoly {

namespace {

using namespace umma;

constexpr int kEpiWarps = 16;
constexpr int kThreads = (kEpiWarps + 1) * 32;

struct TArgs {
  const uint8_t* tab;  // table block of residue 0
  TdgtLayout L;
  const ModConst* mc;
  ulonglong2* data;            // output
  const ulonglong2* fsrc;      // forward input
  InvSrc isrc;                 // inverse input
  const int* rid_list;         // work list (rows of one element block each) or nullptr
  int nlist, nprimes;
  int nres, rid_off, npolys, S;
  long long poly_stride;       // elements
  int b2;                      // which of the inverse's middle matrices (prescale)
  unsigned units_per_prime, nunits;  // not for work lists
  int* err;
};

// Shared memory: the data, then the pass matrices, then the list order.
template <int M>
struct Cfg {
  static constexpr int NM = 1 << M, LOGN = M + 8, N = 1 << LOGN, N2 = N / 16;
  static constexpr int UNIT = M == 5 ? 8192 : 4096;   // elements per unit
  static constexpr int G = UNIT / N;                  // residues per unit
  static constexpr int TILES = UNIT / 2048;           // tiles of 128 rows x 16 elements
  static constexpr int DATA = UNIT * 16;
  static constexpr int B1 = 65536, B2 = 64 * NM * NM, B3 = 65536;
  // N = 8192: the three matrices take turns in one buffer; else all stay resident.
  static constexpr int MATS = M == 5 ? 65536 : B1 + B2 + B3;
  static constexpr int SMEM = DATA + MATS + 1024;
};

// a w mod p for any a < 2^64 and w = {w, w 2^32 mod p}, left below 2^64: the 32-bit halves of a
// times the two constants stay below 2^96, so one fold by 2^64 = 2 c is left (and the carry of
// that fold).  Five wide multiply-adds and the carry's; Shoup's product without its correction
// takes seven and two 32-bit ones (31.1 against 26.3 cycles a warp and sub-partition).
__device__ __forceinline__ uint64_t mul_lazy(uint64_t a, ulonglong2 w, const Red& r) {
  const uint32_t C = 2 * r.c;
  uint32_t l0, l1, k;
  asm("{\n\t.reg .u32 h0, h1, kk;\n\t"
      "mul.lo.u32 %0, %3, %5;\n\tmul.hi.u32 %1, %3, %5;\n\t"
      "mad.lo.cc.u32 %0, %4, %7, %0;\n\tmadc.hi.cc.u32 %1, %4, %7, %1;\n\taddc.u32 kk, 0, 0;\n\t"
      "mul.lo.u32 h0, %3, %6;\n\tmul.hi.u32 h1, %3, %6;\n\t"
      "mad.lo.cc.u32 h0, %4, %8, h0;\n\tmadc.hi.u32 h1, %4, %8, h1;\n\t"
      "add.cc.u32 %1, %1, h0;\n\taddc.u32 h1, h1, kk;\n\t"
      "mad.lo.cc.u32 %0, h1, %9, %0;\n\tmadc.hi.cc.u32 %1, h1, %9, %1;\n\taddc.u32 %2, 0, 0;\n\t}"
      : "=&r"(l0), "=&r"(l1), "=&r"(k)
      : "r"((uint32_t)a), "r"((uint32_t)(a >> 32)), "r"((uint32_t)w.x), "r"((uint32_t)(w.x >> 32)), "r"((uint32_t)w.y),
        "r"((uint32_t)(w.y >> 32)), "r"(C));
  return mad_wide(k, C, pack64(l0, l1));
}

// A twiddle pair (32 bytes, aligned) in one load: half the load instructions between the
// reductions (with the pairs loaded three steps ahead, inverse at N = 4096: 195 us before, 181 so).
__device__ __forceinline__ void ldg32(ulonglong2 (&w)[2], const ulonglong2* p) {
  asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(w[0].x), "=l"(w[0].y), "=l"(w[1].x), "=l"(w[1].y) : "l"(p));
}

__device__ __forceinline__ void sts8(uint32_t a, uint64_t v) {
  asm volatile("st.shared.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ void sts16(uint32_t a, uint64_t x, uint64_t y) {
  asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(a), "l"(x), "l"(y) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// One residue (element block) of the launch.
struct Item {
  size_t off;   // element offset of the output (and of the input of mode 0)
  size_t pair;  // gather mode: offset inside the operand
  int j;        // gather mode: operand
  int q, blk;   // polynomial (list: row) and element block in it
};

template <int M, bool INV>
__device__ __forceinline__ Item item_of(const TArgs& A, unsigned r, unsigned it) {
  constexpr int LOGN = Cfg<M>::LOGN;
  Item I;
  const unsigned h = it & ((1u << A.S) - 1);
  const unsigned q = it >> A.S;
  const size_t inner = ((size_t)r << (LOGN + A.S)) + ((size_t)h << LOGN);
  I.j = 0;
  I.pair = 0;
  if (INV && A.isrc.mode == 2) {
    I.j = (int)(q / A.isrc.npairs);
    I.pair = (q % A.isrc.npairs) * A.poly_stride + inner;
  }
  I.off = q * A.poly_stride + inner;
  I.q = (int)q;
  I.blk = (int)((r << A.S) + h);
  return I;
}

// The reductions between the products, by 8 warps over a tile of 128 rows: thread (row, wh) takes
// 8 elements (u, v), half wh of the row's outputs.  `wait` waits for the tile's product, `read`
// tells that its columns are in registers.
template <int M, bool INV>
struct Epilogue {
  using C = Cfg<M>;
  static constexpr int N2 = C::N2, NM = C::NM;
  static constexpr int kAhead = 3;  // steps between a twiddle's load and its use
  uint32_t sdat;  // the unit's shared memory
  uint32_t tl;    // the buffer's tensor memory, this warp's lanes
  int warp, lane, row, wh;
  Red R_;

  // 8 steps of 16 columns: two sums a step by `sums`, then `body` on them one step later, so
  // that the two dependent chains of a step overlap the next step's; and the columns after
  // those are on their way meanwhile.
  template <class Read, class Ld, class Sums, class Body>
  __device__ __forceinline__ void steps(Read read, Ld ld, Sums sums, Body body) const {
    uint32_t c[2][16];
    uint64_t x[2], y[2];
    ld(0, c[0]);
#pragma unroll
    for (int s = 0; s < 9; ++s) {
      if (s < 8) {
        tmem_ld_wait(c[s & 1]);
        if (s == 7) read();  // the buffer's columns are in registers
        if (s < 7) ld(s + 1, c[(s + 1) & 1]);
        sums(c[s & 1], x[s & 1], y[s & 1], R_);
      }
      if (s > 0) body(s - 1, x[(s - 1) & 1], y[(s - 1) & 1]);
    }
  }
  static __device__ __forceinline__ void sum2(const uint32_t* c, uint64_t& x, uint64_t& y, const Red& r) {
    x = col_sum(c, r);
    y = col_sum(c + 8, r);
  }

  // First pass of tile t: columns -> twiddled -> the middle pass's operand.
  template <class Wait, class Read>
  __device__ __forceinline__ void first(int t, const ulonglong2* T1, const ulonglong2* T2, Wait wait, Read read) const {
    auto ld_seq = [&](int s, uint32_t(&c)[16]) { tmem_ld16(c, tl + 128 * wh + 16 * s); };
    if (!INV) {
      const int nmi = M == 2 ? (row >> 4) & 3 : row >> 4, nl = row & 15;
      const int n2 = M >= 4 ? 128 * t + row : (M == 3 ? row : row & 63);
      const ulonglong2* Tw = T1 + 2 * (8 * wh * N2 + n2);
      ulonglong2 w[kAhead + 1][2];
      auto ldw = [&](int s) {
        ldg32(w[s & kAhead], Tw + 2 * s * N2);
      };
#pragma unroll
      for (int s = 0; s < kAhead; ++s) ldw(s);
      wait();
      const int R0 = (M == 2 ? (row >> 6) * 512 : 0) + wh * 256 + nl;  // q1 = 8 wh, u
      constexpr int RB = M == 2 ? 32 : 64;
      const uint32_t base = sdat + t * 32768 + R0 * RB + (nmi & 1) * 8 +
                            (((nmi >> 1) ^ (M == 2 ? (R0 >> 2) & 1 : (R0 >> 1) & 3)) << 4);
      steps(read, ld_seq, sum2, [&](int s, uint64_t x, uint64_t y) {
        if (s + kAhead < 8) ldw(s + kAhead);
        sts8(base + s * 16 * RB, mul_lazy(x, w[s & kAhead][0], R_));
        sts8(base + (128 + s * 16) * RB, mul_lazy(y, w[s & kAhead][1], R_));
      });
    } else {
      const int qm = row & (NM - 1), q1l = M == 2 ? (row >> 2) & 15 : row >> M;
      // digit nl = 8 wh + j: every layout xors bits of nl below the first that depends on wh
      uint32_t base;
      int ch;  // swizzled chunk before the xor with bits of nl
      if (M == 4) {
        base = t * 32768 + (q1l * 16 + 8 * wh) * 128 + (qm & 1) * 8;
        ch = qm >> 1;
      } else if (M == 5) {
        base = t * 32768 + (qm >> 4) * 16384 + (q1l * 16 + 8 * wh) * 128 + (qm & 1) * 8;
        ch = (qm & 15) >> 1;
      } else if (M == 3) {
        base = t * 32768 + ((q1l >> 3) * 256 + (q1l & 7) * 16 + 8 * wh) * 64 + (qm & 1) * 8;
        ch = qm >> 1;
      } else {
        base = t * 32768 + ((row >> 6) * 512 + (q1l >> 3) * 256 + (q1l & 7) * 16 + 8 * wh) * 32 + (qm & 1) * 8;
        ch = qm >> 1;
      }
      base += sdat;
      constexpr int RB = M >= 4 ? 128 : (M == 3 ? 64 : 32);
      constexpr int UV = M == 4 ? 16384 : (M == 5 ? 64 * 128 : 128 * RB);
      const ulonglong2* Tw = T2 + 8 * wh * NM + qm;
      wait();
      steps(read, ld_seq, sum2, [&](int j, uint64_t x, uint64_t y) {
        const ulonglong2 w = __ldg(Tw + j * NM);
        const int sw = M >= 4 ? j : (M == 3 ? (j >> 1) & 3 : (j >> 2) & 1);
        const uint32_t a = base + j * RB + ((ch ^ sw) << 4);
        sts8(a, mul_lazy(x, w, R_));
        sts8(a + UV, mul_lazy(y, w, R_));
      });
    }
  }

  // Middle pass of tile t: N = 4096 forward: t = half h; N = 8192 forward: t = 2 h + s.
  template <class Wait, class Read>
  __device__ __forceinline__ void middle(int t, const ulonglong2* T1, const ulonglong2* T2, Wait wait, Read read) const {
    auto ld_seq = [&](int s, uint32_t(&c)[16]) { tmem_ld16(c, tl + 128 * wh + 16 * s); };
    // u and v of output s of this half
    auto ld_uv = [&](int s, uint32_t(&c)[16]) {
      if (M >= 4)
        tmem_ld8x2(c, tl + 64 * wh + 8 * s, tl + 128 + 64 * wh + 8 * s);
      else if (M == 3)
        tmem_ld8x2(c, tl + 128 * wh + 8 * s, tl + 128 * wh + 64 + 8 * s);
      else
        tmem_ld8x2(c, tl + (2 * wh + (s >> 2)) * 64 + 8 * (s & 3), tl + (2 * wh + (s >> 2)) * 64 + 32 + 8 * (s & 3));
    };
    const int q1l = row >> 4, nl = row & 15;
    if (!INV) {
      const int o0 = M == 5 ? 16 * (t & 1) + 8 * wh : (M == 4 ? 8 * wh : 0);  // first digit qm
      const ulonglong2* Tw = T2 + o0 * 16 + nl;
      wait();
      steps(read, ld_uv, sum2, [&](int s, uint64_t x, uint64_t y) {
        const int oj = M == 2 ? s & 3 : s;
        const ulonglong2 w = __ldg(Tw + oj * 16);
        const int qm = o0 + oj, pn = nl >> 3;
        int r3;
        uint32_t a;
        if (M == 5) {
          r3 = q1l * 32 + qm;
          a = (pn * 2 + (r3 >> 7)) * 32768 + (t >> 1) * 16384 + (r3 & 127) * 128;
        } else if (M == 4) {
          r3 = q1l * 16 + qm;
          a = pn * 32768 + t * 16384 + r3 * 128;
        } else if (M == 3) {
          r3 = (wh * 8 + q1l) * 8 + qm;
          a = t * 32768 + pn * 16384 + r3 * 128;
        } else {
          r3 = wh * 64 + ((s >> 2) * 8 + q1l) * 4 + qm;
          a = t * 32768 + pn * 16384 + r3 * 128;
        }
        sts16(sdat + a + (((nl & 7) ^ (r3 & 7)) << 4), mul_lazy(x, w, R_), mul_lazy(y, w, R_));
      });
    } else if (M != 5) {
      // M == 2: row tiles 2 wh (q1 = q1l) and 2 wh + 1 (q1 = 8 + q1l) of residue wh, 4 outputs each
      const int q1 = M == 4 ? 8 * t + q1l : (M == 3 ? wh * 8 + q1l : q1l);
      const int o0 = M == 4 ? 8 * wh : 0;  // first digit nm
      const ulonglong2* Tw = T1 + 2 * (q1 * N2 + 16 * o0 + nl);
      auto tw_off = [&](int s) { return M == 2 ? 2 * ((s >> 2) * 8 * N2 + 16 * (s & 3)) : 32 * s; };
      ulonglong2 w[kAhead + 1][2];
      auto ldw = [&](int s) {
        ldg32(w[s & kAhead], Tw + tw_off(s));
      };
#pragma unroll
      for (int s = 0; s < kAhead; ++s) ldw(s);
      wait();
      const int n2 = 16 * o0 + nl;
      const uint32_t a = sdat + t * 32768 +
                         (M == 4 ? n2 * 128 : (M == 3 ? wh * 16384 + n2 * 128 : (wh * 64 + n2) * 128)) +
                         ((q1l ^ (nl & 7)) << 4);
      steps(read, ld_uv, sum2, [&](int s, uint64_t x, uint64_t y) {
        if (s + kAhead < 8) ldw(s + kAhead);
        sts16(a + (M == 2 ? (s & 3) * 2048 + (s >> 2) * 16384 : s * 2048), mul_lazy(x, w[s & kAhead][0], R_),
              mul_lazy(y, w[s & kAhead][1], R_));
      });
    } else {  // N = 8192: rows of u (lanes 0 .. 63) or of v; 16 outputs each
      const int uv = row >> 6, q1 = 4 * t + ((row >> 4) & 3), o0 = 16 * wh;
      const ulonglong2* Tw = T1 + 2 * (q1 * N2 + 16 * o0 + nl) + uv;
      ulonglong2 w[kAhead + 1][2];
      auto ldw = [&](int s) {
#pragma unroll
        for (int i = 0; i < 2; ++i) w[s & kAhead][i] = __ldg(Tw + 32 * (2 * s + i));
      };
#pragma unroll
      for (int s = 0; s < kAhead; ++s) ldw(s);
      wait();
      const uint32_t a = sdat + (t >> 1) * 65536 + (16 * o0 + nl) * 128 + (((q1 & 7) ^ (nl & 7)) << 4) + uv * 8;
      steps(read, ld_seq, sum2, [&](int s, uint64_t x, uint64_t y) {
        if (s + kAhead < 8) ldw(s + kAhead);
        sts8(a + 2 * s * 2048, mul_lazy(x, w[s & kAhead][0], R_));
        sts8(a + (2 * s + 1) * 2048, mul_lazy(y, w[s & kAhead][1], R_));
      });
    }
  }

  // Last pass of tile t: canonical results to global memory; out(g) is item g of the unit or nullptr.
  template <class Out, class Read>
  __device__ __forceinline__ void last(int t, Out out, Read read) const {
    auto ld_seq = [&](int s, uint32_t(&c)[16]) { tmem_ld16(c, tl + 128 * wh + 16 * s); };
    if (INV) {
      const int g = M >= 4 ? 0 : (M == 3 ? t : 2 * t + (row >> 6));
      const int n2 = M >= 4 ? 128 * t + row : (M == 3 ? row : row & 63);
      ulonglong2* x0 = out(g);
      const bool live = x0 != nullptr;
      ulonglong2* x = x0 + 8 * wh * N2 + n2;
      steps(read, ld_seq, sum2, [&](int s, uint64_t a, uint64_t b) {
        if (live) x[s * N2] = make_ulonglong2(red2p(a, R_.p), red2p(b, R_.p));
      });
    } else {
      // A row's results are contiguous: four neighbouring lanes take four elements of a row
      // (64 bytes a store), so that a store instruction touches 8 lines and not 32.
      const int rw = (warp & 3) * 32;  // rows of this warp; M == 2: all of one residue
      const int g = M >= 4 ? 0 : (M == 3 ? t : 2 * t + (rw >> 6));
      const int r0 = M >= 4 ? 128 * t + rw : (M == 3 ? rw : rw & 63);
      ulonglong2* x0 = out(g);
      const bool live = x0 != nullptr;
      ulonglong2* x = x0 + (r0 + (lane >> 2)) * 16 + 8 * wh + (lane & 3);
      uint64_t z0 = 0, z1 = 0;
      // step: 16-lane half s >> 2, group of 4 elements (s >> 1) & 1, component s & 1
      steps(read, [&](int s, uint32_t(&c)[16]) {
        tmem_ld_quad(c, tl + ((uint32_t)((s >> 2) * 16) << 16) + 128 * wh + 32 * (s & 3));
      }, [](const uint32_t* c, uint64_t& x, uint64_t& y, const Red& R_) {
        x = col_sum(c[0], c[1], c[4], c[5], c[8], c[9], c[12], c[13], R_);
        y = col_sum(c[2], c[3], c[6], c[7], c[10], c[11], c[14], c[15], R_);
      }, [&](int s, uint64_t a, uint64_t b) {
        a = red2p(a, R_.p);
        b = red2p(b, R_.p);
        if (s & 1) {
          ulonglong2* y = x + (s >> 2) * 256 + 4 * ((s >> 1) & 1);
          if (live) {
            y[0] = make_ulonglong2(z0, a);
            y[128] = make_ulonglong2(z1, b);
          }
        } else {
          z0 = a;
          z1 = b;
        }
      });
    }
  }
};

// Inverse: tiles t0, t0 + dt, ... of a unit's operand into shared memory by 256 threads (gtid),
// swizzled rows of 16 elements; item(g) is item g < count of the unit.
template <int M, class ItemOf>
__device__ __forceinline__ void load_inverse(const TArgs& A, uint32_t sdat, int gtid, int t0, int dt, int count,
                                             ItemOf item) {
#pragma unroll 1
  for (int t = t0; t < Cfg<M>::TILES; t += dt) {
#pragma unroll 1
    for (int g0 = 0; g0 < (M == 2 ? 2 : 1); ++g0) {
      const int g = M == 2 ? 2 * t + g0 : (M == 3 ? t : 0);
      if (g >= count) continue;
      const Item I = item(g);
      constexpr int E = M == 2 ? 1024 : 2048;  // elements of this item in this tile
      const int eo = M >= 4 ? t * 2048 : 0;    // their first element in the item
      const int er0 = (gtid >> 4) + (M == 2 ? g0 * 64 : 0), ql = gtid & 15;
      // rows er0, er0 + 16, ...: the swizzle term does not change
      const uint32_t dst0 = sdat + t * 32768 + (ql >> 3) * 16384 + er0 * 128 + (((ql & 7) ^ (er0 & 7)) << 4);
      const ulonglong2* src =
          (A.isrc.mode == 0 ? A.isrc.p[0] + I.off : inv_src_ptr(A.isrc, I.j) + I.pair) + eo + gtid;
#pragma unroll
      for (int i = 0; i < E / 256; ++i) cp_async16(dst0 + i * 2048, src + i * 256);
    }
  }
}

// Orders the rows of a work list by prime (each CTA for itself: no scratch memory, no second
// launch): rows cnt[r] .. cnt[r + 1] of `order` have prime r, and units of at most GR rows start
// at ustart[r].  Returns the number of units.
template <int GR>
__device__ __forceinline__ unsigned order_rows(const TArgs& A, unsigned* s_cnt, unsigned* s_ustart, uint16_t* s_order,
                                               int warp, int lane, int tid, int threads) {
  for (int i = tid; i <= kMaxResidues; i += threads) s_cnt[i] = 0;
  __syncthreads();
  for (int i = tid; i < A.nlist; i += threads) {
    const unsigned r = (unsigned)A.rid_list[i];
    if (r < (unsigned)A.nprimes) atomicAdd(&s_cnt[r + 1], 1u);  // a row of no prime of the engine is left out
  }
  __syncthreads();
  if (tid == 0) {
    unsigned u = 0, c = 0;
    for (int r = 0; r < kMaxResidues; ++r) {
      const unsigned n = s_cnt[r + 1];
      s_ustart[r] = u;
      u += (n + GR - 1) / GR;
      s_cnt[r] = c;  // first row of prime r in the order
      c += n;
    }
    s_ustart[kMaxResidues] = u;
    s_cnt[kMaxResidues] = c;
  }
  __syncthreads();
  // stable order without atomics: a warp takes every (threads / 32)-th prime
  for (int r = warp; r < kMaxResidues; r += (threads >> 5)) {
    unsigned at = s_cnt[r];
    const unsigned end = s_cnt[r + 1];
    for (int b = 0; b < A.nlist && at < end; b += 32) {
      const bool mine = b + lane < A.nlist && A.rid_list[b + lane] == r;
      const unsigned m = __ballot_sync(0xFFFFFFFFu, mine);
      if (mine) s_order[at + __popc(m & ((1u << lane) - 1))] = (uint16_t)(b + lane);
      at += __popc(m);
    }
  }
  return s_ustart[kMaxResidues];
}

// `fmap` (forward): the input as a tensor of 64-bit words, {2 N2, 16 x blocks, polynomials}; for
// N = 1024 {2 N2, polynomials, 16 x blocks}.  A box is one tile's part of the input in the
// order in which the first pass reads it.
template <int M, bool INV>
__global__ void __launch_bounds__(kThreads, 1)
    k_tdgt(const __grid_constant__ TArgs A, const __grid_constant__ CUtensorMap fmap) {
  using C = Cfg<M>;
  constexpr int N2 = C::N2, NM = C::NM, G = C::G, TILES = C::TILES;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t s_bar[12];
  __shared__ uint32_t s_slot;
  __shared__ int s_fail;
  __shared__ unsigned s_cnt[kMaxResidues + 1], s_ustart[kMaxResidues + 1];
  __shared__ uint16_t s_order[kTdgtListMax];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sdat = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sB1 = sdat + C::DATA;
  const uint32_t sB2 = M == 5 ? sB1 : sB1 + C::B1;
  const uint32_t sB3 = M == 5 ? sB1 : sB2 + C::B2;
  const uint32_t bar0 = smem_u32(s_bar);
  const uint32_t bD = bar0, bE = bar0 + 16, bA = bar0 + 32, bB = bar0 + 64;  // D[2], E[2], A[4], B[3]
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(bD + 8 * i, 1);
      mbar_init(bE + 8 * i, kEpiWarps / 2);
    }
    for (int i = 0; i < 4; ++i) mbar_init(bA + 8 * i, INV ? kEpiWarps / 2 : 1);
    for (int i = 0; i < 3; ++i) mbar_init(bB + 8 * i, 1);
    mbar_init_fence();
    s_fail = 0;
  }
  if (warp == kEpiWarps) tmem_alloc(smem_u32(&s_slot), 512);
  const bool list = A.rid_list != nullptr;
  unsigned nunits = A.nunits;
  if (list) nunits = order_rows<G>(A, s_cnt, s_ustart, s_order, warp, lane, tid, kThreads);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = s_slot;
  const unsigned u0 = (unsigned)((unsigned long long)blockIdx.x * nunits / gridDim.x);
  const unsigned u1 = (unsigned)((unsigned long long)(blockIdx.x + 1) * nunits / gridDim.x);

  // the prime and the items [first, first + count) of a unit
  int cur_r = 0;  // list: the prime whose units contain the last unit asked for
  auto unit_of = [&](unsigned u, int& r, unsigned& first, int& count) {
    unsigned v, n;
    if (list) {
      while (u >= s_ustart[cur_r + 1]) ++cur_r;
      r = cur_r;
      v = u - s_ustart[r];
      n = s_cnt[r + 1] - s_cnt[r];
      first = s_cnt[r] + v * G;
    } else {
      r = (int)(u / A.units_per_prime);
      v = u - (unsigned)r * A.units_per_prime;
      n = (unsigned)A.npolys << A.S;
      first = v * G;
    }
    const unsigned left = n - v * G;
    count = left < (unsigned)G ? (int)left : G;
  };
  auto item_at = [&](int r, unsigned it) -> Item {
    if (list) return item_of<M, INV>(A, 0, (unsigned)s_order[it]);
    return item_of<M, INV>(A, (unsigned)r, it);
  };
  auto rid_of = [&](int r) { return list ? r : A.rid_off + r; };

  if (warp == kEpiWarps) {
    constexpr int N2C = M >= 4 ? 128 : NM * 8;  // columns of a middle product
    const uint32_t id256 = idesc_u8(128, 256);
    const uint32_t idm = idesc_u8(128, N2C);
    // descriptors of the buffers' first bytes; a step adds bytes / 16 to the low word
    const uint64_t dat_lin = smem_desc(sdat, 2048, 128, kSwzNone);
    const uint64_t dat128 = smem_desc(sdat, 16, 1024, kSwz128);
    const uint64_t dat64 = smem_desc(sdat, 16, 512, kSwz64);
    const uint64_t dat32 = smem_desc(sdat, 16, 256, kSwz32);
    const uint64_t db1 = smem_desc(sB1, 4096, 128, kSwzNone), db3 = smem_desc(sB3, 4096, 128, kSwzNone);
    const uint64_t db2 = smem_desc(sB2, M == 5 ? 4096 : NM * 128, 128, kSwzNone);
    uint32_t pe[2] = {0, 0}, pa = 0, pb = 0, pd[2] = {0, 0};
    // waits for the epilogue's next arrival on buffer d
    auto waitE = [&](int d) {
      mbar_wait(bE + 8 * d, pe[d] & 1, &s_fail);
      ++pe[d];
    };
    auto waitD = [&]() {  // every product issued so far is done
      for (int d = 0; d < 2; ++d) mbar_wait(bD + 8 * d, (pd[d] - 1) & 1, &s_fail);
    };
    auto commit = [&](int d) {
      if (lane == 0) mma_commit(bD + 8 * d);
      ++pd[d];
    };
    // a 16-element pass over 256 bytes of K: operand panels of 128-byte rows at byte offsets a0, a1
    auto pass16 = [&](int d, uint32_t a0, uint32_t a1, uint64_t b) {
      if (lane == 0) {
        const uint64_t da0 = dat128 + (a0 >> 4), da1 = dat128 + (a1 >> 4);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          mma_u8(tmem + 256 * d, (ks < 4 ? da0 : da1) + (ks & 3) * 2, b + ks * 512, id256, ks > 0);
      }
      commit(d);
    };
    auto load_matrix = [&](uint32_t dst, const uint8_t* src, uint32_t bytes, uint32_t bar) {
      if (lane == 0) {
        mbar_expect_tx(bar, bytes);
        bulk_load(dst, src, bytes, bar);
      }
    };
    int prev_rid = -1;
    for (unsigned u = u0; u < u1; ++u) {
      int r, count;
      unsigned first;
      unit_of(u, r, first, count);
      const int rid = rid_of(r);
      const uint8_t* tab = A.tab + (size_t)rid * A.L.stride;
      const uint8_t* gB1 = tab + (INV ? A.L.i_b1 : A.L.f_b1);
      const uint8_t* gB2 = tab + (INV ? A.L.i_b2[A.b2] : A.L.f_b2);
      const uint8_t* gB3 = tab + (INV ? A.L.i_b3 : A.L.f_b3);
      const bool newb = M == 5 || rid != prev_rid;
      prev_rid = rid;
      Item ld0{}, ld1{};
      if (!INV) {
        ld0 = item_at(r, first);
        ld1 = M == 3 && count > 1 ? item_at(r, first + 1) : ld0;
      }
      if (u > u0) waitD();  // the last pass of the previous unit has read the data and the matrices
      if (!INV) {
#pragma unroll
        for (int t = 0; t < TILES; ++t) {
          const uint32_t dst = sdat + t * 32768, bar = bA + 8 * t;
          if (M >= 3) {
            if (lane == 0) {
              if (M >= 4 || t < count) {
                mbar_expect_tx(bar, 32768);
                tensor_load3(dst, &fmap, M >= 4 ? t * 256 : 0, 16 * (t == 1 && M == 3 ? ld1 : ld0).blk,
                             (t == 1 && M == 3 ? ld1 : ld0).q, bar);
              } else {
                mbar_arrive(bar);
              }
            }
          } else if (!list) {  // two consecutive polynomials; beyond the last one the box is filled with zeros
            if (lane == 0) {
              if (2 * t < count) {
                mbar_expect_tx(bar, 32768);
                tensor_load3(dst, &fmap, 0, ld0.q + 2 * t, 16 * ld0.blk, bar);
              } else {
                mbar_arrive(bar);
              }
            }
          } else {  // rows of a list: 1 KB pieces, spread over the lanes
            const int have = count - 2 * t < 0 ? 0 : (count - 2 * t > 2 ? 2 : count - 2 * t);
            if (lane == 0) {
              if (have)
                mbar_expect_tx(bar, have * 16384);
              else
                mbar_arrive(bar);
            }
            __syncwarp();
            if ((lane >> 4) < have) {
              const int gl = lane >> 4, n1 = lane & 15;
              bulk_load(dst + n1 * 2048 + gl * 1024, A.fsrc + item_at(r, first + 2 * t + gl).off + n1 * N2, 1024, bar);
            }
          }
        }
      }
      if (newb) {
        load_matrix(sB1, gB1, C::B1, bB);
        if (M != 5) {
          load_matrix(sB2, gB2, C::B2, bB + 8);
          load_matrix(sB3, gB3, C::B3, bB + 16);
        }
      }
      // ---- pass 1 ----
      if (newb) mbar_wait(bB, pb & 1, &s_fail);
      for (int t = 0; t < TILES; ++t) {
        const int d = t & 1;
        mbar_wait(bA + 8 * t, pa & 1, &s_fail);
        if (u > u0 || t >= 2) waitE(d);
        fence_after_sync();
        if (INV) {
          pass16(d, t * 32768, t * 32768 + 16384, db1);
        } else {
          if (lane == 0) {
            const uint64_t da = dat_lin + t * 2048;
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) mma_u8(tmem + 256 * d, da + ks * 256, db1 + ks * 512, id256, ks > 0);
          }
          commit(d);
        }
      }
      ++pa;
      if (u + 1 < u1) {  // the next unit's operands into L2
        int rn, cn;
        unsigned fn;
        unit_of(u + 1, rn, fn, cn);
        if (lane < cn) {
          const Item I = item_at(rn, fn + lane);
          constexpr uint32_t bytes = C::N * 16;
          if (!INV) {
            prefetch_l2(A.fsrc + I.off, bytes);
          } else {
            prefetch_l2(A.isrc.mode == 0 ? A.isrc.p[0] + I.off : inv_src_ptr(A.isrc, I.j) + I.pair, bytes);
          }
        }
        if (list) cur_r = r;  // unit_of walks forward only
      }
      // ---- middle pass ----
      if (M == 5) {  // the middle matrix replaces the first one
        waitD();
        load_matrix(sB2, gB2, C::B2, bB + 8);
      }
      if (newb) mbar_wait(bB + 8, pb & 1, &s_fail);
      if (M == 4 && !INV) {
        waitE(0);
        waitE(1);
        fence_after_sync();
        for (int h = 0; h < 2; ++h) {
          if (lane == 0) {
#pragma unroll
            for (int uv = 0; uv < 2; ++uv)
#pragma unroll
              for (int ks = 0; ks < 4; ++ks)
                mma_u8(tmem + 256 * h + 128 * uv, dat64 + (ks >> 1) * 2048 + (h * 2 + uv) * 512 + (ks & 1) * 2,
                       db2 + ks * 256, idm, ks > 0);
          }
          commit(h);
        }
      } else if (M <= 4) {
        for (int t = 0; t < 2; ++t) {
          waitE(t);
          fence_after_sync();
          if (lane == 0) {
            if (M == 4) {
#pragma unroll
              for (int uv = 0; uv < 2; ++uv)
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                  mma_u8(tmem + 256 * t + 128 * uv, dat128 + t * 2048 + uv * 1024 + ks * 2, db2 + ks * 256, idm, ks > 0);
            } else if (M == 3) {
#pragma unroll
              for (int tile = 0; tile < 4; ++tile)
#pragma unroll
                for (int ks = 0; ks < 2; ++ks)
                  mma_u8(tmem + 256 * t + 64 * tile, dat64 + t * 2048 + tile * 512 + ks * 2, db2 + ks * 128, idm, ks > 0);
            } else {
#pragma unroll
              for (int tile = 0; tile < 8; ++tile)
                mma_u8(tmem + 256 * t + 32 * tile, dat32 + t * 2048 + tile * 256, db2, idm, 0);
            }
          }
          commit(t);
        }
      } else if (!INV) {  // M == 5
        waitE(0);
        waitE(1);
        for (int h = 0; h < 2; ++h)
          for (int s = 0; s < 2; ++s) {
            if (h > 0) waitE(s);
            fence_after_sync();
            if (lane == 0) {
#pragma unroll
              for (int uv = 0; uv < 2; ++uv)
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)
                  mma_u8(tmem + 256 * s + 128 * uv, dat64 + (ks >> 1) * 2048 + (h * 2 + uv) * 512 + (ks & 1) * 2,
                         db2 + ks * 512 + s * 128, idm, ks > 0);
            }
            commit(s);
          }
      } else {  // M == 5 inverse
        waitE(0);
        waitE(1);
        for (int t = 0; t < 4; ++t) {
          if (t >= 2) waitE(t & 1);
          fence_after_sync();
          pass16(t & 1, t * 32768, t * 32768 + 16384, db2);
        }
      }
      // ---- last pass ----
      if (M == 5) {
        waitD();
        load_matrix(sB3, gB3, C::B3, bB + 16);
      }
      if (newb) {
        mbar_wait(bB + 16, pb & 1, &s_fail);
        ++pb;
      }
      if (M == 4 && INV) {  // every row reads both halves of the middle pass's results
        waitE(0);
        waitE(1);
        fence_after_sync();
        for (int t = 0; t < 2; ++t) pass16(t, t * 16384, 32768 + t * 16384, db3);
      } else if (M <= 4) {
        for (int t = 0; t < 2; ++t) {
          waitE(t);
          fence_after_sync();
          if (M == 4)
            pass16(t, t * 16384, 32768 + t * 16384, db3);
          else
            pass16(t, t * 32768, t * 32768 + 16384, db3);
        }
      } else {  // M == 5
        waitE(0);
        waitE(1);
        for (int t = 0; t < 4; ++t) {
          if (t >= 2) waitE(t & 1);
          fence_after_sync();
          if (!INV) {
            const int h = t >> 1, rb = t & 1;
            pass16(t & 1, rb * 32768 + h * 16384, (2 + rb) * 32768 + h * 16384, db3);
          } else {
            pass16(t & 1, t * 16384, 65536 + t * 16384, db3);
          }
        }
      }
    }
    __syncwarp();
  } else {
    // Two groups of 8 warps: group d reduces the products of buffer d, so one group's waits
    // and fences overlap the other's arithmetic.
    const int d = warp >> 3, gtid = tid & 255;
    uint32_t k8 = 256;  // see Red
    asm volatile("" : "+r"(k8));
    Epilogue<M, INV> ep;
    ep.sdat = sdat;
    ep.warp = warp;
    ep.lane = lane;
    ep.row = (warp & 3) * 32 + lane;
    ep.wh = (warp >> 2) & 1;
    ep.tl = tmem + 256 * d + ((uint32_t)((warp & 3) * 32) << 16);
    uint32_t pd = 0;
    auto waitD = [&]() {
      mbar_wait(bD + 8 * d, pd & 1, &s_fail);
      ++pd;
      fence_after_sync();
    };
    // The product of the same step into buffer 1 is done as well.  Only group 0 has to wait, and
    // after its own product: products complete in issue order, so buffer 1 is then past its
    // previous phase, and its next product waits for group 0, so it is at most one phase ahead.
    auto waitD_both = [&]() {
      waitD();
      if (d == 0) mbar_wait(bD + 8, (pd - 1) & 1, &s_fail);
    };
    // this warp has read its buffer (and written its part of the next operand)
    auto doneE = [&]() {
      fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bE + 8 * d);
    };
    auto doneE_smem = [&]() {
      fence_async_smem();
      doneE();
    };
    auto none = []() {};
    auto load_unit = [&](unsigned u) {
      int r, count;
      unsigned first;
      unit_of(u, r, first, count);
      load_inverse<M>(A, sdat, gtid, d, 2, count, [&](int g) { return item_at(r, first + g); });
    };
    auto load_done = [&]() {
      cp_async_wait();
      fence_async_smem();
      __syncwarp();
      if (lane == 0)
        for (int t = d; t < TILES; t += 2) mbar_arrive(bA + 8 * t);
    };
    if (INV && u0 < u1) {
      load_unit(u0);
      load_done();
    }
    for (unsigned u = u0; u < u1; ++u) {
      int r, count;
      unsigned first;
      unit_of(u, r, first, count);
      const int rid = rid_of(r);
      const uint64_t p = A.mc[rid].p;
      ep.R_ = Red{p, (uint32_t)((1ull << 63) - p), k8, k8 << 8};
      const uint8_t* tab = A.tab + (size_t)rid * A.L.stride;
      const ulonglong2* T1 = reinterpret_cast<const ulonglong2*>(tab + (INV ? A.L.i_t1 : A.L.f_t1));
      const ulonglong2* T2 = reinterpret_cast<const ulonglong2*>(tab + (INV ? A.L.i_t2 : A.L.f_t2));
#pragma unroll 1
      for (int t = d; t < TILES; t += 2) {
        ep.first(t, T1, T2, waitD, none);
        doneE_smem();
      }
#pragma unroll 1
      for (int t = d; t < TILES; t += 2) {  // N = 8192: both products of a half have read what the results replace
        if (M == 5)
          ep.middle(t, T1, T2, waitD_both, none);
        else
          ep.middle(t, T1, T2, waitD, none);
        doneE_smem();
      }
#pragma unroll 1
      for (int t = d; t < TILES; t += 2) {
        const bool last = t + 2 >= TILES;
        if (INV && M >= 4 && last)
          waitD_both();  // for the loads below
        else
          waitD();
        if (INV && last && u + 1 < u1) {
          // every product that reads this group's tiles is done: the next operand can come in
          load_unit(u + 1);
        }
        ep.last(t, [&](int g) { return g < count ? A.data + item_at(r, first + g).off : nullptr; }, doneE);
      }
      if (INV && u + 1 < u1) load_done();
    }
  }
  fence_before_sync();
  __syncthreads();
  settle(&s_fail);
  if (warp == kEpiWarps) tmem_dealloc(tmem, 512);
  if (tid == 0 && s_fail) atomicOr(A.err, kErrWait);
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's tensor-map encoder, looked up once (the library links only the runtime).
EncodeFn encoder() {
  static EncodeFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult res;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &res) != cudaSuccess ||
        res != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<EncodeFn>(f);
  }();
  return fn;
}

template <int M>
int forward_map(const TArgs& A, CUtensorMap* map) {
  using C = Cfg<M>;
  EncodeFn enc = encoder();
  if (!enc) {
    set_error("dgt (tensor cores): cuTensorMapEncodeTiled not found");
    return CP_ERR_CUDA_;
  }
  const cuuint64_t rows = 16ull * ((cuuint64_t)A.nres << A.S), polys = (cuuint64_t)A.npolys;
  const cuuint64_t row_bytes = C::N2 * 16ull, poly_bytes = (cuuint64_t)A.poly_stride * 16;
  const cuuint32_t ones[3] = {1, 1, 1};
  cuuint64_t dims[3] = {2ull * C::N2, rows, polys}, strides[2] = {row_bytes, poly_bytes};
  cuuint32_t box[3] = {256, 16, 1};
  if (M == 2) {
    dims[1] = polys;
    dims[2] = rows;
    strides[0] = poly_bytes;
    strides[1] = row_bytes;
    box[0] = 128;
    box[1] = 2;
    box[2] = 16;
  }
  const CUresult rc = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, const_cast<ulonglong2*>(A.fsrc), dims, strides, box,
                          ones, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) {
    set_error("dgt (tensor cores): cuTensorMapEncodeTiled failed (status " + std::to_string((int)rc) + ")");
    return CP_ERR_CUDA_;
  }
  return 0;
}

template <int M, bool INV>
int launch_m(const TArgs& A, unsigned grid, cudaStream_t st) {
  CUtensorMap fmap{};
  if (!INV)
    if (int rc = forward_map<M>(A, &fmap)) return rc;
  static std::atomic<unsigned long long> done{0};
  constexpr int smem = Cfg<M>::SMEM;
  if (int rc = ensure_smem(k_tdgt<M, INV>, smem, done)) return rc;
  k_tdgt<M, INV><<<grid, kThreads, smem, st>>>(A, fmap);
  return check_launch("dgt (tensor cores)");
}

int launch_any(int M, bool inv, const TArgs& A, unsigned grid, cudaStream_t st) {
  switch (M * 2 + (inv ? 1 : 0)) {
    case 4: return launch_m<2, false>(A, grid, st);
    case 5: return launch_m<2, true>(A, grid, st);
    case 6: return launch_m<3, false>(A, grid, st);
    case 7: return launch_m<3, true>(A, grid, st);
    case 8: return launch_m<4, false>(A, grid, st);
    case 9: return launch_m<4, true>(A, grid, st);
    case 10: return launch_m<5, false>(A, grid, st);
    case 11: return launch_m<5, true>(A, grid, st);
  }
  set_error("dgt (tensor cores): no kernel for this size");
  return CP_ERR_UNSUPPORTED_;
}

}  // namespace

int launch_tdgt(const Engine& e, ulonglong2* data, const ulonglong2* fsrc, const InvSrc& isrc, int nres, int rid_off,
                int npolys, long long poly_stride, bool inverse, cudaStream_t st, const int* rid_list) {
  const int M = e.tlayout.logNc - 8;
  TArgs A{};
  A.tab = e.d_ttab;
  A.L = e.tlayout;
  A.mc = e.d_mc;
  A.data = data;
  A.fsrc = fsrc ? fsrc : data;
  A.isrc = isrc;
  A.rid_list = nullptr;
  A.nres = nres;
  A.rid_off = rid_off;
  A.npolys = npolys;
  A.S = e.tlayout.S;
  A.poly_stride = poly_stride;
  A.b2 = inverse && A.S == 0 ? isrc.untwist : 0;
  A.err = e.d_err;
  const long long G = M >= 4 ? 1 : (M == 3 ? 2 : 4);  // residues per unit
  if (inverse && isrc.mode != 0 && isrc.mode != 2) {
    set_error("dgt (tensor cores): products are formed before the transform");
    return CP_ERR_INVALID_;
  }
  if (rid_list && A.S > 0) {
    set_error("dgt (tensor cores): a work list needs a whole-CTA size");
    return CP_ERR_INVALID_;
  }
  if (!rid_list) {
    const long long per = (((long long)npolys << A.S) + G - 1) / G;
    if (per * nres > 0x7fffffffLL || ((long long)npolys << A.S) > 0x7fffffffLL) {
      set_error("dgt: grid too large");
      return CP_ERR_INVALID_;
    }
    A.units_per_prime = (unsigned)per;
    A.nunits = (unsigned)(per * nres);
    return launch_any(M, inverse, A, std::min(A.nunits, (unsigned)e.sms), st);
  }
  for (int i0 = 0; i0 < npolys; i0 += kTdgtListMax) {  // rows of the list, kTdgtListMax at a time
    const int n = npolys - i0 < kTdgtListMax ? npolys - i0 : kTdgtListMax;
    const size_t o = (size_t)i0 * poly_stride;
    TArgs B = A;
    B.rid_list = rid_list + i0;
    B.nlist = n;
    B.nprimes = e.k + e.kl;
    B.npolys = n;
    B.data = data + o;
    B.fsrc = A.fsrc + o;
    for (int v = 0; v < 4; ++v) B.isrc.p[v] = isrc.p[v] ? isrc.p[v] + o : nullptr;
    if (int rc = launch_any(M, inverse, B, std::min((unsigned)n, (unsigned)e.sms), st)) return rc;
  }
  return 0;
}

}  // namespace cpoly
