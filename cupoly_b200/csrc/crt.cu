// Coefficient I/O on the device: big-integer coefficients <-> RNS residues,
// and the binary residue wire format.
//
// Replaces cuPoly's host-side NTL conversions poly_crt / poly_icrt
// (src/arithmetic/polynomial.cu:190-296), which reduce every ZZ coefficient
// modulo each prime on the host and recombine with NTL's CRT on read-back,
// and the string forms poly_export_residues / poly_import_residues
// (polynomial.cu:1291-1383).
//
// Coefficient layout: unsigned integers of `nlimbs` 64-bit limbs, least
// significant first, coefficient-major: uint64_t[npolys][nphi][nlimbs].
//  * CRT: residue r of coefficient x = sum_l x_l (2^(64 l) mod q_r), a lazy
//    192-bit dot product with one final reduction, or a byte matrix product.
//  * ICRT: the mixed-radix digits d_i of X (exact, word-size), then
//    X = d_0 + q_0 (d_1 + q_1 (d_2 + ...)) by multi-limb Horner; X in [0, Q); or
//    the CRT sum as a byte matrix product, from the overflow count.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>
#include <utility>
#include <vector>

#include "../../include/cupoly_b200.h"
#include "launch.cuh"
#include "product_sums.cuh"
#include "umma.cuh"

namespace cpoly {

namespace {

constexpr int kCrtTensor = 32;    // most limbs of cp_crt on the tensor cores (256 bytes: column sums below 2^24)
constexpr int kIcrtFirst = 5, kIcrtTensor = 16;  // primes of cp_icrt on the tensor cores (at most 256 columns of tensor memory)
constexpr int kMaxIcrt = 24;  // largest base recombined by cp_icrt (|Q|, |B| <= 24)
constexpr int kIcrtHeld = 15;  // primes whose digits and limbs k_icrt keeps in registers

// i / d for i < 2^16, 2 <= d <= 64, with m = ceil(2^32 / d).
__device__ __forceinline__ int div_small(int i, uint32_t m) { return (int)__umulhi((uint32_t)i, m); }

__device__ __forceinline__ void cp_async8(uint32_t shared, const uint64_t* global) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(shared), "l"(global) : "memory");
}

// R residues from rid on of one Gaussian element whose limbs are at s0 and s1.
template <int R>
__device__ __forceinline__ void crt_rows(ulonglong2* __restrict__ out, const uint64_t* s0, const uint64_t* s1,
                                         int nlimbs, int N, int rid, const ModConst* __restrict__ mc,
                                         const uint64_t* __restrict__ pow64) {
  const uint64_t* w = pow64 + (size_t)rid * kMaxLimbs;
  ProductSum<true> x[R], y[R];
#pragma unroll 2
  for (int l = 0; l < nlimbs; ++l) {  // each product < 2^127; 64 terms < 2^133
    const uint64_t a = s0[l], b = s1[l];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint64_t wl = __ldg(w + r * kMaxLimbs + l);
      x[r].mac(a, wl);
      y[r].mac(b, wl);
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint64_t p = mc[rid + r].p;
    const uint32_t c = (uint32_t)((1ull << 63) - p);
    out[(size_t)r * N] = make_ulonglong2(canon(x[r].fold(c), c, p), canon(y[r].fold(c), c, p));
  }
}

// One thread per Gaussian element (coefficients j and j + N) of one residue, blockIdx.y its polynomial
// and residue.  PM: every prime has 63 bits (BFV engines).
template <bool PM>
__global__ void __launch_bounds__(256) k_crt_direct(ulonglong2* __restrict__ out, const uint64_t* __restrict__ coefs,
                                                    int nlimbs, int N, int nres, int rid_off,
                                                    const ModConst* __restrict__ mc,
                                                    const uint64_t* __restrict__ pow64,
                                                    const uint64_t* __restrict__ pow64m) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  const int y = blockIdx.y, rid = rid_off + y % nres;
  const ModConst m = mc[rid];
  const uint64_t* c0 = coefs + ((size_t)(y / nres) * 2 * N + j) * nlimbs;
  const uint64_t* c1 = c0 + (size_t)N * nlimbs;
  uint64_t a0 = 0, a1 = 0;
  if (PM || m.pm) {
    const uint64_t* w = pow64 + (size_t)rid * kMaxLimbs;
    const uint32_t c = (uint32_t)((1ull << 63) - m.p);
    ProductSum<true> x0, x1;
    auto step = [&](int l) {
      const uint64_t wl = __ldg(w + l);
      x0.mac(c0[l], wl);
      x1.mac(c1[l], wl);
    };
    if constexpr (PM) {
#pragma unroll 4
      for (int l = 0; l < nlimbs; ++l) step(l);
    } else {
      for (int l = 0; l < nlimbs; ++l) step(l);
    }
    a0 = canon(x0.fold(c), c, m.p);
    a1 = canon(x1.fold(c), c, m.p);
  } else {
    const uint64_t* wm = pow64m + (size_t)rid * kMaxLimbs;
    for (int l = 0; l < nlimbs; ++l) {
      const uint64_t wl = __ldg(wm + l);
      a0 = add_mod(a0, mont_mul(c0[l], wl, m.p, m.pneg), m.p);
      a1 = add_mod(a1, mont_mul(c1[l], wl, m.p, m.pneg), m.p);
    }
  }
  out[(size_t)y * N + j] = make_ulonglong2(a0, a1);
}

// Residues of T Gaussian elements (coefficients j and j + N) of polynomial blockIdx.y, four at a
// time: groups blockIdx.z, blockIdx.z + gridDim.z, ... of the base.  The limbs are read once, in
// order, into shared memory (rows of an odd number of words: no bank conflicts); one thread per
// element and residue instead read each limb once per residue, 8 bytes from a line at a time
// (nphi 8192, 5 residues of 5 limbs, 128 polynomials, 13 us of traffic: 54 us, 40 us so; the integer
// multiply pipe is busy 64 % of that).
__global__ void __launch_bounds__(128) k_crt(ulonglong2* __restrict__ out, const uint64_t* __restrict__ coefs,
                                             int nlimbs, int N, int nres, int rid_off,
                                             const ModConst* __restrict__ mc, const uint64_t* __restrict__ pow64,
                                             const uint64_t* __restrict__ pow64m, uint32_t inv_nlimbs, int pm) {
  extern __shared__ uint64_t s_limbs[];
  const int T = blockDim.x, j0 = blockIdx.x * T, nt = N - j0 < T ? N - j0 : T, row = nlimbs | 1;
  const uint64_t* c0 = coefs + ((size_t)blockIdx.y * 2 * N + j0) * nlimbs;
  const uint64_t* c1 = c0 + (size_t)N * nlimbs;
  const uint32_t base = umma::smem_u32(s_limbs);
  for (int i = threadIdx.x; i < nt * nlimbs; i += T) {
    const int e = nlimbs == 1 ? i : div_small(i, inv_nlimbs), at = e * row + (i - e * nlimbs);
    cp_async8(base + 8 * at, c0 + i);  // all of them in flight together
    cp_async8(base + 8 * (T * row + at), c1 + i);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if ((int)threadIdx.x >= nt) return;
  const uint64_t* s0 = s_limbs + threadIdx.x * row;
  const uint64_t* s1 = s0 + T * row;
  ulonglong2* o = out + (size_t)blockIdx.y * nres * N + j0 + threadIdx.x;
  for (int r0 = 4 * blockIdx.z; r0 < nres; r0 += 4 * gridDim.z) {
    const int n = nres - r0 < 4 ? nres - r0 : 4;
    if (pm) {  // 63-bit primes: lazy sums, one reduction
      switch (n) {
        case 1: crt_rows<1>(o + (size_t)r0 * N, s0, s1, nlimbs, N, rid_off + r0, mc, pow64); break;
        case 2: crt_rows<2>(o + (size_t)r0 * N, s0, s1, nlimbs, N, rid_off + r0, mc, pow64); break;
        case 3: crt_rows<3>(o + (size_t)r0 * N, s0, s1, nlimbs, N, rid_off + r0, mc, pow64); break;
        default: crt_rows<4>(o + (size_t)r0 * N, s0, s1, nlimbs, N, rid_off + r0, mc, pow64);
      }
      continue;
    }
    for (int r = r0; r < r0 + n; ++r) {  // other primes: one Montgomery product per limb with 2^(64 l) in Montgomery form
      const ModConst m = mc[rid_off + r];
      if (m.pm) {
        crt_rows<1>(o + (size_t)r * N, s0, s1, nlimbs, N, rid_off + r, mc, pow64);
        continue;
      }
      const uint64_t* wm = pow64m + (size_t)(rid_off + r) * kMaxLimbs;
      uint64_t a0 = 0, a1 = 0;
      for (int l = 0; l < nlimbs; ++l) {
        const uint64_t wl = __ldg(wm + l);
        a0 = add_mod(a0, mont_mul(s0[l], wl, m.p, m.pneg), m.p);
        a1 = add_mod(a1, mont_mul(s1[l], wl, m.p, m.pneg), m.p);
      }
      o[(size_t)r * N] = make_ulonglong2(a0, a1);
    }
  }
}

// One thread per coefficient of polynomial blockIdx.y: threads 0 .. 63 of a block take the first
// halves of 64 Gaussian elements, the others the second halves.  NS is a template argument so that
// the digits and limbs stay in registers (indexed by a loop they lay in local memory), and the
// coefficients leave through shared memory in order (nphi 8192, 5 residues, 128 polynomials, 13 us of
// traffic: 48 us before, 32 us so; bound by the integer multiply pipe).
template <int NS>
__global__ void __launch_bounds__(128) k_icrt(uint64_t* __restrict__ coefs, int nlimbs,
                                              const ulonglong2* __restrict__ in, int N, int src_off,
                                              const ModConst* __restrict__ mc, const uint64_t* __restrict__ inv,
                                              const uint64_t* __restrict__ inv_s, uint32_t inv_nlimbs) {
  constexpr int ROW = NS | 1;
  __shared__ uint64_t s_x[128 * ROW];
  const int tid = threadIdx.x, half = tid >> 6, j0 = blockIdx.x * 64, nt = N - j0 < 64 ? N - j0 : 64;
  const int j = j0 + (tid & 63);
  uint64_t d[NS];
  if ((tid & 63) < nt) {
    const uint64_t* src = reinterpret_cast<const uint64_t*>(in + (size_t)blockIdx.y * NS * N + j) + half;
#pragma unroll
    for (int i = 0; i < NS; ++i) d[i] = src[(size_t)i * 2 * N];
    // mixed-radix digits: d_i = (x_i - d_0 - d_1 s_0 - ...) / (s_0 ... s_{i-1}) mod s_i, all i > l
    // one step at a time: independent of each other
#pragma unroll
    for (int l = 0; l < NS - 1; ++l) {
#pragma unroll
      for (int i = l + 1; i < NS; ++i) {
        const uint64_t si = mc[src_off + i].p;
        uint64_t dl = d[l];  // d_l < s_l: one subtraction for primes of one size, a division otherwise
        if (dl >= si) dl = dl - si < si ? dl - si : dl % si;
        const int c = i * (i - 1) / 2 + l;
        d[i] = shoup_mul(d[i] + si - dl, __ldg(inv + c), __ldg(inv_s + c), si);
      }
    }
    // X = d_{NS-1}; X = X s_i + d_i for i = NS-2 .. 0, in 64-bit limbs: below s_i ... s_{NS-1}, so
    // NS - i limbs after step i
    uint64_t X[NS];
    X[0] = d[NS - 1];
#pragma unroll
    for (int i = NS - 2; i >= 0; --i) {
      const uint64_t si = mc[src_off + i].p;
      uint64_t carry = d[i];
#pragma unroll
      for (int l = 0; l < NS - 1 - i; ++l) {
        uint64_t lo, hi;
        mul128(X[l], si, lo, hi);
        const uint64_t s = lo + carry;
        carry = hi + (s < lo);
        X[l] = s;
      }
      X[NS - 1 - i] = carry;
    }
#pragma unroll
    for (int l = 0; l < NS; ++l) s_x[tid * ROW + l] = X[l];
  }
  __syncthreads();
  uint64_t* o = coefs + ((size_t)blockIdx.y * 2 * N + j0 + (size_t)half * N) * nlimbs;
  for (int i = tid & 63; i < nt * nlimbs; i += 64) {
    const int e = nlimbs == 1 ? i : div_small(i, inv_nlimbs), l = i - e * nlimbs;
    o[i] = l < NS ? s_x[(64 * half + e) * ROW + l] : 0;
  }
}

// The same for a base of ns > kIcrtHeld primes, a coefficient's digits and limbs in one row of shared
// memory: in registers they spill and the unrolled products no longer fit the instruction cache (us, 24
// primes at nphi 8192, 1 polynomial: local memory 53, registers 70, so 50; 20 polynomials 166, 213, 152).  Digit i
// lies at word i; when step i takes it, limbs 0 .. ns - 2 - i of X lie at words ns - 1 .. i + 1, and the limb
// that the step adds takes its place.
__global__ void __launch_bounds__(128) k_icrt_wide(uint64_t* __restrict__ coefs, int nlimbs,
                                                   const ulonglong2* __restrict__ in, int N, int ns, int src_off,
                                                   const ModConst* __restrict__ mc, const uint64_t* __restrict__ inv,
                                                   const uint64_t* __restrict__ inv_s, uint32_t inv_nlimbs) {
  constexpr int ROW = kMaxIcrt | 1;
  __shared__ uint64_t s_x[128 * ROW];
  const int tid = threadIdx.x, half = tid >> 6, j0 = blockIdx.x * 64, nt = N - j0 < 64 ? N - j0 : 64;
  const int j = j0 + (tid & 63);
  if ((tid & 63) < nt) {
    uint64_t* x = s_x + tid * ROW;
    const uint64_t* src = reinterpret_cast<const uint64_t*>(in + (size_t)blockIdx.y * ns * N + j) + half;
    for (int i = 0; i < ns; ++i) {
      const uint64_t si = mc[src_off + i].p;
      uint64_t y = src[(size_t)i * 2 * N];
      for (int l = 0; l < i; ++l) {
        uint64_t dl = x[l];
        if (dl >= si) dl = dl - si < si ? dl - si : dl % si;
        const int c = i * (i - 1) / 2 + l;
        y = shoup_mul(y + si - dl, __ldg(inv + c), __ldg(inv_s + c), si);
      }
      x[i] = y;
    }
    for (int i = ns - 2; i >= 0; --i) {
      const uint64_t si = mc[src_off + i].p;
      uint64_t carry = x[i];
      for (int w = ns - 1; w > i; --w) {
        const uint64_t v = x[w], lo = v * si, s = lo + carry;
        carry = mulhi64(v, si) + (s < lo);
        x[w] = s;
      }
      x[i] = carry;
    }
  }
  __syncthreads();
  uint64_t* o = coefs + ((size_t)blockIdx.y * 2 * N + j0 + (size_t)half * N) * nlimbs;
  for (int i = tid & 63; i < nt * nlimbs; i += 64) {
    const int e = div_small(i, inv_nlimbs), l = i - e * nlimbs;
    o[i] = l < ns ? s_x[(64 * half + e) * ROW + ns - 1 - l] : 0;
  }
}

using IcrtFn = void (*)(uint64_t*, int, const ulonglong2*, int, int, const ModConst*, const uint64_t*,
                        const uint64_t*, uint32_t);
template <int... I>
IcrtFn icrt_kernel(int ns, std::integer_sequence<int, I...>) {
  static constexpr IcrtFn table[] = {k_icrt<I + 1>...};
  return table[ns - 1];
}

// ---- on the tensor cores ----
//
// Both directions are constant linear maps of bytes (see tdgt.cu): a coefficient's limbs are its
// row of the operand as they are, residue r has 8 columns, and byte b of limb l contributes the
// bytes of 2^(64 l + 8 b) mod q_r.  Back, with y_i = x_i (Q/q_i)^-1 mod q_i,
//   X = sum_i y_i (Q/q_i) - v Q,  v = floor(sum_i y_i / q_i),
// whose limb has 8 columns, modulo 2^(64 NS); v, counted in FP64 and rounded down, is one more
// byte (times 2^(64 NS) - Q), and at most one subtraction of Q is left.  Per output 8 column sums
// and one fold (a carry) are left of NS products and a reduction on the integer multiply pipe.
// A CTA of 128 threads takes 128 Gaussian elements: coefficients j and j + N are rows of two
// tiles.  crt / icrt of 128 polynomials (us; CUDA cores below), nphi 8192, 5
// residues (13 us of traffic each): 23 / 29 (36 / 31); 32 polynomials, nphi 16384, 12 residues (16
// us): 29 / 40 (69 / 115).  What is left is the latency of a tile's steps, four CTAs a SM.
struct IoTensor {
  const uint8_t* mat;
  int cols, tiles_per_poly, ntiles;
  uint32_t inv_nlimbs;
  int* err;
};

__global__ void __launch_bounds__(128, 4)
    k_crt_tensor(ulonglong2* __restrict__ out, const uint64_t* __restrict__ coefs, int nlimbs, int N, int nres,
                 int rid_off, const ModConst* __restrict__ mc, IoTensor io) {
  using namespace umma;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ uint64_t s_bar[2];
  __shared__ uint32_t s_slot;
  __shared__ int s_fail;
  const int tid = threadIdx.x;
  const ConvShape sh{nlimbs, nres};
  const int grp = sh.group(), ngrp = sh.groups(), cols = sh.cols();
  const int KB = (8 * nlimbs + 31) / 32 * 32, CH = KB / 16;
  const uint32_t sA = smem_u32(smem_raw), sB = sA + 2 * 128 * KB;
  const uint32_t bD = smem_u32(s_bar), bB = bD + 8;
  if (tid == 0) {
    mbar_init(bD, 1);
    mbar_init(bB, 1);
    mbar_init_fence();
    s_fail = 0;
    mbar_expect_tx(bB, CH * cols * 16);
    for (int ch = 0; ch < CH; ++ch)
      bulk_load(sB + ch * cols * 16, io.mat + ((size_t)ch * io.cols + 8 * rid_off) * 16, cols * 16, bB);
  }
  if (tid < 32) tmem_alloc(smem_u32(&s_slot), 128);
  auto word = [&](int comp, int row, int l) { return sA + comp * 128 * KB + (l >> 1) * 2048 + row * 16 + (l & 1) * 8; };
  for (int l = nlimbs; l < KB / 8; ++l)
    for (int comp = 0; comp < 2; ++comp)
      asm volatile("st.shared.b64 [%0], %1;" ::"r"(word(comp, tid, l)), "l"(0ull) : "memory");
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = s_slot, tl = tmem + ((uint32_t)(tid & 96) << 16);
  const uint32_t idesc = idesc_u8(128, 8 * grp);
  const uint64_t dA = smem_desc(sA, 2048, 128, kSwzNone), dB = smem_desc(sB, cols * 16, 128, kSwzNone);
  uint32_t k8 = 256;
  asm volatile("" : "+r"(k8));
  uint32_t pd = 0;
  auto load = [&](int tile) {
    const int poly = tile / io.tiles_per_poly, j0 = (tile % io.tiles_per_poly) * 128;
    const uint64_t* c0 = coefs + ((size_t)poly * 2 * N + j0) * nlimbs;
    const uint64_t* c1 = c0 + (size_t)N * nlimbs;
    for (int i = tid; i < 128 * nlimbs; i += 128) {
      const int e = nlimbs == 1 ? i : div_small(i, io.inv_nlimbs), l = i - e * nlimbs;
      cp_async8(word(0, e, l), c0 + i);
      cp_async8(word(1, e, l), c1 + i);
    }
  };
  if ((int)blockIdx.x < io.ntiles) load(blockIdx.x);
  bool first = true;
  for (int tile = blockIdx.x; tile < io.ntiles; tile += gridDim.x) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    fence_async_smem();
    fence_before_sync();
    __syncthreads();  // every row is written, and the last tile's products are read
    auto issue = [&](int g) {
      if (tid == 0) {
        fence_after_sync();
        for (int comp = 0; comp < 2; ++comp)
          for (int ks = 0; ks < KB / 32; ++ks)
            mma_u8(tmem + 64 * comp, dA + (comp * 128 * KB + ks * 4096) / 16, dB + (ks * 2 * cols + g * grp * 8), idesc,
                   ks > 0);
        mma_commit(bD);
      }
    };
    if (first) mbar_wait(bB, 0, &s_fail);
    first = false;
    issue(0);
    const int poly = tile / io.tiles_per_poly, j = (tile % io.tiles_per_poly) * 128 + tid;
    ulonglong2* o = out + (size_t)poly * nres * N + j;
    for (int g = 0; g < ngrp; ++g) {
      const int t0 = g * grp, t1 = t0 + grp < nres ? t0 + grp : nres;
      mbar_wait(bD, pd & 1, &s_fail);
      ++pd;
      fence_after_sync();
      // the operand has been read: the next tile's limbs are on their way during the sums
      if (g == ngrp - 1 && tile + (int)gridDim.x < io.ntiles) load(tile + gridDim.x);
      uint32_t c0[16], c1[16];
      auto ld = [&](int t, uint32_t(&c)[16]) { tmem_ld8x2(c, tl + 8 * (t - t0), tl + 64 + 8 * (t - t0)); };
      auto one = [&](int t, const uint32_t(&c)[16]) {
        const uint64_t p = mc[rid_off + t].p;
        const Red R{p, (uint32_t)((1ull << 63) - p), k8, k8 << 8};
        o[(size_t)t * N] = make_ulonglong2(red2p(col_sum(c, R), p), red2p(col_sum(c + 8, R), p));
      };
      ld(t0, c0);
#pragma unroll 1
      for (int t = t0; t < t1; t += 2) {  // the next residue's columns are on their way while one is summed
        tmem_ld_wait(c0);
        if (t + 1 < t1) ld(t + 1, c1);
        one(t, c0);
        if (t + 1 < t1) {
          tmem_ld_wait(c1);
          if (t + 2 < t1) ld(t + 2, c0);
          one(t + 1, c1);
        }
      }
      if (g + 1 < ngrp) {
        fence_before_sync();
        __syncthreads();  // the group's products are read
        issue(g + 1);
      }
    }
  }
  fence_before_sync();
  __syncthreads();
  settle(&s_fail);
  if (tid < 32) tmem_dealloc(tmem, 128);
  if (tid == 0 && s_fail) atomicOr(io.err, kErrWait);
}

// Shapes and constants of cp_icrt's matrix: K bytes (NS residues and the count), columns (limbs,
// a multiple of 16), then the words (Q/q_i)^-1 mod q_i, their Shoup quotients, 1/q_i as FP64 and
// the limbs of Q.
__host__ __device__ constexpr int icrt_kbytes(int ns) { return (8 * ns + 1 + 31) / 32 * 32; }
__host__ __device__ constexpr int icrt_cols(int ns) { return (8 * ns + 15) / 16 * 16; }
constexpr size_t icrt_bytes(int ns) { return (size_t)icrt_kbytes(ns) * icrt_cols(ns) + 4 * 8 * (size_t)ns; }

template <int NS>
__global__ void __launch_bounds__(128, NS <= 8 ? 4 : 2)
    k_icrt_tensor(uint64_t* __restrict__ coefs, int nlimbs, const ulonglong2* __restrict__ in, int N, int src_off,
                  const ModConst* __restrict__ mc, IoTensor io) {
  using namespace umma;
  constexpr int KB = icrt_kbytes(NS), CH = KB / 16, COLS = icrt_cols(NS), HALF = NS <= 8 ? 64 : 128;
  constexpr int ROW = NS | 1;  // words between the staged coefficients, in the operand's own place
  static_assert(ROW * 8 <= KB, "staging");
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ uint64_t s_bar[2];
  __shared__ uint32_t s_slot;
  __shared__ int s_fail;
  const int tid = threadIdx.x;
  const uint32_t sA = smem_u32(smem_raw), sB = sA + 2 * 128 * KB;
  const uint32_t bD = smem_u32(s_bar), bB = bD + 8;
  if (tid == 0) {
    mbar_init(bD, 1);
    mbar_init(bB, 1);
    mbar_init_fence();
    s_fail = 0;
    mbar_expect_tx(bB, KB * COLS);
    bulk_load(sB, io.mat, KB * COLS, bB);
  }
  if (tid < 32) tmem_alloc(smem_u32(&s_slot), 2 * HALF);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = s_slot, tl = tmem + ((uint32_t)(tid & 96) << 16);
  const uint32_t idesc = idesc_u8(128, COLS);
  const uint64_t dA = smem_desc(sA, 2048, 128, kSwzNone), dB = smem_desc(sB, COLS * 16, 128, kSwzNone);
  const uint64_t* inv = reinterpret_cast<const uint64_t*>(io.mat + KB * COLS);
  const uint64_t *inv_s = inv + NS, *recip = inv + 2 * NS, *Q = inv + 3 * NS;
  uint32_t k8 = 256;
  asm volatile("" : "+r"(k8));
  const uint32_t k16 = k8 << 8;
  ulonglong2 x[NS];
  auto load = [&](int tile) {
    const ulonglong2* p = in + (size_t)(tile / io.tiles_per_poly) * NS * N + (tile % io.tiles_per_poly) * 128 + tid;
#pragma unroll
    for (int i = 0; i < NS; ++i) x[i] = p[(size_t)i * N];
  };
  if ((int)blockIdx.x < io.ntiles) load(blockIdx.x);
  uint32_t pd = 0;
  for (int tile = blockIdx.x; tile < io.ntiles; tile += gridDim.x) {
#pragma unroll
    for (int comp = 0; comp < 2; ++comp) {
      uint64_t y[NS + 1];
      double f = -0x1p-40;  // FP64 errors are below 2^-45: v is never too large, and one too small at most
#pragma unroll
      for (int i = 0; i < NS; ++i) {
        y[i] = shoup_mul(comp ? x[i].y : x[i].x, __ldg(inv + i), __ldg(inv_s + i), mc[src_off + i].p);
        const double c = __longlong_as_double(__ldg(recip + i));
        f = __fma_rn(u32_to_double((uint32_t)y[i]), c, f);
        f = __fma_rn(u32_to_double((uint32_t)(y[i] >> 32)), c * 4294967296.0, f);
      }
      y[NS] = f > 0.0 ? (uint64_t)(uint32_t)__double2int_rd(f) : 0;
      const uint32_t row = sA + comp * 128 * KB + tid * 16;
#pragma unroll
      for (int ch = 0; ch < CH; ++ch) {
        const uint64_t lo = 2 * ch <= NS ? y[2 * ch <= NS ? 2 * ch : 0] : 0;
        const uint64_t hi = 2 * ch + 1 <= NS ? y[2 * ch + 1 <= NS ? 2 * ch + 1 : 0] : 0;
        asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(row + ch * 2048), "l"(lo), "l"(hi) : "memory");
      }
    }
    fence_async_smem();
    fence_before_sync();
    __syncthreads();  // every row is written, and the last tile's products are read
    if (pd == 0) mbar_wait(bB, 0, &s_fail);
    if (tid == 0) {
      fence_after_sync();
#pragma unroll
      for (int comp = 0; comp < 2; ++comp)
#pragma unroll
        for (int ks = 0; ks < KB / 32; ++ks)
          mma_u8(tmem + HALF * comp, dA + (comp * 128 * KB + ks * 4096) / 16, dB + ks * 2 * COLS, idesc, ks > 0);
      mma_commit(bD);
    }
    const int poly = tile / io.tiles_per_poly, j0 = (tile % io.tiles_per_poly) * 128;
    if (tile + (int)gridDim.x < io.ntiles) load(tile + gridDim.x);  // on their way during the products
    mbar_wait(bD, pd & 1, &s_fail);
    ++pd;
    fence_after_sync();
#pragma unroll 1
    for (int comp = 0; comp < 2; ++comp) {
      uint64_t X[NS], D[NS];
      uint32_t carry = 0;
      uint32_t c[2][16];
      tmem_ld16(c[0], tl + HALF * comp);
#pragma unroll
      for (int l = 0; l < NS; ++l) {  // two limbs a load; the columns past the last limb are zero
        const uint32_t* s = c[(l >> 1) & 1] + 8 * (l & 1);
        if ((l & 1) == 0) {
          tmem_ld_wait(c[(l >> 1) & 1]);
          if (l + 2 < NS) tmem_ld16(c[((l >> 1) + 1) & 1], tl + HALF * comp + 8 * (l + 2));
        }
        // as col_sum: a 17-bit carry fits on top of a word of two columns
        const uint32_t a0 = s[1] * k8 + s[0] + carry, a1 = s[3] * k8 + s[2];
        const uint32_t a2 = s[5] * k8 + s[4], a3 = s[7] * k8 + s[6];
        const uint64_t t = mad_wide(a1, k16, pack64(a0, a2));
        const uint64_t h = mad_wide(a3, k16, (uint64_t)(t >> 32));
        X[l] = pack64((uint32_t)t, (uint32_t)h);
        carry = (uint32_t)(h >> 32);
      }
      uint64_t borrow = 0;
#pragma unroll
      for (int l = 0; l < NS; ++l) {
        const uint64_t q = __ldg(Q + l), d = X[l] - q;
        D[l] = d - borrow;
        borrow = (X[l] < q) | (d < borrow);
      }
      const uint32_t at = sA + comp * 128 * KB + tid * ROW * 8;
#pragma unroll
      for (int l = 0; l < NS; ++l)
        asm volatile("st.shared.b64 [%0], %1;" ::"r"(at + 8 * l), "l"(borrow ? X[l] : D[l]) : "memory");
    }
    fence_before_sync();
    __syncthreads();
    for (int comp = 0; comp < 2; ++comp) {
      uint64_t* o = coefs + ((size_t)poly * 2 * N + (size_t)comp * N + j0) * nlimbs;
      const uint64_t* sx = reinterpret_cast<const uint64_t*>(smem_raw + comp * 128 * KB);
      for (int i = tid; i < 128 * nlimbs; i += 128) {
        const int e = nlimbs == 1 ? i : div_small(i, io.inv_nlimbs), l = i - e * nlimbs;
        o[i] = l < NS ? sx[e * ROW + l] : 0;
      }
    }
    __syncthreads();  // the staged coefficients are read
  }
  fence_before_sync();
  __syncthreads();
  settle(&s_fail);
  if (tid < 32) tmem_dealloc(tmem, 2 * HALF);
  if (tid == 0 && s_fail) atomicOr(io.err, kErrWait);
}

using IcrtTensorFn = void (*)(uint64_t*, int, const ulonglong2*, int, int, const ModConst*, IoTensor);
template <int... I>
IcrtTensorFn icrt_tensor_kernel(int ns, std::integer_sequence<int, I...>) {
  static constexpr IcrtTensorFn table[] = {k_icrt_tensor<I + kIcrtFirst>...};
  return table[ns - kIcrtFirst];
}

int io_ctas(const Engine& e, int smem_bytes, int most_per_sm) {
  const int fit = 220 * 1024 / (smem_bytes + 1024);
  return e.sms * std::max(1, std::min(fit, most_per_sm));
}

__global__ void __launch_bounds__(256) k_icrt_t(uint64_t* __restrict__ coefs, int nlimbs,
                                                const ulonglong2* __restrict__ in, int N) {
  const int jj = blockIdx.x * blockDim.x + threadIdx.x;
  if (jj >= 2 * N) return;
  const int poly = blockIdx.y;
  const ulonglong2 x = in[(size_t)poly * N + (jj < N ? jj : jj - N)];
  uint64_t* o = coefs + ((size_t)poly * 2 * N + jj) * nlimbs;
  o[0] = jj < N ? x.x : x.y;
  for (int l = 1; l < nlimbs; ++l) o[l] = 0;
}

// Wire header: 16 little-endian 32-bit words.
struct WireHeader {
  uint32_t magic, version, nphi, nres, base, npolys, domain, flags;
  uint32_t reserved[8];
};
static_assert(sizeof(WireHeader) == 64, "wire header is 64 bytes");

// Whether cp_crt runs with a thread per element and residue (k_crt_direct) where the tensor cores do not
// take it.  k_crt's blocks stage the limbs and then take the residues one after the other: with fewer blocks than
// the SMs hold, with one residue (nothing is read twice) or with the long Montgomery chains of CKKS primes that
// costs more than the limbs read again (us, k_crt / direct: nphi 8192, 5 residues and limbs, 1 polynomial 3.4 /
// 2.4, 2 3.4 / 3.0, 4 3.6 / 3.5, 8 4.8 / 5.1; 1 residue of 6 limbs, 100 polynomials 12.9 / 9.9; CKKS, 6 residues of 7 limbs, 1
// polynomial 6.7 / 3.1, 64 46 / 48; 24 of 25 limbs at nphi 32768, 4 polynomials 178 / 155).  Rows of a multiple of 8
// words fall on few sets of L1 and favour k_crt (12 residues of 24 limbs, nphi 8192, 1 polynomial 7.1 / 10.8).
bool crt_direct(const Engine& e, int nres, int nlimbs, int npolys) {
  const long long blocks = (long long)npolys * nres * ((e.N + 255) / 256), sms = e.sms;
  const bool strided = nlimbs % 8 == 0;
  if (e.N < 128 && (nres > 2 || e.ckks_prec)) return e.ckks_prec || 4 * blocks <= (strided ? 9 : 16) * sms;
  if (e.ckks_prec) {
    if (!strided) return nres <= 2 || blocks <= 55 * sms;
    if (nlimbs == 8) return blocks <= 4 * sms;
    return nres >= 4 && 2 * blocks <= (nlimbs % 16 ? 5 : 2) * sms;
  }
  if (nres == 1) return nlimbs <= 7 || (nlimbs <= 12 && !strided && blocks <= 9 * sms);
  if (blocks <= sms && (nlimbs <= 14 || (nlimbs % 16 && nlimbs <= (nres >= 4 ? 40 : nres == 3 ? 23 : 0)))) return true;
  if (4 * blocks <= 11 * sms && nlimbs <= (nres >= 4 ? 7 : 6)) return true;
  return blocks <= 2 * sms && nres >= 4 && nlimbs <= 12 && !strided;
}

uint32_t inv_small(int d) { return d < 2 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d); }  // see div_small

const uint64_t* base_primes(const Engine& e, int base, uint64_t* tmp) {
  if (base == CP_TBASE) {
    tmp[0] = e.t;
    return tmp;
  }
  return e.primes.data() + e.rid_offset(base);
}

}  // namespace

// The matrices and constants of k_crt_tensor and k_icrt_tensor.
int build_io_tables(Engine& e) {
  const int R = e.k + e.kl;
  std::vector<uint8_t> io;
  e.io_cols = 0;
  if (!e.ckks_prec) {  // column sums fold by 2^63 = c
    e.io_cols = 8 * (R + 24);  // a base's columns are read up to a multiple of its groups
    io.assign((size_t)kCrtTensor / 2 * e.io_cols * 16, 0);
    for (int r = 0; r < R; ++r) {
      uint64_t f = 1;  // 2^(8 kb) mod p
      for (int kb = 0; kb < 8 * kCrtTensor; ++kb) {
        uint8_t* at = io.data() + ((size_t)(kb >> 4) * e.io_cols + 8 * r) * 16 + (kb & 15);
        for (int j = 0; j < 8; ++j) at[16 * j] = (uint8_t)(f >> (8 * j));
        f = h_mul(f, 256, e.mconst[r]);
      }
    }
  }
  for (int v = 0; v < 2; ++v) {
    const int ns = v ? e.kl : e.k;
    if (ns < kIcrtFirst || ns > kIcrtTensor) continue;
    const uint64_t* p = e.primes.data() + (v ? e.k : 0);
    const ModConst* m = e.mconst.data() + (v ? e.k : 0);
    const int kb_n = icrt_kbytes(ns), cols = icrt_cols(ns);
    e.io_icrt[v] = io.size();
    io.resize(io.size() + ((icrt_bytes(ns) + 127) & ~(size_t)127), 0);
    uint8_t* mat = io.data() + e.io_icrt[v];
    uint64_t* words = reinterpret_cast<uint64_t*>(mat + (size_t)kb_n * cols);
    auto product = [&](int skip) {  // of the base's primes, in ns limbs
      std::vector<uint64_t> x(ns, 0);
      x[0] = 1;
      for (int i = 0; i < ns; ++i) {
        if (i == skip) continue;
        uint64_t carry = 0;
        for (int l = 0; l < ns; ++l) {
          const unsigned __int128 w = (unsigned __int128)x[l] * p[i] + carry;
          x[l] = (uint64_t)w;
          carry = (uint64_t)(w >> 64);
        }
      }
      return x;
    };
    auto put = [&](int kb, const std::vector<uint64_t>& x, int shift) {  // bytes of x 2^(8 shift) mod 2^(64 ns)
      for (int c = shift; c < 8 * ns; ++c)
        mat[(size_t)(kb >> 4) * cols * 16 + (size_t)c * 16 + (kb & 15)] = (uint8_t)(x[(c - shift) >> 3] >> (8 * ((c - shift) & 7)));
    };
    const std::vector<uint64_t> Q = product(-1);
    std::vector<uint64_t> neg(ns);  // 2^(64 ns) - Q
    uint64_t carry = 1;
    for (int l = 0; l < ns; ++l) {
      neg[l] = ~Q[l] + carry;
      carry = carry && neg[l] == 0;
    }
    put(8 * ns, neg, 0);
    for (int i = 0; i < ns; ++i) {
      const std::vector<uint64_t> x = product(i);
      for (int b = 0; b < 8; ++b) put(8 * i + b, x, b);
      uint64_t f = 1;
      for (int l = 0; l < ns; ++l)
        if (l != i) f = h_mul(f, p[l] % p[i], m[i]);
      const uint64_t w = h_invmod(f, p[i]);
      const double rec = 1.0 / (double)p[i];
      words[i] = w;
      words[ns + i] = h_shoup(w, m[i]);
      std::memcpy(words + 2 * ns + i, &rec, 8);
      words[3 * ns + i] = Q[i];
    }
  }
  if (io.empty()) return 0;
  cudaError_t err = cudaMalloc(&e.d_io, io.size());
  if (err != cudaSuccess) {
    set_error(std::string("cudaMalloc failed for engine tables: ") + cudaGetErrorString(err));
    return 4;
  }
  if ((err = cudaMemcpy(e.d_io, io.data(), io.size(), cudaMemcpyHostToDevice)) != cudaSuccess) {
    set_error(std::string("table upload failed: ") + cudaGetErrorString(err));
    return 2;
  }
  return 0;
}

}  // namespace cpoly

using namespace cpoly;


#define CRT_REQUIRE(cond, msg) \
  do {                         \
    if (!(cond)) {             \
      set_error(msg);          \
      return CP_ERR_INVALID;   \
    }                          \
  } while (0)

extern "C" {

int cp_crt(const cp_engine* h, void* out, const uint64_t* coefs, int nlimbs, int base, int npolys, void* stream) {
  CRT_REQUIRE(h && out && coefs, "cp_crt: NULL argument");
  CRT_REQUIRE(base == CP_QBASE || base == CP_BBASE || base == CP_QBBASE, "cp_crt: base must be Q, B or QB");
  CRT_REQUIRE(nlimbs >= 1 && nlimbs <= kMaxLimbs, "cp_crt: nlimbs must be in [1, 64]");
  CRT_REQUIRE(npolys >= 0, "cp_crt: npolys < 0");
  const Engine& e = h->e;
  const int nres = e.n_residues(base);
  if (npolys == 0) return CP_OK;
  CRT_REQUIRE((long long)npolys * nres <= 65535, "cp_crt: npolys x residues exceeds 65535");
  if (e.d_io && e.io_cols && nlimbs <= kCrtTensor && e.N >= 128) {
    const int kb = (8 * nlimbs + 31) / 32 * 32;
    const long long tiles = (long long)npolys * (e.N / 128);
    const int smem = std::max(2 * 128 * kb + kb * ConvShape{nlimbs, nres}.cols(), 46 * 1024);
    // Below some 16 K tile x limb x residue steps the CUDA cores are faster (us, 5 limbs and residues:
    // 512 tiles 6.8 there and 7.7 here, 4096 tiles 36 and 23; 12: 128 tiles 7.9 and 7.2, 512 tiles 20 and 11); with
    // two residues below 32 K (7 limbs, 1600 tiles 6 % faster there, 2560 tiles as fast), with one always (6 limbs, 3200
    // tiles 9.9 and 14.1, 8000 tiles 27 and 32).
    if (smem <= 200 * 1024 && nres > 1 && tiles * nlimbs * nres >= (nres == 2 ? 32768 : 16384)) {
      static std::atomic<unsigned long long> done{0};
      if (int rc = ensure_smem(k_crt_tensor, 200 * 1024, done)) return rc;
      const IoTensor io{e.d_io, e.io_cols, e.N / 128, (int)tiles, inv_small(nlimbs), e.d_err};
      k_crt_tensor<<<(unsigned)std::min<long long>(tiles, io_ctas(e, smem, 4)), 128, smem,
                     reinterpret_cast<cudaStream_t>(stream)>>>(reinterpret_cast<ulonglong2*>(out), coefs, nlimbs, e.N,
                                                               nres, e.rid_offset(base), e.d_mc, io);
      return check_launch("cp_crt");
    }
  }
  if (crt_direct(e, nres, nlimbs, npolys)) {
    const auto direct = e.ckks_prec ? k_crt_direct<false> : k_crt_direct<true>;
    direct<<<dim3((e.N + 255) / 256, npolys * nres), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<ulonglong2*>(out), coefs, nlimbs, e.N, nres, e.rid_offset(base), e.d_mc, e.d_hps + e.ho.pow64,
        e.d_hps + e.ho.pow64m);
    return check_launch("cp_crt");
  }
  // elements per block: the limbs take at most 48 KB
  const int T = nlimbs <= 23 ? 128 : (nlimbs <= 47 ? 64 : 32);
  const unsigned bx = (unsigned)((e.N + T - 1) / T), groups = (unsigned)((nres + 3) / 4);
  // The blocks of a small call take one group of residues each (a group's serial chain is the
  // whole time); with four blocks on each SM reading the limbs once is worth more.
  const long long blocks = (long long)bx * npolys;
  const long long fill = 4LL * e.sms;
  const unsigned gz = blocks >= fill ? 1u : (unsigned)std::min<long long>(groups, (fill + blocks - 1) / blocks);
  k_crt<<<dim3(bx, (unsigned)npolys, gz), T, (size_t)2 * T * (nlimbs | 1) * 8, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<ulonglong2*>(out), coefs, nlimbs, e.N, nres, e.rid_offset(base), e.d_mc, e.d_hps + e.ho.pow64,
      e.d_hps + e.ho.pow64m, inv_small(nlimbs), e.ckks_prec ? 0 : 1);
  return check_launch("cp_crt");
}

int cp_icrt(const cp_engine* h, uint64_t* coefs, int nlimbs, const void* in, int base, int npolys, void* stream) {
  CRT_REQUIRE(h && coefs && in, "cp_icrt: NULL argument");
  CRT_REQUIRE(base == CP_QBASE || base == CP_BBASE || base == CP_TBASE, "cp_icrt: base must be Q, B or T");
  CRT_REQUIRE(npolys >= 0 && npolys <= 65535, "cp_icrt: npolys must be in [0, 65535]");
  const Engine& e = h->e;
  const int ns = e.n_residues(base);
  CRT_REQUIRE(nlimbs >= ns && nlimbs <= kMaxLimbs, "cp_icrt: nlimbs must be in [residues of the base, 64]");
  if (npolys == 0) return CP_OK;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const ulonglong2* src = reinterpret_cast<const ulonglong2*>(in);
  if (base == CP_TBASE) {
    dim3 grid((2 * e.N + 255) / 256, npolys);
    k_icrt_t<<<grid, 256, 0, st>>>(coefs, nlimbs, src, e.N);
    return check_launch("cp_icrt");
  }
  CRT_REQUIRE(ns <= kMaxIcrt, "cp_icrt: base larger than 24 primes");
  if (e.d_io && ns >= kIcrtFirst && ns <= kIcrtTensor && e.N >= 128) {
    const long long tiles = (long long)npolys * (e.N / 128);
    // The CUDA cores' chain grows with the square of the base (us: 12 residues 128 tiles 15 there and 6.0
    // here, 2048 tiles 115 and 40; 6 residues 1024 tiles 13 and 10.5; 5 residues 512 tiles 6.0 and 7.2,
    // 2048 tiles 16.9 and 15.6); up to 4 residues it is short (4 residues 4096 tiles 21 and 25).
    if (ns >= 8 || tiles * ns * ns >= 32768) {
      const int per = ns <= 8 ? 4 : 2;
      const int smem = std::max(2 * 128 * icrt_kbytes(ns) + icrt_kbytes(ns) * icrt_cols(ns), per == 4 ? 46 * 1024 : 80 * 1024);
      IcrtTensorFn fn = icrt_tensor_kernel(ns, std::make_integer_sequence<int, kIcrtTensor - kIcrtFirst + 1>());
      static std::atomic<unsigned long long> done[kIcrtTensor + 1];
      if (int rc = ensure_smem(fn, smem, done[ns])) return rc;
      const IoTensor io{e.d_io + e.io_icrt[base == CP_QBASE ? 0 : 1], 0, e.N / 128, (int)tiles, inv_small(nlimbs), e.d_err};
      fn<<<(unsigned)std::min<long long>(tiles, io_ctas(e, smem, per)), 128, smem, st>>>(coefs, nlimbs, src, e.N,
                                                                                      e.rid_offset(base), e.d_mc, io);
      return check_launch("cp_icrt");
    }
  }
  const uint64_t* inv = e.d_hps + (base == CP_QBASE ? e.ho.qb_inv : e.ho.bq_inv);
  const uint64_t* inv_s = e.d_hps + (base == CP_QBASE ? e.ho.qb_inv_s : e.ho.bq_inv_s);
  if (ns > kIcrtHeld)
    k_icrt_wide<<<dim3((e.N + 63) / 64, npolys), 128, 0, st>>>(coefs, nlimbs, src, e.N, ns, e.rid_offset(base), e.d_mc,
                                                               inv, inv_s, inv_small(nlimbs));
  else
    icrt_kernel(ns, std::make_integer_sequence<int, kIcrtHeld>())<<<dim3((e.N + 63) / 64, npolys), 128, 0, st>>>(
        coefs, nlimbs, src, e.N, e.rid_offset(base), e.d_mc, inv, inv_s, inv_small(nlimbs));
  return check_launch("cp_icrt");
}

size_t cp_wire_bytes(const cp_engine* h, int base, int npolys) {
  if (!h || base < 0 || base > 3 || npolys < 0) return 0;
  const int nres = h->e.n_residues(base);
  return sizeof(WireHeader) + (size_t)nres * 8 + (size_t)npolys * nres * h->e.N * 16;
}

int cp_export_residues(const cp_engine* h, void* host_out, size_t cap, const void* poly, int base, int npolys,
                       int domain, void* stream) {
  CRT_REQUIRE(h && host_out && poly, "cp_export_residues: NULL argument");
  CRT_REQUIRE(base >= 0 && base <= 3 && npolys >= 0, "cp_export_residues: bad base or npolys");
  CRT_REQUIRE(domain == 0 || domain == 1, "cp_export_residues: domain must be 0 (coefficient) or 1 (DGT)");
  const size_t need = cp_wire_bytes(h, base, npolys);
  CRT_REQUIRE(cap >= need, "cp_export_residues: output buffer too small");
  const Engine& e = h->e;
  const int nres = e.n_residues(base);
  WireHeader hd;
  std::memset(&hd, 0, sizeof(hd));
  hd.magic = CP_WIRE_MAGIC;
  hd.version = CP_WIRE_VERSION;
  hd.nphi = (uint32_t)e.nphi;
  hd.nres = (uint32_t)nres;
  hd.base = (uint32_t)base;
  hd.npolys = (uint32_t)npolys;
  hd.domain = (uint32_t)domain;
  unsigned char* o = reinterpret_cast<unsigned char*>(host_out);
  std::memcpy(o, &hd, sizeof(hd));
  uint64_t tmp[1];
  std::memcpy(o + sizeof(hd), base_primes(e, base, tmp), (size_t)nres * 8);
  const size_t body = (size_t)npolys * nres * e.N * 16;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const cudaError_t err = cudaMemcpyAsync(o + sizeof(hd) + (size_t)nres * 8, poly, body, cudaMemcpyDeviceToHost, st);
  if (err != cudaSuccess) return cuda_fail("cp_export_residues", err);
  return sync_and_check(e, "cp_export_residues", st);
}

int cp_import_residues(const cp_engine* h, void* poly, const void* host_in, size_t size, int base, int npolys,
                       int* domain_out, void* stream) {
  CRT_REQUIRE(h && poly && host_in, "cp_import_residues: NULL argument");
  CRT_REQUIRE(base >= 0 && base <= 3 && npolys >= 0, "cp_import_residues: bad base or npolys");
  CRT_REQUIRE(size >= sizeof(WireHeader), "cp_import_residues: truncated header");
  const Engine& e = h->e;
  const int nres = e.n_residues(base);
  WireHeader hd;
  const unsigned char* in = reinterpret_cast<const unsigned char*>(host_in);
  std::memcpy(&hd, in, sizeof(hd));
  CRT_REQUIRE(hd.magic == CP_WIRE_MAGIC, "cp_import_residues: bad magic");
  CRT_REQUIRE(hd.version == CP_WIRE_VERSION, "cp_import_residues: unsupported version");
  CRT_REQUIRE(hd.nphi == (uint32_t)e.nphi, "cp_import_residues: ring degree differs from the engine's");
  CRT_REQUIRE(hd.base == (uint32_t)base && hd.nres == (uint32_t)nres, "cp_import_residues: base differs");
  CRT_REQUIRE(hd.npolys == (uint32_t)npolys, "cp_import_residues: polynomial count differs");
  CRT_REQUIRE(hd.domain <= 1 && hd.flags == 0, "cp_import_residues: bad domain or flags");
  CRT_REQUIRE(size == cp_wire_bytes(h, base, npolys), "cp_import_residues: size does not match the header");
  uint64_t tmp[1];
  const uint64_t* primes = base_primes(e, base, tmp);
  CRT_REQUIRE(std::memcmp(in + sizeof(hd), primes, (size_t)nres * 8) == 0,
              "cp_import_residues: primes differ from the engine's");
  const uint64_t* body = reinterpret_cast<const uint64_t*>(in + sizeof(hd) + (size_t)nres * 8);
  // every residue must be canonical: a malformed request is refused before it reaches the GPU.
  // Rows (polynomial, residue) are checked on up to 8 host threads for large payloads.
  const long long rows = (long long)npolys * nres;
  const size_t row_words = (size_t)2 * e.N;
  std::atomic<bool> bad{false};
  auto check_rows = [&](long long lo, long long hi) {
    for (long long y = lo; y < hi && !bad.load(std::memory_order_relaxed); ++y) {
      const uint64_t q = primes[y % nres];
      const uint64_t* row = body + (size_t)y * row_words;
      uint64_t worst = 0;
      for (size_t j = 0; j < row_words; ++j) worst = row[j] > worst ? row[j] : worst;
      if (worst >= q) bad.store(true);
    }
  };
  const size_t bytes = (size_t)rows * row_words * 8;
  const unsigned hw = std::thread::hardware_concurrency();
  // at most 8 threads and half the host's cores: on a 16-core host 8 threads measured best
  // (42 MB: 2.6 ms with the copy; 16 threads 4.5 ms, as the copy then runs at pageable speed)
  const long long nthreads =
      bytes < ((size_t)4 << 20) ? 1 : std::min<long long>(std::min(hw > 1 ? hw / 2 : 1u, 8u), rows);
  if (nthreads <= 1) {
    check_rows(0, rows);
  } else {
    // no exception may cross the C ABI: if a thread cannot be started, the rows it would
    // have checked are checked on this thread
    std::vector<std::thread> pool;
    long long started = 0;
    try {
      for (; started < nthreads; ++started)
        pool.emplace_back(check_rows, rows * started / nthreads, rows * (started + 1) / nthreads);
    } catch (...) {
    }
    if (started < nthreads) check_rows(rows * started / nthreads, rows);
    for (auto& th : pool) th.join();
  }
  if (bad.load()) {
    set_error("cp_import_residues: residue not reduced modulo its prime");
    return CP_ERR_INVALID;
  }
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  cudaError_t err = cudaMemcpyAsync(poly, body, (size_t)npolys * nres * e.N * 16, cudaMemcpyHostToDevice, st);
  if (err == cudaSuccess) err = cudaStreamSynchronize(st);
  if (err != cudaSuccess) return cuda_fail("cp_import_residues", err);
  if (domain_out) *domain_out = (int)hd.domain;
  return CP_OK;
}

}  // extern "C"
