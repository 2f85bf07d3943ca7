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
//    192-bit dot product with one final reduction.
//  * ICRT: the mixed-radix digits d_i of X (exact, word-size), then
//    X = d_0 + q_0 (d_1 + q_1 (d_2 + ...)) by multi-limb Horner; X in [0, Q).
#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>
#include <utility>
#include <vector>

#include "../../include/cupoly_b200.h"
#include "launch.cuh"
#include "product_sums.cuh"

namespace cpoly {

namespace {

constexpr int kMaxIcrt = 24;  // largest base recombined by cp_icrt (|Q|, |B| <= 24)

// i / d for i < 2^16, 2 <= d <= 64, with m = ceil(2^32 / d).
__device__ __forceinline__ int div_small(int i, uint32_t m) { return (int)__umulhi((uint32_t)i, m); }

__device__ __forceinline__ void cp_async8(uint64_t* shared, const uint64_t* global) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(shared)), "l"(global)
               : "memory");
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
  for (int i = threadIdx.x; i < nt * nlimbs; i += T) {
    const int e = nlimbs == 1 ? i : div_small(i, inv_nlimbs), at = e * row + (i - e * nlimbs);
    cp_async8(s_limbs + at, c0 + i);  // all of them in flight together
    cp_async8(s_limbs + T * row + at, c1 + i);
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

using IcrtFn = void (*)(uint64_t*, int, const ulonglong2*, int, int, const ModConst*, const uint64_t*,
                        const uint64_t*, uint32_t);
template <int... I>
IcrtFn icrt_kernel(int ns, std::integer_sequence<int, I...>) {
  static constexpr IcrtFn table[] = {k_icrt<I + 1>...};
  return table[ns - 1];
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

uint32_t inv_small(int d) { return d < 2 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d); }  // see div_small

const uint64_t* base_primes(const Engine& e, int base, uint64_t* tmp) {
  if (base == CP_TBASE) {
    tmp[0] = e.t;
    return tmp;
  }
  return e.primes.data() + e.rid_offset(base);
}

}  // namespace

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
  // elements per block: the limbs take at most 48 KB
  const int T = nlimbs <= 23 ? 128 : (nlimbs <= 47 ? 64 : 32);
  const unsigned bx = (unsigned)((e.N + T - 1) / T), groups = (unsigned)((nres + 3) / 4);
  // The blocks of a small call take one group of residues each (a group's serial chain is the
  // whole time); with four blocks on each of 148 SMs reading the limbs once is worth more.
  const long long blocks = (long long)bx * npolys;
  const unsigned gz = blocks >= 592 ? 1u : (unsigned)std::min<long long>(groups, (592 + blocks - 1) / blocks);
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
  const uint64_t* inv = e.d_hps + (base == CP_QBASE ? e.ho.qb_inv : e.ho.bq_inv);
  const uint64_t* inv_s = e.d_hps + (base == CP_QBASE ? e.ho.qb_inv_s : e.ho.bq_inv_s);
  icrt_kernel(ns, std::make_integer_sequence<int, kMaxIcrt>())<<<dim3((e.N + 63) / 64, npolys), 128, 0, st>>>(
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
  cudaError_t err = cudaMemcpyAsync(o + sizeof(hd) + (size_t)nres * 8, poly, body, cudaMemcpyDeviceToHost, st);
  if (err == cudaSuccess) err = cudaStreamSynchronize(st);
  if (err != cudaSuccess) return cuda_fail("cp_export_residues", err);
  return CP_OK;
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
