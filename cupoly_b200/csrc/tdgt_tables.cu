// Host-side construction of the tensor-core DGT tables (see tdgt.cu for the passes).
//
// A pass matrix entry pair (output o, input k) with coefficient f in Z_p becomes an 8 x 8 block
// of bytes: row (column of the product) 8 o + j, K byte 8 k + i holds byte j of f 2^(8 i) mod p.
// Index digits: element n = n1 N2 + 16 nm + nl, stored position pos = q1 N2 + 16 qm + ql, where
// q1, qm, ql are the bit-reversed digits of the frequency k = k1 + 16 km + 16 NM kl.
#include <cstring>

#include "engine.cuh"

namespace cpoly {

namespace {

int brev(int x, int bits) {
  int r = 0;
  for (int i = 0; i < bits; ++i) {
    r = (r << 1) | (x & 1);
    x >>= 1;
  }
  return r;
}

struct Mat {
  uint8_t* m;
  int cols;  // columns (8 per output)
  const ModConst& mc;
  bool quad = false;  // columns of four elements interleaved for tmem_ld_quad (umma.cuh)
  // column of byte j of output o
  int col(int o, int j) const {
    if (!quad) return 8 * o + j;
    const int g = o >> 3, e = (o >> 1) & 3, comp = o & 1;  // element 4 g + e
    return 64 * g + 8 * (4 * comp + (j >> 1)) + 2 * e + (j & 1);
  }
  // input k (its 8 K bytes), output o (its 8 columns), coefficient f
  void put(int o, int k, uint64_t f) {
    // the 8 x 8 byte block transposed in words: word j collects byte j of f 2^(8 i) at byte i
    uint64_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int i = 0; i < 8; ++i) {
      for (int j = 0; j < 8; ++j) w[j] |= (uint64_t)(uint8_t)(f >> (8 * j)) << (8 * i);
      f = mul_mod(f, 256, mc);
    }
    uint8_t* at = m + (size_t)(k >> 1) * cols * 16 + (k & 1) * 8;
    for (int j = 0; j < 8; ++j) std::memcpy(at + (size_t)col(o, j) * 16, &w[j], 8);
  }
};

void build_residue(const Engine& e, int r, uint64_t pre0, uint64_t pre1, uint8_t* T) {
  const TdgtLayout& L = e.tlayout;
  const ModConst& mc = e.mconst[r];
  const uint64_t p = mc.p;
  const int Nc = 1 << L.logNc, M = L.logNc - 8, NM = 1 << M, N2 = Nc / 16;
  const bool twist = L.S == 0;
  auto mul = [&](uint64_t a, uint64_t b) { return mul_mod(a, b, mc); };
  auto pw = [&](uint64_t w) {  // powers 0 .. Nc - 1
    std::vector<uint64_t> v(Nc);
    v[0] = 1;
    for (int i = 1; i < Nc; ++i) v[i] = mul(v[i - 1], w);
    return v;
  };
  const uint64_t w = h_powmod(e.roots[r], (p - 1) / (uint64_t)Nc, p);
  const std::vector<uint64_t> W = pw(w);
  auto Wi = [&](long long x) { return W[(size_t)((Nc - x % Nc) % Nc)]; };  // w^-x
  const uint64_t s = h_powmod(e.roots[r], (p - 1) / 4, p);
  const uint64_t half = (p + 1) / 2, half_s = mul(half, h_invmod(s, p));
  // the twist root in the two factors: xi_re +- s xi_im, and their inverses' powers
  const uint64_t xr = e.xi[r].first, xs = mul(s, e.xi[r].second);
  const uint64_t xi[2] = {add_mod(xr, xs, p), sub_mod(xr, xs, p)};
  std::vector<uint64_t> X[2], Xi[2];
  for (int v = 0; v < 2; ++v) {
    X[v] = pw(twist ? xi[v] : 1);
    Xi[v] = pw(twist ? h_invmod(xi[v], p) : 1);
  }
  const uint64_t ninv = twist ? h_invmod((uint64_t)Nc, p) : 1;

  Mat fb1{T + L.f_b1, 256, mc}, fb2{T + L.f_b2, 8 * NM, mc}, fb3{T + L.f_b3, 256, mc, true};
  Mat ib1{T + L.i_b1, 256, mc}, ib3{T + L.i_b3, 256, mc};
  for (int q = 0; q < 16; ++q) {
    const int k = brev(q, 4);
    for (int n = 0; n < 16; ++n) {
      const uint64_t f = W[(size_t)(n * k % 16) * (Nc / 16)], fi = Wi((long long)(n * k % 16) * (Nc / 16));
      for (int v = 0; v < 2; ++v) {
        // forward first pass: element (n, comp) -> (q, factor v), with the twist of digit n
        const uint64_t a = mul(f, X[v][(size_t)n * N2 % Nc]);
        fb1.put(2 * q + v, 2 * n, a);
        fb1.put(2 * q + v, 2 * n + 1, v ? neg_mod(mul(a, s), p) : mul(a, s));
        // forward last pass: (n, factor v) -> element (q, comp)
        const uint64_t h = mul(f, half), hs = mul(f, half_s);
        fb3.put(2 * q, 2 * n + v, h);
        fb3.put(2 * q + 1, 2 * n + v, v ? neg_mod(hs, p) : hs);
        // inverse first pass: element (q, comp) -> (n, factor v)
        ib1.put(2 * n + v, 2 * q, fi);
        ib1.put(2 * n + v, 2 * q + 1, v ? neg_mod(mul(fi, s), p) : mul(fi, s));
        // inverse last pass: (q, factor v) -> element (n, comp), with the untwist of digit n and 1/N
        const uint64_t g = mul(mul(fi, ninv), Xi[v][(size_t)n * N2 % Nc]);
        ib3.put(2 * n, 2 * q + v, mul(g, half));
        ib3.put(2 * n + 1, 2 * q + v, v ? neg_mod(mul(g, half_s), p) : mul(g, half_s));
      }
    }
  }
  const uint64_t scale[3] = {1, pre0, pre1};
  for (int q = 0; q < NM; ++q) {
    const int k = brev(q, M);
    for (int n = 0; n < NM; ++n) {
      const size_t ex = (size_t)(n * k % NM) * (Nc / NM);
      fb2.put(q, n, W[ex]);
      for (int v = 0; v < 3; ++v) Mat{T + L.i_b2[v], 8 * NM, mc}.put(n, q, mul(Wi((long long)ex), scale[v]));
    }
  }
  auto tw = [&](uint64_t v) { return make_ulonglong2(v, mul(v, 1ull << 32)); };
  ulonglong2* f1 = reinterpret_cast<ulonglong2*>(T + L.f_t1);
  ulonglong2* i1 = reinterpret_cast<ulonglong2*>(T + L.i_t1);
  for (int q = 0; q < 16; ++q)
    for (int n2 = 0; n2 < N2; ++n2) {
      const size_t ex = (size_t)brev(q, 4) * n2 % Nc;
      for (int v = 0; v < 2; ++v) {
        f1[2 * ((size_t)q * N2 + n2) + v] = tw(mul(W[ex], X[v][n2]));
        i1[2 * ((size_t)q * N2 + n2) + v] = tw(mul(Wi((long long)ex), Xi[v][n2]));
      }
    }
  ulonglong2* f2 = reinterpret_cast<ulonglong2*>(T + L.f_t2);
  ulonglong2* i2 = reinterpret_cast<ulonglong2*>(T + L.i_t2);
  for (int q = 0; q < NM; ++q)
    for (int nl = 0; nl < 16; ++nl) {
      const size_t ex = (size_t)nl * brev(q, M) % N2 * 16;
      f2[q * 16 + nl] = tw(W[ex]);
      i2[nl * NM + q] = tw(Wi((long long)ex));
    }
}

}  // namespace

// 63-bit primes (the kernels reduce by 2^63 = c), blocks of 2^10 .. 2^13 elements; above, the main
// plan's split stage does the default 2 bits.
bool tensor_possible(const Engine& e) {
  return !e.ckks_prec && e.logN >= 10 && (e.logN <= 13 || (e.plan.S == 2 && e.plan.logNc == e.logN - 2));
}

void place_tensor_line(Engine& e) {
  // Launches of at most this many residue transforms keep the CUDA-core plans, whose small
  // launches spread one residue over several CTAs: a tensor-core unit takes 11 us however few
  // there are (22 us at N = 8192).  Forward + inverse at the line, us, CUDA cores / tensor cores:
  // nphi 2048: 288 residues 19 / 24, 384 25 / 24; 4096: 64 18 / 23, 96 22 / 23, 148 24 / 23;
  // 8192: 32 19 / 24, 64 24 / 24; 16384: 32 28 / 44, 64 43 / 44; 32768: 1 36 / 31.
  static const int above[5] = {320, 96, 64, 64, 0};
  // Rows of a work list fill a unit with residues of one prime only, load apart from each other at N = 1024, and are
  // ordered first.  Forward / inverse of the list, us, CUDA cores; tensor cores: nphi 2048: 1000 rows 24 / 25.4; 27 /
  // 25.1, 1600 37 / 39; 38 / 34, 2400 53 / 57; 57 / 50, 2800 60.5 / 63.5; 59 / 52; 4096: 140 rows 12.2 / 12.6; 13.9 /
  // 13.5, 150 14.9 / 15.3; 14.0 / 13.6; 8192: 65 rows 12.6 / 13.0; 14.1 / 14.1, 75 16.0 / 16.4; 14.2 / 14.1; 16384:
  // 65 21 / 22; 24 / 23, 75 27 / 28; 24 / 24.
  static const int list_above[4][2] = {{2600, 1150}, {148, 148}, {74, 74}, {74, 74}};
  const int at = e.logN < 10 ? 0 : (e.logN < 14 ? e.logN - 10 : 4);
  e.tensor_above = e.tensor == 2 ? 0 : above[at];
  for (int v = 0; v < 2; ++v) e.tensor_above_list[v] = e.tensor == 2 || at == 4 ? 0 : list_above[at][v];
}

// Places and fills the tensor-core tables when the engine can use them.
int build_tensor_tables(Engine& e) {
  e.tlayout = TdgtLayout{};
  if (!e.tensor || !tensor_possible(e)) return 0;
  place_tensor_line(e);
  const int logNc = e.logN <= 13 ? e.logN : e.logN - 2;
  TdgtLayout& L = e.tlayout;
  L.logNc = logNc;
  L.S = e.logN - logNc;
  const size_t Nc = (size_t)1 << logNc, NM = Nc / 256;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += (bytes + 127) & ~(size_t)127;
    return o;
  };
  L.f_b1 = take(65536);
  L.f_b2 = take(64 * NM * NM);
  L.f_b3 = take(65536);
  L.f_t1 = take(32 * Nc);
  L.f_t2 = take(Nc);
  L.i_b1 = take(65536);
  for (auto& o : L.i_b2) o = take(64 * NM * NM);
  L.i_b3 = take(65536);
  L.i_t1 = take(32 * Nc);
  L.i_t2 = take(Nc);
  L.stride = off;
  const int nres = e.k + e.kl;
  std::vector<uint64_t> pre0, pre1;
  prescale_factors(e, pre0, pre1);
  std::vector<uint8_t> host(L.stride * nres);
  struct Job {
    const Engine* e;
    const uint64_t *p0, *p1;
    uint8_t* out;
  } job{&e, pre0.data(), pre1.data(), host.data()};
  parallel_for_host(
      nres,
      [](int r, void* a) {
        const Job& j = *static_cast<Job*>(a);
        build_residue(*j.e, r, j.p0[r], j.p1[r], j.out + j.e->tlayout.stride * r);
      },
      &job);
  cudaError_t err;
  if ((err = cudaMalloc(&e.d_ttab, host.size())) != cudaSuccess) {
    set_error(std::string("cudaMalloc failed for engine tables: ") + cudaGetErrorString(err));
    return 4;
  }
  if ((err = cudaMemcpy(e.d_ttab, host.data(), host.size(), cudaMemcpyHostToDevice)) != cudaSuccess) {
    set_error(std::string("table upload failed: ") + cudaGetErrorString(err));
    return 2;
  }
  return 0;
}

}  // namespace cpoly
