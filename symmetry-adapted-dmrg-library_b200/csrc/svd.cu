// svd.cu -- one-sided (Hestenes) block Jacobi SVD of the psi sector blocks.
//
// Replaces the per-sector LAPACK gesvd of the reference
// (src/dense_inst.cpp:447-541, called from src/block_tensor_inst.cpp:535-557).
// Method: Hestenes one-sided Jacobi (Hestenes 1958; Demmel & Veselic 1992,
// with the parallel block ordering of Brent & Luk and the norm-sorted column
// order of de Rijk 1989).  The C = min(m,n) columns of W (A, or A^H when m < n)
// are ordered by decreasing norm at the start of every sweep and split into
// column blocks of b = 8 or 16 (chosen per call).  Every round of a sweep
// pairs the blocks by the circle method; one CTA forms the 2b x 2b Gram matrix
// of its pair on the FP64 tensor cores (DMMA), runs a cyclic sweep of the
// one-sided rotations on it, and applies the accumulated 2b x 2b rotation to
// the pair's columns of W and V (DMMA again).  Sweeps repeat until a full sweep
// performs no rotation, so the result keeps the columnwise relative accuracy of
// one-sided Jacobi on small singular values, which the reference's 1e-10
// relative cut-off depends on.
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.hpp"
#include "kernels.cuh"
#include "ptx.cuh"

namespace sadmrg {

constexpr int kSvdThreads = 512;
constexpr int kSvdWarps = kSvdThreads / 32;
// columns per block (a visit takes two blocks): 8 or 16, chosen per call by run_jacobi_svd

// What one CTA of the Jacobi kernel does: sectors order[j0 .. j0 + nj - 1] one after
// another, as CTA `rank` of the `size` that share each of them and barrier `group`.
struct SvdCta {
  int group, rank, size, j0, nj;
};

template <bool CPLX> struct SvdT;
template <> struct SvdT<false> { using T = double; };
template <> struct SvdT<true> { using T = double2; };

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// scalar helpers for T = double / double2 (complex)
__device__ __forceinline__ double cj_mul(double a, double b) { return a * b; }   // conj(a) b
__device__ __forceinline__ double2 cj_mul(double2 a, double2 b) {
  return make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ double cmul(double a, double b) { return a * b; }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double cadd(double a, double b) { return a + b; }
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double cconj(double a) { return a; }
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double cre(double a) { return a; }
__device__ __forceinline__ double cre(double2 a) { return a.x; }
__device__ __forceinline__ double cim(double) { return 0.0; }
__device__ __forceinline__ double cim(double2 a) { return a.y; }
template <class T> __device__ __forceinline__ T czero();
template <> __device__ __forceinline__ double czero<double>() { return 0.0; }
template <> __device__ __forceinline__ double2 czero<double2>() { return make_double2(0.0, 0.0); }

// D (8 x 8) += A (8 x 4, row-major) B (4 x 8, col-major) on the FP64 tensor cores.
// Lane l holds A(l / 4, l % 4), B(l % 4, l / 4) and D(l / 4, 2 (l % 4) + i), i = 0, 1.
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// 2^-k for a normal double m = 2^k (1 + f): m times it lies in [1, 2) (built from the
// exponent bits, exact)
__device__ __forceinline__ double pow2_scale_of(double m) {
  const int e = (__double2hiint(m) >> 20) & 0x7ff;
  return __hiloint2double((2046 - e) << 20, 0);
}
// The one-sided rotation of a pair with squared norms a, b and |<w_p, w_q>| = g > 0,
// as on the columns themselves: t = tan(theta) = 2 g sgn(d) / (|d| + r) with d = b - a,
// r = sqrt(d^2 + 4 g^2).  With u = |d| + r and q = 1 / sqrt(2 r u) (since
// 1 + t^2 = 2 r / u): c = cos(theta) = u q, s = sin(theta) = 2 g q sgn(d) and
// t = 4 g r q^2 sgn(d) -- two inverse square roots and no division on the chain
// that sets the time of an inner round.  d and g are first scaled by a power of two,
// so that the squares neither overflow nor underflow; c, s and t do not depend on the
// scale.  The scale takes the larger of a and b, which bounds |d| and (up to rounding) g,
// into [1, 2): known before g is.  Returns c, s sgn (sgn = 1 or -1) and t g.
__device__ __forceinline__ void jacobi_rotation(double a, double b, double g, double sgn, double& c, double& s,
                                                double& tg) {
  const double d = b - a, sc = pow2_scale_of(fmax(a, b)), sd = d >= 0.0 ? 1.0 : -1.0;
  const double dn = fabs(d) * sc, h = g * (2.0 * sc);
  const double x = fma(dn, dn, __dmul_rn(h, h));
  const double r = __dmul_rn(x, rsqrt(x));
  const double u = __dadd_rn(dn, r);
  const double q = rsqrt(__dmul_rn(2.0 * r, u));
  c = u * q;
  s = (sd * sgn * h) * q;
  tg = (2.0 * h * r * q * q) * (sd * g);
}

constexpr int kChunk = 128;            // rows per streamed chunk of W

template <bool CPLX, int B>            // B: columns per block
struct SvdGeom {
  static constexpr int Nc = 2 * B;                          // columns of one visit
  static constexpr int TD = Nc / 8;                         // 8 x 8 DMMA tiles along one side of G
  // strides in shared memory, in elements, are 32 bytes past a multiple of 128: the four
  // rows and four columns that half a warp reads of a DMMA fragment then lie in different
  // banks (at Nc + 1 the Gram of a 128-row chunk took 5,200 cycles, four times its mma)
  static constexpr int Pad = CPLX ? 2 : 4;
  static constexpr int Ld = Nc + Pad;                       // rows of G, columns of Q
  static constexpr int LdC = kChunk + Pad;                  // columns of a row chunk of W
  // columns of all rows of W or V (a resident visit)
  __host__ __device__ static constexpr int ldr(int rows) { return ((rows + 15) & ~15) + Pad; }
  static constexpr int Split = B == 8 ? 4 : 1;              // row parts of a resident visit's Gram
  static constexpr int TU = TD * (TD + 1) / 2;              // tiles on and above the diagonal
  static constexpr int Units = B == 8 ? 1 : 4;              // of a streamed one: GramUnit
  // threads of the inner sweep: a deciding warp, one thread per 2 x 2 block of G, and
  // those that rotate Q
  static constexpr int GT = B * B, QT = B == 8 ? 64 : 128;
  static constexpr int IT = 32 + GT + QT;
  static_assert(IT <= kSvdThreads && GT % 32 == 0 && QT % Nc == 0, "threads of a visit");
};

template <bool CPLX, int B>
constexpr size_t svd_smem_bytes() {   // G twice, Q and two row-chunk buffers
  using Gm = SvdGeom<CPLX, B>;
  return (size_t)(3 * Gm::Ld + 2 * Gm::LdC) * Gm::Nc * (CPLX ? 16 : 8);
}
// shared memory of a resident visit (all rows of the pair's W and V columns) of an
// R x C block; launches whose largest pair needs more stream row chunks instead
template <bool CPLX, int B>
constexpr size_t svd_res_smem_bytes(int R, int C) {
  using Gm = SvdGeom<CPLX, B>;
  return (size_t)(3 * Gm::Ld + Gm::ldr(R) + Gm::ldr(C)) * Gm::Nc * (CPLX ? 16 : 8) + (size_t)kSvdWarps * 32 * 4 * 8;
}
constexpr size_t kSvdResMax = 188 * 1024;

// Tiles of G on and above the diagonal that one warp forms, from the fragments of nl
// column groups of 8: tile t is between the groups l[x[t]] and l[y[t]] (l, x and y are
// lists of digits, the first lowest).  Of 4 groups
// (B = 16) by four warps, of 2 (B = 8) by one as the last two of 4: 10 fragments for 10
// mma instead of 20, which took as long as the mma.
template <int U> struct GramUnit;
__device__ constexpr int digit(int list, int i) { return list >> 4 * i & 15; }
template <> struct GramUnit<0> { static constexpr int nl = 2, nt = 2, l = 0x10, x = 0x00, y = 0x10; };
template <> struct GramUnit<1> { static constexpr int nl = 3, nt = 2, l = 0x320, x = 0x00, y = 0x21; };
template <> struct GramUnit<2> { static constexpr int nl = 3, nt = 3, l = 0x321, x = 0x000, y = 0x210; };
template <> struct GramUnit<3> { static constexpr int nl = 2, nt = 3, l = 0x32, x = 0x100, y = 0x110; };

__device__ __forceinline__ void gram_mma(double* g, double x, double y) { dmma(g[0], g[1], x, y); }
__device__ __forceinline__ void gram_mma(double* g, double2 x, double2 y) {   // conj(x) y
  dmma(g[0], g[1], x.x, y.x);
  dmma(g[0], g[1], x.y, y.y);
  dmma(g[2], g[3], x.x, y.y);
  dmma(g[2], g[3], -x.y, y.x);
}
// g[t] += tiles of unit U over the k steps k0, k0 + STEP, ... < k1 of four rows each, of
// columns at D (column-major, stride ldd; D points to this lane's row and column)
template <int U, int TD, int STEP, class T, int NG>
__device__ __forceinline__ void gram_unit(const T* D, int ldd, int k0, int k1, double (&g)[3][NG]) {
  using Un = GramUnit<U>;
#pragma unroll 4
  for (int k = k0; k < k1; k += STEP) {
    T f[Un::nl];
#pragma unroll
    for (int i = 0; i < Un::nl; ++i) f[i] = D[(digit(Un::l, i) - 4 + TD) * 8 * ldd + k];
#pragma unroll
    for (int t = 0; t < Un::nt; ++t) gram_mma(g[t], f[digit(Un::x, t)], f[digit(Un::y, t)]);
  }
}
template <int TD, int STEP, class T, int NG>
__device__ __forceinline__ void gram_any(int unit, const T* D, int ldd, int k0, int k1, double (&g)[3][NG]) {
  if constexpr (TD == 2) {
    gram_unit<3, TD, STEP>(D, ldd, k0, k1, g);
  } else {
    if (unit == 0) gram_unit<0, TD, STEP>(D, ldd, k0, k1, g);
    else if (unit == 1) gram_unit<1, TD, STEP>(D, ldd, k0, k1, g);
    else if (unit == 2) gram_unit<2, TD, STEP>(D, ldd, k0, k1, g);
    else gram_unit<3, TD, STEP>(D, ldd, k0, k1, g);
  }
}

template <int U, int TD, class F, int NG>
__device__ __forceinline__ void gram_unit_tiles(F f, const double (&g)[3][NG]) {
  using Un = GramUnit<U>;
#pragma unroll
  for (int t = 0; t < Un::nt; ++t)
    f(digit(Un::l, digit(Un::x, t)) - 4 + TD, digit(Un::l, digit(Un::y, t)) - 4 + TD, g[t]);
}
// f(row tile, column tile, sums) for the tiles of a unit
template <int TD, class F, int NG>
__device__ __forceinline__ void gram_tiles(int unit, F f, const double (&g)[3][NG]) {
  if (TD == 2 || unit == 3) gram_unit_tiles<3, TD>(f, g);
  else if (unit == 0) gram_unit_tiles<0, TD>(f, g);
  else if (unit == 1) gram_unit_tiles<1, TD>(f, g);
  else gram_unit_tiles<2, TD>(f, g);
}

// A pair's rotation, c and s e^{i phi} (on = 0: none).
struct SvdRot {
  double c, sr, si;
  int on;
};
// Columns x, y <- c x - conj(s) y, s x + c y.  The real form names its roundings: the
// signs of singular vectors of blocks of about 1,400 columns depend on each.
__device__ __forceinline__ void rot_cols(double& x, double& y, const SvdRot& t) {
  const double u = x, v = y;
  x = __fma_rn(t.c, u, -__dmul_rn(t.sr, v));
  y = __fma_rn(t.sr, u, __dmul_rn(t.c, v));
}
__device__ __forceinline__ void rot_cols(double2& x, double2& y, const SvdRot& t) {
  const double2 u = x, v = y, ep = make_double2(t.sr, t.si), em = make_double2(-t.sr, t.si);
  x = cadd(make_double2(t.c * u.x, t.c * u.y), cmul(v, em));
  y = cadd(cmul(u, ep), make_double2(t.c * v.x, t.c * v.y));
}
// rows x, y <- c x - s y, conj(s) x + c y
__device__ __forceinline__ void rot_rows(double& x, double& y, const SvdRot& t) { rot_cols(x, y, t); }
__device__ __forceinline__ void rot_rows(double2& x, double2& y, const SvdRot& t) {
  const double2 u = x, v = y, mp = make_double2(-t.sr, -t.si), pm = make_double2(t.sr, -t.si);
  x = cadd(make_double2(t.c * u.x, t.c * u.y), cmul(mp, v));
  y = cadd(cmul(pm, u), make_double2(t.c * v.x, t.c * v.y));
}
// the first or second of the two that rot_cols (row = 0) or rot_rows (row = 1) returns
__device__ __forceinline__ double rot_one(double u, double v, const SvdRot& t, bool second, int) {
  const double a = second ? t.sr : t.c, b = second ? t.c : -t.sr;
  const double w = __fma_rn(a, u, __dmul_rn(b, v));
  return t.on ? w : second ? v : u;
}
__device__ __forceinline__ double2 rot_one(double2 u, double2 v, const SvdRot& t, bool second, int row) {
  double2 x = u, y = v;
  if (row) rot_rows(x, y, t);
  else rot_cols(x, y, t);
  return second ? (t.on ? y : v) : (t.on ? x : u);
}

// A pair of a round: its columns p < q (p + 256 q) and the 2 x 2 block of the round
// before that its G_pq comes from: rows of pair i, columns of pair j (j + 256 i), p and q
// being the second of them (+ 32768, + 128), and the offsets of its entries in G.
struct alignas(16) SvdLook {
  unsigned short o00, o01, o10, o11, pq, ij;
};

template <class P>
__device__ __forceinline__ void swap_ptr(P*& a, P*& b) { P* const t = a; a = b; b = t; }

// pair k of round rnd of the circle method over N (even) columns, p < q
__device__ __forceinline__ void circle_pair(int N, int rnd, int k, int& p, int& q) {
  int u = rnd + k, v = k == 0 ? N - 1 : rnd - k;
  if (u >= N - 1) u -= N - 1;
  if (v < 0) v += N - 1;
  p = min(u, v);
  q = max(u, v);
}

// One visit of a column-block pair (Hestenes one-sided Jacobi in Gram form):
//   1. G = Wp^H Wp for the pair's nc <= 2B columns Wp;
//   2. cyclic one-sided Jacobi on G: rotation (p, q) from a = G_pp, b = G_qq,
//      g = G_pq exactly as on the columns themselves, G <- J^H G J, Q <- Q J,
//      with the rotated diagonal set to a - t|g|, b + t|g| and G_pq to 0 (one sweep:
//      more cut the outer sweeps by less than they cost);
//   3. Wp <- Wp Q and Vp <- Vp Q.
// The rotations rotate the Gram entries of the columns exactly as the column updates
// would (a rotation that mixes a small column with a large one has |s| <=
// sqrt(a_small / a_large)), so the entries keep the columnwise relative accuracy of the
// direct method; W itself changes only by the orthogonal Q.  Adds the number of
// rotations to *rotations.  Every thread of the block calls it.
//
// The Gram and the application of Q run on the FP64 tensor cores.  When the launch's
// largest pair fits in shared memory (RES) the pair's W columns are read there first and
// its V columns by idle warps during part 2; otherwise half of the warps read W in row
// chunks while the others form the Gram, and the application reads its fragments straight
// from L2.  Only the Gram tiles on and above the diagonal are formed, and new columns go
// from registers to memory.
//
// Part 2 is a chain of Nc - 1 rounds and the longest part of a resident visit: a load of
// the deciding entries, two inverse square roots and a barrier.  One warp computes the
// rotations and runs a round ahead: the entry G_pq that decides a pair of the next round
// comes from one 2 x 2 block of G and two rotations of this round, so it computes that
// entry itself (SvdLook) while others, one thread per 2 x 2 block, write the rotated G to
// a second copy and others again rotate Q.  The deciding warp passes alone over rounds in
// which no pair rotates.  950 cycles a round (b = 8) and 1,130 (b = 16), after 1,300 with
// the test, the rotations and the rotation of G one after another.
//
// Cycles of a visit, real: b = 8, 344 x 344 (D = 512): load 1,340, Gram 2,350, part 2
// 14,000, part 3 5,200, between visits 5,000: 4.6 ms of Jacobi after 7.8; b = 16,
// 1,319 x 1,319 (D = 2,048): Gram 32,600, part 2 35,000, part 3 63,600 (44,000 of mma),
// between visits 11,500: 46.9 ms after 115.
//
// The sums run in a fixed order: of a resident visit's Gram in kSplit row parts of one
// chain each, of a streamed one over even and odd k steps apart.  With blocks of about
// 1,400 columns the signs of singular vectors depend on every rounding, so the orders
// are part of the result.
template <bool CPLX, int B, bool RES>
__device__ __forceinline__ void jacobi_pair_visit(typename SvdT<CPLX>::T* W, int R, typename SvdT<CPLX>::T* V, int C, const int* cols,
                                  int nc, double tol, unsigned char* smem_raw, SvdLook (*looks)[B], int& looks_n, int* rotations) {
  using T = typename SvdT<CPLX>::T;
  using Gm = SvdGeom<CPLX, B>;
  constexpr int kNc = Gm::Nc, kTD = Gm::TD, kLdG = Gm::Ld, kTU = Gm::TU, kSplit = Gm::Split, kUnits = Gm::Units;
  constexpr int kE = CPLX ? 4 : 2;
  __shared__ double dg[kNc];             // the diagonal of G
  // by pair of the round: its rotation, its columns p < q as p + 256 q + 65536 on
  __shared__ double par_c[2][B], par_sr[2][B], par_si[2][CPLX ? B : 1];
  __shared__ int par_pq[2][B];
  __shared__ int msg[2];                 // 1: par holds rotations (2: the last), 0: it holds none, -1: end
  __shared__ int nrot_sh;
  T* G = reinterpret_cast<T*>(smem_raw); // kNc x kLdG, row-major
  T* G2 = G + kNc * kLdG;                // the other copy of G
  T* Q = G2 + kNc * kLdG;                // kNc x kLdG, column-major
  T* Ck = Q + kNc * kLdG;                // two row chunks of W, column-major
  // resident visit: all R rows of the pair's W columns, then all C rows of its V columns
  const int ldw = Gm::ldr(R), ldv = Gm::ldr(C);
  T* Ws = Ck;
  T* Vs = Ws + kNc * ldw;
  double* Gp = reinterpret_cast<double*>(Vs + kNc * ldv);   // Gram partials, 4 per lane per warp
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // Rows r0, r0 + 32, ... of column c of M (zeros past the column or past nc): read
  // together, so that a thread's loads are in flight at once (cp.async of 8 bytes
  // passed at 12 bytes a cycle: 7,500 cycles for 350 rows of W and V)
  auto load = [&](const T* M, int ld, int c, int r0, auto& v) {
    const T* src = M + (long long)cols[min(c, nc - 1)] * ld;
#pragma unroll
    for (int u = 0; u < (int)(sizeof(v) / sizeof(T)); ++u)
      v[u] = c < nc && r0 + u * 32 < ld ? __ldcg(src + r0 + u * 32) : czero<T>();
  };
  // all rows of the columns of M, and zeros to a multiple of four, by nw warps
  auto load_all = [&](const T* M, int ld, T* dst, int ldd, int w, int nw) {
    T v[CPLX ? 6 : 12];
    const int ldz = (ld + 3) & ~3;
    constexpr int kU = sizeof(v) / sizeof(T);
    for (int c = w; c < kNc; c += nw)
      for (int r0 = lane; r0 < ldz; r0 += 32 * kU) {
        load(M, ld, c, r0, v);
#pragma unroll
        for (int u = 0; u < kU; ++u)
          if (r0 + u * 32 < ldz) dst[c * ldd + r0 + u * 32] = v[u];
      }
  };

  // 1. Gram matrix
  const int fr = lane >> 2, fk = lane & 3;
  // tiles of this warp, a resident visit: one in one part of the rows; streamed: GramUnit
  double g[RES ? 1 : 3][kE] = {};   // Re (and Im) of D(fr, 2 fk + i)
  int pt = 0, qt = 0, unit = warp % kUnits;
  bool gram_warp = warp < (RES ? kTU : kUnits);   // of which the tiles are stored
  if constexpr (RES) {
    load_all(W, R, Ws, ldw, warp, kSvdWarps);
    qt = warp % kTU;
    while (qt >= kTD - pt) { qt -= kTD - pt; ++pt; }
    qt += pt;
    const int part = warp / kTU;
    __syncthreads();
    if (part < kSplit) {
      const int rs = (((R + kSplit - 1) / kSplit) + 3) & ~3;
      const int k0s = part * rs, k1s = min(R, k0s + rs);
      const T* xa = Ws + (pt * 8 + fr) * ldw + fk;   // A(p, r) = conj(W(r, p))
      const T* yb = Ws + (qt * 8 + fr) * ldw + fk;   // B(r, q) = W(r, q)
#pragma unroll 4
      for (int k0 = k0s; k0 < k1s; k0 += 4) gram_mma(g[0], xa[k0], yb[k0]);
    }
    if constexpr (kSplit > 1) {
      if (part > 0 && part < kSplit)
#pragma unroll
        for (int e = 0; e < kE; ++e) Gp[(warp * kE + e) * 32 + lane] = g[0][e];
      __syncthreads();
      if (part == 0)
        for (int pp = 1; pp < kSplit; ++pp)
#pragma unroll
          for (int e = 0; e < kE; ++e) g[0][e] += Gp[((warp + pp * kTU) * kE + e) * 32 + lane];
    }
  } else {
    // Row chunks of W in two shared buffers: half of the warps read the next chunk while
    // the first 2 kUnits multiply one, even and odd k steps apart (units so that each
    // quarter of the SM gets as many mma)
    const bool loads = warp >= kSvdWarps / 2;
    const int odd = warp / kUnits;
    if (odd == 1) unit = (warp + 2) % kUnits;
    const int nch = (R + kChunk - 1) / kChunk;
    for (int ch = -1; ch < nch; ++ch) {
      if (loads && ch + 1 < nch) {
        constexpr int kCols = kNc / (kSvdWarps / 2), kAt = CPLX ? 1 : kCols;
        T* Cn = Ck + ((ch + 1) & 1) * kNc * Gm::LdC + lane;
        for (int i0 = 0; i0 < kCols; i0 += kAt) {
          T v[kAt][kChunk / 32];
#pragma unroll
          for (int i = 0; i < kAt; ++i) load(W, R, warp - kSvdWarps / 2 + (i0 + i) * (kSvdWarps / 2), (ch + 1) * kChunk + lane, v[i]);
#pragma unroll
          for (int i = 0; i < kAt; ++i)
#pragma unroll
            for (int u = 0; u < kChunk / 32; ++u)
              Cn[(warp - kSvdWarps / 2 + (i0 + i) * (kSvdWarps / 2)) * Gm::LdC + u * 32] = v[i][u];
        }
      } else if (odd < 2 && ch >= 0) {
        const int kend = min(kChunk, (R - ch * kChunk + 7) & ~7);   // zero rows beyond add nothing
        gram_any<kTD, 8>(unit, Ck + (ch & 1) * kNc * Gm::LdC + fr * Gm::LdC + fk, Gm::LdC, odd * 4, kend, g);
      }
      __syncthreads();
    }
    double* sums = reinterpret_cast<double*>(Ck);   // of the odd steps
    if (odd == 1)
#pragma unroll
      for (int t = 0; t < 3; ++t)
#pragma unroll
        for (int e = 0; e < kE; ++e) sums[((unit * 3 + t) * kE + e) * 32 + lane] = g[t][e];
    __syncthreads();
    if (gram_warp)
#pragma unroll
      for (int t = 0; t < 3; ++t)
#pragma unroll
        for (int e = 0; e < kE; ++e) g[t][e] += sums[((unit * 3 + t) * kE + e) * 32 + lane];
  }
  // stored from the tiles on and above the diagonal, mirrored, so that G is exactly Hermitian
  auto store = [&](int pt, int qt, const double* d) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int p = pt * 8 + fr, q = qt * 8 + 2 * fk + i;
      if (p > q) continue;
      T v;
      if constexpr (CPLX) v = make_double2(d[i], d[2 + i]);
      else v = d[i];
      if (p == q) {
        dg[p] = cre(v);
      } else {
        G[p * kLdG + q] = v;
        G[q * kLdG + p] = cconj(v);
      }
    }
  };
  if (gram_warp) {
    if constexpr (RES) store(pt, qt, g[0]);
    else gram_tiles<kTD>(unit, store, g);
  }
  for (int e = tid; e < kNc * kNc; e += kSvdThreads) {
    const int r = e / kNc, c = e % kNc;
    Q[r * kLdG + c] = czero<T>();
    if (r == c) reinterpret_cast<double*>(Q + r * kLdG + c)[0] = 1.0;
  }
  __syncthreads();

  // the rounds over N columns, made when N changes (the last block of a sector is narrower)
  const int N = nc + (nc & 1), np = N / 2;
  if (N != looks_n)
    for (int e = tid; e < (N - 1) * np; e += kSvdThreads) {
      const int rnd = e / np, k = e % np;
      // columns rnd + k and rnd - k were in pairs k + 1 and k - 1 of the round before
      const int pu = min(k + 1, np - 1), pv = max(k - 1, 0);
      int p, q, p0, p1, q0, q1;
      circle_pair(N, rnd, k, p, q);
      const bool uv = p == (rnd + k >= N - 1 ? rnd + k - (N - 1) : rnd + k);
      const int i = uv ? pu : pv, j = uv ? pv : pu;
      circle_pair(N, max(rnd - 1, 0), i, p0, p1);
      circle_pair(N, max(rnd - 1, 0), j, q0, q1);
      SvdLook L;
      L.pq = (unsigned short)(p + 256 * q);
      L.ij = (unsigned short)(j + 256 * i + (p == p1 ? 32768 : 0) + (q == q1 ? 128 : 0));
      L.o00 = (unsigned short)(p0 * kLdG + q0);
      L.o01 = (unsigned short)(p0 * kLdG + q1);
      L.o10 = (unsigned short)(p1 * kLdG + q0);
      L.o11 = (unsigned short)(p1 * kLdG + q1);
      looks[rnd][k] = L;
    }
  // a pair that needs no rotation on the fresh G keeps the inner sweep from
  // rotating at all: skip the visit when no pair of it does
  {
    int need = 0;
    for (int e = tid; e < kNc * kNc; e += kSvdThreads) {
      const int p = e / kNc, q = e % kNc;
      if (p >= q || q >= nc) continue;
      const double ab = dg[p] * dg[q];
      const T gpq = G[p * kLdG + q];
      double g2;
      if constexpr (CPLX) g2 = gpq.x * gpq.x + gpq.y * gpq.y; else g2 = gpq * gpq;
      if (ab > 0.0 && g2 > tol * tol * ab) need = 1;
    }
    const int any = __syncthreads_or(need);
    if (tid == 0) looks_n = N;
    if (!any) return;
  }

  // 2. the inner sweep on G
  constexpr int GT = Gm::GT;
  auto sync = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(Gm::IT) : "memory"); };
  auto rot_of = [&](int buf, int pair) {
    SvdRot t;
    t.c = par_c[buf][pair];
    t.sr = par_sr[buf][pair];
    t.si = CPLX ? par_si[buf][pair] : 0.0;
    t.on = par_pq[buf][pair] >> 16;
    return t;
  };
  if (warp == 0) {
    // lane k decides pair k of a round.  ahead: the others are still applying the
    // rotations par[buf] of the round before to Gc, else Gc is as it should be.
    T* Gc = G;
    T* Gn = G2;
    int nrot = 0, buf = 0;
    bool ahead = false;
    const int k = min(lane, np - 1);
    SvdLook L = looks[0][k];
    int pp = 0, pq = 0;             // the last rotation's columns and their new diagonal,
    double pa = 0.0, pb = 0.0;      // stored while the next G_pq is on its way
    bool pend = false;
    for (int rnd = 0; rnd < N - 1; ++rnd) {
      T b00, b01, b10, b11;
      SvdRot ri, rj;
      const int p = L.pq & 255, q = L.pq >> 8 & 255;
      const bool p_second = L.ij & 32768, q_second = L.ij & 128;
      if (ahead) {
        b00 = Gc[L.o00];
        b01 = Gc[L.o01];
        b10 = Gc[L.o10];
        b11 = Gc[L.o11];
        ri = rot_of(buf, L.ij >> 8 & 127);
        rj = rot_of(buf, L.ij & 127);
      } else {
        b00 = Gc[p * kLdG + q];
      }
      L = looks[min(rnd + 1, N - 2)][k];
      if (pend) {
        dg[pp] = pa;
        dg[pq] = pb;
      }
      __syncwarp();
      const double a = dg[p], b = dg[q];
      T gpq = b00;
      if (ahead)
        gpq = rot_one(rot_one(b00, b01, rj, q_second, 0), rot_one(b10, b11, rj, q_second, 0), ri, p_second, 1);
      const double gr = cre(gpq), gi = cim(gpq);
      const double g2 = gr * gr + gi * gi;
      // rotate when |g| > tol sqrt(ab), compared squared
      const bool act = lane < np && q < nc && a * b > 0.0 && g2 > tol * tol * (a * b);
      // the rotation before the test's outcome is known (unused where !act)
      double c, sr, si = 0.0, tg;
      if constexpr (CPLX) {
        const double gn = sqrt(g2);
        const double ig = 1.0 / gn;
        double sn;
        jacobi_rotation(a, b, gn, 1.0, c, sn, tg);
        sr = sn * (gr * ig);
        si = sn * (gi * ig);
      } else {
        jacobi_rotation(a, b, fabs(gr), gr >= 0.0 ? 1.0 : -1.0, c, sr, tg);
      }
      const unsigned on = __ballot_sync(0xffffffffu, act);
      pend = act;
      if (on == 0) {
        if (ahead) {              // let the others finish the round before
          buf ^= 1;
          if (lane == 0) msg[buf] = 0;
          sync();
          swap_ptr(Gc, Gn);
          ahead = false;
        }
        continue;
      }
      if (ahead) swap_ptr(Gc, Gn);
      buf ^= 1;
      ahead = true;
      if (lane < np) {
        par_c[buf][lane] = c;
        par_sr[buf][lane] = sr;
        if constexpr (CPLX) par_si[buf][lane] = si;
        par_pq[buf][lane] = p + 256 * q + (act ? 65536 : 0);
      }
      if (lane == 0) msg[buf] = rnd == N - 2 ? 2 : 1;
      sync();
      pp = p;                     // the rotated 2 x 2 block is set to its exact values
      pq = q;
      pa = __dsub_rn(a, tg);
      pb = __dadd_rn(b, tg);
      nrot += __popc(on);
    }
    if (lane == 0) {
      msg[buf ^ 1] = -1;
      nrot_sh = nrot;
    }
    sync();
  } else if (tid < 32 + GT) {
    const int e = tid - 32, bi = e / np, bj = e % np;   // rows of pair bi, columns of pair bj
    T* Gc = G;
    T* Gn = G2;
    for (int buf = 1;; buf ^= 1) {
      sync();
      const int m = msg[buf];
      if (m < 0) break;
      if (m != 1 || bi >= np) continue;   // (nobody reads G after the last round)
      const int pi = par_pq[buf][bi], pj = par_pq[buf][bj];
      const SvdRot ri = rot_of(buf, bi), rj = rot_of(buf, bj);
      const int r0 = (pi & 255) * kLdG, r1 = (pi >> 8 & 255) * kLdG, q0 = pj & 255, q1 = pj >> 8 & 255;
      if (bi != bj) {
        T b00 = Gc[r0 + q0], b01 = Gc[r0 + q1], b10 = Gc[r1 + q0], b11 = Gc[r1 + q1];
        if (rj.on) {   // columns: [x y] <- [x y] [[c, s e^{i phi}], [-s e^{-i phi}, c]]
          rot_cols(b00, b01, rj);
          rot_cols(b10, b11, rj);
        }
        if (ri.on) {   // rows: G <- J^H G
          rot_rows(b00, b10, ri);
          rot_rows(b01, b11, ri);
        }
        Gn[r0 + q0] = b00;
        Gn[r0 + q1] = b01;
        Gn[r1 + q0] = b10;
        Gn[r1 + q1] = b11;
      } else {
        Gn[r0 + q1] = ri.on ? czero<T>() : Gc[r0 + q1];
        Gn[r1 + q0] = ri.on ? czero<T>() : Gc[r1 + q0];
      }
      swap_ptr(Gc, Gn);
    }
  } else if (tid < Gm::IT) {
    constexpr int kG = Gm::QT / kNc, kU = B / kG;   // pairs at a time, and in turn
    const int t = tid - 32 - GT;
    T* const Qr = Q + t % kNc;                      // row t % kNc of Q
    for (int buf = 1;; buf ^= 1) {
      sync();
      const int m = msg[buf];
      if (m < 0) break;
      if (m == 0) continue;
      T x[kU], y[kU];
      int pq[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int k = t / kNc + u * kG;
        pq[u] = k < np ? par_pq[buf][k] : 0;
        x[u] = Qr[(pq[u] & 255) * kLdG];
        y[u] = Qr[(pq[u] >> 8 & 255) * kLdG];
      }
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        const int k = t / kNc + u * kG;
        if (k >= np) continue;
        if (!(pq[u] >> 16)) continue;
        rot_cols(x[u], y[u], rot_of(buf, k));
        Qr[(pq[u] & 255) * kLdG] = x[u];
        Qr[(pq[u] >> 8 & 255) * kLdG] = y[u];
      }
    }
  }
  if (RES && tid >= Gm::IT) load_all(V, C, Vs, ldv, warp - Gm::IT / 32, kSvdWarps - Gm::IT / 32);
  __syncthreads();
  const int nrot = nrot_sh;
  if (nrot == 0) return;        // nothing moved: W and V stay as they are

  // 3. Wp <- Wp Q and Vp <- Vp Q: each warp takes RT 8-row tiles of W, then of V, at a
  //    time, reads them whole (from shared memory: the next on their way) and writes their
  //    new columns
  const int ntw = (R + 7) / 8, nt = ntw + (C + 7) / 8;
  constexpr int RT = CPLX || RES ? 1 : 2;
  T x[RT][kNc / 4], xn[RES ? kNc / 4 : 1];
  auto next = [&](int t) {
    const bool isw = t < ntw;
    const int r = (isw ? t : t - ntw) * 8 + fr, lds = isw ? ldw : ldv;
    const bool in = t < nt && r < (isw ? R : C);
    const T* sm = (isw ? Ws : Vs) + r + fk * lds;
#pragma unroll
    for (int k = 0; k < kNc / 4; ++k) xn[k] = in ? sm[k * 4 * lds] : czero<T>();
  };
  if constexpr (RES) next(warp);
  for (int t0 = warp * RT; t0 < nt; t0 += kSvdWarps * RT) {
    T* base[RT];
    int ld[RT];
    bool in[RT];
#pragma unroll
    for (int u = 0; u < RT; ++u) {
      const int t = t0 + u;
      const bool isw = t < ntw;
      const int r = (isw ? t : t - ntw) * 8 + fr;
      ld[u] = isw ? R : C;
      base[u] = (isw ? W : V) + r;
      in[u] = t < nt && r < ld[u];
      if constexpr (RES) {
#pragma unroll
        for (int k = 0; k < kNc / 4; ++k) x[u][k] = xn[k];
        next(t + kSvdWarps);
      } else {
#pragma unroll
        for (int k = 0; k < kNc / 4; ++k)
          x[u][k] = in[u] && k * 4 + fk < nc ? __ldcg(base[u] + (long long)cols[k * 4 + fk] * ld[u]) : czero<T>();
      }
    }
    double acc[RT][kTD][kE] = {};
#pragma unroll
    for (int k = 0; k < kNc / 4; ++k)
#pragma unroll
      for (int j = 0; j < kTD; ++j) {
        const T y = Q[(j * 8 + fr) * kLdG + k * 4 + fk];
#pragma unroll
        for (int u = 0; u < RT; ++u) {
          if constexpr (CPLX) {
            dmma(acc[u][j][0], acc[u][j][1], x[u][k].x, y.x);
            dmma(acc[u][j][0], acc[u][j][1], -x[u][k].y, y.y);
            dmma(acc[u][j][2], acc[u][j][3], x[u][k].x, y.y);
            dmma(acc[u][j][2], acc[u][j][3], x[u][k].y, y.x);
          } else {
            dmma(acc[u][j][0], acc[u][j][1], x[u][k], y);
          }
        }
      }
#pragma unroll
    for (int u = 0; u < RT; ++u) {
      if (!in[u]) continue;
#pragma unroll
      for (int j = 0; j < kTD; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c = j * 8 + 2 * fk + e;
          T v;
          if constexpr (CPLX) v = make_double2(acc[u][j][e], acc[u][j][2 + e]);
          else v = acc[u][j][e];
          if (c < nc) base[u][(long long)cols[c] * ld[u]] = v;
        }
    }
  }
  if (tid == 0) atomicAdd(rotations, nrot);
}

constexpr unsigned long long kSvdBarrierNs = 2000000000ull;

struct SvdCtl {
  unsigned count;             // of the QR kernels' barrier
  int status;                 // 0, or 1 when a barrier ran out of time
  int sweeps, failed;         // sweeps taken; 1 when max_sweeps was reached
  unsigned long long t0, t1;  // device clock (ns) at the start and end of block 0
};

__device__ __forceinline__ unsigned long long svd_gtime() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Barrier of `size` CTAs (those that share a sector, or all): *count grows by one per CTA
// and phase.
// Returns false when it ran out of time.
__device__ bool svd_group_sync(unsigned* count, int size, unsigned& phase, SvdCtl* ctl) {
  __shared__ int ok_sh;
  __syncthreads();
  if (size == 1) return true;
  ++phase;
  if (threadIdx.x == 0) {
    ok_sh = 1;
    __threadfence();
    atomicAdd(count, 1u);
    const unsigned want = phase * (unsigned)size;
    const volatile unsigned* seen = count;
    const unsigned long long t0 = svd_gtime();
    for (long long it = 0; (int)(*seen - want) < 0; ++it) {
      if (it > (1ll << 30) || ((it & 255) == 255 && svd_gtime() - t0 > kSvdBarrierNs)) {
        ok_sh = 0;
        atomicExch(&ctl->status, 1);
        break;
      }
      if (it > 16) __nanosleep(32);
    }
    __threadfence();
  }
  __syncthreads();
  return ok_sh != 0;
}

// All sweeps of all sectors in one cooperative launch.  Sectors are independent: each
// has its own CTAs (SvdCta), its own barrier between rounds and its own end, so a round
// of a narrow sector doesn't wait for the visits of the widest one (with one barrier
// for all, waiting took 39,000 of 190,000 cycles a round at D = 2048; with its own
// 11,500).  Rotations are counted in three rotating counter sets (sweep s adds into set s % 3; the set of sweep s + 1 is
// cleared during sweep s, when nobody reads it any more); every CTA of a sector takes
// the same decisions from the same counts, read after the barrier that ends the sweep.
template <bool CPLX, int B, bool RES>
__global__ void __launch_bounds__(kSvdThreads) jacobi_coop_kernel(const SvdJob* __restrict__ jobs, int nj,
                                                                  const SvdCta* __restrict__ ctas,
                                                                  const int* __restrict__ order, unsigned* bars,
                                                                  void* work, void* vmat, double* nrm, int* perm,
                                                                  double tol, int* cnt, SvdCtl* ctl, int max_sweeps) {
  using T = typename SvdT<CPLX>::T;
  constexpr int kNc = SvdGeom<CPLX, B>::Nc;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int cols[kNc];
  __shared__ SvdLook looks[2 * B - 1][B];   // the rounds over looks_n columns
  __shared__ int looks_n;
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) {
    looks_n = 0;
    atomicMin(&ctl->t0, svd_gtime());
  }
  const SvdCta me = ctas[blockIdx.x];
  unsigned* bar = bars + me.group * 32;
  unsigned phase = 0;
  for (int jj = 0; jj < me.nj; ++jj) {
    const int j = order[me.j0 + jj];
    const SvdJob J = jobs[j];
    const int R = J.trans ? J.n : J.m, C = J.trans ? J.m : J.n;
    if (C <= 0) {                // an empty sector: nothing to rotate
      if (me.rank == 0 && tid == 0) atomicMax(&ctl->sweeps, 1);
      continue;
    }
    T* W = static_cast<T*>(work) + J.woff;
    T* V = static_cast<T*>(vmat) + J.voff;
    int* pj = perm + J.soff;
    // rounds of the circle method over N blocks (odd nblk: the last is a dummy), npair
    // pairs each
    const int nblk = (C + B - 1) / B, N = nblk + (nblk & 1);
    const int nr = nblk <= 1 ? 1 : N - 1, npair = nblk <= 1 ? 1 : nblk / 2;
    // column of this thread (of the first kNc) in pair i of round r; nc: the pair's columns
    int nc = 0;
    auto column = [&](int r, int i) {
      int b0 = 0, b1 = 0;
      nc = min(B, C);
      if (nblk > 1) {
        circle_pair(N, r, i + (nblk & 1), b0, b1);
        nc = B + min(B, C - b1 * B);
      }
      return tid < nc ? __ldcg(pj + (tid < B ? b0 * B + tid : b1 * B + tid - B)) : 0;
    };
    int sweeps = -1;
    for (int sw = 0; sw < max_sweeps; ++sw) {
      int* cur = cnt + (sw % 3) * nj + j;
      if (me.rank == 0 && tid == 0) cnt[((sw + 1) % 3) * nj + j] = 0;
      // column order of this sweep: decreasing norm (de Rijk), ties by index.  Norms
      // one warp per column, then every column's rank counted by a warp.  A NaN counts as
      // -1: the order is a permutation whatever the input, so no two visits of a round
      // share a column.
      const int gw = (me.rank * kSvdThreads + tid) >> 5, nw = me.size * kSvdWarps;
      for (int c = gw; c < C; c += nw) {
        double a = 0.0;
        for (int r = lane; r < R; r += 32) {
          const T x = __ldcg(W + r + (long long)c * R);
          if constexpr (CPLX) a += x.x * x.x + x.y * x.y;
          else a += x * x;
        }
        a = wsum(a);
        if (lane == 0) nrm[J.soff + c] = a;
      }
      if (!svd_group_sync(bar, me.size, phase, ctl)) return;
      for (int c = gw; c < C; c += nw) {
        const double v = fmax(__ldcg(nrm + J.soff + c), -1.0);
        int rank = 0;
        for (int k = lane; k < C; k += 32) {
          const double u = fmax(__ldcg(nrm + J.soff + k), -1.0);
          rank += (u > v || (u == v && k < c)) ? 1 : 0;
        }
        rank = __reduce_add_sync(0xffffffffu, rank);
        if (lane == 0) pj[rank] = c;
      }
      if (!svd_group_sync(bar, me.size, phase, ctl)) return;
      int col = me.rank < npair ? column(0, me.rank) : 0;
      for (int r = 0; r < nr; ++r) {
        for (int i = me.rank; i < npair; i += me.size) {
          if (i != me.rank) {
            col = column(r, i);
            __syncthreads();     // the visit before is done with cols
          }
          if (tid < nc) cols[tid] = col;
          __syncthreads();
          jacobi_pair_visit<CPLX, B, RES>(W, R, V, C, cols, nc, tol, smem_raw, looks, looks_n, cur);
        }
        // the next round's columns, on their way while the barrier is
        if (r + 1 < nr && me.rank < npair) col = column(r + 1, me.rank);
        if (!svd_group_sync(bar, me.size, phase, ctl)) return;
      }
      if (*reinterpret_cast<volatile int*>(cur) == 0) {
        sweeps = sw + 1;
        break;
      }
    }
    if (me.rank == 0 && tid == 0) {
      if (sweeps < 0) atomicExch(&ctl->failed, 1);
      else atomicMax(&ctl->sweeps, sweeps);
    }
  }
  if (tid == 0) atomicMax(&ctl->t1, svd_gtime());
}

// W = A (m >= n) or A^H (m < n); V = I (copy = 0: only the column order, when the
// caller has set W and V itself)
template <bool CPLX>
__global__ void jacobi_init_kernel(const SvdJob* jobs, const void* a, void* work, void* vmat, int* perm, int copy) {
  chain_begin();
  using T = typename SvdT<CPLX>::T;
  const SvdJob J = jobs[blockIdx.x];
  const int R = J.trans ? J.n : J.m, C = J.trans ? J.m : J.n;
  const T* A = static_cast<const T*>(a) + J.aoff;
  T* W = static_cast<T*>(work) + J.woff;
  T* V = static_cast<T*>(vmat) + J.voff;
  if (blockIdx.y == 0)
    for (int c = threadIdx.x; c < C; c += blockDim.x) perm[J.soff + c] = c;
  if (!copy) return;
  for (long long e = threadIdx.x + (long long)blockIdx.y * blockDim.x; e < (long long)R * C;
       e += (long long)blockDim.x * gridDim.y) {
    const int r = (int)(e % R), c = (int)(e / R);
    if (!J.trans) W[e] = A[r + (long long)c * J.m];
    else {
      T v = A[c + (long long)r * J.m];  // A^H(r, c) = conj(A(c, r))
      if (CPLX) reinterpret_cast<double2&>(v).y = -reinterpret_cast<double2&>(v).y;
      W[e] = v;
    }
  }
  for (long long e = threadIdx.x + (long long)blockIdx.y * blockDim.x; e < (long long)C * C;
       e += (long long)blockDim.x * gridDim.y) {
    const int r = (int)(e % C), c = (int)(e / C);
    if (CPLX) reinterpret_cast<double2*>(V)[e] = make_double2(r == c ? 1.0 : 0.0, 0.0);
    else reinterpret_cast<double*>(V)[e] = r == c ? 1.0 : 0.0;
  }
}

template <bool CPLX>
__global__ void jacobi_norms_kernel(const SvdJob* jobs, const void* work, double* sv) {
  chain_begin();
  using T = typename SvdT<CPLX>::T;
  const SvdJob J = jobs[blockIdx.x];
  const int R = J.trans ? J.n : J.m, C = J.trans ? J.m : J.n;
  const T* W = static_cast<const T*>(work) + J.woff;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int c = blockIdx.y * nw + warp; c < C; c += gridDim.y * nw) {
    double s = 0.0;
    for (int r = lane; r < R; r += 32) {
      if (CPLX) { const double2 v = reinterpret_cast<const double2*>(W)[r + (long long)c * R]; s += v.x * v.x + v.y * v.y; }
      else { const double v = reinterpret_cast<const double*>(W)[r + (long long)c * R]; s += v * v; }
    }
    s = wsum(s);
    if (lane == 0) sv[J.soff + c] = sqrt(s);
  }
}

// ---------------------------------------------------------------------------
// QR preconditioning (Drmac & Veselic, "New fast and accurate Jacobi SVD
// algorithm I", SIAM J. Matrix Anal. Appl. 29, 2008): with the columns of
// W0 = op(A) ordered by decreasing norm (P), W0 = Q R and R^H = Q1 R1 by
// Householder reflections, and the one-sided Jacobi runs on R1^H (C x C) instead
// of W0:
//   R1^H V2 = U2 S  =>  op(A) = (Q U2) S (P Q1 V2)^H,
// so the outputs keep the meaning they have without preconditioning -- W =
// Q [R1^H V2; 0] = Q U2 S, the left factor times S, and V = P Q1 V2 -- with no
// division by S.  The graded rows of R make the Jacobi converge in well under
// the sweeps it takes on W0 itself.  Each QR is
// blocked (panels of NB columns, compact WY form H_1 ... H_NB = I - Y T Y^H as in
// LAPACK's larft): one CTA factors a job's panel in shared memory, then every
// CTA updates one NB-column tile of a trailing matrix; Q (V1 S) applies the same
// block reflectors in reverse.  All panels run in one cooperative launch with
// bounded grid barriers.
template <bool CPLX> struct QrGeom {
  static constexpr int NB = CPLX ? 8 : 16;     // panel width
  static constexpr int RC = 256;               // rows per chunk of a tile update
  static constexpr int LD = RC + 1;            // shared row stride of a chunk (odd: no bank conflicts)
  static constexpr int NT = NB * NB;
  static constexpr int G = kSvdThreads / NT;   // row groups of the Y = V^H X sums
};
constexpr size_t kQrSmemMax = 200 * 1024;       // largest panel kept in shared memory
// Calls whose widest block has fewer columns run the Jacobi directly: it needs a
// few rounds per sweep there, so the QRs would cost about what they save.  (It
// also keeps the first steps of an iDMRG warm-up -- blocks of a few columns,
// some of pure rounding noise, whose kept count the 1e-16 floor of the
// per-sector cut-off then decides -- on the path of the plain Jacobi.)
constexpr int kQrMinCols = 32;

struct QrJob {
  long long aoff;             // input block (m x n, lda m)
  long long qoff;             // the matrix factored (R x C, ld R), then R above and the reflectors below the diagonal
  long long toff;             // T factors of the panels, NB x NB each (column-major)
  long long jwoff, jvoff;     // the Jacobi's W = R1^H and V (C x C each)
  long long woff, voff, soff; // outputs as in SvdJob; for a Q application: the matrix it multiplies (ld R)
  int m, n, trans, R, C;
  int x_in_q;                 // Q application: the matrix is in the QR buffer (1) or in the output W (0)
};
struct QrTile {
  int job, c1;                // a tile of NB columns starting at column c1
};

__device__ __forceinline__ double cabs2(double a) { return a * a; }
__device__ __forceinline__ double cabs2(double2 a) { return a.x * a.x + a.y * a.y; }
__device__ __forceinline__ double csub(double a, double b) { return a - b; }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
template <class T> __device__ __forceinline__ T cmake(double re, double im);
template <> __device__ __forceinline__ double cmake<double>(double re, double) { return re; }
template <> __device__ __forceinline__ double2 cmake<double2>(double re, double im) { return make_double2(re, im); }
__device__ __forceinline__ double wsum_t(double v) { return wsum(v); }
__device__ __forceinline__ double2 wsum_t(double2 v) { return make_double2(wsum(v.x), wsum(v.y)); }
__device__ __forceinline__ double cscale(double a, double s) { return a * s; }
__device__ __forceinline__ double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }

// column c of op(A) at row r: A(r, c), or conj(A(c, r)) when the job works on A^H
template <class T>
__device__ __forceinline__ T op_a(const T* A, int m, int trans, int r, int c) {
  return trans ? cconj(A[c + (long long)r * m]) : A[r + (long long)c * m];
}

// Column norms of op(A).  (One block per sector for these, the order and jacobi_norms took
// 1.8 ms at D = 2048: 7 of 148 SMs.)
template <bool CPLX>
__global__ void qr_norms_kernel(const QrJob* jobs, const void* a, double* nrm) {
  chain_begin();
  using T = typename SvdT<CPLX>::T;
  const QrJob J = jobs[blockIdx.x];
  const T* A = static_cast<const T*>(a) + J.aoff;
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int c = blockIdx.y * nw + (threadIdx.x >> 5); c < J.C; c += gridDim.y * nw) {
    double s = 0.0;
    for (int r = lane; r < J.R; r += 32) s += cabs2(op_a(A, J.m, J.trans, r, c));
    s = wsum(s);
    if (lane == 0) nrm[J.soff + c] = s;
  }
}
// Their order (decreasing, ties by index): P; a warp counts a column's rank.
template <bool CPLX>
__global__ void qr_order_kernel(const QrJob* jobs, const double* nrm, int* perm) {
  chain_begin();
  const QrJob J = jobs[blockIdx.x];
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const double* nj = nrm + J.soff;
  for (int c = blockIdx.y * nw + (threadIdx.x >> 5); c < J.C; c += gridDim.y * nw) {
    const double v = fmax(nj[c], -1.0);   // (a NaN counts as -1: a permutation whatever the input)
    int rank = 0;
    for (int k = lane; k < J.C; k += 32) {
      const double u = fmax(nj[k], -1.0);
      rank += (u > v || (u == v && k < c)) ? 1 : 0;
    }
    rank = __reduce_add_sync(0xffffffffu, rank);
    if (lane == 0) perm[J.soff + rank] = c;
  }
}

// W0 = op(A) P
template <bool CPLX>
__global__ void qr_gather_kernel(const QrJob* jobs, const void* a, void* qbuf, const int* perm) {
  chain_begin();
  using T = typename SvdT<CPLX>::T;
  const QrJob J = jobs[blockIdx.x];
  const T* A = static_cast<const T*>(a) + J.aoff;
  T* W = static_cast<T*>(qbuf) + J.qoff;
  const int* p = perm + J.soff;
  for (long long e = threadIdx.x + (long long)blockIdx.y * blockDim.x; e < (long long)J.R * J.C;
       e += (long long)blockDim.x * gridDim.y) {
    const int r = (int)(e % J.R), i = (int)(e / J.R);
    W[e] = op_a(A, J.m, J.trans, r, p[i]);
  }
}

// Panel k of job J: Householder reflections of its NB columns (rows k NB .. R-1)
// in shared memory (LAPACK larfg: beta = -sign(Re alpha) |x|, tau = (beta -
// alpha) / beta, v = x / (alpha - beta) below the unit diagonal; no reflection
// when the column below the diagonal is zero and alpha is real), each applied as
// H^H to the panel's later columns; then T of the compact WY form (forward,
// columnwise).  Writes R's panel rows, the reflectors and T back.
// The panel is what bounds a step: a chain of columns (norm, scale, dots, update) in one
// CTA while the other SMs wait.  Cycles of a panel of 172 x 16 on average (D = 512): load
// 1,900, columns 33,400, S 5,200, T 3,200, after 67,800 with one element in flight per lane, a
// dot at a time and T's sums through shared memory; a QR of D = 512 blocks 1.18 -> 0.83 ms, of
// D = 2048 10.1 -> 7.1.  The order of every sum is as it was (see jacobi_pair_visit on signs).
template <bool CPLX>
__device__ void qr_panel(const QrJob& J, int k, void* qbuf, unsigned char* smem) {
  using T = typename SvdT<CPLX>::T;
  constexpr int NB = QrGeom<CPLX>::NB;
  const int r0 = k * NB, nr = J.R - r0, w = min(NB, J.C - r0);
  T* A = static_cast<T*>(qbuf) + J.qoff;
  T* P = reinterpret_cast<T*>(smem);   // nr x w, column-major, ld nr
  __shared__ T tau_sh[NB];
  __shared__ T S_sh[NB * NB];          // S(k, j) = v_k^H v_j, k < j
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // kU elements of a column from i on, every 32nd (zeros past the rows): read together, as a
  // column is a chain of four passes over it and each element's latency would add to it (one
  // element at a time a column of 172 rows took 4,200 cycles)
  constexpr int kU = CPLX ? 4 : 8;
  auto take = [&](const T* x, int i, T (&a)[kU]) {
#pragma unroll
    for (int u = 0; u < kU; ++u) a[u] = i + 32 * u < nr ? x[i + 32 * u] : czero<T>();
  };
  for (int l = warp; l < w; l += kSvdWarps) {
    const T* src = A + r0 + (long long)(r0 + l) * J.R;
    for (int i = lane; i < nr; i += 32 * kU) {
      T a[kU];
      take(src, i, a);
#pragma unroll
      for (int u = 0; u < kU; ++u)
        if (i + 32 * u < nr) P[l * nr + i + 32 * u] = a[u];
    }
  }
  __syncthreads();
  for (int j = 0; j < w; ++j) {
    T* x = P + (long long)j * nr;
    if (warp == 0) {
      double s2 = 0.0;
      for (int i = j + 1 + lane; i < nr; i += 32 * kU) {
        T a[kU];
        take(x, i, a);
#pragma unroll
        for (int u = 0; u < kU; ++u) s2 += cabs2(a[u]);
      }
      s2 = wsum(s2);
      const T alpha = x[j];
      T tau = czero<T>();
      const bool refl = s2 > 0.0 || cim(alpha) != 0.0;
      double beta = 0.0;
      if (refl) {
        beta = -copysign(sqrt(cabs2(alpha) + s2), cre(alpha));
        tau = cmake<T>((beta - cre(alpha)) / beta, -cim(alpha) / beta);
        // 1 / (alpha - beta)
        T scale;
        if constexpr (CPLX) {
          const double dr = alpha.x - beta, di = alpha.y, dd = 1.0 / (dr * dr + di * di);
          scale = make_double2(dr * dd, -di * dd);
        } else {
          scale = 1.0 / (alpha - beta);
        }
        for (int i = j + 1 + lane; i < nr; i += 32 * kU) {
          T a[kU];
          take(x, i, a);
#pragma unroll
          for (int u = 0; u < kU; ++u)
            if (i + 32 * u < nr) x[i + 32 * u] = cmul(a[u], scale);
        }
      }
      __syncwarp();
      if (lane == 0) {
        tau_sh[j] = tau;
        if (refl) x[j] = cmake<T>(beta, 0.0);
      }
    }
    __syncthreads();
    const T tau = tau_sh[j];
    if (warp < w - 1 - j && cabs2(tau) != 0.0) {
      T* y = P + (long long)(j + 1 + warp) * nr;
      T d = lane == 0 ? y[j] : czero<T>();   // v_j = 1
      for (int i = j + 1 + lane; i < nr; i += 32 * kU) {
        T a[kU], b[kU];
        take(x, i, a);
        take(y, i, b);
#pragma unroll
        for (int u = 0; u < kU; ++u) d = cadd(d, cj_mul(a[u], b[u]));
      }
      d = wsum_t(d);
      const T f = cmul(cconj(tau), d);
      if (lane == 0) y[j] = csub(y[j], f);
      for (int i = j + 1 + lane; i < nr; i += 32 * kU) {
        T a[kU], b[kU];
        take(x, i, a);
        take(y, i, b);
#pragma unroll
        for (int u = 0; u < kU; ++u)
          if (i + 32 * u < nr) y[i + 32 * u] = csub(b[u], cmul(a[u], f));
      }
    }
    __syncthreads();
  }
  // S(q, j) = v_q^H v_j for q < j (rows j .. nr-1; v_j(j) = 1, v_q(j) = P(j, q)); a warp
  // takes a j, kQ of its sums side by side
  constexpr int kQ = CPLX ? 2 : 4;
  for (int j = warp; j < w; j += kSvdWarps)
    for (int q0 = 0; q0 < j; q0 += kQ) {
      const T* vj = P + (long long)j * nr;
      T d[kQ];
#pragma unroll
      for (int q = 0; q < kQ; ++q) d[q] = lane == 0 ? cconj(P[(long long)min(q0 + q, j - 1) * nr + j]) : czero<T>();
      for (int i = j + 1 + lane; i < nr; i += 32 * kU) {
        T b[kU];
        take(vj, i, b);
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
          T a[kU];
          take(P + (long long)min(q0 + q, j - 1) * nr, i, a);
#pragma unroll
          for (int u = 0; u < kU; ++u) d[q] = cadd(d[q], cj_mul(a[u], b[u]));
        }
      }
#pragma unroll
      for (int q = 0; q < kQ; ++q) d[q] = wsum_t(d[q]);
#pragma unroll
      for (int q = 0; q < kQ; ++q)
        if (lane == 0 && q0 + q < j) S_sh[q0 + q + j * NB] = d[q];
    }
  __syncthreads();
  // T: T(j, j) = tau_j, T(0:j, j) = -tau_j T(0:j, 0:j) S(0:j, j)
  T* Tm = static_cast<T*>(qbuf) + J.toff + (long long)k * NB * NB;
  if (warp == 0) {
    T row[NB];                           // lane's row of T
#pragma unroll
    for (int j = 0; j < NB; ++j) {
      row[j] = czero<T>();
      if (j < w) {
        const T tj = tau_sh[j];
        T v = czero<T>();
#pragma unroll
        for (int q = 0; q < j; ++q)
          if (q >= lane) v = cadd(v, cmul(row[q], S_sh[q + j * NB]));
        if (lane < j) row[j] = cmul(cscale(tj, -1.0), v);
        if (lane == j) row[j] = tj;
      }
    }
#pragma unroll
    for (int j = 0; j < NB; ++j)
      if (lane < NB) Tm[lane + j * NB] = row[j];
  }
  for (int l = warp; l < w; l += kSvdWarps) {
    T* dst = A + r0 + (long long)(r0 + l) * J.R;
#pragma unroll 4
    for (int i = lane; i < nr; i += 32) dst[i] = P[l * nr + i];
  }
  __syncthreads();   // P, tau_sh and S_sh are reused by the next panel this CTA takes
}

// X(r0:R, c1:c1+tw) <- H X with H = I - Y T Y^H (adj = 0) or H^H = I - Y T^H Y^H
// (adj = 1), Y = the unit lower trapezoidal reflectors of panel k.  Two passes
// over row chunks: Z = T' (Y^H X), then X -= Y Z (a single chunk stays in shared
// memory between the passes).
template <bool CPLX>
__device__ void qr_apply_tile(const QrJob& J, int k, int c1, int ncols, int adj, const void* qbuf, void* xbase,
                              long long xoff, unsigned char* smem) {
  using T = typename SvdT<CPLX>::T;
  using Gm = QrGeom<CPLX>;
  constexpr int NB = Gm::NB, RC = Gm::RC, LD = Gm::LD, NT = Gm::NT, G = Gm::G;
  const int r0 = k * NB, nr = J.R - r0, w = min(NB, J.C - r0), tw = min(NB, ncols - c1);
  const T* A = static_cast<const T*>(qbuf) + J.qoff;
  const T* Tm = static_cast<const T*>(qbuf) + J.toff + (long long)k * NB * NB;
  T* X = static_cast<T*>(xbase) + xoff;
  T* Vs = reinterpret_cast<T*>(smem);      // RC x NB (ld LD)
  T* Xs = Vs + LD * NB;                    // RC x NB (ld LD)
  T* Yp = Xs + LD * NB;                    // G partial sums of Y (NB x NB each)
  T* Zs = Yp + G * NT;                     // Z (NB x NB)
  const int tid = threadIdx.x;
  const int g = tid / NT, l = (tid % NT) / NB, t = tid % NB;
  const int nch = (nr + RC - 1) / RC;
  // (four elements of each at a time: their latencies one after another were half of a tile)
  auto load = [&](int rr0, int rows) {
    constexpr int U = 4;
    for (int e0 = tid; e0 < RC * NB; e0 += U * kSvdThreads) {
      T v[U], x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u * kSvdThreads, i = e % RC, c = e / RC, gi = rr0 + i;
        v[u] = czero<T>();
        x[u] = czero<T>();
        if (i < rows && c < w && gi >= c) v[u] = gi == c ? cmake<T>(1.0, 0.0) : A[(r0 + gi) + (long long)(r0 + c) * J.R];
        if (i < rows && c < tw) x[u] = X[(r0 + gi) + (long long)(c1 + c) * J.R];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = e0 + u * kSvdThreads, i = e % RC, c = e / RC;
        Vs[i + c * LD] = v[u];
        Xs[i + c * LD] = x[u];
      }
    }
  };
  static_assert(RC * NB % (4 * kSvdThreads) == 0, "whole groups of four");
  T acc = czero<T>();
  for (int ch = 0; ch < nch; ++ch) {
    const int rr0 = ch * RC, rows = min(RC, nr - rr0);
    load(rr0, rows);
    __syncthreads();
#pragma unroll 8
    for (int i = g; i < rows; i += G) acc = cadd(acc, cj_mul(Vs[i + l * LD], Xs[i + t * LD]));
    __syncthreads();
  }
  Yp[g * NT + l * NB + t] = acc;
  __syncthreads();
  if (tid < NT) {
    T y = czero<T>();
    for (int q = 0; q < G; ++q) y = cadd(y, Yp[q * NT + l * NB + t]);
    Zs[l * NB + t] = y;   // Y(l, t), row-major
  }
  __syncthreads();
  T z = czero<T>();
  if (tid < NT) {
    // Z(l, t) = sum_q T'(l, q) Y(q, t), T' = T (upper) or T^H (lower)
    for (int q = 0; q < w; ++q) {
      const T tq = adj ? cconj(Tm[q + l * NB]) : Tm[l + q * NB];
      z = cadd(z, cmul(tq, Zs[q * NB + t]));
    }
  }
  __syncthreads();
  if (tid < NT) Zs[l * NB + t] = z;
  __syncthreads();
  for (int ch = 0; ch < nch; ++ch) {
    const int rr0 = ch * RC, rows = min(RC, nr - rr0);
    if (nch > 1) {
      load(rr0, rows);
      __syncthreads();
    }
    for (int e = tid; e < RC * NB; e += kSvdThreads) {
      const int i = e % RC, c = e / RC;
      if (i >= rows || c >= tw) continue;
      T x = Xs[i + c * LD];
#pragma unroll
      for (int q = 0; q < NB; ++q) x = csub(x, cmul(Vs[i + q * LD], Zs[q * NB + c]));
      X[(r0 + rr0 + i) + (long long)(c1 + c) * J.R] = x;
    }
    __syncthreads();
  }
}

template <bool CPLX>
constexpr size_t qr_tile_smem() {
  using Gm = QrGeom<CPLX>;
  return (size_t)(2 * Gm::LD * Gm::NB + Gm::G * Gm::NT + Gm::NT) * (CPLX ? 16 : 8);
}

// The blocked QR of every job: step k factors panel k of every job that has one,
// then updates every NB-column tile right of it; a bounded grid barrier after
// each phase.
template <bool CPLX>
__global__ void __launch_bounds__(kSvdThreads, 1) qr_coop_kernel(const QrJob* __restrict__ jobs,
                                                              const int* __restrict__ panels, const int* __restrict__ poff,
                                                              const QrTile* __restrict__ tiles, const int* __restrict__ toff,
                                                              int steps, void* qbuf, SvdCtl* ctl) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned phase = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->t0 = svd_gtime();
  for (int k = 0; k < steps; ++k) {
    for (int p = poff[k] + blockIdx.x; p < poff[k + 1]; p += gridDim.x) qr_panel<CPLX>(jobs[panels[p]], k, qbuf, smem_raw);
    if (!svd_group_sync(&ctl->count, gridDim.x, phase, ctl)) return;
    for (int t = toff[k] + blockIdx.x; t < toff[k + 1]; t += gridDim.x) {
      const QrTile tl = tiles[t];
      const QrJob& J = jobs[tl.job];
      qr_apply_tile<CPLX>(J, k, tl.c1, J.C, 1, qbuf, qbuf, J.qoff, smem_raw);
    }
    if (!svd_group_sync(&ctl->count, gridDim.x, phase, ctl)) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->t1 = svd_gtime();
}

// X <- Q X for every job: its block reflectors applied from the last panel to
// the first to X (R x C at woff, in the output W or in the QR buffer).
template <bool CPLX>
__global__ void __launch_bounds__(kSvdThreads) qr_unmq_kernel(const QrJob* __restrict__ jobs,
                                                              const QrTile* __restrict__ tiles, const int* __restrict__ toff,
                                                              int steps, void* qbuf, void* out, SvdCtl* ctl) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned phase = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->t0 = svd_gtime();
  for (int k = steps - 1; k >= 0; --k) {
    for (int t = toff[k] + blockIdx.x; t < toff[k + 1]; t += gridDim.x) {
      const QrTile tl = tiles[t];
      const QrJob& J = jobs[tl.job];
      qr_apply_tile<CPLX>(J, k, tl.c1, J.C, 0, qbuf, J.x_in_q ? qbuf : out, J.woff, smem_raw);
    }
    if (k > 0 && !svd_group_sync(&ctl->count, gridDim.x, phase, ctl)) return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) ctl->t1 = svd_gtime();
}

// R^H (lower triangular, C x C) of src's factor into dst's matrix to factor
// (to_jacobi = 0), or into dst's Jacobi W with V = I (to_jacobi = 1).
template <bool CPLX>
__global__ void qr_rh_kernel(const QrJob* src, const QrJob* dst, void* qbuf, int to_jacobi) {
  chain_begin();
  using T = typename SvdT<CPLX>::T;
  const QrJob S = src[blockIdx.x], D = dst[blockIdx.x];
  const T* A = static_cast<const T*>(qbuf) + S.qoff;
  T* W = static_cast<T*>(qbuf) + (to_jacobi ? D.jwoff : D.qoff);
  T* V = static_cast<T*>(qbuf) + D.jvoff;
  const int C = S.C;
  for (long long e = threadIdx.x + (long long)blockIdx.y * blockDim.x; e < (long long)C * C;
       e += (long long)blockDim.x * gridDim.y) {
    const int r = (int)(e % C), c = (int)(e / C);
    W[e] = r >= c ? cconj(A[c + (long long)r * S.R]) : czero<T>();
    if (to_jacobi) V[e] = cmake<T>(r == c ? 1.0 : 0.0, 0.0);
  }
}

// Before the Q applications: the output W = [R1^H V2; 0] (R x C).
template <bool CPLX>
__global__ void qr_wout_kernel(const QrJob* jobs, const void* qbuf, void* work) {
  chain_begin();
  using T = typename SvdT<CPLX>::T;
  const QrJob J = jobs[blockIdx.x];
  const T* Wj = static_cast<const T*>(qbuf) + J.jwoff;
  T* W = static_cast<T*>(work) + J.woff;
  for (long long e = threadIdx.x + (long long)blockIdx.y * blockDim.x; e < (long long)J.R * J.C;
       e += (long long)blockDim.x * gridDim.y) {
    const int r = (int)(e % J.R), c = (int)(e / J.R);
    W[e] = r < J.C ? Wj[r + (long long)c * J.C] : czero<T>();
  }
}

// After them: the output V = P (Q1 V2), rows put back in the order of op(A)'s columns.
template <bool CPLX>
__global__ void qr_vout_kernel(const QrJob* jobs, const void* qbuf, void* vmat, const int* perm) {
  chain_begin();
  using T = typename SvdT<CPLX>::T;
  const QrJob J = jobs[blockIdx.x];
  const T* Vj = static_cast<const T*>(qbuf) + J.jvoff;
  T* V = static_cast<T*>(vmat) + J.voff;
  const int* p = perm + J.soff;
  for (long long e = threadIdx.x + (long long)blockIdx.y * blockDim.x; e < (long long)J.C * J.C;
       e += (long long)blockDim.x * gridDim.y) {
    const int i = (int)(e % J.C), c = (int)(e / J.C);
    V[p[i] + (long long)c * J.C] = Vj[e];
  }
}

// CTAs of the Jacobi kernel for nsect sectors with pairs[j] pairs per round, rounds[j]
// rounds per sweep and visits of cost[j] each: of all shares of ncta CTAs the one whose
// longest sector ends first (every sector taking as many sweeps).  A sector that ends in
// time on one CTA may share it with others.  Fills the sectors' order and the CTAs.
static void jacobi_shares(const std::vector<int>& pairs, const std::vector<int>& rounds, const std::vector<double>& cost,
                          int ncta, std::vector<int>& order, std::vector<SvdCta>& ctas) {
  const int nj = (int)pairs.size();
  std::vector<int> by(nj);
  for (int j = 0; j < nj; ++j) by[j] = j;
  auto alone = [&](int j) { return rounds[j] * cost[j] * pairs[j]; };
  std::stable_sort(by.begin(), by.end(), [&](int a, int b) { return alone(a) > alone(b); });
  std::vector<std::vector<int>> bins;
  // CTAs needed to end by time t (> ncta: no)
  auto fits = [&](double t) {
    bins.clear();
    std::vector<double> left;
    long long n = 0;
    for (const int j : by) {
      const double turns = std::floor(t / (rounds[j] * cost[j]) * (1 + 1e-12));
      if (turns < 1.0) return false;
      const int size = (int)((pairs[j] + std::min(turns, 1e6) - 1) / std::floor(std::min(turns, 1e6)));
      if (size > 1) {
        n += size;
        continue;
      }
      size_t b = 0;
      while (b < bins.size() && left[b] < alone(j)) ++b;
      if (b == bins.size()) {
        bins.emplace_back();
        left.push_back(t);
      }
      bins[b].push_back(j);
      left[b] -= alone(j);
    }
    return n + (long long)bins.size() <= ncta;
  };
  double lo = 0.0, hi = 0.0;
  for (int j = 0; j < nj; ++j) hi += alone(j);
  for (int it = 0; it < 50; ++it) {
    const double t = 0.5 * (lo + hi);
    (fits(t) ? hi : lo) = t;
  }
  fits(hi);
  int group = 0;
  for (const int j : by) {
    const double turns = std::min(std::floor(hi / (rounds[j] * cost[j]) * (1 + 1e-12)), 1e6);
    const int size = (int)((pairs[j] + turns - 1) / turns);
    if (size <= 1) continue;
    for (int r = 0; r < size; ++r) ctas.push_back({group, r, size, (int)order.size(), 1});
    order.push_back(j);
    ++group;
  }
  for (const auto& b : bins) {
    ctas.push_back({group++, 0, 1, (int)order.size(), (int)b.size()});
    order.insert(order.end(), b.begin(), b.end());
  }
}

// Host driver of the Jacobi: all sweeps in one cooperative launch.  Returns the number
// of sweeps taken, or -1 when max_sweeps was reached.
template <bool CPLX, int B>
static int jacobi_run(const void* a, void* work, void* vmat, double* sv, const std::vector<SvdJob>& hjobs,
                      int max_sweeps, cudaStream_t s, double* kernel_ms, int copy = 1, int stream = 0) {
  const int nj = (int)hjobs.size();
  std::vector<int> pairs(nj), rounds(nj);
  std::vector<double> cost(nj);
  int maxR = 0;
  long long nsv = 1;   // singular-value slots (the column order lives at the same offsets)
  size_t smem = svd_smem_bytes<CPLX, B>(), res_smem = 0;
  for (int j = 0; j < nj; ++j) {
    const int R = hjobs[j].trans ? hjobs[j].n : hjobs[j].m;
    const int C = hjobs[j].trans ? hjobs[j].m : hjobs[j].n;
    maxR = std::max(maxR, R);
    res_smem = std::max(res_smem, svd_res_smem_bytes<CPLX, B>(R, C));
    nsv = std::max<long long>(nsv, hjobs[j].soff + C);
    const int nblk = (C + B - 1) / B;
    pairs[j] = std::max(nblk / 2, 1);
    rounds[j] = std::max(nblk + (nblk & 1) - 1, 1);
    // a visit's load, Gram and application take as long per row as 1,000 rows take for
    // its inner sweep and barrier (b = 8: 17,000 cycles + 12 a row; b = 16: 35,000 + 40)
    cost[j] = R + C + 1000.0;
  }
  // visits hold the pair's columns of W and V in shared memory when the largest fits
  const bool res = !stream && res_smem <= kSvdResMax;
  if (res) smem = std::max(smem, res_smem);
  const auto kernel = res ? jacobi_coop_kernel<CPLX, B, true> : jacobi_coop_kernel<CPLX, B, false>;
  static unsigned char limit[2][kMaxDevices] = {{0}};
  ensure_smem_limit((const void*)kernel, (int)std::max(svd_smem_bytes<CPLX, B>(), res ? kSvdResMax : 0), limit[res]);
  int dev = 0, nsm = 0, per_sm = 0;
  SADMRG_CUDA(cudaGetDevice(&dev));
  SADMRG_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  SADMRG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSvdThreads, smem));
  SADMRG_REQUIRE(per_sm > 0, SADMRG_ERR_CUDA, "jacobi svd: the kernel does not fit on this device");
  std::vector<int> order;
  std::vector<SvdCta> ctas;
  jacobi_shares(pairs, rounds, cost, per_sm * nsm, order, ctas);
  // one copy: jobs, CTAs, order; one cleared area: control, counters, barriers
  const size_t o_cta = sizeof(SvdJob) * nj, o_ord = o_cta + sizeof(SvdCta) * ctas.size();
  std::vector<char> host(o_ord + sizeof(int) * nj);
  std::memcpy(host.data(), hjobs.data(), o_cta);
  std::memcpy(host.data() + o_cta, ctas.data(), o_ord - o_cta);
  std::memcpy(host.data() + o_ord, order.data(), sizeof(int) * nj);
  const size_t o_cnt = sizeof(SvdCtl), o_bar = (o_cnt + sizeof(int) * 3 * nj + 127) & ~(size_t)127;
  const size_t nzero = o_bar + 128 * ctas.size();
  DevBuf dlists(host.size(), s), dzero(nzero, s), dperm(sizeof(int) * nsv, s);
  SADMRG_CUDA(cudaMemcpyAsync(dlists.get(), host.data(), host.size(), cudaMemcpyHostToDevice, s));
  SADMRG_CUDA(cudaMemsetAsync(dzero.get(), 0, nzero, s));
  char* lists = dlists.as<char>();
  char* zero = dzero.as<char>();
  SvdCtl* pctl = reinterpret_cast<SvdCtl*>(zero);
  SADMRG_CUDA(cudaMemsetAsync(&pctl->t0, 0xff, sizeof(pctl->t0), s));
  const SvdJob* pj = reinterpret_cast<const SvdJob*>(lists);
  const SvdCta* pcta = reinterpret_cast<const SvdCta*>(lists + o_cta);
  const int* pord = reinterpret_cast<const int*>(lists + o_ord);
  int* pcnt = reinterpret_cast<int*>(zero + o_cnt);
  unsigned* pbar = reinterpret_cast<unsigned*>(zero + o_bar);
  int* pperm = dperm.as<int>();
  launch_chained(jacobi_init_kernel<CPLX>, dim3(nj, 16), 256, 0, s, pj, a, work, vmat, pperm, copy);
  SADMRG_CUDA(cudaGetLastError());
  double tol = std::sqrt((double)std::max(maxR, 1)) * 2.220446049250313e-16;
  int njv = nj;
  double* nrm = sv;   // column norms of each sweep; the final singular values overwrite them
  void* args[] = {(void*)&pj,   (void*)&njv, (void*)&pcta,  (void*)&pord, (void*)&pbar, (void*)&work,       (void*)&vmat,
                  (void*)&nrm,  (void*)&pperm, (void*)&tol, (void*)&pcnt, (void*)&pctl, (void*)&max_sweeps};
  SADMRG_CUDA(cudaLaunchCooperativeKernel((const void*)kernel, dim3((unsigned)ctas.size()), dim3(kSvdThreads), args, smem, s));
  SvdCtl hctl{};
  SADMRG_CUDA(cudaMemcpyAsync(&hctl, pctl, sizeof(SvdCtl), cudaMemcpyDeviceToHost, s));
  launch_chained(jacobi_norms_kernel<CPLX>, dim3(nj, 16), 256, 0, s, pj, work, sv);
  SADMRG_CUDA(cudaGetLastError());
  SADMRG_CUDA(cudaStreamSynchronize(s));
  SADMRG_REQUIRE(hctl.status == 0, SADMRG_ERR_CUDA, "jacobi svd: a barrier ran out of time");
  if (kernel_ms) *kernel_ms = (double)(hctl.t1 - hctl.t0) * 1e-6;
  return hctl.failed ? -1 : hctl.sweeps;
}

// Column blocks of the Jacobi for these jobs: 8 when a round of all sectors'
// 16-column pairs would keep fewer than half the SMs busy, else 16.
static bool narrow_blocks(const std::vector<SvdJob>& hjobs) {
  int dev = 0, nsm = 0;
  SADMRG_CUDA(cudaGetDevice(&dev));
  SADMRG_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  long long pairs16 = 0;
  for (const SvdJob& J : hjobs) {
    const int C = J.trans ? J.m : J.n;
    const int nb = (C + 15) / 16;
    pairs16 += nb <= 1 ? 1 : nb / 2;
  }
  return 2 * pairs16 < nsm;
}

// Launches a cooperative kernel (whose shared-memory limit is set) on the largest grid the
// device keeps resident, capped at `want` CTAs.  Returns false (nothing launched) when it cannot.
static bool coop_launch(const void* fn, int want, size_t smem, void** args, cudaStream_t s) {
  int dev = 0, coop = 0, nsm = 0, per_sm = 0;
  SADMRG_CUDA(cudaGetDevice(&dev));
  SADMRG_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  SADMRG_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  SADMRG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kSvdThreads, smem));
  if (!coop || per_sm <= 0) return false;
  const int grid = std::max(1, std::min(want, per_sm * nsm));
  SADMRG_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kSvdThreads), args, smem, s));
  return true;
}

// Per-step work lists of a set of QrJobs: the panels and trailing tiles of the
// QR (qr_coop_kernel), or the tiles of a Q application (qr_unmq_kernel).
struct QrLists {
  std::vector<int> panels, poff, toff;
  std::vector<QrTile> tiles;
  int steps = 0, want = 1;
};
template <int NB>
static QrLists qr_lists(const std::vector<QrJob>& jobs, bool unmq) {
  QrLists L;
  for (const QrJob& J : jobs) L.steps = std::max(L.steps, (J.C + NB - 1) / NB);
  L.poff.assign(L.steps + 1, 0);
  L.toff.assign(L.steps + 1, 0);
  for (int k = 0; k < L.steps; ++k) {
    L.poff[k] = (int)L.panels.size();
    L.toff[k] = (int)L.tiles.size();
    for (int j = 0; j < (int)jobs.size(); ++j) {
      if (jobs[j].C <= k * NB) continue;
      if (!unmq) L.panels.push_back(j);
      for (int c1 = unmq ? 0 : (k + 1) * NB; c1 < jobs[j].C; c1 += NB) L.tiles.push_back({j, c1});
    }
    L.want = std::max({L.want, (int)L.panels.size() - L.poff[k], (int)L.tiles.size() - L.toff[k]});
  }
  L.poff[L.steps] = (int)L.panels.size();
  L.toff[L.steps] = (int)L.tiles.size();
  return L;
}

// Device copies of a job array and its lists, and the cooperative launch of the
// QR (unmq = false) or of the Q application (unmq = true).  Returns false when
// the device cannot run it cooperatively.
template <bool CPLX>
struct QrLaunch {
  DevBuf dj, dpan, dpoff, dtl, dtoff;
  QrLists L;
  bool run(const std::vector<QrJob>& jobs, bool unmq, void* qbuf, void* out, SvdCtl* ctl, cudaStream_t s) {
    constexpr int NB = QrGeom<CPLX>::NB;
    L = qr_lists<NB>(jobs, unmq);
    int maxR = 0;
    for (const QrJob& J : jobs) maxR = std::max(maxR, J.R);
    dj.alloc(sizeof(QrJob) * jobs.size(), s);
    dpan.alloc(sizeof(int) * std::max<size_t>(L.panels.size(), 1), s);
    dpoff.alloc(sizeof(int) * (L.steps + 1), s);
    dtl.alloc(sizeof(QrTile) * std::max<size_t>(L.tiles.size(), 1), s);
    dtoff.alloc(sizeof(int) * (L.steps + 1), s);
    SADMRG_CUDA(cudaMemcpyAsync(dj.get(), jobs.data(), sizeof(QrJob) * jobs.size(), cudaMemcpyHostToDevice, s));
    if (!L.panels.empty())
      SADMRG_CUDA(cudaMemcpyAsync(dpan.get(), L.panels.data(), sizeof(int) * L.panels.size(), cudaMemcpyHostToDevice, s));
    if (!L.tiles.empty())
      SADMRG_CUDA(cudaMemcpyAsync(dtl.get(), L.tiles.data(), sizeof(QrTile) * L.tiles.size(), cudaMemcpyHostToDevice, s));
    SADMRG_CUDA(cudaMemcpyAsync(dpoff.get(), L.poff.data(), sizeof(int) * (L.steps + 1), cudaMemcpyHostToDevice, s));
    SADMRG_CUDA(cudaMemcpyAsync(dtoff.get(), L.toff.data(), sizeof(int) * (L.steps + 1), cudaMemcpyHostToDevice, s));
    const QrJob* pj = dj.as<QrJob>();
    const int* pp = dpan.as<int>();
    const int* ppo = dpoff.as<int>();
    const QrTile* pt = dtl.as<QrTile>();
    const int* pto = dtoff.as<int>();
    int st = L.steps;
    void* qb = qbuf;
    void* o = out;
    SvdCtl* pc = ctl;
    static unsigned char limit[2][kMaxDevices] = {{0}};
    if (unmq) {
      ensure_smem_limit((const void*)qr_unmq_kernel<CPLX>, (int)qr_tile_smem<CPLX>(), limit[1]);
      void* args[] = {(void*)&pj, (void*)&pt, (void*)&pto, (void*)&st, (void*)&qb, (void*)&o, (void*)&pc};
      return coop_launch((const void*)qr_unmq_kernel<CPLX>, L.want, qr_tile_smem<CPLX>(), args, s);
    }
    const size_t smem = std::max((size_t)maxR * NB * sizeof(typename SvdT<CPLX>::T), qr_tile_smem<CPLX>());
    ensure_smem_limit((const void*)qr_coop_kernel<CPLX>, (int)std::max(kQrSmemMax, qr_tile_smem<CPLX>()), limit[0]);
    void* args[] = {(void*)&pj, (void*)&pp, (void*)&ppo, (void*)&pt, (void*)&pto, (void*)&st, (void*)&qb, (void*)&pc};
    return coop_launch((const void*)qr_coop_kernel<CPLX>, L.want, smem, args, s);
  }
};

// The QR-preconditioned SVD (see the QR preconditioning notes above).  Returns
// the Jacobi sweeps (as jacobi_run), or 0 with *fallback set when the device
// cannot run the cooperative kernels (the call then runs without
// preconditioning).
template <bool CPLX>
static int qr_jacobi_run(const void* a, void* work, void* vmat, double* sv, const std::vector<SvdJob>& hjobs,
                         int max_sweeps, cudaStream_t s, double* kernel_ms, bool* fallback, int stream, int block) {
  using T = typename SvdT<CPLX>::T;
  constexpr int NB = QrGeom<CPLX>::NB;
  *fallback = false;
  const int nj = (int)hjobs.size();
  // q1: op(A) P = Q R (R x C); q2: R^H = Q1 R1 (C x C), whose Jacobi W = R1^H and V
  // live at jwoff / jvoff; the second Q application multiplies that V
  std::vector<QrJob> q1(nj), q2(nj);
  long long tot = 0, nsv = 1;
  for (int j = 0; j < nj; ++j) {
    const SvdJob& J = hjobs[j];
    const int R = std::max(J.m, J.n), C = std::min(J.m, J.n), np = (C + NB - 1) / NB;
    QrJob& A = q1[j];
    QrJob& B = q2[j];
    A = QrJob{};
    A.aoff = J.aoff; A.woff = J.woff; A.voff = J.voff; A.soff = J.soff;
    A.m = J.m; A.n = J.n; A.trans = J.trans; A.R = R; A.C = C; A.x_in_q = 0;
    A.qoff = tot;  tot += (long long)R * C;
    A.toff = tot;  tot += (long long)np * NB * NB;
    B = A;
    B.m = B.n = B.R = C; B.trans = 0;
    B.qoff = tot;  tot += (long long)C * C;
    B.toff = tot;  tot += (long long)np * NB * NB;
    A.jwoff = B.jwoff = tot; tot += (long long)C * C;
    A.jvoff = B.jvoff = tot; tot += (long long)C * C;
    B.woff = B.jvoff;   // the second Q application multiplies the Jacobi's V
    B.x_in_q = 1;
    nsv = std::max<long long>(nsv, J.soff + C);
  }
  DevBuf qbuf(sizeof(T) * std::max<long long>(tot, 1), s), dperm(sizeof(int) * nsv, s), dctl(3 * sizeof(SvdCtl), s);
  SADMRG_CUDA(cudaMemsetAsync(dctl.get(), 0, 3 * sizeof(SvdCtl), s));
  SvdCtl* ctl = dctl.as<SvdCtl>();
  QrLaunch<CPLX> L1, L2, LU;
  // P and W0 = op(A) P need the job array on the device: the first QR's copy
  L1.dj.alloc(sizeof(QrJob) * nj, s);
  SADMRG_CUDA(cudaMemcpyAsync(L1.dj.get(), q1.data(), sizeof(QrJob) * nj, cudaMemcpyHostToDevice, s));
  launch_chained(qr_norms_kernel<CPLX>, dim3(nj, 32), 256, 0, s, static_cast<const QrJob*>(L1.dj.get()), a, sv);
  launch_chained(qr_order_kernel<CPLX>, dim3(nj, 32), 256, 0, s, static_cast<const QrJob*>(L1.dj.get()), (const double*)sv, dperm.as<int>());
  launch_chained(qr_gather_kernel<CPLX>, dim3(nj, 32), 256, 0, s, static_cast<const QrJob*>(L1.dj.get()), a, qbuf.get(), dperm.as<int>());
  SADMRG_CUDA(cudaGetLastError());
  if (!L1.run(q1, false, qbuf.get(), work, ctl, s)) {
    *fallback = true;
    return 0;
  }
  L2.dj.alloc(sizeof(QrJob) * nj, s);
  SADMRG_CUDA(cudaMemcpyAsync(L2.dj.get(), q2.data(), sizeof(QrJob) * nj, cudaMemcpyHostToDevice, s));
  launch_chained(qr_rh_kernel<CPLX>, dim3(nj, 16), 256, 0, s, static_cast<const QrJob*>(L1.dj.get()), static_cast<const QrJob*>(L2.dj.get()), qbuf.get(), 0);
  SADMRG_CUDA(cudaGetLastError());
  SADMRG_REQUIRE(L2.run(q2, false, qbuf.get(), work, ctl + 1, s), SADMRG_ERR_CUDA,
                 "svd: the second cooperative QR cannot be launched");
  launch_chained(qr_rh_kernel<CPLX>, dim3(nj, 16), 256, 0, s, static_cast<const QrJob*>(L2.dj.get()), static_cast<const QrJob*>(L2.dj.get()), qbuf.get(), 1);
  SADMRG_CUDA(cudaGetLastError());
  // the Jacobi on R1^H (C x C, W and V in qbuf)
  std::vector<SvdJob> jj(nj);
  for (int j = 0; j < nj; ++j) {
    SvdJob& J = jj[j];
    J.aoff = 0;
    J.woff = q2[j].jwoff;
    J.voff = q2[j].jvoff;
    J.soff = q2[j].soff;
    J.m = J.n = q2[j].C;
    J.trans = 0;
  }
  double jms = -1.0;
  const bool narrow = block == 8 || (block == 0 && narrow_blocks(jj));
  const int sweeps = narrow
                         ? jacobi_run<CPLX, 8>(nullptr, qbuf.get(), qbuf.get(), sv, jj, max_sweeps, s, &jms, 0, stream)
                         : jacobi_run<CPLX, 16>(nullptr, qbuf.get(), qbuf.get(), sv, jj, max_sweeps, s, &jms, 0, stream);
  if (sweeps <= 0) return sweeps;
  // W = Q [R1^H V2; 0] and Q1 V2, both Q applications in one launch, then V = P (Q1 V2)
  launch_chained(qr_wout_kernel<CPLX>, dim3(nj, 16), 256, 0, s, static_cast<const QrJob*>(L1.dj.get()), qbuf.get(), work);
  SADMRG_CUDA(cudaGetLastError());
  std::vector<QrJob> qu(q1);
  qu.insert(qu.end(), q2.begin(), q2.end());
  SADMRG_REQUIRE(LU.run(qu, true, qbuf.get(), work, ctl + 2, s), SADMRG_ERR_CUDA,
                 "svd: the cooperative Q application cannot be launched");
  launch_chained(qr_vout_kernel<CPLX>, dim3(nj, 16), 256, 0, s, static_cast<const QrJob*>(L1.dj.get()), qbuf.get(), vmat, dperm.as<int>());
  SADMRG_CUDA(cudaGetLastError());
  SvdCtl hctl[3];
  SADMRG_CUDA(cudaMemcpyAsync(hctl, dctl.get(), 3 * sizeof(SvdCtl), cudaMemcpyDeviceToHost, s));
  SADMRG_CUDA(cudaStreamSynchronize(s));
  SADMRG_REQUIRE(hctl[0].status == 0 && hctl[1].status == 0 && hctl[2].status == 0, SADMRG_ERR_CUDA,
                 "svd: a grid barrier of the QR preconditioning ran out of time");
  if (kernel_ms && jms >= 0.0) {
    *kernel_ms = jms;
    for (const SvdCtl& c : hctl) *kernel_ms += (double)(c.t1 - c.t0) * 1e-6;
  }
  return sweeps;
}

int run_jacobi_svd(bool cplx, const void* a, void* work, void* vmat, double* sv, const std::vector<SvdJob>& hjobs,
                   int max_sweeps, cudaStream_t s, double* kernel_ms, int precondition, int stream, int block) {
  if (kernel_ms) *kernel_ms = -1.0;
  if (hjobs.empty()) return 0;
  if (precondition) {
    // the panel of the tallest block must fit in shared memory
    int maxR = 0, maxC = 0;
    for (const SvdJob& J : hjobs) {
      maxR = std::max(maxR, std::max(J.m, J.n));
      maxC = std::max(maxC, std::min(J.m, J.n));
    }
    const size_t panel = (size_t)maxR * (cplx ? QrGeom<true>::NB * 16 : QrGeom<false>::NB * 8);
    if (panel <= kQrSmemMax && (maxC >= kQrMinCols || precondition == 2)) {
      bool fallback = false;
      const int sw = cplx ? qr_jacobi_run<true>(a, work, vmat, sv, hjobs, max_sweeps, s, kernel_ms, &fallback, stream, block)
                          : qr_jacobi_run<false>(a, work, vmat, sv, hjobs, max_sweeps, s, kernel_ms, &fallback, stream, block);
      if (!fallback) return sw;
    }
  }
  // column blocks of 16, or of 8 when a round of all sectors' 16-column pairs would
  // keep fewer than half the SMs busy: narrower pairs double the CTAs per round
  // and cut each visit's work to a quarter, which wins while SMs are idle and loses
  // once they are not.  One truncation with 8 and 16 columns, ms: SU(2) D = 512 7.2 and
  // 7.7, 768 14.7 and 16.3, 1,024 25.0 and 23.3, 2,048 107 and 80; complex U(1) D = 384
  // 4.8 and 5.2, 1,024 24.5 and 27.5, 1,536 52.0 and 59.7, 2,048 145 and 106.  The rule
  // takes 8 up to 1,024 in both, so it is 7% off the better width at SU(2) D = 1,024
  // and 14% at complex D = 1,536.
  const bool narrow = block == 8 || (block == 0 && narrow_blocks(hjobs));
  if (cplx)
    return narrow ? jacobi_run<true, 8>(a, work, vmat, sv, hjobs, max_sweeps, s, kernel_ms, 1, stream)
                  : jacobi_run<true, 16>(a, work, vmat, sv, hjobs, max_sweeps, s, kernel_ms, 1, stream);
  return narrow ? jacobi_run<false, 8>(a, work, vmat, sv, hjobs, max_sweeps, s, kernel_ms, 1, stream)
                : jacobi_run<false, 16>(a, work, vmat, sv, hjobs, max_sweeps, s, kernel_ms, 1, stream);
}

}  // namespace sadmrg
