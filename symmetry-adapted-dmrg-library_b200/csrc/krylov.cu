// krylov.cu -- vector kernels of the Lanczos solves, for one problem and for many
// independent ones stored back to back.
//
// A launch works on a VecSpan: segments cut into ranges, one thread block per
// range.  Reductions are deterministic: every block writes its partial sums, and
// the last of a segment's blocks to finish adds them in block order, so the result
// does not depend on which block is last.
//
// What bounds them is reading the Krylov vectors (8 or 16 bytes per
// multiply-add); a step of the recurrence reads each of them twice.  So the passes
// of a step are fused where they touch the same elements: the two-term update runs
// inside the pass that takes the dots for the reorthogonalisation, the norm inside
// the pass that applies it, and the scalars that the host needs go from the last
// block straight to page-locked memory.  Many problems: ranges of about 1/1024 of
// all elements keep the chip full whatever the segments' lengths (64 segments of
// 1,000 to 43,000 elements, 40 steps: one block per segment took 82 ms for the
// vector kernels of a solve).
#include <cuda_runtime.h>
#include <algorithm>

#include "kernels.cuh"
#include "ptx.cuh"

namespace sadmrg {
namespace {

constexpr int kVT = 256;             // threads per block
constexpr int kVW = kVT / 32;
constexpr int kG = 8;                // dots per pass over a block's range
// coefficients that a block keeps in shared memory (complex 32 KB); those of further
// vectors, which no solve has in earnest, are read where they are
constexpr int kStaged = 2048;

template <bool CX> struct VT_;
template <> struct VT_<false> { using T = double; };
template <> struct VT_<true> { using T = double2; };

__device__ __forceinline__ double vzero(double) { return 0.0; }
__device__ __forceinline__ double2 vzero(double2) { return make_double2(0.0, 0.0); }
// s + conj(a) b
__device__ __forceinline__ double dot_acc(double s, double a, double b) { return s + a * b; }
__device__ __forceinline__ double2 dot_acc(double2 s, double2 a, double2 b) {
  return make_double2(s.x + (a.x * b.x + a.y * b.y), s.y + (a.x * b.y - a.y * b.x));
}
// x - c v
__device__ __forceinline__ double sub_mul(double x, double c, double v) { return x - c * v; }
__device__ __forceinline__ double2 sub_mul(double2 x, double2 c, double2 v) {
  return make_double2(x.x - (c.x * v.x - c.y * v.y), x.y - (c.x * v.y + c.y * v.x));
}
// y + c v, real c
__device__ __forceinline__ double add_rmul(double y, double c, double v) { return y + c * v; }
__device__ __forceinline__ double2 add_rmul(double2 y, double c, double2 v) {
  return make_double2(y.x + c * v.x, y.y + c * v.y);
}
__device__ __forceinline__ double rmul(double x, double f) { return x * f; }
__device__ __forceinline__ double2 rmul(double2 x, double f) { return make_double2(x.x * f, x.y * f); }
__device__ __forceinline__ double vabs2(double x) { return x * x; }
__device__ __forceinline__ double vabs2(double2 x) { return x.x * x.x + x.y * x.y; }
__device__ __forceinline__ double vre(double x) { return x; }
__device__ __forceinline__ double vre(double2 x) { return x.x; }
__device__ __forceinline__ double vreal(double r, double) { return r; }
__device__ __forceinline__ double2 vreal(double r, double2) { return make_double2(r, 0.0); }

struct Range {
  long long lo, hi;
  int seg, first, count;             // its segment, and that segment's blocks [first, first + count)
};

__device__ __forceinline__ bool block_range(const VecSpan& v, Range& r) {
  if (!v.blk) {
    r.lo = v.per * blockIdx.x;
    r.hi = min(v.n, r.lo + v.per);
    r.seg = 0;
    r.first = 0;
    r.count = v.nblk;
  } else {
    const VecBlk b = v.blk[blockIdx.x];
    r.lo = b.lo;
    r.hi = b.lo + b.n;
    r.seg = b.seg;
    r.first = v.blk0[b.seg];
    r.count = v.blk0[b.seg + 1] - r.first;
  }
  return !v.active || v.active[r.seg];
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Sums of 8 values over the warp with 9 shuffles instead of 40: each of the first
// three exchanges halves the values a lane still carries.  On return lane l with
// l % 4 == 0 (and its three neighbours) holds the sum of value l / 4.
__device__ __forceinline__ double warp_sum8(double (&a)[8], int lane) {
#pragma unroll
  for (int o = 16, cnt = 8; cnt > 1; o >>= 1, cnt >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < cnt / 2; ++i) {
      const double keep = up ? a[i + cnt / 2] : a[i], send = up ? a[i] : a[i + cnt / 2];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double s = a[0];
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  return s;
}

// True (in every thread) in the last of the segment's blocks to get here; the
// partial sums that any of them wrote before are then visible.  The counter is left zero.
__device__ __forceinline__ bool last_block(unsigned* counter, const Range& r) {
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(counter + r.seg, 1u) == (unsigned)r.count - 1u;
    if (last) counter[r.seg] = 0u;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

__device__ __forceinline__ void norm_out(const VecOut& o, int seg, double sum) {
  const double nr = sqrt(fabs(sum));
  static_cast<double*>(o.scal)[(long long)seg * o.sstride] = nr;
  if (o.host) static_cast<double*>(o.host)[(long long)seg * o.hstride] = nr;
}

// out[seg * nv + j] = <V_j | x>, after x -= uc[0] u0 + uc[1] u1 when u1 is given
// (u0 may be null).  See VecOut for what the last block does with the sums.
template <bool CX>
__global__ void __launch_bounds__(kVT) vec_dots(VecSpan v, const typename VT_<CX>::T* V, long long ldv,
                                                int nv, typename VT_<CX>::T* x, const typename VT_<CX>::T* u0,
                                                const typename VT_<CX>::T* u1, const typename VT_<CX>::T* uc,
                                                double* partial, typename VT_<CX>::T* out, unsigned* counter,
                                                VecOut o) {
  using T = typename VT_<CX>::T;
  __shared__ double red[2][CX ? 2 : 1][kVW][kG];
  chain_begin();
  Range r;
  if (!block_range(v, r)) return;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  T c0 = vzero(T()), c1 = vzero(T());
  if (u1) {
    c1 = uc[2 * r.seg + 1];
    if (u0) c0 = uc[2 * r.seg];
  }
  int buf = 0;
  for (int j0 = 0; j0 < nv; j0 += kG, buf ^= 1) {
    const int g = min(kG, nv - j0);
    const T* Vg = V + j0 * ldv;
    T s[kG];
#pragma unroll
    for (int u = 0; u < kG; ++u) s[u] = vzero(T());
    auto body = [&](long long i, int gg) {
      T b = x[i];
      if (u1 && j0 == 0) {
        if (u0) b = sub_mul(b, c0, u0[i]);
        b = sub_mul(b, c1, u1[i]);
        x[i] = b;
      }
#pragma unroll
      for (int u = 0; u < kG; ++u)
        if (u < gg) s[u] = dot_acc(s[u], Vg[u * ldv + i], b);
    };
    if (g == kG) {
#pragma unroll 2
      for (long long i = r.lo + threadIdx.x; i < r.hi; i += kVT) body(i, kG);
    } else {
      for (long long i = r.lo + threadIdx.x; i < r.hi; i += kVT) body(i, g);
    }
    double re[kG], im[kG];
#pragma unroll
    for (int u = 0; u < kG; ++u) {
      if constexpr (CX) { re[u] = s[u].x; im[u] = s[u].y; }
      else re[u] = s[u];
    }
    const double a = warp_sum8(re, l);
    if ((l & 3) == 0) red[buf][0][w][l >> 2] = a;
    if constexpr (CX) {
      const double b = warp_sum8(im, l);
      if ((l & 3) == 0) red[buf][1][w][l >> 2] = b;
    }
    __syncthreads();
    if (w == 0 && l < g) {   // the next pass writes the other buffer
      double ta = 0.0, tb = 0.0;
#pragma unroll
      for (int k = 0; k < kVW; ++k) {
        ta += red[buf][0][k][l];
        if constexpr (CX) tb += red[buf][1][k][l];
      }
      double* p = partial + ((long long)blockIdx.x * nv + j0 + l) * (CX ? 2 : 1);
      p[0] = ta;
      if constexpr (CX) p[1] = tb;
    }
  }
  if (!last_block(counter, r)) return;
  for (int j = w; j < nv; j += kVW) {
    double a = 0.0, b = 0.0;
#pragma unroll 4
    for (int p = l; p < r.count; p += 32) {
      const double* q = partial + ((long long)(r.first + p) * nv + j) * (CX ? 2 : 1);
      a += __ldcg(q);
      if constexpr (CX) b += __ldcg(q + 1);
    }
    a = warp_sum(a);
    if constexpr (CX) b = warp_sum(b);
    if (l == 0) {
      T t;
      if constexpr (CX) t = make_double2(a, b);
      else t = a;
      out[(long long)r.seg * nv + j] = t;
      if (o.op == VO_HOST) static_cast<T*>(o.host)[(long long)r.seg * o.hstride + j] = t;
      if (j == 0 && o.op == VO_COEF) {
        T* sc = static_cast<T*>(o.scal) + 2 * (long long)r.seg;
        sc[0] = vreal(o.beta[(long long)r.seg * o.bstride], T());
        sc[1] = vreal(a, T());
        static_cast<double*>(o.host)[(long long)r.seg * o.hstride] = a;
      }
      if (j == 0 && o.op == VO_NORM) norm_out(o, r.seg, a);
    }
  }
}

// x -= sum_j c[seg * cstride + j] V_j; with a partial buffer also |x| of the result
// to o.scal and o.host (as VO_NORM).
template <bool CX>
__global__ void __launch_bounds__(kVT) vec_axpy(VecSpan v, typename VT_<CX>::T* x,
                                                const typename VT_<CX>::T* V, long long ldv, int nv,
                                                const typename VT_<CX>::T* c, int cstride, double* partial,
                                                unsigned* counter, VecOut o) {
  using T = typename VT_<CX>::T;
  extern __shared__ __align__(16) unsigned char csm[];
  __shared__ double red[kVW];
  T* cs = reinterpret_cast<T*>(csm);
  chain_begin();
  Range r;
  if (!block_range(v, r)) return;
  const auto* cg = c + (long long)r.seg * cstride;
  const int ns = min(nv, kStaged);
  for (int j = threadIdx.x; j < ns; j += kVT) cs[j] = cg[j];
  __syncthreads();
  double s2 = 0.0;
  for (long long i = r.lo + threadIdx.x; i < r.hi; i += kVT) {
    T a = x[i];
    int j = 0;
    for (; j + kG <= ns; j += kG) {
      T t[kG];
#pragma unroll
      for (int u = 0; u < kG; ++u) t[u] = V[(j + u) * ldv + i];
#pragma unroll
      for (int u = 0; u < kG; ++u) a = sub_mul(a, cs[j + u], t[u]);
    }
    for (; j < ns; ++j) a = sub_mul(a, cs[j], V[j * ldv + i]);
    for (; j < nv; ++j) a = sub_mul(a, cg[j], V[j * ldv + i]);
    x[i] = a;
    s2 += vabs2(a);
  }
  if (!partial) return;
  s2 = warp_sum(s2);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = s2;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < kVW; ++k) t += red[k];
    partial[blockIdx.x] = t;
  }
  if (!last_block(counter, r) || w != 0) return;
  double t = 0.0;
#pragma unroll 4
  for (int p = l; p < r.count; p += 32) t += __ldcg(partial + r.first + p);
  t = warp_sum(t);
  if (l == 0) norm_out(o, r.seg, t);
}

// y = sum_j c[seg * cstride + j] V_j (real c); with a partial buffer also |y| (as VO_NORM)
template <bool CX>
__global__ void __launch_bounds__(kVT) vec_lincomb(VecSpan v, typename VT_<CX>::T* y,
                                                   const typename VT_<CX>::T* V, long long ldv, int nv,
                                                   const double* c, int cstride, double* partial, unsigned* counter,
                                                   VecOut o) {
  using T = typename VT_<CX>::T;
  extern __shared__ __align__(16) unsigned char csm[];
  __shared__ double red[kVW];
  double* cs = reinterpret_cast<double*>(csm);
  chain_begin();
  Range r;
  if (!block_range(v, r)) return;
  const auto* cg = c + (long long)r.seg * cstride;
  const int ns = min(nv, kStaged);
  for (int j = threadIdx.x; j < ns; j += kVT) cs[j] = cg[j];
  __syncthreads();
  double s2 = 0.0;
  for (long long i = r.lo + threadIdx.x; i < r.hi; i += kVT) {
    T a = vzero(T());
    int j = 0;
    for (; j + kG <= ns; j += kG) {
      T t[kG];
#pragma unroll
      for (int u = 0; u < kG; ++u) t[u] = V[(j + u) * ldv + i];
#pragma unroll
      for (int u = 0; u < kG; ++u) a = add_rmul(a, cs[j + u], t[u]);
    }
    for (; j < ns; ++j) a = add_rmul(a, cs[j], V[j * ldv + i]);
    for (; j < nv; ++j) a = add_rmul(a, cg[j], V[j * ldv + i]);
    y[i] = a;
    s2 += vabs2(a);
  }
  if (!partial) return;
  s2 = warp_sum(s2);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = s2;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < kVW; ++k) t += red[k];
    partial[blockIdx.x] = t;
  }
  if (!last_block(counter, r) || w != 0) return;
  double t = 0.0;
#pragma unroll 4
  for (int p = l; p < r.count; p += 32) t += __ldcg(partial + r.first + p);
  t = warp_sum(t);
  if (l == 0) norm_out(o, r.seg, t);
}

// y = x / scal[seg * sstride] (y2 too when given); values not above floor divide by 1
template <bool CX>
__global__ void __launch_bounds__(kVT) vec_div(VecSpan v, const typename VT_<CX>::T* x, typename VT_<CX>::T* y,
                                               typename VT_<CX>::T* y2, const double* scal, int sstride, double floor) {
  chain_begin();
  Range r;
  if (!block_range(v, r)) return;
  const double d = scal[(long long)r.seg * sstride];
  const double f = d <= floor ? 1.0 : 1.0 / d;
  for (long long i = r.lo + threadIdx.x; i < r.hi; i += kVT) {
    const auto t = rmul(x[i], f);
    y[i] = t;
    if (y2) y2[i] = t;
  }
}

}  // namespace

VecSpan vec_span(long long n, int max_blocks) {
  VecSpan v{};
  v.n = n;
  long long per = (n + max_blocks - 1) / max_blocks;
  per = (per + kVT - 1) / kVT * kVT;
  v.per = per > kVT ? per : kVT;
  v.nblk = (int)((n + v.per - 1) / v.per);
  if (v.nblk < 1) v.nblk = 1;
  v.nseg = 1;
  return v;
}

void launch_vec_dots(bool cplx, const VecSpan& v, const void* V, long long ldv, int nv, void* x, const void* u0,
                     const void* u1, const void* uc, double* partial, void* out, unsigned* counter, const VecOut& o,
                     cudaStream_t s) {
  if (nv <= 0 || v.nblk <= 0) return;
  if (cplx)
    launch_chained(vec_dots<true>, v.nblk, kVT, 0, s, v, (const double2*)V, ldv, nv, (double2*)x, (const double2*)u0,
                                          (const double2*)u1, (const double2*)uc, partial, (double2*)out, counter, o);
  else
    launch_chained(vec_dots<false>, v.nblk, kVT, 0, s, v, (const double*)V, ldv, nv, (double*)x, (const double*)u0,
                                           (const double*)u1, (const double*)uc, partial, (double*)out, counter, o);
}

void launch_vec_axpy(bool cplx, const VecSpan& v, void* x, const void* V, long long ldv, int nv, const void* c,
                     int cstride, double* partial, unsigned* counter, const VecOut& o, cudaStream_t s) {
  if (v.nblk <= 0) return;
  const size_t smem = std::min(nv, kStaged) * (cplx ? sizeof(double2) : sizeof(double));
  if (cplx)
    launch_chained(vec_axpy<true>, v.nblk, kVT, smem, s, v, (double2*)x, (const double2*)V, ldv, nv,
                   (const double2*)c, cstride, partial, counter, o);
  else
    launch_chained(vec_axpy<false>, v.nblk, kVT, smem, s, v, (double*)x, (const double*)V, ldv, nv,
                   (const double*)c, cstride, partial, counter, o);
}

void launch_vec_lincomb(bool cplx, const VecSpan& v, void* y, const void* V, long long ldv, int nv, const double* c,
                        int cstride, double* partial, unsigned* counter, const VecOut& o, cudaStream_t s) {
  if (v.nblk <= 0) return;
  const size_t smem = std::min(nv, kStaged) * sizeof(double);
  if (cplx)
    launch_chained(vec_lincomb<true>, v.nblk, kVT, smem, s, v, (double2*)y, (const double2*)V, ldv, nv, c, cstride,
                   partial, counter, o);
  else
    launch_chained(vec_lincomb<false>, v.nblk, kVT, smem, s, v, (double*)y, (const double*)V, ldv, nv, c, cstride,
                   partial, counter, o);
}

void launch_vec_div(bool cplx, const VecSpan& v, const void* x, void* y, void* y2, const double* scal, int sstride,
                    double floor, cudaStream_t s) {
  if (v.nblk <= 0) return;
  if (cplx)
    launch_chained(vec_div<true>, v.nblk, kVT, 0, s, v, (const double2*)x, (double2*)y, (double2*)y2, scal, sstride, floor);
  else
    launch_chained(vec_div<false>, v.nblk, kVT, 0, s, v, (const double*)x, (double*)y, (double*)y2, scal, sstride, floor);
}

}  // namespace sadmrg
