// tridiag.cu -- the lowest eigenpair of many small symmetric tridiagonal matrices.
//
// A batched Lanczos diagonalises one tridiagonal per instance at every check point
// (replaces LAPACK dstev, src/dmrg_inst.cpp:1216-1231).  One warp per matrix runs the
// implicit QL of tridiag_eig (dmrg.cpp) with the same operations and roundings in the same
// order and one hypot (hypot.hpp), so the eigenvalues and vectors are those of the host's
// solver to the last bit (but for the rare quotient named at `rotation`): the sign of a
// vector depends on how often an almost converged coupling is swept, which the roundings
// decide.
//
// The time is the chain of a rotation, 0.2 us.  All lanes compute it, and each lane
// rotates its own rows of the eigenvectors in shared memory while the next one is on its
// way.  64 matrices of 32 / 40 / 64 rows: 0.29 / 0.52 / 1.4 ms; the host takes 0.04 us a
// rotation, but one matrix after another (64 of 40 rows: 6 ms).
#include <cuda_runtime.h>
#include <algorithm>

#include "common.hpp"
#include "hypot.hpp"
#include "kernels.cuh"
#include "ptx.cuh"

namespace sadmrg {
namespace {

using rn::add;
using rn::mul;
using rn::sub;

// r = hypot(f, g), s = f / r, c = g / r.  In the usual range without CUDA's division and
// square root after one another (0.39 us a rotation, 0.21 like this): from one inverse
// square root y of x^2 + y^2, the square root and the quotients by Markstein's final
// corrections (IBM J. Res. Dev. 34, 1990).  They round as the exact results do but where an
// exact quotient lies within about 2^-52 of an ulp from halfway between two numbers (so does
// the correction of h, which is below an ulp of it): one in some 10^15.
__device__ __forceinline__ void rotation(double f, double g, double& r, double& s, double& c) {
  const double af = fabs(f), ag = fabs(g), x = fmax(af, ag), y = fmin(af, ag);
  if (y >= rn::kHypotLo && x <= rn::kHypotHi) {
    const double q = add(mul(x, x), mul(y, y)), i0 = rsqrt(q), h0 = mul(q, i0);
    const double h = fma(fma(-h0, h0, q), mul(0.5, i0), h0);
    const double t = sub(h, y), u = sub(h, x);
    const double n1 = add(mul(x, fma(2.0, t, -x)), mul(fma(-2.0, sub(x, y), t), t));
    const double n2 = add(mul(u, mul(2.0, fma(-2.0, y, x))), add(mul(fma(4.0, u, -y), y), mul(u, u)));
    r = sub(h, mul(h <= mul(2.0, y) ? n1 : n2, mul(0.5, i0)));
    const double ir = fma(fma(-r, i0, 1.0), i0, i0), s0 = mul(f, ir), c0 = mul(g, ir);
    s = fma(fma(-s0, r, f), ir, s0);
    c = fma(fma(-c0, r, g), ir, c0);
  } else {
    r = rn::hypot(f, g);
    s = rn::div(f, r);
    c = rn::div(g, r);
  }
}

// first m in [l, n - 1) whose coupling is negligible, else n - 1 (whole warp)
__device__ __forceinline__ int split_at(const double* d, const double* e, int l, int n) {
  const int lane = threadIdx.x;
  for (int m0 = l; m0 < n - 1; m0 += 32) {
    const int m = m0 + lane;
    bool small = false;
    if (m < n - 1) small = fabs(e[m]) <= mul(2.220446049250313e-16, add(fabs(d[m]), fabs(d[m + 1])));
    const unsigned b = __ballot_sync(0xffffffffu, small);
    if (b) return m0 + __ffs(b) - 1;
  }
  return n - 1;
}

// NR: rows of the eigenvectors per lane
template <int NR>
__global__ void __launch_bounds__(32) tridiag_lowest_kernel(int ns, const int* nn, int nmax, const double* a,
                                                            const double* b, double* z0, int zstride, double* e0,
                                                            int* status) {
  extern __shared__ double sm[];
  chain_begin();
  const int s = blockIdx.x, n = nn[s], lane = threadIdx.x;
  if (n <= 0) return;
  double* d = sm;               // a of row i: a[i * ns + s]; coupling of i and i + 1: b[(i + 1) * ns + s]
  double* e = d + n;
  double* z = e + n;            // column-major, n x n
  for (int i = lane; i < n; i += 32) {
    d[i] = a[(size_t)i * ns + s];
    e[i] = i + 1 < n ? b[(size_t)(i + 1) * ns + s] : 0.0;
  }
  for (int i = lane; i < n * n; i += 32) z[i] = i / n == i % n ? 1.0 : 0.0;
  __syncwarp();
  bool ok = true;
  for (int l = 0; l < n && ok; ++l) {
    for (int iter = 0;; ++iter) {
      const int m = split_at(d, e, l, n);
      if (m == l) break;
      if (iter == 100) {
        ok = false;
        break;
      }
      const double el = e[l], dl = d[l];
      double g = rn::div(sub(d[l + 1], dl), mul(2.0, el));
      const double r0 = rn::hypot(g, 1.0);
      g = add(sub(d[m], dl), rn::div(el, add(g, g >= 0.0 ? r0 : -r0)));
      double sn = 1.0, cc = 1.0, pp = 0.0;
      double col[NR];           // the eigenvectors' column i + 1
#pragma unroll
      for (int u = 0; u < NR; ++u) col[u] = lane + 32 * u < n ? z[m * n + lane + 32 * u] : 0.0;
      double dn = d[m], en = e[m - 1];
      int i = m - 1;
      bool deflated = false;
      for (; i >= l; --i) {
        const double f = mul(sn, en), bb = mul(cc, en), di1 = dn;
        dn = d[i];
        if (i > l) en = e[i - 1];
        double r, s1, c1;
        rotation(f, g, r, s1, c1);
        __syncwarp();
        if (lane == 0) e[i + 1] = r;
        if (r == 0.0) {
          if (lane == 0) {
            d[i + 1] = sub(di1, pp);
            e[m] = 0.0;
          }
          deflated = true;
          break;
        }
        sn = s1;
        cc = c1;
        g = sub(di1, pp);
        const double t = add(mul(sub(dn, g), sn), mul(mul(2.0, cc), bb));
        pp = mul(sn, t);
        if (lane == 0) d[i + 1] = add(g, pp);
        g = sub(mul(cc, t), bb);
#pragma unroll
        for (int u = 0; u < NR; ++u)
          if (lane + 32 * u < n) {
            const double zi = z[i * n + lane + 32 * u], f1 = col[u];
            z[(i + 1) * n + lane + 32 * u] = add(mul(sn, zi), mul(cc, f1));
            col[u] = sub(mul(cc, zi), mul(sn, f1));
          }
      }
#pragma unroll
      for (int u = 0; u < NR; ++u)
        if (lane + 32 * u < n) z[(i + 1) * n + lane + 32 * u] = col[u];
      __syncwarp();
      if (!deflated && lane == 0) {
        d[l] = sub(d[l], pp);
        e[l] = g;
        e[m] = 0.0;
      }
      __syncwarp();
    }
  }
  int lo = 0;
  for (int i = 1; i < n; ++i)
    if (d[i] < d[lo]) lo = i;
  for (int i = lane; i < nmax; i += 32) z0[(size_t)s * zstride + i] = ok && i < n ? z[lo * n + i] : 0.0;
  if (lane == 0) {
    e0[s] = d[lo];
    if (!ok) *status = 1;
  }
}

size_t smem_of(int n) { return sizeof(double) * ((size_t)n * n + 2 * (size_t)n); }

template <int NR>
void launch(int ns, const int* n, int nmax, const double* a, const double* b, double* z0, int zstride, double* e0,
            int* status, cudaStream_t s) {
  // the limit belongs to the kernel, for every thread that launches it: its largest size, once
  static unsigned char attr[kMaxDevices] = {0};
  ensure_smem_limit((const void*)tridiag_lowest_kernel<NR>, (int)smem_of(32 * NR), attr);
  launch_chained(tridiag_lowest_kernel<NR>, ns, 32, smem_of(nmax), s, ns, n, nmax, a, b, z0, zstride, e0, status);
  SADMRG_CUDA(cudaGetLastError());
}

}  // namespace

void launch_tridiag_lowest(int ns, const int* n, int nmax, const double* a, const double* b, double* z0, int zstride,
                           double* e0, int* status, cudaStream_t s) {
  if (ns <= 0 || nmax <= 0) return;
  SADMRG_REQUIRE(nmax <= kTridiagMax, SADMRG_ERR_LIMIT, "tridiagonal: too many rows for the device solver");
  if (nmax <= 32) launch<1>(ns, n, nmax, a, b, z0, zstride, e0, status, s);
  else if (nmax <= 64) launch<2>(ns, n, nmax, a, b, z0, zstride, e0, status, s);
  else launch<4>(ns, n, nmax, a, b, z0, zstride, e0, status, s);
}

}  // namespace sadmrg
