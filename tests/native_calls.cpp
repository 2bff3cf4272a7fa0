// native_calls.cpp -- test infrastructure: C entries to functions of the library that its
// C ABI has no call for (built by native.py, linked against libsadmrg_b200.so).  A call
// that throws returns 1.
#include <cuda_runtime.h>
#include <vector>

#include "hypot.hpp"
#include "kernels.cuh"

namespace sadmrg {
void tridiag_eig(int n, std::vector<double>& d, std::vector<double> e, std::vector<double>& z);
}
using namespace sadmrg;

template <class F>
static int call(F f) {
  try {
    f();
    return 0;
  } catch (...) {
    return 1;
  }
}

extern "C" {

void nc_hypot(long long n, const double* a, const double* b, double* out) {
  for (long long i = 0; i < n; ++i) out[i] = rn::hypot(a[i], b[i]);
}

// d: n diagonal, e: n - 1 couplings; the lowest eigenvalue and its vector
int nc_tridiag_host(int n, const double* d, const double* e, double* e0, double* z0) {
  return call([&] {
    std::vector<double> dd(d, d + n), ee(e, e + (n > 1 ? n - 1 : 0)), z;
    tridiag_eig(n, dd, ee, z);
    *e0 = dd[0];
    for (int i = 0; i < n; ++i) z0[i] = z[i];
  });
}

int nc_tridiag_device(int ns, const int* n, int nmax, const double* a, const double* b, double* z0, int zstride,
                      double* e0, int* status, void* stream) {
  return call([&] {
    launch_tridiag_lowest(ns, n, nmax, a, b, z0, zstride, e0, status, static_cast<cudaStream_t>(stream));
  });
}

// one segment of n elements: x -= sum_j c_j V_j and its norm
int nc_axpy(int cplx, long long n, void* x, const void* V, int nv, const void* c, double* partial, unsigned* counter,
            double* norm, void* stream) {
  return call([&] {
    VecOut o;
    o.op = VO_NORM;
    o.scal = norm;
    launch_vec_axpy(cplx != 0, vec_span(n, 592), x, V, n, nv, c, 0, partial, counter, o,
                    static_cast<cudaStream_t>(stream));
  });
}
// y = sum_j c_j V_j (real c) and its norm
int nc_lincomb(int cplx, long long n, void* y, const void* V, int nv, const double* c, double* partial,
               unsigned* counter, double* norm, void* stream) {
  return call([&] {
    VecOut o;
    o.op = VO_NORM;
    o.scal = norm;
    launch_vec_lincomb(cplx != 0, vec_span(n, 592), y, V, n, nv, c, 0, partial, counter, o,
                       static_cast<cudaStream_t>(stream));
  });
}


// SVD of column-major blocks m[j] x n[j] lying back to back in a; work, vmat and sv hold
// max x min, min x min and min elements per block, back to back.  The sweeps, -1, or -2.
int nc_jacobi(int cplx, const void* a, void* work, void* vmat, double* sv, int nj, const int* m, const int* n,
              int precondition, int stream_rows, int block) {
  int sweeps = -2;
  call([&] {
    std::vector<SvdJob> jobs(nj);
    long long ao = 0, wo = 0, vo = 0, so = 0;
    for (int j = 0; j < nj; ++j) {
      const int R = m[j] < n[j] ? n[j] : m[j], C = m[j] < n[j] ? m[j] : n[j];
      jobs[j] = {ao, wo, vo, so, m[j], n[j], m[j] < n[j] ? 1 : 0};
      ao += (long long)m[j] * n[j];
      wo += (long long)R * C;
      vo += (long long)C * C;
      so += C;
    }
    sweeps = run_jacobi_svd(cplx != 0, a, work, vmat, sv, jobs, 60, nullptr, nullptr, precondition, stream_rows, block);
  });
  return sweeps;
}

}  // extern "C"
