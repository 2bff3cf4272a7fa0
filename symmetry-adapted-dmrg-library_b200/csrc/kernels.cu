// kernels.cu -- sm_100a kernels for the two-site DMRG hot path.
//
//  Block utilities: segment axpy, block transpose, fuse fill, SVD gather, scaling.
//  (The grouped block-GEMM executors are in gemm.cu and umma.cu, the Krylov vector
//  kernels in krylov.cu, the block SVD in svd.cu.)
#include <cuda_runtime.h>
#include <cstdio>

#include "kernels.cuh"
#include "ptx.cuh"

namespace sadmrg {

// --------------------------------------------------------------------------
// block utilities
template <bool CPLX>
__global__ void seg_axpy_kernel(void* y, const void* x, const Seg* segs) {
  chain_begin();
  const Seg sg = segs[blockIdx.x];
  const long long stride = (long long)blockDim.x * gridDim.y;
  for (long long i = (long long)blockIdx.y * blockDim.x + threadIdx.x; i < sg.n; i += stride) {
    if (CPLX) {
      const double2 v = static_cast<const double2*>(x)[sg.soff + i];
      double2& o = static_cast<double2*>(y)[sg.doff + i];
      o.x += v.x * sg.ar - v.y * sg.ai;
      o.y += v.x * sg.ai + v.y * sg.ar;
    } else {
      static_cast<double*>(y)[sg.doff + i] += sg.ar * static_cast<const double*>(x)[sg.soff + i];
    }
  }
}

void launch_seg_axpy(bool cplx, void* y, const void* x, const Seg* segs, int nseg, cudaStream_t s) {
  if (nseg <= 0) return;
  dim3 grid(nseg, 16);
  if (cplx) launch_chained(seg_axpy_kernel<true>, grid, 256, 0, s, y, x, segs);
  else launch_chained(seg_axpy_kernel<false>, grid, 256, 0, s, y, x, segs);
}

template <class T>
__global__ void block_transpose_kernel(T* dst, const T* src, const Transp* jobs) {
  chain_begin();
  __shared__ T tile[32][33];
  const Transp tj = jobs[blockIdx.x];
  const int tr = (tj.rows + 31) / 32, tc = (tj.cols + 31) / 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  for (int tIdx = blockIdx.y; tIdx < tr * tc; tIdx += gridDim.y) {
    const int bi = (tIdx % tr) * 32, bj = (tIdx / tr) * 32;
    for (int k = ty; k < 32; k += 8) {
      const int r = bi + tx, c = bj + k;
      if (r < tj.rows && c < tj.cols) tile[k][tx] = src[tj.soff + r + (long long)c * tj.rows];
    }
    __syncthreads();
    for (int k = ty; k < 32; k += 8) {
      const int r = bj + tx, c = bi + k;  // dst is cols x rows
      if (r < tj.cols && c < tj.rows) dst[tj.doff + r + (long long)c * tj.cols] = tile[tx][k];
    }
    __syncthreads();
  }
}

void launch_block_transpose(bool cplx, void* dst, const void* src, const Transp* t, int nt, cudaStream_t s) {
  if (nt <= 0) return;
  dim3 grid(nt, 32);
  if (cplx) launch_chained(block_transpose_kernel<double2>, grid, 256, 0, s, (double2*)dst, (const double2*)src, t);
  else launch_chained(block_transpose_kernel<double>, grid, 256, 0, s, (double*)dst, (const double*)src, t);
}

// leg permutation of 3-leg blocks: one block of threads per tensor block, every
// destination element gathered from its source position (the tensors this serves,
// projected lower states of an excited-state sweep, are small)
template <class T>
__global__ void permute3_kernel(T* dst, const T* src, const Perm3* jobs) {
  chain_begin();
  const Perm3 J = jobs[blockIdx.x];
  const long long nd0 = J.d[J.p[0]], nd1 = J.d[J.p[1]], n = (long long)J.d[0] * J.d[1] * J.d[2];
  const long long st[3] = {1, J.d[0], (long long)J.d[0] * J.d[1]};   // source strides
  for (long long e = threadIdx.x + (long long)blockIdx.y * blockDim.x; e < n; e += (long long)blockDim.x * gridDim.y) {
    const long long i0 = e % nd0, i1 = (e / nd0) % nd1, i2 = e / (nd0 * nd1);
    dst[J.doff + e] = src[J.soff + i0 * st[J.p[0]] + i1 * st[J.p[1]] + i2 * st[J.p[2]]];
  }
}

void launch_permute3(bool cplx, void* dst, const void* src, const Perm3* t, int nt, cudaStream_t s) {
  if (nt <= 0) return;
  dim3 grid(nt, 8);
  if (cplx) launch_chained(permute3_kernel<double2>, grid, 256, 0, s, (double2*)dst, (const double2*)src, t);
  else launch_chained(permute3_kernel<double>, grid, 256, 0, s, (double*)dst, (const double*)src, t);
}

template <bool CPLX>
__global__ void fuse_fill_kernel(void* data, const FuseFill* f) {
  chain_begin();
  const FuseFill ff = f[blockIdx.x];
  const long long plane = (long long)ff.d0 * ff.d1;
  for (long long e = threadIdx.x; e < plane; e += blockDim.x) {
    const int a = (int)(e % ff.d0), b = (int)(e / ff.d0);
    const long long idx = ff.off + a + (long long)b * ff.d0 + (long long)(ff.pos + b * ff.d0 + a) * plane;
    if (CPLX) static_cast<double2*>(data)[idx] = make_double2(1.0, 0.0);
    else static_cast<double*>(data)[idx] = 1.0;
  }
}

void launch_fuse_fill(bool cplx, void* data, const FuseFill* f, int nf, cudaStream_t s) {
  if (nf <= 0) return;
  if (cplx) launch_chained(fuse_fill_kernel<true>, nf, 256, 0, s, data, f);
  else launch_chained(fuse_fill_kernel<false>, nf, 256, 0, s, data, f);
}

template <bool CPLX>
__global__ void gather_kernel(void* dst, const void* src, const double* w, const int* perm, const Gather* g) {
  chain_begin();
  const Gather G = g[blockIdx.x];
  const long long total = (long long)G.rows * G.kept;
  for (long long e = (long long)blockIdx.y * blockDim.x + threadIdx.x; e < total; e += (long long)blockDim.x * gridDim.y) {
    const int r = (int)(e % G.rows), c = (int)(e / G.rows);
    const double wv = w[G.woff + c];
    double sc = 1.0;
    if (G.p != 0.0) sc = (wv > 0.0) ? pow(wv, G.p) : 0.0;
    const long long si = G.soff + r + (long long)perm[G.poff + c] * G.lds;
    if (CPLX) {
      double2 v = static_cast<const double2*>(src)[si];
      if (G.conj) v.y = -v.y;
      v.x *= sc; v.y *= sc;
      static_cast<double2*>(dst)[G.doff + e] = v;
    } else {
      static_cast<double*>(dst)[G.doff + e] = static_cast<const double*>(src)[si] * sc;
    }
  }
}

void launch_gather(bool cplx, void* dst, const void* src, const double* w, const int* perm, const Gather* g, int ng,
                   cudaStream_t s) {
  if (ng <= 0) return;
  dim3 grid(ng, 8);
  if (cplx) launch_chained(gather_kernel<true>, grid, 256, 0, s, dst, src, w, perm, g);
  else launch_chained(gather_kernel<false>, grid, 256, 0, s, dst, src, w, perm, g);
}

template <bool CPLX>
__global__ void scale_kernel(void* x, double ar, double ai, long long n) {
  chain_begin();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)blockDim.x * gridDim.x) {
    if (CPLX) {
      const double2 v = static_cast<double2*>(x)[i];
      static_cast<double2*>(x)[i] = make_double2(v.x * ar - v.y * ai, v.x * ai + v.y * ar);
    } else {
      static_cast<double*>(x)[i] *= ar;
    }
  }
}

void launch_scale(bool cplx, void* x, double ar, double ai, long long n, cudaStream_t s) {
  if (n <= 0) return;
  const int blocks = (int)min((n + 255) / 256, 148LL * 8);
  if (cplx) launch_chained(scale_kernel<true>, blocks, 256, 0, s, x, ar, ai, n);
  else launch_chained(scale_kernel<false>, blocks, 256, 0, s, x, ar, ai, n);
}

// Reads bytes (a multiple of 16) of x; writes sink only when the xor of all
// words is a value no data here holds in practice, so the loads cannot be dropped.
__global__ void read_kernel(const uint4* __restrict__ x, long long n16, unsigned* sink) {
  unsigned acc = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += (long long)blockDim.x * gridDim.x) {
    const uint4 v = __ldcg(x + i);
    acc ^= v.x ^ v.y ^ v.z ^ v.w;
  }
  if (acc == 0x9e3779b9u && sink) *sink = acc;
}

void launch_read(const void* x, long long bytes, unsigned* sink, cudaStream_t s) {
  if (bytes < 16) return;
  read_kernel<<<148 * 8, 256, 0, s>>>(static_cast<const uint4*>(x), bytes / 16, sink);
}

template <bool CPLX>
__global__ void fill_kernel(void* x, double vr, double vi, long long n) {
  chain_begin();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)blockDim.x * gridDim.x) {
    if (CPLX) static_cast<double2*>(x)[i] = make_double2(vr, vi);
    else static_cast<double*>(x)[i] = vr;
  }
}

void launch_fill(bool cplx, void* x, double vr, double vi, long long n, cudaStream_t s) {
  if (n <= 0) return;
  const int blocks = (int)min((n + 255) / 256, 148LL * 8);
  if (cplx) launch_chained(fill_kernel<true>, blocks, 256, 0, s, x, vr, vi, n);
  else launch_chained(fill_kernel<false>, blocks, 256, 0, s, x, vr, vi, n);
}

}  // namespace sadmrg
