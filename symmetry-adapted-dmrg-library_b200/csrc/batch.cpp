// batch.cpp -- many independent two-site problems solved together.
//
// Each instance is a frozen H_eff plan (one centre step of its own chain).  The
// plans are merged into one: instance i's psi / H psi segment starts at seg[i]
// of one long vector, its operators and stage-0 products at their own offsets of
// one operator buffer and one scratch buffer, so every batched matvec is one
// launch per stage for all instances (mma.sync for FP64, tcgen05 for 3xTF32).
// The Krylov recurrence runs segment-wise (krylov.cu: every segment cut into
// ranges, a block each), and every instance has its own tridiagonal problem; the
// recurrence and its checks are those of lanczos1 (Lanczos::lanczos1,
// src/dmrg_inst.cpp:1286-1348), applied per instance.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "dmrg.hpp"

namespace sadmrg {

namespace {
template <class S> constexpr bool kCxB = ScalarInfo<S>::cplx;
}

template <class S>
void HeffBatch<S>::add(Ctx& c, const HeffPlan<S>& H) {
  SADMRG_REQUIRE(!ready, SADMRG_ERR_STATE, "batch: already finalized");
  Part p;
  p.job_terms = H.plan.job_terms;
  p.jobs = H.plan.jobs;
  p.job_stage = H.plan.job_stage;
  p.scratch = H.plan.scratch_elems;
  p.n = H.n;
  p.flops = H.flops;
  // The operators are copied on the batch's stream and the copy is awaited here:
  // the instance's buffers belong to its own handle (and stream), which the
  // caller may destroy as soon as this returns.
  const size_t bytes = H.opsbuf ? H.opsbuf->bytes() : 0;
  if (bytes) {
    p.ops = std::make_shared<DevBuf>(bytes, c.stream);
    SADMRG_CUDA(cudaMemcpyAsync(p.ops->get(), H.opsbuf->get(), bytes, cudaMemcpyDeviceToDevice, c.stream));
    SADMRG_CUDA(cudaStreamSynchronize(c.stream));
  }
  parts.push_back(std::move(p));
}

template <class S>
void HeffBatch<S>::finalize(Ctx& c) {
  SADMRG_REQUIRE(!ready, SADMRG_ERR_STATE, "batch: already finalized");
  SADMRG_REQUIRE(!parts.empty(), SADMRG_ERR_STATE, "batch: no instances");
  const int np = (int)parts.size();
  seg.assign(np + 1, 0);
  std::vector<long long> ooff(np + 1, 0), xoff(np + 1, 0);
  for (int i = 0; i < np; ++i) {
    seg[i + 1] = seg[i] + parts[i].n;
    ooff[i + 1] = ooff[i] + (long long)(parts[i].ops ? parts[i].ops->bytes() / sizeof(S) : 0);
    xoff[i + 1] = xoff[i] + parts[i].scratch;
  }
  HeffPlan<S>& M = merged;
  M.n = seg[np];
  M.opsbuf = std::make_shared<DevBuf>(sizeof(S) * std::max<long long>(ooff[np], 1), c.stream);
  for (int i = 0; i < np; ++i)
    if (parts[i].ops && ooff[i + 1] > ooff[i])
      SADMRG_CUDA(cudaMemcpyAsync(M.opsbuf->template as<S>() + ooff[i], parts[i].ops->get(),
                                  sizeof(S) * (ooff[i + 1] - ooff[i]), cudaMemcpyDeviceToDevice, c.stream));
  GemmPlan& P = M.plan;
  for (int i = 0; i < np; ++i) {
    const Part& q = parts[i];
    auto base = [&](int buf) -> long long { return buf == 2 ? ooff[i] : buf == 3 ? xoff[i] : seg[i]; };
    for (size_t j = 0; j < q.jobs.size(); ++j) {
      const GemmJob& J = q.jobs[j];
      const int nj = P.add_job(q.job_stage[j], J.cbuf, J.coff + base(J.cbuf), J.m, J.n, J.ldc);
      P.jobs[nj].tag = i;   // a masked matvec skips the jobs of converged instances
      for (const GemmTerm& t : q.job_terms[j])
        P.add_term(nj, t.abuf, t.aoff + base(t.abuf), t.lda, t.bbuf, t.boff + base(t.bbuf), t.ldb, t.k, t.flags,
                   t.ar, t.ai);
    }
    P.scratch_elems += q.scratch;
    M.flops += q.flops;
  }
  Bases cb{};
  cb.p[2] = M.opsbuf->get();
  P.finalize(c, kCxB<S>, /*mixed=*/true, &cb);
  M.scratch = std::make_shared<DevBuf>(sizeof(S) * std::max<long long>(P.scratch_elems, 1), c.stream);
  M.ntasks = (int)P.flat_terms.size();
  // ranges of the vector kernels: about 1024 of equal length over all segments (7 blocks
  // of 256 threads per SM), whole multiples of a block's threads
  long long per = (M.n + 1023) / 1024;
  per = std::max<long long>(256, (per + 255) / 256 * 256);
  std::vector<VecBlk> blk;
  std::vector<int> blk0(np + 1, 0);
  for (int i = 0; i < np; ++i) {
    for (long long lo = seg[i]; lo < seg[i + 1]; lo += per)
      blk.push_back(VecBlk{lo, (int)std::min(per, seg[i + 1] - lo), i});
    blk0[i + 1] = (int)blk.size();
  }
  nblk = (int)blk.size();
  const size_t bytes_blk = (sizeof(VecBlk) * blk.size() + 255) & ~size_t(255);
  d_blk = std::make_shared<DevBuf>(bytes_blk + sizeof(int) * blk0.size(), c.stream);
  if (nblk)
    SADMRG_CUDA(cudaMemcpyAsync(d_blk->get(), blk.data(), sizeof(VecBlk) * blk.size(), cudaMemcpyHostToDevice, c.stream));
  SADMRG_CUDA(cudaMemcpyAsync(d_blk->as<unsigned char>() + bytes_blk, blk0.data(), sizeof(int) * blk0.size(),
                              cudaMemcpyHostToDevice, c.stream));
  span = VecSpan{};
  span.blk = d_blk->as<VecBlk>();
  span.blk0 = reinterpret_cast<const int*>(d_blk->as<unsigned char>() + bytes_blk);
  span.nblk = nblk;
  span.nseg = np;
  span.n = M.n;
  SADMRG_CUDA(cudaStreamSynchronize(c.stream));
  parts.clear();   // the merged buffers hold everything now
  ready = true;
}

namespace {

// device and page-locked host work space of one batched Lanczos solve
template <class S>
struct BatchKrylov {
  Ctx& c;
  long long N;
  int ns, mlanc;                // segments, Krylov size
  VecSpan all;                  // every segment; the launches of a step and of a check mask it
  DevBuf ff, vh, dots, coef, beta, cdev, mask, norm, active, partial, counter;
  double* h_a = nullptr;        // a of step m, segment s: h_a[(m - 1) * ns + s]
  double* h_beta = nullptr;     // b: h_beta[m * ns + s]
  S* h_dots = nullptr;          // 2 per segment
  double* h_cdev = nullptr;     // Ritz coefficients (ns x (mlanc + 1))
  int* h_mask = nullptr;
  double* h_e0 = nullptr;       // lowest Ritz values
  int* h_n = nullptr;           // rows of the tridiagonals of a check, then their status
  int* h_active = nullptr;      // instances whose matvec work still runs (written only after a stream sync)
  BatchKrylov(Ctx& cc, const HeffBatch<S>& B, int ml) : c(cc), N(B.merged.n), ns(B.nseg()), mlanc(ml), all(B.span) {
    ff.alloc(sizeof(S) * N * (mlanc + 1), c.stream);
    vh.alloc(sizeof(S) * N * 2, c.stream);
    dots.alloc(sizeof(S) * (size_t)ns * (mlanc + 2), c.stream);
    coef.alloc(sizeof(S) * (size_t)ns * 2, c.stream);
    beta.alloc(sizeof(double) * (size_t)ns * (mlanc + 2), c.stream);
    cdev.alloc(sizeof(double) * (size_t)ns * (mlanc + 1), c.stream);
    mask.alloc(sizeof(int) * ns, c.stream);
    norm.alloc(sizeof(double) * ns, c.stream);
    active.alloc(sizeof(int) * ns, c.stream);
    partial.alloc(sizeof(S) * (size_t)std::max(all.nblk, 1) * (mlanc + 1), c.stream);
    counter.alloc(sizeof(unsigned) * ns, c.stream);
    SADMRG_CUDA(cudaMemsetAsync(beta.get(), 0, beta.bytes(), c.stream));
    SADMRG_CUDA(cudaMemsetAsync(counter.get(), 0, counter.bytes(), c.stream));
    SADMRG_CUDA(cudaMemsetAsync(norm.get(), 0, norm.bytes(), c.stream));
    // page-locked scalars, one allocation: the dots, which may be complex, first (16-byte
    // aligned), then doubles, then ints
    const size_t na = (size_t)ns * (mlanc + 1), nb = (size_t)ns * (mlanc + 2);
    void* pinned = nullptr;
    SADMRG_CUDA(cudaMallocHost(&pinned, sizeof(S) * 2 * ns + sizeof(double) * (2 * na + nb + ns) + sizeof(int) * (3 * (size_t)ns + 1)));
    h_dots = static_cast<S*>(pinned);
    h_a = reinterpret_cast<double*>(h_dots + 2 * ns);
    h_beta = h_a + na;
    h_cdev = h_beta + nb;
    h_e0 = h_cdev + na;
    h_mask = reinterpret_cast<int*>(h_e0 + ns);
    h_active = h_mask + ns;
    h_n = h_active + ns;
    // an instance without elements has no block to write its scalars: they read as zero
    std::memset(h_a, 0, sizeof(double) * (size_t)ns * (mlanc + 1));
    std::memset(h_beta, 0, sizeof(double) * (size_t)ns * (mlanc + 2));
    std::memset(static_cast<void*>(h_dots), 0, sizeof(S) * (size_t)ns * 2);
    std::fill(h_active, h_active + ns, 1);
    SADMRG_CUDA(cudaMemcpyAsync(active.get(), h_active, sizeof(int) * ns, cudaMemcpyHostToDevice, c.stream));
  }
  ~BatchKrylov() {
    cudaStreamSynchronize(c.stream);
    cudaFreeHost(h_dots);
  }
  S* F(int i) { return ff.as<S>() + (size_t)i * N; }
  VecSpan on(const DevBuf& m) const {   // the segments whose flag in m is set
    VecSpan v = all;
    v.active = m.as<int>();
    return v;
  }
  void mdot(const VecSpan& v, const S* V, int nv, const S* x, const VecOut& o, const S* u0 = nullptr,
            const S* u1 = nullptr) {
    launch_vec_dots(kCxB<S>, v, V, N, nv, const_cast<S*>(x), u0, u1, coef.get(), partial.as<double>(), dots.get(),
                    counter.as<unsigned>(), o, c.stream);
    ++c.launches;
  }
};

template <class S>
BatchStats batch_lanczos1(Ctx& c, const HeffBatch<S>& B, S* v, int mlanc, int prec) {
  constexpr bool CX = kCxB<S>;
  const HeffPlan<S>& H = B.merged;
  const int ns = B.nseg();
  const long long N = H.n;
  BatchKrylov<S> K(c, B, mlanc);
  const double tol = 1.e-6;
  BatchStats st;
  st.energy.assign(ns, 0.0);
  st.matvecs.assign(ns, 0);
  std::vector<char> done(ns, 0);
  // Converged instances are switched off in the matvec (their jobs skip all
  // work; their segments of the output keep stale values that nothing reads).
  auto matvec = [&](const S* in, S* out) {
    c.job_mask = K.active.template as<int>();
    try {
      H.apply(c, in, out, prec);
    } catch (...) {
      c.job_mask = nullptr;
      throw;
    }
    c.job_mask = nullptr;
    ++st.launches_matvec;
    for (int s = 0; s < ns; ++s)
      if (!done[s]) ++st.matvecs[s];
  };
  VecOut to_norm;
  to_norm.op = VO_NORM;
  to_norm.scal = K.norm.get();
  to_norm.sstride = 1;
  // Lowest Ritz pair of the masked segments, whose tridiagonals have K.h_n[s] <= nv rows
  // (0 elsewhere): the Ritz vectors into v and their norms.  Tridiagonals of at least
  // kTridiagDev instances are solved on the device (0.2 us a rotation, all at once), of
  // fewer on the host (0.04 us, one after another): 8 of 40 rows 0.52 ms against 0.8.
  constexpr int kTridiagDev = 8;
  std::vector<double> eig, z;
  auto ritz = [&](int nv) {
    int open = 0;
    for (int s = 0; s < ns; ++s) open += K.h_mask[s] != 0;
    K.h_n[ns] = 0;
    if (open >= kTridiagDev && nv <= kTridiagMax) {
      launch_tridiag_lowest(ns, K.h_n, nv, K.h_a, K.h_beta, K.cdev.template as<double>(), mlanc + 1, K.h_e0, K.h_n + ns,
                            c.stream);
      ++c.launches;
    } else {
      std::fill(K.h_cdev, K.h_cdev + (size_t)ns * (mlanc + 1), 0.0);
      for (int s = 0; s < ns; ++s) {
        const int m = K.h_n[s];
        if (m == 0) continue;
        eig.resize(m);
        std::vector<double> e(m, 0.0);
        for (int i = 0; i < m; ++i) eig[i] = K.h_a[(size_t)i * ns + s];
        for (int i = 0; i + 1 < m; ++i) e[i] = K.h_beta[(size_t)(i + 1) * ns + s];
        tridiag_eig(m, eig, e, z);
        K.h_e0[s] = eig[0];
        std::copy(z.begin(), z.begin() + m, K.h_cdev + (size_t)s * (mlanc + 1));
      }
      SADMRG_CUDA(cudaMemcpyAsync(K.cdev.get(), K.h_cdev, sizeof(double) * (size_t)ns * (mlanc + 1),
                                  cudaMemcpyHostToDevice, c.stream));
    }
    SADMRG_CUDA(cudaMemcpyAsync(K.mask.get(), K.h_mask, sizeof(int) * ns, cudaMemcpyHostToDevice, c.stream));
    launch_vec_lincomb(CX, K.on(K.mask), v, K.F(0), N, nv, K.cdev.template as<double>(), mlanc + 1,
                       K.partial.template as<double>(), K.counter.template as<unsigned>(), to_norm, c.stream);
    ++c.launches;
  };
  // Lanczos::check_eigenvector on the masked segments' Ritz vectors: normalise v (norms
  // below 1e-12 are left alone), |<v|Hv>| / |Hv|
  std::vector<double> ov(ns, 0.0);
  auto check = [&]() {
    S* vv = K.vh.template as<S>();
    S* hv = vv + N;
    const VecSpan m = K.on(K.mask);
    launch_vec_div(CX, m, v, v, vv, K.norm.template as<double>(), 1, 1e-12, c.stream);
    ++c.launches;
    matvec(vv, hv);
    VecOut o;
    o.op = VO_HOST;
    o.host = K.h_dots;
    o.hstride = 2;
    K.mdot(m, vv, 2, hv, o);
    SADMRG_CUDA(cudaStreamSynchronize(c.stream));
    if (K.h_n[ns]) throw Error(SADMRG_ERR_NUMERIC, "tridiagonal QL did not converge");
    for (int s = 0; s < ns; ++s) {
      if (!K.h_mask[s]) continue;
      const double prod = std::sqrt(std::fabs(real_of(K.h_dots[2 * s + 1])));
      ov[s] = prod > 0 ? std::abs(K.h_dots[2 * s]) / prod : 0.0;
    }
  };
  // F(0) = normalised v
  K.mdot(K.all, v, 1, v, to_norm);
  launch_vec_div(CX, K.all, v, K.F(0), nullptr, K.norm.template as<double>(), 1, 1e-12, c.stream);
  ++c.launches;

  int synced = 0;
  auto step = [&](int m) {
    const VecSpan act = K.on(K.active);
    double* bm = K.beta.template as<double>() + (size_t)m * ns;
    matvec(K.F(m - 1), K.F(m));
    VecOut o;
    o.op = VO_COEF;
    o.beta = bm - ns;
    o.bstride = 1;
    o.scal = K.coef.get();
    o.host = K.h_a + (size_t)(m - 1) * ns;
    o.hstride = 1;
    K.mdot(act, K.F(m - 1), 1, K.F(m), o);
    VecOut nb;
    nb.op = VO_NORM;
    nb.scal = bm;
    nb.sstride = 1;
    nb.host = K.h_beta + (size_t)m * ns;
    nb.hstride = 1;
    if (m >= 2) {
      K.mdot(act, K.F(0), m, K.F(m), VecOut{}, K.F(m - 2), K.F(m - 1));
      launch_vec_axpy(CX, act, K.F(m), K.F(0), N, m, K.dots.get(), m, K.partial.template as<double>(),
                      K.counter.template as<unsigned>(), nb, c.stream);
    } else {
      launch_vec_axpy(CX, act, K.F(m), K.F(m - 1), N, 1, K.coef.template as<S>() + 1, 2,
                      K.partial.template as<double>(), K.counter.template as<unsigned>(), nb, c.stream);
    }
    launch_vec_div(CX, act, K.F(m), K.F(m), nullptr, bm, 1, -1.0, c.stream);
    c.launches += 2;
  };
  auto sync_to = [&](int m, std::vector<int>& brk) {
    SADMRG_CUDA(cudaStreamSynchronize(c.stream));
    brk.assign(ns, 0);
    for (int s = 0; s < ns; ++s) {
      if (done[s]) continue;
      for (int j = synced + 1; j <= m; ++j) {
        if (!brk[s] && j >= 2 && K.h_beta[(size_t)j * ns + s] < tol) brk[s] = j;
      }
    }
    synced = m;
  };

  std::vector<int> brk;
  std::vector<int> finishing(ns, 0);
  step(1);
  if (mlanc > 2) {
    for (int m = 2; m < mlanc; ++m) {
      step(m);
      if (m % 4 != 0 && m != mlanc - 1) continue;
      sync_to(m, brk);
      bool any = false;
      std::fill(K.h_mask, K.h_mask + ns, 0);
      std::fill(K.h_n, K.h_n + ns, 0);
      for (int s = 0; s < ns; ++s) {
        finishing[s] = 0;
        if (done[s]) continue;
        if (!brk[s] && m % 4 != 0) continue;
        K.h_n[s] = brk[s] ? brk[s] : m;
        K.h_mask[s] = 1;
        finishing[s] = brk[s] ? 1 : 0;
        any = true;
      }
      if (!any) continue;
      ritz(m + 1);
      check();
      bool all = true, changed = false;
      for (int s = 0; s < ns; ++s) {
        if (K.h_mask[s] && (finishing[s] || std::fabs(ov[s] - 1.0) < c.lanczos_ov_tol)) {
          done[s] = 1;
          st.energy[s] = K.h_e0[s];
          K.h_active[s] = 0;
          changed = true;
        }
        if (!done[s]) all = false;
      }
      if (all) return st;
      if (changed)   // check() synchronised the stream, so h_active is not being read by an earlier copy
        SADMRG_CUDA(cudaMemcpyAsync(K.active.get(), K.h_active, sizeof(int) * ns, cudaMemcpyHostToDevice, c.stream));
    }
  }
  // instances still open after mlanc - 1 steps: one more matvec, then the Ritz vector
  const int last = mlanc > 2 ? mlanc - 1 : 1;
  matvec(K.F(last), K.F(last + 1));
  VecOut od;
  od.op = VO_HOST;
  od.host = K.h_dots;
  od.hstride = 1;
  K.mdot(K.on(K.active), K.F(last), 1, K.F(last + 1), od);
  SADMRG_CUDA(cudaStreamSynchronize(c.stream));
  std::fill(K.h_mask, K.h_mask + ns, 0);
  std::fill(K.h_n, K.h_n + ns, 0);
  for (int s = 0; s < ns; ++s) {
    if (done[s]) continue;
    K.h_a[(size_t)last * ns + s] = real_of(K.h_dots[s]);
    K.h_n[s] = last + 1;
    K.h_mask[s] = 1;
  }
  ritz(last + 1);
  check();
  for (int s = 0; s < ns; ++s)
    if (!done[s]) {
      done[s] = 1;
      st.energy[s] = K.h_e0[s];
    }
  return st;
}

}  // namespace

template <class S>
BatchStats batch_lanczos_solve(Ctx& c, const HeffBatch<S>& B, S* v, int mlanc, int prec) {
  SADMRG_REQUIRE(B.ready, SADMRG_ERR_STATE, "batch: not finalized");
  SADMRG_REQUIRE(mlanc >= 3, SADMRG_ERR_ARG, "batch lanczos: mlanc >= 3");
  if (prec == PREC_FP64) return batch_lanczos1<S>(c, B, v, mlanc, PREC_FP64);
  const double tol = c.lanczos_ov_tol;
  c.lanczos_ov_tol = std::max(tol, 1e-10);   // the split-precision phase stops no tighter (see lanczos_solve)
  BatchStats a;
  try {
    a = batch_lanczos1<S>(c, B, v, mlanc, prec);
  } catch (...) {
    c.lanczos_ov_tol = tol;
    throw;
  }
  c.lanczos_ov_tol = tol;
  BatchStats b = batch_lanczos1<S>(c, B, v, mlanc, PREC_FP64);   // FP64 restart
  for (size_t s = 0; s < b.matvecs.size(); ++s) b.matvecs[s] += a.matvecs[s];
  b.launches_matvec += a.launches_matvec;
  return b;
}

template struct HeffBatch<double>;
template struct HeffBatch<dcmplex>;
template BatchStats batch_lanczos_solve<double>(Ctx&, const HeffBatch<double>&, double*, int, int);
template BatchStats batch_lanczos_solve<dcmplex>(Ctx&, const HeffBatch<dcmplex>&, dcmplex*, int, int);

}  // namespace sadmrg
