// gemm.cu -- grouped FP64 block-GEMM executor with deterministic split-K.
//
// A plan is a list of jobs (output blocks C, m x n) with accumulation lists of
// terms alpha * op(A) * op(B).  Work is cut into items of one output tile and a
// contiguous range of the job's concatenated reduction dimension (the k of all
// its terms laid end to end), so a matvec with a few large output blocks still
// fills all 148 SMs.  An item that covers the whole range writes C directly;
// otherwise it writes its partial tile to a workspace slot, and the last item of
// the tile to finish sums the slots in a fixed order -- results are bitwise
// reproducible and there is no separate reduction launch.
//
// The products run on the double-precision tensor path (mma.sync m8n8k4 .f64;
// tcgen05 has no f64 kind).  Every FP64 mma shape runs at the same 36.5-37
// TFLOP/s here (m8n8k4 at 8 warps per SM: 35.7), plain FMAs at 29.8, so the
// smallest shape costs nothing and lets a tile skip the 8 x 8 strips that lie
// outside its block.
#include <cuda_runtime.h>
#include <cstdint>
#include <mutex>

#include "kernels.cuh"
#include "ptx.cuh"

namespace sadmrg {

constexpr int kThreads = 128;

__device__ __forceinline__ void dmma884(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}
template <bool CX> struct GTile;
template <> struct GTile<false> {
  using T = double;
  static constexpr int BM = 64, BN = 64, BK = 16, PAD = 4;   // PAD: of a k-major row, see items_f64
};
template <> struct GTile<true> {
  using T = double2;
  static constexpr int BM = 64, BN = 32, BK = 8, PAD = 2;
};
constexpr int kF64Stages = 3;
template <bool CX>
struct GSmem {
  using G = GTile<CX>;
  static constexpr int SKA = G::BM + G::PAD, SKB = G::BN + G::PAD;   // k-major row strides
  static constexpr int SM = G::BK + 4;                               // m/n-major row stride
  static constexpr int ABUF = G::BM * SM > G::BK * SKA ? G::BM * SM : G::BK * SKA;
  static constexpr int BBUF = G::BN * SM > G::BK * SKB ? G::BN * SM : G::BK * SKB;
  static constexpr int bytes = kF64Stages * (ABUF + BBUF) * (int)sizeof(typename G::T);
};

template <bool B> struct BoolC { static constexpr bool value = B; };
__device__ __forceinline__ double gzero(double) { return 0.0; }
__device__ __forceinline__ double2 gzero(double2) { return make_double2(0.0, 0.0); }
__device__ __forceinline__ double gadd(double a, double b) { return a + b; }
__device__ __forceinline__ double2 gadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

__device__ __forceinline__ double gmul(double a, double f) { return a * f; }
__device__ __forceinline__ double2 gmul(double2 a, double f) { return make_double2(a.x * f, a.y * f); }
__device__ __forceinline__ double gconj(double a, int) { return a; }
__device__ __forceinline__ double2 gconj(double2 a, int on) { return make_double2(a.x, on ? -a.y : a.y); }
__device__ __forceinline__ double gscale(double a, double ar, double) { return a * ar; }
__device__ __forceinline__ double2 gscale(double2 a, double ar, double ai) {
  return make_double2(a.x * ar - a.y * ai, a.x * ai + a.y * ar);
}

// ---------------------------------------------------------------------------
// Split-K fixup, run by every thread of an item that wrote a partial tile: the last
// item of the tile to finish (per-tile atomic count) sums all its partial tiles in
// slot order -- the same order whichever item is last -- writes C and clears the count
// for the next launch.  All of a thread's loads of one slot are in flight together.
template <bool CX>
__device__ __forceinline__ void split_fixup(const WorkItem& it, typename GTile<CX>::T* C,
                                            const typename GTile<CX>::T* work, int* tile_cnt) {
  using T = typename GTile<CX>::T;
  constexpr int BM = GTile<CX>::BM, BN = GTile<CX>::BN, E = BM * BN / kThreads;
  static_assert(kThreads % BM == 0, "a thread keeps its row");
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&tile_cnt[it.red], 1) == it.nslot - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int r = threadIdx.x % BM, c0 = threadIdx.x / BM;
  constexpr int CS = kThreads / BM;                 // columns between a thread's elements
  if (r < it.mv) {
    T sum[E];
#pragma unroll
    for (int u = 0; u < E; ++u) sum[u] = gzero(T());
    for (int k = 0; k < it.nslot; ++k) {
      const T* W = work + (long long)(it.slot0 + k) * BM * BN + threadIdx.x;
#pragma unroll
      for (int u = 0; u < E; ++u)
        if (c0 + u * CS < it.nv) sum[u] = gadd(sum[u], __ldcg(W + u * kThreads));
    }
#pragma unroll
    for (int u = 0; u < E; ++u) {
      const int c = c0 + u * CS;
      if (c < it.nv) C[r + (long long)c * it.ldc] = gmul(sum[u], it.alpha);
    }
  }
  if (threadIdx.x == 0) tile_cnt[it.red] = 0;
}

// one element global -> shared, zero-filled instead when !ok (src must still be a valid address)
__device__ __forceinline__ void cp_elem(double* smem, const double* gmem, bool ok) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(ok ? 8 : 0));
}
__device__ __forceinline__ void cp_elem(double2* smem, const double2* gmem, bool ok) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(ok ? 16 : 0));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// ---------------------------------------------------------------------------
struct ItemArgs {             // what a launch is given (kernel parameters, read where needed)
  const WorkItem* items;
  const ItemSeg* segs;
  const int* mask;
  void* work;
  int* tile_cnt;
  Bases bases;
};

// This warp's quarter of one operand slab, global -> shared with cp.async, zero-filled
// past the block and past the slab's k up to the next multiple of 4 (8 x 8 strips and k
// steps of 4 that lie outside are neither copied nor read).  The slab is kept in the
// layout its global copy is contiguous in.  Out-of-range copies read nothing and are
// given the address of a valid element.
template <class T, int ROWS, int BK, int SK, int SM>
__device__ __forceinline__ void copy_slab(T* dst, const T* src, int ld, bool kmajor, int valid, int k0, int kt, int warp,
                                          int lane) {
  constexpr int NW = kThreads / 32;
  if (kmajor) {                        // element (r, k) at src[r + k ld] -> dst[k SK + r]
    const long long step = (long long)NW * ld;
#pragma unroll
    for (int h = 0; h < ROWS / 32; ++h) {
      if (h * 32 >= valid) break;
      const int r = lane + 32 * h;
      const bool ok = r < valid;
      T* d = dst + warp * SK + r;
      if (kt == BK) {
        const T* s = src + min(r, valid - 1) + (long long)(k0 + warp) * ld;
#pragma unroll
        for (int q = 0; q < BK / NW; ++q) {
          cp_elem(d + q * NW * SK, s, ok);
          s += step;
        }
      } else {
        const int kr = (kt + 3) & ~3;
#pragma unroll 1
        for (int k = warp; k < kr; k += NW) {
          cp_elem(d, src + min(r, valid - 1) + (long long)(k0 + min(k, kt - 1)) * ld, ok && k < kt);
          d += NW * SK;
        }
      }
    }
  } else {                             // element (r, k) at src[k + r ld] -> dst[r SM + k]
    constexpr int RP = 32 / BK, Q = ROWS / RP / NW;   // rows of one warp copy, copies of a warp
    const int k = lane % BK, r0 = warp * RP + lane / BK;
    const bool kok = k < kt;
    const T* s = src + k0 + min(k, kt - 1);
    T* d = dst + r0 * SM + k;
    if (valid == ROWS) {
      const long long step = (long long)(NW * RP) * ld;
      s += (long long)r0 * ld;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        cp_elem(d + q * NW * RP * SM, s, kok);
        s += step;
      }
    } else {
      const int r8 = (valid + 7) & ~7;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (q * NW * RP >= r8) break;
        const int r = q * NW * RP + r0;
        cp_elem(d + q * NW * RP * SM, s + (long long)min(r, valid - 1) * ld, kok && r < valid);
      }
    }
  }
}

// One item, by warps that own at most MT x NT strips each.
template <bool CX, int MT, int NT>
__device__ __forceinline__ void run_item(const ItemArgs& a, const WorkItem& it, typename GTile<CX>::T* smem) {
  using G = GTile<CX>;
  using S = GSmem<CX>;
  using T = typename G::T;
  constexpr int STAGES = kF64Stages, NP = CX ? 2 : 1, BK = G::BK;
  __shared__ double sh_ar[STAGES], sh_ai[STAGES];
  __shared__ int sh_flags[STAGES], sh_kt[STAGES];
  T* const As = smem;                        // STAGES x ABUF
  T* const Bs = smem + STAGES * S::ABUF;     // STAGES x BBUF
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = warp >> 1, wn = warp & 1;
  double acc[MT][NT][NP][2];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int p = 0; p < NP; ++p) acc[i][j][p][0] = acc[i][j][p][1] = 0.0;

  // the slab that is copied next: its segment, first k and width
  int seg = 0, k0 = 0;
  ItemSeg sg = a.segs[it.seg0], sn = a.segs[it.seg0 + min(1, it.nseg)];
  const T *A = nullptr, *B = nullptr;
  auto bind = [&]() {
    A = static_cast<const T*>(a.bases.p[sg.abuf]) + sg.aoff;
    B = static_cast<const T*>(a.bases.p[sg.bbuf]) + sg.boff;
  };
  bind();
  auto more = [&]() { return seg < it.nseg; };
  auto copy_a = [&](int st) {
    copy_slab<T, G::BM, BK, S::SKA, S::SM>(As + st * S::ABUF, A, sg.lda, !(sg.flags & TF_TA), it.mv, k0,
                                           min(BK, sg.k - k0), warp, lane);
    if (threadIdx.x == 0) {
      sh_ar[st] = sg.ar;
      sh_ai[st] = sg.ai;
      sh_flags[st] = sg.flags;
      sh_kt[st] = min(BK, sg.k - k0);
    }
  };
  auto copy_b = [&](int st) {                // ... and on to the next slab
    copy_slab<T, G::BN, BK, S::SKB, S::SM>(Bs + st * S::BBUF, B, sg.ldb, sg.flags & TF_TB, it.nv, k0,
                                           min(BK, sg.k - k0), warp, lane);
    k0 += BK;
    if (k0 >= sg.k) {
      k0 = 0;
      ++seg;
      sg = sn;
      sn = a.segs[it.seg0 + min(seg + 1, it.nseg)];   // a term is often one slab long: loaded one ahead
      bind();
    }
  };

  int issued = 0;
#pragma unroll 1
  for (int st = 0; st < STAGES - 1; ++st) {
    if (more()) {
      copy_a(st);
      copy_b(st);
      ++issued;
    }
    cp_async_commit();
  }
#pragma unroll 1
  for (int c = 0; c < issued; ++c) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    const int st = c % STAGES, sw = (c + STAGES - 1) % STAGES;
    const int fl = sh_flags[st], kt = sh_kt[st];
    const double ar = sh_ar[st], ai = CX ? sh_ai[st] : 0.0;
    // fragment addresses: element (row r, k) of the A slab at r * sr + k * sk, of B at c * sc + k * sq
    const int sr = (fl & TF_TA) ? S::SM : 1, sk = (fl & TF_TA) ? 1 : S::SKA;
    const int sc = (fl & TF_TB) ? 1 : S::SM, sq = (fl & TF_TB) ? S::SKB : 1;
    const T* as = As + st * S::ABUF + (wm * 8 + (lane >> 2)) * sr + (lane & 3) * sk;
    const T* bs = Bs + st * S::BBUF + (wn * 8 + (lane >> 2)) * sc + (lane & 3) * sq;
    // the products of one k step (4 deep); plain: no scaling or conjugation
    auto step = [&](auto plain) {
      T af[MT], bf[NT];
#pragma unroll
      for (int mi = 0; mi < MT; ++mi) {
        af[mi] = as[mi * 16 * sr];
        if constexpr (!decltype(plain)::value) af[mi] = gscale(gconj(af[mi], fl & TF_CA), ar, ai);
      }
#pragma unroll
      for (int ni = 0; ni < NT; ++ni) {
        bf[ni] = bs[ni * 16 * sc];
        if constexpr (!decltype(plain)::value) bf[ni] = gconj(bf[ni], fl & TF_CB);
      }
#pragma unroll
      for (int mi = 0; mi < MT; ++mi)
#pragma unroll
        for (int ni = 0; ni < NT; ++ni) {
          if constexpr (CX) {
            dmma884(acc[mi][ni][0][0], acc[mi][ni][0][1], af[mi].x, bf[ni].x);
            dmma884(acc[mi][ni][1][0], acc[mi][ni][1][1], af[mi].x, bf[ni].y);
          } else {
            dmma884(acc[mi][ni][0][0], acc[mi][ni][0][1], af[mi], bf[ni]);
          }
        }
      if constexpr (CX) {
#pragma unroll
        for (int mi = 0; mi < MT; ++mi)
#pragma unroll
          for (int ni = 0; ni < NT; ++ni) {
            dmma884(acc[mi][ni][0][0], acc[mi][ni][0][1], -af[mi].y, bf[ni].y);
            dmma884(acc[mi][ni][1][0], acc[mi][ni][1][1], af[mi].y, bf[ni].x);
          }
      }
      as += 4 * sk;
      bs += 4 * sq;
    };
    const bool plain = ar == 1.0 && ai == 0.0 && !(CX && (fl & (TF_CA | TF_CB)));
    const bool next = more();
    if (next) copy_a(sw);
    if (plain && kt == BK) {
#pragma unroll
      for (int k4 = 0; k4 < BK; k4 += 4) step(BoolC<true>());
    } else {
#pragma unroll 1
      for (int k4 = 0; k4 < kt; k4 += 4) step(BoolC<false>());
    }
    if (next) {
      copy_b(sw);
      ++issued;
    }
    cp_async_commit();
  }
  cp_async_wait<0>();
  const bool split = it.slot >= 0;
  const double alpha = split ? 1.0 : it.alpha;
  T* const C = static_cast<T*>(a.bases.p[it.cbuf]) + it.out;
  const int ldo = split ? G::BM : it.ldc;
  T* out = split ? static_cast<T*>(a.work) + (long long)it.slot * G::BM * G::BN : C;
  out += wm * 8 + (lane >> 2) + (long long)(wn * 8 + 2 * (lane & 3)) * ldo;
#pragma unroll
  for (int ni = 0; ni < NT; ++ni)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      T* o = out + (long long)(ni * 16 + e) * ldo;
      const bool in = (ni * 2 + wn) * 8 + 2 * (lane & 3) + e < it.nv;
#pragma unroll
      for (int mi = 0; mi < MT; ++mi) {
        T v;
        if constexpr (CX) v = make_double2(acc[mi][ni][0][e], acc[mi][ni][1][e]);
        else v = acc[mi][ni][0][e];
        if (in && (mi * 2 + wm) * 8 + (lane >> 2) < it.mv) o[mi * 16] = gmul(v, alpha);
      }
    }
  if (split) split_fixup<CX>(it, C, static_cast<const T*>(a.work), a.tile_cnt);
}

// The item kernel, real (64 x 64 tiles, slabs of 16 k) and complex (64 x 32, 8): slabs
// copied global -> shared with cp.async, STAGES-1 in flight while the tensor cores
// consume one, three CTAs per SM hiding each other's barriers.
//
// A full slab is 1024 cycles of an SM's FP64 tensor path against 16 KB of operands, so
// the bound is that path, if the copies' instructions stay few: blocks start at any
// element and have odd leading dimensions, so copies are of one element, and with 64-bit
// addresses formed per element 9 instructions were issued per mma (the path 63% busy on
// full tiles).  Here a warp steps one address through its quarter of a slab, and the
// segment after the current one is loaded ahead.
//
// Blocks are 1 to some hundreds wide and rarely multiples of 64, so the tile is cut into
// 8 x 8 strips dealt to the warps in turn (warp row wm takes row strips wm, wm + 2, ...;
// columns alike), and the item is compiled for 1, 2 or 4 (complex: 1 or 2 column) strips
// per warp: on 8..512 log-uniform blocks whole 64 x 64 tiles are 1.55 times the useful
// products.
//
// Measured (one H_eff*psi, graph replay): SU(2) D = 512 bond 145 -> 83 us, SU(2) ladder
// centre 274 -> 217, SU(2) D = 1500 bond 1594 -> 1114 (24.6 TFLOP/s), U(1) D = 64 bond
// 37 -> 13, complex U(1) D = 1024 bond 2351 -> 1219 (27.1 TFLOP/s).  Tried and slower: a
// predicate on each mma instead of compiled strip counts (2x); one copying warp beside
// four multiplying ones (it issues at one warp's rate: 90 us at D = 512); that with
// persistent CTAs and both stages in one launch (130 us).
template <bool CX>
__global__ void __launch_bounds__(kThreads, 3) items_f64(const __grid_constant__ ItemArgs args) {
  using T = typename GTile<CX>::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chain_begin();
  const WorkItem it = args.items[blockIdx.x];
  if (args.mask && !args.mask[it.tag]) return;   // instance switched off for this launch
  T* const smem = reinterpret_cast<T*>(smem_raw);
  const int mt = (it.mv + 15) >> 4, nt = (it.nv + 15) >> 4;   // strips per warp, at most
  if (nt <= 1) {
    if (mt <= 1) run_item<CX, 1, 1>(args, it, smem);
    else if (mt <= 2) run_item<CX, 2, 1>(args, it, smem);
    else run_item<CX, 4, 1>(args, it, smem);
  } else if (CX || nt <= 2) {
    if (mt <= 1) run_item<CX, 1, 2>(args, it, smem);
    else if (mt <= 2) run_item<CX, 2, 2>(args, it, smem);
    else run_item<CX, 4, 2>(args, it, smem);
  } else if constexpr (!CX) {
    if (mt <= 1) run_item<CX, 1, 4>(args, it, smem);
    else if (mt <= 2) run_item<CX, 2, 4>(args, it, smem);
    else run_item<CX, 4, 4>(args, it, smem);
  }
}

int gemm_tile_m(bool cplx) { return cplx ? GTile<true>::BM : GTile<false>::BM; }
int gemm_tile_n(bool cplx) { return cplx ? GTile<true>::BN : GTile<false>::BN; }

template <bool CX>
static void launch_items_t(const ItemArgs& a, int nitems, cudaStream_t s) {
  static unsigned char attr[kMaxDevices] = {0};
  ensure_smem_attr((const void*)items_f64<CX>, GSmem<CX>::bytes, attr);
  launch_chained(items_f64<CX>, nitems, kThreads, GSmem<CX>::bytes, s, a);
}

void launch_items(bool cplx, const WorkItem* items, const ItemSeg* segs, int nitems, const Bases& b, void* work,
                  int* tile_cnt, const int* mask, cudaStream_t s) {
  if (nitems <= 0) return;
  const ItemArgs a{items, segs, mask, work, tile_cnt, b};
  if (cplx) launch_items_t<true>(a, nitems, s);
  else launch_items_t<false>(a, nitems, s);
}

// ---------------------------------------------------------------------------
// Fixed scratch for the allocation-free H_eff*psi entry point.  It lives for the
// life of the process on every device that loads the library.  Host code must not
// use the symbol's host-side name as a device address: the device address is
// looked up once per device with cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

int noalloc_scratch(void** ptr) {
  static std::mutex mu;
  static void* cache[kMaxDevices] = {nullptr};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= kMaxDevices) return (int)cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> g(mu);
  if (!cache[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return (int)e;
    cache[dev] = p;
  }
  *ptr = cache[dev];
  return 0;
}


}  // namespace sadmrg
