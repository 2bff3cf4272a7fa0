// kernels.cuh -- device task formats and launchers.
//
// Every contraction on the hot path (H_eff*psi, environment updates, the
// projector products after the SVD) is lowered on the host to a list of dense
// sector GEMMs; one launch executes a whole list.  Operands are addressed as
// (base buffer id, element offset) so a plan built once per bond can be run on
// any psi / output vector by swapping base pointers.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <vector>

namespace sadmrg {

enum TermFlags : int { TF_TA = 1, TF_CA = 2, TF_TB = 4, TF_CB = 8 };
enum Precision : int { PREC_FP64 = 0, PREC_TF32X3 = 1 };
constexpr int kMaxBases = 8;

struct GemmTerm {             // alpha * op(A) * op(B), A: m x k, B: k x n after op
  long long aoff, boff;       // element offsets (elements of the scalar type)
  int abuf, bbuf;             // base buffer ids
  int lda, ldb, k, flags;
  double ar, ai;              // alpha (imaginary part ignored for real data)
};
struct GemmJob {              // C (m x n, column-major, ldc) = the sum of its terms
  long long coff;
  int cbuf, m, n, ldc;
  int t0, nt;
  int tag;                    // instance of a merged batch plan (0 otherwise): a launch given a mask
                              // skips every item of a job whose mask[tag] is 0
};
struct WorkItem {             // one output tile x a contiguous range of the job's concatenated k
  long long out;              // element offset of the tile's (0, 0) in C
  double alpha;               // C = alpha sum(terms)
  int cbuf, ldc, mv, nv;      // mv x nv: the tile's extent inside the block
  int tag;                    // as GemmJob::tag
  int seg0, nseg;             // its segments
  int slot;                   // < 0: write C directly; otherwise the partial-tile slot
  int red;                    // split items: their tile's counter, and the tile's slots
  int slot0, nslot;           // [slot0, slot0 + nslot), summed in this order
  int pad;
};
struct ItemSeg {              // a run of k inside one term of an item; A, B: first element of the tile's rows / columns
  long long aoff, boff;
  int abuf, bbuf, lda, ldb, k, flags;
  double ar, ai;
  long long pad;
};
static_assert(sizeof(WorkItem) == 64 && sizeof(ItemSeg) == 64, "one 64-byte load each");
struct Bases {
  void* p[kMaxBases];
};


// Grouped FP64 GEMM over work items (deterministic split-K; see gemm.cu).
// Split items write partial tiles; the last of a tile's items sums them (tile_cnt
// holds one zeroed counter per split tile and is left zeroed).
// mask: null, or per job tag; items of a job with mask[tag] == 0 do nothing.
void launch_items(bool cplx, const WorkItem* items, const ItemSeg* segs, int nitems, const Bases& b, void* work,
                  int* tile_cnt, const int* mask, cudaStream_t s);

// ---- tcgen05 3xTF32 over TF32 hi/lo operand panels (umma.cu) --------------
// An operand (rows x K after op) is stored as panels: panel (p, s) holds rows
// [p*T, p*T + T) and k [32 s, 32 s + 32) as groups of 8 rows, each a hi plane then a lo
// plane, each [kg = 0..7][row = 0..7][4 consecutive k] of TF32 bit patterns (x ~ hi + lo),
// zero padded in k; it starts at dst + (p * nslab + s) * T * 256 bytes.  This is the
// K-major, no-swizzle core-matrix layout tcgen05.mma reads, and the rows that a block has
// are the first bytes of its panel: one contiguous bulk copy of them moves into shared
// memory, whatever the tile is padded to.
// Complex products run as real ones of twice the size: C = A B (complex m x n,
// k) is Ch = Ah Bh with Ch (2m x n) and Bh (2k x n) the interleaved storage of
// C and B read as real column-major matrices (no copy), and Ah (2m x 2k) the
// real form of A, Ah(2i+p, 2j+q) = Re A(i,j) for p == q, -Im A(i,j) for
// (p, q) = (0, 1), Im A(i,j) for (1, 0).  The real flop count is the complex
// one (8 per complex multiply-add), and the pack kernel writes Ah / Bh panels
// straight from the complex operands (cmode 1 / 2).
constexpr int kPanelK = 32;
constexpr int kUmmaTileM = 128;
struct PackJob {              // FP64 matrix -> panels
  long long src;              // element offset in its source buffer
  long long dst;              // byte offset of panel (0, 0) in the packed buffer
  long long chunk0;           // first 16-byte chunk of this job in the launch (a multiple of 256)
  int srcbuf, ld, rows, K, trans, T;   // trans 0: (r, k) at src[r + k*ld]; 1: at src[k + r*ld]
  int cmode;                  // 0 real; complex source (src, ld in complex elements, rows / K of the real
                              // form): 1 Ah (rows 2m, K 2k), 2 Bh read as rows n x K 2k
  int conj;                   // complex: conjugate the source elements first
  int sparse;                 // 1: chunks of the real rows and k only (the padding of the
                              // panels is zero already and never written), 0: whole panels
};
struct USlab {                // one slab of a job's concatenated reduction
  long long a, b;             // byte offsets of its A and B panels of tile row / column 0
  int nslab;                  // slabs of its term: panels of tile row p start p * nslab panels further on
  int info;                   // its k (1..32), + 256 (+ 512): the A (B) panel is a per-apply one, else constant
  int adep, bdep;             // dependency counter of the A / B panels written in the same launch, or -1
};
struct UJob {                 // output tile grid of one job
  long long coff;             // FP64 output: bases.p[cbuf] + coff, column-major, ldc
  long long pack;             // >= 0: the result becomes A panels (T = 128) at this byte offset of the
                              // per-apply buffer, scaled by alpha, with pack_nslab slabs per panel
  double alpha;
  int cbuf, m, n, ldc, pack_nslab;
  int dep;                    // counter bumped per finished tile (results read as panels later), or -1
  int tag;                    // as GemmJob::tag
  int cx;                     // complex plan: the tile is a real-form block (rows 2i, 2i+1 = Re, Im of
                              // row i); panels of the result are written in the real form Xh (cmode 1)
};
struct UItem {                // one output tile x a run of consecutive slabs
  int job, tm, tn, q0, nslab, slot;   // q0: first slab (absolute); slot < 0: direct
  int red;                    // split items: their tile's URed
  int arows, brows;           // rows of the A and B panels that the tile's block has, to a multiple of 8
};
struct URed {                 // C tile = sum of FP32 partial slots [slot0, slot0 + nslot) in fixed order
  int job, tm, tn, slot0, nslot;
};
struct UBufs {
  const unsigned char* pconst;
  unsigned char* pvar;
  float* slots;
  int* tile_cnt;              // per URed: items of the tile finished in this launch (reset by the last)
  int* deps;                  // dependency counters (psi pack jobs, then stage-0 results), zero between launches
  const int* dep_target;      // value each counter reaches once its panels are complete
  unsigned* fin;              // CTAs finished (the last one clears deps)
  const int* mask;            // null, or per job tag: 0 skips the job's items (not with wait_deps)
};
constexpr int kMaxPackJobs = 1024;   // psi pack jobs one fused launch can count
struct UPhase {               // what one launch does besides its items
  const PackJob* pk;          // psi -> panels jobs packed at the start of the launch
  const int* pk_blk;          // pack block (256 chunks) -> job
  int npk_blocks;             // 0: no packing in this launch
  int npk_jobs;
  int wait_deps;              // items wait for panels written in this launch (cooperative launch)
  int ndeps;
  long long wait_ns;          // limit of every bounded wait; 0: the default (2 s)
  int ctas_per_sm;            // 2: two CTAs per SM, each with a 2-stage ring (tile width 64 only); else one
};
// one 256-thread block per 256 chunks; blk_job[block] = its job
void launch_pack(const PackJob* jobs, const int* blk_job, int nblocks, const Bases& b, unsigned char* dst,
                 cudaStream_t s);
// One launch of the tcgen05 executor: optional psi packing, then the items.  With
// ph.wait_deps the whole matvec (pack, stage 0, stage 1) runs as one cooperative
// launch, every item waiting (bounded) for the panels it reads.
void launch_umma_items(int bn, const USlab* slabs, const UJob* jobs, const UItem* items, const URed* reds, int nitems,
                       const Bases& b, const UBufs& u, const UPhase& ph, cudaStream_t s);
// status word of the tcgen05 kernels: 0 = fine, otherwise a bounded wait ran out
// (the tiles it guarded were not written); reset clears it.  -1 if unreadable.
int umma_status(bool reset);
int device_sm_count();
constexpr int kMaxDevices = 64;
// cudaFuncSetAttribute(fn, MaxDynamicSharedMemorySize, bytes) once per device (the
// attribute belongs to the kernel on a device and holds for every host thread, so bytes is
// the most that any launch of it takes); done[] holds one flag per device ordinal
void ensure_smem_limit(const void* fn, int bytes, unsigned char* done);
// the same, and the largest shared-memory carve-out
void ensure_smem_attr(const void* fn, int bytes, unsigned char* done);
// Fixed device scratch of the allocation-free H_eff*psi entry point (gemm.cu).
constexpr size_t kNoAllocScratchBytes = (size_t)32 << 20;
// Device address of that scratch on the current device (looked up once per
// device); returns 0 or a cudaError_t value.
int noalloc_scratch(void** ptr);
int gemm_tile_m(bool cplx);
int gemm_tile_n(bool cplx);

// ---- block utilities -------------------------------------------------------
struct Seg {                  // y[doff + i] (+)= alpha * x[soff + i], i < n
  long long doff, soff;
  long long n;
  double ar, ai;
};
void launch_seg_axpy(bool cplx, void* y, const void* x, const Seg* segs, int nseg, cudaStream_t s);

struct Transp {               // dst (cols x rows) = src (rows x cols)^T
  long long soff, doff;
  int rows, cols;
};
void launch_block_transpose(bool cplx, void* dst, const void* src, const Transp* t, int nt, cudaStream_t s);

struct Perm3 {                // dst block = src block (d0 x d1 x d2, column-major) with its legs
  long long soff, doff;       // permuted: leg k of dst is leg p[k] of src
  int d[3], p[3];
};
void launch_permute3(bool cplx, void* dst, const void* src, const Perm3* t, int nt, cudaStream_t s);

struct FuseFill {             // identity embedding of a fuse block (d0,d1,d2): 1 at (a,b,pos+b*d0+a)
  long long off;
  int d0, d1, d2, pos;
};
void launch_fuse_fill(bool cplx, void* data, const FuseFill* f, int nf, cudaStream_t s);

struct Gather {               // dst (rows x kept) = src[rows, perm[c]] * w[c]^p  (optionally conjugated)
  long long soff, doff;       // soff: first row of the source column block (column 0)
  int lds, rows, kept, conj;
  long long woff;             // sorted singular values (double) offset
  long long poff;             // offset into the column permutation
  double p;                   // exponent applied to singular values (0 => none)
};
void launch_gather(bool cplx, void* dst, const void* src, const double* w, const int* perm, const Gather* g, int ng,
                   cudaStream_t s);
// x *= alpha (host scalar)
void launch_scale(bool cplx, void* x, double ar, double ai, long long n, cudaStream_t s);
// read bytes (a multiple of 16) of x and discard them (sink: a device word, written
// only by an unlikely data pattern)
void launch_read(const void* x, long long bytes, unsigned* sink, cudaStream_t s);
// fill with a constant
void launch_fill(bool cplx, void* x, double vr, double vi, long long n, cudaStream_t s);

// ---- Krylov vector operations (krylov.cu) ----------------------------------
struct VecBlk {               // one thread block's range of a segment
  long long lo;
  int n, seg;
};
struct VecSpan {              // the vectors a launch works on: one segment of n elements in ranges of
  const VecBlk* blk;          // `per` (blk null), or the ranges blk[0 .. nblk) of nseg segments, segment
  const int* blk0;            // s owning blocks [blk0[s], blk0[s + 1])
  const int* active;          // null, or per segment: 0 = leave the segment alone
  long long n, per;
  int nblk, nseg;
};
// one segment of n elements in at most max_blocks ranges
VecSpan vec_span(long long n, int max_blocks);
enum VecOp : int {
  VO_NONE = -1,
  VO_COEF = 0,                // scal[2 seg] = beta[seg * bstride], scal[2 seg + 1] = Re out[0] (elements of the
                              // scalar type: the two-term recurrence's coefficients), host = Re out[0]
  VO_NORM = 1,                // scal[seg * sstride] = host = sqrt(|Re out[0]|) (doubles)
  VO_HOST = 2                 // host[seg * hstride + j] = out[j] (elements of the scalar type)
};
struct VecOut {               // what the last block of a segment does with its sums; host: page-locked
  int op = VO_NONE;           // host memory (readable after a synchronisation), may be null for VO_NORM
  const double* beta = nullptr;
  int bstride = 0;
  void* scal = nullptr;
  int sstride = 0;
  void* host = nullptr;
  int hstride = 0;
};
// out[seg * nv + j] = <V_j | x> (conjugated first argument), after x -= uc[2 seg] u0 + uc[2 seg + 1] u1
// when u1 is given (u0 may be null).  partial: nblk * nv elements of the scalar type; counter: a zeroed
// word per segment (left zero).  Deterministic, one launch.
void launch_vec_dots(bool cplx, const VecSpan& v, const void* V, long long ldv, int nv, void* x, const void* u0,
                     const void* u1, const void* uc, double* partial, void* out, unsigned* counter, const VecOut& o,
                     cudaStream_t s);
// x -= sum_j c[seg * cstride + j] V_j; partial (nblk doubles) given: then |x| as VO_NORM
void launch_vec_axpy(bool cplx, const VecSpan& v, void* x, const void* V, long long ldv, int nv, const void* c,
                     int cstride, double* partial, unsigned* counter, const VecOut& o, cudaStream_t s);
// y = sum_j c[seg * cstride + j] V_j (real c); partial given: then |y| as VO_NORM
void launch_vec_lincomb(bool cplx, const VecSpan& v, void* y, const void* V, long long ldv, int nv, const double* c,
                        int cstride, double* partial, unsigned* counter, const VecOut& o, cudaStream_t s);
// y = x / scal[seg * sstride], copied to y2 when given; a value not above floor divides by 1
void launch_vec_div(bool cplx, const VecSpan& v, const void* x, void* y, void* y2, const double* scal, int sstride,
                    double floor, cudaStream_t s);

// Lowest eigenvalue (e0[s]) and its vector (z0[s * zstride + i], zeros to i = nmax) of ns
// symmetric tridiagonals of n[s] <= nmax <= kTridiagMax rows (0: none), diagonal a[i * ns + s],
// coupling of i and i + 1 b[(i + 1) * ns + s]; as tridiag_eig (dmrg.cpp) bit for bit (tridiag.cu).
// *status = 1 where one did not converge.  n, a, b, e0 and status may be page-locked host
// memory.
constexpr int kTridiagMax = 128;
void launch_tridiag_lowest(int ns, const int* n, int nmax, const double* a, const double* b, double* z0, int zstride,
                           double* e0, int* status, cudaStream_t s);

// ---- one-sided Jacobi SVD of sector blocks --------------------------------
struct SvdJob {
  long long aoff;             // input block (m x n, lda = m) in the input buffer
  long long woff;             // work: max(m,n) x min(m,n) columns being orthogonalised
  long long voff;             // accumulated rotations: min(m,n) x min(m,n)
  long long soff;             // singular values (double), min(m,n)
  int m, n, trans;            // trans = 1 when m < n (work on A^H)
};
// Host driver: all sweeps in one cooperative launch.  Returns the sweeps taken, or -1 if
// max_sweeps was reached.  kernel_ms (optional): device time of that launch (with the
// QR preconditioning: plus the QR and the Q application).
// precondition: Jacobi on R1^H after Householder QRs of the norm-ordered columns
// and of R^H (fewer sweeps): 0 never, 1 when the widest block has at least 32
// columns, 2 always; the outputs have the same meaning either way.
// stream: 1 streams every visit's rows in chunks even where the pair's columns
// would fit in shared memory (same results; covers that path on small problems).
// block: Jacobi column blocks of 8 or 16, 0 for the rule (8 when a round of all sectors'
// 16-column pairs would keep fewer than half the SMs busy).
int run_jacobi_svd(bool cplx, const void* a, void* work, void* vmat, double* sv, const std::vector<SvdJob>& jobs,
                   int max_sweeps, cudaStream_t s, double* kernel_ms = nullptr, int precondition = 1,
                   int stream = 0, int block = 0);

}  // namespace sadmrg
