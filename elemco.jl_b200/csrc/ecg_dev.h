// ecg_dev.h — the device layer of libecgpu: memory, copies and kernel
// launchers.  The host orchestration (residuals, DIIS, drivers) talks to the
// GPU only through these functions; dev_cuda.cu implements them with CUDA
// kernels for sm_100a.  Every launcher is asynchronous on the given stream
// and returns 0 or a nonzero CUDA error code.
#pragma once
#include <cstddef>
#include <cstdint>
#include <vector>

namespace ecg {
namespace dev {

using stream_t = void*;

int set_device(int device);
int stream_create(stream_t* s);
// Waits for s, frees the scratch the layer holds for it (splitk_buffer,
// split_scratch) and destroys it.
void stream_destroy(stream_t s);
int sync(stream_t s);
const char* error_string(int code);
int check_launch();  // cudaGetLastError as int

void* dmalloc(size_t bytes);   // nullptr on failure
void dfree(void* p);
void* hmalloc_pinned(size_t bytes);
void hfree_pinned(void* p);
int h2d(void* dst, const void* src, size_t bytes, stream_t s);
int d2h(void* dst, const void* src, size_t bytes, stream_t s);
int d2d(void* dst, const void* src, size_t bytes, stream_t s);
// d2h for results that may be large and go to pageable memory; the data has
// arrived on return (where it was not staged: once the stream is synchronised).
int d2h_large(void* dst, const void* src, size_t bytes, stream_t s);
int memset0(void* dst, size_t bytes, stream_t s);
// Record the launches issued on s after graph_capture_begin into a CUDA graph;
// graph_capture_run ends the capture, runs the graph once, waits for it and
// frees it (*nodes: the number of graph nodes).
int graph_capture_begin(stream_t s);
int graph_capture_run(stream_t s, int64_t* nodes);
void graph_capture_abort(stream_t s);  // end a capture in progress, discarding it
// As graph_capture_run, but hands the graph to the caller (graph_free) instead
// of running it; graph_launch queues it once more.
int graph_capture_keep(stream_t s, void** exec, int* kernels);
int graph_launch(stream_t s, void* exec, int kernels);
void graph_free(void* exec);
// Whether launches on s may be recorded: not while they are timed or tuned.
bool graphs_usable(stream_t s);

// C(m,n) = alpha * sum_k opA(A)(m,k) opB(B)(k,n) + beta * C(m,n), column-major;
// ta/tb = 'N' or 'T'.  batch > 1 uses strides sa/sb/sc between instances.
int gemm(stream_t s, char ta, char tb, int64_t m, int64_t n, int64_t k, double alpha,
         const double* A, int64_t lda, const double* B, int64_t ldb, double beta,
         double* C, int64_t ldc, int64_t batch = 1, int64_t sa = 0, int64_t sb = 0,
         int64_t sc = 0);

// Fully strided batched GEMM: C(m,n) = alpha sum_k A(m,k) B(k,n) + beta C(m,n)
// with A(m,k) = A[b*sab + m*sam + k*sak], B(k,n) = B[b*sbb + k*sbk + n*sbn],
// C(m,n) = C[b*scb + m*scm + n*scn] for batch b.  Batches must not write
// overlapping C elements.  tri > 0 (batch 1, beta 0): elements with
// n / tri < m / tri are not needed, and tiles that hold nothing else are
// skipped (such elements of C may keep their old values or get their product).
struct Gemm {
  int64_t m = 0, n = 0, k = 0, batch = 1;
  double alpha = 1.0, beta = 0.0;
  const double* A = nullptr;
  int64_t sam = 1, sak = 0, sab = 0;
  const double* B = nullptr;
  int64_t sbk = 1, sbn = 0, sbb = 0;
  double* C = nullptr;
  int64_t scm = 1, scn = 0, scb = 0;
  int64_t tri = 0;
};
int gemm_strided(stream_t s, const Gemm& g);
// Share of C's elements that g computes (1 unless tri > 0; counted by tri x tri
// squares).
inline double gemm_kept(int64_t m, int64_t n, int64_t tri) {
  if (tri <= 0) return 1.0;
  const double a = (double)((m + tri - 1) / tri), b = (double)((n + tri - 1) / tri);
  return a <= b ? 1.0 - (a - 1.0) / (2.0 * b) : (b + 1.0) / (2.0 * a);
}
inline double gemm_kept(const Gemm& g) { return gemm_kept(g.m, g.n, g.tri); }
// FP64 GEMM with TMA-staged operands (dev_dgemm.cu): C with unit row stride,
// each operand contiguous along its row index or along k with its other
// strides even (16-byte multiples) and a 16-byte-aligned base.  cfg selects the
// tile (0: 64x64, 1: 32x32, 2: 64x32, 3: 64x64 with eight MMA warps); nsplit > 1
// (batch 1) cuts K into slices summed in a fixed order.  Returns -1, launching
// nothing, when TMA cannot address an operand; dgemm_tma_usable tells
// beforehand.  dgemm_tma_rule picks cfg and nsplit by estimated time.
constexpr int DTMA_CONFIGS = 4;
bool dgemm_tma_usable(const Gemm& q);
// Returns that time (us).
double dgemm_tma_rule(const Gemm& q, int* cfg, int* nsplit);
int dgemm_tma(stream_t s, const Gemm& q, int cfg, int nsplit);

// The (T) K builds in FP64 (dev_kbuild.cu): for each item z of a batch
//   C_z(r,c) = beta C_z(r,c) + sum_{s < nseg} sum_{k < k[s]} A_s(r,k) B_s(c,k)
// with r < m, c < n and beta 0 or 1.  Operand X(i,k) of item index z sits at
// X[i + k*sk + z*sz] (i < ni, z < nz; X 16-byte aligned, sk and sz even);
// items[z] (device memory) names the item of each segment's A and B and the
// offset of C_z.  C(r,c) sits at (r % dm)*scm + (r / dm)*scm2 + c*scn (dm = 0:
// r*scm + c*scn).  even_items: every item's C offset is even.  One launch.
constexpr int KB_MAX_SEG = 4;
struct KbOperand {
  const double* X = nullptr;
  int64_t ni = 0, sk = 0, nz = 1, sz = 2;
};
struct KbItem {
  int32_t a[KB_MAX_SEG], b[KB_MAX_SEG];
  int64_t c;
};
struct KbGemm {
  int64_t m = 0, n = 0;
  int nseg = 0;
  int64_t k[KB_MAX_SEG] = {0, 0, 0, 0};
  KbOperand A[KB_MAX_SEG], B[KB_MAX_SEG];
  double beta = 0.0;
  double* C = nullptr;
  int64_t scm = 1, dm = 0, scm2 = 0, scn = 0;
  bool even_items = false;
};
int kbuild(stream_t s, const KbGemm& g, int nitems, const KbItem* items);
// Split-BF16 tensor-core version of gemm_strided (batch 1).
int gemm_strided_mixed(stream_t s, const Gemm& g);

// Pre-split operand of the tensor-core GEMM: X(r,k) as `slices` (2 or 3)
// BF16 slices [slices][rows_p][k_p] (k fastest; rows padded to 128, k to 64,
// zero filled) and the TMA descriptor over them.  tc_operand_elems() is the
// BF16 element count of the storage; tc_split() fills it (dst 16-byte
// aligned) from the FP64 source X(r,k) = src[r*sr + k*sk] and encodes the
// descriptor.  Three slices reproduce FP32-level products, two slices
// ~2^-16 relative.
struct TcOperand {
  alignas(64) unsigned char map[128];
  // the same operand with 160- and 256-row boxes, for 160- and 256-column
  // tiles when it is the B operand (each encoded, and its flag set, when the
  // row extent is at least the box)
  alignas(64) unsigned char map_w[128];
  alignas(64) unsigned char map_x[128];
  bool wide = false, xwide = false;
  int64_t rows = 0, rows_p = 0, k = 0, k_p = 0;
  int slices = 0;
  void* base = nullptr;        // first BF16 element of row 0, slice 0
  int64_t slice_stride = 0;    // BF16 elements between slices
};
size_t tc_operand_elems(int64_t rows, int64_t k, int slices);
int tc_split(stream_t s, const double* src, int64_t rows, int64_t k, int64_t sr, int64_t sk,
             int slices, void* dst, TcOperand* op);
// Rows [row0, row0 + rows) of a split operand as an operand of their own (no
// copy: a descriptor over the same storage; rows past the view read as zero).
int tc_view(const TcOperand& parent, int64_t row0, int64_t rows, TcOperand* out);
// Descriptor over slices already written to dst in tc_split's layout
// ([slice][tc_pad_rows(rows)][tc_pad_k(k)], K fastest, zero K padding).
int tc_bind(void* dst, int64_t rows, int64_t k, int slices, TcOperand* op);
int64_t tc_pad_rows(int64_t rows);
int64_t tc_pad_k(int64_t k);
// ladder_pack_v fused with the three-slice split of its outputs: the a-block's
// V (FP32 when v_f32, else FP64; layout of ladder_pack_v) is packed into the
// symmetric (rows: the block's npairs pairs, K = v(v+1)/2) and antisymmetric
// (rows: its a < b pairs, K = v(v-1)/2) operands, written as BF16 slices in
// tc_split's layout at Vp / Vm (bind them with tc_bind).
int ladder_pack_v_split(stream_t s, int nv, int a0, int na, int npairs, const int* pairs,
                        const int* cdp, const void* V, bool v_f32, void* Vp, void* Vm);
// C(m,n) = alpha sum_k A(m,k) B(k,n) + beta C(m,n) over pre-split operands
// (all with the same slice count): the K sum runs over up to TC_MAX_SEG
// segments A[s]/B[s], s = 0, 1, ... (the first null A[s] ends the list), each
// with its own K depth and operands.  An FP64 C may be computed in K slices
// summed in FP64 (to fill the GPU and to bound the FP32 accumulation length).
// C is FP64, or FP32 when f32, at C[m*scm + n*scn]; stores are coalesced when
// scm == 1.
constexpr int TC_MAX_SEG = 4;
// Longest K one FP32 tensor-memory accumulator sums: FP64 outputs with a
// longer K are computed in K slices whose partial products are added in FP64;
// FP32 outputs are one accumulation, so callers keep their K within this.
constexpr int64_t TC_ACC_K = 1024;
struct TcGemm {
  int64_t m = 0, n = 0;
  double alpha = 1.0, beta = 0.0;
  const TcOperand* A[TC_MAX_SEG] = {nullptr, nullptr, nullptr, nullptr};
  const TcOperand* B[TC_MAX_SEG] = {nullptr, nullptr, nullptr, nullptr};
  void* C = nullptr;
  bool f32 = false;
  int64_t scm = 1, scn = 0;
  // tri > 0: as Gemm::tri
  int64_t tri = 0;
};
int tc_gemm(stream_t s, const TcGemm& g);
// A stack of `items` operands of equal shape, each as tc_split writes one (two
// slices), back to back.  tc_split_stack fills it: item i's X(r,k) sits at
// src[(i % d)*s0 + (i / d)*s1 + rowoff(r) + k*sk], rowoff(r) = (r % dr) + (r /
// dr)*sr (dr = 0: r*sr).
struct TcStack {
  const void* base = nullptr;
  int64_t rows = 0, k = 0, items = 0;
};
int tc_split_stack(stream_t s, const double* src, int64_t rows, int64_t k, int64_t sr, int64_t sk,
                   int64_t dr, int64_t items, int64_t d, int64_t s0, int64_t s1, void* dst,
                   TcStack* out);
// The (T) K builds on the tensor cores (dev_tckbuild.cu): kbuild's products
// with FP32 C and BF16-split operands; beta adds to C.  pad4: rows of C are
// followed by room for whole groups of four columns (scn == 1), and every item
// starts on 16 bytes.  Items run in chunks of `chunk` consecutive ones, which
// should share operands A.
struct TcKbuild {
  int64_t m = 0, n = 0;
  int nseg = 0;
  TcStack A[KB_MAX_SEG], B[KB_MAX_SEG];
  bool beta = false, pad4 = false;
  float* C = nullptr;
  int64_t scm = 1, dm = 0, scm2 = 0, scn = 0;
};
int tc_kbuild(stream_t s, const TcKbuild& g, int nitems, const KbItem* items, int chunk);

// out = alpha * permute(in) + beta * out.  in has rank nd with dims
// in_dims (column-major, first fastest); out dimension d is in dimension
// perm[d].  beta == 0 never reads out.
int permute(stream_t s, int nd, const int64_t* in_dims, const int* perm, double alpha,
            const double* in, double beta, double* out);

// dst[x + ldd*r] = src[x + lds*r], x < n, r < rows: a copy between row pitches.
int repitch(stream_t s, int64_t n, int64_t rows, const double* src, int64_t lds, double* dst,
            int64_t ldd);

// y = alpha * x + beta * y   (beta == 0: y = alpha * x)
int axpby(stream_t s, int64_t n, double alpha, const double* x, double beta, double* y);

// out[b] = beta*out[b] + alpha * sum_{k<nk} in[b*sb + k*sk]
int strided_sum(stream_t s, int64_t nb, int64_t sb, int64_t nk, int64_t sk, double alpha,
                const double* in, double beta, double* out);

// Doubles (or singles) update with level shift, in place:
// T[a,b,i,j] += -R[a,b,i,j] / (ev[a]+ev[b]-eo[i]-eo[j]+shift)
int update_doubles(stream_t s, int nv, int no, const double* eo, const double* ev,
                   double shift, const double* R, double* T);
int update_singles(stream_t s, int nv, int no, const double* eo, const double* ev,
                   double shift, const double* R, double* T);

// Deterministic reductions (fixed grouping and order), all jobs in one launch:
//   DOT_PLAIN  out[0] = sum X*Y over n
//   DOT_CS     for nv x nv x no x no:  out[0] = sum X[a,b,i,j] Y[a,b,i,j],
//              out[1] = sum X[b,a,i,j] Y[a,b,i,j]
//   DOT_CS_T1  DOT_CS of X[a,b,i,j] = X[a,i] X[b,j] (X nv x no)
// `scratch` must hold at least reduce_scratch_len() doubles, zero before its
// first use; calls that share it run on one stream.
enum { DOT_PLAIN = 0, DOT_CS = 1, DOT_CS_T1 = 2 };
constexpr int DOT_MAX = 16;
struct DotJob {
  int type;
  const double* X;
  const double* Y;
  int64_t n;  // DOT_PLAIN
  double* out;
};
int64_t reduce_scratch_len();
int dots(stream_t s, int nv, int no, int njobs, const DotJob* jobs, double* scratch);
int dot(stream_t s, int64_t n, const double* x, const double* y, double* scratch, double* out);
int cs_dot(stream_t s, int nv, int no, const double* X, const double* Y, double* scratch,
           double* out);

// Doubles amplitudes as the ring terms read them, in one pass over T2[a,b,i,j]:
//   X1[a,i,b,j] = T2[a,b,i,j], X2[a,i,b,j] = T2[a,b,j,i], Xt = 2 X1 - X2,
//   Tt[a,b,i,j] = 2 T2[a,b,i,j] - T2[a,b,j,i]
int ring_split(stream_t s, int nv, int no, const double* T2, double* X1, double* X2, double* Xt,
               double* Tt);
// In place over n elements: W, Y, Z <- Y - W, 2 W - Y - Z, Q/2 - Z (Y and Q read
// as zero, and Q not at all, when Q is null).
int ring_combine(stream_t s, int64_t n, double* W, double* Y, double* Z, const double* Q);
// R2[a,b,i,j] += D[a,i,b,j] + D[b,j,a,i] + E[b,i,a,j] + E[a,j,b,i]
int ring_add(stream_t s, int nv, int no, const double* D, const double* E, double* R2);
// Fock matrix blocks: f = dh + 2 sum_Q B[:,:,Q] J[Q] + G, written to f (n x n) and
// as dense blocks foo [i,j], fvo [a,i], fov [a,i] (of f[i,a]) and fvv [a,b].  G
// holds the dense blocks oo, vo [a,i], ov [i,a], vv back to back.
int fock_blocks(stream_t s, int no, int nv, int nq, const double* dh, const double* Boo,
                const double* Bvo, const double* Bov, const double* Bvv, const double* J,
                const double* G, double* f, double* foo, double* fvo, double* fov, double* fvv);
// Level-shifted update of T = [T1 | T2] by R = [R1 | R2], in place, with copies
// of both at Tsave and Rsave:
//   T1 -= R1 / (ev[a] - eo[i] + shifts), T2 -= R2 / (ev[a] + ev[b] - eo[i] - eo[j] + shiftp)
int update_save(stream_t s, int nv, int no, const double* eo, const double* ev, double shifts,
                double shiftp, const double* R, double* T, double* Tsave, double* Rsave);

// C(i,j) = alpha * A(i,j) + beta * C(i,j) for an m x n column-major block
// (leading dimensions lda, ldc); beta == 0 never reads C.
int geam(stream_t s, int64_t m, int64_t n, double alpha, const double* A, int64_t lda,
         double beta, double* C, int64_t ldc);

// out[a,b,i,j] = alpha * X[a,i] * Y[b,j] + beta * out[a,b,i,j]
// (X: na x ni, Y: nb x nj, out: na x nb x ni x nj).
int outer(stream_t s, int64_t na, int64_t ni, int64_t nb, int64_t nj, double alpha,
          const double* X, const double* Y, double beta, double* out);

// out = sum_{k<m} coef[k] * X[k]
int combine(stream_t s, int64_t n, int m, const double* const* X, const double* coef,
            double* out);

// y[i] = (float)x[i]
int to_f32(stream_t s, int64_t n, const double* x, float* y);
// out[i] = (float(a[i]), float(b[i])) as float2 pairs (out 8-byte aligned)
int to_f32_pairs(stream_t s, int64_t n, const double* a, const double* b, void* out);
// *flag = 1 if any of x[0..n) is an infinity or NaN, else 0 (device double)
int nonfinite(stream_t s, int64_t n, const double* x, double* flag);

// (T) energies of occupied triplets (src/cc/cc_triples.jl:113-156) from
// K[a,b,c] (FP64, or FP32 when k_f32), without storing X:
//   X[a,b,c] = (4K[abc]-2K[acb]-2K[cba]-2K[bac]+K[cab]+K[bca]) / (eijk-ev[a]-ev[b]-ev[c])
//   out[0]   = sum KE*X      (KE = KU when given, else K)
//   out[1]   = sum X*Y,  Y[a,b,c] = g0[a] M0[b,c] + g1[b] M1[a,c] + g2[c] M2[a,b]
//                              + f0[a] N0[b,c] + f1[b] N1[a,c] + f2[c] N2[a,b]
// The 8^3 cubes of K are visited in orbits of the index permutations, so each
// element of K is read once.  `tri` holds the cube triples A <= B <= C (3
// ints each) for nt = ceil(nv/8) cubes per axis: triples_cube_count(nv) of
// them, written by triples_cube_table().  g, f (length nv) and M, N (nv x nv)
// hold elements of K's precision; ev (FP64) the virtual orbital energies.
// nv <= 1290 (32-bit element offsets).
struct TriplesTerms {
  const void* g[3];
  const void* f[3];
  const void* M[3];
  const void* N[3];
};
int64_t triples_cube_count(int nv);
void triples_cube_table(int nv, int* tri);
// FP64 K: item b reads K + b*kstride (KU likewise), eijk_tab[b] and tt_tab[b]
// (device tables) and writes out[2b], out[2b+1]; partial sums land in
// `scratch` (at least triples_energy_scratch_len(nv, nitems) doubles) and are
// summed in a fixed order.  One launch (plus one fixed-order reduction
// launch).  k_f32 must be false (FP32 K: triples_energy_f32_batched).
int64_t triples_energy_scratch_len(int nv, int nitems);
// blocks per batch item of the FP64 / FP32 energy kernels
int64_t triples_energy_grid(int nv);
int64_t triples_energy_f32_grid(int nv);
int triples_energy_batched(stream_t s, int nv, int nitems, const void* K, const void* KU,
                           int64_t kstride, bool k_f32, const double* eijk_tab, const double* ev,
                           const TriplesTerms* tt_tab, const int* tri, double* scratch,
                           double* out);
// The same for FP32 K (and K') (dev_energy.cu).  K[a,b,c] of slot i sits at
// K + i*kstride + a + vp*(b + v*c), vp >= v a multiple of 4 (TMA strides of
// 16 bytes); nslots >= nitems slots at K (and KU), 16-byte aligned.  The
// (M, N) terms are FP32 pairs per occupied pair p = x + o*y, packed by
// triples_mn_pack: mn[p][a + vpe*b] and their transposes mt[p][b + vpe*a]
// (vpe = v rounded up to even; triples_mn_elems float2 each).  Per item,
// gf[r] points at the (g, f)[a] FP32 pairs of occupied index r of the triplet
// (i, j, k) and mnpair[w] is the pair index of (j,k), (i,k), (i,j).
struct TriplesTermsF {
  const void* gf[3];
  int32_t mnpair[3];
};
int64_t triples_mn_elems(int nv, int64_t npairs);
int triples_mn_pack(stream_t s, int nv, int64_t npairs, const double* M, const double* N,
                    void* mn, void* mt);
int triples_energy_f32_batched(stream_t s, int nv, int vp, int nitems, int nslots, const float* K,
                               const float* KU, int64_t kstride, const void* mn, const void* mt,
                               int64_t npairs, const double* eijk_tab, const double* ev,
                               const TriplesTermsF* tt_tab, const int* tri, double* scratch,
                               double* out);

// Split-K GEMM (column-major, device pointers) whose partial products use a
// fixed file-scope device array instead of allocated memory; m*n must not
// exceed noalloc_scratch_doubles().  *nsplit receives the K split used.
size_t noalloc_scratch_doubles();
int gemm_splitk_noalloc(stream_t s, char ta, char tb, int64_t m, int64_t n, int64_t k,
                        double alpha, const double* A, int64_t lda, const double* B, int64_t ldb,
                        double beta, double* C, int64_t ldc, int* nsplit);

// Split-BF16 tensor-core GEMM (tcgen05, FP32 accumulate, ~FP32 accuracy),
// same interface as gemm().  tc_error() returns and clears the time-out codes
// of stream s's kernels with bounded mbarrier waits (s synchronised; 0 = none; 1-4 tensor-core GEMM,
// 17 TMA-staged FP64 GEMM, 33 FP32 (T) energy kernel, 49 FP64 K builds,
// 65-68 tensor-core K builds).
int gemm_mixed(stream_t s, char ta, char tb, int64_t m, int64_t n, int64_t k, double alpha,
               const double* A, int64_t lda, const double* B, int64_t ldb, double beta,
               double* C, int64_t ldc);
int tc_error(stream_t s, int* codes);  // codes[WAIT_KERNELS]
// Where those kernels leave them: a word of the stream's for each kind of kernel, in
// pinned host memory that the device maps (nullptr: it could not be allocated).
enum { WAIT_TC, WAIT_DGEMM, WAIT_ENERGY, WAIT_KBUILD, WAIT_TCKBUILD, WAIT_KERNELS };
int* wait_error(stream_t s, int kernel);
// Split-K scratch of stream s on the current device (at least n doubles;
// grown on demand, after s has drained, never during stream capture: nullptr
// then, or when the allocation fails) and its fixed-order reduction
// C(i,j) = alpha sum_z P[z][i + j m] + beta C(i,j), C at C[i*scm + j*scn].
double* splitk_buffer(stream_t s, size_t n);
// Scratch of stream s for gemm_mixed's BF16 operand slices (same rules).
void* split_scratch(stream_t s, size_t bytes);
// What stream s holds of it; release_scratch waits for s and gives it back.
size_t scratch_bytes(stream_t s);
void release_scratch(stream_t s);
// The copies in even pitches that the FP64 GEMM makes for TMA live in it too, as
// long as it stays within `bytes` (no bound to begin with).
void set_copy_room(stream_t s, size_t bytes);
// Bound (ns) of the tensor-core kernels' main-loop waits on stream s
// (0 = the default second); the kernels' final waits keep the second.
int set_tc_wait(stream_t s, uint64_t ns);
uint64_t tc_wait(stream_t s);
int splitk_reduce(stream_t s, int64_t m, int64_t n, int S, const double* P, double alpha,
                  double beta, double* C, int64_t scm, int64_t scn);
// The same for FP32 partials (summed in FP64).
int splitk_reduce_f32(stream_t s, int64_t m, int64_t n, int S, const float* P, double alpha,
                      double beta, double* C, int64_t scm, int64_t scn);

// Event timing of kernel families (process-wide diagnostic): enable, then
// read and reset a family's summed device ms, launch count and algorithmic
// work (flops for the GEMMs, bytes for the (T) energy kernel).  Launches
// during stream capture are not timed.  ktime_begin returns a slot (-1: not
// timed) for ktime_end, which records the end event and adds the work.
enum { KT_DGEMM = 0, KT_TCGEMM = 1, KT_TRIPLES = 2, KT_FAMILIES = 3 };
void gemm_timing(bool enable);
void gemm_time(double* ms, int64_t* launches, double* flops);  // KT_DGEMM
void kernel_time(int family, double* ms, int64_t* launches, double* work);
int ktime_begin(stream_t s, int family);
void ktime_end(stream_t s, int family, int slot, double work);

// Symmetric/antisymmetric particle-particle ladder helpers.  Pair tables hold
// (x,y) as int pairs: cdp enumerates c<=d (d outer), ijp i<=j, pairs the
// (a,b), a<=b of one a-block.  Packed "minus" indices follow arithmetically:
// idx-(c,d) = idx+(c,d) - d (c<d); pair-(a,b) = pair+(a,b) - (a-a0) - 1 (a<b).
//   ladder_pack_t: Ts[cd+,ij+] = (T[c,d,i,j]+T[d,c,i,j])/2, Ta[cd-,ij-] = (T[c,d,i,j]-T[d,c,i,j])/2
//   ladder_pack_v: Vblk[c,a',d,b''] (a' = a-a0, b'' = b-a0) ->
//                  Vp[cd+,pair+] = V[acbd]+V[adbc] (c<d), V[acbc] (c=d);  Vm[cd-,pair-] = V[acbd]-V[adbc]
//   ladder_unpack: R2[a,b,i,j] += Lp+Lm, R2[b,a,i,j] += Lp-Lm, R2[a,b,j,i] += Lp-Lm, R2[b,a,j,i] += Lp+Lm
// The packed cd index runs fastest, with leading dimensions ldp (>= v(v+1)/2)
// for Ts / Vp and ldm (>= v(v-1)/2) for Ta / Vm (even values let TMA stage them).
int ladder_pack_t(stream_t s, int nv, int no, const double* T2, const int* cdp, const int* ijp,
                  double* Ts, double* Ta, int64_t ldp, int64_t ldm);
int ladder_pack_v(stream_t s, int nv, int a0, int na, int npairs, const int* pairs,
                  const int* cdp, const double* Vblk, double* Vp, double* Vm, int64_t ldp,
                  int64_t ldm);
int ladder_unpack(stream_t s, int nv, int no, int a0, int npairs, const int* pairs,
                  const int* ijp, const double* Lp, const double* Lm, double* R2);

// Gaussian integrals over contracted Cartesian shells (dev_ints.cu).  A shell
// has centre (x, y, z), angular momentum l <= INT_LMAX, nprim primitives whose
// exponents/coefficients start at poff in the exponent/coefficient arrays,
// and its first Cartesian function at boff of the output dimension.
// Components of degree l are ordered i = l..0, j = l-i..0 (x^i y^j z^k).
// Outputs are accumulated (zero them first).
constexpr int INT_LMAX = 4;   // largest shell angular momentum (g)
constexpr int INT_LTOT = 12;  // largest l_a + l_b + l_c (+ l_d) of a Coulomb integral
struct IntShell {
  double x, y, z;
  int l, nprim, poff, boff;
};
// kind 0 overlap, 1 kinetic, 2 nuclear attraction (natom charges Z at xyz),
// 3 dipole about origin (three nn x nn matrices); out[m + nn*n].
int int1e_cart(stream_t s, int kind, const IntShell* sh, int nsh, const double* ex,
               const double* co, int natom, const double* Z, const double* xyz,
               const double* origin, int64_t nn, double* out);
// (P|Q), out[P + np*Q]
int int2c2e_cart(stream_t s, const IntShell* aux, int nsh, const double* ex, const double* co,
                 int64_t np, double* out);
// (mn|P) over real solid harmonics, normalised: out[m + n*(m' + n*P)].  build()
// collects on the host the AO shell pairs by class with their primitive pairs,
// and the fitting shells by degree (boff: first spherical function; exponents
// and coefficients as for the other integrals, each basis with its own
// arrays); it returns -1 for a function of zero norm.  run() uploads them to
// `tables` (table_doubles(), 16-byte aligned) and launches.
struct IntPair {
  int pp0, npp, aoff, boff;  // primitive pairs, first functions (la >= lb)
  int64_t hoff;              // its first Hermite expansion
};
struct IntPrimPair {
  double p, x, y, z;
};
struct IntPairPrimSrc {
  double p, pa[3], pb[3], f;
  int64_t hoff;
  int la, lb;
};
struct Int3cPlan {
  std::vector<IntPair> pairs;
  std::vector<IntPrimPair> prims;
  std::vector<IntPairPrimSrc> src;
  std::vector<IntShell> aux;
  std::vector<double> ex, co;
  // by class la*(INT_LMAX+1) + lb: first pair, pairs, and how many of them (the
  // first ones) are contracted
  int pair0[(INT_LMAX + 1) * (INT_LMAX + 1)] = {}, npair[(INT_LMAX + 1) * (INT_LMAX + 1)] = {};
  int nsplit[(INT_LMAX + 1) * (INT_LMAX + 1)] = {};
  int aux0[INT_LMAX + 1] = {}, naux[INT_LMAX + 1] = {};
  int64_t hlen = 0;
  int build(const IntShell* ao, int nao_sh, const double* aoex, const double* aoco,
            const IntShell* fit, int nfit_sh, const double* fex, const double* fco);
  int64_t table_doubles() const;
  int run(stream_t s, double* tables, int64_t n, double* out) const;
};

// Count of kernels launched through this layer in this process.
int64_t launches();
void note_launches(int n);  // add n launches made outside dev_cuda.cu

}  // namespace dev
}  // namespace ecg
