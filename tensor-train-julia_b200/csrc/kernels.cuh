// Launchers of the device kernels of libttcuda (all FP64 unless stated).
#pragma once
#include "common.cuh"

namespace ttc {

// Elements of an element-wise launch's problems: the largest, and all together.
struct ElemCount {
  long long max = 0, total = 0;
  void add(long long n) {
    max = n > max ? n : max;
    total += n;
  }
};
// Blocks per problem of an element-wise launch over `count` problems (the grid's y dimension) on nsm SMs; a
// block takes per_block elements at least, its threads striding over the problem.  Sixteen blocks per SM (two
// waves of the resident ones) are shared among the problems: of problems alike each gets as many.  A problem
// much larger than the others gets up to sixteen, as far as its part of the elements goes, also where a share
// by number is less; every other one starts as many, most of them with nothing to do.  The element-wise launches
// of a rounding of one train of rank 700 and 1400 of rank 2 (d 22): one block per problem 14.7 ms, sixteen 2.1,
// 32 2.2, 64 3.3; of one of rank 300 and 1400 of rank 2 (d 20) 3.6, 1.3, 1.7, 2.5; with 90 or 200 small ones the
// same.  One block per per_block elements of the largest problem, whatever the count, started up to 4 million:
// 16.9 and 6.8 ms, and the operand conversion of 60 sketches (3689 problems) 830 us, 262 so with its transposes
// in tiles.
inline unsigned elem_blocks(const ElemCount& e, int per_block, int count, int nsm) {
  const double part = 16.0 * nsm * (double)e.max / (double)(e.total > 0 ? e.total : 1);
  const long long fit = (e.max + per_block - 1) / per_block, like = 16LL * nsm / (count > 0 ? count : 1);
  const long long share = (long long)part, most = like > 16 ? like : 16;
  const long long b = fit < share ? fit : share;
  return (unsigned)(b < 1 ? 1 : b < most ? b : most);
}

// ---- grouped FP64 GEMM (gemm_f64.cu)
// tile: one of the output tile shapes (gemm_pick_tile), for which the descriptors' tile_start is filled.
constexpr int kGemmTiles = 4;
void launch_gemm_f64(const GemmDesc* d_descs, int nd, long long total_tiles, int tile, cudaStream_t s);
// The tile shape for one launch of nd problems (ksplit set) on nsm SMs.
int gemm_pick_tile(const GemmDesc* d, int nd, int nsm);
long long gemm_tiles(const GemmDesc& d, int tile);
// Tile 0 (64 x 64), in which the K splits are counted.
constexpr int kGemmRefTile = 0;
// Split-K count for one FP64 problem of a launch of launch_tiles reference tiles on nsm SMs (1: no
// split), and the partial-tile workspace (doubles) a split problem needs.
int gemm_pick_ksplit(const GemmDesc& d, long long launch_tiles, int nsm);
long long gemm_split_ws_doubles(const GemmDesc& d, int tile);
// ---- the same problems with float data in A, B and C, FP32 accumulation (gemm_f32.cu)
constexpr int kGemm32Tiles = 3;
void launch_gemm_f32(const GemmDesc* d_descs, int nd, long long total_tiles, int tile, cudaStream_t s);
int gemm32_pick_tile(const GemmDesc* d, int nd, int nsm);
long long gemm32_tiles(const GemmDesc& d, int tile);

// Device-side size bound: min(cap, mult * *p) when p is given (a rank that an earlier kernel of
// the same plan wrote), else cap.  Rows or columns beyond the bound are exactly zero in the
// operand, so the kernels leave them out.
__device__ __forceinline__ int dev_bound(int cap, const int* p, int mult) {
  return p ? min(cap, max(0, mult * *p)) : cap;
}

// Dynamic shared memory that keeps a second CTA off an SM (227 KB at most per SM and CTA).
constexpr size_t kLoneCtaSmem = 116 * 1024;
// Clusters of csize CTAs of that size which the current device holds at once.  Fewer than its SMs have room for:
// a cluster lies within one group of SMs, and what is left over of a group goes unused (of 148 SMs 15 clusters of
// eight, 33 of four).  A launch of more clusters would run in two turns where CTAs share SMs in one: 16 Jacobi
// problems of 256 x 256 2.43 ms alone on their SMs, 1.73 sharing, 35 of 128 x 128 0.96 and 0.65.
int lone_clusters(int csize);

// ---- batched Householder QR (qr_householder.cu)
// A (m x n, col-major, lda) is overwritten.  Q (m x K, ldq) and R (K x n, ldr),
// K = min(m, n), like LAPACK geqrf + orgqr (Julia `qr`, `Matrix(F.Q)`, `F.R`).
// Q == nullptr skips the Q formation, R == nullptr skips R.
struct QRDesc {
  int m, n;
  double* A; int lda;
  double* Q; int ldq;
  double* R; int ldr;
  double* Tws;      // >= ceil(K/16)*16*16 doubles of workspace for the block reflectors
  int r_trans;      // 1: R is written transposed, R^T[j][i] at R[i*ldr + j]
  // optional device bounds: rows >= m_mult * *m_dev and columns >= n_mult * *n_dev of A are
  // zero; the factorization runs on the bounded block (Q and R keep their full shapes)
  const int* m_dev; int m_mult;
  const int* n_dev; int n_mult;
  double* Rt; int ldrt;   // optional second copy of R, transposed: R^T[j][i] at Rt[i*ldrt + j]
};
constexpr int QR_MAX_M = 1536;
// dependent: as a plan's launches (launch_dep); false on a caller's stream, whose capture would take the
// programmatic edge that this makes into the caller's graph, and then cannot list its edges (cuGraphGetEdges).
void launch_qr(const QRDesc* d_descs, int count, int max_m, cudaStream_t s, int* d_flags, bool dependent = true);
// The same factorisation with every sum over all rows in one order (qr_sequential.cu).
void launch_qr_seq(const QRDesc* d_descs, int count, int max_m, cudaStream_t s, int* d_flags);

// B <- Q B with Q = H_1 ... H_K the Householder factor a QR launch left in A (reflectors below
// the diagonal, T factors in Tws): B is m x nb (ld ldb); columns >= *n_dev (when given) are
// zero and stay zero, so they are not touched.
struct QApplyDesc {
  int m, K;
  const double* A; int lda;
  const double* Tws;
  double* B; int ldb; int nb;
  const int* n_dev;
  const int* m_dev; int m_mult;   // the row bound the QR launch was given (Q acts on those rows)
};
void launch_qr_apply(const QApplyDesc* d_descs, int count, int max_m, cudaStream_t s);

// ---- batched one-sided Jacobi SVD (svd_jacobi.cu)
// X (m x n, col-major, ldx, m >= n) is overwritten by X*W whose columns are
// orthogonal; W (n x n, ldw) accumulates the rotations when not null.
// sigma[i] = ||column i||; perm lists columns by decreasing sigma.
struct JacobiDesc {
  int m, n;
  double* X; int ldx;
  double* W; int ldw;
  double* sigma;    // n
  int* perm;        // n
  int* info;        // optional: sweeps used (negative if the sweep cap was hit)
  const int* m_dev; int m_mult;   // optional: rows >= m_mult * *m_dev of X are zero
};
// `order` (count ints of device workspace, or nullptr): the launch first ranks the problems by
// their size (rows after the device bound x columns^2, largest first) so that the clusters,
// which the hardware starts in index order, take the longest problems first.
constexpr int kJacobiOrderMax = 4096;
// max_sweeps: sweep cap; a problem still rotating after it sets DFLAG_JACOBI_NOCONV.
constexpr int kJacobiDefaultSweeps = 40;
void launch_jacobi(const JacobiDesc* d_descs, int count, int max_m, int max_n, bool accw, cudaStream_t s,
                   int* d_flags, int* order = nullptr, int max_sweeps = kJacobiDefaultSweeps);

// ---- truncation rule (tt_kernels.cu): floor(s, tol) then min(k, rmax, #(s>0))
struct TruncDesc {
  const double* sigma;  // unsorted singular values
  const int* perm;      // order by decreasing sigma
  int n;                // number of singular values
  int* rank_out;        // where k is written (device rank array slot)
};
void launch_truncate(const TruncDesc* d, int count, double tol, long long rmax, cudaStream_t s);

// Build Ut (rows x cols, ld) with Ut[:, i] = X[:, perm[i]] / sigma[perm[i]] for i < k and
// 0 for i >= k (k read from *rank); with `unit_w` the columns are taken from W unscaled.
struct SelectDesc {
  const double* X; int ldx;  // source columns
  const double* sigma; const int* perm; const int* rank;
  int rows, cols;            // output rows and column capacity
  int src_cols;              // columns of X (perm entries are < src_cols)
  double* U; int ldu;
  int scale;                 // 1: divide by sigma; 0: copy; 2: multiply by sigma
  int zrows;                 // when above rows: rows [rows, zrows) of every output column are zeroed
};
void launch_select(const SelectDesc* d, int count, const ElemCount& e, cudaStream_t s);

// ---- general strided copy / permute of up to 4-D tensors (tt_kernels.cu)
// dst[i0*ds0 + i1*ds1 + i2*ds2 + i3*ds3] = alpha * src[i0*ss0 + ...] for i < ext.
struct CopyDesc {
  const double* src; double* dst;
  long long ext[4];
  long long ss[4];
  long long ds[4];
  double alpha;
};
void launch_copy(const CopyDesc* d, int count, const ElemCount& e, cudaStream_t s);

// Zero a set of flat ranges.
struct ZeroDesc { double* p; long long n; };
void launch_zero(const ZeroDesc* d, int count, const ElemCount& e, cudaStream_t s);

// Sum of squares of `n` doubles per problem, written to out[i] (FP64, deterministic order).
struct NormDesc { const double* p; long long n; double* out; };
void launch_sumsq(const NormDesc* d, int count, cudaStream_t s);

// ---- MPO x TT apply (tt_kernels.cu), src/tt_operations.jl:170-194, internal layouts.
struct ApplyDesc {
  const double* H;   // internal MPO core (R, n_out, n_in, R')  col-major
  const double* V;   // internal TT core  (r, n_in, r')         col-major
  double* Y;         // internal TT core  ((R r), n_out, (R' r')) col-major, R index fastest
  int R, Rn, r, rn, n;
};
// one CTA per right rank index nu' of each problem: grid (max rn, count).  Staged in shared memory:
// V[:, :, nu'] and, one a' at a time, H[:, :, :, a'].
__host__ __device__ inline long long apply_smem_doubles(const ApplyDesc& d) {
  return (long long)d.n * d.r + (long long)d.n * d.n * d.R;
}
void launch_apply(const ApplyDesc* d, int count, int max_rn, int max_smem_doubles, cudaStream_t s);

// ---- Philox sketch generation (tt_kernels.cu): Gaussian block entries
// dst (Julia layout of the block, flat index e) = scale * N(0,1)_{seed, stream, e}.
struct PhiloxDesc { double* dst; long long count; unsigned long long seed; unsigned stream; double scale; };
void launch_philox(const PhiloxDesc* d, int count, long long max_count, cudaStream_t s);

// ---- FP64 -> BF16 conversion and the tcgen05 BF16 GEMM (gemm_bf16_tc.cu)
// Operands are BF16, or FP32 read as TF32 in a launch with tf32 = true.
struct Bf16GemmDesc {
  int m, n, k, m0;                // m0: row split (row i = i0 + m0*i1) of the outputs
  const void* A; long long lda;   // operand type, K-major: A(i, kk) at A[i*lda + kk]
  const void* B; long long ldb;   // operand type, K-major: B(j, kk) at B[j*ldb + kk]
  double* C64; float* C32;        // outputs sharing strides: (i0*c_i0 + i1*c_i1 + j0*c_j + j1*c_j1)
  void* C16;                      // output in the operand type (BF16 or FP32), strides (h_i0, h_i1, h_j, h_j1)
  long long c_i0, c_i1, c_j, h_i0, h_i1, h_j;
  double alpha;
  long long tile_start;
  int n0;                         // column split j = j0 + n0*j1 of the outputs (0: no split)
  long long c_j1, h_j1;
};
void launch_gemm_bf16_tc(const Bf16GemmDesc* d, int nd, long long total_tiles, cudaStream_t s, int* d_flags,
                         bool tf32 = false);
long long bf16_gemm_tiles(const Bf16GemmDesc& d);
// Poll limit of the tensor-core GEMM's mbarrier waits on the current device (default 2^24); tests
// set 0 to make the waits give up on purpose.
void set_tc_wait_limit(long long polls);

}  // namespace ttc
