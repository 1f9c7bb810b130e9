// Batched one-sided (Hestenes) Jacobi SVD, FP64, one thread-block cluster per problem.
//
// Replaces the LAPACK gesdd/gesvd call of the truncated-SVD sweep
// (src/tt_rounding.jl:191-195, :235-239).  The sweep driver first QR-factors the
// unfolding, so the Jacobi input is a small square factor (one-sided Jacobi preconditioned
// by QR converges in few sweeps and keeps singular values accurate to O(eps * ||X||), the
// backward-error level of LAPACK).
//
// Parallel block ordering.  Columns are split into nblk blocks of bw columns.  One sweep =
// (a) the pairs inside every block, then (b) nblk'-1 rounds of the circle method over the
// blocks (nblk' = nblk rounded up to even): in a round the block pairs are disjoint, so the
// C CTAs of the cluster take them in turn, each streaming its two blocks from global memory
// (L2-resident) into shared memory, rotating all b x b cross pairs and writing them back.
// Rounds are separated by cluster barriers (barrier.cluster with release/acquire semantics,
// which orders the global-memory writes of one CTA before the reads of the next round);
// the "any rotation" flag of a sweep is OR-reduced into CTA 0's shared memory through
// distributed shared memory.  Control flow is identical in every CTA of a cluster, so
// every CTA reaches every barrier.
//
// Cross phase: each warp keeps its OWNT columns of the first block in registers, and only
// the partner column of the second block moves through shared memory; the OWNT rotations
// of a warp are independent and interleaved for instruction-level parallelism.
//
// Rotation: with alpha = ||x||^2, beta = ||y||^2, gamma = x.y, rotate when
// gamma^2 > tol^2 alpha beta; with d = beta - alpha and h = sqrt(d^2 + 4 gamma^2) the angle of
// modulus <= pi/4 has cos 2theta = |d|/h, sin 2theta = sign(d) 2 gamma / h, so
// c = sqrt((1 + cos 2theta)/2), s = sin 2theta / (2c) -- the rotation of Rutishauser's
// t = sign(d) 2 gamma / (|d| + h), computed with two reciprocal square roots and no division.
//
// Inert columns: a column whose squared norm is at most the numerical-zero threshold is never
// rotated (see make_rot), so its norm never changes.  Such columns (for example the
// (rank-deficient) trailing columns of an oversampled randomized-rounding factor) are left
// out of the sweeps: every CTA builds the same list of active columns and the blocks are
// gathered from it.
// alpha, beta, gamma are scaled by a power of two that brings ||X||_F^2 into [1/4, 1], so
// the squares cannot overflow or underflow (the rotation is scale invariant).
#include <cooperative_groups.h>

#include <algorithm>

#include "kernels.cuh"

namespace cg = cooperative_groups;

namespace ttc {
namespace {
constexpr int NT = 256;
constexpr int NW = NT / 32;

// Rotation threshold |a_i.a_j| > tol * ||a_i|| ||a_j|| with tol = max(m, 16) eps, the worst-case
// rounding error of an m-term FP64 dot product.  A threshold nearer the typical error
// (sqrt(m) eps) is crossed by noise alone on a few of the ~m^2/2 pairs of every sweep when m is
// a few hundred, and the iteration would never stop.
__device__ __forceinline__ double jac_tol(int m) { return (double)(m > 16 ? m : 16) * 2.220446049250313e-16; }

struct Rot { double c, s, t; bool apply; };   // t = s / c (= s rsqrt(c^2): no division)

// Parameters shared by all rotations of one problem.
struct RotCfg {
  double sc;     // power-of-two scale applied to alpha, beta, gamma
  double tol2;   // tol^2
  double zthr;   // scaled squared norm below which a column is numerically zero
};

// Columns whose squared norm is <= zthr (= (tol * ||A||_F)^2) are numerically zero: they are
// left alone, as in LAPACK's dgesvj.  Without this rule a rank-deficient matrix (more columns
// than the dimension of its column space) keeps rotating noise columns that cannot all be
// mutually orthogonal, and the iteration never stops.
__device__ __forceinline__ Rot make_rot(double alpha, double beta, double gamma, const RotCfg& q) {
  Rot r{1.0, 0.0, 0.0, false};
  alpha *= q.sc; beta *= q.sc; gamma *= q.sc;
  if (alpha <= q.zthr || beta <= q.zthr) return r;
  const double g2 = gamma * gamma;
  if (!(g2 > q.tol2 * alpha * beta)) return r;
  const double d = beta - alpha;
  const double rh = rsqrt(fma(d, d, 4.0 * g2));
  const double c2 = fma(0.5 * fabs(d), rh, 0.5);
  const double rc = rsqrt(c2);
  r.c = c2 * rc;
  r.s = copysign(1.0, d) * gamma * rh * rc;
  r.t = r.s * rc;
  r.apply = true;
  return r;
}

// Rotate columns x, y (both in shared memory, m rows) with one warp.  W columns (n rows,
// shared) follow along.  Returns whether a rotation was applied.
__device__ bool rotate_smem(double* x, double* y, int m, double* wx, double* wy, int n, const RotCfg& q) {
  const int lane = threadIdx.x & 31;
  double a = 0.0, b = 0.0, g = 0.0;
  for (int r = lane; r < m; r += 32) {
    const double u = x[r], v = y[r];
    a = fma(u, u, a); b = fma(v, v, b); g = fma(u, v, g);
  }
  a = warp_sum(a); b = warp_sum(b); g = warp_sum(g);
  const Rot R = make_rot(a, b, g, q);
  if (!R.apply) return false;
  for (int r = lane; r < m; r += 32) {
    const double u = x[r], v = y[r];
    x[r] = R.c * u - R.s * v;
    y[r] = fma(R.s, u, R.c * v);
  }
  if (wx)
    for (int r = lane; r < n; r += 32) {
      const double u = wx[r], v = wy[r];
      wx[r] = R.c * u - R.s * v;
      wy[r] = fma(R.s, u, R.c * v);
    }
  return true;
}

// Cross rotations between block I (in S0, cI columns) and block J (in S1, cJ columns), both
// of width bw = NW * OWNT.  Warp w owns the columns a = w + NW*o of block I in registers; in
// step s it rotates a against b = (a + s) mod bw of block J.  Requires m <= 32 * RPLT.
template <int OWNT, int RPLT>
__device__ __forceinline__ bool cross_regs(double* S0, double* S1, int m, int ms, int cI, int cJ, const RotCfg& q) {
  constexpr int bw = NW * OWNT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double xr[OWNT][RPLT];
#pragma unroll
  for (int o = 0; o < OWNT; ++o) {
    const int a = warp + NW * o;
#pragma unroll
    for (int t = 0; t < RPLT; ++t) {
      const int r = lane + 32 * t;
      xr[o][t] = (a < cI && r < m) ? S0[a * ms + r] : 0.0;
    }
  }
  bool any = false;
  for (int s = 0; s < bw; ++s) {
    double yr[OWNT][RPLT];
    double al[OWNT], be[OWNT], ga[OWNT];
    bool act[OWNT];
#pragma unroll
    for (int o = 0; o < OWNT; ++o) {
      const int a = warp + NW * o;
      const int b = (a + s) % bw;
      act[o] = (a < cI) && (b < cJ);
      const double* y = S1 + b * ms;
      al[o] = 0.0; be[o] = 0.0; ga[o] = 0.0;
#pragma unroll
      for (int t = 0; t < RPLT; ++t) {
        const int r = lane + 32 * t;
        yr[o][t] = (act[o] && r < m) ? y[r] : 0.0;
      }
    }
#pragma unroll
    for (int t = 0; t < RPLT; ++t)
#pragma unroll
      for (int o = 0; o < OWNT; ++o) {
        al[o] = fma(xr[o][t], xr[o][t], al[o]);
        be[o] = fma(yr[o][t], yr[o][t], be[o]);
        ga[o] = fma(xr[o][t], yr[o][t], ga[o]);
      }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
      for (int o = 0; o < OWNT; ++o) {
        al[o] += __shfl_xor_sync(0xffffffffu, al[o], off);
        be[o] += __shfl_xor_sync(0xffffffffu, be[o], off);
        ga[o] += __shfl_xor_sync(0xffffffffu, ga[o], off);
      }
#pragma unroll
    for (int o = 0; o < OWNT; ++o) {
      const Rot R = act[o] ? make_rot(al[o], be[o], ga[o], q) : Rot{1.0, 0.0, false};
      if (R.apply) {
        any = true;
        const int a = warp + NW * o;
        double* y = S1 + ((a + s) % bw) * ms;
#pragma unroll
        for (int t = 0; t < RPLT; ++t) {
          const int r = lane + 32 * t;
          const double u = xr[o][t], v = yr[o][t];
          xr[o][t] = R.c * u - R.s * v;
          if (r < m) y[r] = fma(R.s, u, R.c * v);
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int o = 0; o < OWNT; ++o) {
    const int a = warp + NW * o;
#pragma unroll
    for (int t = 0; t < RPLT; ++t) {
      const int r = lane + 32 * t;
      if (a < cI && r < m) S0[a * ms + r] = xr[o][t];
    }
  }
  return any;
}

// Cross rotations through shared memory only (W accumulation, or m beyond the register path).
__device__ bool cross_smem(double* S0, double* S1, double* W0, double* W1, int m, int ms, int n, int bw, int cI,
                           int cJ, const RotCfg& q) {
  const int warp = threadIdx.x >> 5;
  bool any = false;
  for (int s = 0; s < bw; ++s) {
    for (int a = warp; a < cI; a += NW) {
      const int b = (a + s) % bw;
      if (b < cJ)
        any |= rotate_smem(S0 + a * ms, S1 + b * ms, m, W0 ? W0 + a * n : nullptr, W1 ? W1 + b * n : nullptr, n, q);
    }
    __syncthreads();
  }
  return any;
}

// Copy `cols` columns of `rows` doubles between global memory and shared memory (or back):
// one warp per column, lanes over rows, four independent loads in flight per lane.
__device__ __forceinline__ void copy_cols(double* __restrict__ dst, long long dld, const double* __restrict__ src,
                                          long long sld, int rows, int cols) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int c = warp; c < cols; c += NW) {
    const double* sc = src + (long long)c * sld;
    double* dc = dst + (long long)c * dld;
    for (int r0 = lane; r0 < rows; r0 += 128) {
      double v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = (r0 + 32 * u < rows) ? sc[r0 + 32 * u] : 0.0;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (r0 + 32 * u < rows) dc[r0 + 32 * u] = v[u];
    }
  }
}

// One column of `rows` doubles copied by one warp (four loads in flight per lane).
__device__ __forceinline__ void copy_col_warp(double* __restrict__ dc, const double* __restrict__ sc, int rows) {
  const int lane = threadIdx.x & 31;
  for (int r0 = lane; r0 < rows; r0 += 128) {
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = (r0 + 32 * u < rows) ? sc[r0 + 32 * u] : 0.0;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (r0 + 32 * u < rows) dc[r0 + 32 * u] = v[u];
  }
}

// Gather the columns idx[0..cols) of a global matrix into packed shared-memory columns, or
// scatter them back; one warp per column.
__device__ __forceinline__ void gather_cols(double* __restrict__ dst, int dld, const double* __restrict__ src,
                                            long long ld, const int* idx, int rows, int cols) {
  for (int c = threadIdx.x >> 5; c < cols; c += NW) copy_col_warp(dst + (long long)c * dld, src + (long long)idx[c] * ld, rows);
}
__device__ __forceinline__ void scatter_cols(double* __restrict__ dst, long long ld, const double* __restrict__ src,
                                             int sld, const int* idx, int rows, int cols) {
  for (int c = threadIdx.x >> 5; c < cols; c += NW) copy_col_warp(dst + (long long)idx[c] * ld, src + (long long)c * sld, rows);
}

// Screening of a block pair in the later sweeps: whether any column pair (a of block I, b of
// block J; a < b inside one block) would be rotated.  The 16 x 16 Gram block S0^T S1 is formed
// on the FP64 tensor cores (mma.sync m8n8k4; warp w: tile w mod 4, half w / 4 of the rows) and
// tested with the column norms exactly as make_rot tests a pair.  A pair that passes needs no
// rotation, so its blocks are left as they are.  bw == 16; every thread gets the same answer.
__device__ bool screen_pair(const double* S0, const double* S1, int m, int ms, int cI, int cJ, bool same,
                            const RotCfg& q, double* scr) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, qr = lane >> 2, qc = lane & 3;
  double* nrm = scr;            // 32 column norms^2
  double* part = scr + 32;      // 4 tiles x 64 partial sums of the upper row half
  for (int c = warp; c < 32; c += NW) {
    const bool ok = (c < 16) ? (c < cI) : (c - 16 < cJ);
    const double* col = (c < 16) ? S0 + c * ms : S1 + (c - 16) * ms;
    double a = 0.0;
    if (ok)
      for (int r = lane; r < m; r += 32) a = fma(col[r], col[r], a);
    a = warp_sum(a);
    if (lane == 0) nrm[c] = a;
  }
  const int t = warp & 3, ti = t >> 1, tj = t & 1, h = warp >> 2;
  const int kh = ((m + 7) >> 3) << 2;
  const int kbeg = h ? kh : 0, kend = h ? m : (kh < m ? kh : m);
  const int ca = 8 * ti + qr, cb = 8 * tj + qr;
  double ga0 = 0.0, ga1 = 0.0, gb0 = 0.0, gb1 = 0.0;   // two accumulator chains
  for (int k0 = kbeg; k0 < kend; k0 += 8) {
    const int k = k0 + qc, k2 = k0 + 4 + qc;
    const double a = (k < kend && ca < cI) ? S0[ca * ms + k] : 0.0;
    const double b = (k < kend && cb < cJ) ? S1[cb * ms + k] : 0.0;
    const double a2 = (k2 < kend && ca < cI) ? S0[ca * ms + k2] : 0.0;
    const double b2 = (k2 < kend && cb < cJ) ? S1[cb * ms + k2] : 0.0;
    dmma(ga0, ga1, a, b);
    dmma(gb0, gb1, a2, b2);
  }
  double g0 = ga0 + gb0, g1 = ga1 + gb1;
  if (h == 1) { part[t * 64 + 2 * lane] = g0; part[t * 64 + 2 * lane + 1] = g1; }
  __syncthreads();
  int need = 0;
  if (h == 0) {
    g0 += part[t * 64 + 2 * lane];
    g1 += part[t * 64 + 2 * lane + 1];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int a = 8 * ti + qr, b = 8 * tj + 2 * qc + e;
      if (a < cI && b < cJ && (!same || a < b)) {
        const double al = nrm[a] * q.sc, be = nrm[16 + b] * q.sc, ga = (e ? g1 : g0) * q.sc;
        if (al > q.zthr && be > q.zthr && ga * ga > q.tol2 * al * be) need = 1;
      }
    }
  }
  return __syncthreads_or(need) != 0;
}

// Column position in the circle-method round robin over an even count `ne` of players.
__device__ __forceinline__ int rr_player(int pos, int round, int ne) {
  if (pos == 0) return 0;
  return ((pos - 1 + round) % (ne - 1)) + 1;
}

// Register-path dispatch on the rows per lane (bw = 16: two own columns per warp), up to
// RMAX rows per lane.
template <int RMAX>
__device__ bool cross_dispatch(double* S0, double* S1, int m, int ms, int cI, int cJ, const RotCfg& q) {
  const int rpl = (m + 31) / 32;
  if (rpl <= 2) return cross_regs<2, 2>(S0, S1, m, ms, cI, cJ, q);
  if (rpl <= 4) return cross_regs<2, 4>(S0, S1, m, ms, cI, cJ, q);
  if (RMAX <= 8 || rpl <= 8) return cross_regs<2, (RMAX < 8 ? RMAX : 8)>(S0, S1, m, ms, cI, cJ, q);
  return cross_regs<2, RMAX>(S0, S1, m, ms, cI, cJ, q);
}
}  // namespace

// Column stride of the shared blocks: rows rounded up to 4 mod 16 doubles, so the tensor-core
// fragment loads of the screening Gram (4 columns x 4 rows per half warp) hit distinct banks.
__host__ __device__ __forceinline__ int smem_stride(int m) { return m + ((4 - m) & 15); }

// Doubles of the dynamic shared memory before the active-column list: two blocks of bw
// columns of stride ms (and their W columns), at least n doubles (column norms, singular values).
__host__ __device__ __forceinline__ size_t dyn_doubles(int bw, int ms, int n, bool accw) {
  const size_t blocks = 2 * (size_t)bw * (size_t)(ms + (accw ? n : 0));
  return blocks > (size_t)n ? blocks : (size_t)n;
}

// grid = count * csize CTAs, clusters of csize CTAs (one cluster per problem).  RMAX bounds
// the register rows per lane of the cross phase (m <= 32 RMAX); RMAX = 8 keeps the kernel
// within 128 registers so that two CTAs share an SM.
template <int RMAX>
__global__ void __launch_bounds__(NT, RMAX <= 8 ? 2 : 1)
    jacobi_svd_kernel(const JacobiDesc* __restrict__ descs, const int* __restrict__ order, int bw, int csize,
                      int* flags, int max_sweeps) {
  dep_wait();
  extern __shared__ double sm[];
  __shared__ int s_any, s_nact;
  __shared__ double s_red[NW];
  __shared__ double s_scr[32 + 4 * 64];
  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)cluster.block_rank();
  const int prob = (int)(blockIdx.x / csize);
  const JacobiDesc D = descs[order ? order[prob] : prob];
  if (D.m <= 0 || D.n <= 0) return;             // uniform across the cluster
  // rows beyond the device bound are zero and stay zero under the rotations (at least one row
  // is kept so that an all-zero problem still reports its zero singular values)
  const int m = max(1, dev_bound(D.m, D.m_dev, D.m_mult)), n = D.n;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool accw = (D.W != nullptr);
  const int ms = smem_stride(m);                 // column stride of the shared blocks
  double* S0 = sm;
  double* S1 = sm + (size_t)bw * ms;
  double* W0 = S1 + (size_t)bw * ms;
  double* W1 = W0 + (accw ? (size_t)bw * n : 0);
  const bool use_regs = !accw && bw == 16 && m <= 32 * RMAX;

  if (accw) {  // W = I (columns split over the cluster)
    for (long long e = tid + (long long)crank * NT; e < (long long)n * n; e += (long long)NT * csize) {
      const int j = (int)(e / n), i = (int)(e - (long long)j * n);
      D.W[(long long)j * D.ldw + i] = (i == j) ? 1.0 : 0.0;
    }
  }
  // column norms (into sm, free until the first block load) and ||X||_F^2, which the
  // rotations leave invariant: scale and numerical-zero threshold
  int* act = reinterpret_cast<int*>(sm + dyn_doubles(bw, ms, n, accw));   // active columns
  {
    double a = 0.0;
    for (int j = warp; j < n; j += NW) {
      const double* xc = D.X + (long long)j * D.ldx;
      double cj = 0.0;
      for (int i = lane; i < m; i += 32) cj = fma(xc[i], xc[i], cj);
      cj = warp_sum(cj);
      if (lane == 0) sm[j] = cj;
      a += cj;
    }
    if (lane == 0) s_red[warp] = a;
  }
  if (tid == 0) s_any = 0;
  __syncthreads();
  double fro2 = 0.0;
#pragma unroll
  for (int i = 0; i < NW; ++i) fro2 += s_red[i];
  RotCfg q;
  {
    const double tol = jac_tol(D.m);   // the stored row count, whatever the device bound
    int e2 = 0;
    if (fro2 > 0.0 && isfinite(fro2)) { frexp(fro2, &e2); e2 = (e2 + 1) & ~1; }   // even exponent
    q.sc = (fro2 > 0.0 && isfinite(fro2)) ? ldexp(1.0, -e2) : 1.0;
    q.tol2 = tol * tol;
    q.zthr = q.tol2 * fro2 * q.sc;
  }
  if (warp == 0) {   // the same list in every CTA of the cluster
    int cnt = 0;
    for (int c0 = 0; c0 < n; c0 += 32) {
      const int c = c0 + lane;
      const bool on = (c < n) && (sm[c] * q.sc > q.zthr);
      const unsigned b = __ballot_sync(0xffffffffu, on);
      if (on) act[cnt + __popc(b & ((1u << lane) - 1u))] = c;
      cnt += __popc(b);
    }
    if (lane == 0) s_nact = cnt;
  }
  __syncthreads();
  const int na = s_nact;
  const int nblk = (na + bw - 1) / bw;
  const int ne = nblk + (nblk & 1);

  auto load_block = [&](int blk, double* S, double* Wd) {
    const int c0 = blk * bw, cn = min(bw, na - c0);
    gather_cols(S, ms, D.X, D.ldx, act + c0, m, cn);
    if (accw) gather_cols(Wd, n, D.W, D.ldw, act + c0, n, cn);
  };
  auto store_block = [&](int blk, const double* S, const double* Wd) {
    const int c0 = blk * bw, cn = min(bw, na - c0);
    scatter_cols(D.X, D.ldx, S, ms, act + c0, m, cn);
    if (accw) scatter_cols(D.W, D.ldw, Wd, n, act + c0, n, cn);
  };
  cluster.sync();   // W = I visible to every CTA

  int* any0 = cluster.map_shared_rank(&s_any, 0);
  bool converged = false;
  int sweep = 0;
  for (; sweep < max_sweeps && !converged; ++sweep) {
    bool any = false;
    const bool screen = (sweep >= 3) && (bw == 16);   // late sweeps: skip block pairs that need no rotation
    // (a) pairs inside each block; blocks dealt to the CTAs of the cluster
    for (int blk = crank; blk < nblk; blk += csize) {
      const int cI = min(bw, na - blk * bw);
      load_block(blk, S0, W0);
      __syncthreads();
      if (screen && !screen_pair(S0, S0, m, ms, cI, cI, true, q, s_scr)) continue;   // block unchanged
      const int nee = cI + (cI & 1);
      for (int rd = 0; rd < nee - 1; ++rd) {
        for (int p = warp; p < nee / 2; p += NW) {
          const int i = rr_player(p, rd, nee), j = rr_player(nee - 1 - p, rd, nee);
          if (i < cI && j < cI)
            any |= rotate_smem(S0 + i * ms, S0 + j * ms, m, accw ? W0 + i * n : nullptr, accw ? W0 + j * n : nullptr,
                               n, q);
        }
        __syncthreads();
      }
      store_block(blk, S0, W0);
      __syncthreads();
    }
    cluster.sync();
    // (b) cross pairs: circle method over the blocks, disjoint pairs per round
    for (int rd = 0; rd < ne - 1; ++rd) {
      for (int p = crank; p < ne / 2; p += csize) {
        const int bi = rr_player(p, rd, ne), bj = rr_player(ne - 1 - p, rd, ne);
        if (bi >= nblk || bj >= nblk) continue;
        const int cI = min(bw, na - bi * bw), cJ = min(bw, na - bj * bw);
        load_block(bi, S0, W0);
        load_block(bj, S1, W1);
        __syncthreads();
        if (screen && !screen_pair(S0, S1, m, ms, cI, cJ, false, q, s_scr)) continue;   // blocks unchanged
        if (use_regs) any |= cross_dispatch<RMAX>(S0, S1, m, ms, cI, cJ, q);
        else any |= cross_smem(S0, S1, accw ? W0 : nullptr, accw ? W1 : nullptr, m, ms, n, bw, cI, cJ, q);
        __syncthreads();
        store_block(bi, S0, W0);
        store_block(bj, S1, W1);
        __syncthreads();
      }
      cluster.sync();
    }
    // OR of the per-CTA flags into CTA 0; every CTA reads it; CTA 0 clears it for the next sweep
    if (any && lane == 0) atomicOr(any0, 1);
    cluster.sync();
    converged = (*any0 == 0);
    cluster.sync();
    if (crank == 0 && tid == 0) s_any = 0;
  }
  if (crank != 0) return;   // no distributed-shared-memory access follows
  if (!converged && tid == 0) atomicOr(flags, DFLAG_JACOBI_NOCONV);
  if (D.info && tid == 0) *D.info = converged ? sweep : -sweep;

  // singular values = column norms; order by decreasing value (ties by index)
  double* sig = sm;   // reuse shared memory
  for (int c = warp; c < n; c += NW) {
    double a = 0.0;
    for (int r = lane; r < m; r += 32) { const double u = D.X[(long long)c * D.ldx + r]; a = fma(u, u, a); }
    a = warp_sum(a);
    if (lane == 0) { sig[c] = sqrt(a); D.sigma[c] = sqrt(a); }
  }
  __syncthreads();
  // the keys order NaN (a non-finite input, flagged by the QR) below every singular value, so
  // that the ranks form a permutation whatever the values and perm stays a valid index list
  for (int c = tid; c < n; c += NT) {
    const double v = (sig[c] == sig[c]) ? sig[c] : -1.0;
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const double w = (sig[j] == sig[j]) ? sig[j] : -1.0;
      rank += (w > v) || (w == v && j < c);
    }
    D.perm[rank] = c;
  }
}

// Block variant for problems without W and with m <= 512 rows (the truncated-SVD sweeps).
//
// The cross steps of jacobi_svd_kernel rotate 256-row columns one pair at a time: every step
// streams a block through shared memory, reduces three dot products across the warp and waits at a
// barrier, and measured per step that is several thousand cycles, 70 % of the kernel.  Here a CTA
// takes its block pair (32 column slots: block I in slots 0-15, block J in 16-31) and
//   1. forms the 32 x 32 Gram matrix G = S^T S on the FP64 tensor cores (mma.sync m8n8k4), the ten
//      tiles on and above the diagonal, each quarter of the rows by two warps;
//   2. runs the Jacobi rotations on G instead of on the columns (two-sided: G <- J^T G J, with the
//      rotations accumulated in V, V <- V J), 16 disjoint pairs per inner round and one barrier
//      per round, on 32-element rows instead of m-row columns;
//   3. applies V to the columns with the tensor cores again (S V, m x 32 x 32), writing the result
//      straight back to the problem's columns in global memory.
// Each rotation is the one jacobi_svd_kernel would take for the same three numbers (make_rot: the
// same threshold, zero rule and formulas), computed from G's entries: alpha = G_ii, beta = G_jj,
// gamma = G_ij.  The diagonal of a rotated pair is updated as alpha - t gamma and beta + t gamma
// (t = s / c) and gamma set to zero, as in the scalar recurrences; the other entries take the rotation
// on both sides.  An entry updated this way keeps an error of the order of eps sqrt(G_ii G_kk) (the
// rotation angle of a large and a small column is small in proportion), so the decisions have the
// relative accuracy of the column-based ones (Demmel and Veselic, SIAM J. Matrix Anal. Appl. 13,
// 1992).  A block pair is left untouched (not stored) when no pair of its Gram matrix passes the
// rotation test.
// Sweep structure: the circle method over the blocks as in jacobi_svd_kernel.  In round 0 every block
// meets its partner with all 496 slot pairs (a full inner sweep, which covers the pairs inside the
// blocks); in the later rounds only the 256 cross pairs (inner round s pairs slot p with
// 16 + (p + s) mod 16).  A sweep thus visits every column pair once, and it converges when no CTA of
// the cluster rotated anything during a whole sweep.
// What bounds it: the inner rounds' chain of instructions, then the two products.  Cycles per visit of
// one 248 x 248 problem (eight CTAs) before and now: inner rounds 15200 and 9100, Gram matrix 6200 and
// 3600, S V 6600 and 5800; one such problem 1.54 and 1.09 ms, 60 of them 4.53 and 3.11 ms.
namespace {
constexpr int GLD = 36;          // leading dimension of G and V in shared memory (= 4 mod 16: no bank conflicts)
constexpr int GSZ = 32 * GLD;
constexpr int kGramPart = 640;   // the ten 8 x 8 tiles on and above the diagonal of a 32 x 32 Gram matrix

// Shared-memory doubles of a launch of jacobi_block_kernel: S (32 slots of stride ms), the two copies of
// G and V (together also the four partial Gram matrices) and the column norms (n); the active-column
// list (n ints) follows.
__host__ __device__ __forceinline__ size_t block_dyn_doubles(int ms, int n) {
  return (size_t)32 * ms + (GSZ + 4 * kGramPart) + (size_t)n;
}

__device__ __forceinline__ void cp_async8(double* dst, const double* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(double* dst, const double* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}

// make_rot without branches on scaled values, for the inner rounds' critical path: a pair that does not
// rotate gets c = 1, s = t = 0.
__device__ __forceinline__ Rot make_rot_nb(double alpha, double beta, double gamma, const RotCfg& q) {
  const double g2 = gamma * gamma, d = beta - alpha;
  const double rh = rsqrt_normal(fma(d, d, 4.0 * g2));
  const bool ap = (alpha > q.zthr) && (beta > q.zthr) && (g2 > q.tol2 * alpha * beta);
  const double c2 = fma(0.5 * fabs(d), rh, 0.5);
  const double gs = copysign(1.0, d) * (gamma * rh);
  const double rc = rsqrt_normal(c2);
  const double s = gs * rc;
  Rot r;
  r.c = ap ? c2 * rc : 1.0;
  r.s = ap ? s : 0.0;
  r.t = ap ? s * rc : 0.0;
  r.apply = ap;
  return r;
}

// Entry (i, j) of a symmetric matrix of which the part i < j is kept.
__device__ __forceinline__ int sym(int i, int j) { return min(i, j) + max(i, j) * GLD; }

// Next slot of a circle-method position: slots 1 .. 31 move round, slot 0 stays.
__device__ __forceinline__ int rr_next(int x) { return x == 0 ? 0 : (x == 31 ? 1 : x + 1); }

__device__ __forceinline__ double flip(double v, int mask) {   // v with the sign bit xor mask
  return __hiloint2double(__double2hiint(v) ^ mask, __double2loint(v));
}

// The barrier of an inner round: the warps arrive from the code of their roles.
__device__ __forceinline__ void round_barrier() {
  __syncwarp();
  asm volatile("bar.sync 1, %0;\n" ::"n"(NT) : "memory");
}

// The inner rounds on G: nr rounds of 16 disjoint pairs, pair p of round r being the slots at positions p
// and 31 - p of the circle method (FULL, 31 rounds: all pairs), or p and 16 + (p + r) mod 16 (16 rounds:
// the pairs across the blocks).  One barrier per round, the roles dealt by warps:
//  * warps 0, 1, 2 and 4 rotate the 120 off-diagonal 2 x 2 blocks of G (pairs p < q, a thread each) from
//    one copy of G into the other, so that the pre-round entries stay readable for the whole round;
//  * lanes 0-15 of warp 7 carry the pairs' own off-diagonal entries over (OFF: zero after a rotation);
//  * warps 5 and 6 rotate V, two lanes to a row, in registers ordered by position (shifted by one place
//    per round: one loop body instead of one per round, which had outgrown the instruction cache);
//  * warp 3, the critical path, with its scheduler almost to itself, computes the rotations of round r + 1, one pair a lane: its slots u, v were paired with u', v' in round r, so after round r
//      G[u,v] = c_u (c_v G[u,v] + s_v G[u,v']) + s_u (c_v G[u',v] + s_v G[u',v'])
//    with the signed sines of u and v (new u = c_u u + s_u u'), and G[u,u], G[v,v] are what the rotations
//    of round r left (alpha - t gamma, beta + t gamma).
// A pair's rotation is kept by pair index: CSP = (c, s of its first slot; the second has -s), DG = the
// two diagonal entries after it.  The place of u and v in round r (pair, side) is the same in every
// round.  Returns whether a pair rotated after round 0 (warp 3's lanes).
template <bool FULL>
__device__ __forceinline__ bool inner_rounds(double* G, double* V, double2 (*CSP)[16], double (*DG)[32], double (*OFF)[16],
                                             const RotCfg& q) {
  constexpr int NR = FULL ? 31 : 16;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  bool any = false;
  if (warp < 3 || warp == 4) {
    const int bk = warp < 3 ? tid : 96 + lane;
    int p = 0, rem = min(bk, 119);
    while (rem >= 15 - p) { rem -= 15 - p; ++p; }
    const int pq = p + 1 + rem;
    const bool on = bk < 120;
    int x = p, y = pq, x1 = FULL ? 31 - p : 16 + p, y1 = FULL ? 31 - pq : 16 + pq;
#pragma unroll 2
    for (int r = 0; r < NR; ++r) {
      const double* Gc = G + (r & 1) * GSZ;
      double* Gn = G + ((r & 1) ^ 1) * GSZ;
      const double2 A = CSP[r & 1][p], B = CSP[r & 1][pq];
      const int i00 = FULL ? sym(x, y) : x + y * GLD, i01 = FULL ? sym(x, y1) : x + y1 * GLD;
      const int i10 = FULL ? sym(x1, y) : y + x1 * GLD, i11 = sym(x1, y1);
      const double g00 = Gc[i00], g01 = Gc[i01], g10 = Gc[i10], g11 = Gc[i11];
      const double u0 = fma(A.y, g10, A.x * g00), v0 = fma(-A.y, g00, A.x * g10);
      const double u1 = fma(A.y, g11, A.x * g01), v1 = fma(-A.y, g01, A.x * g11);
      if (on) {
        Gn[i00] = fma(B.y, u1, B.x * u0);
        Gn[i01] = fma(-B.y, u0, B.x * u1);
        Gn[i10] = fma(B.y, v1, B.x * v0);
        Gn[i11] = fma(-B.y, v0, B.x * v1);
      }
      if (FULL) { x = rr_next(x); x1 = rr_next(x1); y = rr_next(y); y1 = rr_next(y1); }
      else { x1 = x1 == 31 ? 16 : x1 + 1; y1 = y1 == 31 ? 16 : y1 + 1; }
      round_barrier();
    }
  } else if (warp == 5 || warp == 6) {
    // row = 16 (warp - 5) + lane mod 16; lane half h holds the pairs 8 h .. 8 h + 7: v[k] the first slot of
    // pair 8 h + k, w[k] the second one (FULL: at positions 31 - 8 h - k)
    const int h = lane >> 4, row = 16 * (warp - 5) + (lane & 15);
    double v[8], w[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      v[k] = (8 * h + k == row) ? 1.0 : 0.0;
      w[k] = ((FULL ? 31 - 8 * h - k : 16 + 8 * h + k) == row) ? 1.0 : 0.0;
    }
    for (int r = 0; r < NR; ++r) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const double2 A = CSP[r & 1][8 * h + k];
        const double a = v[k], b = w[k];
        v[k] = fma(A.y, b, A.x * a);
        w[k] = fma(-A.y, a, A.x * b);
      }
      // one place on: position j takes the slot at j + 1 (FULL: 1 .. 31, else 16 .. 31 in a circle); one
      // slot crosses between the lane halves each way
      if (FULL) {
        const double out = __shfl_xor_sync(0xffffffffu, h ? v[0] : w[7], 16), first = v[1];
#pragma unroll
        for (int k = 0; k < 7; ++k)
          if (k > 0) v[k] = v[k + 1];
        if (h) v[0] = first;
        v[7] = h ? w[7] : out;                  // position 15 takes 16, position 7 takes 8
#pragma unroll
        for (int k = 7; k > 0; --k) w[k] = w[k - 1];
        w[0] = h ? out : first;                 // position 23 takes 24, position 31 takes 1
      } else {
        const double out = __shfl_xor_sync(0xffffffffu, w[0], 16);
#pragma unroll
        for (int k = 0; k < 7; ++k) w[k] = w[k + 1];
        w[7] = out;
      }
      round_barrier();
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      V[row + (8 * h + k) * GLD] = v[k];
      V[row + (FULL ? 31 - 8 * h - k : 16 + 8 * h + k) * GLD] = w[k];
    }
  } else if (warp == 3) {
    const int p = lane & 15;
    int u, v, u1, v1, ia, ib, da, db, ma, mb;   // slots in round r + 1 and their partners in round r
    const int neg = (int)0x80000000;
    if (FULL) {
      u = (p == 0) ? 0 : p + 1;  v = (p == 0) ? 1 : 32 - p;                 // round 1
      u1 = (p == 0) ? 31 : 30 - p;                                          // partners in round 0
      v1 = (p == 0) ? 30 : p - 1;
      const int pu = (p == 0) ? 0 : p + 1, pv = (p == 0) ? 1 : 32 - p;      // positions in round r
      ia = min(pu, 31 - pu); ma = pu > 15 ? neg : 0; da = 2 * ia + (pu > 15);
      ib = min(pv, 31 - pv); mb = pv > 15 ? neg : 0; db = 2 * ib + (pv > 15);
    } else {
      u = p; v = 16 + ((p + 1) & 15); u1 = 16 + p; v1 = (p + 1) & 15;
      ia = p; ma = 0; da = 2 * p;
      ib = (p + 1) & 15; mb = neg; db = 2 * ib + 1;
    }
#pragma unroll 2
    for (int r = 0; r < NR; ++r) {
      if (r + 1 < NR) {
        const double* Gc = G + (r & 1) * GSZ;
        const double2 A = CSP[r & 1][ia], B = CSP[r & 1][ib];
        const double al = DG[r & 1][da], be = DG[r & 1][db];
        const int j00 = FULL ? sym(u, v) : u + v * GLD, j01 = sym(u, v1);
        const int j10 = sym(u1, v), j11 = FULL ? sym(u1, v1) : v1 + u1 * GLD;
        const double g00 = Gc[j00], g01 = Gc[j01], g10 = Gc[j10], g11 = Gc[j11];
        const double su = flip(A.y, ma), sv = flip(B.y, mb);
        const double t1 = fma(sv, g01, B.x * g00), t2 = fma(sv, g11, B.x * g10);
        const double ga = fma(su, t2, A.x * t1);
        const Rot R = make_rot_nb(al, be, ga, q);
        if (lane < 16) {
          CSP[(r & 1) ^ 1][p] = make_double2(R.c, -R.s);
          *reinterpret_cast<double2*>(&DG[(r & 1) ^ 1][2 * p]) = make_double2(fma(-R.t, ga, al), fma(R.t, ga, be));
          OFF[(r & 1) ^ 1][p] = R.apply ? 0.0 : ga;
        }
        any |= R.apply;
        if (FULL) { u = rr_next(u); v = rr_next(v); u1 = rr_next(u1); v1 = rr_next(v1); }
        else { v = v == 31 ? 16 : v + 1; u1 = u1 == 31 ? 16 : u1 + 1; }
      }
      round_barrier();
    }
  } else {
    const int p = lane & 15;
    int x = p, x1 = FULL ? 31 - p : 16 + p;
    for (int r = 0; r < NR; ++r) {
      if (lane < 16) G[((r & 1) ^ 1) * GSZ + sym(x, x1)] = OFF[r & 1][p];
      if (FULL) { x = rr_next(x); x1 = rr_next(x1); }
      else x1 = x1 == 31 ? 16 : x1 + 1;
      round_barrier();
    }
  }
  return any;
}
}  // namespace

__global__ void __launch_bounds__(NT, 2)
    jacobi_block_kernel(const JacobiDesc* __restrict__ descs, const int* __restrict__ order, int csize, int* flags,
                        int max_sweeps) {
  dep_wait();
  extern __shared__ __align__(16) double sm[];
  __shared__ int s_any, s_nact;
  __shared__ double s_red[NW];
  __shared__ double2 s_csp[2][16];
  __shared__ __align__(16) double s_dg[2][32];
  __shared__ double s_off[2][16];
  __shared__ int s_rot;
  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)cluster.block_rank();
  const int prob = (int)(blockIdx.x / csize);
  const JacobiDesc D = descs[order ? order[prob] : prob];
  if (D.m <= 0 || D.n <= 0) return;             // uniform across the cluster
  const int m = max(1, dev_bound(D.m, D.m_dev, D.m_mult)), n = D.n;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, qr = lane >> 2, qc = lane & 3;
  const int ms = smem_stride(m);
  const int m4 = (m + 3) & ~3;                  // rows m .. m4 - 1 of S are zero
  double* S = sm;
  double* G = S + (size_t)32 * ms;              // G[0]; the partial Gram matrices lie behind it, over G[1] and V
  double* part = G + GSZ;
  double* V = G + 2 * GSZ;
  double* nrm = G + GSZ + 4 * kGramPart;
  int* act = reinterpret_cast<int*>(sm + block_dyn_doubles(ms, n));
  const bool vec = ((D.ldx & 1) == 0) && ((reinterpret_cast<uintptr_t>(D.X) & 15) == 0);

  // column norms and ||X||_F^2: scale and numerical-zero threshold, as in jacobi_svd_kernel
  {
    double a = 0.0;
    for (int j = warp; j < n; j += NW) {
      const double* xc = D.X + (long long)j * D.ldx;
      double cj = 0.0;
      for (int i = lane; i < m; i += 32) cj = fma(xc[i], xc[i], cj);
      cj = warp_sum(cj);
      if (lane == 0) nrm[j] = cj;
      a += cj;
    }
    if (lane == 0) s_red[warp] = a;
  }
  if (tid == 0) s_any = 0;
  __syncthreads();
  double fro2 = 0.0;
#pragma unroll
  for (int i = 0; i < NW; ++i) fro2 += s_red[i];
  RotCfg q;
  {
    const double tol = jac_tol(D.m);
    int e2 = 0;
    if (fro2 > 0.0 && isfinite(fro2)) { frexp(fro2, &e2); e2 = (e2 + 1) & ~1; }
    q.sc = (fro2 > 0.0 && isfinite(fro2)) ? ldexp(1.0, -e2) : 1.0;
    q.tol2 = tol * tol;
    q.zthr = q.tol2 * fro2 * q.sc;
  }
  if (warp == 0) {   // the same list in every CTA of the cluster
    int cnt = 0;
    for (int c0 = 0; c0 < n; c0 += 32) {
      const int c = c0 + lane;
      const bool on = (c < n) && (nrm[c] * q.sc > q.zthr);
      const unsigned b = __ballot_sync(0xffffffffu, on);
      if (on) act[cnt + __popc(b & ((1u << lane) - 1u))] = c;
      cnt += __popc(b);
    }
    if (lane == 0) s_nact = cnt;
  }
  __syncthreads();
  const int na = s_nact;
  const int nblk = (na + 15) / 16;
  const int ne = nblk + (nblk & 1);
  cluster.sync();   // every CTA of the cluster runs before the first distributed-shared-memory access

  // Gram tiles (a, b), a <= b, of 8 x 8 entries: five of them for each of the two warps that share a
  // quarter of the rows
  const int kq = ((m4 + 15) / 16) * 4, kbeg = min(m4, (warp >> 1) * kq), kend = min(m4, kbeg + kq);
  int* any0 = cluster.map_shared_rank(&s_any, 0);
  bool converged = false;
  int sweep = 0;
  for (; sweep < max_sweeps && !converged; ++sweep) {
    bool any = false;
    for (int rd = 0; rd < ne - 1; ++rd) {
      const bool full = (rd == 0);
      for (int p = crank; p < ne / 2; p += csize) {
        int bi = rr_player(p, rd, ne), bj = rr_player(ne - 1 - p, rd, ne);
        if (bi >= nblk || bj >= nblk) {       // partner is the phantom of an odd block count
          if (!full) continue;
          bi = min(bi, bj);
          bj = -1;
        }
        const int cI = min(16, na - bi * 16), cJ = bj >= 0 ? min(16, na - bj * 16) : 0;
        auto valid = [&](int slot) { return slot < 16 ? slot < cI : slot - 16 < cJ; };
        // load the valid slots: a warp per slot, lanes over rows, every copy in flight at once; the other
        // slots, and the rows up to a multiple of four, are zero
#pragma unroll
        for (int k4 = 0; k4 < 32 / NW; ++k4) {
          const int slot = warp + NW * k4;
          double* dst = S + (size_t)slot * ms;
          if (valid(slot)) {
            const double* src = D.X + (long long)act[slot < 16 ? bi * 16 + slot : bj * 16 + slot - 16] * D.ldx;
            if (vec) {
              for (int r = 2 * lane; r + 1 < m; r += 64) cp_async16(dst + r, src + r);
              if ((m & 1) && lane == 0) cp_async8(dst + m - 1, src + m - 1);
            } else {
              for (int r = lane; r < m; r += 32) cp_async8(dst + r, src + r);
            }
            if (m + lane < m4) dst[m + lane] = 0.0;
          } else {
            for (int r = lane; r < m4; r += 32) dst[r] = 0.0;
          }
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        // G = S^T S, scaled: the upper ten tiles, each quarter of the rows by two warps
        {
          const double* Sq = S + qr * ms + qc;
          const int hw = warp & 1;
          double g[5][2] = {};
          // four K steps' fragments in flight; the two halves of the tiles in loops of their own (a branch
          // inside the loop is turned into predicated multiplications, which take the tensor core's time
          // all the same: 5400 cycles against 2870 at 256 rows)
          auto loop = [&](auto step) {
            int k = kbeg;
            for (; k + 16 <= kend; k += 16) {
              double f[4][4];
#pragma unroll
              for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int t = 0; t < 4; ++t) f[u][t] = Sq[8 * t * ms + k + 4 * u];
#pragma unroll
              for (int u = 0; u < 4; ++u) step(f[u][0], f[u][1], f[u][2], f[u][3]);
            }
            for (; k < kend; k += 4) step(Sq[k], Sq[8 * ms + k], Sq[16 * ms + k], Sq[24 * ms + k]);
          };
          if (hw == 0)
            loop([&](double f0, double f1, double f2, double f3) {
              dmma(g[0][0], g[0][1], f0, f0);
              dmma(g[1][0], g[1][1], f0, f1);
              dmma(g[2][0], g[2][1], f0, f2);
              dmma(g[3][0], g[3][1], f0, f3);
              dmma(g[4][0], g[4][1], f1, f1);
            });
          else
            loop([&](double, double f1, double f2, double f3) {
              dmma(g[0][0], g[0][1], f1, f2);
              dmma(g[1][0], g[1][1], f1, f3);
              dmma(g[2][0], g[2][1], f2, f2);
              dmma(g[3][0], g[3][1], f2, f3);
              dmma(g[4][0], g[4][1], f3, f3);
            });
          double* pt = part + (warp >> 1) * kGramPart + hw * 320 + lane * 2;
#pragma unroll
          for (int t = 0; t < 5; ++t) *reinterpret_cast<double2*>(pt + 64 * t) = make_double2(g[t][0], g[t][1]);
        }
        __syncthreads();
        for (int e = tid; e < kGramPart; e += NT) {
          const double v = ((part[e] + part[kGramPart + e]) + (part[2 * kGramPart + e] + part[3 * kGramPart + e])) * q.sc;
          const int t = e >> 6, l = (e & 63) >> 1;
          const int a = t < 4 ? 0 : (t < 7 ? 1 : (t < 9 ? 2 : 3)), b = t < 4 ? t : (t < 7 ? t - 3 : (t < 9 ? t - 5 : 3));
          const int i = 8 * a + (l >> 2), j = 8 * b + 2 * (l & 3) + (e & 1);
          if (i <= j) G[i + j * GLD] = v;
        }
        __syncthreads();
        // does any pair of this visit (all slot pairs in round 0, the cross pairs later) need a rotation?
        int need = 0;
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
          const int e = tid + NT * k4, i = e & 31, j = e >> 5;
          if (i < j && (full || (i < 16 && j >= 16))) {
            const double al = G[i * (GLD + 1)], be = G[j * (GLD + 1)], ga = G[i + j * GLD];
            need |= (al > q.zthr) && (be > q.zthr) && (ga * ga > q.tol2 * al * be);
          }
        }
        if (!__syncthreads_or(need)) continue;   // block pair unchanged
        if (tid < 16) {   // the rotations of inner round 0 (pair index = tid)
          const int x = tid, y = full ? 31 - tid : 16 + tid;
          const double al = G[x * (GLD + 1)], be = G[y * (GLD + 1)], ga = G[x + y * GLD];
          const Rot R = make_rot_nb(al, be, ga, q);
          s_csp[0][tid] = make_double2(R.c, -R.s);
          s_dg[0][2 * tid] = fma(-R.t, ga, al);
          s_dg[0][2 * tid + 1] = fma(R.t, ga, be);
          s_off[0][tid] = R.apply ? 0.0 : ga;
          const unsigned b = __ballot_sync(0xffffu, R.apply);
          if (tid == 0) s_rot = b != 0;
        }
        __syncthreads();
        const bool rot = full ? inner_rounds<true>(G, V, s_csp, s_dg, s_off, q)
                              : inner_rounds<false>(G, V, s_csp, s_dg, s_off, q);
        if (rot) s_rot = 1;
        __syncthreads();   // V complete
        any |= (s_rot != 0);
        // columns <- S V, written to the problem's columns: 8-row tiles dealt to the warps, V's fragments
        // in registers
        {
          double vf[8][4];
#pragma unroll
          for (int k = 0; k < 8; ++k)
#pragma unroll
            for (int tn = 0; tn < 4; ++tn) vf[k][tn] = V[4 * k + qc + (8 * tn + qr) * GLD];
          int off[8];                           // this lane's columns of X (slots 8 tn + 2 qc + e), -1: none
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const int slot = 8 * (u >> 1) + 2 * qc + (u & 1);
            off[u] = valid(slot) ? (slot < 16 ? act[bi * 16 + slot] : act[bj * 16 + slot - 16]) * D.ldx : -1;
          }
          double a[8];
          const double* Sa = S + qc * ms;
          if (warp * 8 < m) {
#pragma unroll
            for (int k = 0; k < 8; ++k) a[k] = Sa[(size_t)(4 * k) * ms + warp * 8 + qr];
          }
          for (int r0 = warp * 8 + qr; r0 - qr < m; r0 += 8 * NW) {
            double c[4][2] = {}, an[8];
            // the next tile's rows (the last tile loads its own again) while this one is multiplied
            const double* Sn = Sa + (r0 - qr + 8 * NW < m ? r0 + 8 * NW : r0);
#pragma unroll
            for (int k = 0; k < 8; ++k) an[k] = Sn[4 * k * ms];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
#pragma unroll
              for (int tn = 0; tn < 4; ++tn) dmma(c[tn][0], c[tn][1], a[k], vf[k][tn]);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) a[k] = an[k];
            if (r0 < m) {
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (off[u] >= 0) D.X[off[u] + r0] = c[u >> 1][u & 1];
            }
          }
        }
        __syncthreads();   // S and V are read before the next visit loads
      }
      cluster.sync();      // the round's columns are in global memory for the next round's loads
    }
    if (any && lane == 0) atomicOr(any0, 1);
    cluster.sync();
    converged = (*any0 == 0);
    cluster.sync();
    if (crank == 0 && tid == 0) s_any = 0;
  }
  if (crank != 0) return;   // no distributed-shared-memory access follows
  if (!converged && tid == 0) atomicOr(flags, DFLAG_JACOBI_NOCONV);
  if (D.info && tid == 0) *D.info = converged ? sweep : -sweep;
  double* sig = nrm;
  for (int c = warp; c < n; c += NW) {
    double a = 0.0;
    for (int r = lane; r < m; r += 32) { const double u = D.X[(long long)c * D.ldx + r]; a = fma(u, u, a); }
    a = warp_sum(a);
    if (lane == 0) { sig[c] = sqrt(a); D.sigma[c] = sqrt(a); }
  }
  __syncthreads();
  for (int c = tid; c < n; c += NT) {
    const double v = (sig[c] == sig[c]) ? sig[c] : -1.0;
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const double w = (sig[j] == sig[j]) ? sig[j] : -1.0;
      rank += (w > v) || (w == v && j < c);
    }
    D.perm[rank] = c;
  }
}

// Small problems (m, n <= 32, no W): one warp per problem, L = 32 / PAIRS lanes per pair of columns, lane h of a
// pair with the rows h, h + L, ... of both (RPL of them).  Pair p holds the columns at positions p and
// ne - 1 - p of the circle method; between rounds the positions 1 .. ne - 1 move on by one, a shuffle from the
// pair above or below.  A round is then a chain of RPL products, log2 L exchanges, the rotation and the move.
// Same rotation, zero threshold and convergence rule as the cluster kernel.
// What bounds it is that chain, 600 to 800 cycles: one warp runs alone on its scheduler.  One problem of
// 8, 16, 20, 32 columns: 20, 37, 81, 149 us, where a column per lane, exchanged whole in every round with its 32
// products in a row, took 65, 145, 206, 393; 600 problems of 32 columns 221 (499).  The block kernel, a CTA
// per problem: 174 for one of 32 columns, 574 for 600.
template <int PAIRS, int RPL>
__global__ void __launch_bounds__(128) jacobi_small_kernel(const JacobiDesc* __restrict__ descs, int count, int* flags,
                                                          int max_sweeps) {
  dep_wait();
  constexpr int L = 32 / PAIRS;
  const int lane = threadIdx.x & 31, p = lane / L, h = lane % L;
  const int prob = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (prob >= count) return;                        // uniform within the warp
  const JacobiDesc D = descs[prob];
  if (D.m <= 0 || D.n <= 0) return;
  const int m = max(1, dev_bound(D.m, D.m_dev, D.m_mult)), n = D.n;
  const int ne = n + (n & 1), cx = p, cy = ne - 1 - p;   // the pair's columns before and after every sweep
  const bool live = p < ne / 2, last = p == ne / 2 - 1;
  double x[RPL], y[RPL];
  double nx = 0.0, ny = 0.0;
#pragma unroll
  for (int i = 0; i < RPL; ++i) {
    const int r = L * i + h;
    x[i] = (live && r < m) ? D.X[(long long)cx * D.ldx + r] : 0.0;
    y[i] = (live && r < m && cy < n) ? D.X[(long long)cy * D.ldx + r] : 0.0;
    nx = fma(x[i], x[i], nx);
    ny = fma(y[i], y[i], ny);
  }
  auto pair_sum = [](double v) {
#pragma unroll
    for (int o = 1; o < L; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  const double fro2 = warp_sum(nx + ny);
  RotCfg q;
  {
    const double tol = jac_tol(D.m);
    int e2 = 0;
    if (fro2 > 0.0 && isfinite(fro2)) { frexp(fro2, &e2); e2 = (e2 + 1) & ~1; }
    q.sc = (fro2 > 0.0 && isfinite(fro2)) ? ldexp(1.0, -e2) : 1.0;
    q.tol2 = tol * tol;
    q.zthr = q.tol2 * fro2 * q.sc;
  }
  bool converged = false;
  int sweep = 0;
  for (; sweep < max_sweeps && !converged; ++sweep) {
    bool any = false;
#pragma unroll 1
    for (int rd = 0; rd < ne - 1; ++rd) {
      double a = x[0] * x[0], b = y[0] * y[0], g = x[0] * y[0];
#pragma unroll
      for (int i = 1; i < RPL; ++i) {
        a = fma(x[i], x[i], a);
        b = fma(y[i], y[i], b);
        g = fma(x[i], y[i], g);
      }
      a = pair_sum(a); b = pair_sum(b); g = pair_sum(g);
      const Rot R = make_rot_nb(a * q.sc, b * q.sc, g * q.sc, q);
      any |= R.apply;
#pragma unroll
      for (int i = 0; i < RPL; ++i) {
        const double u = R.c * x[i] - R.s * y[i], v = fma(R.s, x[i], R.c * y[i]);
        const double up = __shfl_down_sync(0xffffffffu, u, L), dn = __shfl_up_sync(0xffffffffu, v, L);
        x[i] = p == 0 ? u : last ? v : up;
        y[i] = p == 0 ? (last ? v : up) : dn;
      }
    }
    converged = !__any_sync(0xffffffffu, any);
  }
  if (!converged && lane == 0) atomicOr(flags, DFLAG_JACOBI_NOCONV);
  if (D.info && lane == 0) *D.info = converged ? sweep : -sweep;
  nx = ny = 0.0;
#pragma unroll
  for (int i = 0; i < RPL; ++i) {
    nx = fma(x[i], x[i], nx);
    ny = fma(y[i], y[i], ny);
  }
  nx = sqrt(pair_sum(nx));
  ny = sqrt(pair_sum(ny));
#pragma unroll
  for (int i = 0; i < RPL; ++i) {
    const int r = L * i + h;
    if (live && r < m) {
      D.X[(long long)cx * D.ldx + r] = x[i];
      if (cy < n) D.X[(long long)cy * D.ldx + r] = y[i];
    }
  }
  // ranking by decreasing value (NaN last, ties by index), as in the cluster kernel
  const double kx = nx == nx ? nx : -1.0, ky = ny == ny ? ny : -1.0;
  int rx = 0, ry = 0;
  for (int j = 0; j < n; ++j) {
    const double w = j < ne / 2 ? __shfl_sync(0xffffffffu, kx, L * j) : __shfl_sync(0xffffffffu, ky, L * (ne - 1 - j));
    rx += (w > kx) || (w == kx && j < cx);
    ry += (w > ky) || (w == ky && j < cy);
  }
  if (live && h == 0) {
    D.sigma[cx] = nx;
    D.perm[rx] = cx;
    if (cy < n) {
      D.sigma[cy] = ny;
      D.perm[ry] = cy;
    }
  }
}

// Problem order of a launch: by decreasing size m x n^2, m the rows left by the device bound and
// n the columns (at most m when bounded: the bounded factor is square), ties by index.
__global__ void jacobi_order_kernel(const JacobiDesc* __restrict__ descs, int count, int* __restrict__ order) {
  dep_wait();
  for (int i = threadIdx.x; i < count; i += blockDim.x) {
    auto key = [&](int j) {
      const JacobiDesc& d = descs[j];
      const double m = dev_bound(d.m, d.m_dev, d.m_mult);
      const double n = d.m_dev ? fmin((double)d.n, m) : (double)d.n;
      return m * n * n;
    };
    const double ki = key(i);
    int rank = 0;
    for (int j = 0; j < count; ++j) {
      const double kj = key(j);
      rank += (kj > ki) || (kj == ki && j < i);
    }
    order[rank] = i;
  }
}


// Block width and dynamic shared memory of a launch: dyn_doubles(bw, ...) doubles and the
// active-column list (max_n ints).
static int jacobi_bw(int max_m, int max_n, bool accw, size_t* smem_out) {
  int bw = 16;
  auto need = [&](int b) {
    return sizeof(double) * dyn_doubles(b, smem_stride(max_m), max_n, accw) + sizeof(int) * (size_t)max_n;
  };
  while (bw > 1 && need(bw) > 200 * 1024) bw >>= 1;
  *smem_out = need(bw);
  return bw;
}

// Cluster size of an ordered launch (measured on the 64-TT rounding: 8 for the two-CTA-per-SM
// instance, 4 for the one-CTA-per-SM instance; 8 there runs 3.5 waves and loses).
template <int RMAX>
constexpr int kOrderedCsize = RMAX <= 8 ? 8 : 4;
template <int RMAX>
static int jacobi_cluster_size(int count, int max_n, int bw, size_t smem, bool ordered) {
  // CTAs per problem: fill the SMs (resident CTAs per SM from registers and shared memory),
  // at most 8 (portable cluster size) and at most the disjoint block pairs of a round.  With
  // the problems ordered largest first the grid may exceed the resident slots (the clusters
  // that start later take the smaller problems): then at least kOrderedCsize<RMAX>.
  int per_sm = 1;
  TTC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, jacobi_svd_kernel<RMAX>, NT, smem));
  per_sm = std::max(1, per_sm);
  const int slots = current_sm_count() * per_sm;
  const int pairs = std::max(1, ((max_n + bw - 1) / bw + 1) / 2);
  int c = std::max(1, slots / std::max(1, count));
  if (ordered) c = std::max(c, kOrderedCsize<RMAX>);
  c = std::min(c, std::min(8, pairs));
  int p2 = 1;
  while (p2 * 2 <= c) p2 *= 2;
  return p2;
}

template <int RMAX>
static void launch_jacobi_t(const JacobiDesc* d_descs, int count, int max_n, int bw, size_t smem, cudaStream_t s,
                            int* d_flags, int* order, int max_sweeps) {
  static PerDeviceOnce attr_once;
  int dev = 0;
  TTC_CUDA(cudaGetDevice(&dev));
  attr_once.run(dev, [] {
    TTC_CUDA(cudaFuncSetAttribute(jacobi_svd_kernel<RMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  });
  if (order) {
    launch_dep(jacobi_order_kernel, 1, 512, 0, s, d_descs, count, order);
    TTC_CHECK_LAUNCH();
  }
  const int csize = jacobi_cluster_size<RMAX>(count, max_n, bw, smem, order != nullptr);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(count * csize));
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)csize;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  TTC_CUDA(cudaLaunchKernelEx(&cfg, jacobi_svd_kernel<RMAX>, d_descs, (const int*)order, bw, csize, d_flags,
                              max_sweeps));
  TTC_CHECK_LAUNCH();
}

// Cluster size of a jacobi_block_kernel launch: as jacobi_cluster_size, for the block kernel's
// occupancy (two CTAs per SM up to 256 rows, one beyond).
static int jacobi_block_csize(int count, int max_n, size_t smem, bool ordered) {
  int per_sm = 1;
  TTC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, jacobi_block_kernel, NT, smem));
  per_sm = std::max(1, per_sm);
  const int slots = current_sm_count() * per_sm;
  const int pairs = std::max(1, ((max_n + 15) / 16 + 1) / 2);
  int c = std::max(1, slots / std::max(1, count));
  if (ordered) c = std::max(c, per_sm >= 2 ? 8 : 4);
  c = std::min(c, std::min(8, pairs));
  // a power of two, rounded up when the launch is ordered: a problem whose block pairs outnumber
  // its CTAs takes two visits per round, which doubles its latency
  int p2 = 1;
  if (ordered) while (p2 < c) p2 *= 2;
  else while (p2 * 2 <= c) p2 *= 2;
  return p2;
}

static void launch_jacobi_block(const JacobiDesc* d_descs, int count, int max_m, int max_n, cudaStream_t s,
                                int* d_flags, int* order, int max_sweeps) {
  static PerDeviceOnce attr_once;
  int dev = 0;
  TTC_CUDA(cudaGetDevice(&dev));
  attr_once.run(dev, [] {
    TTC_CUDA(cudaFuncSetAttribute(jacobi_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  });
  const size_t smem = sizeof(double) * block_dyn_doubles(smem_stride(max_m), max_n) + sizeof(int) * (size_t)max_n;
  TTC_REQUIRE(smem <= 200 * 1024, TTC_EDIM, "jacobi: matrix too large for the shared-memory blocks");
  if (order) {
    launch_dep(jacobi_order_kernel, 1, 512, 0, s, d_descs, count, order);
    TTC_CHECK_LAUNCH();
  }
  const int csize = jacobi_block_csize(count, max_n, smem, order != nullptr);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(count * csize));
  cfg.blockDim = dim3(NT);
  // Launches that leave every CTA an SM of its own ask for more than half of an SM's shared memory:
  // otherwise two CTAs of a cluster may land on one SM and share its tensor cores (one 248 x 248 problem
  // 1.37 ms, 1.30 apart)
  cfg.dynamicSmemBytes = count <= lone_clusters(csize) ? std::max(smem, kLoneCtaSmem) : smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)csize;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  TTC_CUDA(cudaLaunchKernelEx(&cfg, jacobi_block_kernel, d_descs, (const int*)order, csize, d_flags, max_sweeps));
  TTC_CHECK_LAUNCH();
}

void launch_jacobi(const JacobiDesc* d_descs, int count, int max_m, int max_n, bool accw, cudaStream_t s,
                   int* d_flags, int* order, int max_sweeps) {
  if (count <= 0) return;
  TTC_REQUIRE(max_sweeps >= 1, TTC_EARG, "jacobi: the sweep cap must be at least 1");
  size_t smem = 0;
  const int bw = jacobi_bw(max_m, max_n, accw, &smem);
  TTC_REQUIRE(smem <= 200 * 1024, TTC_EDIM, "jacobi: matrix too large for the shared-memory blocks");
  if (count > kJacobiOrderMax) order = nullptr;
  if (!accw && max_m <= 32 && max_n <= 32) {       // every problem fits one warp's registers
    const unsigned grid = (unsigned)((count + 3) / 4);
    if (max_m <= 16 && max_n <= 16) launch_dep(jacobi_small_kernel<8, 4>, grid, 128, 0, s, d_descs, count, d_flags, max_sweeps);
    else launch_dep(jacobi_small_kernel<16, 16>, grid, 128, 0, s, d_descs, count, d_flags, max_sweeps);
    TTC_CHECK_LAUNCH();
    return;
  }
  if (!accw && max_m <= 512) {
    launch_jacobi_block(d_descs, count, max_m, max_n, s, d_flags, order, max_sweeps);
    return;
  }
  if (max_m <= 256) launch_jacobi_t<8>(d_descs, count, max_n, bw, smem, s, d_flags, order, max_sweeps);
  else launch_jacobi_t<16>(d_descs, count, max_n, bw, smem, s, d_flags, order, max_sweeps);
}

}  // namespace ttc
