// Householder QR of the range finders of operator and Hadamard products (rand_rounding_general,
// hadamard_rounding_host), row-sequential: every product with a column is summed over all rows by one
// warp in one fixed order, whatever the cluster size.
//
// The sketches of these roundings are recursive Gaussian ones, whose right-hand levels multiply square
// Gaussian blocks (b_k = n b_{k+1}): Z = y_k W_{k+1} reaches condition numbers of 1e8 (rank 138, 32
// sites), and its trailing Q columns follow the rounding of every sum to eight digits.  The kernel of
// qr_householder.cu, which shares a column's rows between warps, gives there another, equally accurate
// basis (1.7e-8 from the 64-bit result's either way, 1e-8 from each other); this one returns the basis
// that results of these roundings were stored with.  It costs 243 us for 276 x 138 with Q, the other 184.
//
// Every sum keeps its order whatever the split of the work: a change of the kernel must not move a bit.
// What bounds it: the 16 column steps of a panel, 1300 cycles each at 276 rows (a barrier, a warp's sum over
// its lanes and the reflector's scalars twice over, and the shared memory's bandwidth for x, which 15 warps
// read), then the L2 latency of the panels and the trailing columns, which few warps walk.  With Q: 276 x 138
// 346 -> 243 us, 640 x 320 1300 -> 964, 1024 x 256 1650 -> 1131 from one warp per octet of the block products,
// loads one 32-row chunk ahead, panels above 512 rows in shared memory and the scalars in every warp.
//
// Layout: panels of NB = 16 columns are factored in shared memory (reflectors with the
// LAPACK dlarfg convention beta = -sign(alpha)*||x||), the block reflector
// I - V T V^T (dlarft) is applied to the trailing columns, and Q is formed backwards from the stored
// panels (dorgqr).
//
// One thread-block cluster of C CTAs per problem.  Every CTA factors each panel itself
// (same data, same arithmetic: identical reflectors, no broadcast needed); the column octets
// (8o .. 8o+7) of the trailing update and of Q are owned by CTA o mod C, so a column is always
// updated by the same CTA.  The block reflectors are applied on the FP64 tensor cores
// (mma.sync m8n8k4).  A cluster barrier (release/acquire at cluster scope) after each
// panel's trailing update makes the next panel visible to every CTA.  The CTAs write the
// factored panel's columns in turn and CTA 0 the T factors, which the Q formation reads.
#include <cooperative_groups.h>

#include <algorithm>

#include "kernels.cuh"

namespace cg = cooperative_groups;

namespace ttc {
namespace {
constexpr int NB = 16;
constexpr int NT = 512;
constexpr int NW = NT / 32;

// Shared memory, in doubles.
constexpr int kT = 0;                    // NB*NB  T of the panel, T[col * NB + row] (upper triangular)
constexpr int kTau = kT + NB * NB;       // NB
constexpr int kRed = kTau + NB;          // NW
constexpr int kSv = kRed + NW;           // NB     reflector scales 1/(alpha - beta)
constexpr int kBet = kSv + NB;           // NB     betas (diagonal of R)
constexpr int kNrm = kBet + NB;          // 2      squared norm below the diagonal of the next column
constexpr int kGs = kNrm + 2;            // NB*NB  x_l . x_i below row i (l < i), unscaled
constexpr int kG = kGs + NB * NB;        // NB*NB  V^T V
constexpr int kTop = kG + NB * NB;       // NB*NB  R's part of the panel, top[col * NB + row]
constexpr int kW = kTop + NB * NB;       // NW/2*256  the W of the octets in work
constexpr int kU = kW + NW / 2 * 256;    // NW/2*128  and their -U
constexpr int kP = kU + NW / 2 * 128;    // panel, panel_ld x NB
extern __shared__ __align__(16) double sm[];   // T is read in pairs

// Block-wide sum; `red` holds NW doubles.  All threads get the result.
__device__ double block_sum(double v, double* red) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int i = 0; i < NW; ++i) s += red[i];
  return s;
}

// 8 bytes global -> shared, asynchronous
__device__ __forceinline__ void cp8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// Stride of a panel of mp rows in shared memory: whole 128-row batches and 4 (4 mod 16, so that the fragment
// loads of 4 rows x 8 columns meet distinct banks).
__host__ __device__ __forceinline__ int panel_ld(int mp) { return (mp + 127) / 128 * 128 + 4; }

// Starts the copy of jb panel columns of mp rows into shared memory (one commit group), a warp per column;
// rows from mp to the end of the last batch, and the columns from jb to NB, become zero.
__device__ __forceinline__ void panel_load(double* P, const double* __restrict__ src, long long ld, int mp, int jb) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mp_ld = panel_ld(mp);
  double* pc = P + warp * mp_ld;
  const double* sc = src + warp * ld;
  for (int r = lane; r < mp_ld - 4; r += 32) {
    if (warp < jb && r < mp) cp8(pc + r, sc + r);
    else pc[r] = 0.0;
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void panel_wait() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// T of a panel from T^{-1} + T^{-T} = V^T V (compact WY): T^{-1} = striu(G) + diag(1/tau), so
// T[r][j] = -tau_r sum_{r < l <= j} G[r][l] T[l][j], T[j][j] = tau_j; lane j of the
// calling warp back-substitutes column j in registers (a zero tau gives a zero row, as in dlarft).
__device__ __noinline__ void form_t(int jb) {
  const double* G = sm + kG;
  const double* tau = sm + kTau;
  const int j = threadIdx.x & 31;
  if (j >= NB) return;
  double tc[NB];
#pragma unroll
  for (int k = 0; k < NB; ++k) tc[k] = (k == j && j < jb) ? tau[k] : 0.0;
#pragma unroll
  for (int r = NB - 2; r >= 0; --r) {
    double a2 = 0.0;
#pragma unroll
    for (int l = r + 1; l < NB; ++l) a2 = fma(G[l * NB + r], tc[l], a2);
    if (r < j && j < jb) tc[r] = -tau[r] * a2;
  }
#pragma unroll
  for (int k = 0; k < NB; ++k) sm[kT + j * NB + k] = tc[k];
}

// The sums of W = V^T C for NH halves of the reflectors from l0 on, over the even (odd = 0) or odd 4-row steps:
// 16 steps (128 rows) at a time, the next ones' loads in flight while they are multiplied (a load takes 700
// cycles, the products of a half 28 each).
template <int NH>
__device__ __forceinline__ void w_sums(double* Ws, const double* V, int mp_ld, int mp, const double* __restrict__ colb,
                                       bool cb_ok, int odd, int l0) {
  const int lane = threadIdx.x & 31, qr = lane >> 2, qc = lane & 3;
  const int q = 4 * odd + qc;
  const double* v = V + (l0 + qr) * mp_ld + q;
  double w[NH][2] = {};
  double bb[16];
#pragma unroll
  for (int u = 0; u < 16; ++u) {
    const int r = 8 * u + q;
    bb[u] = (cb_ok && r < mp) ? colb[r] : 0.0;
  }
#pragma unroll 1
  for (int k0 = 0; k0 < mp; k0 += 128) {
    double bn[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int r = k0 + 128 + 8 * u + q;
      bn[u] = (cb_ok && r < mp) ? colb[r] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 16; ++u)
#pragma unroll
      for (int h = 0; h < NH; ++h) dmma(w[h][0], w[h][1], v[8 * h * mp_ld + k0 + 8 * u], bb[u]);
#pragma unroll
    for (int u = 0; u < 16; ++u) bb[u] = bn[u];
  }
#pragma unroll
  for (int h = 0; h < NH; ++h) {
    double* o = Ws + 128 * odd + (l0 + 8 * h + qr) * 8 + 2 * qc;
    o[0] = w[h][0];
    o[1] = w[h][1];
  }
}

// Apply I - V S V^T to columns [c_begin, c_end) of the global matrix M (rows r0..m-1, ld), with V (mp x jb,
// panel_load's layout) and S^T in shared memory: T there applies I - V T^T V^T, its transpose I - V T V^T.
// Octet o of 8 columns belongs to CTA o mod csize; G warps share one, NW / G octets at a time.  Both
// products run on the FP64 tensor cores: W (16 x 8) = V^T C accumulated over 4-row steps, U = S W,
// then C -= V U per 8-row tile.  W is always four sums (reflectors 0-7 and 8-15, even and odd steps), and the
// tiles of C do not meet, so the warps divide the sums and the tiles and no result depends on G.
// With `make_t`, the last warp forms T first, which is used after a barrier.  Every warp of the CTA calls this
// (it holds barriers).  The code is kept short, loops and one body for every G: unrolled per G it was slower
// than one warp per octet, every panel reading its instructions anew (8400 cycles for U, 11700 for W).
__device__ __noinline__ void apply_block_reflector(double* M, long long ld, int r0, int m, int c_begin, int c_end, int jb,
                                                   bool make_t, int crank, int csize) {
  const double* V = sm + kP;
  const double* T = sm + kT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qr = lane >> 2, qc = lane & 3;
  const int mp = m - r0, mp_ld = panel_ld(mp);
  const int o_begin = c_begin >> 3, o_end = (c_end + 7) >> 3;
  const int o_first = o_begin + ((crank - o_begin) % csize + csize) % csize;
  const int mine = o_first < o_end ? (o_end - 1 - o_first) / csize + 1 : 0;
  const int lg = mine <= NW / 4 ? 2 : 1;                    // log2 of G
  const int G = 1 << lg, g = warp & (G - 1), slot = warp >> lg;
  double* Ws = sm + kW + slot * 256;
  double* Us = sm + kU + slot * 128;
  if (make_t && warp == NW - 1) form_t(jb);
  bool first = true;
  for (int ob = o_first; first || ob < o_end; ob += (NW >> lg) * csize) {
    const int c0 = 8 * (ob + slot * csize);
    const bool live = ob + slot * csize < o_end;
    if (live) {
      // pass 1: this warp's sums of W
      const int cb = c0 + qr;
      const bool cb_ok = cb >= c_begin && cb < c_end;
      const double* colb = M + (cb_ok ? cb : c_begin) * ld + r0;
      if (G == 4) w_sums<1>(Ws, V, mp_ld, mp, colb, cb_ok, g & 1, 4 * (g & 2));
      else w_sums<2>(Ws, V, mp_ld, mp, colb, cb_ok, g, 0);
    }
    first = false;
    __syncthreads();
    if (live) {
      // U = S W, its rows in turn among the octet's warps; -U is kept
#pragma unroll 1
      for (int l = 4 * g + qc; l < NB; l += 4 * G) {
        double u = 0.0;
#pragma unroll
        for (int i = 0; i < NB; i += 2) {
          const double2 tv = *reinterpret_cast<const double2*>(&T[l * NB + i]);
          u = fma(tv.x, Ws[i * 8 + qr] + Ws[128 + i * 8 + qr], u);
          u = fma(tv.y, Ws[i * 8 + 8 + qr] + Ws[136 + i * 8 + qr], u);
        }
        Us[l * 8 + qr] = -u;
      }
    }
    __syncthreads();
    if (live) {
      double ub[4];
#pragma unroll
      for (int sidx = 0; sidx < 4; ++sidx) ub[sidx] = Us[(4 * sidx + qc) * 8 + qr];
      // pass 2: C[rt..rt+7][c0..c0+7] -= V[rt.., 0..15] U; 32-row sets of four 8-row tiles, every G-th set, the
      // next one's loads in flight while one is multiplied and stored
      const int ca = c0 + 2 * qc;
      const bool ok0 = ca >= c_begin && ca < c_end, ok1 = ca + 1 >= c_begin && ca + 1 < c_end;
      double* col0 = M + (ok0 ? ca : c_begin) * ld + r0;
      double* col1 = M + (ok1 ? ca + 1 : c_begin) * ld + r0;
      double d0[4], d1[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = 32 * g + 8 * u + qr;
        d0[u] = (ok0 && r < mp) ? col0[r] : 0.0;
        d1[u] = (ok1 && r < mp) ? col1[r] : 0.0;
      }
#pragma unroll 1
      for (int rt = 32 * g; rt < mp; rt += 32 * G) {
        double e0[4], e1[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int r = rt + 32 * G + 8 * u + qr;
          e0[u] = (ok0 && r < mp) ? col0[r] : 0.0;
          e1[u] = (ok1 && r < mp) ? col1[r] : 0.0;
        }
        const double* v = V + qc * mp_ld + rt + qr;
#pragma unroll
        for (int sidx = 0; sidx < 4; ++sidx)
#pragma unroll
          for (int u = 0; u < 4; ++u) dmma(d0[u], d1[u], v[4 * sidx * mp_ld + 8 * u], ub[sidx]);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int r = rt + 8 * u + qr;
          if (ok0 && r < mp) col0[r] = d0[u];
          if (ok1 && r < mp) col1[r] = d1[u];
          d0[u] = e0[u];
          d1[u] = e1[u];
        }
      }
    }
    __syncthreads();                                       // W and U are rewritten for the next octets
  }
}

// Column steps of a panel held in registers (panel rows mp <= 32 * RMAX): warp w keeps panel
// column (w + 1) mod NW, lane l its rows l + 32 i, for the whole panel.  Step jj reads only the
// reflector column x = P[:, jj] and its diagonal from shared memory.  While the warp of column jj, which
// has nothing left to do with it, forms the reflector's scalars (dlarfg: a square root and two divisions, as
// long as a product with a column), the others form theirs, x . c; then the warps of the columns
// c > jj apply reflector jj to their column (x unscaled, as in the shared-memory loop below), those of the
// finished columns c < jj note x_c . x_jj below row jj for V^T V, and the warp of column jj + 1 returns its
// squared norm below the diagonal and publishes the column to P, where it is the next step's reflector.
// The order of the sums: up to 512 rows lane l adds its rows in four chains, i mod 4.  Above (RMAX > 16), as
// the shared-memory loop adds: two chains, and the lanes are added up counted from row jj + 1.
template <int RMAX>
__device__ __noinline__ bool panel_steps_regs(int mp, int jb) {
  double *P = sm + kP, *nrm2 = sm + kNrm, *tau = sm + kTau, *sv = sm + kSv, *bet = sm + kBet, *gs = sm + kGs;
  constexpr bool WIDE = RMAX > 16;
  constexpr int NC = WIDE ? 2 : 4;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mp_ld = panel_ld(mp);
  const int c = (warp + 1) % NW;
  const bool own = c < jb;
  double* pc = P + c * mp_ld + lane;
  double cr[RMAX];
  bool bad = false;
#pragma unroll
  for (int i = 0; i < RMAX; ++i) {
    cr[i] = pc[32 * i];                                    // rows from mp on are zero
    bad |= !isfinite(cr[i]);
  }
  auto total = [&](const double (&v)[NC], int jj) {
    if (!WIDE) return warp_sum((v[0] + v[1]) + (v[2 % NC] + v[3 % NC]));
    return warp_sum(__shfl_sync(0xffffffffu, v[0] + v[1], (lane + jj + 1) & 31));
  };
#pragma unroll 1
  for (int jj = 0; jj < jb; ++jj) {
    const double* x = P + jj * mp_ld + lane;
    double xv[4];
    double d = 0.0;
    if (c == jj) {
      const double s = nrm2[jj & 1], alpha = P[jj * mp_ld + jj];
      double beta = alpha, t = 0.0, scal = 0.0;
      if (s != 0.0) {
        beta = -copysign(sqrt(fma(alpha, alpha, s)), alpha);
        t = (beta - alpha) / beta;
        scal = 1.0 / (alpha - beta);
      }
      if (lane == 0) { tau[jj] = t; sv[jj] = scal; bet[jj] = beta; }
    } else if (own) {
      double dd[NC] = {};
#pragma unroll
      for (int i = 0; i < RMAX; i += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) xv[u] = x[32 * (i + u)];
        if (i == 0 && lane <= jj) xv[0] = 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u) dd[u % NC] = fma(xv[u], cr[i + u], dd[u % NC]);
      }
      d = total(dd, jj);
    }
    __syncthreads();
    if (own && c < jj) {
      if (lane == 0) gs[c * NB + jj] = d;
    } else if (own && c > jj) {
      const double t = tau[jj], scal = sv[jj];
      const double cj = __shfl_sync(0xffffffffu, cr[0], jj);   // row jj < 32: lane jj, i = 0
      const double w = fma(scal, d, cj) * t;                   // tau v^T c
      const double ws = w * scal;
#pragma unroll
      for (int i = 0; i < RMAX; i += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u) xv[u] = x[32 * (i + u)];
        if (i == 0 && lane <= jj) xv[0] = 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u) cr[i + u] = fma(-ws, xv[u], cr[i + u]);
      }
      const double below = lane > jj + 1 ? cr[0] : 0.0;
      if (lane == jj) cr[0] = cj - w;
      if (c == jj + 1) {
        double qq[NC] = {};
        qq[0] = fma(below, below, 0.0);
#pragma unroll
        for (int i = 0; i < RMAX; ++i) {
          pc[32 * i] = cr[i];
          if (i > 0) qq[i % NC] = fma(cr[i], cr[i], qq[i % NC]);
        }
        const double q = total(qq, jj);
        if (lane == 0) nrm2[(jj + 1) & 1] = q;
      }
    }
    __syncthreads();
  }
  return bad;
}

}  // namespace

__global__ void __launch_bounds__(NT, 1) householder_qr_seq_kernel(const QRDesc* __restrict__ descs, int csize, int* flags) {
  dep_wait();
  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)cluster.block_rank();
  const QRDesc D = descs[blockIdx.x / csize];
  if (D.m <= 0 || D.n <= 0) return;
  // the factored block (rows and columns beyond the device bounds are zero) and the shapes of
  // R (Kc x D.n) and Q (D.m x Kc)
  const int m = dev_bound(D.m, D.m_dev, D.m_mult), n = dev_bound(D.n, D.n_dev, D.n_mult);
  const int K = min(m, n), Kc = min(D.m, D.n);
  double *T = sm + kT, *tau = sm + kTau, *red = sm + kRed, *sv = sm + kSv, *bet = sm + kBet, *nrm2 = sm + kNrm;
  double *gs = sm + kGs, *G = sm + kG, *top = sm + kTop, *P = sm + kP;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  double* A = D.A;
  const int lda = D.lda;
  bool nonfinite = false;

  for (int j0 = 0; j0 < K; j0 += NB) {
    const int jb = min(NB, K - j0);
    const int mp = m - j0;
    const int mp_ld = panel_ld(mp);
    // 1. load panel
    panel_load(P, A + (long long)j0 * lda + j0, lda, mp, jb);
    panel_wait();
    __syncthreads();
    // this CTA has read the panel; CTA 0 overwrites it only when all have
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    // 2. factor panel, one CTA barrier per column: reflector jj (dlarfg: beta =
    //    -sign(alpha) ||(alpha, x)||, tau = (beta - alpha)/beta, v = [1; x/(alpha - beta)]) is
    //    applied to columns c > jj with x unscaled; the warp that updates column jj+1 also
    //    returns its squared norm below the diagonal for the next reflector.  The reflector
    //    columns are scaled, and the betas stored, after the loop.
    {
      double s0 = 0.0;
      for (int r = 1 + tid; r < mp; r += NT) { const double x = P[r]; s0 = fma(x, x, s0); }
      s0 = block_sum(s0, red);
      if (tid == 0) nrm2[0] = s0;
      __syncthreads();
    }
    // the panel's own row count picks the column-step routine (uniform across the cluster):
    // registers up to 1024 rows, else the shared-memory loop below
    switch ((mp + 127) / 128) {
      case 1: nonfinite |= panel_steps_regs<4>(mp, jb); break;
      case 2: nonfinite |= panel_steps_regs<8>(mp, jb); break;
      case 3: nonfinite |= panel_steps_regs<12>(mp, jb); break;
      case 4: nonfinite |= panel_steps_regs<16>(mp, jb); break;
      case 5: nonfinite |= panel_steps_regs<20>(mp, jb); break;
      case 6: nonfinite |= panel_steps_regs<24>(mp, jb); break;
      case 7: nonfinite |= panel_steps_regs<28>(mp, jb); break;
      case 8: nonfinite |= panel_steps_regs<32>(mp, jb); break;
      default:
        for (int r = lane; r < mp; r += 32) nonfinite |= !isfinite(P[warp * mp_ld + r]);
        __syncthreads();
    }
    if (mp > 1024) for (int jj = 0; jj < jb; ++jj) {
      const double s = nrm2[jj & 1];
      const double alpha = P[jj * mp_ld + jj];
      double beta, t, scal;
      if (s == 0.0) { t = 0.0; beta = alpha; scal = 0.0; }
      else {
        beta = -copysign(sqrt(fma(alpha, alpha, s)), alpha);
        t = (beta - alpha) / beta;
        scal = 1.0 / (alpha - beta);
      }
      const double* x = P + jj * mp_ld;
      // slot k of warp k mod NW: column k < jj gives x_k . x_jj below row jj (for V^T V),
      // column k + 1 > jj gets the reflector
      for (int k = warp; k < jb - 1; k += NW) {
        if (k < jj) {
          const double* pl = P + k * mp_ld;
          double g = 0.0, g2 = 0.0;
          for (int r = jj + 1 + lane; r < mp; r += 64) {
            g = fma(pl[r], x[r], g);
            if (r + 32 < mp) g2 = fma(pl[r + 32], x[r + 32], g2);
          }
          g = warp_sum(g + g2);
          if (lane == 0) gs[k * NB + jj] = g;
          continue;
        }
        const int c = k + 1;
        double* pc = P + c * mp_ld;
        const double cj = pc[jj];
        double d = 0.0, d2 = 0.0;       // two chains
        for (int r = jj + 1 + lane; r < mp; r += 64) {
          d = fma(x[r], pc[r], d);
          if (r + 32 < mp) d2 = fma(x[r + 32], pc[r + 32], d2);
        }
        d = warp_sum(d + d2);
        const double w = fma(scal, d, cj) * t;     // tau v^T c
        const double ws = w * scal;
        double q = 0.0, q2 = 0.0;
        for (int r = jj + 1 + lane; r < mp; r += 64) {
          const double u = fma(-ws, x[r], pc[r]);
          pc[r] = u;
          if (r > jj + 1) q = fma(u, u, q);
          if (r + 32 < mp) {
            const double u2 = fma(-ws, x[r + 32], pc[r + 32]);
            pc[r + 32] = u2;
            q2 = fma(u2, u2, q2);
          }
        }
        q += q2;
        if (c == jj + 1) {
          q = warp_sum(q);
          if (lane == 0) nrm2[(jj + 1) & 1] = q;
        }
        if (lane == 0) pc[jj] = cj - w;
      }
      if (tid == 0) { tau[jj] = t; sv[jj] = scal; bet[jj] = beta; }
      __syncthreads();
    }
    // 3. G = V^T V (l < i) from the dot products of the panel loop: v_l[i] = scal_l x_l[i], v_i[i] = 1, rows
    //    below i scaled by both (x unscaled here and there)
    for (int e = tid; e < NB * NB; e += NT) {
      const int i = e / NB, l = e - i * NB;
      if (l < i) G[i * NB + l] = (i < jb) ? sv[l] * fma(sv[i], gs[l * NB + i], P[l * mp_ld + i]) : 0.0;
    }
    __syncthreads();
    for (int c = warp; c < jb; c += NW) {
      double* pc = P + c * mp_ld;
      const double sc = sv[c];
      for (int r = c + 1 + lane; r < mp; r += 32) pc[r] *= sc;
      if (lane <= c) {                               // the entries of R aside, V's unit triangle in their place
        top[c * NB + lane] = lane == c ? bet[c] : pc[lane];
        pc[lane] = lane == c ? 1.0 : 0.0;
      }
    }
    __syncthreads();
    // 4. trailing update with H^T = I - V T^T V^T (this CTA's column octets); T is formed between its passes
    if (j0 + jb < n) {
      apply_block_reflector(A, lda, j0, m, j0 + jb, n, jb, true, crank, csize);
    } else {
      if (warp == 0) form_t(jb);
      __syncthreads();
    }
    // 5. the CTAs write back the panel's columns in turn, CTA 0 keeps T
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    for (int c = crank + csize * warp; c < jb; c += csize * NW)
      for (int r = lane; r < mp; r += 32) A[(long long)(j0 + c) * lda + j0 + r] = r <= c ? top[c * NB + r] : P[c * mp_ld + r];
    if (crank == 0 && D.Tws)
      for (int e = tid; e < NB * NB; e += NT) D.Tws[(j0 / NB) * NB * NB + e] = T[e];
    cluster.sync();   // trailing columns and the panel visible to every CTA
  }
  if (nonfinite && crank == 0) atomicOr(flags, DFLAG_NONFINITE);

  // R = upper triangle of A[0:Kc, 0:D.n] (zero outside the factored block)
  if (D.R) {
    for (int j = (int)(threadIdx.x >> 5) + NW * crank; j < D.n; j += NW * csize)
      for (int i = (int)(threadIdx.x & 31); i < Kc; i += 32) {
        const double v = (i <= j) ? A[(long long)j * lda + i] : 0.0;
        if (D.r_trans) D.R[(long long)i * D.ldr + j] = v;
        else D.R[(long long)j * D.ldr + i] = v;
        if (D.Rt) D.Rt[(long long)i * D.ldrt + j] = v;
      }
  }
  if (!D.Q) return;
  // Q = H_1 ... H_K [I; 0], accumulated backwards panel by panel.  Each CTA initialises
  // and updates only its own column octets, so the panels need no barrier between them.
  // The reflectors act on rows < m; identity columns c >= K are untouched unless a column
  // bound leaves some of them with c < m.
  for (int c = 0; c < Kc; ++c) {
    if (((c >> 3) % csize) != crank) continue;
    for (int i = tid; i < D.m; i += NT) D.Q[(long long)c * D.ldq + i] = (i == c) ? 1.0 : 0.0;
  }
  __syncthreads();
  const int qc_end = (n < D.n) ? Kc : K;
  const int npan = (K + NB - 1) / NB;
  for (int p = npan - 1; p >= 0; --p) {
    const int j0 = p * NB, jb = min(NB, K - j0), mp = m - j0;
    panel_load(P, A + (long long)j0 * lda + j0, lda, mp, jb);
    for (int e = tid; e < NB * NB; e += NT) T[e % NB * NB + e / NB] = D.Tws[p * NB * NB + e];   // T^T
    panel_wait();
    __syncwarp();
    if (warp < jb && lane <= warp) P[warp * panel_ld(mp) + lane] = lane == warp ? 1.0 : 0.0;   // V's triangle
    __syncthreads();
    apply_block_reflector(D.Q, D.ldq, j0, m, j0, qc_end, jb, false, crank, csize);
  }
}

namespace {
size_t qr_smem(int max_m) {
  return sizeof(double) * (kP + (size_t)panel_ld(max_m) * NB);
}

constexpr int kQrWaves = 2;
void launch_qr_cfg(const QRDesc* d_descs, int count, int max_m, cudaStream_t s, int* d_flags) {
  const size_t smem = qr_smem(max_m);
  static PerDeviceOnce attr_once;
  int dev = 0;
  TTC_CUDA(cudaGetDevice(&dev));
  attr_once.run(dev, [] {
    TTC_CUDA(cudaFuncSetAttribute(householder_qr_seq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)qr_smem(QR_MAX_M)));
  });
  const int nsm = current_sm_count();
  // CTAs per problem: up to two waves of the resident-CTA slots of the GPU (the planner puts the
  // largest problems first, so the second wave holds the short ones), at most 8 (portable cluster)
  int per_sm = 1;
  TTC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, householder_qr_seq_kernel, NT, smem));
  const int slots = nsm * std::max(1, per_sm);
  int c = std::min(8, std::max(1, kQrWaves * slots / count));
  int csize = 1;
  while (csize * 2 <= c) csize *= 2;
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
  TTC_CUDA(cudaLaunchKernelEx(&cfg, householder_qr_seq_kernel, d_descs, csize, d_flags));
  TTC_CHECK_LAUNCH();
}
}  // namespace

void launch_qr_seq(const QRDesc* d_descs, int count, int max_m, cudaStream_t s, int* d_flags) {
  if (count <= 0) return;
  TTC_REQUIRE(max_m <= QR_MAX_M, TTC_EDIM, "qr: row count exceeds the supported maximum (1536)");
  launch_qr_cfg(d_descs, count, max_m, s, d_flags);
}

}  // namespace ttc
