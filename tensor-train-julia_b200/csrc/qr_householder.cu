// Batched blocked Householder QR, one thread-block cluster per problem.
//
// Replaces Julia `qr(A)` / `qr!(Z)` + `Matrix(F.Q)` (LAPACK geqrf + orgqr) on the
// tall-skinny unfoldings of the orthogonalisation sweep (src/tt_rounding.jl:75-78) and of
// the randomized range finder (src/tt_randtools.jl:134-135).  Householder is used (not
// CholeskyQR) because the range-finder matrices are rank deficient by construction when
// the sketch rank exceeds the TT rank, and zero-padded cores give exactly zero columns;
// Householder returns an orthonormal Q for any input, like LAPACK.
//
// Layout: panels of NB = 16 columns are factored in registers (reflectors with the LAPACK dlarfg
// convention beta = -sign(alpha)*||x||), the block reflector I - V T V^T (dlarft) is applied to
// the trailing columns in octets of 8, several warps sharing an octet's rows, and Q is formed
// backwards from the stored panels (dorgqr).
//
// One thread-block cluster of C CTAs per problem.  Every CTA factors each panel itself
// (same data, same arithmetic: identical reflectors, no broadcast needed); the column octets
// (8o .. 8o+7) of the trailing update and of Q are owned by CTA o mod C, so a column is always
// updated by the same CTA.  The block reflectors are applied on the FP64 tensor cores
// (mma.sync m8n8k4).  A cluster barrier (release/acquire at cluster scope) after each
// panel's trailing update makes the next panel visible to every CTA.  The CTAs write the
// factored panel's columns in turn and CTA 0 the T factors, which the Q formation reads after one
// more barrier.
//
// What bounds it: the chain of column steps (n of them, one barrier each), so a step is kept
// short: the columns of the panel stay in registers, the reflector column is published once in
// shared memory with its leading rows zeroed (no row masks in the dot products and updates), and
// the scalars of a reflector (one reciprocal square root and one reciprocal, no branch) are computed
// while the dot products are reduced.  Cycles per column step on one SM, with a square root and two
// divisions in every warp and the columns in shared memory before: 64 rows 2020, now 790; 256 rows
// 2290 and 1020; 512 rows 5600 and 1600.  One problem with Q: 128 x 64 126 us before and 65 now,
// 256 x 256 530 and 293, 512 x 256 870 and 446; the QR family of a 64-TT rounding 32.9
// and 20.7 ms.
// The rest is the trailing update and the Q formation, on 8-column octets held in registers from the
// first product to the second (read and written once; 0.33 and 0.52 of 2.5 M cycles for 512 x 256
// before, 0.14 and 0.17 now).
#include <cooperative_groups.h>

#include <algorithm>

#include "kernels.cuh"

namespace cg = cooperative_groups;

namespace ttc {
namespace {
constexpr int NB = 16;

__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }

// Rows r and r + 1 (r even) of a column with mp rows, zero where masked.  VEC: one 16-byte access; the
// columns are 16-byte aligned and mp is even (vec_ok).
template <bool VEC>
__device__ __forceinline__ void load2(double (&v)[2], const double* col, int r, int mp, bool on) {
  if (VEC) {
    double2 t = make_double2(0.0, 0.0);
    if (on && r < mp) t = *reinterpret_cast<const double2*>(col + r);
    v[0] = t.x; v[1] = t.y;
  } else {
    v[0] = (on && r < mp) ? col[r] : 0.0;
    v[1] = (on && r + 1 < mp) ? col[r + 1] : 0.0;
  }
}
template <bool VEC>
__device__ __forceinline__ void store2(const double (&v)[2], double* col, int r, int mp, bool on) {
  if (VEC) {
    if (on && r < mp) *reinterpret_cast<double2*>(col + r) = make_double2(v[0], v[1]);
  } else {
    if (on && r < mp) col[r] = v[0];
    if (on && r + 1 < mp) col[r + 1] = v[1];
  }
}
__device__ __forceinline__ bool vec_ok(const double* p, int ld, int mp) {
  return ((reinterpret_cast<uintptr_t>(p) & 15) == 0) && (((ld | mp) & 1) == 0);
}

// The reflectors V of a panel in shared memory: column l at l * panel_ld(mp), its rows in groups of
// eight whose two halves are swapped in the columns with bit 1 of l set.  With a column stride of
// 8 mod 16 doubles the fragment loads of both passes of apply_block meet no bank twice.  The unit
// diagonal and the zeros above it and below row mp (to the next multiple of 8) are stored.
__host__ __device__ __forceinline__ int panel_ld(int mp) {
  const int r = (mp + 7) & ~7;
  return (r & 15) ? r : r + 8;
}
__device__ __forceinline__ int panel_at(int l, int r, int ld) { return l * ld + (r ^ (((l >> 1) & 1) << 2)); }

// Shared-memory doubles before the panel: T, the scalars, two NB x NB tables and the exchange
// buffer of apply_block.
template <int NW>
constexpr int kExchange = (NW <= 8 ? 2 : 1) * NW * 128;
template <int NW>
constexpr int kFixed = 3 * NB * NB + 4 * NB + kExchange<NW>;

// Apply (I - V T^T V^T) [trans] or (I - V T V^T) to columns [c_begin, c_end) and rows r0 .. r0 + mp - 1
// of the global matrix M, with V (16 columns) in shared memory at p_off as above, T[col * 16 + row] at the
// start of shared memory and the exchange buffer behind it.  G
// warps share an octet of 8 columns, warp g its 8-row tiles g, g + G, ..., which it holds in
// registers from the first pass to the second, so the columns are read and written once.  Both
// passes run on the FP64 tensor cores, transposed:
//   pass 1  W^T (8 x 16) += C^T V   (K = 4 rows of a tile at a time, rows 2 qc + s in step s)
//   U^T = W^T T or W^T T^T, whose column order gives lane qc the entries 4 s + qc of pass 2
//   pass 2  C^T (8 x 8 rows) -= U^T V^T
// Rows mp must not exceed 8 G MAXT.
template <int NW, int G, int MAXT>
__device__ __noinline__ void apply_block_g(double* M, int ld, int r0, int mp, int c_begin, int c_end, int p_off,
                                           bool trans, int crank, int csize) {
  extern __shared__ __align__(16) double sm[];
  const double* T = sm;
  double* Wx = sm + NB * NB;
  const double* P = sm + p_off;
  const int mp_ld = panel_ld(mp);
  constexpr int NG = NW / G;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, qr = lane >> 2, qc = lane & 3;
  const int grp = warp / G, gw = warp % G;
  const bool vec = vec_ok(M + r0, ld, mp);
  const int o_begin = c_begin >> 3, o_end = (c_end + 7) >> 3;
  const int o_first = o_begin + ((crank - o_begin) % csize + csize) % csize;
  if (o_first + grp * csize >= o_end) return;
  // B fragments of the U product: T[l][sigma] (trans) or T[sigma][l], l = 8 h + 2 qc + e,
  // sigma = (qr >> 1) + 4 (qr & 1) + 8 h2
  double tf[2][2][2];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int h2 = 0; h2 < 2; ++h2) {
        const int l = 8 * h + 2 * qc + e, sg = (qr >> 1) + 4 * (qr & 1) + 8 * h2;
        tf[h][e][h2] = trans ? T[sg * NB + l] : T[l * NB + sg];
      }
  const double* p1 = P + qr * mp_ld + ((2 * qc) ^ (((qr >> 1) & 1) << 2));   // pass 1: columns qr, qr + 8
  const double* p2 = P + qc * mp_ld + (qr ^ (((qc >> 1) & 1) << 2));         // pass 2: columns 4 s + qc
  int it = 0;
  for (int o = o_first + grp * csize; o < o_end; o += NG * csize, ++it) {
    const int c = 8 * o + qr;
    const bool cok = (c >= c_begin && c < c_end);
    double* col = M + (long long)(cok ? c : c_begin) * ld + r0;
    double cc[MAXT][2];
    if (vec) {
#pragma unroll
      for (int t = 0; t < MAXT; ++t) load2<true>(cc[t], col, 8 * (gw + G * t) + 2 * qc, mp, cok);
    } else {
#pragma unroll
      for (int t = 0; t < MAXT; ++t) load2<false>(cc[t], col, 8 * (gw + G * t) + 2 * qc, mp, cok);
    }
    double w[2][2][2] = {};
#pragma unroll
    for (int t = 0; t < MAXT; ++t) {
      // leave the loop: multiplications predicated off would take the tensor core's time all the same
      const int rt = 8 * (gw + G * t);
      if (rt >= mp) break;
      const double2 v0 = *reinterpret_cast<const double2*>(p1 + rt);
      const double2 v1 = *reinterpret_cast<const double2*>(p1 + 8 * mp_ld + rt);
      dmma(w[0][0][0], w[0][0][1], cc[t][0], v0.x);
      dmma(w[1][0][0], w[1][0][1], cc[t][0], v1.x);
      dmma(w[0][1][0], w[0][1][1], cc[t][1], v0.y);
      dmma(w[1][1][0], w[1][1][1], cc[t][1], v1.y);
    }
    double ws[2][2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e) ws[h][e] = w[h][0][e] + w[h][1][e];
    if (G > 1) {   // add the G partial products in the same order in every warp
      double* X = Wx + ((NW <= 8) ? (it & 1) * NW * 128 : 0) + grp * G * 128;
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<double2*>(X + gw * 128 + h * 64 + lane * 2) = make_double2(ws[h][0], ws[h][1]);
      asm volatile("bar.sync %0, %1;\n" ::"r"(1 + grp), "n"(G * 32) : "memory");
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        double2 a = *reinterpret_cast<const double2*>(X + h * 64 + lane * 2);
#pragma unroll
        for (int g = 1; g < G; ++g) {
          const double2 b = *reinterpret_cast<const double2*>(X + g * 128 + h * 64 + lane * 2);
          a.x += b.x; a.y += b.y;
        }
        ws[h][0] = a.x; ws[h][1] = a.y;
      }
      // with one buffer, every read is done before the next octet's writes
      if (NW > 8) asm volatile("bar.sync %0, %1;\n" ::"r"(1 + grp), "n"(G * 32) : "memory");
    }
    double u[2][2] = {};
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) dmma(u[h2][0], u[h2][1], ws[h][e], tf[h][e][h2]);
#pragma unroll
    for (int t = 0; t < MAXT; ++t) {
      const int rt = 8 * (gw + G * t);
      if (rt >= mp) break;
#pragma unroll
      for (int s = 0; s < 4; ++s) dmma(cc[t][0], cc[t][1], -u[s >> 1][s & 1], p2[4 * s * mp_ld + rt]);
      if (vec) store2<true>(cc[t], col, rt + 2 * qc, mp, cok);
      else store2<false>(cc[t], col, rt + 2 * qc, mp, cok);
    }
  }
}

// Warps per octet by the panel's rows: 16 tiles of 8 rows per warp at most.
template <int NW>
__device__ __forceinline__ void apply_block(double* M, int ld, int r0, int mp, int c_begin, int c_end, int p_off,
                                            bool trans, int crank, int csize) {
  if constexpr (NW <= 8) {
    if (mp <= 256) apply_block_g<NW, 4, 8>(M, ld, r0, mp, c_begin, c_end, p_off, trans, crank, csize);
    else apply_block_g<NW, 4, 16>(M, ld, r0, mp, c_begin, c_end, p_off, trans, crank, csize);
  } else {
    if (mp <= 512) apply_block_g<NW, 8, 8>(M, ld, r0, mp, c_begin, c_end, p_off, trans, crank, csize);
    else if (mp <= 1024) apply_block_g<NW, 8, 16>(M, ld, r0, mp, c_begin, c_end, p_off, trans, crank, csize);
    else apply_block_g<NW, 16, 12>(M, ld, r0, mp, c_begin, c_end, p_off, trans, crank, csize);
  }
}

// A stored panel (R in and above its diagonal, the reflectors below) into shared memory as V.
template <int NW>
__device__ __forceinline__ void load_panel_v(double* P, int mp_ld, const double* A, int lda, int mp, int jb) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool vec = vec_ok(A, lda, mp);
  const int mp8 = (mp + 7) & ~7;
#pragma unroll
  for (int q = 0; q < NB / NW; ++q) {
    const int c = warp + NW * q;
    const double* col = A + (long long)c * lda;
    for (int b = 2 * lane; b < mp8; b += 512) {
      double v[8][2];
      if (vec) {
#pragma unroll
        for (int i = 0; i < 8; ++i) load2<true>(v[i], col, b + 64 * i, mp, c < jb);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) load2<false>(v[i], col, b + 64 * i, mp, c < jb);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = b + 64 * i;
        if (i == 0 && r < NB) {
          if (r <= c) v[i][0] = (r == c && c < jb) ? 1.0 : 0.0;
          if (r + 1 <= c) v[i][1] = (r + 1 == c && c < jb) ? 1.0 : 0.0;
        }
        if (r < mp8) *reinterpret_cast<double2*>(P + panel_at(c, r, mp_ld)) = make_double2(v[i][0], v[i][1]);
      }
    }
  }
}

// Shared-memory tables of a panel's factorisation.
struct PanelSm {
  double *T, *sv, *tau, *pub, *gs, *xl, *Wx, *P;
};
template <int NW>
__device__ __forceinline__ PanelSm panel_sm(double* sm) {
  PanelSm S;
  S.T = sm;                          // NB*NB
  S.Wx = S.T + NB * NB;              // exchange buffer of apply_block
  S.gs = S.Wx + kExchange<NW>;       // NB*NB  x_l . x_i below row i (l < i), unscaled; then V^T V
  S.xl = S.gs + NB * NB;             // NB*NB  x_l[i] (l < i), unscaled
  S.sv = S.xl + NB * NB;             // NB     reflector scales 1/(alpha - beta)
  S.tau = S.sv + NB;                 // NB
  S.pub = S.tau + NB;                // 2*NB   alpha and squared norm below the diagonal of the published columns
  S.P = S.pub + 2 * NB;              // panel, 16 columns of panel_ld(mp)
  return S;
}

// The reflector of a column step from the published alpha and s = ||x||^2: with norm = ||(alpha, x)||,
// beta = -sign(alpha) norm, v = [alpha - beta; x] and g = |alpha| + norm, H = I - v v^T / (norm g), that
// is c -= ws v with ws = (v^T c) rn rg.  H = I (nz false) when x = 0 or the squared norm is subnormal
// (a column of norm below 2e-154, whose square would carry no digits).
struct Reflector {
  double alpha, norm, rn, rg;
  bool nz;
  __device__ __forceinline__ explicit Reflector(double2 as) {
    const double n2 = fma(as.x, as.x, as.y);
    alpha = as.x;
    nz = as.y != 0.0 && n2 >= 2.2250738585072014e-308;
    rn = rsqrt_normal(n2);
    norm = n2 * rn;
    rg = rcp_normal(fabs(as.x) + norm);
  }
  __device__ __forceinline__ double u() const { return copysign(fabs(alpha) + norm, alpha); }        // alpha - beta
  __device__ __forceinline__ double tau() const { return nz ? fma(fabs(alpha), rn, 1.0) : 0.0; }     // (beta - alpha) / beta
  __device__ __forceinline__ double scale() const { return nz ? copysign(rg, alpha) : 0.0; }         // 1 / (alpha - beta)
  __device__ __forceinline__ double beta() const { return nz ? -copysign(norm, alpha) : alpha; }
};

// T from the products gs, xl and the scales, by one warp.  G = V^T V (l < i): v_l[i] = scal_l x_l[i],
// v_i[i] = 1, rows below i scaled by both.  T forward (dlarft): T[r][l] = -tau_l sum_{r <= k < l} T[r][k]
// G[k][l], T[l][l] = tau_l; lane r holds row r and adds T[r][l] G[l][j] to every later column's sum at
// once.  Loads, chain and stores are kept apart, so that no load waits for a store.
template <int NW>
__device__ __forceinline__ void form_t(const PanelSm& S, int jb, double* Tg) {
  const int lane = threadIdx.x & 31, r = lane & 15;
  double a[NB];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int e = lane + 32 * k, l = e >> 4, i = e & 15;
    a[k] = (l < i && i < jb) ? S.sv[l] * fma(S.sv[i], S.gs[e], S.xl[e]) : 0.0;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) S.gs[lane + 32 * k] = a[k];
  __syncwarp();
#pragma unroll
  for (int j = 0; j < NB; ++j) a[j] = 0.0;
  double2 g[NB / 2], gn[NB / 2];
  const double2* gr = reinterpret_cast<const double2*>(S.gs);
#pragma unroll
  for (int k = 0; k < NB / 2; ++k) g[k] = gr[k];
  double tl = S.tau[0];
#pragma unroll
  for (int l = 0; l < NB; ++l) {
    double tn = 0.0;
    if (l + 1 < NB) {                          // row l + 1 while row l is used
      tn = S.tau[l + 1];
#pragma unroll
      for (int k = (l + 2) / 2; k < NB / 2; ++k) gn[k] = gr[(l + 1) * (NB / 2) + k];
    }
    a[l] = (r == l) ? tl : (r < l ? -tl * a[l] : 0.0);
#pragma unroll
    for (int j = l + 1; j < NB; ++j) a[j] = fma(a[l], (j & 1) ? g[j / 2].y : g[j / 2].x, a[j]);
#pragma unroll
    for (int k = 0; k < NB / 2; ++k) g[k] = gn[k];
    tl = tn;
  }
  if (lane < NB) {
#pragma unroll
    for (int l = 0; l < NB; ++l) S.T[l * NB + r] = a[l];
    if (Tg) {
#pragma unroll
      for (int l = 0; l < NB; ++l) Tg[l * NB + r] = a[l];
    }
  }
}

// One panel: A points at its first diagonal entry, mp rows, jb <= 16 columns.  A column belongs to LPC
// lanes of a warp, lane hl holding its rows 2 LPC i + 2 hl + {0, 1} in registers (mp <= 2 LPC RI); a
// warp has CW adjacent columns, side by side (LPC = 32 / CW) or CPW to a lane (LPC = 32).
// Column step jj: the reflector column x = column jj below row jj lies in shared memory, zero in the
// rows <= jj and beyond mp, with its squared norm and alpha.  Every column forms x . c; the columns
// c > jj then take the reflector (x unscaled), for c < jj the product is an entry of V^T V.  The warp of
// column jj + 1 publishes that column and its squared norm.  The reflectors are scaled, and T formed,
// after the last step.
// The panel is factored times a power of two that brings its largest entry to 2^480, so that no square
// leaves the normal range (columns of norms from 1e-290 to 1e300; without it from 1.5e-154 to 1e154): the
// reflectors and T do not depend on the scale, and R takes it back.  Every operation commutes with it, so it
// does not change a bit of what is in range without it.
template <int NW, int LPC, int RI>
__device__ __noinline__ bool factor_panel(double* A, int lda, int mp, int jb, int crank, int csize, double* Tws) {
  extern __shared__ __align__(16) double sm[];
  const PanelSm S = panel_sm<NW>(sm);
  const int mp_ld = panel_ld(mp);
  constexpr int CW = NB / NW, CPW = CW * LPC / 32, CH = 2 * LPC, XLD = CH * RI;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, hl = lane & (LPC - 1);
  const int c0 = warp * CW + lane / LPC;      // column q of this lane: c0 + q
  const bool vec = vec_ok(A, lda, mp);
  double* X = S.P;                            // two published columns (the panel region is free until the end)
  double cr[CPW][RI][2];
  if (vec) {
#pragma unroll
    for (int q = 0; q < CPW; ++q)
#pragma unroll
      for (int i = 0; i < RI; ++i)
        load2<true>(cr[q][i], A + (long long)(c0 + q) * lda, CH * i + 2 * hl, mp, c0 + q < jb);
  } else {
#pragma unroll
    for (int q = 0; q < CPW; ++q)
#pragma unroll
      for (int i = 0; i < RI; ++i)
        load2<false>(cr[q][i], A + (long long)(c0 + q) * lda, CH * i + 2 * hl, mp, c0 + q < jb);
  }
  int hi = 0;
#pragma unroll
  for (int q = 0; q < CPW; ++q)
#pragma unroll
    for (int i = 0; i < RI; ++i)
      hi = max(hi, max(__double2hiint(cr[q][i][0]) & 0x7fffffff, __double2hiint(cr[q][i][1]) & 0x7fffffff));
  hi = __reduce_max_sync(0xffffffffu, hi);
  int* his = reinterpret_cast<int*>(S.sv);    // free until the scales are written
  if (lane == 0) his[warp] = hi;
  __syncwarp();
  cluster_arrive();                           // this CTA has read the panel (waited for before it is overwritten)
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NW; ++w) hi = max(hi, his[w]);
  const int sh = min(1000, 480 - ((hi >> 20) - 1023));
  const double up = __hiloint2double((1023 + sh) << 20, 0), down = __hiloint2double((1023 - sh) << 20, 0);
#pragma unroll
  for (int q = 0; q < CPW; ++q)
#pragma unroll
    for (int i = 0; i < RI; ++i) { cr[q][i][0] *= up; cr[q][i][1] *= up; }

  // column j = c0 + q of some lanes of this warp
  auto publish = [&](const double (&v)[RI][2], int j, bool me) {
    double* x = X + (j & 1) * XLD + 2 * hl;
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    {
      const int r = 2 * hl;
      const double v0 = (r > j) ? v[0][0] : 0.0, v1 = (r + 1 > j) ? v[0][1] : 0.0;
      if (me) *reinterpret_cast<double2*>(x) = make_double2(v0, v1);
      if (me && hl < NB / 2) *reinterpret_cast<double2*>(S.xl + j * NB + 2 * hl) = make_double2(v0, v1);
      a[0] = v0 * v0; a[1] = v1 * v1;
    }
#pragma unroll
    for (int i = 1; i < RI; ++i) {
      if (me) *reinterpret_cast<double2*>(x + CH * i) = make_double2(v[i][0], v[i][1]);
      a[2 * (i & 1)] = fma(v[i][0], v[i][0], a[2 * (i & 1)]);
      a[2 * (i & 1) + 1] = fma(v[i][1], v[i][1], a[2 * (i & 1) + 1]);
    }
    double s = RI > 1 ? (a[0] + a[1]) + (a[2] + a[3]) : a[0] + a[1];
#pragma unroll
    for (int o = LPC / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (me && hl == (j >> 1)) *reinterpret_cast<double2*>(S.pub + 2 * j) = make_double2((j & 1) ? v[0][1] : v[0][0], s);
  };
  if (warp == 0) publish(cr[0], 0, c0 == 0);

  // unrolled by two (the parity of jj is then fixed): in full, the loop outgrows the instruction cache
#pragma unroll 2
  for (int jj = 0; jj < NB; ++jj) {
    if (jj >= jb) break;
    __syncthreads();
    const double* x = X + (jj & 1) * XLD + 2 * hl;
    const double2 as = *reinterpret_cast<const double2*>(S.pub + 2 * jj);
    constexpr bool KEEP = (1 + CPW) * RI <= 16;   // x stays in registers from the product to the update
    double xr[KEEP ? RI : 1][2];
    double acc[CPW][4] = {};
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      if (!KEEP && i > 0 && i % 4 == 0) asm volatile("" ::: "memory");   // bounds the loads hoisted at once
      const double2 t = *reinterpret_cast<const double2*>(x + CH * i);
      if (KEEP) { xr[i][0] = t.x; xr[i][1] = t.y; }
#pragma unroll
      for (int q = 0; q < CPW; ++q) {
        acc[q][2 * (i & 1)] = fma(t.x, cr[q][i][0], acc[q][2 * (i & 1)]);
        acc[q][2 * (i & 1) + 1] = fma(t.y, cr[q][i][1], acc[q][2 * (i & 1) + 1]);
      }
    }
    double d[CPW];
#pragma unroll
    for (int q = 0; q < CPW; ++q)
      d[q] = RI > 1 ? (acc[q][0] + acc[q][1]) + (acc[q][2] + acc[q][3]) : acc[q][0] + acc[q][1];
    const Reflector H(as);                    // the scalars, without branches, beside the reduction of the products
#pragma unroll
    for (int o = LPC / 2; o > 0; o >>= 1)
#pragma unroll
      for (int q = 0; q < CPW; ++q) d[q] += __shfl_xor_sync(0xffffffffu, d[q], o);
#pragma unroll
    for (int q = 0; q < CPW; ++q)
      if (c0 + q < jj && hl == 0) S.gs[(c0 + q) * NB + jj] = d[q];
    if (warp * CW + CW - 1 > jj) {            // a column of this warp is not finished
      const double u = H.u(), rr = H.rn * H.rg;
#pragma unroll
      for (int q = 0; q < CPW; ++q) {
        const int c = c0 + q;
        const double cj = __shfl_sync(0xffffffffu, (jj & 1) ? cr[q][0][1] : cr[q][0][0], (lane & ~(LPC - 1)) | (jj >> 1));
        const bool on = c > jj && H.nz;
        const double ws = on ? rr * fma(u, cj, d[q]) : 0.0;
#pragma unroll
        for (int i = 0; i < RI; ++i) {
          if (!KEEP && i % 4 == 0) asm volatile("" ::: "memory");
          double x0, x1;
          if (KEEP) { x0 = xr[i][0]; x1 = xr[i][1]; }
          else {
            const double2 t2 = *reinterpret_cast<const double2*>(x + CH * i);
            x0 = t2.x; x1 = t2.y;
          }
          cr[q][i][0] = fma(-ws, x0, cr[q][i][0]);
          cr[q][i][1] = fma(-ws, x1, cr[q][i][1]);
        }
        if (on && hl == (jj >> 1)) {
          const double w = fma(-ws, u, cj);
          if (jj & 1) cr[q][0][1] = w; else cr[q][0][0] = w;
        }
      }
#pragma unroll
      for (int q = 0; q < CPW; ++q)
        if (warp == (jj + 1) / CW && jj + 1 < jb && (CPW == 1 || c0 + q == jj + 1))
          publish(cr[q], jj + 1, CPW > 1 || c0 == jj + 1);
    }
  }
  __syncthreads();
  cluster_wait();                             // every CTA holds the panel: it may be overwritten
  double sc[CPW], bc[CPW];
#pragma unroll
  for (int q = 0; q < CPW; ++q) {
    const int c = c0 + q;
    const Reflector H(*reinterpret_cast<const double2*>(S.pub + 2 * min(c, jb - 1)));
    sc[q] = (c < jb) ? H.scale() : 0.0;
    bc[q] = H.beta() * down;
    if (hl == 0) { S.sv[c] = sc[q]; S.tau[c] = (c < jb) ? H.tau() : 0.0; }
  }
  __syncthreads();
  const int mp8 = (mp + 7) & ~7;
#pragma unroll
  for (int q = 0; q < CPW; ++q) {
    const int c = c0 + q;
    const bool own = c < jb, out = own && (c % csize == crank);
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const int r = CH * i + 2 * hl;
      double v[2], g[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        v[e] = cr[q][i][e] * sc[q];
        g[e] = v[e];
        if (i == 0 && r + e <= c) {           // on and above the diagonal: R in global memory, V in the panel
          g[e] = (r + e == c) ? bc[q] : cr[q][i][e] * down;
          v[e] = (r + e == c && own) ? 1.0 : 0.0;
        }
      }
      if (r < mp8) *reinterpret_cast<double2*>(S.P + panel_at(c, r, mp_ld)) = make_double2(v[0], v[1]);
      if (vec) store2<true>(g, A + (long long)c * lda, r, mp, out);
      else store2<false>(g, A + (long long)c * lda, r, mp, out);
    }
  }
  if (warp == 0) form_t<NW>(S, jb, (crank == 0) ? Tws : nullptr);   // its columns' registers are free by now
  __syncthreads();
  return hi >= 0x7ff00000;
}
}  // namespace

// T layout in shared memory: T[col * NB + row] (upper triangular).
template <int NW>
__global__ void __launch_bounds__(NW * 32, NW <= 8 ? 2 : 1)
    householder_qr_kernel(const QRDesc* __restrict__ descs, int csize, int* flags) {
  dep_wait();
  extern __shared__ __align__(16) double sm[];
  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)cluster.block_rank();
  const QRDesc D = descs[blockIdx.x / csize];
  if (D.m <= 0 || D.n <= 0) return;
  // the factored block (rows and columns beyond the device bounds are zero) and the shapes of
  // R (Kc x D.n) and Q (D.m x Kc)
  const int m = dev_bound(D.m, D.m_dev, D.m_mult), n = dev_bound(D.n, D.n_dev, D.n_mult);
  const int K = min(m, n), Kc = min(D.m, D.n);
  const PanelSm S = panel_sm<NW>(sm);
  const int tid = threadIdx.x;
  double* A = D.A;
  const int lda = D.lda;
  bool nonfinite = false;

  for (int j0 = 0; j0 < K; j0 += NB) {
    const int jb = min(NB, K - j0), mp = m - j0;
    double* Ap = A + (long long)j0 * lda + j0;
    double* Tws = D.Tws ? D.Tws + (j0 / NB) * NB * NB : nullptr;
    // registers per lane for the panel's own row count (uniform across the cluster)
    if constexpr (NW <= 8) {
      if (mp <= 64) nonfinite |= factor_panel<NW, 16, 2>(Ap, lda, mp, jb, crank, csize, Tws);
      else if (mp <= 128) nonfinite |= factor_panel<NW, 16, 4>(Ap, lda, mp, jb, crank, csize, Tws);
      else if (mp <= 256) nonfinite |= factor_panel<NW, 32, 4>(Ap, lda, mp, jb, crank, csize, Tws);
      else nonfinite |= factor_panel<NW, 32, 8>(Ap, lda, mp, jb, crank, csize, Tws);
    } else {
      if (mp <= 128) nonfinite |= factor_panel<NW, 32, 2>(Ap, lda, mp, jb, crank, csize, Tws);
      else if (mp <= 256) nonfinite |= factor_panel<NW, 32, 4>(Ap, lda, mp, jb, crank, csize, Tws);
      else if (mp <= 512) nonfinite |= factor_panel<NW, 32, 8>(Ap, lda, mp, jb, crank, csize, Tws);
      else if (mp <= 1024) nonfinite |= factor_panel<NW, 32, 16>(Ap, lda, mp, jb, crank, csize, Tws);
      else nonfinite |= factor_panel<NW, 32, 24>(Ap, lda, mp, jb, crank, csize, Tws);
    }
    // trailing update with H^T = I - V T^T V^T (this CTA's column octets)
    if (j0 + jb < n) apply_block<NW>(A, lda, j0, mp, j0 + jb, n, (int)(S.P - sm), true, crank, csize);
    __syncwarp();
    cluster_arrive();   // trailing columns and the panel visible to every CTA
    cluster_wait();
  }
  if (nonfinite && crank == 0) atomicOr(flags, DFLAG_NONFINITE);

  // R = upper triangle of A[0:Kc, 0:D.n] (zero outside the factored block)
  if (D.R) {
    for (int j = (tid >> 5) + NW * crank; j < D.n; j += NW * csize)
      for (int i = tid & 31; i < Kc; i += 32) {
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
  for (int c = tid >> 5; c < Kc; c += NW) {
    if (((c >> 3) % csize) != crank) continue;
    for (int i = tid & 31; i < D.m; i += 32) D.Q[(long long)c * D.ldq + i] = (i == c) ? 1.0 : 0.0;
  }
  const int qc_end = (n < D.n) ? Kc : K;
  const int npan = (K + NB - 1) / NB;
  for (int p = npan - 1; p >= 0; --p) {
    const int j0 = p * NB, jb = min(NB, K - j0), mp = m - j0, mp_ld = panel_ld(mp);
    __syncthreads();    // the identity columns, then the previous panel's products
    load_panel_v<NW>(S.P, mp_ld, A + (long long)j0 * lda + j0, lda, mp, jb);
    for (int e = tid; e < NB * NB; e += NW * 32) S.T[e] = D.Tws[p * NB * NB + e];
    __syncthreads();
    apply_block<NW>(D.Q, D.ldq, j0, mp, j0, qc_end, (int)(S.P - sm), false, crank, csize);
  }
}

// B <- Q B from the stored panels, backwards (as the Q formation, but from B instead of the
// identity and over all its columns).  CTA problem / csize owns the column octets o with
// o mod csize == CTA rank; the panels are only read, so no CTA waits for another.
template <int NW>
__global__ void __launch_bounds__(NW * 32, NW <= 8 ? 2 : 1)
    householder_apply_q_kernel(const QApplyDesc* __restrict__ descs, int csize) {
  dep_wait();
  extern __shared__ __align__(16) double sm[];
  const int crank = (int)(blockIdx.x % csize);
  const QApplyDesc D = descs[blockIdx.x / csize];
  const int m = dev_bound(D.m, D.m_dev, D.m_mult), K = min(D.K, m);   // H_k = I for k >= m
  if (m <= 0 || K <= 0 || D.nb <= 0) return;
  const int nb = D.n_dev ? min(D.nb, *D.n_dev) : D.nb;
  if (nb <= 0) return;
  double* T = sm;                                  // NB*NB, then the exchange buffer of apply_block
  double* P = T + NB * NB + kExchange<NW>;         // panel
  const int tid = threadIdx.x;
  const int npan = (K + NB - 1) / NB;
  for (int p = npan - 1; p >= 0; --p) {
    const int j0 = p * NB, jb = min(NB, K - j0), mp = m - j0, mp_ld = panel_ld(mp);
    __syncthreads();
    load_panel_v<NW>(P, mp_ld, D.A + (long long)j0 * D.lda + j0, D.lda, mp, jb);
    for (int e = tid; e < NB * NB; e += NW * 32) T[e] = D.Tws[p * NB * NB + e];
    __syncthreads();
    apply_block<NW>(D.B, D.ldb, j0, mp, 0, nb, (int)(P - sm), false, crank, csize);
  }
}

namespace {
// Rows up to which the eight-warp kernels (two CTAs per SM) hold a panel's registers and tiles.
constexpr int kSmallM = 512;

template <int NW>
size_t qr_smem(int max_m) {
  return sizeof(double) * (kFixed<NW> + (size_t)NB * panel_ld(std::max(max_m, 1)));
}
template <int NW>
size_t qr_apply_smem(int max_m) {
  return sizeof(double) * (NB * NB + kExchange<NW> + (size_t)NB * panel_ld(std::max(max_m, 1)));
}

template <int NW>
void launch_qr_apply_t(const QApplyDesc* d_descs, int count, int max_m, cudaStream_t s) {
  constexpr int lim = NW <= 8 ? kSmallM : QR_MAX_M;
  const size_t smem = qr_apply_smem<NW>(max_m);
  static PerDeviceOnce attr_once;
  int dev = 0;
  TTC_CUDA(cudaGetDevice(&dev));
  attr_once.run(dev, [] {
    TTC_CUDA(cudaFuncSetAttribute(householder_apply_q_kernel<NW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)std::max(qr_apply_smem<NW>(lim), kLoneCtaSmem)));
  });
  int per_sm = 1;
  TTC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, householder_apply_q_kernel<NW>, NW * 32, smem));
  const int csize = std::min(8, std::max(1, current_sm_count() * std::max(1, per_sm) / count));
  const size_t smem_l = count * csize <= current_sm_count() ? std::max(smem, kLoneCtaSmem) : smem;
  launch_dep(householder_apply_q_kernel<NW>, (unsigned)(count * csize), NW * 32, smem_l, s, d_descs, csize);
  TTC_CHECK_LAUNCH();
}

template <int NW>
void launch_qr_t(const QRDesc* d_descs, int count, int max_m, cudaStream_t s, int* d_flags, bool dependent) {
  constexpr int lim = NW <= 8 ? kSmallM : QR_MAX_M;
  const size_t smem = qr_smem<NW>(max_m);
  static PerDeviceOnce attr_once;
  int dev = 0;
  TTC_CUDA(cudaGetDevice(&dev));
  attr_once.run(dev, [] {
    TTC_CUDA(cudaFuncSetAttribute(householder_qr_kernel<NW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)std::max(qr_smem<NW>(lim), kLoneCtaSmem)));
  });
  // CTAs per problem: one wave of the resident-CTA slots of the two-per-SM kernel (a CTA's column steps
  // run beside its neighbour's products), two waves of the one-per-SM kernel (the planner puts the
  // largest problems first, so the second wave holds the short ones), at most 8 (portable cluster)
  int per_sm = 1;
  TTC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, householder_qr_kernel<NW>, NW * 32, smem));
  const int slots = current_sm_count() * std::max(2, per_sm);
  const int c = std::min(8, std::max(1, slots / count));
  int csize = 1;
  while (csize * 2 <= c) csize *= 2;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(count * csize));
  cfg.blockDim = dim3(NW * 32);
  // one CTA per SM while all clusters have room so
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
  cfg.numAttrs = dependent ? 2 : 1;
  TTC_CUDA(cudaLaunchKernelEx(&cfg, householder_qr_kernel<NW>, d_descs, csize, d_flags));
  TTC_CHECK_LAUNCH();
}
}  // namespace

void launch_qr_apply(const QApplyDesc* d_descs, int count, int max_m, cudaStream_t s) {
  if (count <= 0) return;
  TTC_REQUIRE(max_m <= QR_MAX_M, TTC_EDIM, "qr apply: row count exceeds the supported maximum (1536)");
  if (max_m <= kSmallM) launch_qr_apply_t<8>(d_descs, count, max_m, s);
  else launch_qr_apply_t<16>(d_descs, count, max_m, s);
}

void launch_qr(const QRDesc* d_descs, int count, int max_m, cudaStream_t s, int* d_flags, bool dependent) {
  if (count <= 0) return;
  TTC_REQUIRE(max_m <= QR_MAX_M, TTC_EDIM, "qr: row count exceeds the supported maximum (1536)");
  // Launches of few problems (every CTA has an SM to itself) and panels beyond 256 rows take sixteen
  // warps: one problem 512 x 256 with Q 446 us (454 with eight), 276 x 138 184 (183), 256 x 256 316 (293)
  const bool alone = max_m > 256 && 8LL * count <= current_sm_count();
  if (max_m <= kSmallM && !alone) launch_qr_t<8>(d_descs, count, max_m, s, d_flags, dependent);
  else launch_qr_t<16>(d_descs, count, max_m, s, d_flags, dependent);
}

}  // namespace ttc
