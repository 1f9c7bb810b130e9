// Grouped, strided-batched FP64 GEMM for the FP64 contractions of the rounding sweeps
// (FR*core, absorb U*S, Z = y_k W, Q^T y_k, environment updates).  One launch runs a
// list of GemmDesc problems; CTA t finds its problem by binary search over the
// descriptors' tile prefix sums, so ranks that differ per TT and per site share one
// launch.  The products run on the FP64 tensor cores (mma.sync m8n8k4); the operand tiles (16 K
// steps at a time) come through a four-stage ring of 8-byte asynchronous copies, which take any strides.
// The split K index (k0 + k0e k1) of every loaded element advances incrementally, with no
// division in the K loop.  Launches of few output tiles and long K (the range finder and
// projections of the operator rounding, K = r R) split K over several CTAs per tile.
//
// What bounds it: the tensor cores' 64 FMA per cycle and SM, that is 1024 cycles for 16 K steps of a
// 64 x 64 tile, so that a launch of a few such tiles leaves most SMs idle for K / 16 of these.  The tile
// is therefore chosen for a whole launch (gemm_pick_tile) among 64 x 64, 64 x 32, 32 x 32 and
// 16 x 16.
// Every output element adds its K steps in the same order whatever the tile, and the K splits are a
// function of the shapes alone, so the choice does not change a bit of the result.
//
// Four warps per tile (at 64 x 64 each 32 x 32: 16 products for 8 fragment loads), three CTAs per SM, the
// fragments of the next 4 K steps loaded ahead of the products, the copies of a later stage issued before
// them.  Eight warps of 32 x 16 with two CTAs per SM, loads at their use: 24.7 TFLOP/s at 4096 x 4096 x 1024
// where this runs 28.0 (the DMMA rate is 37); copies issued between the products instead: 27.4, and 23.8 ->
// 22.5 at 1280 x 1280 x 2048; 128 x 64 tiles: 28.0, but 17.6 at 1280 x 1280 x 2048.
// Measured here against one 64 x 64 tile shape: 4096 x 4096 x 1024 24.4 -> 28.0, 1280 x 1280 x 2048
// 18.5 -> 23.8, 640 x 1920 x 1024 14.7 -> 19.5 TFLOP/s; 256 x 256 x 320 30 -> 20 us.
#include <algorithm>

#include "common.cuh"
#include "gemm_grouped.cuh"
#include "kernels.cuh"

namespace ttc {

namespace {
constexpr int BK = 16;
// the tile that the K splits are counted in
constexpr int REF_BM = 64, REF_BN = 64;

// bm x bn, the CTAs that an SM holds, and what a turn of n CTAs on an SM costs: once + n each (gemm_pick_tile)
struct TileShape { int bm, bn, per_sm; double once, each; };
constexpr TileShape kTiles[kGemmTiles] = {{64, 64, 3, 0.52, 1.0}, {64, 32, 3, 0.29, 0.55}, {32, 32, 6, 0.30, 0.35},
                                          {16, 16, 8, 0.092, 0.18}};

// 8 bytes global -> shared; zero when !on (the address is not read)
__device__ __forceinline__ void cp8(unsigned dst, const double* src, bool on) {
  const int sz = on ? 8 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(sz) : "memory");
}

// Shared memory: STAGES x (As[BK][BM + 4], Bs[BK][BN + 4]); a pad of 4 mod 16 doubles, so that the
// fragment loads (4 k x 4 rows per half warp) hit distinct banks.
template <int BM, int BN>
constexpr int kStageDoubles = BK * (BM + 4 + BN + 4);
template <int BM, int BN, int STAGES>
constexpr size_t kGemmSmem = sizeof(double) * STAGES * kStageDoubles<BM, BN>;
}  // namespace

// WM x WN warps, each a (BM / WM) x (BN / WN) part of the tile in 8 x 8 fragments.
template <int BM, int BN, int WM, int WN, int STAGES, int MINB>
__global__ void __launch_bounds__(WM * WN * 32, MINB) gemm_f64_grouped_kernel(const GemmDesc* __restrict__ descs, int nd) {
  dep_wait();
  constexpr int NT = WM * WN * 32, PA = BM + 4, PB = BN + 4;
  constexpr int FM = BM / WM / 8, FN = BN / WN / 8;
  constexpr int LA = BM * BK / NT, LB = BN * BK / NT;      // elements of A and B a thread loads per stage
  constexpr int KQ = NT / 16;                              // rows (columns) that one pass of the threads covers
  extern __shared__ __align__(16) double smem[];
  __shared__ int s_last;

  const int tid = threadIdx.x;
  const long long tile = blockIdx.x;
  const int di = find_desc(descs, nd, tile);
  const GemmDesc D = descs[di];
  const int tm = ceil_div(D.m, BM), tn = ceil_div(D.n, BN);
  const long long local = tile - D.tile_start;
  const int per = tm * tn;
  const int ks = D.ksplit > 1 ? D.ksplit : 1;
  const long long tiles_out = (long long)per * D.batch;          // output tiles of this problem
  if (per == 0 || local >= tiles_out * ks) return;
  const int split = (int)(local / tiles_out);
  const long long lt = local - (long long)split * tiles_out;     // output tile
  const int b = (int)(lt / per);
  const int rem = (int)(lt - (long long)b * per);
  const int bm = rem % tm, bn = rem / tm;
  const int row0 = bm * BM, col0 = bn * BN;
  if (D.n_dev && col0 >= *D.n_dev) {          // every column of this tile is known to be zero
    if (D.beta != 0.0 || split != 0) return;  // (the same decision in every split: no counting)
    double* __restrict__ Cz = D.C + (long long)b * D.c_b;
    for (int e = threadIdx.x; e < BM * BN; e += NT) {
      const int li = e % BM, lj = e / BM;
      const int gi = row0 + li, gj = col0 + lj;
      if (gi < D.m && gj < D.n)
        Cz[(long long)(gi % D.m0) * D.c_i0 + (long long)(gi / D.m0) * D.c_i1 + (long long)(gj % D.n0) * D.c_j0 +
           (long long)(gj / D.n0) * D.c_j1] = 0.0;
    }
    return;
  }

  const double* __restrict__ A = D.A + (long long)b * D.a_b;
  const double* __restrict__ B = D.B + (long long)b * D.b_b;

  // Loader mappings: contiguous along the unit-stride index when there is one.  A thread copies its
  // elements at one K index, rows (columns) NT / 16 apart.
  const bool a_rowfast = (D.a_i0 == 1);          // consecutive rows contiguous
  const bool b_colfast = (D.b_j0 == 1);          // consecutive cols contiguous
  const int k0e = D.k0e, kdim = D.k;
  const int a_k = a_rowfast ? (tid / KQ) : (tid & 15);
  const int b_k = b_colfast ? (tid / KQ) : (tid & 15);
  const int ar0 = a_rowfast ? (tid % KQ) : (tid >> 4), bc0 = b_colfast ? (tid % KQ) : (tid >> 4);
  const bool m_one = D.m0 >= D.m, n_one = D.n0 >= D.n;    // most dimensions are not split: no divisions
  unsigned a_ok = 0, b_ok = 0;
  long long a_roff[LA], b_coff[LB];
#pragma unroll
  for (int t = 0; t < LA; ++t) {
    const int gi = row0 + ar0 + KQ * t;
    a_ok |= (gi < D.m ? 1u : 0u) << t;
    a_roff[t] = (gi < D.m) ? split_off(gi, D.m0, m_one, D.a_i0, D.a_i1) : 0;
  }
#pragma unroll
  for (int t = 0; t < LB; ++t) {
    const int gj = col0 + bc0 + KQ * t;
    b_ok |= (gj < D.n ? 1u : 0u) << t;
    b_coff[t] = (gj < D.n) ? split_off(gj, D.n0, n_one, D.b_j0, D.b_j1) : 0;
  }
  // this CTA's K range, in BK-wide steps
  const int nk_all = ceil_div(kdim, BK);
  const int chunk = ceil_div(nk_all, ks);
  const int kt_beg = min(nk_all, split * chunk), kt_end = min(nk_all, kt_beg + chunk);
  // running split K coordinate of this thread's A and B elements: kr = gk mod k0e and the
  // element offset kr k_0 + (gk / k0e) k_1, advanced by BK per step without a division
  const long long a_wrap = D.a_k1 - (long long)k0e * D.a_k0, b_wrap = D.b_k1 - (long long)k0e * D.b_k0;
  const long long a_step = BK * D.a_k0, b_step = BK * D.b_k0;
  int a_kr, b_kr;
  long long a_ko, b_ko;
  {
    const int ga = kt_beg * BK + a_k, gb = kt_beg * BK + b_k;
    a_kr = ga % k0e; a_ko = (long long)a_kr * D.a_k0 + (long long)(ga / k0e) * D.a_k1;
    b_kr = gb % k0e; b_ko = (long long)b_kr * D.b_k0 + (long long)(gb / k0e) * D.b_k1;
  }
  const unsigned sbase = (unsigned)__cvta_generic_to_shared(smem);
  const unsigned sa0 = sbase + 8u * (unsigned)(a_k * PA + ar0), sb0 = sbase + 8u * (unsigned)(BK * PA + b_k * PB + bc0);
  // Issues the copies of K step kt and advances the running coordinates.  A copy that is off has an
  // address inside the operand all the same.
  auto load_stage = [&](int kt) {
    if (kt < kt_end) {
      const int k0 = kt * BK;
      const bool ka = k0 + a_k < kdim, kb = k0 + b_k < kdim;
      const unsigned so = 8u * (unsigned)(((kt - kt_beg) % STAGES) * kStageDoubles<BM, BN>);
      const unsigned oka = ka ? a_ok : 0u, okb = kb ? b_ok : 0u;
      const double* Ak = A + (ka ? a_ko : 0);
      const double* Bk = B + (kb ? b_ko : 0);
#pragma unroll
      for (int t = 0; t < LA; ++t) cp8(sa0 + so + 8u * KQ * t, Ak + a_roff[t], (oka >> t) & 1u);
#pragma unroll
      for (int t = 0; t < LB; ++t) cp8(sb0 + so + 8u * KQ * t, Bk + b_coff[t], (okb >> t) & 1u);
      a_kr += BK; a_ko += a_step;
      while (a_kr >= k0e) { a_kr -= k0e; a_ko += a_wrap; }
      b_kr += BK; b_ko += b_step;
      while (b_kr >= k0e) { b_kr -= k0e; b_ko += b_wrap; }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  // Fragment coordinates: A[qr][qc] = As[k + qc][i + qr], B[qc][qr] = Bs[k + qc][j + qr], D[qr][2qc + {0,1}].
  const int warp = tid >> 5, lane = tid & 31, qr = lane >> 2, qc = lane & 3;
  const int wr = (warp % WM) * (BM / WM), wc = (warp / WM) * (BN / WN);
  const bool busy = row0 + wr < D.m && col0 + wc < D.n;    // this warp's part holds an output
  double acc[FM][FN][2];
#pragma unroll
  for (int i = 0; i < FM; ++i)
#pragma unroll
    for (int j = 0; j < FN; ++j) { acc[i][j][0] = 0.0; acc[i][j][1] = 0.0; }

#pragma unroll 1
  for (int p = 0; p < STAGES - 1; ++p) load_stage(kt_beg + p);
  for (int kt = kt_beg; kt < kt_end; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                                       // stage kt is there, stage kt - 1 is read
    load_stage(kt + STAGES - 1);
    if (busy) {
      const double* As = smem + ((kt - kt_beg) % STAGES) * kStageDoubles<BM, BN>;
      const double* Bs = As + BK * PA;
      // the fragments of one K group ahead of the products
      double a[2][FM], bv[2][FN];
      auto frags = [&](int kk, int h) {
#pragma unroll
        for (int i = 0; i < FM; ++i) a[h][i] = As[(kk + qc) * PA + wr + 8 * i + qr];
#pragma unroll
        for (int j = 0; j < FN; ++j) bv[h][j] = Bs[(kk + qc) * PB + wc + 8 * j + qr];
      };
      frags(0, 0);
#pragma unroll
      for (int kk = 0; kk < BK; kk += 4) {
        const int h = (kk >> 2) & 1;
        if (kk + 4 < BK) frags(kk + 4, h ^ 1);
#pragma unroll
        for (int i = 0; i < FM; ++i)
#pragma unroll
          for (int j = 0; j < FN; ++j) dmma(acc[i][j][0], acc[i][j][1], a[h][i], bv[h][j]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");

  if (ks > 1) {
    // this split's partial tile into its slot, then the last CTA of the tile to arrive sums
    // the ks slots in split order
    double* slots = D.ws + lt * ks * (long long)(BM * BN) + tid;
    double* mine = slots + (long long)split * (BM * BN);
#pragma unroll
    for (int i = 0; i < FM; ++i)
#pragma unroll
      for (int j = 0; j < FN; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) mine[((i * FN + j) * 2 + e) * NT] = acc[i][j][e];
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = (atomicAdd(D.cnt + lt, 1u) == (unsigned)(ks - 1));
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // a row of fragments at a time, the loads of several splits in flight (its own partial is read back as well)
#pragma unroll
    for (int i = 0; i < FM; ++i) {
      double v[FN][2] = {};
#pragma unroll 4
      for (int s2 = 0; s2 < ks; ++s2) {
        const double* from = slots + (long long)s2 * (BM * BN) + i * FN * 2 * NT;
#pragma unroll
        for (int j = 0; j < FN; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) v[j][e] += __ldcg(from + (j * 2 + e) * NT);
      }
#pragma unroll
      for (int j = 0; j < FN; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) acc[i][j][e] = v[j][e];
    }
    if (tid == 0) D.cnt[lt] = 0u;   // zero again for the next launch of the plan
  }
  if (!busy) return;
  // Each fragment row is 8 consecutive rows (or 8 consecutive columns) of C: 64-byte runs along a unit
  // stride, written from the registers.
  const double alpha = D.alpha, beta = D.beta;
  double* __restrict__ C = D.C + (long long)b * D.c_b;
  long long coff[FN][2];
#pragma unroll
  for (int j = 0; j < FN; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int gj = col0 + wc + 8 * j + 2 * qc + e;
      coff[j][e] = (gj < D.n) ? split_off(gj, D.n0, n_one, D.c_j0, D.c_j1) : -1;
    }
#pragma unroll
  for (int i = 0; i < FM; ++i) {
    const int gi = row0 + wr + 8 * i + qr;
    if (gi >= D.m) continue;
    double* Cr = C + split_off(gi, D.m0, m_one, D.c_i0, D.c_i1);
#pragma unroll
    for (int j = 0; j < FN; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (coff[j][e] >= 0) {
          double* p = Cr + coff[j][e];
          const double v = alpha * acc[i][j][e];
          *p = (beta == 0.0) ? v : fma(beta, *p, v);
        }
  }
}

namespace {
template <int BM, int BN, int WM, int WN, int STAGES, int MINB>
void launch_t(const GemmDesc* d_descs, int nd, long long total_tiles, cudaStream_t s) {
  static PerDeviceOnce attr_once;
  int dev = 0;
  TTC_CUDA(cudaGetDevice(&dev));
  attr_once.run(dev, [] {
    TTC_CUDA(cudaFuncSetAttribute(gemm_f64_grouped_kernel<BM, BN, WM, WN, STAGES, MINB>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem<BM, BN, STAGES>));
  });
  launch_dep(gemm_f64_grouped_kernel<BM, BN, WM, WN, STAGES, MINB>, (unsigned)total_tiles, WM * WN * 32,
             kGemmSmem<BM, BN, STAGES>, s, d_descs, nd);
  TTC_CHECK_LAUNCH();
}
}  // namespace

// Host launcher: descs already resident on the device (tile_start filled for the tile shape).
void launch_gemm_f64(const GemmDesc* d_descs, int nd, long long total_tiles, int tile, cudaStream_t s) {
  if (nd <= 0 || total_tiles <= 0) return;
  TTC_REQUIRE(total_tiles < (1LL << 31), TTC_EINTERNAL, "gemm: too many tiles in one launch");
  switch (tile) {
    case 0: launch_t<64, 64, 2, 2, 4, 3>(d_descs, nd, total_tiles, s); break;
    case 1: launch_t<64, 32, 2, 2, 5, 3>(d_descs, nd, total_tiles, s); break;
    case 2: launch_t<32, 32, 2, 2, 4, 6>(d_descs, nd, total_tiles, s); break;
    default: launch_t<16, 16, 2, 2, 4, 8>(d_descs, nd, total_tiles, s); break;
  }
}

long long gemm_tiles(const GemmDesc& d, int tile) {
  if (d.m <= 0 || d.n <= 0 || d.batch <= 0) return 0;
  return (long long)ceil_div(d.m, kTiles[tile].bm) * ceil_div(d.n, kTiles[tile].bn) * d.batch *
         (d.ksplit > 1 ? d.ksplit : 1);
}

int gemm_pick_ksplit(const GemmDesc& d, long long launch_tiles, int nsm) {
  // enough CTAs for two per SM over the whole launch, each split at least 32 K steps deep
  const long long want = 2LL * nsm;
  if (launch_tiles <= 0 || launch_tiles >= want) return 1;
  const int nk = ceil_div(d.k, BK);
  const long long by_fill = (want + launch_tiles - 1) / launch_tiles;
  const long long by_depth = nk / 32;
  return (int)std::max(1LL, std::min({by_fill, by_depth, 16LL}));
}

long long gemm_split_ws_doubles(const GemmDesc& d, int tile) {
  if (d.ksplit <= 1) return 0;
  return gemm_tiles(d, tile) * (kTiles[tile].bm * kTiles[tile].bn);
}

int gemm_pick_tile(const GemmDesc* d, int nd, int nsm) {
  // The shape with the least time, for as many turns as the SMs' CTAs need.  A turn's time per K step grows with
  // the CTAs on an SM, but from a part that one CTA alone pays as well (four warps do not fill an SM's tensor
  // cores): fitted to 160 launches, 1 to 840 tiles of 64 x 64, K 64 to 10240, all four layouts, each shape timed.
  // The choice is 1.2 % above the best shape on average and nowhere above the time of 64 x 64 tiles of eight
  // warps; counting turns of one tile per SM by area alone was 3.8 % above it, 20 to 37 % for 112 to 148 tiles
  // (700^3 55 -> 45 us, transposed 66 -> 48; eight 1000 x 60 x 1000 88 -> 71).
  int best = 0;
  double best_t = 0.0;
  for (int t = 0; t < kGemmTiles; ++t) {
    const TileShape& T = kTiles[t];
    long long tiles = 0;
    for (int i = 0; i < nd; ++i) tiles += gemm_tiles(d[i], t);
    const long long per = (tiles + nsm - 1) / nsm, rest = per % T.per_sm;
    const double time = (double)(per / T.per_sm) * (T.once + T.per_sm * T.each) + (rest ? T.once + (double)rest * T.each : 0.0);
    if (t == 0 || time < best_t) { best = t; best_t = time; }
  }
  return best;
}

}  // namespace ttc
