// Grouped, strided-batched FP32 GEMM (FP32 operands, FP32 accumulation, CUDA-core FMA) for the
// FP32 variant of the Rayleigh-quotient gradient: the same GemmDesc problems as the FP64 grouped
// GEMM (split row/column/K indices, batches, alpha/beta, the device column bound), with A, B
// and C holding float data, and the same scheme: CTA t finds its problem among the descriptors' tile
// prefix sums, 16 K steps at a time come through a ring of asynchronous copies, which take any strides,
// and the split K index advances without a division.  Every element adds its K steps in order with one FMA
// each (no K splits), so the result does not depend on the tile.
//
// What bounds it: the FMA pipes (128 per cycle and SM) and the issue of the copies and fragment loads, which
// the two-column FMA and the 8 x 4 part per thread keep to 11 loads and copies per 16 FMAs; at few tiles, the
// latency of a K step.  A gradient at d 32, r 192, R 18 (51 GF; 98 launches): 64 x 64 tiles of 256 threads with
// one tile prefetched in registers 6.1 ms; this kernel 3.5 at 64 x 64, 4.0 at 64 x 32, 4.6 at 32 x 32;
// 128 x 64 tiles 3.9 (8 x 8 or 8 x 4 per thread), 64 x 64 with 4 x 4 per thread 3.9, with three stages and four
// CTAs per SM 3.6.
#include "common.cuh"
#include "gemm_grouped.cuh"
#include "kernels.cuh"

namespace ttc {

namespace {
constexpr int BK = 16;
struct TileShape { int bm, bn; };
constexpr TileShape kTiles[kGemm32Tiles] = {{64, 64}, {64, 32}, {32, 32}};

// 4 bytes global -> shared; zero when !on (the address is not read)
__device__ __forceinline__ void cp4(unsigned dst, const float* src, bool on) {
  const int sz = on ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(sz) : "memory");
}

// d = a b + d in both halves, each rounded as fmaf rounds
__device__ __forceinline__ void fma2(float2& d, float2 a, float2 b) {
  unsigned long long& dd = reinterpret_cast<unsigned long long&>(d);
  asm("fma.rn.f32x2 %0, %1, %2, %0;\n"
      : "+l"(dd)
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
}

// Shared memory: STAGES x (As[BK][BM + 4], Bs[BK][BN + 4]), then the C tile [BN][BM + 1] over it.
template <int BM, int BN>
constexpr int kStageFloats = BK * (BM + 4 + BN + 4);
template <int BM, int BN, int STAGES>
constexpr size_t kSmem32 = sizeof(float) * (STAGES * kStageFloats<BM, BN> > BN * (BM + 1) ? STAGES * kStageFloats<BM, BN>
                                                                                          : BN * (BM + 1));
}  // namespace

// Each thread a TM x TN part of the tile in blocks of 4 rows BM / (TM / 4) apart (columns alike); a warp covers
// 4 x 8 threads.
template <int BM, int BN, int TM, int TN, int STAGES, int MINB>
__global__ void __launch_bounds__(BM / TM * (BN / TN), MINB) gemm_f32_grouped_kernel(const GemmDesc* __restrict__ descs, int nd) {
  dep_wait();
  constexpr int NT = BM / TM * (BN / TN), PA = BM + 4, PB = BN + 4;
  constexpr int LA = BM * BK / NT, LB = BN * BK / NT, KQ = NT / BK;
  constexpr int GM = BM / TM, GN = BN / TN;                  // threads along rows and columns
  constexpr int WN = GN / 8;                                 // warps along the columns
  static_assert(GM % 4 == 0 && GN % 8 == 0 && TM % 4 == 0 && TN % 4 == 0 && NT % BM == 0 && NT % BN == 0, "tile");
  extern __shared__ __align__(16) float smem32[];
  const int tid = threadIdx.x;
  const long long tile = blockIdx.x;
  const GemmDesc D = descs[find_desc(descs, nd, tile)];
  const int tm = ceil_div(D.m, BM), tn = ceil_div(D.n, BN);
  const int per = tm * tn;
  const long long local = tile - D.tile_start;
  if (per == 0 || local < 0 || local >= (long long)per * D.batch) return;
  const int b = (int)(local / per);
  const int rem = (int)(local - (long long)b * per);
  const int row0 = (rem % tm) * BM, col0 = (rem / tm) * BN;
  const bool m_one = D.m0 >= D.m, n_one = D.n0 >= D.n;
  float* __restrict__ C = reinterpret_cast<float*>(D.C) + (long long)b * D.c_b;
  if (D.n_dev && col0 >= *D.n_dev) {          // every column of this tile is known to be zero
    if (D.beta != 0.0) return;
    for (int e = tid; e < BM * BN; e += NT) {
      const int gi = row0 + e % BM, gj = col0 + e / BM;
      if (gi < D.m && gj < D.n) C[split_off(gi, D.m0, m_one, D.c_i0, D.c_i1) + split_off(gj, D.n0, n_one, D.c_j0, D.c_j1)] = 0.f;
    }
    return;
  }
  const float* __restrict__ A = reinterpret_cast<const float*>(D.A) + (long long)b * D.a_b;
  const float* __restrict__ Bm = reinterpret_cast<const float*>(D.B) + (long long)b * D.b_b;

  // Loader mappings as in the FP64 kernel: contiguous along the unit-stride index when there is one.
  const bool a_rowfast = (D.a_i0 == 1), b_colfast = (D.b_j0 == 1);
  const int a_k = a_rowfast ? (tid / KQ) : (tid & 15);
  const int b_k = b_colfast ? (tid / KQ) : (tid & 15);
  const int ar0 = a_rowfast ? (tid % KQ) : (tid >> 4), bc0 = b_colfast ? (tid % KQ) : (tid >> 4);
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
  const int k0e = D.k0e, kdim = D.k;
  const long long a_wrap = D.a_k1 - (long long)k0e * D.a_k0, b_wrap = D.b_k1 - (long long)k0e * D.b_k0;
  const long long a_step = BK * D.a_k0, b_step = BK * D.b_k0;
  int a_kr = a_k % k0e, b_kr = b_k % k0e;
  long long a_ko = (long long)a_kr * D.a_k0 + (long long)(a_k / k0e) * D.a_k1;
  long long b_ko = (long long)b_kr * D.b_k0 + (long long)(b_k / k0e) * D.b_k1;
  const unsigned sbase = (unsigned)__cvta_generic_to_shared(smem32);
  const unsigned sa0 = sbase + 4u * (unsigned)(a_k * PA + ar0), sb0 = sbase + 4u * (unsigned)(BK * PA + b_k * PB + bc0);
  const int nk = ceil_div(kdim, BK);
  // Issues the copies of K step kt and advances the running coordinates.  A copy that is off has an
  // address inside the operand all the same.
  auto load_stage = [&](int kt) {
    if (kt < nk) {
      const int k0 = kt * BK;
      const bool ka = k0 + a_k < kdim, kb = k0 + b_k < kdim;
      const unsigned so = 4u * (unsigned)((kt % STAGES) * kStageFloats<BM, BN>);
      const unsigned oka = ka ? a_ok : 0u, okb = kb ? b_ok : 0u;
      const float* Ak = A + (ka ? a_ko : 0);
      const float* Bk = Bm + (kb ? b_ko : 0);
#pragma unroll
      for (int t = 0; t < LA; ++t) cp4(sa0 + so + 4u * KQ * t, Ak + a_roff[t], (oka >> t) & 1u);
#pragma unroll
      for (int t = 0; t < LB; ++t) cp4(sb0 + so + 4u * KQ * t, Bk + b_coff[t], (okb >> t) & 1u);
      a_kr += BK; a_ko += a_step;
      while (a_kr >= k0e) { a_kr -= k0e; a_ko += a_wrap; }
      b_kr += BK; b_ko += b_step;
      while (b_kr >= k0e) { b_kr -= k0e; b_ko += b_wrap; }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  const int warp = tid >> 5, lane = tid & 31;
  const int ty = warp / WN * 4 + (lane >> 3), tx = warp % WN * 8 + (lane & 7);
  float2 acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 1
  for (int p = 0; p < STAGES - 1; ++p) load_stage(p);
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                                       // stage kt is there, stage kt - 1 is read
    load_stage(kt + STAGES - 1);
    const float* As = smem32 + (kt % STAGES) * kStageFloats<BM, BN>;
    const float* Bs = As + BK * PA;
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM];
      float2 bv[TN / 2];
#pragma unroll
      for (int i = 0; i < TM; i += 4)
        *reinterpret_cast<float4*>(&a[i]) = *reinterpret_cast<const float4*>(&As[kk * PA + i / 4 * (4 * GM) + ty * 4]);
#pragma unroll
      for (int j = 0; j < TN; j += 4)
        *reinterpret_cast<float4*>(&bv[j / 2]) = *reinterpret_cast<const float4*>(&Bs[kk * PB + j / 4 * (4 * GN) + tx * 4]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], make_float2(a[i], a[i]), bv[j]);
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  // stage the C tile (column-major), then store along C's unit stride
  constexpr int PC = BM + 1;
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j)
      smem32[(j / 4 * (4 * GN) + tx * 4 + j % 4) * PC + i / 4 * (4 * GM) + ty * 4 + i % 4] = j % 2 ? acc[i][j / 2].y : acc[i][j / 2].x;
  __syncthreads();
  const float alpha = (float)D.alpha, beta = (float)D.beta;
  auto put = [&](long long off, int li, int lj) {
    const float v = alpha * smem32[lj * PC + li];
    C[off] = (beta == 0.f) ? v : fmaf(beta, C[off], v);
  };
  if (D.c_j0 == 1 && D.c_i0 != 1) {
    const int lj = tid % BN, gj = col0 + lj;
    if (gj >= D.n) return;
    const long long oj = split_off(gj, D.n0, n_one, D.c_j0, D.c_j1);
    for (int li = tid / BN; li < BM && row0 + li < D.m; li += NT / BN)
      put(oj + split_off(row0 + li, D.m0, m_one, D.c_i0, D.c_i1), li, lj);
  } else {
    const int li = tid % BM, gi = row0 + li;
    if (gi >= D.m) return;
    const long long oi = split_off(gi, D.m0, m_one, D.c_i0, D.c_i1);
    for (int lj = tid / BM; lj < BN && col0 + lj < D.n; lj += NT / BM)
      put(oi + split_off(col0 + lj, D.n0, n_one, D.c_j0, D.c_j1), li, lj);
  }
}

namespace {
template <int BM, int BN, int TM, int TN, int STAGES, int MINB>
void launch_t(const GemmDesc* d_descs, int nd, long long total_tiles, cudaStream_t s) {
  static PerDeviceOnce attr_once;
  int dev = 0;
  TTC_CUDA(cudaGetDevice(&dev));
  attr_once.run(dev, [] {
    TTC_CUDA(cudaFuncSetAttribute(gemm_f32_grouped_kernel<BM, BN, TM, TN, STAGES, MINB>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem32<BM, BN, STAGES>));
  });
  launch_dep(gemm_f32_grouped_kernel<BM, BN, TM, TN, STAGES, MINB>, (unsigned)total_tiles, BM / TM * (BN / TN),
             kSmem32<BM, BN, STAGES>, s, d_descs, nd);
  TTC_CHECK_LAUNCH();
}
}  // namespace

void launch_gemm_f32(const GemmDesc* d_descs, int nd, long long total_tiles, int tile, cudaStream_t s) {
  if (nd <= 0 || total_tiles <= 0) return;
  TTC_REQUIRE(total_tiles < (1LL << 31), TTC_EINTERNAL, "gemm: too many tiles in one launch");
  switch (tile) {
    case 0: launch_t<64, 64, 8, 4, 4, 3>(d_descs, nd, total_tiles, s); break;
    case 1: launch_t<64, 32, 4, 4, 4, 4>(d_descs, nd, total_tiles, s); break;
    default: launch_t<32, 32, 4, 4, 4, 6>(d_descs, nd, total_tiles, s); break;
  }
}

long long gemm32_tiles(const GemmDesc& d, int tile) {
  if (d.m <= 0 || d.n <= 0 || d.batch <= 0) return 0;
  return (long long)ceil_div(d.m, kTiles[tile].bm) * ceil_div(d.n, kTiles[tile].bn) * d.batch;
}

int gemm32_pick_tile(const GemmDesc* d, int nd, int nsm) {
  // The shape with the least time at one tile per SM and turn.  The costs are times per output element and
  // turn, measured in the gradient's last launch (8.8 GF, K to 3456): 333 tiles of 64 x 64 0.33 ms, 657 of
  // 64 x 32 0.40, 1299 of 32 x 32 0.46.
  constexpr double cost[kGemm32Tiles] = {1.0, 1.45, 1.86};
  int best = 0;
  double best_t = 0.0;
  for (int t = 0; t < kGemm32Tiles; ++t) {
    long long tiles = 0;
    for (int i = 0; i < nd; ++i) tiles += gemm32_tiles(d[i], t);
    const double turns = (double)((tiles + nsm - 1) / nsm) * kTiles[t].bm * kTiles[t].bn * cost[t];
    if (t == 0 || turns < best_t) { best = t; best_t = turns; }
  }
  return best;
}

}  // namespace ttc
