// Simple tiled GEMM over general strides, templated on the element type.
//
// The FP64 DGEMM (the FP64 oracle and the double variants of the benchmarks).
//   op(X)[r][k] = X[r * s_r + k * s_k]
//   C[m][n] = alpha * (sum_k op(A)[m][k] op(B)[k][n]  [+ op(A2) op(B2)]) + beta * C[m][n]
// 16 x 16 of C per group of 64 threads, BK = 16; persistent CTAs of eight such
// groups, one CTA per SM, walk the tiles.  beta == 0 does not read C.  `lower`
// (symmetric products, M == N): only tiles on or below the diagonal are
// computed; a tile below it also stores its transpose.
//
// Bound: the FP64 pipe, two FMA per cycle and SM (1.26 TFLOP/s), so slow that
// a small tile's extra loads cost nothing, while how evenly the tiles fall on
// the SMs decides: N = 1024 took 2.06 ms with 256 CTAs of 64 x 64, 1.81 with
// 4096 CTAs of 16 x 16, which the hardware spreads unevenly, and takes 1.76 ms
// (floor 1.71) with tile t on SM t mod 152; 573 x 417 x 398 411, 311 and 182 us.
#pragma once
#include "gbpoly_internal.cuh"

namespace gbpoly {

template <typename T>
struct TiledOperand {
  const T* p;
  int64_t s_r, s_k;
};

constexpr int kTiledTile = 16;
constexpr int kTiledGroups = 8;  // groups of 64 threads per CTA

template <typename T>
__global__ void __launch_bounds__(64 * kTiledGroups, 1) tiled_gemm_kernel(int64_t M, int64_t N, int64_t K, T alpha,
    TiledOperand<T> a, TiledOperand<T> b, bool dual, TiledOperand<T> a2, TiledOperand<T> b2, T beta, T* __restrict__ C,
    int64_t ldc, bool lower, int64_t tiles_n, int64_t tiles) {
  constexpr int TILE = kTiledTile, R = TILE / 8, BK = 16;  // R x R outputs per thread (8 x 8 threads)
  __shared__ T As_all[kTiledGroups][BK][TILE + 1];
  __shared__ T Bs_all[kTiledGroups][BK][TILE + 1];
  pdl_enter();
  const int group = threadIdx.x >> 6, tid = threadIdx.x & 63;
  T(&As)[BK][TILE + 1] = As_all[group];
  T(&Bs)[BK][TILE + 1] = Bs_all[group];
  auto sync_group = [&] { asm volatile("bar.sync %0, 64;" ::"r"(group + 1) : "memory"); };
  const int tx = tid & 7, ty = tid >> 3;
  // group 0 of every CTA first, then group 1, ...: the tiles of a round fall evenly on the SMs
  for(int64_t t = blockIdx.x + int64_t(group) * gridDim.x; t < tiles; t += int64_t(kTiledGroups) * gridDim.x) {
    int64_t tm = t / tiles_n, tn = t - tm * tiles_n;
    if(lower) {  // row-major walk of the lower triangle: t = tm (tm + 1) / 2 + tn
      tm = int64_t((sqrtf(8.f * float(t) + 1.f) - 1.f) * 0.5f);
      while(tm * (tm + 1) / 2 > t) --tm;
      while((tm + 1) * (tm + 2) / 2 <= t) ++tm;
      tn = t - tm * (tm + 1) / 2;
    }
    const int64_t m0 = tm * TILE, n0 = tn * TILE;
    T acc[R][R];
#pragma unroll
    for(int i = 0; i < R; ++i)
#pragma unroll
      for(int j = 0; j < R; ++j) acc[i][j] = T(0);
    const int passes = dual ? 2 : 1;
    for(int p = 0; p < passes; ++p) {
      const TiledOperand<T> oa = p ? a2 : a;
      const TiledOperand<T> ob = p ? b2 : b;
      for(int64_t k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for(int e = 0; e < TILE * BK / 64; ++e) {
          const int idx = tid + e * 64;
          // rows fastest when the operand is contiguous along rows, else k fastest
          const int r = (oa.s_r == 1) ? (idx % TILE) : (idx / BK);
          const int kk = (oa.s_r == 1) ? (idx / TILE) : (idx % BK);
          const int64_t gm = m0 + r, gk = k0 + kk;
          As[kk][r] = (gm < M && gk < K) ? oa.p[gm * oa.s_r + gk * oa.s_k] : T(0);
          const int rb = (ob.s_r == 1) ? (idx % TILE) : (idx / BK);
          const int kb = (ob.s_r == 1) ? (idx / TILE) : (idx % BK);
          const int64_t gn = n0 + rb, gkb = k0 + kb;
          Bs[kb][rb] = (gn < N && gkb < K) ? ob.p[gn * ob.s_r + gkb * ob.s_k] : T(0);
        }
        sync_group();
#pragma unroll
        for(int kk = 0; kk < BK; ++kk)
#pragma unroll
          for(int i = 0; i < R; ++i)
#pragma unroll
            for(int j = 0; j < R; ++j) acc[i][j] = fma(As[kk][ty * R + i], Bs[kk][tx + 8 * j], acc[i][j]);
        sync_group();
      }
    }
    // C values are loaded before the first store (a load cannot move above a
    // store that may alias it); then, below the diagonal, the transposed tile C[n][m]
#pragma unroll
    for(int w = 0; w < 2; ++w) {
      if(w == 1 && !(lower && tm != tn)) break;
      T cv[R][R];
#pragma unroll
      for(int i = 0; i < R; ++i)
#pragma unroll
        for(int j = 0; j < R; ++j) {
          const int64_t m = m0 + ty * R + i, n = n0 + tx + 8 * j;
          cv[i][j] = (beta != T(0) && m < M && n < N) ? (w ? C[n * ldc + m] : C[m * ldc + n]) : T(0);
        }
#pragma unroll
      for(int i = 0; i < R; ++i)
#pragma unroll
        for(int j = 0; j < R; ++j) {
          const int64_t m = m0 + ty * R + i, n = n0 + tx + 8 * j;
          if(m < M && n < N) (w ? C[n * ldc + m] : C[m * ldc + n]) = fma(beta, cv[i][j], alpha * acc[i][j]);
        }
    }
  }
}

template <typename T>
gbpoly_status launch_tiled_gemm(gbpoly_ctx* ctx, int64_t M, int64_t N, int64_t K, T alpha, TiledOperand<T> a,
    TiledOperand<T> b, bool dual, TiledOperand<T> a2, TiledOperand<T> b2, T beta, T* C, int64_t ldc,
    bool lower = false) {
  if(M == 0 || N == 0) return GBPOLY_OK;
  const int64_t gx = (N + kTiledTile - 1) / kTiledTile, gy = (M + kTiledTile - 1) / kTiledTile;
  if((M + 63) / 64 > 65535) return fail(GBPOLY_ERR_UNSUPPORTED, "matrix too tall for the tiled kernel grid");
  lower = lower && M == N;
  const int64_t tiles = lower ? gy * (gy + 1) / 2 : gx * gy;
  if(tiles >= (1ll << 31)) return fail(GBPOLY_ERR_UNSUPPORTED, "matrix too large for the tiled kernel grid");
  ProfileScope prof(ctx, "dgemm_tiled");
  const unsigned ctas = unsigned(std::min<int64_t>(tiles, std::max(1, ctx->sm_count)));
  GBPOLY_CUDA_TRY(launch_pdl(ctx, tiled_gemm_kernel<T>, ctas, 64 * kTiledGroups, 0, M, N, K, alpha, a, b, dual, a2, b2,
      beta, C, ldc, lower, gx, tiles));
  return GBPOLY_OK;
}

}  // namespace gbpoly
