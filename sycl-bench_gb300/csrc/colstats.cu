// Column statistics and column normalisation for the covariance and
// correlation benchmarks (polybench/covariance.cpp, polybench/correlation.cpp):
// the passes that prepare the data matrix before its X^T.X contraction.
//
// The reference gives one work-item per column and walks the rows
// sequentially through global memory (covariance.cpp:84-96,
// correlation.cpp:111-142).  Here a CTA of 8 warps owns 32 adjacent columns and
// one chunk of rows; lane j of every warp reads column j (a warp reads 128
// contiguous bytes of a row), each thread keeps eight independent loads in
// flight, and the 8 warps are combined in shared memory into one partial sum
// per (chunk, column).  Then, in chunk order, the partials are added and the
// division (and, for standard deviations, the square root and the eps clamp)
// applied:
//   * up to 4096 x 4096: the (at most eight) chunks of a column block are a
//     cluster, whose first CTA reads the others' partials from their shared
//     memory: one launch;
//   * beyond: partials in global memory, a second launch of one thread per
//     column; about four CTAs per SM stream the matrix.
// The result does not depend on the launch beyond that fixed summation tree
// (same inputs and shape, same bits).  All arithmetic is FP32.
//
// Bound: HBM or L2, one read of the matrix (3000 x 2000: 3.5 us at the measured
// copy rate).  Mean and standard deviation together, us, clusters / partials in
// global memory: 100 x 100 4.8 / 5.8, 1000 x 1300 6.8 / 10.8, 3000 x 2000 11.0 /
// 12.6, 4096 x 4096 20.0 / 22.2, 4096 x 600 9.5 / 9.7; but 100000 x 1300 260 /
// 178, 1000000 x 500 2376 / 667, 20000 x 8192 231 / 214, 5000 x 16384 119 / 108,
// 2000 x 30000 103 / 85: a cluster's eight chunks are too few CTAs for a high
// matrix, and more than a wave of them for a wide one.  Between, clusters would
// still win (8000 x 1300 15.9 / 19.1, 10000 x 1300 18.4 / 21.2).
//
// No kernel here triggers the next one early: CTAs of later kernels would be
// resident, waiting, on whichever SMs had room, and a grid of a wave of CTAs
// so placed leaves other SMs idle (100000 x 1300, calls queued back to back:
// 252 us with the early trigger, 185 without).
#include "gbpoly_internal.cuh"

namespace gbpoly {
namespace {

constexpr int kColsPerBlock = 32;
constexpr int kWarps = 8;
constexpr int64_t kClusterRows = 4096, kClusterCols = 4096;  // largest matrix reduced by clusters

// sum over rows [r0, r1) of f(X[r][j]) for this thread's column j, rows
// warp, warp + 8, ... of the chunk; eight loads in flight.  What is left after
// the full batches is loaded together (TAIL: short chunks, where it is a good
// part of the work) or row by row (long chunks: the tail's predicates cost
// registers and with them resident CTAs; 2000 x 30000, mean and deviation, 99
// us against 88).  Rows are unsigned: the end of a chunk and a step past the
// last row may lie beyond 2^31 (as signed numbers 4096 x 4096, mean, 11.7 us
// against 9.6).
template <bool CENTERED, bool TAIL>
__device__ __forceinline__ float column_chunk_sum(const float* __restrict__ col, int64_t ldx, unsigned r0, unsigned r1,
    unsigned warp, float m) {
  constexpr int kLoads = 8;
  float a[kLoads];
#pragma unroll
  for(int k = 0; k < kLoads; ++k) a[k] = 0.f;
  auto add = [&](float& s, float x) {
    if constexpr(CENTERED) {
      const float c = x - m;
      s = fmaf(c, c, s);
    } else {
      s += x;
    }
  };
  unsigned r = r0 + warp;
  for(; r + (kLoads - 1) * kWarps < r1; r += kLoads * kWarps) {
    float v[kLoads];
#pragma unroll
    for(int k = 0; k < kLoads; ++k) v[k] = col[int64_t(r + k * kWarps) * ldx];
#pragma unroll
    for(int k = 0; k < kLoads; ++k) add(a[k], v[k]);
  }
  if constexpr(TAIL) {
    float v[kLoads];
#pragma unroll
    for(int k = 0; k < kLoads; ++k) v[k] = r + k * kWarps < r1 ? col[int64_t(r + k * kWarps) * ldx] : 0.f;
#pragma unroll
    for(int k = 0; k < kLoads; ++k)
      if(r + k * kWarps < r1) add(a[k], v[k]);  // beyond the chunk nothing: m - m is NaN for an infinite mean
  } else {
    for(; r < r1; r += kWarps) add(a[0], col[int64_t(r) * ldx]);
  }
  return ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
}

// The chunk's sum for column lane of the block, in every lane of warp 0 (all threads call it).
template <bool CENTERED, bool TAIL>
__device__ __forceinline__ float block_chunk_sum(const float* __restrict__ X, int64_t ldx, int cols, unsigned r0, unsigned r1,
    int j, const float* __restrict__ mean) {
  __shared__ float red[kWarps][kColsPerBlock + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float s = 0.f;
  if(j < cols) s = column_chunk_sum<CENTERED, TAIL>(X + j, ldx, r0, r1, warp, CENTERED ? mean[j] : 0.f);
  red[warp][lane] = s;
  __syncthreads();
  float t = red[0][lane];
#pragma unroll
  for(int w = 1; w < kWarps; ++w) t += red[w][lane];
  return t;
}

template <bool STDDEV>
__device__ __forceinline__ float finish(float s, float divisor, float eps) {
  s = s / divisor;
  if constexpr(STDDEV) {
    s = sqrtf(s);
    s = s <= eps ? 1.f : s;
  }
  return s;
}

// Cluster of 1 x gridDim.y CTAs: one column block, its chunks of rows.
template <bool STDDEV>
__global__ void __launch_bounds__(kWarps * 32) column_cluster_kernel(const float* __restrict__ X, int64_t ldx, int rows,
    int cols, int rows_per_chunk, const float* __restrict__ mean, float divisor, float eps, float* __restrict__ out) {
  __shared__ float part[kColsPerBlock];
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int j = blockIdx.x * kColsPerBlock + lane;
  const int r0 = blockIdx.y * rows_per_chunk, r1 = min(rows, r0 + rows_per_chunk);
  const float t = block_chunk_sum<STDDEV, true>(X, ldx, cols, r0, r1, j, mean);
  if(warp == 0) part[lane] = t;
  cluster_sync();
  if(blockIdx.y == 0 && warp == 0) {
    float s = 0.f;
    for(unsigned c = 0; c < gridDim.y; ++c) s += ld_cluster_f32(cluster_map(&part[lane], c));
    if(j < cols) out[j] = finish<STDDEV>(s, divisor, eps);
  }
  cluster_sync();  // no CTA leaves while its partials are being read
}

// partial[chunk][j] = sum over the chunk's rows of X[r][j] (or (X[r][j] - mean[j])^2).
// Eight CTAs per SM: with six (40 registers) a grid of 938 is two waves (means
// of 2000 x 30000 56.4 us against 42.6).
template <bool CENTERED>
__global__ void __launch_bounds__(kWarps * 32, 8) column_partial_kernel(const float* __restrict__ X, int64_t ldx,
    int rows, int cols, int rows_per_chunk, const float* __restrict__ mean, float* __restrict__ partial) {
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int j = blockIdx.x * kColsPerBlock + lane;
  const unsigned r0 = blockIdx.y * unsigned(rows_per_chunk), r1 = min(unsigned(rows), r0 + unsigned(rows_per_chunk));
  const float t = block_chunk_sum<CENTERED, false>(X, ldx, cols, r0, r1, j, mean);
  if(warp == 0 && j < cols) partial[int64_t(blockIdx.y) * cols + j] = t;
}

// out[j] = (sum of the chunks' partials) / divisor; for standard deviations
// then sqrt, and 1 where the result is <= eps.
template <bool STDDEV>
__global__ void column_final_kernel(const float* __restrict__ partial, int chunks, int cols, float divisor, float eps,
    float* __restrict__ out) {
  pdl_wait();
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if(j >= cols) return;
  float s = 0.f;
#pragma unroll 8
  for(int c = 0; c < chunks; ++c) s += partial[int64_t(c) * cols + j];
  out[j] = finish<STDDEV>(s, divisor, eps);
}

// Y[r][j] = X[r][j] - mean[j], or ((X[r][j] - mean[j]) / scale_div) / stddev[j].
template <bool SCALED>
__global__ void __launch_bounds__(256) center_columns_kernel(const float* X, int64_t ldx, int rows, int cols,
    const float* __restrict__ mean, const float* __restrict__ stddev, float scale_div, float* Y, int64_t ldy,
    int rows_per_block) {
  pdl_wait();
  const int j = blockIdx.x * 32 + (threadIdx.x & 31);
  if(j >= cols) return;
  const float m = mean[j];
  const float sd = SCALED ? stddev[j] : 1.f;
  const int r0 = blockIdx.y * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  // eight rows per batch, all loaded before the first store (Y may be X, so a
  // load could not otherwise move above the previous store)
  constexpr int kBatch = 8;
  for(int rb = r0 + (threadIdx.x >> 5); rb < r1; rb += 8 * kBatch) {
    float v[kBatch];
#pragma unroll
    for(int k = 0; k < kBatch; ++k) {
      const int r = rb + 8 * k;
      v[k] = r < r1 ? X[int64_t(r) * ldx + j] : 0.f;
    }
#pragma unroll
    for(int k = 0; k < kBatch; ++k) {
      const int r = rb + 8 * k;
      float y = v[k] - m;
      if constexpr(SCALED) y = (y / scale_div) / sd;
      if(r < r1) Y[int64_t(r) * ldy + j] = y;
    }
  }
}

__global__ void set_diagonal_kernel(int64_t n, float value, float* C, int64_t ldc) {
  pdl_wait();
  for(int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
    C[i * ldc + i] = value;
}

gbpoly_status check_block(const char* name, const void* p, int64_t rows, int64_t cols, int64_t ld) {
  if(rows > 0 && cols > 0) {
    if(!p) return fail(GBPOLY_ERR_INVALID, std::string(name) + ": null pointer");
    if(ld < cols) return fail(GBPOLY_ERR_INVALID, std::string(name) + ": leading dimension smaller than columns");
  }
  return GBPOLY_OK;
}

gbpoly_status check_args(gbpoly_ctx* ctx, int64_t rows, int64_t cols) {
  if(!ctx) return fail(GBPOLY_ERR_INVALID, "null context");
  GBPOLY_CUDA_TRY(cudaSetDevice(ctx->device));
  if(rows < 0 || cols < 0) return fail(GBPOLY_ERR_INVALID, "negative dimension");
  if(rows >= (1ll << 31) || cols >= (1ll << 31)) return fail(GBPOLY_ERR_UNSUPPORTED, "dimension too large");
  return GBPOLY_OK;
}

// Column reduction: partial pass into the context's stats scratch, final pass into out.
template <bool STDDEV>
gbpoly_status column_reduce(gbpoly_ctx* ctx, int64_t rows, int64_t cols, const float* X, int64_t ldx, const float* mean,
    float divisor, float eps, float* out) {
  if(cols == 0) return GBPOLY_OK;
  const int col_blocks = int((cols + kColsPerBlock - 1) / kColsPerBlock);
  const int cluster = int(std::max<int64_t>(1, std::min<int64_t>(8, (rows + 63) / 64)));
  if(rows <= kClusterRows && cols <= kClusterCols) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    cfg.gridDim = dim3(unsigned(col_blocks), unsigned(cluster));
    cfg.blockDim = dim3(kWarps * 32);
    cfg.stream = ctx->stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1, attr[0].val.clusterDim.y = unsigned(cluster), attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_pdl
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    ProfileScope prof(ctx, STDDEV ? "column_stddev" : "column_mean");
    GBPOLY_CUDA_TRY(cudaLaunchKernelEx(&cfg, column_cluster_kernel<STDDEV>, X, ldx, int(rows), int(cols),
        std::max(int((rows + cluster - 1) / cluster), 1), mean, divisor, eps, out));
    return GBPOLY_OK;
  }
  // about four CTAs per SM, at least 64 rows per chunk
  const int64_t want = std::max<int64_t>(1, (4ll * std::max(ctx->sm_count, 1) + col_blocks - 1) / col_blocks);
  const int64_t chunks = std::max<int64_t>(1, std::min<int64_t>(want, (rows + 63) / 64));
  const int rows_per_chunk = int((rows + chunks - 1) / chunks);
  gbpoly_status st = ensure_scratch(ctx, ctx->stats, size_t(chunks) * size_t(cols) * sizeof(float), "column scratch");
  if(st != GBPOLY_OK) return st;
  float* partial = static_cast<float*>(ctx->stats.ptr);
  {
    ProfileScope prof(ctx, STDDEV ? "column_sumsq" : "column_sum");
    GBPOLY_CUDA_TRY(launch_pdl(ctx, column_partial_kernel<STDDEV>, dim3(unsigned(col_blocks), unsigned(chunks)),
        kWarps * 32, 0, X, ldx, int(rows), int(cols), std::max(rows_per_chunk, 1), mean, partial));
  }
  ProfileScope prof(ctx, STDDEV ? "column_stddev_final" : "column_mean_final");
  GBPOLY_CUDA_TRY(launch_pdl(ctx, column_final_kernel<STDDEV>, unsigned((cols + 255) / 256), 256, 0, partial,
      int(rows > 0 ? chunks : 0), int(cols), divisor, eps, out));
  return GBPOLY_OK;
}

}  // namespace
}  // namespace gbpoly

using namespace gbpoly;

extern "C" {

gbpoly_status gbpoly_column_mean_f32(gbpoly_ctx* ctx, int64_t rows, int64_t cols, const float* X, int64_t ldx,
    float divisor, float* mean) {
  gbpoly_status st = check_args(ctx, rows, cols);
  if(st != GBPOLY_OK) return st;
  if((st = check_block("X", X, rows, cols, ldx)) != GBPOLY_OK) return st;
  if(cols > 0 && !mean) return fail(GBPOLY_ERR_INVALID, "mean: null pointer");
  return column_reduce<false>(ctx, rows, cols, X, ldx, nullptr, divisor, 0.f, mean);
}

gbpoly_status gbpoly_column_stddev_f32(gbpoly_ctx* ctx, int64_t rows, int64_t cols, const float* X, int64_t ldx,
    const float* mean, float divisor, float eps, float* stddev) {
  gbpoly_status st = check_args(ctx, rows, cols);
  if(st != GBPOLY_OK) return st;
  if((st = check_block("X", X, rows, cols, ldx)) != GBPOLY_OK) return st;
  if(cols > 0 && (!mean || !stddev)) return fail(GBPOLY_ERR_INVALID, "mean/stddev: null pointer");
  return column_reduce<true>(ctx, rows, cols, X, ldx, mean, divisor, eps, stddev);
}

gbpoly_status gbpoly_center_columns_f32(gbpoly_ctx* ctx, int64_t rows, int64_t cols, const float* X, int64_t ldx,
    const float* mean, const float* stddev, float scale_div, float* Y, int64_t ldy) {
  gbpoly_status st = check_args(ctx, rows, cols);
  if(st != GBPOLY_OK) return st;
  if((st = check_block("X", X, rows, cols, ldx)) != GBPOLY_OK) return st;
  if((st = check_block("Y", Y, rows, cols, ldy)) != GBPOLY_OK) return st;
  if(cols > 0 && !mean) return fail(GBPOLY_ERR_INVALID, "mean: null pointer");
  if(X == Y && ldx != ldy) return fail(GBPOLY_ERR_INVALID, "in-place centring needs ldy == ldx");
  if(rows == 0 || cols == 0) return GBPOLY_OK;
  constexpr int kRowsPerBlock = 64;
  const dim3 grid(unsigned((cols + 31) / 32), unsigned((rows + kRowsPerBlock - 1) / kRowsPerBlock));
  if(grid.y > 65535u) return fail(GBPOLY_ERR_UNSUPPORTED, "too many rows");
  ProfileScope prof(ctx, stddev ? "normalize_columns" : "center_columns");
  if(stddev)
    GBPOLY_CUDA_TRY(launch_pdl(ctx, center_columns_kernel<true>, grid, 256, 0, X, ldx, int(rows), int(cols), mean, stddev,
        scale_div, Y, ldy, kRowsPerBlock));
  else
    GBPOLY_CUDA_TRY(launch_pdl(ctx, center_columns_kernel<false>, grid, 256, 0, X, ldx, int(rows), int(cols), mean,
        nullptr, 1.f, Y, ldy, kRowsPerBlock));
  return GBPOLY_OK;
}

gbpoly_status gbpoly_covariance_f32(gbpoly_ctx* ctx, gbpoly_precision prec, int64_t rows, int64_t cols, const float* X,
    int64_t ldx, const float* mean, const float* stddev, float scale_div, float* C, int64_t ldc) {
  gbpoly_status st = check_args(ctx, rows, cols);
  if(st != GBPOLY_OK) return st;
  if((st = check_block("X", X, rows, cols, ldx)) != GBPOLY_OK) return st;
  if((st = check_block("C", C, cols, cols, ldc)) != GBPOLY_OK) return st;
  if(cols > 0 && !mean) return fail(GBPOLY_ERR_INVALID, "mean: null pointer");
  if(cols == 0) return GBPOLY_OK;
  GemmF32Args a{};
  a.M = cols, a.N = cols, a.K = rows, a.alpha = 1.f, a.beta = 0.f, a.op_a = GBPOLY_OP_T, a.op_b = GBPOLY_OP_N;
  a.C = C, a.ldc = ldc;
  const bool split_form = prec == GBPOLY_PREC_TF32 || prec == GBPOLY_PREC_BF16X3 || prec == GBPOLY_PREC_TF32X3 ||
                          prec == GBPOLY_PREC_BF16X6 || prec == GBPOLY_PREC_FP16X3;
  if(split_form && rows > 0) {
    // centred in the split pass: X itself is both operands
    a.A = X, a.lda = ldx, a.B = X, a.ldb = ldx;
    a.xf = RowXform{mean, stddev, scale_div};
    return launch_gemm_tensor(ctx, prec, a);
  }
  if(prec != GBPOLY_PREC_FP32 && prec != GBPOLY_PREC_FP8 && !split_form)
    return fail(GBPOLY_ERR_INVALID, "unknown precision");
  // a centred copy with 16-byte-aligned rows, then the contraction
  const int64_t ldy = (cols + 3) / 4 * 4;
  if((st = ensure_scratch(ctx, ctx->centred, size_t(std::max<int64_t>(rows, 1)) * size_t(ldy) * 4 + 256,
          "centred copy")) != GBPOLY_OK)
    return st;
  float* Y = static_cast<float*>(ctx->centred.ptr);
  if((st = gbpoly_center_columns_f32(ctx, rows, cols, X, ldx, mean, stddev, scale_div, Y, ldy)) != GBPOLY_OK)
    return st;
  a.A = Y, a.lda = ldy, a.B = Y, a.ldb = ldy;
  return prec == GBPOLY_PREC_FP32 ? launch_gemm_f32_simt(ctx, a) : launch_gemm_tensor(ctx, prec, a);
}

gbpoly_status gbpoly_set_diagonal_f32(gbpoly_ctx* ctx, int64_t n, float value, float* C, int64_t ldc) {
  gbpoly_status st = check_args(ctx, n, n);
  if(st != GBPOLY_OK) return st;
  if((st = check_block("C", C, n, n, ldc)) != GBPOLY_OK) return st;
  if(n == 0) return GBPOLY_OK;
  ProfileScope prof(ctx, "set_diagonal");
  GBPOLY_CUDA_TRY(launch_pdl(ctx, set_diagonal_kernel, unsigned(std::min<int64_t>((n + 255) / 256, 4096)), 256, 0, n,
      value, C, ldc));
  return GBPOLY_OK;
}

}  // extern "C"
