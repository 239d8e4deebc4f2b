// Matrix-vector products of the PolyBench BLAS-2 benchmarks (atax, bicg,
// mvt, gesummv), HBM-bound: every kernel reads each matrix element once.
//
// The reference runs one work-item per output element: row dots walk a row
// per work-item (uncoalesced across the work-group), column sums walk a
// column (polybench/atax.cpp:73-97, bicg.cpp:77-100, mvt.cpp:75-98,
// gesummv.cpp:84-98).  Here one pass over the matrix serves up to two row
// dots (y = A x, or A x and B x for gesummv) and one column sum (A^T v):
//   * a CTA of 256 threads owns a 1024-column tile (per thread 4 adjacent
//     columns, one 128-bit load, where rows are 16-byte aligned; else columns
//     t, t + 256, ..., four 32-bit loads of adjacent lanes) and a group of
//     rows; each row of the tile is one coalesced 4 KB read, 16 rows in flight
//     per thread (8 per matrix for two);
//   * row dots: a thread's 4 columns give one term per row; each group of rows
//     in flight is reduced across the warp at once (a halving transpose
//     exchange: 16 shuffles for 16 rows), the 8 warps in shared memory per
//     32-row block, into one partial per (column tile, row);
//   * column sums: 4 accumulators per thread, a batch of 16 (8) rows summed by
//     itself and added to the group's, one partial per (row group, column);
//   * a final kernel (1 to 16 warps per 32 outputs, by the number of partials)
//     adds them in a fixed order and applies y = beta * y + alpha * sum
//     (gesummv: tmp += A x, y = alpha tmp + beta (y + B x)).
// Deterministic: the summation tree depends only on the shape and SM count.
// No kernel here triggers the next one early: its waiting CTAs would settle on
// the SMs that drain first (queued calls 0.5 to 1 us slower).
#include "gbpoly_internal.cuh"

namespace gbpoly {
namespace {

constexpr int kThreads = 256;
constexpr int kTileCols = 4 * kThreads;  // 1024
constexpr int kRowBlock = 32;
constexpr int kRowBatch = 16;  // row groups are multiples of this
// rows in flight per thread: 16 for one matrix, 8 each for two (gesummv)
template <bool TWO>
constexpr int rows_in_flight() {
  return TWO ? 8 : 16;
}

struct GemvArgs {
  const float* A;
  int64_t lda;
  const float* B;  // second matrix (gesummv), row dot 1 reads it with xr[1]
  int64_t ldb;
  int rows, cols;
  const float* xr[2];  // row-dot vectors (cols entries)
  const float* xc;     // column-sum weights (rows entries)
  float* row_part;     // [NR][col_tiles][rows]
  float* col_part;     // [row_groups][cols]
  int col_tiles, rows_per_group;
};

// The four columns of thread t in a 1024-column tile starting at c0: 4 t .. + 3
// (VEC), or t, t + 256, t + 512, t + 768, so that every 32-bit load of a warp is
// one 128-byte segment (measured with odd rows, against 4 t .. + 3 and the final
// kernel of 8 warps: bicg 7000 x 7001 48.9 -> 41.8 us, gesummv 76.3 -> 66.9).
template <bool VEC>
__device__ __forceinline__ float4 load4(const float* __restrict__ p, int c0, int cols) {
  const int t = threadIdx.x;
  if constexpr(VEC) {
    const int c = c0 + 4 * t;
    return c < cols ? *reinterpret_cast<const float4*>(p + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const int c = c0 + t;
  return make_float4(c < cols ? p[c] : 0.f, c + 256 < cols ? p[c + 256] : 0.f, c + 512 < cols ? p[c + 512] : 0.f,
      c + 768 < cols ? p[c + 768] : 0.f);
}
template <bool VEC>
__device__ __forceinline__ void store4(float* __restrict__ p, int c0, int cols, float4 v) {
  const int t = threadIdx.x;
  if constexpr(VEC) {
    const int c = c0 + 4 * t;
    if(c < cols) *reinterpret_cast<float4*>(p + c) = v;
    return;
  }
  const int c = c0 + t;
  if(c < cols) p[c] = v.x;
  if(c + 256 < cols) p[c + 256] = v.y;
  if(c + 512 < cols) p[c + 512] = v.z;
  if(c + 768 < cols) p[c + 768] = v.w;
}

__device__ __forceinline__ float dot4(float4 a, float4 x) {
  return fmaf(a.w, x.w, fmaf(a.z, x.z, fmaf(a.y, x.y, a.x * x.x)));
}

// Warp-wide sums of V (8 or 16) values per lane: halving exchanges (V/2 +
// ... + 1 shuffles) leave lane l with the sum of v[l % V] over its group of V
// lanes, butterfly steps add the 32 / V groups.  Every lane ends with the
// total of v[lane % V].
template <int V>
__device__ __forceinline__ float reduce_rows(float (&v)[V], int lane) {
#pragma unroll
  for(int s = V / 2; s >= 1; s >>= 1) {
    const bool upper = (lane & s) != 0;
#pragma unroll
    for(int i = 0; i < s; ++i) {
      const float send = upper ? v[i] : v[i + s];
      const float keep = upper ? v[i + s] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
    }
  }
  float r = v[0];
#pragma unroll
  for(int s = V; s < 32; s <<= 1) r += __shfl_xor_sync(0xffffffffu, r, s);
  return r;
}

// v(0) + ... + v(7), the eight warps' sums, in pairs.
template <class V>
__device__ __forceinline__ float sum8(V v) {
  static_assert(kThreads / 32 == 8, "eight warps");
  return ((v(0) + v(1)) + (v(2) + v(3))) + ((v(4) + v(5)) + (v(6) + v(7)));
}

// NR row dots (0..2), NC: one column sum, TWO: row dot 1 reads B.
// VEC: 16-byte aligned rows and columns a multiple of 4 (128-bit loads).
template <int NR, bool NC, bool TWO, bool VEC>
__global__ void __launch_bounds__(kThreads, 2) gemv_partial_kernel(const GemvArgs g) {
  __shared__ float red[NR > 0 ? NR : 1][kThreads / 32][kRowBlock];
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tile = blockIdx.x;
  const int c0 = tile * kTileCols;
  // Rows are numbered from -kBase, so that no step past the last one reaches 2^31
  // (numbered from the group's first row, A x of 2000 x 2000 took 5.5 us for 4.85).
  constexpr int kBase = 2 * kRowBlock;
  const int rg0 = int(blockIdx.y * g.rows_per_group) - kBase;
  const int rg1 = rg0 + min(g.rows_per_group, g.rows - kBase - rg0);
  const float* const A = g.A + kBase * g.lda;
  const float* const B = TWO ? g.B + kBase * g.ldb : nullptr;
  const float* const xc = NC ? g.xc + kBase : nullptr;

  float4 xr[NR > 0 ? NR : 1];
#pragma unroll
  for(int t = 0; t < NR; ++t) xr[t] = load4<VEC>(g.xr[t], c0, g.cols);
  float4 colacc = make_float4(0.f, 0.f, 0.f, 0.f);

  constexpr int kInFlight = rows_in_flight<TWO>();
  for(int r0 = rg0; r0 < rg1; r0 += kRowBlock) {
    // a thread's 4 columns of a row give one term of that row's dot product;
    // each group of rows in flight is reduced across the warp at once
#pragma unroll 1
    for(int rr = 0; rr < kRowBlock; rr += kInFlight) {
      float4 a[kInFlight], b[TWO ? kInFlight : 1];
#pragma unroll
      for(int k = 0; k < kInFlight; ++k) {
        const int r = r0 + rr + k;
        const bool ok = r < rg1;
        a[k] = ok ? load4<VEC>(A + int64_t(r) * g.lda, c0, g.cols) : make_float4(0.f, 0.f, 0.f, 0.f);
        if constexpr(TWO) b[k] = ok ? load4<VEC>(B + int64_t(r) * g.ldb, c0, g.cols) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for(int t = 0; t < NR; ++t) {
        float v[kInFlight];
#pragma unroll
        for(int k = 0; k < kInFlight; ++k) v[k] = dot4((TWO && t == 1) ? b[TWO ? k : 0] : a[k], xr[t]);
        const float rs = reduce_rows<kInFlight>(v, lane);
        if(lane < kInFlight) red[t][warp][rr + lane] = rs;
      }
      if constexpr(NC) {
        // the batch by itself, then onto the group's sum: a chain of 16 terms and
        // one of batches, not one of all the group's rows
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for(int k = 0; k < kInFlight; ++k) {
          const int r = r0 + rr + k;
          const float w = r < rg1 ? __ldg(xc + r) : 0.f;
          sum.x = fmaf(a[k].x, w, sum.x);
          sum.y = fmaf(a[k].y, w, sum.y);
          sum.z = fmaf(a[k].z, w, sum.z);
          sum.w = fmaf(a[k].w, w, sum.w);
        }
        colacc.x += sum.x, colacc.y += sum.y, colacc.z += sum.z, colacc.w += sum.w;
      }
    }
    if constexpr(NR > 0) {
      __syncthreads();
      if(warp < NR) {
        const float s = sum8([&](int w) { return red[warp][w][lane]; });
        const int r = r0 + lane;
        if(r < rg1) g.row_part[(int64_t(warp) * g.col_tiles + tile) * g.rows + kBase + r] = s;
      }
      __syncthreads();
    }
  }
  if constexpr(NC) store4<VEC>(g.col_part + int64_t(blockIdx.y) * g.cols, c0, g.cols, colacc);
}

struct Term {
  float alpha, beta;
  float* y;
};

// alpha * s + beta * y[i]; y is not read when beta == 0 (NaN in y does not propagate)
__device__ __forceinline__ float apply(const Term& t, float s, int i) {
  return t.beta == 0.f ? t.alpha * s : fmaf(t.alpha, s, t.beta * t.y[i]);
}

// Final pass: the partials of each output added in a fixed order, then
//   row terms:   y_r[i] = beta y_r[i] + alpha sum over column tiles of row_part[t][.][i]
//   column term: y_c[j] = beta y_c[j] + alpha sum over row groups of col_part[.][j]
//   GESUMMV:     tmp += S0, y = alpha tmp + beta (y + S1) (row terms 0, 1)
// W warps share 32 outputs (lane = output): warp w of them adds the partials
// w, w + W, ..., eight loads in flight, and their sums are combined in shared
// memory in pairs, in warp order.  A CTA of 16 warps holds 16 / W such groups; the first
// row_blocks CTAs take the row outputs, the others the column outputs, each
// with the W that final_warps gives for its number of partials.
//
// Bound: starting CTAs where outputs are many and their partials few, the
// latency of the chain of loads where the partials are many, so W follows both
// (us of the whole call, 16 warps for every 32 outputs / this rule: mvt 1000000
// x 200 613 / 386, bicg 200 x 1000000 231 / 143, bicg 4096 x 4096 12.3 / 10.2).
constexpr int kFinalWarps = 16, kFinalLoads = 8;

// Groups of 32 outputs that share a CTA's warps, as CTAs.
int64_t final_blocks(int64_t outputs, int w) { return (outputs + 32 * kFinalWarps / w - 1) / (32 * kFinalWarps / w); }

// The least power of two of warps whose loads in flight cover n partials; more
// while the outputs give fewer CTAs than the device has SMs.
int final_warps(int64_t outputs, int n, int sms) {
  int w = 1;
  while(w < kFinalWarps && (n > kFinalLoads * w || final_blocks(outputs, w) < sms)) w *= 2;
  return w;
}

// Sum over p[g * stride], g = first, first + step, ... < n.
__device__ __forceinline__ float strided_sum(const float* __restrict__ p, int64_t stride, int n, int first, int step) {
  float s[kFinalLoads];
#pragma unroll
  for(int k = 0; k < kFinalLoads; ++k) s[k] = 0.f;
  for(int g = first; g < n; g += kFinalLoads * step) {
#pragma unroll
    for(int k = 0; k < kFinalLoads; ++k) {
      const int i = g + k * step;
      s[k] += i < n ? p[int64_t(i) * stride] : 0.f;
    }
  }
  return ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
}

template <int NR, bool NC, bool GESUMMV>
__global__ void __launch_bounds__(32 * kFinalWarps) gemv_final_kernel(const float* __restrict__ row_part, int col_tiles,
    int rows, int row_warps, int row_blocks, const float* __restrict__ col_part, int row_groups, int cols, int col_warps,
    Term r0, Term r1, Term cterm) {
  constexpr int kSums = NR > 1 ? NR : 1;
  __shared__ float red[kSums][kFinalWarps][32];
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool row_side = NR > 0 && (!NC || int(blockIdx.x) < row_blocks);
  const int W = row_side ? row_warps : col_warps, part = warp & (W - 1);
  const int block = int(blockIdx.x) - (row_side ? 0 : row_blocks);
  const int64_t i = ((int64_t(block) * kFinalWarps + warp) >> (31 - __clz(W))) * 32 + lane;
  if(row_side) {
#pragma unroll
    for(int t = 0; t < NR; ++t)
      red[t][warp][lane] =
          i < rows ? strided_sum(row_part + int64_t(t) * col_tiles * rows + i, rows, col_tiles, part, W) : 0.f;
  } else if constexpr(NC) {
    red[0][warp][lane] = i < cols ? strided_sum(col_part + i, cols, row_groups, part, W) : 0.f;
  }
  __syncthreads();
  if(part != 0) return;
  float sum[kSums];
#pragma unroll
  for(int t = 0; t < kSums; ++t) {
    if(t > 0 && !row_side) break;
    sum[t] = red[t][warp][lane];
    if(W > 1) sum[t] += red[t][warp + 1][lane];
    for(int w = 2; w < W; w += 2) sum[t] += red[t][warp + w][lane] + red[t][warp + w + 1][lane];
  }
  if(row_side) {
    if(NR == 0 || i >= rows) return;
    if constexpr(GESUMMV) {
      const float tmp = r0.y[i] + sum[0];
      r0.y[i] = tmp;
      r1.y[i] = r1.beta == 0.f ? r1.alpha * tmp : fmaf(r1.alpha, tmp, r1.beta * (r1.y[i] + sum[NR > 1 ? 1 : 0]));
    } else {
      r0.y[i] = apply(r0, sum[0], i);
      if constexpr(NR > 1) r1.y[i] = apply(r1, sum[1], i);
    }
  } else if constexpr(NC) {
    if(i < cols) cterm.y[i] = apply(cterm, sum[0], i);
  }
}

// The final pass over `rows` row outputs of col_tiles partials and `cols` column outputs of row_groups partials.
template <int NR, bool NC, bool GESUMMV>
gbpoly_status launch_final(gbpoly_ctx* ctx, const float* row_part, int col_tiles, int rows, const float* col_part,
    int row_groups, int cols, Term r0, Term r1, Term ct) {
  const int rw = final_warps(rows, col_tiles, ctx->sm_count), cw = final_warps(cols, row_groups, ctx->sm_count);
  const int64_t row_blocks = NR > 0 ? final_blocks(rows, rw) : 0, all = row_blocks + (NC ? final_blocks(cols, cw) : 0);
  if(all == 0) return GBPOLY_OK;
  ProfileScope prof(ctx, "gemv_final");
  GBPOLY_CUDA_TRY(launch_pdl(ctx, gemv_final_kernel<NR, NC, GESUMMV>, unsigned(all), 32 * kFinalWarps, 0, row_part,
      col_tiles, rows, rw, int(row_blocks), col_part, row_groups, cols, cw, r0, r1, ct));
  return GBPOLY_OK;
}

template <int NR, bool NC, bool TWO, bool GESUMMV>
gbpoly_status launch_gemv(gbpoly_ctx* ctx, GemvArgs g, Term r0, Term r1, Term ct, const char* name) {
  // An empty matrix runs only the final kernel, with empty sums: y = beta y,
  // and for gesummv tmp unchanged, y = alpha tmp + beta y.
  const int col_tiles = std::max(1, (g.cols + kTileCols - 1) / kTileCols);
  // Two CTAs per SM are resident.  Long row groups run as two full waves; where
  // those would be short (under 64 rows; 16 of two matrices), one wave of twice the rows leaves no
  // part-filled second one (bicg 4096: 17.7 us against 18.4 with 128 groups of 32 rows).
  const int64_t ctas = 2ll * std::max(ctx->sm_count, 1);
  const int64_t two_waves = std::max<int64_t>(1, 2 * ctas / col_tiles), one_wave = std::max<int64_t>(1, ctas / col_tiles);
  const int64_t want_groups = g.rows / two_waves >= (TWO ? 16 : 64) ? two_waves : one_wave;
  // whole batches of loads: a last one of a few rows takes as long as a full one (bicg 1000000 x 200 370 -> 356 us)
  const int rpg = int((std::max<int64_t>(1, (g.rows + want_groups - 1) / want_groups) + kRowBatch - 1) / kRowBatch * kRowBatch);
  const int row_groups = int(std::max<int64_t>(1, (int64_t(g.rows) + rpg - 1) / rpg));
  if(row_groups > 65535) return fail(GBPOLY_ERR_UNSUPPORTED, "too many rows");
  g.col_tiles = col_tiles;
  g.rows_per_group = rpg;
  const size_t row_floats = size_t(NR) * col_tiles * size_t(g.rows);
  const size_t col_floats = NC ? size_t(row_groups) * size_t(g.cols) : 0;
  const size_t row_bytes = (row_floats * 4 + 255) / 256 * 256;
  gbpoly_status st = ensure_scratch(ctx, ctx->stats, row_bytes + col_floats * 4 + 256, "matrix-vector scratch");
  if(st != GBPOLY_OK) return st;
  g.row_part = static_cast<float*>(ctx->stats.ptr);
  g.col_part = reinterpret_cast<float*>(static_cast<char*>(ctx->stats.ptr) + row_bytes);
  const bool vec = (g.cols % 4 == 0) && (g.lda % 4 == 0) && ((reinterpret_cast<uintptr_t>(g.A) & 15) == 0) &&
                   (!TWO || ((g.ldb % 4 == 0) && ((reinterpret_cast<uintptr_t>(g.B) & 15) == 0))) &&
                   (NR < 1 || (reinterpret_cast<uintptr_t>(g.xr[0]) & 15) == 0) &&
                   (NR < 2 || (reinterpret_cast<uintptr_t>(g.xr[1]) & 15) == 0);
  if(g.rows > 0 && g.cols > 0) {
    ProfileScope prof(ctx, name);
    const dim3 grid{unsigned(col_tiles), unsigned(row_groups), 1u};
    if(vec)
      GBPOLY_CUDA_TRY(launch_pdl(ctx, gemv_partial_kernel<NR, NC, TWO, true>, grid, kThreads, 0, g));
    else
      GBPOLY_CUDA_TRY(launch_pdl(ctx, gemv_partial_kernel<NR, NC, TWO, false>, grid, kThreads, 0, g));
  }
  const bool some = g.rows > 0 && g.cols > 0;
  return launch_final<NR, NC, GESUMMV>(ctx, g.row_part, some ? col_tiles : 0, g.rows, g.col_part, some ? row_groups : 0,
      g.cols, r0, r1, ct);
}

// atax in one kernel and one read of A: tmp += A x, then y += A^T tmp.  A CTA
// owns a contiguous range of rows and holds ROWS of them at a time in registers
// (CHUNKS 1024-column tiles, cols <= CHUNKS * 1024, at most 8): it reduces their
// row dots over the CTA (one barrier; tmp of those rows is then final) and adds
// A[r][c] tmp[r] from the same registers into its column accumulators, written
// once at the end as the CTA's row of col_part.  Two CTAs per SM up to 4096
// columns, so that one's loads run while the other reduces.
//
// Bound: HBM, one read of A.  Reading the rows again from L2 for the second
// product (16 rows, two barriers) kept fewer loads in flight: 4096 x 4096, A
// from HBM, 21.6 -> 18.9 us (floor 9.9); odd rows, which took two passes, 45 ->
// 21.5 us at 4095 x 4097 and 88.6 -> 43.7 at 7000 x 7001.
constexpr int atax_rows(int chunks) { return chunks == 1 ? 16 : (chunks == 2 ? 8 : 4); }
constexpr int atax_ctas(int chunks) { return chunks <= 4 ? 2 : 1; }  // per SM

template <int CHUNKS, bool VEC>
__global__ void __launch_bounds__(kThreads, atax_ctas(CHUNKS)) atax_kernel(const float* __restrict__ A, int64_t lda,
    int rows, int cols, const float* __restrict__ x, float* __restrict__ tmp, float* __restrict__ col_part) {
  constexpr int R = atax_rows(CHUNKS);
  __shared__ float red[2][kThreads / 32 + 1][R];  // warp sums and the old tmp, alternating sets
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int begin = int(int64_t(rows) * blockIdx.x / gridDim.x);
  const int count = int(int64_t(rows) * (blockIdx.x + 1) / gridDim.x) - begin;
  float4 xr[CHUNKS], colacc[CHUNKS];
#pragma unroll
  for(int ch = 0; ch < CHUNKS; ++ch) {
    xr[ch] = load4<VEC>(x, ch * kTileCols, cols);
    colacc[ch] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for(int i = 0, it = 0; i < count; i += R, it ^= 1) {  // (begin + i, stepped, could pass the largest row count)
    const int r0 = begin + i, nr = min(R, count - i);
    float4 a[R][CHUNKS];
#pragma unroll
    for(int k = 0; k < R; ++k)
#pragma unroll
      for(int ch = 0; ch < CHUNKS; ++ch)
        a[k][ch] = k < nr ? load4<VEC>(A + int64_t(r0 + k) * lda, ch * kTileCols, cols) : make_float4(0.f, 0.f, 0.f, 0.f);
    if(tid < R) red[it][kThreads / 32][tid] = tid < nr ? tmp[r0 + tid] : 0.f;
    float acc[R];
#pragma unroll
    for(int k = 0; k < R; ++k) {
      acc[k] = 0.f;
#pragma unroll
      for(int ch = 0; ch < CHUNKS; ++ch) acc[k] += dot4(a[k][ch], xr[ch]);
    }
    const float rs = reduce_rows<R>(acc, lane);
    // (zero beyond nr, where a zero row times an infinite x is NaN)
    if(lane < R) red[it][warp][lane] = lane < nr ? rs : 0.f;
    __syncthreads();  // (a set is rewritten two groups later, after the next group's barrier)
#pragma unroll
    for(int k = 0; k < R; ++k) {
      const float sum = sum8([&](int w) { return red[it][w][k]; });
      const float t = red[it][kThreads / 32][k] + sum;  // tmp += A x (atax.cpp:78-83); zero beyond nr
      if(tid == 0 && k < nr) tmp[r0 + k] = t;
#pragma unroll
      for(int ch = 0; ch < CHUNKS; ++ch) {  // y += A^T tmp (atax.cpp:91-96)
        colacc[ch].x = fmaf(a[k][ch].x, t, colacc[ch].x);
        colacc[ch].y = fmaf(a[k][ch].y, t, colacc[ch].y);
        colacc[ch].z = fmaf(a[k][ch].z, t, colacc[ch].z);
        colacc[ch].w = fmaf(a[k][ch].w, t, colacc[ch].w);
      }
    }
  }
#pragma unroll
  for(int ch = 0; ch < CHUNKS; ++ch)
    store4<VEC>(col_part + int64_t(blockIdx.x) * cols, ch * kTileCols, cols, colacc[ch]);
}

template <int CHUNKS>
gbpoly_status launch_atax(gbpoly_ctx* ctx, const float* A, int64_t lda, int rows, int cols, const float* x, float* tmp,
    float* y, bool vec) {
  const int ctas = atax_ctas(CHUNKS) * std::max(ctx->sm_count, 1);
  const int grid = std::max(1, std::min((rows - 1) / atax_rows(CHUNKS) + 1, ctas));
  gbpoly_status st = ensure_scratch(ctx, ctx->stats, size_t(grid) * size_t(cols) * 4 + 256, "matrix-vector scratch");
  if(st != GBPOLY_OK) return st;
  float* col_part = static_cast<float*>(ctx->stats.ptr);
  {
    ProfileScope prof(ctx, "atax");
    GBPOLY_CUDA_TRY(launch_pdl(ctx, vec ? atax_kernel<CHUNKS, true> : atax_kernel<CHUNKS, false>, grid, kThreads, 0, A, lda,
        rows, cols, x, tmp, col_part));
  }
  return launch_final<0, true, false>(ctx, nullptr, 0, 0, col_part, grid, cols, Term{}, Term{}, Term{1.f, 1.f, y});
}

gbpoly_status check_common(gbpoly_ctx* ctx, int64_t rows, int64_t cols, const float* A, int64_t lda) {
  if(!ctx) return fail(GBPOLY_ERR_INVALID, "null context");
  GBPOLY_CUDA_TRY(cudaSetDevice(ctx->device));
  if(rows < 0 || cols < 0) return fail(GBPOLY_ERR_INVALID, "negative dimension");
  if(rows >= (1ll << 31) || cols >= (1ll << 31) - kTileCols) return fail(GBPOLY_ERR_UNSUPPORTED, "dimension too large");
  if(rows > 0 && cols > 0) {
    if(!A) return fail(GBPOLY_ERR_INVALID, "matrix: null pointer");
    if(lda < cols) return fail(GBPOLY_ERR_INVALID, "matrix: leading dimension smaller than columns");
  }
  return GBPOLY_OK;
}

}  // namespace
}  // namespace gbpoly

using namespace gbpoly;

extern "C" {

gbpoly_status gbpoly_gemv_pair_f32(gbpoly_ctx* ctx, int64_t rows, int64_t cols, const float* A, int64_t lda,
    const gbpoly_gemv_term* terms, int count) {
  gbpoly_status st = check_common(ctx, rows, cols, A, lda);
  if(st != GBPOLY_OK) return st;
  if(!terms || count < 1 || count > 2) return fail(GBPOLY_ERR_INVALID, "one or two terms");
  const gbpoly_gemv_term* rt[2] = {nullptr, nullptr};
  const gbpoly_gemv_term* cterm = nullptr;
  int nr = 0;
  for(int i = 0; i < count; ++i) {
    const gbpoly_gemv_term& t = terms[i];
    if(t.op != GBPOLY_OP_N && t.op != GBPOLY_OP_T) return fail(GBPOLY_ERR_INVALID, "bad term op");
    const int64_t xlen = t.op == GBPOLY_OP_N ? cols : rows, ylen = t.op == GBPOLY_OP_N ? rows : cols;
    if((xlen > 0 && !t.x) || (ylen > 0 && !t.y)) return fail(GBPOLY_ERR_INVALID, "term vector: null pointer");
    if(t.op == GBPOLY_OP_N) {
      rt[nr++] = &t;
    } else {
      if(cterm) return fail(GBPOLY_ERR_UNSUPPORTED, "at most one transposed term");
      cterm = &t;
    }
  }
  GemvArgs g{};
  g.A = A, g.lda = lda, g.rows = int(rows), g.cols = int(cols);
  Term r0{}, r1{}, ct{};
  if(nr > 0) g.xr[0] = rt[0]->x, r0 = Term{rt[0]->alpha, rt[0]->beta, rt[0]->y};
  if(nr > 1) g.xr[1] = rt[1]->x, r1 = Term{rt[1]->alpha, rt[1]->beta, rt[1]->y};
  if(cterm) g.xc = cterm->x, ct = Term{cterm->alpha, cterm->beta, cterm->y};
  if(nr == 1 && !cterm) return launch_gemv<1, false, false, false>(ctx, g, r0, r1, ct, "gemv_n");
  if(nr == 0 && cterm) return launch_gemv<0, true, false, false>(ctx, g, r0, r1, ct, "gemv_t");
  if(nr == 1 && cterm) return launch_gemv<1, true, false, false>(ctx, g, r0, r1, ct, "gemv_nt");
  return launch_gemv<2, false, false, false>(ctx, g, r0, r1, ct, "gemv_nn");
}

gbpoly_status gbpoly_gemv_f32(gbpoly_ctx* ctx, gbpoly_op op, int64_t rows, int64_t cols, float alpha, const float* A,
    int64_t lda, const float* x, float beta, float* y) {
  gbpoly_gemv_term t{op, alpha, beta, x, y};
  return gbpoly_gemv_pair_f32(ctx, rows, cols, A, lda, &t, 1);
}

gbpoly_status gbpoly_atax_f32(gbpoly_ctx* ctx, int64_t rows, int64_t cols, const float* A, int64_t lda, const float* x,
    float* tmp, float* y) {
  gbpoly_status st = check_common(ctx, rows, cols, A, lda);
  if(st != GBPOLY_OK) return st;
  if((cols > 0 && (!x || !y)) || (rows > 0 && !tmp)) return fail(GBPOLY_ERR_INVALID, "vector: null pointer");
  if(rows == 0 || cols == 0) return GBPOLY_OK;  // empty sums: tmp and y unchanged
  const bool vec = (cols % 4 == 0) && (lda % 4 == 0) && ((reinterpret_cast<uintptr_t>(A) & 15) == 0) &&
                   ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
  const int chunks = int((cols + kTileCols - 1) / kTileCols);
  if(chunks <= 8) {
    switch(chunks) {
    case 1: return launch_atax<1>(ctx, A, lda, int(rows), int(cols), x, tmp, y, vec);
    case 2: return launch_atax<2>(ctx, A, lda, int(rows), int(cols), x, tmp, y, vec);
    case 3: return launch_atax<3>(ctx, A, lda, int(rows), int(cols), x, tmp, y, vec);
    case 4: return launch_atax<4>(ctx, A, lda, int(rows), int(cols), x, tmp, y, vec);
    case 5: return launch_atax<5>(ctx, A, lda, int(rows), int(cols), x, tmp, y, vec);
    case 6: return launch_atax<6>(ctx, A, lda, int(rows), int(cols), x, tmp, y, vec);
    case 7: return launch_atax<7>(ctx, A, lda, int(rows), int(cols), x, tmp, y, vec);
    default: return launch_atax<8>(ctx, A, lda, int(rows), int(cols), x, tmp, y, vec);
    }
  }
  // wide matrices: the two passes
  if((st = gbpoly_gemv_f32(ctx, GBPOLY_OP_N, rows, cols, 1.f, A, lda, x, 1.f, tmp)) != GBPOLY_OK) return st;
  return gbpoly_gemv_f32(ctx, GBPOLY_OP_T, rows, cols, 1.f, A, lda, tmp, 1.f, y);
}

gbpoly_status gbpoly_gesummv_f32(gbpoly_ctx* ctx, int64_t rows, int64_t cols, float alpha, const float* A,
    int64_t lda, const float* B, int64_t ldb, const float* x, float beta, float* tmp, float* y) {
  gbpoly_status st = check_common(ctx, rows, cols, A, lda);
  if(st != GBPOLY_OK) return st;
  if((st = check_common(ctx, rows, cols, B, ldb)) != GBPOLY_OK) return st;
  if((cols > 0 && !x) || (rows > 0 && (!tmp || !y))) return fail(GBPOLY_ERR_INVALID, "vector: null pointer");
  GemvArgs g{};
  g.A = A, g.lda = lda, g.B = B, g.ldb = ldb, g.rows = int(rows), g.cols = int(cols);
  g.xr[0] = x, g.xr[1] = x;
  return launch_gemv<2, false, true, true>(ctx, g, Term{1.f, 1.f, tmp}, Term{alpha, beta, y}, Term{}, "gesummv");
}

}  // extern "C"
