// Plain FP32 SIMT contraction kernels for sm_103a: the drop-in form of the
// PolyBench kernels polybench/gemm.cpp:82-91, 2mm.cpp:99-122, 3mm.cpp:120-157,
// syrk.cpp:74-83 and syr2k.cpp:78-87.
//
// The reference launches one work-item per C element that walks the whole k
// range through global memory.  Here one CTA owns a 128x128 tile of C:
//   * a producer warpgroup streams BK=32 slices of the A and B panels into a
//     ring of shared-memory stages, each guarded by a full/empty mbarrier
//     pair.  Both tiles lie [k][row or column] there, whatever the operand's
//     layout (Fetch, below);
//   * eight consumer warps (256 threads) each keep an 8x8 block of C in
//     registers and run packed FFMA over 128-bit shared-memory loads;
//   * the epilogue applies C = alpha*acc + beta*C with bounds checks.
// Short K on operands off 16-byte boundaries runs on 64x64 tiles instead
// (use_tile64, below).
// Grids that would not fill the device split K over the CTAs of a cluster.
// syr2k's two products (A_i.B_j + B_i.A_j) stream four tiles per stage into
// the same accumulator.  Symmetric updates (syrk, syr2k, X^T.X) compute only
// the tiles on and below the diagonal; a tile below it also stores its
// transpose (with its own beta * C term), so the full square is written.
//
// Bound: the FP32 pipe, 152 SMs x 128 x 2 x 2070 MHz = 80.5 TFLOP/s; whole
// tiles (M = 2432, N = 4096, K = 2048; op N/N, N/T, T/N, T/T) run at 63.4,
// 62.3, 68.3 and 64.4 TFLOP/s, against 55.7, 52.9, 57.2 and 53.7 with scalar
// FFMA on tiles in their stored layout.  The packed FFMA (two products per
// instruction) takes its operands from register pairs: with both tiles
// [k][...] a pair of B values is half a 16-byte load and only A's 8 values
// per k are duplicated; K-major tiles, whose loads hold 4 k of one row, had
// to be paired by moves (N/N 54, N/T 36 TFLOP/s), and pairs along k need
// twice the accumulators (N/N 26).
#include <algorithm>

#include "gbpoly_internal.cuh"
#include "umma.cuh"

namespace gbpoly {
namespace {

constexpr int kBM = 128, kBN = 128, kBK = 32;
constexpr int kProducers = 128;  // warpgroup 0
constexpr int kConsumers = 256;  // warpgroups 1 and 2: 8 consumer warps
constexpr int kThreads = kProducers + kConsumers;
// Registers per thread after the split: 128 x 40 + 256 x 232 = 64,512, what
// the 384 threads are launched with (168 each).
constexpr uint32_t kRegsProducer = 40, kRegsConsumer = 232;
constexpr int kTileBytes = kBM * kBK * 4;  // 16 KB, same for every tile shape used
constexpr int kMaxSplit = 8;               // CTAs of a cluster (portable cluster size)
// Costs of a CTA besides its k tiles, in k tiles' time (2.4 us; best_split):
// a 64 x 64 x 64 call takes 10.4 us for two k tiles; a split one about 2 us more
constexpr double kFixedTiles = 1.5, kSplitTiles = 0.8;

using umma::regs_decrease;
using umma::regs_increase;

// How a 128-wide, 32-deep operand tile gets into shared memory as
// [32 k][128 rows or columns]:
//   Tma   MN-major operand (rows or columns contiguous) with a 16-byte-aligned
//         base and leading dimension: one 2-D tiled copy;
//   Rows  the same at any alignment: 4-byte cp.async by the 128 producer threads;
//   Turn  K-major operand (k contiguous), any alignment: 4-byte cp.async, the
//         tile turned on the way.  A warp copies 4 rows x 8 k per instruction
//         (four 32-byte sectors) and the 16-byte chunks of k row k are permuted
//         by k % 8, so its 32 words fall in 32 banks.
// The words cost 128 instructions per tile over four warps, against 4096
// cycles of products per tile pair.
enum class Fetch { Tma, Rows, Turn };

// One operand as stored: X[r * ld + c], R x Cn elements.
struct Operand {
  const float* X;
  int64_t ld;
  int R, Cn;
};

__device__ __forceinline__ void cp_async_word(uint32_t dst, const float* src, bool ok) {
  const uint32_t n = ok ? 4u : 0u;  // 0 source bytes: the word is filled with zero
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// One producer thread's words of the tile whose first row or column is x0, zero beyond the matrix.
template <Fetch F>
__device__ __forceinline__ void fetch_words(uint32_t dst, const Operand& o, int x0, int k0) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if constexpr(F == Fetch::Turn) {
    const int kl = lane & 7, rl = lane >> 3;
    const float* p = o.X + int64_t(x0 + 4 * warp + rl) * o.ld + k0 + kl;
#pragma unroll 2
    for(int i = 0; i < 8; ++i) {  // chunks of four rows warp, warp + 4, ...
      const int c = warp + 4 * i;
      const bool row = x0 + 4 * c + rl < o.R;
      const uint32_t d = dst + kl * 512 + ((c ^ kl) << 4) + 4 * rl;
#pragma unroll
      for(int g = 0; g < 4; ++g) {
        const bool ok = row && k0 + 8 * g + kl < o.Cn;
        cp_async_word(d + 8 * 512 * g, ok ? p + 8 * g : o.X, ok);
      }
      p += 16 * o.ld;
    }
  } else {
#pragma unroll 2
    for(int i = 0; i < 8; ++i) {  // k rows warp, warp + 4, ...
      const int k = warp + 4 * i;
      const bool kin = k0 + k < o.R;
      const float* p = o.X + int64_t(k0 + (kin ? k : 0)) * o.ld + x0;
#pragma unroll
      for(int e = 0; e < 4; ++e) {
        const int c = lane + 32 * e;
        const bool ok = kin && x0 + c < o.Cn;
        cp_async_word(dst + 512 * k + 4 * c, ok ? p + c : o.X, ok);
      }
    }
  }
}

// A thread's 8 x 8 block: rows  4 li + 16 (i / 4) + i % 4 of its warp's 32,
// columns 4 lj + 32 (j / 4) + j % 4 of its warp's 64 (lanes 4 x 8, warps 4 x
// 2): per k two 16-byte loads of A (4 distinct in a warp) and two of B (8
// distinct: one shared-memory wavefront each).
__device__ __forceinline__ int owned_row(int li, int i) { return 4 * li + 16 * (i >> 2) + (i & 3); }
__device__ __forceinline__ int owned_col(int lj, int j) { return 4 * lj + 32 * (j >> 2) + (j & 3); }

// Two FP32 fused multiply-adds in one instruction (each rounded as fmaf).
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
  asm volatile("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));  // volatile: keeps the order below
}

// One k tile.  oa, ob: the thread's first 16 bytes of a k row (unpermuted).
// acc[i][h] holds columns 2h and 2h + 1 of row i; a pair of B values is used
// by all eight rows before the next, so that it is read once.
template <bool TURN_A, bool TURN_B>
__device__ __forceinline__ void mma_tile(const char* ta, const char* tb, uint32_t oa, uint32_t ob,
    uint64_t (&acc)[8][4]) {
#pragma unroll
  for(int k8 = 0; k8 < kBK; k8 += 8) {
#pragma unroll
    for(int kk = 0; kk < 8; kk += 4) {
      float a[4][8], b[4][8];
#pragma unroll
      for(int e = 0; e < 4; ++e) {
        const int x = kk + e;  // k % 8
        // a turned tile's chunk c lies at c ^ x; the thread's chunks are its first one plus 4 (A) or 8 (B)
        const char* ra = ta + (TURN_A ? oa ^ (x << 4) : oa) + x * 512;
        const char* rb = tb + (TURN_B ? ob ^ (x << 4) : ob) + x * 512;
        const float4 a0 = *reinterpret_cast<const float4*>(ra);
        const float4 a1 = *reinterpret_cast<const float4*>(ra + (TURN_A && (x & 4) ? -64 : 64));
        const float4 b0 = *reinterpret_cast<const float4*>(rb);
        const float4 b1 = *reinterpret_cast<const float4*>(rb + 128);
        a[e][0] = a0.x, a[e][1] = a0.y, a[e][2] = a0.z, a[e][3] = a0.w;
        a[e][4] = a1.x, a[e][5] = a1.y, a[e][6] = a1.z, a[e][7] = a1.w;
        b[e][0] = b0.x, b[e][1] = b0.y, b[e][2] = b0.z, b[e][3] = b0.w;
        b[e][4] = b1.x, b[e][5] = b1.y, b[e][6] = b1.z, b[e][7] = b1.w;
      }
#pragma unroll
      for(int e = 0; e < 4; ++e)
#pragma unroll
        for(int h = 0; h < 4; ++h) {
          const uint64_t bp = pack2(b[e][2 * h], b[e][2 * h + 1]);
#pragma unroll
          for(int i = 0; i < 8; ++i) fma2(acc[i][h], pack2(a[e][i], a[e][i]), bp);
        }
    }
    ta += 8 * 512, tb += 8 * 512;
  }
}

// Tile rasterisation: groups of 8 tile-rows walk the tile-columns together so
// that concurrently resident CTAs share A and B panels in L2.
__device__ __forceinline__ void tile_coords(int id, int tiles_m, int tiles_n, int& tile_m, int& tile_n) {
  constexpr int G = 8;
  const int per_group = G * tiles_n;
  const int group = id / per_group;
  const int first = group * G;
  const int gsz = min(tiles_m - first, G);
  const int r = id - group * per_group;
  tile_m = first + r % gsz;
  tile_n = r / gsz;
}

// Row-major walk of the lower triangle of tiles: t = tm (tm + 1) / 2 + tn, tn <= tm.
__device__ __forceinline__ void lower_coords(int t, int& tile_m, int& tile_n) {
  int tm = int((sqrtf(8.f * float(t) + 1.f) - 1.f) * 0.5f);
  while(tm * (tm + 1) / 2 > t) --tm;
  while((tm + 1) * (tm + 2) / 2 <= t) ++tm;
  tile_m = tm;
  tile_n = t - tm * (tm + 1) / 2;
}

// syr2k's walk: the tiles below the diagonal, then the diagonal ones, which take half as long.
__device__ __forceinline__ void dual_coords(int t, int tiles, int& tile_m, int& tile_n) {
  const int below = tiles * (tiles - 1) / 2;
  if(t < below) {
    lower_coords(t, tile_m, tile_n);
    ++tile_m;
  } else {
    tile_m = tile_n = t - below;
  }
}

// C = alpha t + beta C for a warp's 32 x 64 block at (m, n), which lies in shared
// memory as t[row][column], and for its mirror: rows of C off 16-byte boundaries.
// The quads' single words would be scattered over a warp's addresses; here a
// lane is a column (of the mirror: a row) and a warp's access a row segment
// (us, quads by words / turned: 8192 x 8192 x 32 262 / 210, 3000 x 3000 x 128 65 /
// 57, syr2k 2000 x 300 67 / 60).  Not inlined: its addresses would cost the
// kernel's other paths registers.
constexpr int kTurnPitch = 65;
__device__ __noinline__ void write_turned(const float* t, int m0, int n0, int M, int N, float alpha, float beta,
    float* __restrict__ C, int64_t ldc, bool mirror) {
  const int lane = threadIdx.x & 31;
  const bool read_c = beta != 0.f;
#pragma unroll 1
  for(int r = 0; r < 32; r += 8) {
    float old[16];
#pragma unroll
    for(int e = 0; e < 16; ++e) {
      const int m = m0 + r + (e >> 1), n = n0 + lane + 32 * (e & 1);
      old[e] = read_c && m < M && n < N ? C[int64_t(m) * ldc + n] : 0.f;
    }
#pragma unroll
    for(int e = 0; e < 16; ++e) {
      const int m = m0 + r + (e >> 1), n = n0 + lane + 32 * (e & 1);
      const float s = t[(r + (e >> 1)) * kTurnPitch + lane + 32 * (e & 1)];
      if(m < M && n < N) C[int64_t(m) * ldc + n] = fmaf(beta, old[e], alpha * s);
    }
  }
  if(!mirror) return;
  const int m = m0 + lane;
#pragma unroll 1
  for(int c = 0; c < 64; c += 16) {
    float old[16];
#pragma unroll
    for(int e = 0; e < 16; ++e) old[e] = read_c && m < M && n0 + c + e < N ? C[int64_t(n0 + c + e) * ldc + m] : 0.f;
#pragma unroll
    for(int e = 0; e < 16; ++e)
      if(m < M && n0 + c + e < N) C[int64_t(n0 + c + e) * ldc + m] = fmaf(beta, old[e], alpha * t[lane * kTurnPitch + c + e]);
  }
}

// FA, FB: how op(A)'s and op(B)'s tiles are fetched.  DUAL: syr2k (both
// operands K-major), tiles A_i, B_j, B_i, A_j.  On the diagonal the second
// product is the first one's transpose, S + S^T: half the copies and half the
// products, the transpose added through shared memory before the exchange.
// (1536: 78 tiles, 12 of them diagonal, as 78 clusters of two on 76 places;
// the last two start when the first diagonal ones end.  132 us against 176
// with both products on every tile, then best as clusters of three in two
// rounds; 512 25.2 -> 20.8, 1280 135 -> 105.  Sizes that run unsplit in whole
// rounds of clusters gain nothing and lose up to 1.6 % to the branch around
// the second product, 2048 330 -> 335; the loop written twice lost 4 % there,
// one body run once or twice 2 % at 1024.)
//
// K split: the gridDim.y CTAs of a cluster take consecutive K ranges of one
// tile.  Each writes its sums to its own shared memory (the drained ring);
// CTA r then adds the cluster's sums of its share of the rows, in rank order
// (every run gives the same bits), and writes them.  No global scratch, no
// second launch: a launch stays independent of every other one, on any
// stream or in any graph.
//
// TURN: unsplit launches on a C whose rows are off 16-byte boundaries, written
// by write_turned.  An instance of its own: beside the quads' path it cost
// syr2k's clusters 1 to 2 us (1000 x 100 15.9 -> 17.7).
template <Fetch FA, Fetch FB, bool DUAL, bool TURN, int STAGES>
__global__ void __launch_bounds__(kThreads, 1) sgemm_kernel(const __grid_constant__ CUtensorMap tmA,
    const __grid_constant__ CUtensorMap tmB, const Operand oa, const Operand ob, int M, int N, int K,
    float alpha, float beta, float* __restrict__ C, int64_t ldc, int lower, int first_tile, int kt_per_split, int* err) {
  constexpr int kTilesPerStage = DUAL ? 4 : 2;
  constexpr int kStageBytes = kTilesPerStage * kTileBytes;
  constexpr int kTmaTiles = DUAL ? 0 : int(FA == Fetch::Tma) + int(FB == Fetch::Tma);
  constexpr bool kWords = kTmaTiles < 2;
  static_assert(!DUAL || (FA == Fetch::Turn && FB == Fetch::Turn), "syr2k: K-major operands");
  extern __shared__ __align__(1024) char smem_raw[];
  // 1024-byte aligned; offset arithmetic keeps the pointer in the shared window
  char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * kStageBytes);
  uint64_t* empty = full + STAGES;

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int tiles_m = (M - 1) / kBM + 1, tiles_n = (N - 1) / kBN + 1;  // (M + kBM could pass 2^31)
  int tile_m, tile_n;
  if constexpr(DUAL)
    dual_coords(first_tile + blockIdx.x, tiles_m, tile_m, tile_n);
  else if(lower)
    lower_coords(first_tile + blockIdx.x, tile_m, tile_n);
  else
    tile_coords(blockIdx.x, tiles_m, tiles_n, tile_m, tile_n);
  const bool diagonal = DUAL && tile_m == tile_n;
  const int m0 = tile_m * kBM, n0 = tile_n * kBN;
  const bool mirror = lower && tile_m != tile_n;
  const int splits = int(gridDim.y), split = int(blockIdx.y);  // the cluster is 1 x splits: split == rank
  const int ktiles = K / kBK + (K % kBK != 0);
  const int kt0 = split * kt_per_split;
  const int nkt = max(0, min(ktiles, kt0 + kt_per_split) - kt0);

  if(tid == 0) {
#pragma unroll
    for(int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], (kTmaTiles > 0 ? 1 : 0) + (kWords ? kProducers : 0));
      mbar_init(&empty[s], kConsumers / 32);
    }
    fence_mbar_init();
  }
  pdl_trigger();
  __syncthreads();
  pdl_wait();

  if(warp < kProducers / 32) {
    // ------------------------------------------------------------ producer
    regs_decrease<kRegsProducer>();
    if(kWords || tid == 0) {
      if constexpr(FA == Fetch::Tma) if(tid == 0) tma_prefetch_desc(&tmA);
      if constexpr(FB == Fetch::Tma) if(tid == 0) tma_prefetch_desc(&tmB);
      int issued = 0;
      for(int i = 0; i < nkt; ++i) {
        const int s = i % STAGES;
        if(i >= STAGES && !mbar_wait(&empty[s], ((i / STAGES) - 1) & 1, err, kDevErrEmptyWait)) break;
        char* st = smem + s * kStageBytes;
        const int k0 = (kt0 + i) * kBK;
        if constexpr(kTmaTiles > 0) {
          if(tid == 0) {
            mbar_arrive_expect_tx(&full[s], kTmaTiles * kTileBytes);
            if constexpr(FA == Fetch::Tma) tma_load_2d(st, &tmA, &full[s], m0, k0);
            if constexpr(FB == Fetch::Tma) tma_load_2d(st + kTileBytes, &tmB, &full[s], n0, k0);
          }
        }
        if constexpr(kWords) {
          const uint32_t d = smem_u32(st);
          if constexpr(FA != Fetch::Tma) fetch_words<FA>(d, oa, m0, k0);
          if constexpr(FB != Fetch::Tma) fetch_words<FB>(d + kTileBytes, ob, n0, k0);
          if(DUAL && !diagonal) {
            fetch_words<FB>(d + 2 * kTileBytes, ob, m0, k0);
            fetch_words<FA>(d + 3 * kTileBytes, oa, n0, k0);
          }
          // one arrival per producer thread, when its copies so far have landed
          asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(smem_u32(&full[s])) : "memory");
        }
        ++issued;
      }
      // Drain: do not leave the CTA while copies into its shared memory are in flight.
      if constexpr(kWords) asm volatile("cp.async.wait_all;" ::: "memory");
      if(kTmaTiles > 0 && tid == 0)
        for(int kt = max(0, issued - STAGES); kt < issued; ++kt)
          if(!mbar_drain(&full[kt % STAGES], (kt / STAGES) & 1, err)) break;
    }
    __syncwarp();
    if(!TURN && splits > 1) {
      cluster_sync();  // the cluster's sums are written
      cluster_arrive();
      cluster_wait();  // and read
    }
    return;
  }

  // -------------------------------------------------------------- consumers
  regs_increase<kRegsConsumer>();
  const int ctid = tid - kProducers, cwarp = ctid >> 5;
  const int li = lane >> 3, lj = lane & 7;
  const int wr = 32 * (cwarp >> 1), wc = 64 * (cwarp & 1);  // the warp's rows and columns of the tile
  uint64_t acc2[8][4];
#pragma unroll
  for(auto& row : acc2)
#pragma unroll
    for(auto& v : row) v = 0;

  bool ok = true;
  for(int kt = 0; kt < nkt; ++kt) {
    if(kt == max(0, nkt - 4) && beta != 0.f) {
      // C of the tile (and of its mirror) into L2 a few k tiles before the
      // epilogue reads it: 512 lines of 128 bytes, two per consumer thread
#pragma unroll
      for(int e = 0; e < 2; ++e) {
        const int line = ctid + kConsumers * e, r = line >> 2, c = 32 * (line & 3);
        if(m0 + r < M && n0 + c < N) prefetch_l2(C + int64_t(m0 + r) * ldc + n0 + c);
        if(mirror && n0 + r < N && m0 + c < M) prefetch_l2(C + int64_t(n0 + r) * ldc + m0 + c);
      }
    }
    const int s = kt % STAGES;
    if(!mbar_wait(&full[s], (kt / STAGES) & 1, err, kDevErrFullWait)) {
      ok = false;
      break;
    }
    const char* st = smem + s * kStageBytes;
    mma_tile<FA == Fetch::Turn, FB == Fetch::Turn>(st, st + kTileBytes, 4 * wr + 16 * li, 4 * wc + 16 * lj, acc2);
    if(DUAL && !diagonal)
      mma_tile<true, true>(st + 2 * kTileBytes, st + 3 * kTileBytes, 4 * wr + 16 * li, 4 * wc + 16 * lj, acc2);
    __syncwarp();
    if(lane == 0) mbar_arrive(&empty[s]);
  }

  // The thread's block as 16 quads: quad f is row f / 2, columns 4 (f % 2) .. + 3.
  float4 acc[16];
#pragma unroll
  for(int f = 0; f < 16; ++f) {
    unpack2(acc2[f / 2][2 * (f & 1)], acc[f].x, acc[f].y);
    unpack2(acc2[f / 2][2 * (f & 1) + 1], acc[f].z, acc[f].w);
  }
  const bool read_c = beta != 0.f;
  const bool vec = (ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;  // 16-byte-aligned rows
  auto row_of = [&](int f) { return m0 + wr + owned_row(li, f >> 1); };
  auto col_of = [&](int f) { return n0 + wc + owned_col(lj, 4 * (f & 1)); };
  auto load_c = [&](int f) {
    const int r = row_of(f), c = col_of(f);
    const float* p = C + static_cast<int64_t>(r) * ldc + c;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if(!read_c || r >= M) return v;
    if(vec && c + 3 < N) return *reinterpret_cast<const float4*>(p);
    if(c < N) v.x = p[0];
    if(c + 1 < N) v.y = p[1];
    if(c + 2 < N) v.z = p[2];
    if(c + 3 < N) v.w = p[3];
    return v;
  };
  auto store_c = [&](int f, float4 s, float4 old) {
    const int r = row_of(f), c = col_of(f);
    float* p = C + static_cast<int64_t>(r) * ldc + c;
    if(r >= M) return;
    const float4 o = make_float4(fmaf(beta, old.x, alpha * s.x), fmaf(beta, old.y, alpha * s.y),
        fmaf(beta, old.z, alpha * s.z), fmaf(beta, old.w, alpha * s.w));
    if(vec && c + 3 < N) {
      *reinterpret_cast<float4*>(p) = o;
      return;
    }
    if(c < N) p[0] = o.x;
    if(c + 1 < N) p[1] = o.y;
    if(c + 2 < N) p[2] = o.z;
    if(c + 3 < N) p[3] = o.w;
  };
  // a mirrored tile's transpose, strictly above the diagonal: C[n][m] from the product element (m, n)
  auto load_t = [&](int f) {
    const int r = row_of(f), c = col_of(f);
    const float* p = C + static_cast<int64_t>(c) * ldc + r;
    const bool ok = read_c && r < M;
    return make_float4(ok && c < N ? p[0] : 0.f, ok && c + 1 < N ? p[ldc] : 0.f, ok && c + 2 < N ? p[2 * ldc] : 0.f,
        ok && c + 3 < N ? p[3 * ldc] : 0.f);
  };
  auto store_t = [&](int f, float4 s, float4 old) {
    const int r = row_of(f), c = col_of(f);
    float* p = C + static_cast<int64_t>(c) * ldc + r;
    if(r >= M) return;
    if(c < N) p[0] = fmaf(beta, old.x, alpha * s.x);
    if(c + 1 < N) p[ldc] = fmaf(beta, old.y, alpha * s.y);
    if(c + 2 < N) p[2 * ldc] = fmaf(beta, old.z, alpha * s.z);
    if(c + 3 < N) p[3 * ldc] = fmaf(beta, old.w, alpha * s.w);
  };

  if(DUAL && diagonal) {
    asm volatile("bar.sync 1, %0;" ::"n"(kConsumers) : "memory");  // as before the exchange below
    constexpr int kPitch = kBN + 1;
    float* t = reinterpret_cast<float*>(smem);
#pragma unroll
    for(int f = 0; f < 16; ++f) {
      float* q = t + (row_of(f) - m0) * kPitch + col_of(f) - n0;
      q[0] = acc[f].x, q[1] = acc[f].y, q[2] = acc[f].z, q[3] = acc[f].w;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kConsumers) : "memory");
#pragma unroll
    for(int f = 0; f < 16; ++f) {
      const float* q = t + (col_of(f) - n0) * kPitch + row_of(f) - m0;
      acc[f].x += q[0], acc[f].y += q[kPitch], acc[f].z += q[2 * kPitch], acc[f].w += q[3 * kPitch];
    }
  }
  if(!TURN && splits > 1) {
    // every consumer warp has read its last stage, every copy has landed (each was waited for)
    asm volatile("bar.sync 1, %0;" ::"n"(kConsumers) : "memory");
    float4* mine = reinterpret_cast<float4*>(smem) + ctid;
#pragma unroll
    for(int f = 0; f < 16; ++f) mine[f * kConsumers] = acc[f];
    cluster_sync();
    // this CTA's quads: f0 .. f1 - 1 (two to eight), all their loads in flight together
    const int f0 = 16 * split / splits, f1 = 16 * (split + 1) / splits;
    float4 sum[8];
#pragma unroll
    for(int e = 0; e < 8; ++e) sum[e] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for(int c = 0; c < kMaxSplit; ++c) {
      if(c >= splits) break;
      const uint32_t theirs = cluster_map(mine, c) + f0 * kConsumers * 16;
      float4 v[8];
#pragma unroll
      for(int e = 0; e < 8; ++e)
        if(f0 + e < f1) v[e] = ld_cluster_f4(theirs + e * kConsumers * 16);
#pragma unroll
      for(int e = 0; e < 8; ++e)
        if(f0 + e < f1) sum[e].x += v[e].x, sum[e].y += v[e].y, sum[e].z += v[e].z, sum[e].w += v[e].w;
    }
    cluster_arrive();
#pragma unroll
    for(int t = 0; t < 2; ++t) {
      if(!ok || (t == 1 && !mirror)) continue;
      float4 old[8];
#pragma unroll
      for(int e = 0; e < 8; ++e)
        if(f0 + e < f1) old[e] = t ? load_t(f0 + e) : load_c(f0 + e);
#pragma unroll
      for(int e = 0; e < 8; ++e)
        if(f0 + e < f1) t ? store_t(f0 + e, sum[e], old[e]) : store_c(f0 + e, sum[e], old[e]);
    }
    __syncwarp();
    cluster_wait();  // no CTA leaves (or is left) while its sums are being read
    return;
  }
  if constexpr(TURN) {
    asm volatile("bar.sync 1, %0;" ::"n"(kConsumers) : "memory");  // the ring is drained, as before the exchange
    float* t = reinterpret_cast<float*>(smem) + cwarp * 32 * kTurnPitch;
#pragma unroll
    for(int f = 0; f < 16; ++f) {
      float* q = t + owned_row(li, f >> 1) * kTurnPitch + owned_col(lj, 4 * (f & 1));
      q[0] = acc[f].x, q[1] = acc[f].y, q[2] = acc[f].z, q[3] = acc[f].w;
    }
    __syncwarp();
    if(ok) write_turned(t, m0 + wr, n0 + wc, M, N, alpha, beta, C, ldc, mirror);
    return;
  }
  if(!ok) return;

  // --------------------------------------------------------------- epilogue
  // C = alpha * acc + beta * C, four rows at a time: the C values of a group
  // are loaded before the group's first store.  A load cannot move above a
  // store that may alias it, so interleaving them per element would serialise
  // one memory round trip per element.
#pragma unroll
  for(int t = 0; t < 2; ++t) {
    if(t == 1 && !mirror) break;
#pragma unroll
    for(int g = 0; g < 16; g += 8) {
      float4 old[8];
#pragma unroll
      for(int e = 0; e < 8; ++e) old[e] = t ? load_t(g + e) : load_c(g + e);
#pragma unroll
      for(int e = 0; e < 8; ++e) t ? store_t(g + e, acc[g + e], old[e]) : store_c(g + e, acc[g + e], old[e]);
    }
  }
}

template <Fetch FA, Fetch FB, bool DUAL, bool TURN = false>
struct Kernel {
  static constexpr int kStages = DUAL ? 3 : 4;
  static constexpr int kSmem = kStages * (DUAL ? 4 : 2) * kTileBytes + 1024 + 2 * kStages * 8;
  static constexpr auto fn = sgemm_kernel<FA, FB, DUAL, TURN, kStages>;

  // Once per device context: shared-memory opt-in and the register check of
  // the warp split (setmaxnreg draws on the registers of the launch).
  static gbpoly_status prepare(gbpoly_ctx* ctx) {
    static ContextMark prepared;
    if(prepared.valid(ctx->device)) return GBPOLY_OK;
    GBPOLY_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    cudaFuncAttributes fa;
    GBPOLY_CUDA_TRY(cudaFuncGetAttributes(&fa, fn));
    if(long(fa.numRegs) * kThreads < long(kProducers) * kRegsProducer + long(kConsumers) * kRegsConsumer)
      return fail(GBPOLY_ERR_UNSUPPORTED, "FP32 kernel built with too few registers for its warp split");
    prepared.set(ctx->device);
    return GBPOLY_OK;
  }

  struct Launch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    Launch(gbpoly_ctx* ctx, unsigned tiles, unsigned splits) {
      cfg.gridDim = dim3(tiles, splits);
      cfg.blockDim = dim3(kThreads);
      cfg.dynamicSmemBytes = kSmem;
      cfg.stream = ctx->stream;
      attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_pdl
      attr[0].val.programmaticStreamSerializationAllowed = 1;
      attr[1].id = cudaLaunchAttributeClusterDimension;
      attr[1].val.clusterDim.x = 1, attr[1].val.clusterDim.y = splits, attr[1].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = splits > 1 ? 2 : 1;
    }
  };
};

// Clusters of 1 x s CTAs to count on at once on the context's device (one CTA
// per SM in every variant of the kernel, so one query serves them all).  GB300
// reports 152, 76, 46, 36, 28, 23, 15 and 15.  Those of 2, 4 and 8 are reached
// (36 tiles as clusters of four in one round: syrk 1024 28.7 us); odd ones do
// not always pack so tightly, the less while the previous launch is ending, and
// one that finds no place takes a round of its own: 429 x 882 x 768, 28 tiles,
// 36.9 us as clusters of five, 22.8 of four; syrk 1536 118 us with 46 clusters
// of three in its first launch, 87 with two.  Hence a sixteenth less for these,
// though no fewer than of the next power of two.
gbpoly_status cluster_capacity(gbpoly_ctx* ctx, int (&cap)[kMaxSplit + 1]) {
  using K = Kernel<Fetch::Tma, Fetch::Tma, false>;
  static std::atomic<int> known_cap[32][kMaxSplit + 1];
  static ContextMark known;
  if(known.valid(ctx->device)) {
    for(int s = 1; s <= kMaxSplit; ++s) cap[s] = known_cap[ctx->device][s];
    return GBPOLY_OK;
  }
  gbpoly_status st = K::prepare(ctx);
  if(st != GBPOLY_OK) return st;
  cap[1] = std::max(1, ctx->sm_count);
  for(int s = 2; s <= kMaxSplit; ++s) {
    typename K::Launch l(ctx, unsigned(ctx->sm_count), unsigned(s));
    l.cfg.attrs = l.attr + 1, l.cfg.numAttrs = 1;  // the cluster size alone
    int n = 0;
    GBPOLY_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, K::fn, &l.cfg));
    cap[s] = n;  // 0: no cluster of this size
  }
  for(int s : {3, 5, 6, 7}) cap[s] = std::max(cap[s] * 15 / 16, cap[s < 4 ? 4 : 8]);
  if(ctx->device >= 0 && ctx->device < 32) {
    for(int s = 1; s <= kMaxSplit; ++s) known_cap[ctx->device][s] = cap[s];
    known.set(ctx->device);
  }
  return GBPOLY_OK;
}

// Time of `whole` tiles of u and then `half` of h on n places: the half ones on
// the places that the last round leaves free, however long these take, or on
// those until the round ends and then on all.
double span(int64_t whole, double u, int64_t half, double h, int n) {
  const int64_t busy = whole % n;
  const double begin = double(whole / n) * u, end = begin + (busy ? u : 0);
  if(half == 0) return end;
  const int64_t early = busy ? std::min<int64_t>(half, (n - busy) * int64_t(u / h)) : 0;
  const double beside = begin + double((half + n - busy - 1) / (n - busy)) * h;
  return std::min(std::max(end, beside), end + double((half - early + n - 1) / n) * h);
}

// Time of a launch of `tiles` tiles and, syr2k, `diagonal` ones of half the
// work, of `ktiles` k tiles each, split over clusters of s, in units of one k
// tile's products; negative where such a launch is not made.  Each CTA spends
// its share of the k tiles, a fixed part (launch, first copies, C) and, when
// split, the exchange of sums.
double split_time(const int (&cap)[kMaxSplit + 1], int64_t tiles, int64_t diagonal, int64_t ktiles, bool dual, int s) {
  if(cap[s] <= 0) return -1;
  const int64_t per = (ktiles + s - 1) / s;
  if(s > 1 && (s > ktiles || (ktiles + per - 1) / per != s)) return -1;  // an empty split
  const double unit = dual ? 2.0 : 1.0;                                   // syr2k: a k tile is two products
  const double fixed = kFixedTiles + (s > 1 ? kSplitTiles : 0);
  return span(tiles, unit * double(per) + fixed, diagonal, double(per) + fixed, cap[s]);
}

// The split that takes the least time.  Measured on GB300, all splits 1 to 8
// of eighteen shapes: within 4 % of the fastest (gemm 1024 47 us with 2
// against 59 with a workspace split and its reduction launch; syr2k 1536 132
// with 2 against 299 unsplit).
int best_split(const int (&cap)[kMaxSplit + 1], int64_t tiles, int64_t diagonal, int64_t ktiles, bool dual,
    double* time = nullptr) {
  int best = 1;
  double best_t = split_time(cap, tiles, diagonal, ktiles, dual, 1);
  for(int s = 2; s <= kMaxSplit; ++s) {
    const double t = split_time(cap, tiles, diagonal, ktiles, dual, s);
    if(t >= 0 && t < 0.97 * best_t) best = s, best_t = t;
  }
  if(time) *time = best_t;
  return best;
}

// Two launches for one contraction: the second one's time besides its CTAs',
// in k tiles' time, and the share of the single launch's time they have to beat.
constexpr double kSecondLaunch = 0.5, kWorth = 0.96;

// A contraction of a few rounds as two launches, by rows of tiles: the first
// one full rounds of clusters of one size, the rest split on its own.  The
// bits of an output depend on its row's split alone, so row panels give the
// whole call's.  1007 x 2632 x 400 66 -> 50 us, 1501 x 1023 x 2047 (72 tiles as
// pairs, 24 as clusters of five) 142 -> 130, 2048 cubed 320 -> 295; of 35
// shapes of 200 to 4000 twelve took two launches, ten of them 1.5 to 31 %
// faster, two 2 % slower.  Not beyond four rounds of CTAs, where the last one
// matters less and the search takes longer; nor up to 25 tiles, which one round
// of clusters of five or more holds.
void best_regions(const int (&cap)[kMaxSplit + 1], int64_t tm, int64_t tn, int64_t ktiles, Fp32Split& split) {
  double best;
  split = Fp32Split{0, 1, best_split(cap, tm * tn, 0, ktiles, false, &best)};
  if(tm * tn <= 25 || tm * tn > 4 * cap[1]) return;
  best *= kWorth;
  for(int s = 1; s <= kMaxSplit; ++s) {
    if(split_time(cap, 1, 0, ktiles, false, s) < 0) continue;
    for(int64_t rows, round = 1; (rows = round * cap[s] / tn) < tm; ++round) {
      if(rows == 0) continue;
      double rest;
      const int r = best_split(cap, (tm - rows) * tn, 0, ktiles, false, &rest);
      const double t = split_time(cap, rows * tn, 0, ktiles, false, s) + rest + kSecondLaunch;
      if(t < best) best = t, split = Fp32Split{rows * kBM, s, r};
    }
  }
}

// The same for syr2k, which launches the tiles below the diagonal and then the
// diagonal ones: `first` CTAs for each of the first `rows` tiles of that walk,
// `rest` for the others (2304 x 512 146 -> 115 us).
void dual_regions(const int (&cap)[kMaxSplit + 1], int64_t tm, int64_t ktiles, Fp32Split& split) {
  const int64_t below = tm * (tm - 1) / 2;
  double best;
  split = Fp32Split{0, 1, best_split(cap, below, tm, ktiles, true, &best)};
  if(below > 4 * cap[1]) return;
  best *= kWorth;
  for(int s = 1; s <= kMaxSplit; ++s) {
    if(split_time(cap, 1, 0, ktiles, true, s) < 0) continue;
    for(int64_t tiles = cap[s]; tiles < below; tiles += cap[s]) {
      double rest;
      const int r = best_split(cap, below - tiles, tm, ktiles, true, &rest);
      const double t = split_time(cap, tiles, 0, ktiles, true, s) + rest + kSecondLaunch;
      if(t < best) best = t, split = Fp32Split{tiles, s, r};
    }
  }
}

// One split for X X^T and for a product of the same shape and operand layout
// with another right operand, so that the triangle of tiles of the one gives
// the bits of the full square of the other (the result does not depend on
// whether the library sees that the operands are the same, and a host-buffer
// call, which has two copies, gives the device call's bits).  The two have
// different best splits, the triangle about half the tiles: the triangle's
// best one among those that cost the square at most 15 % (us with this rule /
// each on its own best plan, two launches among them: 1024 cubed N/T 52 / 45,
// its triangle 28.5 / 28.5; 1536 121 / 121, 125 / 87; 2304 446 / 407, 257 / 225;
// 3000 x 1000, triangle 182 / 182).
constexpr double kSquareMost = 1.15;

int square_split(const int (&cap)[kMaxSplit + 1], int64_t tm, int64_t ktiles) {
  const int64_t square = tm * tm, triangle = tm * (tm + 1) / 2;
  double most = split_time(cap, square, 0, ktiles, false, 1);
  for(int s = 2; s <= kMaxSplit; ++s) {
    const double t = split_time(cap, square, 0, ktiles, false, s);
    if(t >= 0) most = std::min(most, t);
  }
  most *= kSquareMost;
  int best = 0;
  double best_t = 0;
  for(int s = 1; s <= kMaxSplit; ++s) {
    const double full = split_time(cap, square, 0, ktiles, false, s);
    if(full < 0 || full > most) continue;
    const double t = split_time(cap, triangle, 0, ktiles, false, s);
    if(best == 0 || t < 0.97 * best_t) best = s, best_t = t;
  }
  return best;
}

// lower: symmetric product (op(A) == op(B)^T as stored, or syr2k), the lower
// triangle of tiles only; split.rows counts tiles of its walk then.  Others
// are one region: split.rest.
template <Fetch FA, Fetch FB, bool DUAL>
gbpoly_status launch_sgemm(gbpoly_ctx* ctx, const GemmF32Args& a, const Operand& oa, const Operand& ob, bool lower,
    const Fp32Split& split) {
  gbpoly_status st = GBPOLY_OK;
  const int64_t tm = (a.M + kBM - 1) / kBM, tn = (a.N + kBN - 1) / kBN, ktiles = (a.K + kBK - 1) / kBK;
  const int64_t tiles = lower ? tm * (tm + 1) / 2 : tm * tn;
  if(tiles >= (1ll << 31)) return fail(GBPOLY_ERR_UNSUPPORTED, "too many output tiles");
  CUtensorMap ta = {}, tb = {};
  auto map = [&](CUtensorMap* t, const Operand& o) {
    return make_tmap_2d(ctx, t, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, o.X, o.R, o.Cn, o.ld, kBK, 128,
        CU_TENSOR_MAP_SWIZZLE_NONE);
  };
  if(FA == Fetch::Tma && (st = map(&ta, oa)) != GBPOLY_OK) return st;
  if(FB == Fetch::Tma && (st = map(&tb, ob)) != GBPOLY_OK) return st;
  const bool turn = (reinterpret_cast<uintptr_t>(a.C) & 15) != 0 || (a.ldc & 3) != 0;
  auto launch = [&](auto kernel, int64_t t0, int64_t t1, int s) -> gbpoly_status {
    using Kn = decltype(kernel);
    if((st = Kn::prepare(ctx)) != GBPOLY_OK) return st;
    ProfileScope prof(ctx, DUAL ? "sgemm_simt_dual" : "sgemm_simt");
    typename Kn::Launch l(ctx, unsigned(t1 - t0), unsigned(s));
    GBPOLY_CUDA_TRY(cudaLaunchKernelEx(&l.cfg, Kn::fn, ta, tb, oa, ob, int(a.M), int(a.N), int(a.K), a.alpha, a.beta,
        a.C, a.ldc, lower ? 1 : 0, int(t0), int((ktiles + s - 1) / s), ctx->err_dev));
    return GBPOLY_OK;
  };
  for(int64_t t0 = 0; t0 < tiles;) {
    const bool first = t0 < split.rows;
    const int64_t t1 = first ? split.rows : tiles;
    const int s = first ? split.first : split.rest;
    st = turn && s == 1 ? launch(Kernel<FA, FB, DUAL, true>{}, t0, t1, s) : launch(Kernel<FA, FB, DUAL>{}, t0, t1, s);
    if(st != GBPOLY_OK) return st;
    t0 = t1;
  }
  return GBPOLY_OK;
}

template <Fetch FA>
gbpoly_status launch_left(gbpoly_ctx* ctx, const GemmF32Args& a, const Operand& oa, const Operand& ob, Fetch fb,
    bool lower, int splits) {
  const Fp32Split split{0, 1, splits};
  switch(fb) {
  case Fetch::Tma: return launch_sgemm<FA, Fetch::Tma, false>(ctx, a, oa, ob, lower, split);
  case Fetch::Rows: return launch_sgemm<FA, Fetch::Rows, false>(ctx, a, oa, ob, lower, split);
  default: return launch_sgemm<FA, Fetch::Turn, false>(ctx, a, oa, ob, lower, split);
  }
}

// A K-major operand is turned on its way; an MN-major one goes by TMA where
// its base and rows are 16-byte aligned (and it is not empty).
Fetch fetch_of(const Operand& o, bool k_major) {
  if(k_major) return Fetch::Turn;
  return (reinterpret_cast<uintptr_t>(o.X) & 15) == 0 && (o.ld & 3) == 0 && o.R > 0 ? Fetch::Tma : Fetch::Rows;
}

// ---------------------------------------------------------------- short K, any strides
// 64 x 64 of C per CTA of 256 threads, 4 x 4 per thread, 16 of K at a time
// through shared memory: any strides, 64-bit indexes, 64 registers and 8 KB, so
// that four CTAs of an SM hide one another's start, copies and C.  The same
// order of K and the same bits as an unsplit sgemm_kernel.
struct Strided {  // op(X)[r][k] = p[r * s_r + k * s_k]
  const float* p;
  int64_t s_r, s_k;
};
constexpr int kT64 = 64, kT64K = 16;

__global__ void __launch_bounds__(256) sgemm_tile64_kernel(int64_t M, int64_t N, int64_t K, float alpha, Strided a,
    Strided b, bool dual, Strided a2, Strided b2, float beta, float* __restrict__ C, int64_t ldc, bool lower) {
  __shared__ float As[kT64K][kT64 + 1];
  __shared__ float Bs[kT64K][kT64 + 1];
  pdl_wait();
  if(lower && blockIdx.x > blockIdx.y) return;  // strictly above the diagonal: the mirror of another tile
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int64_t m0 = static_cast<int64_t>(blockIdx.y) * kT64, n0 = static_cast<int64_t>(blockIdx.x) * kT64;
  float acc[4][4];
#pragma unroll
  for(int i = 0; i < 4; ++i)
#pragma unroll
    for(int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  const int passes = dual ? 2 : 1;
  for(int p = 0; p < passes; ++p) {
    const Strided oa = p ? a2 : a;
    const Strided ob = p ? b2 : b;
    for(int64_t k0 = 0; k0 < K; k0 += kT64K) {
#pragma unroll
      for(int e = 0; e < 4; ++e) {
        const int idx = tid + e * 256;
        // rows fastest when the operand is contiguous along rows, else k fastest
        const int r = (oa.s_r == 1) ? (idx & 63) : (idx >> 4);
        const int kk = (oa.s_r == 1) ? (idx >> 6) : (idx & 15);
        const int64_t gm = m0 + r, gk = k0 + kk;
        As[kk][r] = (gm < M && gk < K) ? oa.p[gm * oa.s_r + gk * oa.s_k] : 0.f;
        const int rb = (ob.s_r == 1) ? (idx & 63) : (idx >> 4);
        const int kb = (ob.s_r == 1) ? (idx >> 6) : (idx & 15);
        const int64_t gn = n0 + rb, gkb = k0 + kb;
        Bs[kb][rb] = (gn < N && gkb < K) ? ob.p[gn * ob.s_r + gkb * ob.s_k] : 0.f;
      }
      __syncthreads();
#pragma unroll
      for(int kk = 0; kk < kT64K; ++kk)
#pragma unroll
        for(int i = 0; i < 4; ++i)
#pragma unroll
          for(int j = 0; j < 4; ++j) acc[i][j] = fmaf(As[kk][ty * 4 + i], Bs[kk][tx + 16 * j], acc[i][j]);
      __syncthreads();
    }
  }
  // C values are loaded before the first store (a load cannot move above a
  // store that may alias it)
  float cv[4][4];
#pragma unroll
  for(int i = 0; i < 4; ++i)
#pragma unroll
    for(int j = 0; j < 4; ++j) {
      const int64_t m = m0 + ty * 4 + i, n = n0 + tx + 16 * j;
      cv[i][j] = (beta != 0.f && m < M && n < N) ? C[m * ldc + n] : 0.f;
    }
#pragma unroll
  for(int i = 0; i < 4; ++i) {
    const int64_t m = m0 + ty * 4 + i;
    if(m >= M) continue;
#pragma unroll
    for(int j = 0; j < 4; ++j) {
      const int64_t n = n0 + tx + 16 * j;
      if(n < N) C[m * ldc + n] = fmaf(beta, cv[i][j], alpha * acc[i][j]);
    }
  }
  if(lower && blockIdx.x < blockIdx.y) {  // the transposed tile, C[n][m]
#pragma unroll
    for(int i = 0; i < 4; ++i)
#pragma unroll
      for(int j = 0; j < 4; ++j) {
        const int64_t m = m0 + ty * 4 + i, n = n0 + tx + 16 * j;
        cv[i][j] = (beta != 0.f && m < M && n < N) ? C[n * ldc + m] : 0.f;
      }
#pragma unroll
    for(int i = 0; i < 4; ++i) {
      const int64_t m = m0 + ty * 4 + i;
      if(m >= M) continue;
#pragma unroll
      for(int j = 0; j < 4; ++j) {
        const int64_t n = n0 + tx + 16 * j;
        if(n < N) C[n * ldc + m] = fmaf(beta, cv[i][j], alpha * acc[i][j]);
      }
    }
  }
}

gbpoly_status launch_tile64(gbpoly_ctx* ctx, const GemmF32Args& a, bool lower) {
  const int64_t gx = (a.N + kT64 - 1) / kT64, gy = (a.M + kT64 - 1) / kT64;
  if(gy > 65535) return fail(GBPOLY_ERR_UNSUPPORTED, "matrix too tall for the 64 x 64 kernel's grid");
  const Strided oa = a.op_a == GBPOLY_OP_N ? Strided{a.A, a.lda, 1} : Strided{a.A, 1, a.lda};
  const Strided ob = a.op_b == GBPOLY_OP_T ? Strided{a.B, a.ldb, 1} : Strided{a.B, 1, a.ldb};
  ProfileScope prof(ctx, "sgemm_tiled");
  GBPOLY_CUDA_TRY(launch_pdl(ctx, sgemm_tile64_kernel, dim3(unsigned(gx), unsigned(gy)), 256, 0, a.M, a.N, a.K, a.alpha,
      oa, ob, a.dual, Strided{a.A2, a.lda2, 1}, Strided{a.B2, a.ldb2, 1}, a.beta, a.C, a.ldc, lower));
  return GBPOLY_OK;
}

bool aligned16(const GemmF32Args& a) {
  return ((reinterpret_cast<uintptr_t>(a.A) | reinterpret_cast<uintptr_t>(a.B)) & 15) == 0 && ((a.lda | a.ldb) & 3) == 0 &&
         a.K > 0;
}

// Which calls take 64 x 64 tiles: those beyond the other kernel's 32-bit
// coordinates, and short K on operands off 16-byte boundaries, where the big
// kernel's start with 200 KB of shared memory and its word copies cost more
// than the products: the fewer tiles, the longer K may be, and for all outputs
// up to K = 16 (us, 128 x 128 / 64 x 64, odd rows: 300 x 300 K = 16 6.9 / 3.2,
// 500 x 500 K = 32 7.9 / 4.4, 64 9.5 / 6.8; 1000 x 1000 K = 48 9.9 / 8.0, 64 10.0 /
// 9.8; 2000 x 2000 K = 16 15.2 / 10.8, 32 15.6 / 16.6; 8192 x 8192 K = 16 164 / 132).
// A mirrored tile is cheaper in the big kernel, which turns it in shared memory
// (2000 x 2000 symmetric K = 16 13.9 / 20.5; syr2k 500 x 32 16.9 / 9.3, 2000 x 32
// 17.4 / 25.7).
bool use_tile64(gbpoly_ctx* ctx, const GemmF32Args& a) {
  if(a.M >= (1ll << 31) || a.N >= (1ll << 31) || a.K >= (1ll << 31)) return true;
  if(aligned16(a) || a.K > 80 || (a.M + kT64 - 1) / kT64 > 65535) return false;
  const int64_t tiles = ((a.M + kBM - 1) / kBM) * ((a.N + kBN - 1) / kBN), sms = std::max(1, ctx->sm_count);
  if(a.dual) return tiles <= (a.K <= 32 ? sms : (a.K <= 64 ? 16 : 0));
  if(a.K <= 32) return symmetric_operand(a) ? tiles <= sms : (a.K <= 16 || 2 * tiles <= 3 * sms);
  return tiles <= (a.K <= 48 ? sms : (a.K <= 64 ? 32 : 16));
}

}  // namespace

gbpoly_status fp32_split(gbpoly_ctx* ctx, const GemmF32Args& a, Fp32Split& split) {
  split = Fp32Split{0, 1, 1, use_tile64(ctx, a)};
  if(split.tile64) return GBPOLY_OK;
  int cap[kMaxSplit + 1] = {};
  gbpoly_status st = cluster_capacity(ctx, cap);
  if(st != GBPOLY_OK) return st;
  const int64_t tm = (a.M + kBM - 1) / kBM, tn = (a.N + kBN - 1) / kBN, ktiles = (a.K + kBK - 1) / kBK;
  if(a.dual)
    dual_regions(cap, tm, ktiles, split);
  else if(a.M == a.N && a.op_a != a.op_b)
    split.rest = square_split(cap, tm, ktiles);
  else
    best_regions(cap, tm, tn, ktiles, split);
  return GBPOLY_OK;
}

size_t fp32_split_k_bytes(int sm_count, int64_t M, int64_t N, int64_t K) {
  const int64_t tiles = ((M + kBM - 1) / kBM) * ((N + kBN - 1) / kBN), ktiles = (K + kBK - 1) / kBK;
  if(tiles <= 0 || tiles * 2 > sm_count || ktiles < 8) return 0;
  const int64_t s = std::min<int64_t>(std::min<int64_t>(sm_count / tiles, ktiles / 4), 8);
  if(s <= 1) return 0;
  const int64_t per = (ktiles + s - 1) / s;
  return size_t((ktiles + per - 1) / per) * size_t(M) * size_t(N) * sizeof(float);
}

gbpoly_status launch_gemm_f32_simt(gbpoly_ctx* ctx, const GemmF32Args& a) {
  if(a.M == 0 || a.N == 0) return GBPOLY_OK;
  const bool a_kmaj = a.op_a == GBPOLY_OP_N;
  const bool b_kmaj = a.op_b == GBPOLY_OP_T;
  const bool symmetric = a.M == a.N && (a.dual || symmetric_operand(a));
  Fp32Split split = a.split;
  gbpoly_status st = GBPOLY_OK;
  if(split.rest == 0 && (st = fp32_split(ctx, a, split)) != GBPOLY_OK) return st;
  if(split.tile64) return launch_tile64(ctx, a, symmetric);

  // op(A) is M x K.  Stored as M x K (K-major) for op N, K x M for op T;
  // op(B) is K x N.  Stored as K x N for op N, N x K (K-major) for op T.
  const int M = int(a.M), N = int(a.N), K = int(a.K);
  const Operand oa = a_kmaj ? Operand{a.A, a.lda, M, K} : Operand{a.A, a.lda, K, M};
  const Operand ob = b_kmaj ? Operand{a.B, a.ldb, N, K} : Operand{a.B, a.ldb, K, N};
  if(!aligned16(a) && (a.M + 63) / 64 > 65535)
    return fail(GBPOLY_ERR_UNSUPPORTED, "matrix too tall for operands off 16-byte boundaries");
  if(a.dual) return launch_sgemm<Fetch::Turn, Fetch::Turn, true>(ctx, a, oa, ob, true, split);
  const Fetch fb = fetch_of(ob, b_kmaj);
  auto launch = [&](const GemmF32Args& part, const Operand& left, int splits) {
    switch(fetch_of(left, a_kmaj)) {
    case Fetch::Tma: return launch_left<Fetch::Tma>(ctx, part, left, ob, fb, symmetric, splits);
    case Fetch::Rows: return launch_left<Fetch::Rows>(ctx, part, left, ob, fb, symmetric, splits);
    default: return launch_left<Fetch::Turn>(ctx, part, left, ob, fb, symmetric, splits);
    }
  };
  const int m1 = int(std::clamp<int64_t>(split.rows - a.split_row, 0, a.M));  // rows of the first region
  if(m1 == M) return launch(a, oa, split.first);
  if(m1 == 0) return launch(a, oa, split.rest);
  GemmF32Args top = a, below = a;
  top.M = m1, below.M = M - m1;
  below.C += m1 * a.ldc;
  const Operand left_top = a_kmaj ? Operand{a.A, a.lda, m1, K} : Operand{a.A, a.lda, K, m1};
  const Operand left_below =
      a_kmaj ? Operand{a.A + m1 * a.lda, a.lda, M - m1, K} : Operand{a.A + m1, a.lda, K, M - m1};
  if((st = launch(top, left_top, split.first)) != GBPOLY_OK) return st;
  return launch(below, left_below, split.rest);
}

}  // namespace gbpoly
