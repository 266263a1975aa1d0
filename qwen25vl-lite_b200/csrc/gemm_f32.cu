// C[M,N] = A[M,K] . W[N,K]^T (+ bias[N]) in true 32-bit.  This is the matrix product of the 32-bit path
// (the reference's tested path is float32 end to end, src/qwen25vl_lite/engine.py:63).  Where K is 256 or more and a multiple of
// 32, and W's rows are aligned to 16 bytes, it runs on tensor cores, every number in three exact parts (gemm_f32x3.cu); this file has the
// others, plain FMA on the CUDA cores.  (Figures of longer K below are from when these kernels took it.  The line lies at 256 because there the
// two are even for one row and tensor cores ahead for more: 1 / 8 / 16 / 17 / 1,024 rows of 320 features, K 256, by FMA 2.2 / 3.4 / 3.6 / 5.4 / 11.5 us, there
// 2.3 / 2.5 / 3.3 / 3.3 / 7.6; of 4,096 features 2.7 / 4.1 / 4.4 / 5.7 / 52 and 3.6 / 4.1 / 4.6 / 6.2 / 17.)
//
// Every output element is summed in one order, which all kernels of this file share: K is cut into
// segments of 128; inside a segment the even and the odd k are one chain of fma each, in order,
// and the segment's value is even + odd; the segments' values are added in order; then + bias.
// The order depends on nothing but K, so a token's result is bit-identical whether it is computed
// alone, in a portion or in a large batch.  (Two chains, because the packed fma.rn.f32x2 takes
// (k, k + 1) of both operands as they lie in memory; segments, because the warps of a CTA and the
// lanes of a warp can then work on different parts of K; and many short chains err less than one
// long one.)
//
//   * up to 16 rows (decode steps), K and the row pitches multiples of 32: gemm_f32_rows_kernel, a stream of the weights;
//   * more rows: gemm_f32_tile_kernel or gemm_f32_split_kernel, bound by the FMA pipes;
//   * operands TMA refuses (K or a row pitch not a multiple of 4, an unaligned base), and few rows with few steps of K:
//     gemm_f32_kernel, plain loads.
#include "common.cuh"
#include "f32x2.cuh"
#include "gemm_f32x3.cuh"
#include "tensor_map.cuh"

#define GF_SEG 128                               // k of one segment

// ---- plain loads ----------------------------------------------------------------------------------------------------
template <int BM, int BN, int BK, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc) {
  pdl_trigger();
  pdl_wait();
  constexpr int THREADS = (BM / TM) * (BN / TN);
  static_assert(GF_SEG % BK == 0 && BK % 2 == 0, "a segment ends with a tile of K");
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tx = threadIdx.x % (BN / TN), ty = threadIdx.x / (BN / TN);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[2][TM][TN], total[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[0][i][j] = acc[1][i][j] = total[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    for (int e = threadIdx.x; e < BM * BK; e += THREADS) {
      const int r = e / BK, c = e % BK;
      const int gm = m0 + r, gk = k0 + c;
      As[c][r] = (gm < M && gk < K) ? A[(size_t)gm * lda + gk] : 0.f;
    }
    for (int e = threadIdx.x; e < BN * BK; e += THREADS) {
      const int r = e / BK, c = e % BK;
      const int gn = n0 + r, gk = k0 + c;
      Ws[c][r] = (gn < N && gk < K) ? W[(size_t)gn * ldw + gk] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = Ws[kk][tx * TN + j];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[kk & 1][i][j] = fmaf(a[i], w[j], acc[kk & 1][i][j]);
    }
    __syncthreads();
    if ((k0 + BK) % GF_SEG == 0 || k0 + BK >= K) {
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          total[i][j] += acc[0][i][j] + acc[1][i][j];
          acc[0][i][j] = acc[1][i][j] = 0.f;
        }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + ty * TM + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx * TN + j;
      if (gn < N) C[(size_t)gm * ldc + gn] = total[i][j] + (bias ? bias[gn] : 0.f);
    }
  }
}

// ---- up to 16 rows: a stream of the weights -------------------------------------------------------------------------
// One persistent CTA per SM; its items are groups of 16 features over all of K (below 256, as longer K runs in gemm_f32x3.cu), one stage of the
// ring each, which two copies fill: a box of 16 rows of W and one of the rows of x.  (The copy engine takes a request about every
// 90 cycles whatever its size.)  K is seen as blocks of 32, and a row of W's box holds 9 of them, the last one not used: with an odd number of
// 128-byte blocks a row, the 128-byte swizzle puts the same block of eight rows into eight different bank groups.  A warp takes the
// items of one stage: lane = (pair of features p and p + 8, segment), so that 16 bytes of x serve two features (the lanes beyond the two
// segments of K idle), and leaves the segments' values in shared memory, where the last warp adds them in order.  The producer
// starts the weights before it waits for the kernel before (early).  MT: rows of a lane; MG: warps that share a stage (rows 0 .. MT - 1
// and MT ..).
#define GR_ROWS 16
#define GR_K 256                                 // k of a stage
#define GR_PITCH (9 * 128)                       // bytes between the rows of W in a stage
#define GR_W_BYTES (GR_ROWS * GR_PITCH)

template <int MT, int MG> struct RowsShape {
  static constexpr int MP = MT * MG;
  static constexpr int STAGE = GR_W_BYTES + MP * GR_K * 4;
  static constexpr int STAGES = MP <= 4 ? 5 : MP == 8 ? 4 : 3;
  static constexpr int RED = GR_K / GF_SEG * GR_ROWS * MP;      // floats of one slot of segment values
  static constexpr int WARPS = STAGES * MG;
  static constexpr int THREADS = (WARPS + 2) * 32;
  static constexpr int SMEM = 1024 + STAGES * (STAGE + RED * 4) + STAGES * 4 * 8;
};

template <int MT, int MG>
__global__ void __launch_bounds__(RowsShape<MT, MG>::THREADS, 1)
gemm_f32_rows_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                     const float* __restrict__ bias, float* __restrict__ C, int M, int N, int K, int ldc, bool early, int* err) {
  using Shape = RowsShape<MT, MG>;
  constexpr int MP = Shape::MP, S = Shape::STAGES;
  extern __shared__ unsigned char gr_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)gr_raw + 1023) & ~(uintptr_t)1023);
  float* red = reinterpret_cast<float*>(smem + S * Shape::STAGE);
  unsigned long long* full = reinterpret_cast<unsigned long long*>(red + S * Shape::RED);
  unsigned long long* empty = full + S;
  unsigned long long* red_full = empty + S;
  unsigned long long* red_empty = red_full + S;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = (N + GR_ROWS - 1) / GR_ROWS, items = (groups - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, MG);
      mbar_init(red_full + s, MG);
      mbar_init(red_empty + s, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  pdl_trigger();

  if (warp == Shape::WARPS) {
    // ---- producer ----
    if (lane == 0) {
      const unsigned long long once = l2_evict_first();
      bool ok = true;
      auto weights = [&](int item) {
        const int s = item % S, g = (int)blockIdx.x + item * (int)gridDim.x;
        mbar_expect_tx(full + s, Shape::STAGE);
        tma_3d_once(smem_u32(smem + s * Shape::STAGE), &map_w, 0, 0, g * GR_ROWS, full + s, once);
      };
      auto rows = [&](int item) {
        const int s = item % S;
        tma_3d(smem_u32(smem + s * Shape::STAGE) + GR_W_BYTES, &map_x, 0, 0, 0, full + s);
      };
      const int ahead = min(S, items);
      if (!early) pdl_wait();
      for (int i = 0; i < ahead; ++i) weights(i);
      pdl_wait();
      for (int i = 0; i < ahead; ++i) rows(i);
      for (int i = ahead; i < items; ++i) {
        if (ok) {
          ok = mbar_wait(empty + i % S, (unsigned)(i / S - 1) & 1);
          if (!ok) { atomicExch(err, 41); break; }               // nobody reads what was not asked for: the readers give up too
        }
        weights(i);
        rows(i);
      }
    }
    return;
  }
  if (warp == Shape::WARPS + 1) {
    // ---- the segments' values, added in order ----
    constexpr int V = (GR_ROWS * MP + 31) / 32;
    pdl_wait();                                                  // the kernel before may still read what this one overwrites
    bool ok = true;
    for (int i = 0; i < items; ++i) {
      const int s = i % S;
      float total[V];
#pragma unroll
      for (int v = 0; v < V; ++v) total[v] = 0.f;
      if (ok) {
        ok = mbar_wait(red_full + s, (unsigned)(i / S) & 1);
        if (!ok && lane == 0) atomicExch(err, 42);
      }
      const float* slot = red + s * Shape::RED;
#pragma unroll
      for (int q = 0; q < GR_K / GF_SEG; ++q)
#pragma unroll
        for (int v = 0; v < V; ++v)
          if (V * 32 == GR_ROWS * MP || lane < GR_ROWS * MP) total[v] += slot[q * (GR_ROWS * MP) + v * 32 + lane];
      __syncwarp();
      if (lane == 0) mbar_arrive(red_empty + s);
      const int n = ((int)blockIdx.x + i * (int)gridDim.x) * GR_ROWS + (lane & 15);
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const int m = v * 2 + (lane >> 4);
        if (m < M && n < N) C[(size_t)m * ldc + n] = total[v] + (bias ? bias[n] : 0.f);
      }
    }
    return;
  }

  // ---- one warp, one stage ----
  const int s = warp / MG, mg = warp % MG, p = lane & 7, seg = lane >> 3;
  bool ok = true;
  unsigned parity = 0;
  const unsigned wa = smem_u32(smem + s * Shape::STAGE) + p * GR_PITCH + seg * 512;
  const unsigned xa = smem_u32(smem + s * Shape::STAGE) + GR_W_BYTES + mg * MT * (GR_K * 4) + seg * 512;
  for (int i = s; i < items; i += S, parity ^= 1) {
    const int blocks = min(4, (K - seg * GF_SEG + 31) / 32);      // may be <= 0
    f32x2 acc[2][MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[0][m] = acc[1][m] = 0;
    if (ok) {
      ok = mbar_wait(full + s, parity);
      if (!ok && lane == 0) atomicExch(err, 43);
    }
    for (int b = 0; b < blocks; ++b) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const unsigned at = wa + b * 128 + ((c ^ ((p + seg * 4 + b) & 7)) << 4);
        const ulonglong2 w0 = lds_pair(at), w1 = lds_pair(at + 8 * GR_PITCH);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const ulonglong2 x = lds_pair(xa + m * (GR_K * 4) + b * 128 + c * 16);
          acc[0][m] = fma2(w0.x, x.x, acc[0][m]);
          acc[1][m] = fma2(w1.x, x.x, acc[1][m]);
          acc[0][m] = fma2(w0.y, x.y, acc[0][m]);
          acc[1][m] = fma2(w1.y, x.y, acc[1][m]);
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + s);
    if (i >= S && ok) {
      ok = mbar_wait(red_empty + s, parity ^ 1);
      if (!ok && lane == 0) atomicExch(err, 44);
    }
    float* slot = red + s * Shape::RED + seg * (GR_ROWS * MP) + mg * (MT * GR_ROWS) + p;
    if (seg < GR_K / GF_SEG) {
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        slot[m * GR_ROWS] = sum2(acc[0][m]);
        slot[m * GR_ROWS + 8] = sum2(acc[1][m]);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(red_full + s);
  }
}

// ---- more rows: tiles -----------------------------------------------------------------------------------------------
// A thread computes 8 x 4 outputs (rows m = ty + 4 i, features n = tx + 8 j of its warp's 32 x 32), both chains of each in
// one 64-bit register pair; twelve 16-byte reads of shared memory feed 64 packed FMAs.  Tiles of 32 k travel by TMA into a
// ring of four stages, in the 128-byte swizzle, in which the rows a warp reads together lie in different banks.
#define GT_BK 32
#define GT_STAGES 4

// 32 k of a warp's 32 x 32 outputs: rows of A at a0, rows of W at w0 (shared addresses of 128-byte rows, swizzled).
__device__ __forceinline__ void f32_tile_fma(unsigned a0, unsigned w0, int tx, int ty, f32x2 (&acc)[8][4]) {
  a0 += ty * 128;
  w0 += tx * 128;
#pragma unroll
  for (int c = 0; c < GT_BK / 4; ++c) {
    ulonglong2 a[8], w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = lds_pair(w0 + j * (8 * 128) + ((c ^ tx) << 4));
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = lds_pair(a0 + i * (4 * 128) + ((c ^ (ty + 4 * (i & 1))) << 4));
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fma2(a[i].x, w[j].x, acc[i][j]);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fma2(a[i].y, w[j].y, acc[i][j]);
  }
}

template <int WM, int WN, int CTAS>
__global__ void __launch_bounds__(WM * WN * 32, CTAS)
gemm_f32_tile_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                     const float* __restrict__ bias, float* __restrict__ C, int M, int N, int K, int ldc, bool early, int* err) {
  constexpr int BM = WM * 32, BN = WN * 32, STAGE = (BM + BN) * 128;
  extern __shared__ unsigned char gt_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)gt_raw + 1023) & ~(uintptr_t)1023);
  unsigned long long* full = reinterpret_cast<unsigned long long*>(smem + GT_STAGES * STAGE);
  unsigned long long* empty = full + GT_STAGES;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int nk = (K + GT_BK - 1) / GT_BK;
  if (threadIdx.x == 0) {
    for (int s = 0; s < GT_STAGES; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, WM * WN);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  pdl_trigger();
  auto load_w = [&](int t) {
    const int s = t % GT_STAGES;
    mbar_expect_tx(full + s, STAGE);
    tma_2d(smem_u32(smem + s * STAGE) + BM * 128, &map_w, t * GT_BK, n0, full + s);
  };
  auto load_a = [&](int t) {
    const int s = t % GT_STAGES;
    tma_2d(smem_u32(smem + s * STAGE), &map_a, t * GT_BK, m0, full + s);
  };
  const int ahead = min(GT_STAGES - 1, nk);
  if (!early) pdl_wait();
  if (threadIdx.x == 0)
    for (int t = 0; t < ahead; ++t) load_w(t);
  pdl_wait();
  if (threadIdx.x == 0)
    for (int t = 0; t < ahead; ++t) load_a(t);

  const int tx = lane & 7, ty = lane >> 3;
  const int wm = warp % WM, wn = warp / WM;
  f32x2 acc[8][4];
  float total[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) { acc[i][j] = 0; total[i][j] = 0.f; }
  bool ok = true;
  for (int t = 0; t < nk; ++t) {
    const int s = t % GT_STAGES;
    if (ok) {
      ok = mbar_wait(full + s, (unsigned)(t / GT_STAGES) & 1);
      if (!ok && lane == 0) atomicExch(err, 45);
    }
    f32_tile_fma(smem_u32(smem + s * STAGE) + wm * (32 * 128), smem_u32(smem + s * STAGE) + (BM + wn * 32) * 128, tx, ty, acc);
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + s);
    // the stage that every warp left a tile ago takes the tile three ahead
    if (threadIdx.x == 0 && t + GT_STAGES - 1 < nk) {
      const int next = t + GT_STAGES - 1;
      if (next >= GT_STAGES && ok) {
        ok = mbar_wait(empty + next % GT_STAGES, (unsigned)(next / GT_STAGES - 1) & 1);
        if (!ok) atomicExch(err, 46);
      }
      if (ok) {
        load_w(next);
        load_a(next);
      }
    }
    __syncwarp();
    if ((t + 1) % (GF_SEG / GT_BK) == 0 || t + 1 == nk) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          total[i][j] += sum2(acc[i][j]);
          acc[i][j] = 0;
        }
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int n = n0 + wn * 32 + tx + 8 * j;
    if (n >= N) continue;
    const float b = bias ? bias[n] : 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = m0 + wm * 32 + ty + 4 * i;
      if (m < M) C[(size_t)m * ldc + n] = total[i][j] + b;
    }
  }
}

// ---- few tiles: the warps of a CTA side by side in K ----------------------------------------------------------------
// The inner loop of gemm_f32_tile_kernel on a 32 x 32 tile, whose four warps take every fourth segment of K each, through
// a ring of their own; after each round of four segments their values meet in shared memory and are added in order.
// Where tiles of 64 x 64 leave SMs without work (64 rows x 2,048 features: 32 tiles) this has four times as many CTAs.
// One CTA of an SM has four stages for each warp; two have two, which is as fast (a warp's tile takes longer than a trip to
// memory) and leaves room for both.
#define GS_WARPS 4
#define GS_SMEM(stages) (1024 + GS_WARPS * (stages) * 64 * 128 + GS_WARPS * 32 * 32 * 4 + GS_WARPS * (stages) * 16)

__global__ void __launch_bounds__(GS_WARPS * 32, 2)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                      const float* __restrict__ bias, float* __restrict__ C, int M, int N, int K, int ldc, int stages, bool early,
                      int* err) {
  constexpr int STAGE = 64 * 128;
  extern __shared__ unsigned char gs_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)gs_raw + 1023) & ~(uintptr_t)1023);
  float* red = reinterpret_cast<float*>(smem + GS_WARPS * stages * STAGE);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned long long* full = reinterpret_cast<unsigned long long*>(red + GS_WARPS * 32 * 32) + warp * 2 * stages;
  unsigned long long* empty = full + stages;
  unsigned char* ring = smem + warp * (stages * STAGE);
  const int m0 = blockIdx.x * 32, n0 = blockIdx.y * 32;
  if (lane == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncwarp();
  pdl_trigger();
  // this warp's tiles of 32 k, in order: tile t is tile t mod 4 of its segment t / 4
  constexpr int per = GF_SEG / GT_BK;
  const int nt = (K + GT_BK - 1) / GT_BK;
  const int rounds = (nt + GS_WARPS * per - 1) / (GS_WARPS * per);
  const int last = nt - ((rounds - 1) * GS_WARPS + warp) * per;                    // tiles of its last segment, if any
  const int tiles = (rounds - 1) * per + max(0, min(per, last));
  auto k_of = [&](int t) { return ((t / per * GS_WARPS + warp) * per + t % per) * GT_BK; };
  auto load_w = [&](int t, int s) {
    mbar_expect_tx(full + s, STAGE);
    tma_2d(smem_u32(ring + s * STAGE) + 32 * 128, &map_w, k_of(t), n0, full + s);
  };
  auto load_a = [&](int t, int s) { tma_2d(smem_u32(ring + s * STAGE), &map_a, k_of(t), m0, full + s); };
  const int ahead = min(stages - 1, tiles);
  if (!early) pdl_wait();
  if (lane == 0)
    for (int t = 0; t < ahead; ++t) load_w(t, t);
  pdl_wait();
  if (lane == 0)
    for (int t = 0; t < ahead; ++t) load_a(t, t);
  __syncwarp();

  const int tx = lane & 7, ty = lane >> 3;
  float total[8];
#pragma unroll
  for (int v = 0; v < 8; ++v) total[v] = 0.f;
  bool ok = true;
  int s = 0;
  unsigned parity = 0;                           // of the stage that is read next; the one filled next is a stage behind
  for (int r = 0, t = 0; r < rounds; ++r) {
    f32x2 acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    for (const int end = min(tiles, (r + 1) * per); t < end; ++t) {
      if (ok) {
        ok = mbar_wait(full + s, parity);
        if (!ok && lane == 0) atomicExch(err, 47);
      }
      if (lane == 0 && t + stages - 1 < tiles) {
        // into the stage of the tile before this one, which the warp has left
        const int f = s == 0 ? stages - 1 : s - 1;
        if (t >= 1 && ok) {
          ok = mbar_wait(empty + f, s == 0 ? parity ^ 1 : parity);
          if (!ok) atomicExch(err, 48);
        }
        if (ok) {
          load_w(t + stages - 1, f);
          load_a(t + stages - 1, f);
        }
      }
      __syncwarp();
      f32_tile_fma(smem_u32(ring + s * STAGE), smem_u32(ring + s * STAGE) + 32 * 128, tx, ty, acc);
      __syncwarp();
      if (lane == 0) mbar_arrive(empty + s);
      if (++s == stages) { s = 0; parity ^= 1; }
    }
    // row m's column n of a warp's values lies at n ^ 8 (m mod 4): the four rows a warp stores lie in different banks
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) red[(warp * 32 + ty + 4 * i) * 32 + tx + 8 * (j ^ ty)] = sum2(acc[i][j]);
    __syncthreads();
#pragma unroll
    for (int v = 0; v < 8; ++v)
#pragma unroll
      for (int w = 0; w < GS_WARPS; ++w) total[v] += red[(w * 32 + warp + 4 * v) * 32 + (lane ^ (8 * warp))];
    __syncthreads();
  }
  const int n = n0 + lane;
  if (n >= N) return;
  const float b = bias ? bias[n] : 0.f;
#pragma unroll
  for (int v = 0; v < 8; ++v) {
    const int m = m0 + warp + 4 * v;
    if (m < M) C[(size_t)m * ldc + n] = total[v] + b;
  }
}

// ---- host -----------------------------------------------------------------------------------------------------------
template <int MT, int MG>
static int launch_rows(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                       bool early, int* err, cudaStream_t s) {
  using Shape = RowsShape<MT, MG>;
  CUtensorMap mx, mw;
  if (!make_blocks_f32(&mx, A, M, K, lda, Shape::MP, GR_K / 32, false) || !make_blocks_f32(&mw, W, N, K, ldw, GR_ROWS, GR_K / 32 + 1, true)) return (int)cudaErrorInvalidValue;
  const cudaError_t e = cudaFuncSetAttribute(gemm_f32_rows_kernel<MT, MG>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::SMEM);
  if (e != cudaSuccess) return (int)e;
  const int sms = device_sm_count(), groups = (N + GR_ROWS - 1) / GR_ROWS;
  if (sms <= 0) return (int)cudaErrorInvalidDevice;
  launch(gemm_f32_rows_kernel<MT, MG>, dim3(groups < sms ? groups : sms), dim3(Shape::THREADS), Shape::SMEM, s, mx, mw, bias, C, M, N, K, ldc,
         early, err);
  return launch_status();
}

// Shared memory to ask for so that no SM takes more than `ctas` CTAs at a time: the block scheduler does not spread a grid
// evenly by itself (128 CTAs of which an SM holds three: some SMs had two and others none, 129 us for the time of one tile, 83).
static int smem_for(int smem, long long ctas) {
  const int room = ctas <= 1 ? 200 * 1024 : ctas == 2 ? 110 * 1024 : 0;
  return smem > room ? smem : room;
}

template <int WM, int WN, int CTAS>
static int launch_tile(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                       bool early, int* err, long long per_sm, cudaStream_t s) {
  const int SMEM = smem_for(1024 + GT_STAGES * (WM + WN) * 32 * 128 + GT_STAGES * 16, per_sm);
  CUtensorMap ma, mw;
  if (!make_map_f32(&ma, A, M, K, lda, WM * 32) || !make_map_f32(&mw, W, N, K, ldw, WN * 32)) return (int)cudaErrorInvalidValue;
  const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tile_kernel<WM, WN, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (e != cudaSuccess) return (int)e;
  launch(gemm_f32_tile_kernel<WM, WN, CTAS>, dim3((M + WM * 32 - 1) / (WM * 32), (N + WN * 32 - 1) / (WN * 32)), dim3(WM * WN * 32), SMEM, s,
         ma, mw, bias, C, M, N, K, ldc, early, err);
  return launch_status();
}

// The zero padding of the K tail adds fma(0, 0, acc) = acc, which leaves the chains unchanged.
// fixed: no kernel writes W, so it may be fetched before the kernel ahead has ended.  scratch: what q25_gemm_f32_scratch says, 16-byte
// aligned, for products that the tensor cores take, but not for up to F32X3_FEW rows that are aligned to 16 bytes.  err: device int that
// gets a code if a bounded wait gave up.
Q25_EXPORT long long q25_gemm_f32_scratch(int M, int N, int K) { return M > 0 && N > 0 && f32x3_takes(K) ? (long long)f32x3_scratch(M, N, K) : 0; }
// Kernels that this thread's last product on tensor cores with scratch memory was.
Q25_EXPORT int q25_gemm_f32_launches() { return f32x3_launches; }
Q25_EXPORT int q25_gemm_f32(const float* A, const float* W, const float* bias, float* C, void* scratch, int M, int N, int K, int lda,
                            int ldw, int ldc, int fixed, int* err, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || !err) return (int)cudaErrorInvalidValue;
  cudaStream_t s = (cudaStream_t)stream;
  const bool early = fixed != 0;
  if (M == 1) lda = K;                             // a single row's pitch says nothing
  if (N == 1) ldw = K;
  if (f32x3_takes(K) && ldw % 4 == 0 && ldw >= K && !((uintptr_t)W & 15)) {
    if (M <= F32X3_FEW && lda % 4 == 0 && lda >= K && !((uintptr_t)A & 15))
      return launch_f32x3_few(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, s);
    if (!scratch || ((uintptr_t)scratch & 15)) return (int)cudaErrorInvalidValue;
    return launch_f32x3_many(A, W, bias, C, scratch, M, N, K, lda, ldw, ldc, early, err, s);
  }
  const bool tma = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && lda >= K && ldw >= K && !((uintptr_t)A & 15) && !((uintptr_t)W & 15);
  // Few steps of K: the other kernels' start counts for more than their loads (a row of K 16: 2.5 against 3.2 us; and for the many
  // CTAs of a large vocabulary, 152,064 features: K 48 and up to four rows 25 against 34, K 64 and eight 35 against 52, K 128
  // and sixteen 70 against 86; from 22,016 features down, and beyond these K, the others are faster).
  const bool brief = M <= 16 && (K <= 16 || (N > 32768 && K <= (M <= 4 ? 48 : M <= 8 ? 64 : 128)));
  if (!tma || brief || (N + 63) / 64 > 65535) {
    if (M <= 16) {
      dim3 grid((N + 63) / 64, (M + 15) / 16);
      launch(gemm_f32_kernel<16, 64, 16, 1, 4>, dim3(grid), dim3(256), 0, s, A, W, bias, C, M, N, K, lda, ldw, ldc);
    } else {
      dim3 grid((N + 63) / 64, (M + 63) / 64);
      launch(gemm_f32_kernel<64, 64, 16, 4, 4>, dim3(grid), dim3(256), 0, s, A, W, bias, C, M, N, K, lda, ldw, ldc);
    }
    return launch_status();
  }
  if (M <= 16 && K <= GR_K && K % 32 == 0 && lda % 32 == 0 && ldw % 32 == 0) {
    if (M == 1) return launch_rows<1, 1>(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, s);
    if (M == 2) return launch_rows<2, 1>(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, s);
    if (M <= 4) return launch_rows<4, 1>(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, s);
    if (M <= 8) return launch_rows<8, 1>(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, s);
    return launch_rows<8, 2>(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, s);
  }
  // Which tile ends first: q CTAs on the fullest SM, each an area of outputs, at the FMAs a clock that an SM was measured to
  // do with one, two or more such CTAs (of 128; 1,500 rows x 22,016 features: 45 TFLOP/s with 64 x 64, 41 with 32 x 32, but
  // 64 rows x 2,048 features, K 11,008: 432 against 112 us, and 1,500 x 2,048: 340 against 321 us).  Of the warps side by side in K
  // only as many work as a round has segments, which counts where an SM has more than one CTA (257 rows x 22,016 features, K
  // 128: 47 us with 64 x 64, 120 with 32 x 32).
  const int sms = device_sm_count();
  if (sms <= 0) return (int)cudaErrorInvalidDevice;
  const long long q64 = ((long long)((M + 63) / 64) * ((N + 63) / 64) + sms - 1) / sms;
  const long long q32 = ((long long)((M + 31) / 32) * ((N + 31) / 32) + sms - 1) / sms;
  const int segments = (K + GF_SEG - 1) / GF_SEG, rounds = (segments + GS_WARPS - 1) / GS_WARPS;
  const double t64 = 4096.0 * q64 / (q64 == 1 ? 53 : q64 == 2 ? 69 : 78);
  const double t32 = 1024.0 * q32 / (q32 == 1 ? 50 : q32 == 2 ? 62 : 70) * (q32 == 1 ? 1.0 : (double)(rounds * GS_WARPS) / segments);
  if (t32 < t64 && (N + 31) / 32 <= 65535) {
    const int stages = q32 == 1 ? 4 : 2;
    CUtensorMap ma, mw;
    if (!make_map_f32(&ma, A, M, K, lda, 32) || !make_map_f32(&mw, W, N, K, ldw, 32)) return (int)cudaErrorInvalidValue;
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return (int)e;
    launch(gemm_f32_split_kernel, dim3((M + 31) / 32, (N + 31) / 32), dim3(GS_WARPS * 32), smem_for(GS_SMEM(stages), q32), s, ma, mw, bias, C, M, N, K, ldc,
           stages, early, err);
    return launch_status();
  }
  return launch_tile<2, 2, 3>(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, q64, s);
}
