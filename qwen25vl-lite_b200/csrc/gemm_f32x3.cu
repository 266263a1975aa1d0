// C[M,N] = A[M,K] . W[N,K]^T (+ bias[N]) of 32-bit operands on the tensor cores: for operands of both signs nearer to 64 bits than by 32-bit
// FMAs, for sums of one sign not always (below).
//
// A 32-bit number is the sum of three bfloat16 numbers, hi + mid + lo: hi is the number rounded, mid what hi leaves, rounded,
// lo the rest; 8 bits of the mantissa each, so nothing is lost (below 2^-109 the rest is less than bfloat16's smallest number, and low
// bits are lost; results so small that this could be seen are computed again).  Of the nine products of two such sums the six largest are taken;
// the others (mid lo, lo mid, lo lo) are below 2^-24 of the product.  bfloat16 products are exact in 32 bits, what remains is how
// they are added.  The tensor core cuts bits off where FMA rounds, so it adds no more than 32 k (two instructions of 16 k for
// each of the six, the small ones first); the values of these chunks are added by ordinary 32-bit additions.  For every
// output element, whatever kernel computes it:
//
//   chunk   32 k: lo.hi, hi.lo, mid.mid, mid.hi, hi.mid, hi.hi (weight . row), 16 k and then the next 16 k of each, into one
//           accumulator that begins at 0;
//   block   256 k: its chunks' values, added in order;
//   result  the blocks' values, added in order; then + bias.
//
// The order depends on nothing but K, so a token's result is bit for bit the same whether it is computed alone, in a portion or in a
// large batch: mma.sync and tcgen05.mma give the same bits for the same 16 k (test_gemm_f32x3_gpu.py holds them to it).
// Error against 64 bits, relative 2-norm, random operands, by FMA (gemm_f32.cu) and here, at K 256 / 2,048 / 11,008: of both signs 1.49e-7 and
// 8.0e-8, 1.66e-7 and 9.8e-8, 2.24e-7 and 1.46e-7; with exponents spread over 2^+-12 1.14e-7 and 9.0e-8, 1.35e-7 and 1.06e-7, 2.02e-7 and
// 1.51e-7.  Sums of one sign collect what is cut off: 6.9e-8 and 7.0e-8, 6.3e-8 and 7.1e-8, 1.44e-7 and 1.15e-7 (and 5.6e-8 and 6.8e-8 at 1,024); with
// spread exponents 9.9e-8 and 1.61e-7, 8.8e-8 and 1.56e-7, 1.46e-7 and 1.75e-7.
// A result that is not finite (an infinite or not-a-number operand has no three parts; a part may round up to infinity), or below 2^-84
// and not zero, is computed again by plain FMA, behind its CTA's pipeline.
//
//   * up to 16 rows (decode steps): f3_rows_kernel, a stream of the weights, mma.sync;
//   * more rows: f3_parts_kernel cuts A into its three parts, f3_tile_kernel multiplies, tcgen05; where its tiles are too few
//     for the SMs, a tile's blocks go to several CTAs and f3_sum_kernel adds them.
#include "f32x2.cuh"
#include "gemm_f32x3.cuh"
#include "tcgen05.cuh"
#include "tensor_map.cuh"

#define F3_CHUNK 32
#define F3_BLOCK 256
#define F3_BLOCK_CHUNKS (F3_BLOCK / F3_CHUNK)

// The parts of two neighbours, packed as the tensor core reads them (the first in the low half).
__device__ __forceinline__ unsigned f3_pack(float lo, float hi) {
  unsigned r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// What a part leaves: number - part, exact.  (The mixed FMA reads the part as it is packed: a pair of numbers is cut up in 10 cycles of
// a scheduler, 12 where the parts are unpacked for a packed subtraction.)
__device__ __forceinline__ float2 f3_less(float2 x, unsigned part) {
  float2 r;
  asm("{\n .reg .b16 a, b, m;\n mov.b32 {a, b}, %2;\n mov.b16 m, 0xbf80;\n"           // m = -1
      " fma.rn.f32.bf16 %0, a, m, %3;\n fma.rn.f32.bf16 %1, b, m, %4;\n}\n" : "=f"(r.x), "=f"(r.y) : "r"(part), "f"(x.x), "f"(x.y));
  return r;
}
__device__ __forceinline__ void f3_split(f32x2 x, unsigned& hi, unsigned& mid, unsigned& lo) {
  float2 v = split2(x);
  hi = f3_pack(v.x, v.y);
  v = f3_less(v, hi);
  mid = f3_pack(v.x, v.y);
  v = f3_less(v, mid);
  lo = f3_pack(v.x, v.y);
}

// Neither infinite nor not a number, nor so small that what operands lose below 2^-109 would be seen: at most 2^-134 each, times partners
// up to 2^10, 2^15 of them, is below half a unit in the last place of 2^-84.
__device__ __forceinline__ bool f3_sound(float v) {
  const float size = fabsf(v);
  return size <= 3.402823466e38f && (size >= 0x1p-84f || size == 0.f);
}

// ---- results that are not finite, or very small --------------------------------------------------------------------------------------
// They are marked where they are stored and computed again when their CTA's pipeline has ended: a dot product of 11,008 terms takes
// some microseconds, during which warps with bounded waits would stand.
//
// Four dot products of a row by plain FMA, by a warp: lane l has k = 4 l .. 4 l + 3 of every 128, in one chain; one order, like all here.
template <int STEPS>
__device__ __forceinline__ void f3_plain_steps(const float* a, const float* const (&w)[4], float (&sum)[4]) {      // STEPS x 128 k; all loads first
  float x[STEPS][4];                             // perhaps not aligned
  float4 v[STEPS][4];
#pragma unroll
  for (int t = 0; t < STEPS; ++t) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[t][j] = __ldcg(reinterpret_cast<const float4*>(w[j] + t * 128));
#pragma unroll
    for (int j = 0; j < 4; ++j) x[t][j] = __ldcg(a + t * 128 + j);
  }
#pragma unroll
  for (int t = 0; t < STEPS; ++t)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      sum[j] = fmaf(x[t][3], v[t][j].w, fmaf(x[t][2], v[t][j].z, fmaf(x[t][1], v[t][j].y, fmaf(x[t][0], v[t][j].x, sum[j]))));
}
__device__ __forceinline__ void f3_plain(const float* a, const float* const (&row)[4], int K, float (&sum)[4]) {
  int k = (threadIdx.x & 31) * 4;
  const float* w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    sum[j] = 0.f;
    w[j] = row[j] + k;
  }
  a += k;
  auto on = [&](int by) {
    k += by;
    a += by;
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] += by;
  };
  for (; k + 128 < K; on(256)) f3_plain_steps<2>(a, w, sum);
  if (k < K) f3_plain_steps<1>(a, w, sum);
#pragma unroll
  for (int j = 0; j < 4; ++j) sum[j] = warp_sum(sum[j]);
}
// All warps of a CTA look at rows m0 .. m0 + rows of features n0 .. n1 (`marks`: a word of shared memory for each 32 features of a row), and
// four features of a row are computed again by a warp.  A row of A that holds a NaN has nothing else to become, and shows it early where all
// of it is NaN: the products after activations that have all turned into NaN take little longer (1,500 rows x 22,016 x 2,048
// 572 -> 646 us, one row 39 -> 47; with one infinity among the 1,500 rows 1,223 us).
__device__ __noinline__ void f3_again(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* C,
                                      unsigned* marks, int m0, int rows, int n0, int n1, int K, int lda, int ldw, int ldc) {
  const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5, lane = threadIdx.x & 31, words = (n1 - n0 + 31) / 32;
  bool any = false;
  for (int r = warp; r < rows; r += warps) {
    const float* a = A + (size_t)(m0 + r) * lda;
    bool looked = false, nan = false;
    for (int i = 0; i < words; ++i) {
      const int n = n0 + i * 32 + lane;
      unsigned mark = nan ? 0 : __ballot_sync(0xffffffffu, n < n1 && !f3_sound(__ldcg(C + (size_t)(m0 + r) * ldc + min(n, n1 - 1))));
      for (int k = lane; mark != 0 && !looked && !nan && k < K; k += 128) {      // K is a multiple of 32: the lanes go together
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (k + 32 * j < K) nan |= isnan(__ldcg(a + k + 32 * j));
        nan = __any_sync(0xffffffffu, nan);
      }
      looked |= mark != 0;
      if (nan) mark = 0;
      any |= mark != 0;
      if (lane == 0) marks[r * words + i] = mark;
    }
  }
  if (__syncthreads_or(any)) {
    for (int u = warp; u < rows * words * 8; u += warps) {
      const unsigned mark = marks[u >> 3] >> (u & 7) * 4 & 15;
      if (mark == 0) continue;
      const int m = m0 + (u >> 3) / words, n = n0 + (u >> 3) % words * 32 + (u & 7) * 4;
      const float* w[4];
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = W + (size_t)min(n + j, n1 - 1) * ldw;
      f3_plain(A + (size_t)m * lda, w, K, v);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (lane == j && (mark >> j & 1)) C[(size_t)m * ldc + n + j] = v[j] + (bias ? bias[n + j] : 0.f);
    }
  }
  __syncthreads();                                               // the marks are free
}

// ---- up to 16 rows: a stream of the weights -------------------------------------------------------------------------
// One persistent CTA per SM; its items are (group of 16 features, of small products with more rows also a group of 16 rows; 512 k), one stage of the ring each, which two copies fill: a
// box of 16 rows of W and one of the rows of x (the copy engine takes a request about every 90 cycles whatever its size).  K is
// seen as lines of 32; a row of W's box holds 17 of them, the last one not used, so that the 128-byte swizzle puts the same
// line of eight rows into eight different bank groups.  A team of four warps has an item, half a block a warp: the weights are
// the 16-row side of mma.sync m16n8k16, the rows of x its 8 columns (two such tiles for 9 to 16 rows), and a thread's 16 bytes
// of a row fill its four k slots (the sum over 16 k has no order).
// Up to 4 rows leave columns idle, and cutting numbers into parts is what a warp spends most on: there the columns are the rows of 2 or
// 4 lines side by side, cut up once, of which the MMAs of a line use their own; a warp works on two lines at a time, as the 12 MMAs of a chunk wait
// for one another; and every chunk's value goes to the warp that adds the blocks.  With more rows the warp of a block's second half adds its chunks to the
// first half's sum, in shared memory; it waits for that sum at an mbarrier (`half_done`), like every wait here with a limit: at a
// hardware barrier it would wait for good once a warp has given up.
// Measured, us for 1 / 2 / 4 / 8 / 16 rows (in a row of launches over weights that are not in L2), by FMA in brackets: 22,016 features x 2,048
// 27.4 / 28.4 / 28.8 / 30.6 / 44.5 (26.7 / 27.7 / 30.9 / 39.4 / 70.4), 2,048 x 11,008 16.2 / 17.6 / 17.8 / 18.5 / 26.5 (15.2 / 16.0 / 18.3 / 24.9 / 41),
// 2,560 x 2,048 6.7 / 6.7 / 7.0 / 6.9 / 10.7 (5.0 / 5.5 / 6.5 / 8.6 / 15.8), 320 x 256 2.3 / 2.3 / 2.2 / 2.6 / 3.4 (2.2 / 2.2 / 2.5 / 3.4 / 3.6).
// One and two rows stay behind FMA where the first stages arrive together: cutting up 32 KB takes four schedulers some 320 cycles, with every
// team's 12 MMAs behind it.  With every line's rows cut up for itself, a line at a time, and divisions in the producer and the adding warp one
// row took 30.2, 18.7 and 7.5 us.  Two warps a stage: 35, 21; stages of 256 k: 39, 23; sixteen warps with a chunk each of every
// stage: 37, 22; two teams of eight warps with two lines each: 32, 20; lines as the MMA's rows and items of 4 features x 2,048 k, the rows
// in shared memory whole: 28.3, 17.0, but 15.3 for 4,608 x 3,584 (12.4).
#define F3R_FEATURES 16
#define F3R_K 512
#define F3R_PITCH (17 * 128)                     // bytes between the rows of W in a stage
#define F3R_W_BYTES (F3R_FEATURES * F3R_PITCH)

template <int MP, int TEAMS> struct F3Rows {     // MP: rows of x in a stage; teams of four warps
  static constexpr int TILES = MP > 8 ? 2 : 1;
  static constexpr int STAGE = F3R_W_BYTES + MP * F3R_K * 4;
  // One row would have room for six, but then no CTA of a small kernel ahead (a norm) fits beside this one, which starts fetching later for it:
  // a generation step of one request, 6 layers of the 3B sizes, 650 us, with five 637.
  static constexpr int STAGES = MP <= 4 ? 5 : MP == 8 ? 4 : 3;
  static constexpr int VALUES = MP < 8 ? F3_BLOCK_CHUNKS : 1;    // that a team leaves of a block: its chunks', or their sum
  static constexpr int RED = F3R_K / F3_BLOCK * VALUES * F3R_FEATURES * MP;          // floats that a team leaves
  static constexpr int THREADS = (TEAMS * 4 + 2) * 32;
  static constexpr int SMEM = 1024 + STAGES * STAGE + TEAMS * RED * 4 + (2 * STAGES + 4 * TEAMS) * 8 + 16;
  static_assert(SMEM <= 227 * 1024 && TEAMS <= STAGES, "shared memory");
};

__device__ __forceinline__ void f3_mma(float (&c)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <int MP, int TEAMS>
__global__ void __launch_bounds__(F3Rows<MP, TEAMS>::THREADS, 1)
f3_rows_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const float* __restrict__ A,
               const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C, int M, int N, int K, int lda, int ldw,
               int ldc, bool early, int* err) {
  using Shape = F3Rows<MP, TEAMS>;
  constexpr int S = Shape::STAGES, TILES = Shape::TILES;
  extern __shared__ unsigned char f3_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)f3_raw + 1023) & ~(uintptr_t)1023);
  float* red = reinterpret_cast<float*>(smem + S * Shape::STAGE);
  unsigned long long* full = reinterpret_cast<unsigned long long*>(red + TEAMS * Shape::RED);
  unsigned long long* empty = full + S;
  unsigned long long* red_full = empty + S;
  unsigned long long* red_empty = red_full + TEAMS;
  unsigned long long* half_done = red_empty + TEAMS;             // two of each team, one a block
  int* odd = reinterpret_cast<int*>(half_done + 2 * TEAMS);      // a result is not sound
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // its items are the spans of units: a group of features of a group of MP rows
  const int spans = (K + F3R_K - 1) / F3R_K, row_groups = (M + MP - 1) / MP, units = (N + F3R_FEATURES - 1) / F3R_FEATURES * row_groups;
  const int items = ((units - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x) * spans;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 4);
    }
    for (int s = 0; s < TEAMS; ++s) {
      mbar_init(red_full + s, MP < 8 ? 4 : 2);
      mbar_init(red_empty + s, 1);
      mbar_init(half_done + 2 * s, 1);
      mbar_init(half_done + 2 * s + 1, 1);
    }
    *odd = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  pdl_trigger();

  if (warp == TEAMS * 4) {
    // ---- producer ----
    if (lane == 0) {
      const unsigned long long once = l2_evict_first();
      // counters: a division stands between a stage that is free and its copies
      struct { int line, unit, at; } w = {0, (int)blockIdx.x, (int)blockIdx.x / row_groups * F3R_FEATURES}, x = {0, (int)blockIdx.x, (int)blockIdx.x % row_groups * MP};
      const int end = spans * (F3R_K / 32);
      auto weights = [&](int s) {
        mbar_expect_tx(full + s, Shape::STAGE);
        if (row_groups == 1) tma_3d_once(smem_u32(smem + s * Shape::STAGE), &map_w, 0, w.line, w.at, full + s, once);
        else tma_3d(smem_u32(smem + s * Shape::STAGE), &map_w, 0, w.line, w.at, full + s);                  // the next group of rows reads them too
        if ((w.line += F3R_K / 32) == end) {
          w.line = 0;
          w.unit += (int)gridDim.x;
          w.at = w.unit / row_groups * F3R_FEATURES;
        }
      };
      auto rows = [&](int s) {
        tma_3d(smem_u32(smem + s * Shape::STAGE) + F3R_W_BYTES, &map_x, 0, x.line, x.at, full + s);
        if ((x.line += F3R_K / 32) == end) {
          x.line = 0;
          x.unit += (int)gridDim.x;
          x.at = x.unit % row_groups * MP;
        }
      };
      const int ahead = min(S, items);
      if (!early) pdl_wait();
      for (int s = 0; s < ahead; ++s) weights(s);
      pdl_wait();
      for (int s = 0; s < ahead; ++s) rows(s);
      int issued = ahead, s = 0;
      unsigned parity = 0;
      for (; issued < items; ++issued) {
        if (!mbar_wait(empty + s, parity)) { atomicExch(err, 51); break; }       // nobody reads what was not asked for: the readers give up too
        weights(s);
        rows(s);
        if (++s == S) { s = 0; parity ^= 1; }
      }
      mbar_landed(full, S, issued);
    }
  } else if (warp == TEAMS * 4 + 1) {
    // ---- the chunks' and the blocks' values, added in order ----
    constexpr int V = (F3R_FEATURES * MP + 31) / 32;
    pdl_wait();                                                  // the kernel before may still read what this one overwrites
    bool ok = true;
    float total[V];
#pragma unroll
    for (int v = 0; v < V; ++v) total[v] = 0.f;
    unsigned parities = 0;                                       // a bit for each team
    int span = 0, unit = (int)blockIdx.x;
    for (int i = 0; i < items; ++i) {
      const int team = i % S % TEAMS;
      if (ok) {
        ok = mbar_wait(red_full + team, parities >> team & 1);
        if (!ok && lane == 0) atomicExch(err, 52);
      }
      parities ^= 1u << team;
      const float* slot = red + team * Shape::RED + lane;
#pragma unroll
      for (int v = 0; v < V; ++v) {
        if (V * 32 != F3R_FEATURES * MP && lane >= F3R_FEATURES * MP) continue;
#pragma unroll
        for (int block = 0; block < F3R_K / F3_BLOCK; ++block) {
          const float* at = slot + block * (Shape::VALUES * F3R_FEATURES * MP) + v * 32;
          float sum = at[0];
#pragma unroll
          for (int c = 1; c < Shape::VALUES; ++c) sum += at[c * (F3R_FEATURES * MP)];
          total[v] += sum;
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(red_empty + team);
      if (++span == spans) {
        const int n = unit / row_groups * F3R_FEATURES + (lane & 15), m0 = unit % row_groups * MP + (lane >> 4);
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const int m = m0 + v * 2;
          if (m < M && n < N && (MP > 1 || lane < F3R_FEATURES)) {
            const float value = total[v] + (bias ? bias[n] : 0.f);
            C[(size_t)m * ldc + n] = value;
            if (!f3_sound(value)) *odd = 1;
          }
          total[v] = 0.f;
        }
        span = 0;
        unit += (int)gridDim.x;
      }
    }
  } else {
  // ---- a team's warps: four lines of its item each, half a block ----
  // MMA row g of the 16 is feature (g mod 2) * 4 + g / 2 of the group, and row g + 8 that + 8: the two rows whose 64 bytes a warp reads
  // together then lie in different halves of the banks.
  constexpr int SHARE = MP >= 8 ? 1 : MP == 4 ? 2 : 4;           // lines whose parts of x lie side by side
  const int team = warp >> 2, line0 = (warp & 3) * 4, block = (warp >> 1) & 1, half = warp & 1, g = lane >> 2, t = lane & 3, f = (g & 1) * 4 + (g >> 1);
  const unsigned wa = smem_u32(smem) + f * F3R_PITCH + line0 * 128;
  const unsigned xa = smem_u32(smem) + F3R_W_BYTES + (g % MP & 7) * (F3R_K * 4) + (line0 + g / MP % SHARE) * 128 + t * 16;
  float* slot = red + team * Shape::RED + block * (Shape::VALUES * F3R_FEATURES * MP) + f;
  unsigned long long* first_half = half_done + 2 * team + block;
  bool ok = true, again = false;
  unsigned turn = 0;                                             // parity of the team's items
  // A team always meets the same stages: it has seen the phase before the one that it waits for, and a parity tells no more.
  // Past the end of K the copies bring zeros, which are multiplied like the rest: a branch around a chunk would keep the compiler from
  // working on two at a time (22,016 features x 2,048, one row: 32.5 -> 31.8 us; 2,048 x 11,008: 25.3 -> 19.2).
  for (int i = team; i < items; turn ^= 1, again = true) {
    const int s = i % S;
    if (ok) {
      ok = mbar_wait(full + s, (unsigned)(i / S) & 1);
      if (!ok && lane == 0) atomicExch(err, 53);
    }
    float v[4][TILES][4];
    unsigned a[2][2][3][4], b[2][TILES][2][3][2];
    auto weights = [&](int c, unsigned (&parts)[2][3][4]) {      // of line c
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const unsigned at = wa + s * Shape::STAGE + c * 128 + (((h * 4 + t) ^ ((f + line0 + c) & 7)) << 4);
        const ulonglong2 w0 = lds_pair(at), w1 = lds_pair(at + 8 * F3R_PITCH);
        f3_split(w0.x, parts[h][0][0], parts[h][1][0], parts[h][2][0]);
        f3_split(w1.x, parts[h][0][1], parts[h][1][1], parts[h][2][1]);
        f3_split(w0.y, parts[h][0][2], parts[h][1][2], parts[h][2][2]);
        f3_split(w1.y, parts[h][0][3], parts[h][1][3], parts[h][2][3]);
      }
    };
    auto rows = [&](int c, unsigned (&parts)[TILES][2][3][2]) {
#pragma unroll
      for (int n = 0; n < TILES; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const ulonglong2 x = lds_pair(xa + s * Shape::STAGE + n * (8 * F3R_K * 4) + c * 128 + h * 64);
          f3_split(x.x, parts[n][h][0][0], parts[n][h][1][0], parts[n][h][2][0]);
          f3_split(x.y, parts[n][h][0][1], parts[n][h][1][1], parts[n][h][2][1]);
        }
    };
    constexpr int wp[6] = {2, 0, 1, 1, 0, 0}, xp[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int n = 0; n < TILES; ++n) v[c][n][0] = v[c][n][1] = v[c][n][2] = v[c][n][3] = 0.f;
    if (MP < 8) {
      // Two lines at a time, whose MMAs wait for one another in turn.  Column n of the MMA is row n mod MP of line n / MP of those that share.
#pragma unroll
      for (int c0 = 0; c0 < 4; c0 += 2) {
        weights(c0, a[0]);
        weights(c0 + 1, a[1]);
        if (c0 == 0 || SHARE == 2) rows(c0, b[0]);
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int c = 0; c < 2; ++c) f3_mma(v[c0 + c][0], a[c][h][wp[p]], b[0][0][h][xp[p]]);
      }
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        weights(c, a[0]);
        rows(c, b[0]);
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int n = 0; n < TILES; ++n) f3_mma(v[c][n], a[0][h][wp[p]], b[0][n][h][xp[p]]);
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + s);
    if (MP < 8 || half == 0) {
      if (again && ok) {
        ok = mbar_wait(red_empty + team, turn ^ 1);
        if (!ok && lane == 0) atomicExch(err, 54);
      }
    } else if (ok) {
      // within one phase: the first half comes again only behind red_empty, so behind this warp's red_full
      ok = mbar_wait(first_half, turn);
      if (!ok && lane == 0) atomicExch(err, 59);
    }
    __syncwarp();
#pragma unroll
    for (int n = 0; n < TILES; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int col = n * 8 + 2 * t + (e & 1);
        float* at = slot + col % MP * F3R_FEATURES + 8 * (e >> 1);
        if (MP < 8) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
            if (col / MP == c % SHARE) at[(half * 4 + c) * (F3R_FEATURES * MP)] = v[c][n][e];
        } else {
          float sum = half == 0 ? v[0][n][e] : *at + v[0][n][e];
          sum += v[1][n][e];
          sum += v[2][n][e];
          *at = sum + v[3][n][e];
        }
      }
    __syncwarp();
    if (lane == 0) mbar_arrive(MP >= 8 && half == 0 ? first_half : red_full + team);
    i += s + TEAMS < S ? TEAMS : S - s + team;
  }
  }
  // every warp gets here: all waits are bounded
  __syncthreads();
  if (*odd != 0) {
    for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
      const int n0 = unit / row_groups * F3R_FEATURES, m0 = unit % row_groups * MP;
      f3_again(A, W, bias, C, reinterpret_cast<unsigned*>(smem), m0, min(MP, M - m0), n0, min(N, n0 + F3R_FEATURES), K, lda, ldw, ldc);
    }
  }
}

// ---- more rows: the parts of A --------------------------------------------------------------------------------------
// parts[3][M][K]: 10 bytes a value pass through memory, once; f3_tile_kernel then reads A's tiles as the tensor core wants them
// (a tile of A is read by N / 128 CTAs, each of which would have to cut it up again).
__global__ void __launch_bounds__(256)
f3_parts_kernel(const float* __restrict__ A, uint4* __restrict__ parts, int M, int K, int lda, bool aligned) {
  pdl_trigger();
  pdl_wait();
  const size_t eighths = (size_t)M * (K / 8);
  for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < eighths; i += (size_t)gridDim.x * 256) {
    const size_t row = i / (K / 8);
    const float* src = A + row * lda + (i - row * (K / 8)) * 8;
    float v[8];
    if (aligned) {
      const float4 p = __ldcg(reinterpret_cast<const float4*>(src)), q = __ldcg(reinterpret_cast<const float4*>(src) + 1);
      v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w;
      v[4] = q.x; v[5] = q.y; v[6] = q.z; v[7] = q.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __ldcg(src + j);
    }
    unsigned p[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) f3_split(pair2(v[2 * j], v[2 * j + 1]), p[0][j], p[1][j], p[2][j]);
#pragma unroll
    for (int q = 0; q < 3; ++q) parts[q * eighths + i] = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
  }
}

// ---- more rows: tiles of 128 features x BN rows ---------------------------------------------------------------------
// One CTA per SM.  The features are the 128 lanes of tensor memory, the rows of A its columns.  An instruction of both operands
// from shared memory would read 8 KB in 64 cycles (BN 128), all of its bandwidth, before W is even cut up.  So W's parts go to tensor
// memory: converter warps take 32 k of W's 128 rows from the ring (32-bit, 16 KB), a thread a row, and store the three parts as the A
// operand (48 columns, two such stages); A's parts come by TMA ready to be read (64 k a stage).
// The MMA warp leaves the value of each chunk of 32 k in one of two accumulators of BN columns; the drain warps add it in
// registers, and a block's value to the result so far, which lies in tensor memory as well (BN columns).
// With splits > 1 a tile's blocks are cut into that many ranges, a CTA each, and every block's value goes to its plane [M][N] of
// `planes`, for f3_sum_kernel.
// Warps: 4 drain a tile of up to 64 rows, 8 a wider one (half of its columns each, which is what their registers hold); then 4
// converters, or 8 where a chunk's MMAs leave less time (the second four take the odd chunks); a producer for W, which runs ahead
// of the kernel before, one for A's parts, and the MMA warp.
// Measured, 1,500 rows x 22,016 x 2,048: 585 us with f3_parts_kernel, 231 TFLOP/s of the product asked for (by FMA 2,988 us); a chunk takes 654 / 551 / 455 /
// 420 ns with tiles of 128 / 96 / 64 / 32 rows, which is the same 61 bytes a ns from L2 into every SM (9 TB/s) for all four: the tensor
// pipe is busy 410 of the 654.  What the warps do between their barriers must stay short: with selects for a block's first chunk
// (and the spills they brought), an error path in each loop and branches around the arrivals it was 814 ns.
template <int BN> struct F3Tile {
  static constexpr int XSTAGE = 3 * BN * 128, WSTAGE = 128 * 128;
  static constexpr int XS = BN >= 96 ? 3 : 4;
  static constexpr int SETS = BN >= 96 ? 1 : 2;                 // of four converter warps
  static constexpr int ROOM = (208 * 1024 - XS * XSTAGE) / WSTAGE;
  static constexpr int WS = ROOM > 8 ? 8 : ROOM / SETS * SETS;  // a stage always serves the same set
  static constexpr int DRAINS = BN >= 96 ? 8 : 4, WIDTH = BN * 4 / DRAINS;         // columns a drain warp has
  static constexpr int STEP = WIDTH % 32 == 0 ? 32 : 16;                           // and takes at a time
  static constexpr int WARPS = DRAINS + 4 * SETS + 3;
  static constexpr int THREADS = WARPS * 32;
  static constexpr int TOTAL = 2 * BN, PARTS = 3 * BN;          // columns: accumulators at 0 and BN, the result so far, W's parts
  static constexpr int SMEM = 1024 + XS * XSTAGE + WS * WSTAGE + 512;
  static_assert(3 * BN + 96 <= 512 && WS % SETS == 0, "tensor memory; stages");
};

// 16 words into this thread's lane of tensor memory; 16 or 32 floats out of it and back.
__device__ __forceinline__ void f3_st16(unsigned taddr, const unsigned (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void f3_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void f3_ld(unsigned taddr, float (&v)[32]) { tc5_ld32(taddr, v); }
__device__ __forceinline__ void f3_ld(unsigned taddr, float (&v)[16]) {
  unsigned r[16];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                 "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void f3_st(unsigned taddr, const float (&v)[32]) { tc5_st32(taddr, v); }
__device__ __forceinline__ void f3_st(unsigned taddr, const float (&v)[16]) {
  unsigned r[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(v[i]);
  f3_st16(taddr, r);
  f3_st_wait();
}
__device__ __forceinline__ void f3_arrive(unsigned long long* bar, int lane) {       // by the first lane, without a branch
  asm volatile("{\n .reg .pred p;\n setp.eq.s32 p, %1, 0;\n @p mbarrier.arrive.shared::cta.b64 _, [%0];\n}\n" ::"r"(smem_u32(bar)), "r"(lane) : "memory");
}
__device__ __forceinline__ bool f3_elect() {
  unsigned e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
  return e != 0;
}
__device__ constexpr unsigned f3_idesc(int n) {                  // bf16 x bf16 -> f32, M 128, N n, both operands K-major
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(128 >> 4) << 24);
}

template <int BN>
__global__ void __launch_bounds__(F3Tile<BN>::THREADS, 1)
f3_tile_kernel(const __grid_constant__ CUtensorMap map_p, const __grid_constant__ CUtensorMap map_w, const float* __restrict__ A,
               const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C, float* __restrict__ planes, int splits, int M,
               int N, int K, int lda, int ldw, int ldc, bool early, int* err) {
  using Shape = F3Tile<BN>;
  constexpr int XS = Shape::XS, WS = Shape::WS, SETS = Shape::SETS;
  extern __shared__ unsigned char f3_raw[];
  unsigned char* xring = reinterpret_cast<unsigned char*>(((uintptr_t)f3_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* wring = xring + XS * Shape::XSTAGE;
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(wring + WS * Shape::WSTAGE);
  unsigned long long *w_full = bars, *w_empty = w_full + WS, *x_full = w_empty + WS, *x_empty = x_full + XS;
  // of each of the two buffers (a stage of W's parts and an accumulator): both are free for the MMAs; these have ended
  unsigned long long *ready = x_empty + XS, *done = ready + 2;
  unsigned* tmem_at = reinterpret_cast<unsigned*>(done + 2);
  int* odd = reinterpret_cast<int*>(tmem_at + 1);                // a result is not sound
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int W_WARP = Shape::DRAINS + 4 * SETS, X_WARP = W_WARP + 1, MMA_WARP = W_WARP + 2;
  const int row_tiles = (M + BN - 1) / BN, tiles = row_tiles * ((N + 127) / 128);
  // this CTA's tiles, and the chunks of K that it takes of each (whole blocks; a split tile's CTAs have one tile)
  const int first_tile = (int)blockIdx.x / splits, part = (int)blockIdx.x % splits, step = (int)gridDim.x;
  const int blocks = (K + F3_BLOCK - 1) / F3_BLOCK;
  const int c_begin = (int)((long long)blocks * part / splits) * F3_BLOCK_CHUNKS;
  const int c_end = min(K / F3_CHUNK, (int)((long long)blocks * (part + 1) / splits) * F3_BLOCK_CHUNKS), chunks = c_end - c_begin;
  const int mine = (tiles - first_tile + step - 1) / step * chunks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < WS; ++s) { mbar_init(w_full + s, 1); mbar_init(w_empty + s, 4); }
    for (int s = 0; s < XS; ++s) { mbar_init(x_full + s, 1); mbar_init(x_empty + s, 1); }
    for (int b = 0; b < 2; ++b) {
      mbar_init(ready + b, 4 + Shape::DRAINS);
      mbar_init(done + b, 1);
    }
    *odd = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  pdl_trigger();
  auto load_w = [&](int it) {
    const int tile = first_tile + it / chunks * step, s = it % WS;
    mbar_expect_tx(w_full + s, Shape::WSTAGE);
    tma_2d(smem_u32(wring + s * Shape::WSTAGE), &map_w, (c_begin + it % chunks) * F3_CHUNK, tile / row_tiles * 128, w_full + s);
  };
  const int ahead = min(WS, mine);
  if (early && warp == W_WARP && lane == 0)
    for (int it = 0; it < ahead; ++it) load_w(it);
  // A's parts come from the kernel before this one, and tensor memory is asked for only when that has gone (gemm_tcgen05.cu)
  pdl_wait();
  if (!early && warp == W_WARP && lane == 0)
    for (int it = 0; it < ahead; ++it) load_w(it);
  __syncwarp();
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_at)), "n"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc5_fence_before();
  __syncthreads();
  tc5_fence_after();
  const unsigned tmem = *tmem_at;
  bool ok = true;

  if (warp == W_WARP) {
    if (lane == 0) {
      int it = ahead;
      for (; it < mine; ++it) {
        if (!mbar_wait(w_empty + it % WS, (unsigned)(it / WS - 1) & 1)) { atomicExch(err, 55); break; }
        load_w(it);
      }
      mbar_landed(w_full, WS, it);
    }
  } else if (warp == X_WARP) {
    if (lane == 0) {
      int xt = 0;
      for (int tile = first_tile; tile < tiles && ok; tile += step)
        for (int c = c_begin; c < c_end; c += 2, ++xt) {
          const int s = xt % XS;
          if (xt >= XS) {
            ok = mbar_wait(x_empty + s, (unsigned)(xt / XS - 1) & 1);
            if (!ok) { atomicExch(err, 56); break; }
          }
          mbar_expect_tx(x_full + s, Shape::XSTAGE);
          tma_3d(smem_u32(xring + s * Shape::XSTAGE), &map_p, c * F3_CHUNK, tile % row_tiles * BN, 0, x_full + s);
        }
      mbar_landed(x_full, XS, xt);
    }
  } else if (warp == MMA_WARP) {
    // The whole warp walks, in uniform registers, and one lane issues: a lane that walks alone moves every operand into them,
    // 55 cycles an instruction, and each barrier costs it 300.
    const bool issues = f3_elect();
    const unsigned base = __shfl_sync(0xffffffffu, tmem, 0);
    const unsigned long long x0 = tc5_desc(__shfl_sync(0xffffffffu, smem_u32(xring), 0), 16, 1024);
    constexpr unsigned idesc = f3_idesc(BN);
    constexpr int wp[6] = {2, 0, 1, 1, 0, 0}, xp[6] = {0, 2, 1, 0, 1, 0};
    int it = 0, xs = 0;
    unsigned x_parity = 0;
    for (int tile = first_tile; tile < tiles && ok; tile += step)
      for (int c = 0; c < chunks; ++c, ++it) {
        const int b = it & 1;
        if ((c & 1) == 0) ok = mbar_wait(x_full + xs, x_parity);
        if (ok) ok = mbar_wait(ready + b, (unsigned)(it >> 1) & 1);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (issues) atomicExch(err, 57);
          break;
        }
        tc5_fence_after();
        const bool x_done = (c & 1) || c + 1 == chunks;
        if (issues) {
          const unsigned long long xd = x0 + (unsigned)(xs * (Shape::XSTAGE / 16) + (c & 1) * 4);
#pragma unroll
          for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int k = 0; k < 2; ++k)          // 16 k: 8 columns of a part of W, 32 bytes along the rows of a part of A
              tc5_mma_ts(base + b * BN, base + Shape::PARTS + b * 48 + wp[p] * 16 + k * 8, xd + xp[p] * (BN * 128 / 16) + k * 2, idesc, (p | k) != 0);
          if (x_done) tc5_commit(x_empty + xs);
          tc5_commit(done + b);
        }
        __syncwarp();
        if (x_done && ++xs == XS) { xs = 0; x_parity ^= 1; }
      }
    // the last commit stands for all products asked for: none of them still runs when tensor memory goes back
    if (it > 0) mbar_wait(done + ((it - 1) & 1), (unsigned)((it - 1) >> 1) & 1);
  } else if (warp >= Shape::DRAINS) {
    // ---- converters ----
    const int set = (warp - Shape::DRAINS) >> 2, quarter = warp & 3, row = quarter * 32 + lane;
    for (int it = set; it < mine; it += SETS) {
      const int s = it % WS, b = it & 1;
      ok = ok && mbar_wait(w_full + s, (unsigned)(it / WS) & 1);
      const unsigned at = smem_u32(wring + s * Shape::WSTAGE) + row * 128;
      ulonglong2 v[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = lds_pair(at + ((c ^ (row & 7)) << 4));
      unsigned p[3][16];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        f3_split(v[c].x, p[0][2 * c], p[1][2 * c], p[2][2 * c]);
        f3_split(v[c].y, p[0][2 * c + 1], p[1][2 * c + 1], p[2][2 * c + 1]);
      }
      __syncwarp();
      f3_arrive(w_empty + s, lane);
      if (it >= 2) ok = ok && mbar_wait(done + b, (unsigned)((it >> 1) - 1) & 1);
      tc5_fence_after();
      const unsigned to = tmem + ((unsigned)(quarter * 32) << 16) + Shape::PARTS + b * 48;
#pragma unroll
      for (int q = 0; q < 3; ++q) f3_st16(to + q * 16, p[q]);
      f3_st_wait();
      tc5_fence_before();
      __syncwarp();
      f3_arrive(ready + b, lane);
    }
  } else {
    // ---- drain: this thread's feature, WIDTH rows of the tile ----
    constexpr int WIDTH = Shape::WIDTH, STEP = Shape::STEP;
    const int col = (warp >> 2) * WIDTH;
    const unsigned lanes = tmem + ((unsigned)((warp & 3) * 32) << 16) + col;
    float acc[WIDTH];                                            // a block's chunks so far
#pragma unroll
    for (int j = 0; j < WIDTH; ++j) acc[j] = 0.f;
    if (lane < 2) mbar_arrive(ready + lane);                     // both accumulators are free
    int it = 0;
    for (int tile = first_tile; tile < tiles; tile += step) {
      const int m0 = tile % row_tiles * BN + col, n = tile / row_tiles * 128 + (warp & 3) * 32 + lane;
      for (int c = 0; c < chunks; ++c, ++it) {
        const int b = it & 1;
        const bool last = c + 1 == chunks;
        ok = ok && mbar_wait(done + b, (unsigned)(it >> 1) & 1);
        tc5_fence_after();
#pragma unroll
        for (int j0 = 0; j0 < WIDTH; j0 += STEP) {
          float v[STEP];
          f3_ld(lanes + b * BN + j0, v);
#pragma unroll
          for (int j = 0; j < STEP; ++j) acc[j0 + j] += v[j];
        }
        tc5_fence_before();
        __syncwarp();
        f3_arrive(ready + b, lane);
        if (!last && (c + 1) % F3_BLOCK_CHUNKS != 0) continue;
        // a block is complete: it joins those before it, or goes to its plane
        const bool whole = splits == 1;
#pragma unroll
        for (int j0 = 0; j0 < WIDTH; j0 += STEP) {
          float v[STEP];
          if (whole && c >= F3_BLOCK_CHUNKS) {
            f3_ld(lanes + Shape::TOTAL + j0, v);
#pragma unroll
            for (int j = 0; j < STEP; ++j) acc[j0 + j] = v[j] + acc[j0 + j];
          }
          if (whole && !last) {
#pragma unroll
            for (int j = 0; j < STEP; ++j) v[j] = acc[j0 + j];
            f3_st(lanes + Shape::TOTAL + j0, v);
          }
        }
        if ((last || !whole) && n < N) {
          const float more = whole && bias ? bias[n] : 0.f;
          const size_t pitch = whole ? ldc : N;
          float* dst = (whole ? C : planes + (size_t)((c_begin + c) / F3_BLOCK_CHUNKS) * M * N) + m0 * pitch + n;
#pragma unroll
          for (int j = 0; j < WIDTH; ++j, dst += pitch) {
            if (m0 + j < M) *dst = acc[j] + more;
            asm volatile("" : "+l"(dst));        // one address after the other: all of them at once do not fit the registers
          }
          if (whole) {                           // the planes' sums are looked at by f3_sum_kernel
            bool sound = true;
#pragma unroll
            for (int j = 0; j < WIDTH; ++j) sound &= f3_sound(acc[j] + more);
            if (!sound) *odd = 1;
          }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < WIDTH; ++j) acc[j] = 0.f;
      }
    }
  }
  // every warp gets here (all waits are bounded); then the tensor memory goes back
  if (!ok && lane == 0) atomicExch(err, 58);
  __syncwarp();
  tc5_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) {
    tc5_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(512) : "memory");
  }
  if (*odd != 0)
    for (int tile = first_tile; tile < tiles; tile += step) {
      const int m0 = tile % row_tiles * BN, n0 = tile / row_tiles * 128;
      f3_again(A, W, bias, C, reinterpret_cast<unsigned*>(xring), m0, min(BN, M - m0), n0, min(N, n0 + 128), K, lda, ldw, ldc);
    }
}

// The planes of a split product, block by block, + bias; a thread has one element of the output.  Results that are not finite are
// computed again by their warp, one after the other, with few registers (f3_again's would leave three CTAs of this kernel to an SM).
__global__ void __launch_bounds__(256, 6)
f3_sum_kernel(const float* __restrict__ planes, const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
              float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc) {
  pdl_trigger();
  pdl_wait();
  const size_t size = (size_t)M * N;
  const int blocks = (K + F3_BLOCK - 1) / F3_BLOCK, lane = threadIdx.x & 31;
  for (size_t i0 = (size_t)blockIdx.x * 256 + (threadIdx.x & ~31); i0 < size; i0 += (size_t)gridDim.x * 256) {       // a warp has 32 of them
    const size_t i = min(i0 + lane, size - 1);
    const int m = (int)(i / N), n = (int)(i - (size_t)m * N);
    float total = 0.f;
    for (int b0 = 0; b0 < blocks; b0 += 8) {     // eight loads on their way at a time
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __ldcg(planes + (size_t)min(b0 + j, blocks - 1) * size + i);
#pragma unroll
      for (int j = 0; j < 8; ++j) total = b0 + j < blocks ? total + v[j] : total;
    }
    const float more = bias ? bias[n] : 0.f;
    total += more;
    for (unsigned todo = __ballot_sync(0xffffffffu, !f3_sound(total)); todo != 0; todo &= todo - 1) {
      const int from = __ffs(todo) - 1, row = __shfl_sync(0xffffffffu, m, from);
      const float* a = A + (size_t)row * lda;
      const float* w = W + (size_t)__shfl_sync(0xffffffffu, n, from) * ldw;
      float sum = 0.f;                           // as f3_plain has it
      bool nan = false;                          // the row holds one: nothing else can come of it
      for (int k0 = 0; k0 < K && !nan; k0 += 128) {
        const int k = k0 + lane * 4;
        if (k < K) {
          const float x0 = __ldcg(a + k), x1 = __ldcg(a + k + 1), x2 = __ldcg(a + k + 2), x3 = __ldcg(a + k + 3);
          const float4 v = __ldcg(reinterpret_cast<const float4*>(w + k));
          sum = fmaf(x3, v.w, fmaf(x2, v.z, fmaf(x1, v.y, fmaf(x0, v.x, sum))));
          nan = isnan(x0) || isnan(x1) || isnan(x2) || isnan(x3);
        }
        nan = __any_sync(0xffffffffu, nan);
      }
      if (nan) todo &= ~__ballot_sync(0xffffffffu, m == row) | 1u << from;
      sum = warp_sum(sum) + more;
      if (lane == from && !nan) total = sum;
    }
    if (i0 + lane < size) C[(size_t)m * ldc + n] = total;
  }
}

// ---- host -----------------------------------------------------------------------------------------------------------
// Boxes of the three parts of bn rows x 64 k of A.
static bool f3_map_parts(CUtensorMap* map, void* base, int M, int K, int bn) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)M, 3};
  const cuuint64_t strides[2] = {(cuuint64_t)K * 2, (cuuint64_t)M * K * 2};
  const cuuint32_t box[3] = {64, (cuuint32_t)bn, 3};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MP, int TEAMS>
static int f3_launch_rows(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                          bool early, int* err, int sms, cudaStream_t s) {
  using Shape = F3Rows<MP, TEAMS>;
  CUtensorMap mx, mw;
  if (!make_blocks_f32(&mx, A, M, K, lda, MP, F3R_K / 32, false) || !make_blocks_f32(&mw, W, N, K, ldw, F3R_FEATURES, 17, true)) return (int)cudaErrorInvalidValue;
  const cudaError_t e = cudaFuncSetAttribute(f3_rows_kernel<MP, TEAMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::SMEM);
  if (e != cudaSuccess) return (int)e;
  const int units = (N + F3R_FEATURES - 1) / F3R_FEATURES * ((M + MP - 1) / MP);
  launch(f3_rows_kernel<MP, TEAMS>, dim3(units < sms ? units : sms), dim3(Shape::THREADS), Shape::SMEM, s, mx, mw, A, W, bias, C, M, N, K, lda, ldw,
         ldc, early, err);
  return launch_status();
}

int launch_f32x3_few(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                     bool early, int* err, cudaStream_t s) {
  const int sms = device_sm_count();
  if (sms <= 0) return (int)cudaErrorInvalidDevice;
  // Three teams leave their warps the registers for two lines at a time and end sooner; over a long stream of one row four ride over its
  // unevenness (us with three and four: 2,048 x 11,008, 22 items a CTA, 17.4 and 18.0, 22,016 x 2,048, 40, 28.5 and 29.8; 3,584 x 18,944, 74,
  // 59.8 and 54.5, 37,888 x 3,584, 112, 83.3 and 82.0, 151,936 x 2,048, 260, 188 and 177; two rows of the last two 79 and 90, 189 and 197).
  const bool longer = (long long)((N + F3R_FEATURES - 1) / F3R_FEATURES + sms - 1) / sms * ((K + F3R_K - 1) / F3R_K) > 56;
  if (M == 1 && longer) return f3_launch_rows<1, 4>(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, sms, s);
  if (M == 1) return f3_launch_rows<1, 3>(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, sms, s);
  if (M == 2) return f3_launch_rows<2, 3>(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, sms, s);
  if (M <= 4) return f3_launch_rows<4, 3>(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, sms, s);
  if (M <= 8) return f3_launch_rows<8, 4>(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, sms, s);
  return f3_launch_rows<16, 3>(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, sms, s);
}

// How f3_tile_kernel takes a product: the width of its tiles, and into how many ranges of blocks a tile is cut.  The one that ends
// first: the chunks of the fullest SM at what a chunk takes (ns), and for a split the trip through its planes (up to 64 MB of them, half of L2).
struct F3Plan { int bn, splits; double ns; };
static F3Plan f3_plan(int M, int N, int K, int sms) {
  const int widths[4] = {128, 96, 64, 32}, ns[4] = {640, 540, 455, 425};
  const int blocks = (K + F3_BLOCK - 1) / F3_BLOCK;
  const double planes = 4.0 * blocks * M * N;
  F3Plan best = {128, 1, 0};
  double least = -1;
  for (int i = 0; i < 4; ++i) {
    const long long tiles = (long long)((M + widths[i] - 1) / widths[i]) * ((N + 127) / 128);
    const long long room = sms / tiles;
    const int splits = planes <= 64e6 ? (int)(room < 1 ? 1 : room < blocks ? room : blocks) : 1;
    double t = splits > 1 ? 8.0 * ((blocks + splits - 1) / splits) * ns[i] + 3000 + planes / 2000 : (double)((tiles + sms - 1) / sms) * (K / F3_CHUNK) * ns[i];
    if (least < 0 || t < least) { best = {widths[i], splits, t}; least = t; }
  }
  return best;
}
static size_t f3_parts_bytes(int M, int K) { return ((size_t)6 * M * K + 255) / 256 * 256; }
size_t f32x3_scratch(int M, int N, int K) {
  const int sms = device_sm_count();
  const F3Plan plan = f3_plan(M, N, K, sms > 0 ? sms : 1);
  return f3_parts_bytes(M, K) + (plan.splits > 1 ? (size_t)4 * ((K + F3_BLOCK - 1) / F3_BLOCK) * M * N : 0);
}

template <int BN>
static int f3_launch_tiles(const float* A, const float* W, const float* bias, float* C, void* parts, float* planes, int splits, int M, int N,
                           int K, int lda, int ldw, int ldc, bool early, int* err, int sms, cudaStream_t s) {
  using Shape = F3Tile<BN>;
  CUtensorMap mp, mw;
  if (!f3_map_parts(&mp, parts, M, K, BN) || !make_map_f32(&mw, W, N, K, ldw, 128)) return (int)cudaErrorInvalidValue;
  const cudaError_t e = cudaFuncSetAttribute(f3_tile_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::SMEM);
  if (e != cudaSuccess) return (int)e;
  const long long tiles = (long long)((M + BN - 1) / BN) * ((N + 127) / 128);
  launch(f3_tile_kernel<BN>, dim3((unsigned)(splits > 1 ? tiles * splits : tiles < sms ? tiles : sms)), dim3(Shape::THREADS), Shape::SMEM, s, mp,
         mw, A, W, bias, C, planes, splits, M, N, K, lda, ldw, ldc, early, err);
  return launch_status();
}

thread_local int f32x3_launches = 1;             // of this thread's last product of more than F32X3_FEW rows
int launch_f32x3_many(const float* A, const float* W, const float* bias, float* C, void* scratch, int M, int N, int K, int lda, int ldw, int ldc,
                      bool early, int* err, cudaStream_t s) {
  const int sms = device_sm_count();
  if (sms <= 0) return (int)cudaErrorInvalidDevice;
  const F3Plan plan = f3_plan(M, N, K, sms);
  // Small products, as groups of 16 rows: one launch instead of two or three.  An item takes 1.1 us and the launch 2.5; tiles have 2.4 us of
  // launches around them, a split one 2 more than its plan counts (us by tiles and this way: 17 rows x 320 features x 256 6.2 and 3.7, 64 x 320 x 512
  // 7.5 and 3.6, 64 x 1,024 x 512 8.0 and 5.5, 17 x 1,024 x 1,024 7.6 and 5.3; 64 x 4,096 x 512 stays with the tiles at 9.5).
  const long long units = (long long)((N + F3R_FEATURES - 1) / F3R_FEATURES) * ((M + 15) / 16);
  if (lda % 4 == 0 && lda >= K && !((uintptr_t)A & 15) && units < 1 << 16 &&
      1100.0 * ((units + sms - 1) / sms) * ((K + F3R_K - 1) / F3R_K) + 2500 < plan.ns + (plan.splits > 1 ? 2000 : 2400)) {
    f32x3_launches = 1;
    return f3_launch_rows<16, 3>(A, W, bias, C, M, N, K, lda, ldw, ldc, early, err, sms, s);
  }
  const size_t most = (size_t)sms * 8, eighths = ((size_t)M * (K / 8) + 255) / 256, elements = ((size_t)M * N + 255) / 256;
  launch(f3_parts_kernel, dim3((unsigned)(eighths < most ? eighths : most)), dim3(256), 0, s, A, (uint4*)scratch, M, K, lda,
         lda % 4 == 0 && !((uintptr_t)A & 15));
  float* planes = reinterpret_cast<float*>(static_cast<char*>(scratch) + f3_parts_bytes(M, K));
  int e;
  if (plan.bn == 128) e = f3_launch_tiles<128>(A, W, bias, C, scratch, planes, plan.splits, M, N, K, lda, ldw, ldc, early, err, sms, s);
  else if (plan.bn == 96) e = f3_launch_tiles<96>(A, W, bias, C, scratch, planes, plan.splits, M, N, K, lda, ldw, ldc, early, err, sms, s);
  else if (plan.bn == 64) e = f3_launch_tiles<64>(A, W, bias, C, scratch, planes, plan.splits, M, N, K, lda, ldw, ldc, early, err, sms, s);
  else e = f3_launch_tiles<32>(A, W, bias, C, scratch, planes, plan.splits, M, N, K, lda, ldw, ldc, early, err, sms, s);
  f32x3_launches = plan.splits == 1 ? 2 : 3;
  if (e != 0 || plan.splits == 1) return e;
  launch(f3_sum_kernel, dim3((unsigned)(elements < most ? elements : most)), dim3(256), 0, s, planes, A, W, bias, C, M, N, K, lda, ldw, ldc);
  return launch_status();
}
