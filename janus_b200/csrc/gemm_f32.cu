// True float32 matrix product on CUDA cores: Y[T, N] (+)= X[T, K] . W[N, K]^T.
// No tensor cores, no reduced-precision mode.  An output element is summed in ONE order whatever kernel a step's size
// selects, how many rows the batch has and where the row sits in it: k runs in segments of 64, whose even and odd k are
// each summed from zero by fused multiply-adds in the order of k and then added; K is cut into at most eight ranges of
// whole 256s, a range adds its segments up in order, and the ranges are added to the output in order (the first one
// stored, where nothing is accumulated).
// Even and odd k apart, because a packed multiply-add (`fma.rn.f32x2`) takes them as they lie in memory: the same 128
// multiply-adds a cycle and SM in half the instructions (1,000 tokens x 16,384 rows x 2,048: 2,079 -> 1,855 us).
// Short sums that meet in a shallow tree are also closer to the exact result than one chain over K (K = 8,192: 1.4e-7
// against 1.6e-6 of the result, 2-norms).
// Formula: crates/janus-engine/src/compute/shaders/gemm_f32.wgsl:23-75
// (weights [N, K] row-major, f32 accumulation over 16-wide k tiles).
#include <cooperative_groups.h>
#include <stdio.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int SEG = 64, SEGS = 4, UNIT = SEG * SEGS, RANGES = 8;

// numbers of k in a range (the last one may hold fewer)
__host__ __device__ inline int range_of(int K) { return ((K + UNIT - 1) / UNIT + RANGES - 1) / RANGES * UNIT; }

// two numbers of neighbouring k, and two sums of even and odd k
using jb::fma2;
using jb::Pair;
__device__ __forceinline__ float even_and_odd(Pair p) { return jb::lo(p) + jb::hi(p); }

__device__ __forceinline__ void async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}
// copies `bytes` (0, 4 or 16 of a piece of 4 or 16) and fills the rest of the piece with zeros
__device__ __forceinline__ void async16_or_zero(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes));
}
__device__ __forceinline__ void async4_or_zero(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(bytes));
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N));
}

// ---- few tokens: the product streams the weights -----------------------------------------------------------------
// A block owns 16 weight rows at a time, each of its up to eight warps a range of k of them, walked by itself in
// units of 256 k: lane (r, s) sums segment s of the unit for rows r and 8 + r and all tokens, so that 32 chains of 64
// products run side by side.  A stage is half of a unit's segments, pieces of 128 contiguous bytes of every row and
// token with 16 bytes of padding between them (the eight lanes of a shared-memory phase read eight different banks);
// a warp's ring of two stages is its own, so nothing synchronises the block until the ranges meet, and it runs on
// over the rows that a block works through one after another.  The first stages' weights are asked for before the
// kernel that makes X has ended.
constexpr int SUB = 32, PIECE = SUB + 4;       // numbers of a piece, and its pitch
constexpr int RL = 2, STAGES = 2;              // rows of a lane, stages of a ring

template <int TT>
__global__ void __launch_bounds__(32 * RANGES) gemm_f32_stream_kernel(const float* __restrict__ X, const float* __restrict__ W,
                                                                      float* __restrict__ Y, int T, int N, int K, int ldx,
                                                                      int ldy, int accumulate) {
  constexpr int ROWS = 8 * RL, W_PIECES = ROWS * SEGS;
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ranges = blockDim.x >> 5;
  const int t0 = (int)blockIdx.y * TT, tokens = min(T - t0, TT);
  const int stage_floats = (W_PIECES + TT * SEGS) * PIECE;
  float* met = smem;                                            // [range][token][row] of the ranges' sums
  float* ring = smem + RANGES * TT * ROWS + (size_t)warp * STAGES * stage_floats;
  const int range = range_of(K), k_begin = warp * range, k_end = min(K, k_begin + range);
  const int steps = 2 * ((k_end - k_begin + UNIT - 1) / UNIT);
  const int blocks = (N + ROWS - 1) / ROWS;
  const int total = ((blocks - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x) * steps;
  X += (size_t)t0 * ldx;
  Y += (size_t)t0 * ldy;

  // where the next stage to load begins: this lane copies 16 bytes of piece (4 i + lane / 8): row i, segment lane / 8
  int load_step = 0, load_n0 = (int)blockIdx.x * ROWS, load_slot = 0;
  const int lk = (lane >> 3) * SEG + (lane & 7) * 4, lo = (lane >> 3) * PIECE + (lane & 7) * 4;
  auto load_w = [&]() {
    const int k = k_begin + (load_step >> 1) * UNIT + (load_step & 1) * SUB + lk;
    float* dst = ring + load_slot * stage_floats + lo;
    if (k < k_end) {
#pragma unroll
      for (int i = 0; i < ROWS; ++i)                            // rows past the last one repeat it, their sums are dropped
        async16(dst + i * SEGS * PIECE, W + (size_t)min(load_n0 + i, N - 1) * K + k);
    }
  };
  auto load_x = [&](bool now) {
    const int k = k_begin + (load_step >> 1) * UNIT + (load_step & 1) * SUB + lk;
    float* dst = ring + load_slot * stage_floats + W_PIECES * PIECE + lo;
    if (k < k_end) {
#pragma unroll
      for (int t = 0; t < TT; ++t) {
        const float* src = X + (size_t)min(t, tokens - 1) * ldx + k;
        if (now) *reinterpret_cast<float4*>(dst + t * SEGS * PIECE) = *reinterpret_cast<const float4*>(src);
        else async16(dst + t * SEGS * PIECE, src);
      }
    }
  };
  auto next = [&]() {
    load_slot = load_slot + 1 == STAGES ? 0 : load_slot + 1;
    if (++load_step == steps) load_step = 0, load_n0 += (int)gridDim.x * ROWS;
  };

  jb::pdl_launch_dependents();
  int loaded = 0;
#pragma unroll
  for (int i = 0; i < STAGES - 1; ++i) {
    if (loaded < total) load_w(), next(), ++loaded;
    async_commit();
  }
  jb::pdl_wait();
  // the first stages' tokens by plain loads: a copy group of their own would only end after all weights asked for so far
  load_step = 0, load_slot = 0, load_n0 = (int)blockIdx.x * ROWS;
  for (int i = 0; i < loaded; ++i) load_x(true), next();

  // A unit's sums, one for each (row, token) and segment, join the range in the order of the segments: the four lanes of a row
  // exchange theirs so that each ends with all four segments of its share of the (row, token) pairs, in as many shuffles as a
  // lane has pairs (every lane asking the others for every pair took four times as many: 8 tokens, 16,384 rows of 2,048, 44.0 us
  // and 41.4 so, 16 tokens 86 and 81, 8 tokens of 50,257 rows of 1,536 97 and 92, 4 tokens 68 and 66).  One or two tokens have too
  // few pairs for the selections to pay: each lane asks for each (one token, 1,536 rows of 1,536, 3.48 us, 3.63 exchanged; two
  // 3.77 and 3.88).
  constexpr int PAIRS = RL * TT;
  constexpr bool EXCHANGED = TT >= 4;
  constexpr int MINE = EXCHANGED ? PAIRS / 4 : PAIRS;
  Pair acc[RL][TT];
  float sum[MINE];
#pragma unroll
  for (int r = 0; r < RL; ++r)
#pragma unroll
    for (int t = 0; t < TT; ++t) acc[r][t] = 0;
#pragma unroll
  for (int i = 0; i < MINE; ++i) sum[i] = 0.0f;
  const int row = lane >> 2, seg = lane & 3;
  int step = 0, n0 = (int)blockIdx.x * ROWS, slot = 0;

  for (int it = 0; it < total; ++it) {
    async_wait<STAGES - 2>();
    __syncwarp();                                              // all lanes' copies of this stage; the stage before is free
    if (loaded < total) load_w(), load_x(false), next(), ++loaded;
    async_commit();
    const float* w = ring + slot * stage_floats + lane * PIECE;
    const float* x = ring + slot * stage_floats + (W_PIECES + seg) * PIECE;
    const int k0 = k_begin + (step >> 1) * UNIT + (step & 1) * SUB, left = k_end - k0 - seg * SEG;
    auto products = [&](int k) {
      ulonglong2 b[RL];
#pragma unroll
      for (int r = 0; r < RL; ++r) b[r] = *reinterpret_cast<const ulonglong2*>(w + r * 32 * PIECE + k);
#pragma unroll
      for (int t = 0; t < TT; ++t) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(x + t * SEGS * PIECE + k);
#pragma unroll
        for (int r = 0; r < RL; ++r) acc[r][t] = fma2(a.y, b[r].y, fma2(a.x, b[r].x, acc[r][t]));
      }
    };
    if (k0 + UNIT - SUB <= k_end) {                            // all four segments reach the end of this stage
#pragma unroll
      for (int k = 0; k < SUB; k += 4) products(k);
    } else {
      for (int k = 0; k < min(left, SUB); k += 4) products(k);
      __syncwarp();
    }
    slot = slot + 1 == STAGES ? 0 : slot + 1;
    if (step & 1) {                                            // the unit's segments join the range in order
      const int u0 = k0 - SUB;
      float one[PAIRS];
#pragma unroll
      for (int i = 0; i < PAIRS; ++i) one[i] = even_and_odd(acc[i / TT][i % TT]), acc[i / TT][i % TT] = 0;
      if constexpr (EXCHANGED) {
        const bool odd = seg & 1, late = seg & 2;
        float two[PAIRS / 2][2];                               // half of the pairs, segments seg & ~1 and seg | 1
#pragma unroll
        for (int i = 0; i < PAIRS / 2; ++i) {
          const float keep = odd ? one[PAIRS / 2 + i] : one[i];
          const float got = __shfl_xor_sync(0xffffffffu, odd ? one[i] : one[PAIRS / 2 + i], 1);
          two[i][0] = odd ? got : keep, two[i][1] = odd ? keep : got;
        }
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
          float four[SEGS];
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const float keep = late ? two[MINE + i][x] : two[i][x];
            const float got = __shfl_xor_sync(0xffffffffu, late ? two[i][x] : two[MINE + i][x], 2);
            four[x] = late ? got : keep, four[2 + x] = late ? keep : got;
          }
#pragma unroll
          for (int x = 0; x < SEGS; ++x)
            if (u0 + x * SEG < k_end) sum[i] += four[x];
        }
      } else {
#pragma unroll
        for (int i = 0; i < PAIRS; ++i)
#pragma unroll
          for (int x = 0; x < SEGS; ++x) {
            const float v = __shfl_sync(0xffffffffu, one[i], (lane & ~3) | x);
            if (u0 + x * SEG < k_end) sum[i] += v;
          }
      }
    }
    if (++step < steps) continue;
    step = 0;
#pragma unroll
    for (int i = 0; i < MINE; ++i) {
      const int pair = EXCHANGED ? (seg & 1) * (PAIRS / 2) + (seg >> 1) * MINE + i : i;
      if (EXCHANGED || i % TT == seg) met[(warp * TT + pair % TT) * ROWS + pair / TT * 8 + row] = sum[i];
      sum[i] = 0.0f;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < tokens * ROWS; e += blockDim.x) {
      const int t = e / ROWS, n = n0 + e % ROWS;
      if (n >= N) continue;
      float* y = Y + (size_t)t * ldy + n;
      float v = accumulate ? *y + met[e] : met[e];
      for (int g = 1; g < ranges; ++g) v += met[g * TT * ROWS + e];
      *y = v;
    }
    __syncthreads();
    n0 += (int)gridDim.x * ROWS;
  }
}

// ---- many tokens -------------------------------------------------------------------------------------------------
// A block of 128 threads makes a tile of 64 tokens x 128 rows, 8 x 8 of it a thread: operands lie in shared memory as
// they lie in memory, [row][32 k] with 16 bytes of padding, and are read 4 k at a time (a thread's rows are 8 or 16
// apart, so the eight lanes of a phase read eight different banks, or one address): 16 16-byte loads feed 256 fused
// multiply-adds.  Two stages by asynchronous copies, two blocks an SM.  A segment's sums are in registers, the range's
// in shared memory (with both in registers the 255 that a thread has did not hold the operands: spilled, the kernel
// took 1.7 x as long).  Where the tiles leave SMs idle, the blocks of a cluster take ranges of k each and add them up
// in order through each other's shared memory.
constexpr int BM = 64, BN = 128, BK = 32, BLD = BK + 4, BT = 128;
constexpr int STAGE_FLOATS = (BM + BN) * BLD;
constexpr int TILE_SMEM = (2 * STAGE_FLOATS + BM * BN) * 4;

template <bool VEC>
__global__ void __launch_bounds__(BT, 2) gemm_f32_tile_kernel(const float* __restrict__ X, const float* __restrict__ W,
                                                              float* __restrict__ Y, int T, int N, int K, int ldx,
                                                              int ldy, int accumulate, int split) {
  extern __shared__ __align__(16) float smem[];
  float4* sums = reinterpret_cast<float4*>(smem + 2 * STAGE_FLOATS);   // [16][thread]: quarters of a thread's 8 rows
  const int rank = (int)blockIdx.x % split, n0 = ((int)blockIdx.x / split) * BN, t0 = (int)blockIdx.y * BM;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int m1 = (warp & 1) * 4 + (lane >> 3), n1 = (warp >> 1) * 8 + (lane & 7);   // rows m1 + 8 i, n1 + 16 j
  const int range = range_of(K), ranges = (K + range - 1) / range;

  // rows past the last one repeat it, their sums are dropped; what lies past the end of K is zero in both operands
  const int lr = threadIdx.x / (BK / 4), lc = (threadIdx.x % (BK / 4)) * 4;
  auto load = [&](int k0, int stage) {
    float* dst = smem + stage * STAGE_FLOATS;
    if (VEC) {
      const int k = k0 + lc, bytes = k < K ? 16 : 0;
#pragma unroll
      for (int i = 0; i < BM / 16; ++i)
        async16_or_zero(dst + (lr + 16 * i) * BLD + lc, X + (size_t)min(t0 + lr + 16 * i, T - 1) * ldx + (bytes ? k : 0), bytes);
#pragma unroll
      for (int i = 0; i < BN / 16; ++i)
        async16_or_zero(dst + (BM + lr + 16 * i) * BLD + lc, W + (size_t)min(n0 + lr + 16 * i, N - 1) * K + (bytes ? k : 0), bytes);
    } else {
      for (int e = threadIdx.x; e < (BM + BN) * BK; e += BT) {
        const int r = e / BK, k = k0 + e % BK, bytes = k < K ? 4 : 0;
        const float* src = r < BM ? X + (size_t)min(t0 + r, T - 1) * ldx : W + (size_t)min(n0 + r - BM, N - 1) * K;
        async4_or_zero(dst + r * BLD + e % BK, src + (bytes ? k : 0), bytes);
      }
    }
  };

  jb::pdl_launch_dependents();
  jb::pdl_wait();
  for (int round = 0; round * split < ranges; ++round) {
    const int k_begin = (round * split + rank) * range, k_end = min(K, k_begin + range);
    const int chunks = k_end > k_begin ? (k_end - k_begin + BK - 1) / BK : 0;
    Pair acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0;
    if (chunks > 0) load(k_begin, 0);
    async_commit();
    for (int c = 0; c < chunks; ++c) {
      if (c + 1 < chunks) load(k_begin + (c + 1) * BK, (c + 1) & 1);
      async_commit();
      async_wait<1>();
      __syncthreads();
      const float* xs = smem + (c & 1) * STAGE_FLOATS + m1 * BLD;
      const float* ws = smem + (c & 1) * STAGE_FLOATS + (BM + n1) * BLD;
#pragma unroll
      for (int k = 0; k < BK; k += 4) {
        ulonglong2 a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(xs + 8 * i * BLD + k);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ws + 16 * j * BLD + k);
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i][j] = fma2(a[i].x, b.x, acc[i][j]);
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i][j] = fma2(a[i].y, b.y, acc[i][j]);
        }
      }
      __syncthreads();
      if ((c + 1) % (SEG / BK) == 0 || c + 1 == chunks) {      // a segment joins the range
        const bool first = c < SEG / BK;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          Pair* p = &acc[q >> 1][(q & 1) * 4];
          float4 v = make_float4(even_and_odd(p[0]), even_and_odd(p[1]), even_and_odd(p[2]), even_and_odd(p[3]));
          p[0] = p[1] = p[2] = p[3] = 0;
          if (!first) {
            const float4 u = sums[q * BT + threadIdx.x];
            v = make_float4(u.x + v.x, u.y + v.y, u.z + v.z, u.w + v.w);
          }
          sums[q * BT + threadIdx.x] = v;
        }
      }
    }
    // the blocks of a cluster each add up their share of the tile's rows over the ranges of this round
    const int here = min(split, ranges - round * split);
    auto store = [&](int q, auto part_of) {
      const int t = t0 + m1 + 8 * (q >> 1);
      float4 v = part_of(0);
      if (t >= T) return;
      float* y = Y + (size_t)t * ldy;
      const bool joins = accumulate || round > 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + n1 + 16 * ((q & 1) * 4 + j);
        float& f = j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w;
        if (joins && n < N) f = y[n] + f;
      }
      for (int g = 1; g < here; ++g) {
        const float4 u = part_of(g);
        v = make_float4(v.x + u.x, v.y + u.y, v.z + u.z, v.w + u.w);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int n = n0 + n1 + 16 * ((q & 1) * 4 + j);
        if (n < N) y[n] = j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w;
      }
    };
    if (split == 1) {
#pragma unroll
      for (int q = 0; q < 16; ++q) store(q, [&](int) { return sums[q * BT + threadIdx.x]; });
      continue;
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int q = rank; q < 16; q += split)
      store(q, [&](int g) { return cluster.map_shared_rank(sums, g)[q * BT + threadIdx.x]; });
    cluster.sync();                                            // nobody's sums are overwritten or gone while they are read
  }
}

template <int TT>
int launch_stream(const float* X, const float* W, float* Y, int T, int N, int K, int ldx, int ldy, int accumulate,
                  cudaStream_t stream) {
  auto* fn = gemm_f32_stream_kernel<TT>;
  const int rows = 8 * RL, blocks = (N + rows - 1) / rows, range = range_of(K), ranges = (K + range - 1) / range;
  const size_t smem = 4 * (size_t)(RANGES * TT * rows + ranges * STAGES * (rows + TT) * SEGS * PIECE);
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int resident = 148 * (int)((size_t)(227 * 1024) / (smem + 1024));
  jb::Launch l(dim3(blocks < resident ? blocks : resident, (T + TT - 1) / TT), dim3(32 * ranges), smem, stream);
  return (int)cudaLaunchKernelEx(&l.c, fn, X, W, Y, T, N, K, ldx, ldy, accumulate);
}

}  // namespace

JB_EXPORT int jb_gemm_f32(const float* X, const float* W, float* Y, int T, int N, int K, int ldx, int ldy,
                          int accumulate, cudaStream_t stream) {
  if (T <= 0 || N <= 0) return 0;
  JB_REFUSE(K <= 0, "gemm_f32: K must be positive, got %d", K);
  // rows of whole 16-byte vectors (K and the rows' starts)
  const bool vec = K % 4 == 0 && ldx % 4 == 0 && (((uintptr_t)X | (uintptr_t)W) & 15) == 0;
  const int tiles = ((N + BN - 1) / BN) * ((T + BM - 1) / BM);
  // The streaming kernel asks for the weights once for every 8 tokens, the tiles need some of them to fill the SMs.  Streamed and
  // tiles from cold memory, microseconds, K = 2,048, before the sums met in fewer shuffles (5 % less since, from 5 tokens on): 16
  // tokens 2,048 rows 20 and 39, 8,192 rows 50 and 82, 32,000 rows 172 and 233; 24 tokens 27 and 39, 72 and 82, 250 and 233 (16,384 rows 133 and 143, 4,096 rows 43 and 41); 32 tokens 33 and 39, 92
  // and 82, 332 and 235 (2,560 rows 39 and 39; 2,048 rows of 8,192 90 and 123); 40 tokens of 2,048 rows 39 and 39.
  if (vec && (T <= 24 || (T <= 32 && N <= 20 * BN))) {
#define JB_GO(TT) return launch_stream<TT>(X, W, Y, T, N, K, ldx, ldy, accumulate, stream)
    if (T == 1) JB_GO(1);
    if (T == 2) JB_GO(2);
    if (T <= 4) JB_GO(4);
    JB_GO(8);                                                  // more than 8: in portions, each streams the weights
#undef JB_GO
  }
  // how many blocks share a tile: what takes the fewest waves of two blocks an SM for the whole, and no more of them
  const int range = range_of(K), ranges = (K + range - 1) / range;
  int split = 1;
  float best = 1e30f;
  for (int s = 1; s <= ranges; s *= 2) {
    const float waves = (float)(((long long)tiles * s + 295) / 296) * (float)((ranges + s - 1) / s);
    if (waves < 0.95f * best) best = waves, split = s;
  }
  auto* fn = vec ? gemm_f32_tile_kernel<true> : gemm_f32_tile_kernel<false>;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, TILE_SMEM);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((N + BN - 1) / BN * split, (T + BM - 1) / BM);
  c.blockDim = dim3(BT);
  c.dynamicSmemBytes = TILE_SMEM;
  c.stream = stream;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeClusterDimension;
  attrs[0].val.clusterDim.x = split;
  attrs[0].val.clusterDim.y = 1;
  attrs[0].val.clusterDim.z = 1;
  attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attrs[1].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = attrs;
  c.numAttrs = jb::pdl_enabled() ? 2 : 1;
  return (int)cudaLaunchKernelEx(&c, fn, X, W, Y, T, N, K, ldx, ldy, accumulate, split);
}
