// Recurrences with a matrix state per head and one decay a token and head, for prompts, by chunks of 32 tokens:
//
//   S_t = a_t S_(t-1) + b_t k_t v_t^T,   y_t = scale S_t^T q_t        (S [d][e], query/key head j = h / (H / G))
//
// With L_t the sum of log a up to token t of a chunk that starts from state S,
//   y_t = scale (exp(L_t) S^T q_t + sum over s <= t of exp(L_t - L_s) b_s (q_t . k_s) v_s),
//   S  <- exp(L_end) S + sum over t of exp(L_end - L_t) b_t k_t v_t^T,
// so what a token-by-token walk does in d x e steps of its own are three small products a chunk.  `state_prepare_kernel`
// (a block per chunk and key head, all chunks side by side) makes P[t][s] = scale exp(L_t - L_s) b_s (q_t . k_s), which knows
// nothing of the state, and the tokens' scales; `state_chunks_kernel` (a block per sequence, head and 64 value columns, the
// state in shared memory) walks the chunks: [exp(L) q, P] [S; v] is one product, whose sums two halves of the block share,
// then the state's update.  A thread has four by four outputs and eight rows by four columns of the state; sums go in pairs
// of neighbouring rows (packed multiply-adds).  Bound by what shared memory delivers (84% of its rate with all SMs full; the
// multiply-adds, which would bound it next, 55%).  Eight sequences of 1,024 tokens, 128 heads of 128 x 64: 2,035 us as
// segments walked token by token, 1,131 so; 16 heads of 128 x 128 with a matrix memory 1,338 and 426; 16 columns a block,
// for which every q and k is read four times as often, took 1.3 and 1.4 times as long.
// All float32 but for the sums L and their differences, which are float64: a sum that has passed a strong decay is large, and
// a difference of two of them would keep few digits in 32 bits.  Decays only appear as exponentials of differences of L of a
// later and an earlier token; L is of their sizes, the signs of those below zero are counted beside it (the walks take any
// number as a decay, and so do the chunks).
// Kinds: MAMBA   q = C, k = B, v = x, a = exp(-exp(A_log) dt), b = dt = softplus(raw + bias), y + D x
//        LIGHTNING q, k, v through SiLU, a one number a head, b = 1
//        CHANNEL a decay for each of a head's d key channels, b = 1 (see `channel_prepare_kernel`)
//        MEMORY  a, b and exp(-m) as `exp_gates` leaves them; values of one make the normalizer n (the first block of a
//                head has it beside its columns), of which the divisor max(|scale n . q|, exp(-m)) + 1e-6 is kept
#include <stdio.h>

#include "common.cuh"

namespace {

constexpr int C = 32, DMAX = 128, LD = DMAX + 4, THREADS = 256;
constexpr int P_FLOATS = C * C, SC_FLOATS = 4 * C, QK_FLOATS = 2 * C * DMAX;
constexpr float DEN_FLOOR = 1e-6f;
enum { MAMBA = 0, LIGHTNING = 1, MEMORY = 2, CHANNEL = 3 };
// scratch of a chunk and head: P, the scales, and for LIGHTNING the activated q and k; CHANNEL: P, the chunk's decay of every
// channel, and the weighted q and k
__host__ __device__ constexpr bool keeps_qk(int kind) { return kind == LIGHTNING || kind == CHANNEL; }
__host__ __device__ constexpr int scratch_floats(int kind) { return P_FLOATS + SC_FLOATS + (keeps_qk(kind) ? QK_FLOATS : 0); }
static_assert(SC_FLOATS == DMAX, "a chunk's decays of all channels take the place of the scales");

__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float4 silu4(float4 z) { return make_float4(silu(z.x), silu(z.y), silu(z.z), silu(z.w)); }

struct Args {
  const float* proj;      // rows of ld: q, k and v at their columns
  int ld, q_col, k_col, v_col;
  const float* gates;     // MAMBA: raw dt, rows of ld_gates; MEMORY: [T][H][4] of a, b, exp(-m); CHANNEL: [T][H d] of a
  int ld_gates;
  const float* rate;      // MAMBA: A_log [H]; LIGHTNING: a [H]
  const float* bias;      // MAMBA: dt_bias [H]
  const float* skip;      // MAMBA: D [H]
  float scale;
  float* out;             // [T][H e]
  float* den;             // MEMORY: [T][H]
  float* state;
  long long slot_stride, state_off;
  const int* q_start;
  const int* seq_slot;
  int H, G, d, e;
  float* scratch;
  int n_seqs, first_tile, tiles, heads_here, packed;
};

// Where the scratch of a sequence's first chunk lies, in chunks: `tiles` a sequence, or (packed) as many as it needs, one
// sequence after another: floor(q_start / C) + seq begins at or past the end of the sequence before.
__device__ __forceinline__ int first_slot(const Args& a, int seq) { return a.packed ? a.q_start[seq] / C + seq : seq * a.tiles; }

// The chunk of a block of a prepare kernel: its first token and how many it has (none: n <= 0).
__device__ __forceinline__ void find_chunk(const Args& a, int& t0, int& n) {
  int seq = (int)blockIdx.x / a.tiles, tile = (int)blockIdx.x % a.tiles;
  if (a.packed) {                                              // the last sequence whose chunks begin up to here
    seq = -1;
    for (int s0 = 0; s0 < a.n_seqs; s0 += THREADS) {
      const int s = s0 + (int)threadIdx.x;
      seq += __syncthreads_count(s < a.n_seqs && first_slot(a, s) <= (int)blockIdx.x);
    }
    tile = (int)blockIdx.x - first_slot(a, seq);
  }
  t0 = a.q_start[seq] + (a.first_tile + tile) * C, n = min(C, a.q_start[seq + 1] - t0);
}

template <int KIND>
__global__ void __launch_bounds__(THREADS) state_prepare_kernel(const Args a) {
  __shared__ __align__(16) float q_s[C][LD], k_s[C][LD];
  __shared__ float qk_s[C][C + 1];
  jb::pdl_launch_dependents();
  const int R = a.H / a.G, j = blockIdx.y;
  const int h_begin = j * R + (int)blockIdx.z * a.heads_here, h_end = min((j + 1) * R, h_begin + a.heads_here);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  jb::pdl_wait();
  int t0, n;
  find_chunk(a, t0, n);
  if (n <= 0) return;
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float4 qv[4], kv[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int t = 4 * warp + u;
    const bool in = t < n && 4 * lane < a.d;
    const float* row = a.proj + (size_t)(t0 + (t < n ? t : 0)) * a.ld + (size_t)j * a.d + (in ? 4 * lane : 0);
    qv[u] = in ? *reinterpret_cast<const float4*>(row + a.q_col) : zero;
    kv[u] = in ? *reinterpret_cast<const float4*>(row + a.k_col) : zero;
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int t = 4 * warp + u;
    if (KIND == LIGHTNING) {                                   // (silu(0) is 0)
      qv[u] = silu4(qv[u]), kv[u] = silu4(kv[u]);
      float* QK_g = a.scratch + ((size_t)blockIdx.x * a.H + j) * scratch_floats(KIND) + P_FLOATS + SC_FLOATS;   // G = H here
      *reinterpret_cast<float4*>(QK_g + t * DMAX + 4 * lane) = qv[u];
      *reinterpret_cast<float4*>(QK_g + (C + t) * DMAX + 4 * lane) = kv[u];
    }
    *reinterpret_cast<float4*>(&q_s[t][4 * lane]) = qv[u];
    *reinterpret_cast<float4*>(&k_s[t][4 * lane]) = kv[u];
  }
  __syncthreads();
  {
    jb::Pair qk[2][2] = {{0, 0}, {0, 0}};                      // two by two entries a thread; above the diagonal nobody reads
#pragma unroll 4
    for (int r = 0; r < DMAX; r += 4) {
      ulonglong2 b[2], c[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        b[x] = *reinterpret_cast<const ulonglong2*>(&q_s[ty + 16 * x][r]);
        c[x] = *reinterpret_cast<const ulonglong2*>(&k_s[tx + 16 * x][r]);
      }
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y <= x; ++y) qk[x][y] = jb::fma2(b[x].y, c[y].y, jb::fma2(b[x].x, c[y].x, qk[x][y]));
    }
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 2; ++y) qk_s[ty + 16 * x][tx + 16 * y] = jb::lo(qk[x][y]) + jb::hi(qk[x][y]);
  }
  __syncthreads();
  for (int h = h_begin + warp; h < h_end; h += THREADS / 32) { // a head a warp, a token a lane
    float log_a = 0.0f, b = 0.0f, floor = 0.0f;
    bool turns = false;                                        // a decay below zero turns the state's sign
    if (lane < n) {
      const size_t t = (size_t)(t0 + lane);
      if (KIND == MAMBA) {
        const float z = a.gates[t * a.ld_gates + h] + a.bias[h];
        b = z > 20.0f ? z : log1pf(expf(z));
        log_a = -expf(a.rate[h]) * b;
      } else if (KIND == LIGHTNING) {
        b = 1.0f;
        turns = a.rate[h] < 0.0f, log_a = logf(fabsf(a.rate[h]));
      } else {
        const float* g = a.gates + (t * a.H + h) * 4;
        turns = g[0] < 0.0f, log_a = logf(fabsf(g[0])), b = g[1], floor = g[2];
      }
      log_a = log_a < -10000.0f ? -10000.0f : log_a;           // a decay of zero; the sums stay finite (and NaN stays NaN)
    }
    double L = log_a;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double before = __shfl_up_sync(0xffffffffu, L, o);
      if (lane >= o) L += before;
    }
    const double end = __shfl_sync(0xffffffffu, L, 31);
    unsigned turned = KIND == MAMBA ? 0u : __ballot_sync(0xffffffffu, turns);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) turned ^= turned << o;                  // bit t: whether the turns up to token t are odd
    const auto decay = [](double log, unsigned odd) { return __uint_as_float(__float_as_uint(expf((float)log)) ^ odd << 31); };
    float* P_g = a.scratch + ((size_t)blockIdx.x * a.H + h) * scratch_floats(KIND);
    // per token: what multiplies q_t S, what multiplies k_t on its way into the state, the chunk's decay, exp(-m)
    reinterpret_cast<float4*>(P_g + P_FLOATS)[lane] = make_float4(decay(L, turned >> lane) * a.scale, decay(end - L, turned >> 31 ^ turned >> lane) * b, decay(end, turned >> 31), floor);
#pragma unroll 8
    for (int t = 0; t < C; ++t) {
      const double Lt = __shfl_sync(0xffffffffu, L, t);
      P_g[t * C + lane] = lane <= t ? decay(Lt - L, turned >> t ^ turned >> lane) * b * a.scale * qk_s[t][lane] : 0.0f;
    }
  }
}

// CHANNEL.  Products of decays stand where the other kinds have exponentials of sums: along the tokens, as a walk makes them, so
// that decays of zero, below zero and not a number need no case, and nothing is divided by.  q_t goes with the product from
// the chunk's start to its own token, k_t with the one from the next token to the chunk's end, both products in float64.
// P[t][s] = scale q_t . (k_s times what lies between): half a warp owns a token s (and then 31 - s, so that all warps have as
// much to do), eight channels a lane, and takes its k along the later tokens; from the end of its four tokens on by products of
// the four and of their first ones, made in float64 too, which leaves twelve roundings where token by token there were 31.
// Four tokens' sums meet in five shuffles.  Eight sequences of 40 to 511 tokens, 16 heads of 128 x 128: 435 us as segments walked
// token by token, 214 by chunks, one of 256 tokens 104 and 62; errors against float64, relative to all outputs and to the state,
// 1.14e-7 and 7.8e-8 by the walk, 1.10e-7 to 1.12e-7 and 7.2e-8 to 7.9e-8 so (1.21e-7 and 9.9e-8 with float32 products throughout).
constexpr int CHANNEL_SMEM = (3 * C * DMAX + C * (C + 4)) * 4;
__global__ void __launch_bounds__(THREADS) channel_prepare_kernel(const Args a) {
  extern __shared__ __align__(16) float smem[];
  float(*q_s)[DMAX] = reinterpret_cast<float(*)[DMAX]>(smem), (*k_s)[DMAX] = q_s + C, (*a_s)[DMAX] = k_s + C;
  float* P_s = smem + 3 * C * DMAX;
  jb::pdl_launch_dependents();
  const int h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  jb::pdl_wait();
  int t0, n;
  find_chunk(a, t0, n);
  if (n <= 0) return;
#pragma unroll
  for (int u = 0; u < 4; ++u) {                                // past the sequence's end and the keys': nothing, kept as it is
    const int t = 4 * warp + u;
    const bool in = t < n && 4 * lane < a.d;
    const size_t row = (size_t)(t0 + (in ? t : 0)), c = (size_t)h * a.d + (in ? 4 * lane : 0);
    float4 q = make_float4(0.0f, 0.0f, 0.0f, 0.0f), k = q, w = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    if (in) {
      q = *reinterpret_cast<const float4*>(a.proj + row * a.ld + a.q_col + c);
      k = *reinterpret_cast<const float4*>(a.proj + row * a.ld + a.k_col + c);
      w = *reinterpret_cast<const float4*>(a.gates + row * a.ld_gates + c);
    }
    *reinterpret_cast<float4*>(&q_s[t][4 * lane]) = make_float4(q.x * a.scale, q.y * a.scale, q.z * a.scale, q.w * a.scale);
    *reinterpret_cast<float4*>(&k_s[t][4 * lane]) = k;
    *reinterpret_cast<float4*>(&a_s[t][4 * lane]) = w;
  }
  __syncthreads();
  float* P_g = a.scratch + ((size_t)blockIdx.x * a.H + h) * scratch_floats(CHANNEL);
  float* Q_g = P_g + P_FLOATS + SC_FLOATS;
  const int g = lane & 15, half = lane >> 4;
  const int first[2] = {2 * warp, 30 - 2 * warp}, own[2] = {2 * warp + half, 31 - 2 * warp - half};
  ulonglong2 r[2][2];                                          // k of the two tokens: channels 4 g and on, 64 + 4 g and on
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int y = 0; y < 2; ++y) r[p][y] = *reinterpret_cast<const ulonglong2*>(&k_s[own[p]][64 * y + 4 * g]);
  __syncthreads();                                             // k's place is taken below
  {
    const int c = threadIdx.x & (DMAX - 1);
    double w = 1.0;
    if (threadIdx.x < DMAX) {
#pragma unroll 8
      for (int t = 0; t < C; ++t) w *= a_s[t][c], Q_g[t * DMAX + c] = (float)(q_s[t][c] * w);
      P_g[P_FLOATS + c] = (float)w;
    } else {
#pragma unroll 2
      for (int t = C - 4; t >= 0; t -= 4) {
        double four[4];                                        // decays, then their products from the first of the four
#pragma unroll
        for (int u = 3; u >= 0; --u) four[u] = a_s[t + u][c], Q_g[(C + t + u) * DMAX + c] = (float)(k_s[t + u][c] * w), w *= four[u];
#pragma unroll
        for (int u = 0; u < 4; ++u) four[u] = u > 0 ? four[u - 1] * four[u] : four[0], k_s[t + u][c] = (float)four[u];
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int s = own[p];
    for (int tb = first[p] & ~3; tb < C; tb += 4) {
      float sum[4];
      const bool here = tb <= s;                               // s is one of the four (of all the warp, or of none)
      ulonglong2 now[2] = {r[p][0], r[p][1]};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int t = tb + u;
        jb::Pair acc = 0;
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(&(here ? a_s : k_s)[t][64 * y + 4 * g]);
          const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(&q_s[t][64 * y + 4 * g]);
          const ulonglong2 from = here ? now[y] : r[p][y];
          if (t > s) now[y] = make_ulonglong2(jb::mul2(from.x, w.x), jb::mul2(from.y, w.y));
          acc = jb::fma2(q.y, now[y].y, jb::fma2(q.x, now[y].x, acc));
        }
        sum[u] = jb::lo(acc) + jb::hi(acc);
      }
      r[p][0] = now[0], r[p][1] = now[1];
      const bool up8 = g & 8, up4 = g & 4;
      float x = (up8 ? sum[2] : sum[0]) + __shfl_xor_sync(0xffffffffu, up8 ? sum[0] : sum[2], 8);
      const float y = (up8 ? sum[3] : sum[1]) + __shfl_xor_sync(0xffffffffu, up8 ? sum[1] : sum[3], 8);
      x = (up4 ? y : x) + __shfl_xor_sync(0xffffffffu, up4 ? x : y, 4);
      x += __shfl_xor_sync(0xffffffffu, x, 2);
      x += __shfl_xor_sync(0xffffffffu, x, 1);
      if ((g & 3) == 0) P_s[(tb + (g >> 2)) * (C + 4) + s] = x;
    }
  }
  __syncthreads();
  const int t = threadIdx.x >> 3, s = (threadIdx.x & 7) * 4;   // what lies above the diagonal is not there (and may be old)
  float4 x = *reinterpret_cast<const float4*>(P_s + t * (C + 4) + s);
  x.x = s <= t ? x.x : 0.0f, x.y = s + 1 <= t ? x.y : 0.0f, x.z = s + 2 <= t ? x.z : 0.0f, x.w = s + 3 <= t ? x.w : 0.0f;
  *reinterpret_cast<float4*>(P_g + t * C + s) = x;
}

// copies 16 bytes, or zeros
__device__ __forceinline__ void async16(float* dst, const float* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 16 : 0));
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;"); }

constexpr int COLS = 64, SLD = 2 * COLS + 4;   // columns of a block; floats of a pair of the state's rows, and padding
constexpr int VLD = COLS + 4;
constexpr int HAND_FLOATS = 4 * 3 * 128 * 4;   // what four parts of a block hand one another
template <int KIND, int D, int SPLIT>
constexpr int chunk_smem() {
  return (3 * C * (D + 4) + 2 * C * (C + 4) + 2 * SC_FLOATS + (D + C) / 2 * SLD + C * VLD + (KIND == MEMORY ? D : 0) +
          (SPLIT > 2 ? HAND_FLOATS : 0)) * 4;
}

// D: keys' numbers at most.  SPLIT times four warps: four of 16 columns for each part of the sums over keys and tokens.  Two
// parts, two blocks an SM; where no SM has a second block, four parts, which shortens a chunk's chain (128 blocks, 1,024 tokens
// of four sequences of 16 heads of 128 x 128 with a matrix memory: 382 us in two parts, 244 in four; one sequence of 256
// tokens 96 and 64).
template <int KIND, int D, int SPLIT>
__global__ void __launch_bounds__(128 * SPLIT, 4 / SPLIT) state_chunks_kernel(const Args a) {
  constexpr int LDD = D + 4, THREADS = 128 * SPLIT, RT = D / (8 * SPLIT);  // RT: the state's rows a thread updates, of four columns
  constexpr int VL = THREADS / C, OWN = 4 / SPLIT;                         // lanes of a token's values; tokens a thread keeps
  extern __shared__ __align__(16) float smem[];
  __shared__ int wild_s;                       // whether a value was not finite
  float* q_b = smem;                           // two buffers of q [C][LDD]
  float* k_s = q_b + 2 * C * LDD;              // k [C][LDD]
  float* P_b = k_s + C * LDD;                  // two buffers of P [C][C + 4]
  float4* sc_b = reinterpret_cast<float4*>(P_b + 2 * C * (C + 4));         // two buffers of the scales [C]
  float* S_s = P_b + 2 * C * (C + 4) + 2 * SC_FLOATS;                      // [D / 2][SLD]: two rows of a column are neighbours
  float* v_s = S_s + D / 2 * SLD;              // the values (the finite ones), laid out as more rows of the state
  float* vk_s = v_s + C / 2 * SLD;             // the values as they join the state [C][VLD]
  float* n_s = vk_s + C * VLD;                 // MEMORY: the normalizer [D], of the first column block
  float* hand_s = n_s + (KIND == MEMORY ? D : 0);
  jb::pdl_launch_dependents();
  const int seq = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * COLS, H = a.H, d = a.d, e = a.e, j = h / (H / a.G);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool pairs = ((e | a.v_col) & 1) == 0 && ((uintptr_t)a.out & 7) == 0;          // columns go two at a time
  const bool has_n = KIND == MEMORY && blockIdx.x == 0;
  if (tid == 0) wild_s = 0;
  __syncthreads();
  jb::pdl_wait();
  const int begin = a.q_start[seq] + a.first_tile * C, n_all = min(a.q_start[seq + 1] - begin, a.tiles * C);
  if (n_all <= 0) return;
  float* S_g = a.state + (size_t)a.seq_slot[seq] * a.slot_stride + a.state_off + (size_t)h * d * (e + (KIND == MEMORY ? 1 : 0));
  const float* scratch_g = a.scratch + ((size_t)first_slot(a, seq) * H + h) * scratch_floats(KIND);
  const size_t per_chunk = (size_t)H * scratch_floats(KIND);
  const int chunks = (n_all + C - 1) / C;

  auto load_rows = [&](float* dst, int chunk, int col, int which) {
    const int t0 = begin + chunk * C, n = min(C, n_all - chunk * C);
    for (int i = tid; i < C * D / 4; i += THREADS) {
      const int t = i / (D / 4), r = (i % (D / 4)) * 4;
      if (keeps_qk(KIND)) {
        async16(dst + t * LDD + r, scratch_g + chunk * per_chunk + P_FLOATS + SC_FLOATS + (which * C + t) * DMAX + r, true);
      } else {
        const bool in = t < n && r < d;
        async16(dst + t * LDD + r, a.proj + (size_t)(t0 + (in ? t : 0)) * a.ld + col + (size_t)j * d + (in ? r : 0), in);
      }
    }
  };
  auto load_qp = [&](int chunk) {
    if (chunk < chunks) {
      load_rows(q_b + (chunk & 1) * C * LDD, chunk, a.q_col, 0);
      const float* P_g = scratch_g + chunk * per_chunk;
      if (tid < P_FLOATS / 4) async16(P_b + (chunk & 1) * C * (C + 4) + (tid / 8) * (C + 4) + (tid % 8) * 4, P_g + tid * 4, true);     // 256 pieces
      if (tid < C) async16(reinterpret_cast<float*>(sc_b + (chunk & 1) * C + tid), P_g + P_FLOATS + 4 * tid, true);
    }
    commit();
  };
  auto load_k = [&](int chunk) {
    if (chunk < chunks) load_rows(k_s, chunk, a.k_col, 1);
    commit();
  };
  // values: a thread two neighbouring columns of every 2 VL of a token, and what the token's key is worth, a chunk ahead
  const int vt = tid / VL, vc = (tid % VL) * 2;
  float2 v[COLS / (2 * VL)];
  float v_scale;
  auto fetch_v = [&](int chunk) {
    const bool in = vt < n_all - chunk * C;
    const float* row = a.proj + (size_t)(begin + chunk * C + (in ? vt : 0)) * a.ld + a.v_col + (size_t)h * e;
    v_scale = KIND == CHANNEL ? 1.0f : chunk < chunks ? scratch_g[chunk * per_chunk + P_FLOATS + 4 * vt + 1] : 0.0f;
#pragma unroll
    for (int i = 0; i < COLS / (2 * VL); ++i) {
      const int c = c0 + 2 * VL * i + vc;
      v[i] = make_float2(0.0f, 0.0f);
      if (in && pairs && c < e) v[i] = *reinterpret_cast<const float2*>(row + c);
      if (in && !pairs) v[i] = make_float2(c < e ? row[c] : 0.0f, c + 1 < e ? row[c + 1] : 0.0f);
    }
  };
  auto store_v = [&] {
    float nothing = 0.0f;                      // zero, or NaN where a value is not finite
#pragma unroll
    for (int i = 0; i < COLS / (2 * VL); ++i) {
      if (KIND == LIGHTNING) v[i] = make_float2(silu(v[i].x), silu(v[i].y));
      float* at = v_s + (vt >> 1) * SLD + 2 * (2 * VL * i + vc) + (vt & 1);
      at[0] = v[i].x, at[2] = v[i].y;
      *reinterpret_cast<float2*>(vk_s + vt * VLD + 2 * VL * i + vc) = make_float2(v[i].x * v_scale, v[i].y * v_scale);
      nothing = fmaf(v[i].x, 0.0f, fmaf(v[i].y, 0.0f, nothing));
    }
    if (nothing != 0.0f) {                     // such values stay out of the product with P, see the end
      wild_s = 1;
#pragma unroll
      for (int i = 0; i < COLS / (2 * VL); ++i) {
        float* at = v_s + (vt >> 1) * SLD + 2 * (2 * VL * i + vc) + (vt & 1);
        if (!isfinite(v[i].x)) at[0] = 0.0f;
        if (!isfinite(v[i].y)) at[2] = 0.0f;
      }
    }
  };
  load_qp(0);
  load_k(0);
  fetch_v(0);
  for (int i = tid; i < D * COLS; i += THREADS) {
    const int r = i / COLS, c = i % COLS;
    S_s[(r >> 1) * SLD + 2 * c + (r & 1)] = (r < d && c0 + c < e) ? S_g[(size_t)r * e + c0 + c] : 0.0f;
  }
  if (has_n && tid < D) n_s[tid] = tid < d ? S_g[(size_t)d * e + tid] : 0.0f;
  store_v();

  // outputs: a thread four tokens tg + 8 i and four columns, col[x] and the one after it, over one part of the sums
  const int part = warp >> 2, tg = lane >> 2;
  const int col[2] = {16 * (warp & 3) + 2 * (lane & 3), 16 * (warp & 3) + 8 + 2 * (lane & 3)};
  // state's update: a thread RT rows, columns uc, uc + 1, uc + 16 and uc + 17
  const int ur = ((warp >> 1) * 4 + (lane >> 3)) * RT, uc = (warp & 1) * 32 + 2 * (lane & 7);
  const float skip = KIND == MAMBA ? a.skip[h] : 0.0f;

  for (int chunk = 0; chunk < chunks; ++chunk) {
    const int t0 = begin + chunk * C, n = min(C, n_all - chunk * C);
    // copies in flight, oldest first: q and P of this chunk, k of it
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();                                                       // values and state are whole too
    load_qp(chunk + 1);
    fetch_v(chunk + 1);
    float* q_s = q_b + (chunk & 1) * C * LDD;
    const float* P_s = P_b + (chunk & 1) * C * (C + 4);
    const float4* sc_s = sc_b + (chunk & 1) * C;
    float o[4][4];
    {
      jb::Pair acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[i][x] = 0;
      // four numbers of the rows' left factors at L, of which the right ones lie at R
      const auto step = [&](const float* L, int ld, const float* R) {
        ulonglong2 l4[4], b[2][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) l4[i] = *reinterpret_cast<const ulonglong2*>(L + (tg + 8 * i) * ld);
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
          for (int x = 0; x < 2; ++x) b[y][x] = *reinterpret_cast<const ulonglong2*>(R + y * SLD + 2 * col[x]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            acc[i][2 * x] = jb::fma2(l4[i].y, b[1][x].x, jb::fma2(l4[i].x, b[0][x].x, acc[i][2 * x]));
            acc[i][2 * x + 1] = jb::fma2(l4[i].y, b[1][x].y, jb::fma2(l4[i].x, b[0][x].y, acc[i][2 * x + 1]));
          }
      };
#pragma unroll 2
      for (int k = part * (D / SPLIT); k < (part + 1) * (D / SPLIT); k += 4) step(q_s + k, LDD, S_s + (k >> 1) * SLD);
#pragma unroll
      for (int i = 0; i < 4 && KIND != CHANNEL; ++i) {                     // (CHANNEL: q has its scale)
        const float s = sc_s[tg + 8 * i].x;
        const jb::Pair ss = jb::pair(s, s);
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[i][x] = jb::mul2(acc[i][x], ss);
      }
#pragma unroll 2
      for (int s = part * (C / SPLIT); s < (part + 1) * (C / SPLIT); s += 4) step(P_s + s, C + 4, v_s + (s >> 1) * SLD);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int x = 0; x < 4; ++x) o[i][x] = jb::lo(acc[i][x]) + jb::hi(acc[i][x]);
    }
    if (KIND == MAMBA) {                                                   // D x, by the part that keeps the token
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i / OWN == part) {
          const int t = tg + 8 * i;
#pragma unroll
          for (int x = 0; x < 4; ++x) o[i][x] = fmaf(skip, v_s[(t >> 1) * SLD + 2 * (col[x >> 1] + (x & 1)) + (t & 1)], o[i][x]);
        }
    }
    if (has_n) {                                                           // divisors: VL lanes a token
      const int l = tid % VL;
      float dot = 0.0f, ones = 0.0f;
#pragma unroll
      for (int r = 4 * l; r < D; r += 4 * VL) {
        const float4 x = *reinterpret_cast<const float4*>(q_s + vt * LDD + r), y = *reinterpret_cast<const float4*>(n_s + r);
        dot = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, dot))));
      }
      const float4 sc = sc_s[vt];
      if (4 * l < C) {
        const float4 p = *reinterpret_cast<const float4*>(P_s + vt * (C + 4) + 4 * l);
        ones = (p.x + p.y) + (p.z + p.w);
      }
      dot = fmaf(dot, sc.x, ones);
#pragma unroll
      for (int w = 1; w < VL; w <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, w);
      if (l == 0 && vt < n) a.den[(size_t)(t0 + vt) * H + h] = fmaxf(fabsf(dot), sc.w) + DEN_FLOOR;
    }
    // in flight: k of this chunk, q and P of the next
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();                                                       // q, P, the values and the state have been read, k is there
    // the parts meet: each keeps OWN tokens and hands the others its share of theirs (two parts: where q was)
    float4* hand = reinterpret_cast<float4*>(SPLIT > 2 ? hand_s : q_s) + (tid & 127);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int keeper = i / OWN;
      if (keeper != part) hand[128 * (i * (SPLIT - 1) + part - (part > keeper))] = make_float4(o[i][0], o[i][1], o[i][2], o[i][3]);
    }
    {
      jb::Pair S[RT / 2][4];
      const float decay = sc_s[0].z;
      const jb::Pair g = jb::pair(decay, decay);
#pragma unroll
      for (int p = 0; p < RT / 2; ++p)
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const ulonglong2 old = *reinterpret_cast<const ulonglong2*>(S_s + ((ur >> 1) + p) * SLD + 2 * (uc + 16 * x));
          S[p][2 * x] = KIND == CHANNEL ? 0 : jb::mul2(old.x, g);          // (CHANNEL: the chunk's sum by itself, see the end)
          S[p][2 * x + 1] = KIND == CHANNEL ? 0 : jb::mul2(old.y, g);
        }
#pragma unroll 4
      for (int t = 0; t < C; ++t) {
        ulonglong2 k[RT / 4];
#pragma unroll
        for (int p = 0; p < RT / 4; ++p) k[p] = *reinterpret_cast<const ulonglong2*>(k_s + t * LDD + ur + 4 * p);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const float2 w = *reinterpret_cast<const float2*>(vk_s + t * VLD + uc + 16 * x);
          const jb::Pair w0 = jb::pair(w.x, w.x), w1 = jb::pair(w.y, w.y);
#pragma unroll
          for (int p = 0; p < RT / 4; ++p) {
            S[2 * p][2 * x] = jb::fma2(k[p].x, w0, S[2 * p][2 * x]);
            S[2 * p][2 * x + 1] = jb::fma2(k[p].x, w1, S[2 * p][2 * x + 1]);
            S[2 * p + 1][2 * x] = jb::fma2(k[p].y, w0, S[2 * p + 1][2 * x]);
            S[2 * p + 1][2 * x + 1] = jb::fma2(k[p].y, w1, S[2 * p + 1][2 * x + 1]);
          }
        }
      }
#pragma unroll
      for (int p = 0; p < RT / 2; ++p)
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          ulonglong2* at = reinterpret_cast<ulonglong2*>(S_s + ((ur >> 1) + p) * SLD + 2 * (uc + 16 * x));
          if (KIND == CHANNEL) {                                           // two channels' decays
            const jb::Pair both = reinterpret_cast<const jb::Pair*>(sc_s)[(ur >> 1) + p];
            const ulonglong2 old = *at;
            S[p][2 * x] = jb::fma2(old.x, both, S[p][2 * x]), S[p][2 * x + 1] = jb::fma2(old.y, both, S[p][2 * x + 1]);
          }
          *at = make_ulonglong2(S[p][2 * x], S[p][2 * x + 1]);
        }
    }
    if (has_n && tid < D) {                                                // n <- decay n + the sum of b k
      float s = n_s[tid] * sc_s[0].z;
#pragma unroll 8
      for (int t = 0; t < C; ++t) s = fmaf(k_s[t * LDD + tid], sc_s[t].y, s);
      n_s[tid] = s;
    }
    __syncthreads();                                                       // k has been read, the parts are there
    load_k(chunk + 1);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i / OWN == part) {
        const int t = tg + 8 * i;
        float y[4] = {o[i][0], o[i][1], o[i][2], o[i][3]};
#pragma unroll
        for (int w = 0; w < SPLIT - 1; ++w) {
          const float4 more = hand[128 * (i * (SPLIT - 1) + w)];
          y[0] += more.x, y[1] += more.y, y[2] += more.z, y[3] += more.w;
        }
        if (t < n) {
          float* dst = a.out + ((size_t)(t0 + t) * H + h) * e + c0;
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int c = col[x];
            if (pairs) {
              if (c0 + c < e) *reinterpret_cast<float2*>(dst + c) = make_float2(y[2 * x], y[2 * x + 1]);
            } else {
              if (c0 + c < e) dst[c] = y[2 * x];
              if (c0 + c + 1 < e) dst[c + 1] = y[2 * x + 1];
            }
          }
        }
      }
    store_v();                                                             // the next chunk's
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  for (int i = tid; i < D * COLS; i += THREADS) {
    const int r = i / COLS, c = i % COLS;
    if (r < d && c0 + c < e) S_g[(size_t)r * e + c0 + c] = S_s[(r >> 1) * SLD + 2 * c + (r & 1)];
  }
  if (has_n && tid < d) S_g[(size_t)d * e + tid] = n_s[tid];
  if (wild_s == 0) return;
  __syncthreads();
  // P's zeros for later tokens would not have kept a value that is not finite out of the sums, so it was left out: what it
  // does to its own token and the later ones of its chunk is added here (to later chunks it came with the state)
  for (int i = tid; i < n_all * COLS; i += THREADS) {
    const int t = i / COLS, c = c0 + i % COLS, first = t / C * C;
    if (c >= e) continue;
    const float* P_g = scratch_g + (t / C) * per_chunk + (t % C) * C;
    float* dst = a.out + ((size_t)(begin + t) * H + h) * e + c;
    for (int s = first; s <= t; ++s) {
      const float raw = a.proj[(size_t)(begin + s) * a.ld + a.v_col + (size_t)h * e + c], value = KIND == LIGHTNING ? silu(raw) : raw;
      if (!isfinite(value)) *dst += P_g[s - first] * value;
    }
  }
}

template <int KIND, int D, int SPLIT>
int launch(Args a, int max_q_len, int tokens, cudaStream_t stream) {
  constexpr int smem = chunk_smem<KIND, D, SPLIT>();
  cudaError_t e = cudaFuncSetAttribute(state_chunks_kernel<KIND, D, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  constexpr int prepare_smem = KIND == CHANNEL ? CHANNEL_SMEM : 0;
  if (e == cudaSuccess && KIND == CHANNEL)
    e = cudaFuncSetAttribute(channel_prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CHANNEL_SMEM);
  if (e != cudaSuccess) return (int)e;
  const int group = a.H / a.G;
  // a block makes the products of a chunk and key head once for its group's heads, or for a share of them where that
  // leaves SMs without a block
  const int slots = a.packed ? tokens / C + a.n_seqs : a.n_seqs * a.tiles;
  const long long chunks = (a.packed ? (long long)tokens / C + 1 : slots) * a.G;       // that have tokens
  int parts = (int)((2 * 148 + chunks - 1) / chunks);
  parts = parts < group ? parts : group;
  a.heads_here = (group + parts - 1) / parts;
  for (a.first_tile = 0; a.first_tile * C < max_q_len; a.first_tile += a.tiles) {
    jb::Launch prepare(dim3(slots, a.G, (group + a.heads_here - 1) / a.heads_here), dim3(THREADS), prepare_smem, stream);
    e = cudaLaunchKernelEx(&prepare.c, KIND == CHANNEL ? channel_prepare_kernel : state_prepare_kernel<KIND == CHANNEL ? MAMBA : KIND>, a);
    if (e != cudaSuccess) return (int)e;
    jb::Launch walk(dim3((a.e + COLS - 1) / COLS, a.H, a.n_seqs), dim3(128 * SPLIT), smem, stream);
    e = cudaLaunchKernelEx(&walk.c, state_chunks_kernel<KIND, D, SPLIT>, a);
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}

}  // namespace

// kind: 0 state-space (MAMBA), 1 LIGHTNING, 2 matrix MEMORY, 3 a decay a CHANNEL, see the top.  d <= 128; d, ld, q_col and k_col multiples of 4,
// proj and scratch 16-byte aligned.  `scratch` (H * 1152 floats a chunk, LIGHTNING and CHANNEL H * 9344) holds `tiles` chunks of every
// sequence; longer prompts go in slabs of as many, one after another from the state the last left.  tiles = 0: it holds
// tokens / 32 + n_seqs chunks, the whole step's, one sequence after another (`tokens`: of all sequences).
JB_EXPORT int jb_state_chunks(int kind, const float* proj, int ld, int q_col, int k_col, int v_col, const float* gates,
                              int ld_gates, const float* rate, const float* bias, const float* skip, float scale, float* out,
                              float* den, float* state, long long slot_stride, long long state_off, const int* q_start,
                              const int* seq_slot, int n_seqs, int H, int G, int d, int e, int max_q_len, float* scratch,
                              int tiles, int tokens, cudaStream_t stream) {
  if (n_seqs <= 0 || max_q_len <= 0) return 0;
  JB_REFUSE(d < 1 || d > DMAX || e < 1 || ((d | ld | q_col | k_col) & 3) != 0 || (((uintptr_t)proj | (uintptr_t)scratch) & 15) != 0,
            "state_chunks: keys of %d numbers in rows of %d at columns %d and %d", d, ld, q_col, k_col);
  JB_REFUSE(G < 1 || H % G != 0 || tiles < 0 || (keeps_qk(kind) && G != H), "state_chunks: %d heads, %d key heads, %d tiles", H, G, tiles);
  const Args a{proj, ld, q_col, k_col, v_col, gates, ld_gates, rate, bias, skip, scale, out, den, state, slot_stride, state_off,
               q_start, seq_slot, H, G, d, e, scratch, n_seqs, 0, tiles > 0 ? tiles : (max_q_len + C - 1) / C, 0, tiles == 0};
  const bool few = (long long)n_seqs * H * ((e + COLS - 1) / COLS) <= 148;           // no SM has a second block
  const auto run = [&](auto small, auto large, auto alone) { return (d <= 64 ? small : few ? alone : large)(a, max_q_len, tokens, stream); };
  if (kind == MAMBA) return run(launch<MAMBA, 64, 2>, launch<MAMBA, 128, 2>, launch<MAMBA, 128, 4>);
  if (kind == LIGHTNING) return run(launch<LIGHTNING, 64, 2>, launch<LIGHTNING, 128, 2>, launch<LIGHTNING, 128, 4>);
  JB_REFUSE(kind == CHANNEL && ((ld_gates & 3) != 0 || ((uintptr_t)gates & 15) != 0), "state_chunks: decays in rows of %d", ld_gates);
  if (kind == CHANNEL) return run(launch<CHANNEL, 64, 2>, launch<CHANNEL, 128, 2>, launch<CHANNEL, 128, 4>);
  JB_REFUSE(kind != MEMORY, "state_chunks: kind %d", kind);
  return run(launch<MEMORY, 64, 2>, launch<MEMORY, 128, 2>, launch<MEMORY, 128, 4>);
}
