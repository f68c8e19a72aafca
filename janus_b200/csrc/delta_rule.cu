// The gated delta rule, a recurrence with a matrix state per head: a walk token by token for single tokens and short or
// unaligned portions, and chunks of 32 tokens for prompts (at the end).  All arithmetic is float32.  Per head h (query/key head j = h / (H / G)) with state S [d, e]:
//
//   q_t = u_q / sqrt(sum(u_q^2) + unit_eps) * d^-1/2,  k_t = u_k / sqrt(sum(u_k^2) + unit_eps)     (unit vectors)
//   beta_t = sigmoid(b_t),  g_t = exp(-exp(A_log_h) softplus(a_t + dt_bias_h))
//   S <- g_t S;  w = beta_t (v_t - S^T k_t);  S <- S + k_t w^T;  o_t = S^T q_t                 (the read-out sees the write)
//
// u_q, u_k, v are columns of `conv` (the projections after their short convolution and activation), b and a columns
// of `raw` (the projection as it left the product).  The state of a sequence lives at state[slot][state_off ...] as
// [H][d][e], is read at the start of a step and written back at its end.
//
// A block owns one (sequence, head, 16 value columns).  Four of its warps walk the recurrence: eight lanes share a
// column, each with a run of RMAX rows of it in registers (d <= 8 RMAX).  With a = S_old^T k and c = S_old^T q of
// the state before the token, w = beta (v - g a) and o = g c + (k . q) w: both sums over the column are taken before
// the update, in one round of shuffles.  Tokens are walked two at a time: with S the state before the pair, all four
// sums S^T k1, S^T q1, S^T k2, S^T q2 are taken in one pass and one round of shuffles, and the second token's follow
// from them, since the state between the two is g1 S + k1 w1^T:
//   a2 = g1 (S^T k2) + (k1 . k2) w1,   c2 = g1 (S^T q2) + (k1 . q2) w1,   S <- g1 g2 S + k1 (g2 w1)^T + k2 w2^T,
// which halves the chain of dependent instructions a token.  The other four warps stage the chunk of tokens that
// comes next into the second of two shared-memory buffers meanwhile: a warp per pair of tokens reads q and k, makes
// them unit vectors in registers and writes them laid out as the walking lanes read them (a lane's run of rows as
// float4s, runs padded so that the eight lanes meet eight different groups of banks), with the token's gates and
// the products k . q, k1 . k2, k1 . q2 behind them.
#include <math_constants.h>
#include <stdio.h>

#include "common.cuh"

namespace {

constexpr int WALKERS = 128;         // threads that walk the recurrence
constexpr int THREADS = 256;         // and as many that stage the next tokens
constexpr int LANES = 8;             // lanes that share a column
constexpr int CT = WALKERS / LANES;  // columns of a block

template <int RMAX, int CH>
__global__ void __launch_bounds__(THREADS) delta_rule_kernel(
    const float* __restrict__ conv, int ldc, int q_col, int k_col, int v_col, const float* __restrict__ raw, int ld,
    int b_col, int a_col, const float* __restrict__ A_log, const float* __restrict__ dt_bias, float unit_eps,
    float* __restrict__ out, float* __restrict__ state, long long slot_stride, long long state_off,
    const int* __restrict__ q_start, const int* __restrict__ seq_slot, int H, int G, int d, int e) {
  constexpr int SEG = RMAX + 4;                          // a lane's run of rows and its padding
  constexpr int DP = LANES * SEG;                        // q (or k) of a token as staged
  constexpr int ROW = 2 * DP + CT + 8;                   // q, k, v tile, g, beta, k . q, k' . k, k' . q (k' of the token before), unused
  constexpr int JMAX = RMAX * LANES / 32;                // numbers of q (or k) a staging lane holds
  constexpr int PER_WARP = CH / 4;                       // tokens of a chunk that one staging warp takes
  static_assert(RMAX % 4 == 0 && CH % 4 == 0, "runs are read as float4s; four warps share a chunk");
  __shared__ __align__(16) float stage[2][CH][ROW];
  jb::pdl_launch_dependents();
  const int seq = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * CT;
  const int j = h / (H / G);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool walker = threadIdx.x < WALKERS;
  const int p = threadIdx.x & (LANES - 1), c = c0 + ((threadIdx.x & (WALKERS - 1)) >> 3);
  const bool has_col = walker && c < e;
  for (int i = threadIdx.x; i < 2 * CH * ROW; i += THREADS) (&stage[0][0][0])[i] = 0.0f;   // rows behind d stay zero
  const float neg_rate = -expf(A_log[h]), bias = dt_bias[h];
  const float q_mult = rsqrtf((float)d);
  jb::pdl_wait();
  const int t0 = q_start[seq], n_tok = q_start[seq + 1] - t0;
  float* S_g = state + (size_t)seq_slot[seq] * slot_stride + state_off + (size_t)h * d * e;
  float S[RMAX];
#pragma unroll
  for (int i = 0; i < RMAX; ++i) {
    const int r = p * RMAX + i;
    S[i] = (has_col && r < d) ? S_g[(size_t)r * e + c] : 0.0f;
  }
  __syncthreads();                                       // the zeros are in place before the first tokens land

  // a staging warp brings its tokens of a chunk: loads first, for all of them, then the sums and the stores
  auto bring = [&](int chunk, int buf) {
    const int first = chunk * CH, n = min(CH, n_tok - first);
    const int sw = warp - WALKERS / 32;
    float qv[PER_WARP][JMAX], kv[PER_WARP][JMAX], vv[PER_WARP], av[PER_WARP], bv[PER_WARP];
#pragma unroll
    for (int u = 0; u < PER_WARP; ++u) {
      const int tt = 2 * (sw + 4 * (u >> 1)) + (u & 1);  // a warp takes both tokens of a pair
      const size_t t = (size_t)(t0 + first + min(tt, n - 1));
      const float* qs = conv + t * ldc + q_col + (size_t)j * d;
      const float* ks = conv + t * ldc + k_col + (size_t)j * d;
#pragma unroll
      for (int x = 0; x < JMAX; ++x) {
        const int r = lane + 32 * x;
        qv[u][x] = r < d ? qs[r] : 0.0f;
        kv[u][x] = r < d ? ks[r] : 0.0f;
      }
      vv[u] = (lane < CT && c0 + lane < e) ? conv[t * ldc + v_col + (size_t)h * e + c0 + lane] : 0.0f;
      av[u] = raw[t * ld + a_col + h];
      bv[u] = raw[t * ld + b_col + h];
    }
    float ik_before = 0.0f;
#pragma unroll
    for (int u = 0; u < PER_WARP; ++u) {
      const int tt = 2 * (sw + 4 * (u >> 1)) + (u & 1);
      if (tt >= n) break;
      float sq = 0.0f, sk = 0.0f, qk = 0.0f, kk = 0.0f, kq = 0.0f;
#pragma unroll
      for (int x = 0; x < JMAX; ++x) {
        sq = fmaf(qv[u][x], qv[u][x], sq);
        sk = fmaf(kv[u][x], kv[u][x], sk);
        qk = fmaf(qv[u][x], kv[u][x], qk);
        if (u & 1) {
          kk = fmaf(kv[u - (u & 1)][x], kv[u][x], kk);
          kq = fmaf(kv[u - (u & 1)][x], qv[u][x], kq);
        }
      }
      sq = jb::warp_sum(sq);
      sk = jb::warp_sum(sk);
      qk = jb::warp_sum(qk);
      if (u & 1) {
        kk = jb::warp_sum(kk);
        kq = jb::warp_sum(kq);
      }
      const float iq = q_mult / sqrtf(sq + unit_eps), ik = 1.0f / sqrtf(sk + unit_eps);
      float* row = stage[buf][tt];
#pragma unroll
      for (int x = 0; x < JMAX; ++x) {
        const int r = lane + 32 * x;
        if (r < d) {
          const int at = (r / RMAX) * SEG + r % RMAX;
          row[at] = qv[u][x] * iq;
          row[DP + at] = kv[u][x] * ik;
        }
      }
      if (lane < CT) row[2 * DP + lane] = vv[u];
      if (lane == 0) {
        const float z = av[u] + bias;
        const float sp = z > 20.0f ? z : log1pf(expf(z));
        row[2 * DP + CT] = expf(neg_rate * sp);
        row[2 * DP + CT + 1] = 1.0f / (1.0f + expf(-bv[u]));
        row[2 * DP + CT + 2] = qk * iq * ik;
        row[2 * DP + CT + 3] = kk * ik_before * ik;
        row[2 * DP + CT + 4] = kq * ik_before * iq;
      }
      ik_before = ik;
    }
  };

  const int n_chunks = (n_tok + CH - 1) / CH;
  if (!walker && n_chunks > 0) bring(0, 0);
  __syncthreads();
  for (int chunk = 0; chunk < n_chunks; ++chunk) {
    const int buf = chunk & 1;
    if (!walker) {
      if (chunk + 1 < n_chunks) bring(chunk + 1, buf ^ 1);
    } else {
      const int first = chunk * CH, n = min(CH, n_tok - first);
      const int col = (threadIdx.x & (WALKERS - 1)) >> 3;
      int tt = 0;
      for (; tt + 1 < n; tt += 2) {                      // two tokens from one pass over the state
        const float* r1 = stage[buf][tt];
        const float* r2 = stage[buf][tt + 1];
        const float4* q1 = reinterpret_cast<const float4*>(r1 + p * SEG);
        const float4* k1 = reinterpret_cast<const float4*>(r1 + DP + p * SEG);
        const float4* q2 = reinterpret_cast<const float4*>(r2 + p * SEG);
        const float4* k2 = reinterpret_cast<const float4*>(r2 + DP + p * SEG);
        float kr1[RMAX], kr2[RMAX];
        float a1 = 0.0f, c1 = 0.0f, a2 = 0.0f, c2 = 0.0f, a1b = 0.0f, c1b = 0.0f, a2b = 0.0f, c2b = 0.0f;
#pragma unroll
        for (int i = 0; i < RMAX; i += 4) {
          const float4 ka = k1[i >> 2], qa = q1[i >> 2], kb = k2[i >> 2], qb = q2[i >> 2];
          kr1[i] = ka.x, kr1[i + 1] = ka.y, kr1[i + 2] = ka.z, kr1[i + 3] = ka.w;
          kr2[i] = kb.x, kr2[i + 1] = kb.y, kr2[i + 2] = kb.z, kr2[i + 3] = kb.w;
          a1 = fmaf(S[i], ka.x, a1), a1b = fmaf(S[i + 1], ka.y, a1b);
          a1 = fmaf(S[i + 2], ka.z, a1), a1b = fmaf(S[i + 3], ka.w, a1b);
          c1 = fmaf(S[i], qa.x, c1), c1b = fmaf(S[i + 1], qa.y, c1b);
          c1 = fmaf(S[i + 2], qa.z, c1), c1b = fmaf(S[i + 3], qa.w, c1b);
          a2 = fmaf(S[i], kb.x, a2), a2b = fmaf(S[i + 1], kb.y, a2b);
          a2 = fmaf(S[i + 2], kb.z, a2), a2b = fmaf(S[i + 3], kb.w, a2b);
          c2 = fmaf(S[i], qb.x, c2), c2b = fmaf(S[i + 1], qb.y, c2b);
          c2 = fmaf(S[i + 2], qb.z, c2), c2b = fmaf(S[i + 3], qb.w, c2b);
        }
        a1 += a1b, c1 += c1b, a2 += a2b, c2 += c2b;
#pragma unroll
        for (int o = 1; o < LANES; o <<= 1) {
          a1 += __shfl_xor_sync(0xffffffffu, a1, o);
          c1 += __shfl_xor_sync(0xffffffffu, c1, o);
          a2 += __shfl_xor_sync(0xffffffffu, a2, o);
          c2 += __shfl_xor_sync(0xffffffffu, c2, o);
        }
        const float g1 = r1[2 * DP + CT], beta1 = r1[2 * DP + CT + 1], kq1 = r1[2 * DP + CT + 2];
        const float g2 = r2[2 * DP + CT], beta2 = r2[2 * DP + CT + 1], kq2 = r2[2 * DP + CT + 2];
        const float k1k2 = r2[2 * DP + CT + 3], k1q2 = r2[2 * DP + CT + 4];
        const float w1 = beta1 * (r1[2 * DP + col] - g1 * a1);
        const float w2 = beta2 * (r2[2 * DP + col] - g2 * fmaf(k1k2, w1, g1 * a2));
        const float gg = g1 * g2, w1g = g2 * w1;
#pragma unroll
        for (int i = 0; i < RMAX; ++i) S[i] = fmaf(kr2[i], w2, fmaf(kr1[i], w1g, gg * S[i]));
        if (p == 0 && has_col) {
          float* dst = out + ((size_t)(t0 + first + tt) * H + h) * e + c;
          dst[0] = fmaf(kq1, w1, g1 * c1);
          dst[(size_t)H * e] = fmaf(kq2, w2, g2 * fmaf(k1q2, w1, g1 * c2));
        }
      }
      for (; tt < n; ++tt) {                             // a token left over
        const float* row = stage[buf][tt];
        const float4* q4 = reinterpret_cast<const float4*>(row + p * SEG);
        const float4* k4 = reinterpret_cast<const float4*>(row + DP + p * SEG);
        float kr[RMAX];
        float a0 = 0.0f, a1 = 0.0f, b0 = 0.0f, b1 = 0.0f;
#pragma unroll
        for (int i = 0; i < RMAX; i += 4) {
          const float4 kk = k4[i >> 2], qq = q4[i >> 2];
          kr[i] = kk.x, kr[i + 1] = kk.y, kr[i + 2] = kk.z, kr[i + 3] = kk.w;
          a0 = fmaf(S[i], kk.x, a0);
          a1 = fmaf(S[i + 1], kk.y, a1);
          a0 = fmaf(S[i + 2], kk.z, a0);
          a1 = fmaf(S[i + 3], kk.w, a1);
          b0 = fmaf(S[i], qq.x, b0);
          b1 = fmaf(S[i + 1], qq.y, b1);
          b0 = fmaf(S[i + 2], qq.z, b0);
          b1 = fmaf(S[i + 3], qq.w, b1);
        }
        float a = a0 + a1, b = b0 + b1;
#pragma unroll
        for (int o = 1; o < LANES; o <<= 1) {
          a += __shfl_xor_sync(0xffffffffu, a, o);
          b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        const float g = row[2 * DP + CT], beta = row[2 * DP + CT + 1], kq = row[2 * DP + CT + 2];
        const float w = beta * (row[2 * DP + col] - g * a);
#pragma unroll
        for (int i = 0; i < RMAX; ++i) S[i] = fmaf(kr[i], w, g * S[i]);
        if (p == 0 && has_col) out[((size_t)(t0 + first + tt) * H + h) * e + c] = fmaf(kq, w, g * b);
      }
    }
    __syncthreads();                                     // the next chunk is staged; this one is done with
  }
  if (has_col) {
#pragma unroll
    for (int i = 0; i < RMAX; ++i) {
      const int r = p * RMAX + i;
      if (r < d) S_g[(size_t)r * e + c] = S[i];
    }
  }
}

// ---- prompts: chunks of 32 tokens ------------------------------------------------------------------------------------
// Within a chunk that starts from state S the writes w_t solve a triangular system: with L_t the sum of the log decays up
// to token t (of the chunk) and A[t][s] = beta_t exp(L_t - L_s) (k_t . k_s) for s < t,
//   (I + A) w = beta v - (beta exp(L) k) S   =>   w = U - V S with (I + A) U = beta v, (I + A) V = beta exp(L) k,
//   o_t = exp(L_t) q_t S + sum over s <= t of P[t][s] w_s,  P[t][s] = exp(L_t - L_s) (q_t . k_s),
//   S <- exp(L_end) S + sum over t of exp(L_end - L_t) k_t w_t^T.
// U, V and P know nothing of the state, so all chunks make them side by side (`delta_prepare_kernel`: a block per chunk and
// head, V and P to scratch, U to where the output will be); what is left to walk (`delta_chunks_kernel`: a block per
// sequence, head and 16 value columns, the state in shared memory) is three small products a chunk.  All in float32 but for the
// sums L and their differences (float64: past a strong decay a difference of two large sums would keep few digits in 32
// bits); the decays only ever appear as exponentials of differences that are not positive.  One sequence of 1,500 tokens, 16 heads of 128 x
// 128: 460 us as the walk above, a chain of 307 ns a token; 39 us of prepare and 153 of chunks so.
constexpr int C = 32, DMAX = 128, LD = DMAX + 4, CHUNK_THREADS = 256;
constexpr int V_FLOATS = C * DMAX, P_FLOATS = C * C, SC_FLOATS = C * 4;
constexpr int SCRATCH_FLOATS = V_FLOATS + P_FLOATS + SC_FLOATS;           // of one chunk and head
constexpr int PREPARE_HEADS = 8;               // heads of a group that a block prepares at most

// Where the scratch of a sequence's first chunk lies, in chunks: `tiles` a sequence, or (packed) as many as it needs, one
// sequence after another: floor(q_start / C) + seq begins at or past the end of the sequence before.
__device__ __forceinline__ int first_slot(const int* q_start, int seq, int tiles, int packed) {
  return packed ? q_start[seq] / C + seq : seq * tiles;
}

__global__ void __launch_bounds__(CHUNK_THREADS, 2) delta_prepare_kernel(
    const float* __restrict__ conv, int ldc, int q_col, int k_col, int v_col, const float* __restrict__ raw, int ld,
    int b_col, int a_col, const float* __restrict__ A_log, const float* __restrict__ dt_bias, float unit_eps,
    float* __restrict__ out, float* __restrict__ scratch, const int* __restrict__ q_start, int n_seqs, int H, int G, int d, int e,
    int first_tile, int tiles, int packed, int heads_here) {
  // products of a chunk's keys with its keys and queries, which the heads of a group share
  __shared__ __align__(16) float q_s[C][LD], k_s[C][LD];
  __shared__ float kk_s[C][C + 1], qk_s[C][C + 1];
  __shared__ double L_s[PREPARE_HEADS][C];
  __shared__ float beta_s[PREPARE_HEADS][C], start_s[PREPARE_HEADS][C], iq_s[C], ik_s[C];
  jb::pdl_launch_dependents();
  const int R = H / G, j = blockIdx.y;
  const int h_begin = j * R + (int)blockIdx.z * heads_here, h_end = min((j + 1) * R, h_begin + heads_here);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const float q_mult = rsqrtf((float)d);
  jb::pdl_wait();
  int seq = (int)blockIdx.x / tiles, tile = (int)blockIdx.x % tiles;
  if (packed) {                                                            // the last sequence whose chunks begin up to here
    seq = -1;
    for (int s0 = 0; s0 < n_seqs; s0 += CHUNK_THREADS) {
      const int s = s0 + (int)threadIdx.x;
      seq += __syncthreads_count(s < n_seqs && first_slot(q_start, s, tiles, packed) <= (int)blockIdx.x);
    }
    tile = (int)blockIdx.x - first_slot(q_start, seq, tiles, packed);
  }
  const int t0 = q_start[seq] + (first_tile + tile) * C, n = min(C, q_start[seq + 1] - t0);
  if (n <= 0) return;
  // four tokens a warp: unit vectors of q and k, zero past the end of the chunk and of a row
  float4 qv[4], kv[4];
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int t = 4 * warp + u;
    const bool in = t < n && 4 * lane < d;
    const float* row = conv + (size_t)(t0 + (t < n ? t : 0)) * ldc + (size_t)j * d + (in ? 4 * lane : 0);
    qv[u] = in ? *reinterpret_cast<const float4*>(row + q_col) : zero;
    kv[u] = in ? *reinterpret_cast<const float4*>(row + k_col) : zero;
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int t = 4 * warp + u;
    const float iq = q_mult / sqrtf(jb::warp_sum(qv[u].x * qv[u].x + qv[u].y * qv[u].y + qv[u].z * qv[u].z + qv[u].w * qv[u].w) + unit_eps);
    const float ik = 1.0f / sqrtf(jb::warp_sum(kv[u].x * kv[u].x + kv[u].y * kv[u].y + kv[u].z * kv[u].z + kv[u].w * kv[u].w) + unit_eps);
    *reinterpret_cast<float4*>(&q_s[t][4 * lane]) = make_float4(qv[u].x * iq, qv[u].y * iq, qv[u].z * iq, qv[u].w * iq);
    *reinterpret_cast<float4*>(&k_s[t][4 * lane]) = make_float4(kv[u].x * ik, kv[u].y * ik, kv[u].z * ik, kv[u].w * ik);
    if (lane == 0) iq_s[t] = iq, ik_s[t] = ik;
  }
  __syncthreads();
  {
    // two by two entries of each product a thread; above the diagonal nobody reads them
    jb::Pair kk[2][2] = {{0, 0}, {0, 0}}, qk[2][2] = {{0, 0}, {0, 0}};
#pragma unroll 4
    for (int r = 0; r < DMAX; r += 4) {
      ulonglong2 a[2], b[2], c[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        a[x] = *reinterpret_cast<const ulonglong2*>(&k_s[ty + 16 * x][r]);
        b[x] = *reinterpret_cast<const ulonglong2*>(&q_s[ty + 16 * x][r]);
        c[x] = *reinterpret_cast<const ulonglong2*>(&k_s[tx + 16 * x][r]);
      }
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y <= x; ++y) {
          kk[x][y] = jb::fma2(a[x].y, c[y].y, jb::fma2(a[x].x, c[y].x, kk[x][y]));
          qk[x][y] = jb::fma2(b[x].y, c[y].y, jb::fma2(b[x].x, c[y].x, qk[x][y]));
        }
    }
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        kk_s[ty + 16 * x][tx + 16 * y] = jb::lo(kk[x][y]) + jb::hi(kk[x][y]);
        qk_s[ty + 16 * x][tx + 16 * y] = jb::lo(qk[x][y]) + jb::hi(qk[x][y]);
      }
  }
  for (int h = h_begin + warp; h < h_end; h += CHUNK_THREADS / 32) {        // a head a warp, a token a lane: log decays, summed, and betas
    double L = 0.0;
    float b = 0.0f;
    if (lane < n) {
      const float z = raw[(size_t)(t0 + lane) * ld + a_col + h] + dt_bias[h];
      // below -10,000 a decay is zero either way, and the sums stay finite (NaN stays NaN)
      const float log_g = -expf(A_log[h]) * (z > 20.0f ? z : log1pf(expf(z)));
      L = log_g < -10000.0f ? -10000.0f : log_g;
      b = 1.0f / (1.0f + expf(-raw[(size_t)(t0 + lane) * ld + b_col + h]));
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double before = __shfl_up_sync(0xffffffffu, L, o);
      if (lane >= o) L += before;
    }
    const double end = __shfl_sync(0xffffffffu, L, 31);
    const float from_start = expf((float)L);
    L_s[h - h_begin][lane] = L;
    beta_s[h - h_begin][lane] = b;
    start_s[h - h_begin][lane] = b * from_start;
    // per token: what multiplies q_t S (raw q), what multiplies k_t (raw k) on its way into the state, the chunk's decay
    float* V_g = scratch + ((size_t)blockIdx.x * H + h) * SCRATCH_FLOATS;
    reinterpret_cast<float4*>(V_g + V_FLOATS + P_FLOATS)[lane] =
        make_float4(from_start * iq_s[lane], lane < n ? expf((float)(end - L)) * ik_s[lane] : 0.0f, expf((float)end), 0.0f);
  }
  __syncthreads();
  // q has been read: two buffers of a head's A, transposed, take its place
  float(*At_b)[C][C + 4] = reinterpret_cast<float(*)[C][C + 4]>(&q_s[0][0]);
  for (int h = h_begin; h < h_end; ++h) {
    const int hh = h - h_begin;
    float* V_g = scratch + ((size_t)blockIdx.x * H + h) * SCRATCH_FLOATS;
    float* P_g = V_g + V_FLOATS;
    float(*At_s)[C + 4] = At_b[hh & 1];
    const float* v0 = conv + (size_t)t0 * ldc + v_col + (size_t)h * e;
    float x[C];
    // a column of the system's right-hand sides a thread: keys, then values, which are asked for before A is made
    const auto ask = [&](int column) {
#pragma unroll
      for (int t = 0; t < C; ++t) x[t] = column >= DMAX && column < DMAX + e && t < n ? v0[(size_t)t * ldc + column - DMAX] : 0.0f;
    };
    ask(threadIdx.x);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const int t = ty + 16 * i, s = tx + 16 * y;
        const float decay = s <= t ? expf((float)(L_s[hh][t] - L_s[hh][s])) : 0.0f;
        At_s[s][t] = s < t ? beta_s[hh][t] * decay * kk_s[t][s] : 0.0f;
        P_g[t * C + s] = s <= t ? decay * qk_s[t][s] : 0.0f;
      }
    __syncthreads();
    for (int column = threadIdx.x; column < DMAX + e; column += CHUNK_THREADS) {
      const bool is_key = column < DMAX;
      if (column >= CHUNK_THREADS) ask(column);
#pragma unroll
      for (int t = 0; t < C; ++t) x[t] = is_key ? start_s[hh][t] * k_s[t][column] : beta_s[hh][t] * x[t];
      // a write that is known is taken off all later ones
#pragma unroll
      for (int s = 0; s < C - 1; ++s) {
#pragma unroll
        for (int t = (s + 1) & ~3; t < C; t += 4) {
          const float4 a = *reinterpret_cast<const float4*>(&At_s[s][t]);   // zero up to the diagonal
          if (t > s) x[t] = fmaf(-a.x, x[s], x[t]);
          if (t + 1 > s) x[t + 1] = fmaf(-a.y, x[s], x[t + 1]);
          if (t + 2 > s) x[t + 2] = fmaf(-a.z, x[s], x[t + 2]);
          x[t + 3] = fmaf(-a.w, x[s], x[t + 3]);
        }
      }
#pragma unroll
      for (int t = 0; t < C; ++t) {
        if (is_key) V_g[t * DMAX + column] = x[t];
        else if (t < n) out[((size_t)(t0 + t) * H + h) * e + column - DMAX] = x[t];
      }
    }
  }
}

// copies 16 bytes, or zeros
__device__ __forceinline__ void async16(float* dst, const float* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 16 : 0));
}

constexpr int SLD = 40;                        // floats of a pair of the state's rows: 16 columns of two, and padding
constexpr int CHUNK_SMEM = (5 * C * LD + C * (C + 4) + DMAX / 2 * SLD + 2 * C * 20 + C * 4) * 4;

// SPLIT times 256 threads, which share the first product's sums over k.  Once, two blocks an SM; twice where no SM has a second
// block, which shortens a chunk's chain (prepare and chunks, one sequence of 16 heads of 128 x 128, 128 blocks: 1,500
// tokens 265 and 192 us, 192 tokens 48 and 38; 8 heads of 72 x 72, 1,500 tokens 249 and 175; 1,000 tokens, 4 heads of 128 x 128,
// 32 blocks, 164 and 117).  Very few blocks have the chip's clock and memory to themselves and are faster with 256 (3 heads, 24 blocks,
// 106 and 115; one head, 2,000 tokens, 190 and 210; 28 blocks level).
template <int SPLIT>
__global__ void __launch_bounds__(CHUNK_THREADS * SPLIT, 2 / SPLIT) delta_chunks_kernel(
    const float* __restrict__ conv, int ldc, int q_col, int k_col, float* __restrict__ out, const float* __restrict__ scratch,
    float* __restrict__ state, long long slot_stride, long long state_off, const int* __restrict__ q_start,
    const int* __restrict__ seq_slot, int H, int G, int d, int e, int first_tile, int tiles, int packed) {
  constexpr int THREADS = CHUNK_THREADS * SPLIT, KS = 4 * SPLIT;             // lanes that share a thread's sums
  constexpr int OWN = 4 / SPLIT, RP = 2 / SPLIT;                             // columns of a row, pairs of the state's rows a thread keeps
  extern __shared__ __align__(16) float smem[];
  float* vq_b = smem;                          // two buffers of V [C][LD], then q [C][LD]: 64 rows to multiply with the state
  float* k_s = vq_b + 4 * C * LD;              // k [C][LD]
  float* P_s = k_s + C * LD;                   // [C][C + 4]
  float* S_s = P_s + C * (C + 4);              // [DMAX / 2][SLD]: two rows of a column are neighbours
  float* w_s = S_s + DMAX / 2 * SLD;           // the writes [C][20], and as they join the state [C][20]
  float* wk_s = w_s + C * 20;
  float4* sc_s = reinterpret_cast<float4*>(wk_s + C * 20);
  jb::pdl_launch_dependents();
  const int seq = blockIdx.z, h = blockIdx.y, c0 = blockIdx.x * 16, j = h / (H / G);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  jb::pdl_wait();
  const int begin = q_start[seq] + first_tile * C, n_all = min(q_start[seq + 1] - begin, tiles * C);
  if (n_all <= 0) return;
  float* S_g = state + (size_t)seq_slot[seq] * slot_stride + state_off + (size_t)h * d * e;
  const float* scratch_g = scratch + ((size_t)first_slot(q_start, seq, tiles, packed) * H + h) * SCRATCH_FLOATS;
  const int chunks = (n_all + C - 1) / C;

  auto load_vq = [&](int chunk) {
    float* vq_s = vq_b + (chunk & 1) * 2 * C * LD;
    const int t0 = begin + chunk * C, n = min(C, n_all - chunk * C);
    const float* V_g = scratch_g + (size_t)chunk * H * SCRATCH_FLOATS;
    for (int i = tid; i < C * DMAX / 4; i += THREADS) {
      const int t = i / (DMAX / 4), r = (i % (DMAX / 4)) * 4;
      async16(vq_s + t * LD + r, V_g + t * DMAX + r, true);
      const bool in = t < n && r < d;
      async16(vq_s + (C + t) * LD + r, conv + (size_t)(t0 + (in ? t : 0)) * ldc + q_col + (size_t)j * d + (in ? r : 0), in);
    }
    asm volatile("cp.async.commit_group;");
  };
  auto load_kp = [&](int chunk) {
    const int t0 = begin + chunk * C, n = min(C, n_all - chunk * C);
    const float* P_g = scratch_g + (size_t)chunk * H * SCRATCH_FLOATS + V_FLOATS;
    for (int i = tid; i < C * DMAX / 4; i += THREADS) {
      const int t = i / (DMAX / 4), r = (i % (DMAX / 4)) * 4;
      const bool in = t < n && r < d;
      async16(k_s + t * LD + r, conv + (size_t)(t0 + (in ? t : 0)) * ldc + k_col + (size_t)j * d + (in ? r : 0), in);
    }
    if (tid < P_FLOATS / 4) async16(P_s + (tid / 8) * (C + 4) + (tid % 8) * 4, P_g + tid * 4, true);
    if (tid < C) async16(reinterpret_cast<float*>(sc_s + tid), P_g + P_FLOATS + 4 * tid, true);
    asm volatile("cp.async.commit_group;");
  };
  load_vq(0);
  load_kp(0);
  if (chunks > 1) load_vq(1);
  else asm volatile("cp.async.commit_group;");
  for (int i = tid; i < DMAX * 16; i += THREADS) {
    const int r = i >> 4, c = i & 15;
    S_s[(r >> 1) * SLD + 2 * c + (r & 1)] = (r < d && c0 + c < e) ? S_g[(size_t)r * e + c0 + c] : 0.0f;
  }

  // first product: a thread four of the 64 rows, four columns, every KS-th group of four k
  const int cg = lane & 3, ks = (lane >> 2) & (KS - 1), rg = SPLIT == 1 ? (warp << 1) | (lane >> 4) : warp;
  const int t_own = (rg * 4 + (ks & 3)) & (C - 1);                         // the row that is this thread's after the sums meet
  const bool is_q = rg >= C / 4;
  // its columns: 2 cg, 2 cg + 1, 8 + 2 cg, 9 + 2 cg; after the sums meet the OWN of them from own[0] on
  const int col[2] = {2 * cg, 8 + 2 * cg}, own[2] = {SPLIT == 1 || ks < 4 ? col[0] : col[1], col[1]};
  // state's update, by the threads without queries: RP pairs of rows, four columns
  const int uc = (tid & 3) * 4, ur = ((tid & (THREADS / 2 - 1)) >> 2) * RP;

  for (int chunk = 0; chunk < chunks; ++chunk) {
    const int t0 = begin + chunk * C, n = min(C, n_all - chunk * C);
    float* mine = out + ((size_t)(t0 + t_own) * H + h) * e + c0;
    float u[OWN];
#pragma unroll
    for (int x = 0; x < OWN; ++x) {
      const int c = own[x >> 1] + (x & 1);
      u[x] = !is_q && t_own < n && c0 + c < e ? mine[c] : 0.0f;
    }
    // groups in flight, oldest first: V and q of this chunk, k and P of it, V and q of the next
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    __syncthreads();
    const float* vq_s = vq_b + (chunk & 1) * 2 * C * LD;
    jb::Pair acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int x = 0; x < 4; ++x) acc[i][x] = 0;
#pragma unroll 2
    for (int it = 0; it < DMAX / (4 * KS); ++it) {
      const int k4 = KS * it + ks;                                         // group of four rows of the state
      ulonglong2 a[4], b[2][2];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(vq_s + (rg * 4 + i) * LD + 4 * k4);
#pragma unroll
      for (int y = 0; y < 2; ++y)
#pragma unroll
        for (int x = 0; x < 2; ++x)
          b[y][x] = *reinterpret_cast<const ulonglong2*>(S_s + (2 * k4 + y) * SLD + 2 * col[x]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          acc[i][2 * x] = jb::fma2(a[i].y, b[1][x].x, jb::fma2(a[i].x, b[0][x].x, acc[i][2 * x]));
          acc[i][2 * x + 1] = jb::fma2(a[i].y, b[1][x].y, jb::fma2(a[i].x, b[0][x].y, acc[i][2 * x + 1]));
        }
      }
    }
    // the KS lanes of a row group and column group add up; lane ks keeps row ks % 4, of eight lanes two columns each
    float r[4][OWN];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (SPLIT == 1) {
#pragma unroll
        for (int x = 0; x < OWN; ++x) r[i][x] = jb::lo(acc[i][x]) + jb::hi(acc[i][x]);
      } else {
        const bool right = ks >= 4;
#pragma unroll
        for (int x = 0; x < OWN; ++x) {
          const float a = jb::lo(acc[i][x]) + jb::hi(acc[i][x]), b = jb::lo(acc[i][2 + x]) + jb::hi(acc[i][2 + x]);
          r[i][x] = (right ? b : a) + __shfl_xor_sync(0xffffffffu, right ? a : b, 16);
        }
      }
    }
    float m[OWN];
#pragma unroll
    for (int x = 0; x < OWN; ++x) {
      // rows 0, 1 go to the lanes with bit 1 of ks clear, rows 2, 3 to the others; then one row each
      const bool up = (ks & 2) != 0, odd = (ks & 1) != 0;
      float a = up ? r[2][x] : r[0][x], b = up ? r[3][x] : r[1][x];
      a += __shfl_xor_sync(0xffffffffu, up ? r[0][x] : r[2][x], 8);
      b += __shfl_xor_sync(0xffffffffu, up ? r[1][x] : r[3][x], 8);
      m[x] = odd ? b : a;
      m[x] += __shfl_xor_sync(0xffffffffu, odd ? a : b, 4);
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");                   // k, P and the scales
    __syncthreads();                                                       // ... for all; V and q have been read
    const float4 sc = sc_s[t_own];
    if (!is_q) {
#pragma unroll
      for (int x = 0; x < OWN; ++x) {
        const float w = u[x] - m[x];
        w_s[t_own * 20 + own[x >> 1] + (x & 1)] = w;
        wk_s[t_own * 20 + own[x >> 1] + (x & 1)] = w * sc.y;
      }
    }
    __syncthreads();
    if (is_q) {
      float o[OWN];
#pragma unroll
      for (int x = 0; x < OWN; ++x) o[x] = m[x] * sc.x;
      const auto four = [&](int s, int seen) {                             // four writes, of which `seen` come up to this token
        const float4 p = *reinterpret_cast<const float4*>(P_s + t_own * (C + 4) + s);
        const float ps[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
        for (int y = 0; y < 4; ++y) {
          float2 w[OWN / 2];
#pragma unroll
          for (int x = 0; x < OWN / 2; ++x) w[x] = *reinterpret_cast<const float2*>(w_s + (s + y) * 20 + own[x]);
          if (y < seen) {
#pragma unroll
            for (int x = 0; x < OWN / 2; ++x) o[2 * x] = fmaf(ps[y], w[x].x, o[2 * x]), o[2 * x + 1] = fmaf(ps[y], w[x].y, o[2 * x + 1]);
          }
        }
      };
#pragma unroll 2
      for (int s = 0; s < (t_own & ~3); s += 4) four(s, 4);
      four(t_own & ~3, (ks & 3) + 1);                                          // (zero times a later write that is infinite would be NaN)
      if (t_own < n) {
#pragma unroll
        for (int x = 0; x < OWN; ++x)
          if (c0 + own[x >> 1] + (x & 1) < e) mine[own[x >> 1] + (x & 1)] = o[x];
      }
    }
    if (!is_q) {
      jb::Pair S[RP][4];
      const jb::Pair g = jb::pair(sc.z, sc.z);
#pragma unroll
      for (int y = 0; y < RP; ++y)
#pragma unroll
        for (int x = 0; x < 4; x += 2) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(S_s + (ur + y) * SLD + 2 * (uc + x));
          S[y][x] = jb::mul2(v.x, g);
          S[y][x + 1] = jb::mul2(v.y, g);
        }
#pragma unroll 8
      for (int t = 0; t < C; ++t) {
        jb::Pair k[RP];
        if constexpr (RP == 2) {
          const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(k_s + t * LD + 2 * ur);
          k[0] = v.x, k[1] = v.y;
        } else {
          k[0] = *reinterpret_cast<const jb::Pair*>(k_s + t * LD + 2 * ur);
        }
        const float4 w = *reinterpret_cast<const float4*>(wk_s + t * 20 + uc);
        const jb::Pair ws[4] = {jb::pair(w.x, w.x), jb::pair(w.y, w.y), jb::pair(w.z, w.z), jb::pair(w.w, w.w)};
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
          for (int y = 0; y < RP; ++y) S[y][x] = jb::fma2(k[y], ws[x], S[y][x]);
      }
#pragma unroll
      for (int y = 0; y < RP; ++y)
#pragma unroll
        for (int x = 0; x < 4; x += 2)
          *reinterpret_cast<ulonglong2*>(S_s + (ur + y) * SLD + 2 * (uc + x)) = make_ulonglong2(S[y][x], S[y][x + 1]);
    }
    __syncthreads();                                                       // the state is whole; k, P and the writes have been read
    if (chunk + 1 < chunks) load_kp(chunk + 1);
    else asm volatile("cp.async.commit_group;");
    if (chunk + 2 < chunks) load_vq(chunk + 2);
    else asm volatile("cp.async.commit_group;");
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  for (int i = tid; i < DMAX * 16; i += THREADS) {
    const int r = i >> 4, c = i & 15;
    if (r < d && c0 + c < e) S_g[(size_t)r * e + c0 + c] = S_s[(r >> 1) * SLD + 2 * c + (r & 1)];
  }
}

}  // namespace

// conv: float32 [T, ldc], queries at q_col ([G][d]), keys at k_col ([G][d]), values at v_col ([H][e]); raw: float32
// [T, ld], beta's argument at b_col ([H]), the decay's at a_col ([H]); A_log, dt_bias: float32 [H]; out: float32
// [T, H e]; state: per slot slot_stride floats, the recurrence's [H][d][e] at state_off.
JB_EXPORT int jb_delta_rule(const float* conv, int ldc, int q_col, int k_col, int v_col, const float* raw, int ld,
                            int b_col, int a_col, const float* A_log, const float* dt_bias, float unit_eps, float* out,
                            float* state, long long slot_stride, long long state_off, const int* q_start,
                            const int* seq_slot, int n_seqs, int H, int G, int d, int e, cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  JB_REFUSE(d < 1 || d > 256 || e < 1, "delta_rule: key size %d is outside [1, 256]", d);
  JB_REFUSE(G < 1 || H % G != 0, "delta_rule: %d heads are not a multiple of %d key heads", H, G);
  jb::Launch cfg(dim3((e + CT - 1) / CT, H, n_seqs), dim3(THREADS), 0, stream);
  cudaError_t err;
#define JB_LAUNCH_DR(RMAX, CH)                                                                                       \
  err = cudaLaunchKernelEx(&cfg.c, delta_rule_kernel<RMAX, CH>, conv, ldc, q_col, k_col, v_col, raw, ld, b_col, a_col, \
                           A_log, dt_bias, unit_eps, out, state, slot_stride, state_off, q_start, seq_slot, H, G, d, e)
  if (d <= 64) JB_LAUNCH_DR(8, 16);
  else if (d <= 128) JB_LAUNCH_DR(16, 16);
  else JB_LAUNCH_DR(32, 8);   // 8 RMAX rows hold d; a chunk's two buffers stay within the static shared memory
#undef JB_LAUNCH_DR
  return (int)err;
}

// The same for prompts, by chunks: d <= 128, d, ldc, q_col and k_col multiples of 4, conv 16-byte aligned.  `scratch` holds
// `tiles` chunks of every sequence; longer prompts go in slabs of as many, one after another from the state the last left.
// tiles = 0: it holds tokens / 32 + n_seqs chunks, the whole step's, one sequence after another (`tokens`: of all sequences).
JB_EXPORT int jb_delta_rule_chunks(const float* conv, int ldc, int q_col, int k_col, int v_col, const float* raw, int ld,
                                   int b_col, int a_col, const float* A_log, const float* dt_bias, float unit_eps, float* out,
                                   float* state, long long slot_stride, long long state_off, const int* q_start,
                                   const int* seq_slot, int n_seqs, int H, int G, int d, int e, int max_q_len, float* scratch,
                                   int tiles, int tokens, cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  JB_REFUSE(d < 1 || d > DMAX || e < 1 || ((d | ldc | q_col | k_col) & 3) != 0 || (((uintptr_t)conv | (uintptr_t)scratch) & 15) != 0,
            "delta_rule_chunks: keys of %d numbers in rows of %d at columns %d and %d", d, ldc, q_col, k_col);
  JB_REFUSE(G < 1 || H % G != 0 || tiles < 0 || max_q_len < 1, "delta_rule_chunks: %d heads are not a multiple of %d key heads", H, G);
  const long long blocks = (long long)n_seqs * H * ((e + 15) / 16);
  const bool few = blocks > 28 && blocks <= 148;                                     // no SM has a second block, many have one
  auto* const walk_kernel = few ? delta_chunks_kernel<2> : delta_chunks_kernel<1>;
  cudaError_t err = cudaFuncSetAttribute(walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CHUNK_SMEM);
  if (err != cudaSuccess) return (int)err;
  const int all = (max_q_len + C - 1) / C, packed = tiles == 0;
  if (packed) tiles = all;
  const int slots = packed ? tokens / C + n_seqs : n_seqs * tiles;
  for (int first = 0; first < all; first += tiles) {
    // (the scratch of a slab is laid out for `tiles` chunks a sequence, whatever is left of it)
    // a block makes the products of a chunk and key head once for its group's heads, or for a share of them where that
    // leaves SMs without a block
    const int group = H / G, chunks = (packed ? tokens / C + 1 : slots) * G;         // that have tokens
    int parts = (2 * 148 + chunks - 1) / chunks;
    parts = parts < group ? parts : group;
    if (parts < (group + PREPARE_HEADS - 1) / PREPARE_HEADS) parts = (group + PREPARE_HEADS - 1) / PREPARE_HEADS;
    const int heads_here = (group + parts - 1) / parts;
    jb::Launch prepare(dim3(slots, G, (group + heads_here - 1) / heads_here), dim3(CHUNK_THREADS), 0, stream);
    err = cudaLaunchKernelEx(&prepare.c, delta_prepare_kernel, conv, ldc, q_col, k_col, v_col, raw, ld, b_col, a_col, A_log,
                             dt_bias, unit_eps, out, scratch, q_start, n_seqs, H, G, d, e, first, tiles, packed, heads_here);
    if (err != cudaSuccess) return (int)err;
    jb::Launch walk(dim3((e + 15) / 16, H, n_seqs), dim3(few ? 2 * CHUNK_THREADS : CHUNK_THREADS), CHUNK_SMEM, stream);
    err = cudaLaunchKernelEx(&walk.c, walk_kernel, conv, ldc, q_col, k_col, out, (const float*)scratch, state, slot_stride,
                             state_off, q_start, seq_slot, H, G, d, e, first, tiles, packed);
    if (err != cudaSuccess) return (int)err;
  }
  return 0;
}
