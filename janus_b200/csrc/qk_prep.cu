// What happens between the projections of an attention mixer and the attention kernel itself, for two mixers
// whose queries and keys are normed over the whole projection.  All arithmetic is float32; the projections are the
// products' float32 accumulators.
//
// qk_norm_rope_cache (attention whose values are its keys as projected):
//   q = proj[:, 0 : H d] + bq,  k = proj[:, H d : (H + G) d] + bk
//   v = k                                             (before norm and rotation; appended to the value pages)
//   q <- q / sqrt(mean(q^2) + eps) * wq               (one root mean square over all H d numbers), k likewise
//   the first `rot` dimensions of every head of q and k are turned in the pairing (i, i + rot/2) by the angle
//   of the token's position (cos and sin from a table [positions][rot/2][2]); the rest pass
//   q is written [T, H dp] in the engine dtype, k is appended to the key pages; dp >= d is the size a head is
//   stored with (a head size that the attention kernel does not take is stored as the next size it takes, the
//   extra columns zero: scores and sums do not change).
//
// latent_prep (latent attention, queries already multiplied into the latent space):
//   q = proj[:, 0 : Q] written [T, Q] in the engine dtype
//   c = proj[:, Q : Q + r] / sqrt(mean(.^2) + eps) * w, appended to the pages as the token's one key row
//
// Pages of one place: [page][kv_head][page_size][size]; dest[t] = page * page_size + row of token t.
// One block per token.
#include <stdio.h>

#include "common.cuh"

namespace {

typedef __nv_bfloat16 bf16;

template <typename TO>
__device__ __forceinline__ void store4(TO* p, const float4& v) {
  if constexpr (sizeof(TO) == 4) {
    *reinterpret_cast<float4*>(p) = v;
  } else {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
    uint2 u;
    u.x = *reinterpret_cast<const uint32_t*>(&lo);
    u.y = *reinterpret_cast<const uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(p) = u;
  }
}

// (cos, sin) of four neighbouring pairs: u and v, the members of each pair, are turned in place
__device__ __forceinline__ void turn4(float4& u, float4& v, const float* cs) {
  const float4 a = *reinterpret_cast<const float4*>(cs), b = *reinterpret_cast<const float4*>(cs + 4);
  const float4 x = u, y = v;
  u = make_float4(x.x * a.x - y.x * a.y, x.y * a.z - y.y * a.w, x.z * b.x - y.z * b.y, x.w * b.z - y.w * b.w);
  v = make_float4(y.x * a.x + x.x * a.y, y.y * a.z + x.y * a.w, y.z * b.x + x.z * b.y, y.w * b.z + x.w * b.w);
}

// qk_norm_rope_cache four numbers a thread and access (sizes and row starts whole groups of four, half a rotation too,
// no padding).  The biases are asked for before the wait for the projection, the norms' weights before the sums meet, so a
// token costs one chain of latencies (8 tokens of 32 + 8 heads of 128: 31 us with one number a thread and two sums one
// after the other, 5.3 so; 2,532 tokens, 83 MB: 95 and 55 us).  QK_CACHE groups of the row a thread are in flight at once.
constexpr int QK_THREADS = 512, QK_CACHE = 4;

template <typename TO>
__global__ void __launch_bounds__(QK_THREADS) qk_norm_rope_rows_kernel(
    const float* __restrict__ proj, int ld, const float* __restrict__ bq, const float* __restrict__ bk,
    const float* __restrict__ wq, const float* __restrict__ wk, float eps, const float* __restrict__ table, int rot,
    const int* __restrict__ positions, TO* __restrict__ q_out, const int* __restrict__ dest, TO* __restrict__ k_cache,
    TO* __restrict__ v_cache, int H, int G, int d, int page_size, int write_kv) {
  extern __shared__ __align__(16) float row_s[];     // q [H d], then k [G d]
  __shared__ float scratch[2][QK_THREADS / 32];
  jb::pdl_launch_dependents();
  const int t = blockIdx.x;
  const int QW = H * d, KW = write_kv ? G * d : 0;
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const auto bias = [&](int i) {
    const float* b = i < QW ? bq : bk;
    return b != nullptr ? *reinterpret_cast<const float4*>(b + (i < QW ? i : i - QW)) : zero;
  };
  float4 b[QK_CACHE], v[QK_CACHE];
#pragma unroll
  for (int c = 0; c < QK_CACHE; ++c) {
    const int i = 4 * ((int)threadIdx.x + c * QK_THREADS);
    if (i < QW + KW) b[c] = bias(i);
  }
  jb::pdl_wait();
  const float* pr = proj + (size_t)t * ld;
#pragma unroll
  for (int c = 0; c < QK_CACHE; ++c) {
    const int i = 4 * ((int)threadIdx.x + c * QK_THREADS);
    if (i < QW + KW) v[c] = *reinterpret_cast<const float4*>(pr + i);
  }
  const size_t page = write_kv ? (size_t)(dest[t] / page_size) : 0;
  const int prow = write_kv ? dest[t] % page_size : 0;
  const int half = rot >> 1;
  const float* cs = (table != nullptr && rot > 0) ? table + (size_t)positions[t] * half * 2 : nullptr;
  float sq = 0.0f, sk = 0.0f;
  const auto take = [&](int i, float4 x, float4 add) {
    x = make_float4(x.x + add.x, x.y + add.y, x.z + add.z, x.w + add.w);
    if (i < QW) {
      sq = fmaf(x.w, x.w, fmaf(x.z, x.z, fmaf(x.y, x.y, fmaf(x.x, x.x, sq))));
    } else {
      sk = fmaf(x.w, x.w, fmaf(x.z, x.z, fmaf(x.y, x.y, fmaf(x.x, x.x, sk))));
      const int g = (i - QW) / d, j = (i - QW) % d;
      store4(v_cache + ((page * G + g) * page_size + prow) * d + j, x);
    }
    *reinterpret_cast<float4*>(row_s + i) = x;
  };
#pragma unroll
  for (int c = 0; c < QK_CACHE; ++c) {
    const int i = 4 * ((int)threadIdx.x + c * QK_THREADS);
    if (i < QW + KW) take(i, v[c], b[c]);
  }
  for (int i = 4 * ((int)threadIdx.x + QK_CACHE * QK_THREADS); i < QW + KW; i += 4 * QK_THREADS)
    take(i, *reinterpret_cast<const float4*>(pr + i), bias(i));

  // an item: four numbers that are not turned, or four pairs of a head
  const int turned = cs != nullptr ? half / 4 : 0, per_head = turned + (cs != nullptr ? d - rot : d) / 4;
  const int items = (H + (write_kv ? G : 0)) * per_head;
  const auto place = [&](int item, int& head, int& j) {
    head = item / per_head;
    const int n = item % per_head;
    j = 4 * (n < turned || cs == nullptr ? n : n + turned);
  };
  const auto weight = [&](int head, int j) {
    return *reinterpret_cast<const float4*>(head < H ? wq + head * d + j : wk + (head - H) * d + j);
  };
  constexpr int AHEAD = 2;
  float4 w[AHEAD][2];
#pragma unroll
  for (int c = 0; c < AHEAD; ++c) {
    const int item = (int)threadIdx.x + c * QK_THREADS;
    if (item >= items) break;
    int head, j;
    place(item, head, j);
    w[c][0] = weight(head, j);
    if (cs != nullptr && j < half) w[c][1] = weight(head, j + half);
  }
  sq = jb::warp_sum(sq), sk = jb::warp_sum(sk);
  if ((threadIdx.x & 31) == 0) scratch[0][threadIdx.x >> 5] = sq, scratch[1][threadIdx.x >> 5] = sk;
  __syncthreads();
  sq = sk = 0.0f;
#pragma unroll
  for (int i = 0; i < QK_THREADS / 32; ++i) sq += scratch[0][i], sk += scratch[1][i];
  const float rq = sqrtf(sq / (float)QW + eps), rk = write_kv ? sqrtf(sk / (float)KW + eps) : 1.0f;
  const auto finish = [&](int item, const float4* early) {
    int head, j;
    place(item, head, j);
    const float r = head < H ? rq : rk;
    TO* out = head < H ? q_out + ((size_t)t * H + head) * d : k_cache + ((page * G + (head - H)) * page_size + prow) * d;
    const auto normed = [&](int at, float4 g) {
      const float4 x = *reinterpret_cast<const float4*>(row_s + head * d + at);
      return make_float4((x.x / r) * g.x, (x.y / r) * g.y, (x.z / r) * g.z, (x.w / r) * g.w);
    };
    float4 u = normed(j, early != nullptr ? early[0] : weight(head, j));
    if (cs != nullptr && j < half) {
      float4 y = normed(j + half, early != nullptr ? early[1] : weight(head, j + half));
      turn4(u, y, cs + 2 * j);
      store4(out + j + half, y);
    }
    store4(out + j, u);
  };
#pragma unroll
  for (int c = 0; c < AHEAD; ++c)
    if ((int)threadIdx.x + c * QK_THREADS < items) finish((int)threadIdx.x + c * QK_THREADS, w[c]);
  for (int item = (int)threadIdx.x + AHEAD * QK_THREADS; item < items; item += QK_THREADS) finish(item, nullptr);
}

template <typename TO>
__global__ void qk_norm_rope_cache_kernel(const float* __restrict__ proj, int ld, const float* __restrict__ bq,
                                          const float* __restrict__ bk, const float* __restrict__ wq,
                                          const float* __restrict__ wk, float eps, const float* __restrict__ table,
                                          int rot, const int* __restrict__ positions, TO* __restrict__ q_out,
                                          const int* __restrict__ dest, TO* __restrict__ k_cache,
                                          TO* __restrict__ v_cache, int H, int G, int d, int dp, int page_size,
                                          int write_kv) {
  extern __shared__ __align__(16) float row_s[];     // q [H d], then k [G d]
  __shared__ float scratch[2][QK_THREADS / 32];
  jb::pdl_launch_dependents();
  jb::pdl_wait();
  const int t = blockIdx.x;
  const int QW = H * d, KW = write_kv ? G * d : 0;
  const float* pr = proj + (size_t)t * ld;
  size_t page = 0;
  int prow = 0;
  if (write_kv) {
    page = (size_t)(dest[t] / page_size);
    prow = dest[t] % page_size;
  }
  float sq = 0.0f, sk = 0.0f;
  // four neighbouring numbers a thread and round, as the kernel above takes them: the same sums bit for bit
  for (int i4 = 4 * (int)threadIdx.x; i4 < QW + KW; i4 += 4 * QK_THREADS) {
    for (int i = i4; i < min(i4 + 4, QW + KW); ++i) {
      float v = pr[i];
      if (i < QW) {
        if (bq != nullptr) v += bq[i];
        sq = fmaf(v, v, sq);
      } else {
        const int c = i - QW;
        if (bk != nullptr) v += bk[c];
        sk = fmaf(v, v, sk);
        const int g = c / d, j = c % d;
        v_cache[((page * G + g) * page_size + prow) * dp + j] = jb::from_f32<TO>(v);
      }
      row_s[i] = v;
    }
  }
  sq = jb::warp_sum(sq), sk = jb::warp_sum(sk);
  if ((threadIdx.x & 31) == 0) scratch[0][threadIdx.x >> 5] = sq, scratch[1][threadIdx.x >> 5] = sk;
  __syncthreads();
  sq = sk = 0.0f;
#pragma unroll
  for (int i = 0; i < QK_THREADS / 32; ++i) sq += scratch[0][i], sk += scratch[1][i];
  const float rq = sqrtf(sq / (float)QW + eps), rk = write_kv ? sqrtf(sk / (float)KW + eps) : 1.0f;
  const int half = rot >> 1;
  const float* cs = (table != nullptr && rot > 0) ? table + (size_t)positions[t] * half * 2 : nullptr;
  // a thread takes a number and, where it is rotated, writes both members of its pair
  for (int i = threadIdx.x; i < QW + KW; i += blockDim.x) {
    const bool is_q = i < QW;
    const int c = is_q ? i : i - QW;
    const int head = c / d, j = c % d;
    const float* w = is_q ? wq : wk;
    const float r = is_q ? rq : rk;
    TO* out = is_q ? q_out + ((size_t)t * H + head) * dp
                   : k_cache + ((page * G + head) * page_size + prow) * dp;
    if (cs != nullptr && j < rot) {
      if (j >= half) continue;                       // written by the thread of the pair's first member
      const float u = (row_s[i] / r) * w[c], v = (row_s[i + half] / r) * w[c + half];
      const float co = cs[2 * j], si = cs[2 * j + 1];
      out[j] = jb::from_f32<TO>(u * co - v * si);
      out[j + half] = jb::from_f32<TO>(v * co + u * si);
    } else {
      out[j] = jb::from_f32<TO>((row_s[i] / r) * w[c]);
    }
  }
  // heads stored wider than they are: the queries' extra columns are zero (those of the pages are never written)
  const int extra = dp - d;
  for (int i = threadIdx.x; i < H * extra; i += blockDim.x)
    q_out[((size_t)t * H + i / extra) * dp + d + i % extra] = jb::from_f32<TO>(0.0f);
}

template <typename TO>
__global__ void latent_prep_kernel(const float* __restrict__ proj, int ld, int Q, int r, int rp, const float* __restrict__ w,
                                   float eps, TO* __restrict__ q_out, const int* __restrict__ dest,
                                   TO* __restrict__ c_cache, int write_c) {
  __shared__ float scratch[33];
  jb::pdl_launch_dependents();
  jb::pdl_wait();
  const int t = blockIdx.x;
  const float* pr = proj + (size_t)t * ld;
  for (int i = threadIdx.x; i < Q; i += blockDim.x) q_out[(size_t)t * Q + i] = jb::from_f32<TO>(pr[i]);
  if (!write_c) return;
  float ss = 0.0f;
  for (int i = threadIdx.x; i < r; i += blockDim.x) ss += pr[Q + i] * pr[Q + i];
  ss = jb::block_sum(ss, scratch);
  const float rms = sqrtf(ss / (float)r + eps);
  TO* out = c_cache + (size_t)dest[t] * rp;         // one key head: row dest[t] of [page * page_size][rp]
  for (int i = threadIdx.x; i < r; i += blockDim.x) out[i] = jb::from_f32<TO>((pr[Q + i] / rms) * w[i]);
}

// latent_prep four numbers a thread and access: blocks (token, slice of the queries), the first slice's also norm the
// latent, whose weight is asked for before the wait.  (8 tokens of 8,192 + 256 numbers: 11 us with one block a token, below 3 so.)
constexpr int LP_THREADS = 256, LP_SLICE = 4 * 4 * LP_THREADS;      // numbers of the queries a block moves, 16 a thread

template <typename TO>
__global__ void __launch_bounds__(LP_THREADS) latent_prep_rows_kernel(const float* __restrict__ proj, int ld, int Q, int r, int rp,
                                                                      const float* __restrict__ w, float eps,
                                                                      TO* __restrict__ q_out, const int* __restrict__ dest,
                                                                      TO* __restrict__ c_cache, int write_c) {
  __shared__ float scratch[LP_THREADS / 32];
  jb::pdl_launch_dependents();
  const int t = blockIdx.x, mine = 4 * (int)threadIdx.x;
  const bool latent = blockIdx.y == 0 && write_c;
  float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f), c = g;
  if (latent && mine < r) g = *reinterpret_cast<const float4*>(w + mine);
  jb::pdl_wait();
  const float* pr = proj + (size_t)t * ld;
  if (latent && mine < r) c = *reinterpret_cast<const float4*>(pr + Q + mine);
  float4 v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = (int)blockIdx.y * LP_SLICE + k * 4 * LP_THREADS + mine;
    if (i < Q) v[k] = *reinterpret_cast<const float4*>(pr + i);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = (int)blockIdx.y * LP_SLICE + k * 4 * LP_THREADS + mine;
    if (i < Q) store4(q_out + (size_t)t * Q + i, v[k]);
  }
  if (!latent) return;
  float ss = jb::warp_sum(c.x * c.x + c.y * c.y + c.z * c.z + c.w * c.w);
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = 0.0f;
#pragma unroll
  for (int i = 0; i < LP_THREADS / 32; ++i) ss += scratch[i];
  const float rms = sqrtf(ss / (float)r + eps);
  if (mine < r)
    store4(c_cache + (size_t)dest[t] * rp + mine, make_float4((c.x / rms) * g.x, (c.y / rms) * g.y, (c.z / rms) * g.z, (c.w / rms) * g.w));
}

// head_norm_rope_cache (grouped-query attention whose queries and keys are normed head by head):
//   q = proj[:, 0 : H d], k = proj[:, H d : (H + G) d], v = proj[:, (H + G) d : (H + G) d + G e]
//   every head of q and of k is divided by its own root mean square over d (eps inside the root) and multiplied by
//   wq (or wk), a weight of size d that all heads share (null: no norm, or with `unit` the division alone, which a
//   rotation commutes with: it keeps every pair's sum of squares); then the first `rot` dimensions are turned as
//   above, and q is multiplied by the query temperature 1 + temp_coef ln(floor((p + 1) / temp_every) + 1) of the
//   token's position p (temp_every 0: none).  With `first` (the value heads of the same tokens in another layer) the value
//   is (1 - mix) v + mix first.  q is written [T, H dp], k is appended to pages whose rows hold dp numbers, v to pages
//   whose rows hold ep (dp >= d, ep >= e; the extra columns of q are zero, those of the pages are never written).  One
//   block per token, a warp per head.
template <typename TO>
__global__ void head_norm_rope_cache_kernel(const float* __restrict__ proj, int ld, const float* __restrict__ wq,
                                            const float* __restrict__ wk, float eps, const float* __restrict__ table,
                                            int rot, const int* __restrict__ positions, TO* __restrict__ q_out,
                                            const int* __restrict__ dest, TO* __restrict__ k_cache,
                                            TO* __restrict__ v_cache, int H, int G, int d, int e, int dp, int ep,
                                            int page_size, int write_kv, int unit, float temp_coef, int temp_every,
                                            const float* __restrict__ first, int ld_first, float mix) {
  jb::pdl_launch_dependents();
  jb::pdl_wait();
  const int t = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const float* pr = proj + (size_t)t * ld;
  size_t page = 0;
  int prow = 0;
  if (write_kv) {
    page = (size_t)(dest[t] / page_size);
    prow = dest[t] % page_size;
  }
  const int half = rot >> 1;
  const float* cs = (table != nullptr && rot > 0) ? table + (size_t)positions[t] * half * 2 : nullptr;
  const int n_heads = H + (write_kv ? 2 * G : 0);
  const float temp = temp_every > 0 ? 1.0f + temp_coef * logf((float)((positions[t] + 1) / temp_every) + 1.0f) : 1.0f;
  for (int head = warp; head < n_heads; head += warps) {
    if (head >= H + G) {                                // a value head: appended as projected, or mixed
      const int g = head - H - G;
      const float* x = pr + (size_t)(H + G) * d + (size_t)g * e;
      TO* out = v_cache + ((page * G + g) * page_size + prow) * ep;
      if (first != nullptr) {
        const float* y = first + (size_t)t * ld_first + (size_t)g * e;
        for (int j = lane; j < e; j += 32) out[j] = jb::from_f32<TO>((1.0f - mix) * x[j] + mix * y[j]);
      } else {
        for (int j = lane; j < e; j += 32) out[j] = jb::from_f32<TO>(x[j]);
      }
      continue;
    }
    const bool is_q = head < H;
    const float* x = pr + (size_t)head * d;
    const float* w = is_q ? wq : wk;
    float inv = 1.0f;
    if (w != nullptr || unit) {
      float ss = 0.0f;
      for (int j = lane; j < d; j += 32) ss = fmaf(x[j], x[j], ss);
      ss = jb::warp_sum(ss);
      inv = 1.0f / sqrtf(ss / (float)d + eps);
    }
    if (is_q) inv *= temp;
    TO* out = is_q ? q_out + ((size_t)t * H + head) * dp
                   : k_cache + ((page * G + (head - H)) * page_size + prow) * dp;
    for (int j = lane; j < d; j += 32) {
      if (cs != nullptr && j < rot) {
        if (j >= half) continue;                        // written with the pair's first member
        const float u = (x[j] * inv) * (w ? w[j] : 1.0f), v = (x[j + half] * inv) * (w ? w[j + half] : 1.0f);
        const float co = cs[2 * j], si = cs[2 * j + 1];
        out[j] = jb::from_f32<TO>(u * co - v * si);
        out[j + half] = jb::from_f32<TO>(v * co + u * si);
      } else {
        out[j] = jb::from_f32<TO>((x[j] * inv) * (w ? w[j] : 1.0f));
      }
    }
    if (is_q)
      for (int j = d + lane; j < dp; j += 32) out[j] = jb::from_f32<TO>(0.0f);
  }
}

// head_norm_rope_cache for heads of at most 128 numbers, four of them a lane (sizes and row starts whole groups of four,
// half a rotation too): a head is one load a lane, pairs meet by shuffles, the shared weights are asked for before the wait.
// (One token of 16 + 2 x 4 heads of 128: 7.1 us with one number a lane and access and three heads a warp one after another,
// 2.7 so.)
// Up to 32 warps a block: more than 64 registers a thread would not launch.
template <typename TO>
__global__ void __launch_bounds__(1024) head_norm_rope_rows_kernel(const float* __restrict__ proj, int ld, const float* __restrict__ wq,
                                           const float* __restrict__ wk, float eps, const float* __restrict__ table, int rot,
                                           const int* __restrict__ positions, TO* __restrict__ q_out,
                                           const int* __restrict__ dest, TO* __restrict__ k_cache, TO* __restrict__ v_cache,
                                           int H, int G, int d, int e, int dp, int ep, int page_size, int write_kv, int unit,
                                           float temp_coef, int temp_every, const float* __restrict__ first, int ld_first,
                                           float mix) {
  jb::pdl_launch_dependents();
  const int t = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5, j = 4 * lane;
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f), one = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
  const float4 gq = wq != nullptr && j < d ? *reinterpret_cast<const float4*>(wq + j) : one;
  const float4 gk = wk != nullptr && j < d ? *reinterpret_cast<const float4*>(wk + j) : one;
  jb::pdl_wait();
  const float* pr = proj + (size_t)t * ld;
  const int n_heads = H + (write_kv ? 2 * G : 0);
  const int at = write_kv ? dest[t] : 0, pos = positions != nullptr ? positions[t] : 0;
  const size_t page = (size_t)(at / page_size);
  const int prow = at % page_size;
  const int half = rot >> 1;
  const float* cs = (table != nullptr && rot > 0) ? table + (size_t)pos * half * 2 : nullptr;
  const float temp = temp_every > 0 ? 1.0f + temp_coef * logf((float)((pos + 1) / temp_every) + 1.0f) : 1.0f;
  float4 c0 = one, c1 = one;                                  // (cos, sin) of this lane's pairs
  if (cs != nullptr && j < rot) {
    const float* p = cs + 2 * (j < half ? j : j - half);
    c0 = *reinterpret_cast<const float4*>(p), c1 = *reinterpret_cast<const float4*>(p + 4);
  }
  for (int head = warp; head < n_heads; head += warps) {
    if (head >= H + G) {                                      // a value head: appended as projected, or mixed
      const int g = head - H - G;
      const float* x = pr + (size_t)(H + G) * d + (size_t)g * e;
      TO* out = v_cache + ((page * G + g) * page_size + prow) * ep;
      for (int i = j; i < e; i += 128) {
        float4 v = *reinterpret_cast<const float4*>(x + i);
        if (first != nullptr) {
          const float4 y = *reinterpret_cast<const float4*>(first + (size_t)t * ld_first + (size_t)g * e + i);
          v = make_float4((1.0f - mix) * v.x + mix * y.x, (1.0f - mix) * v.y + mix * y.y, (1.0f - mix) * v.z + mix * y.z,
                          (1.0f - mix) * v.w + mix * y.w);
        }
        store4(out + i, v);
      }
      continue;
    }
    const bool is_q = head < H;
    float4 x = j < d ? *reinterpret_cast<const float4*>(pr + (size_t)head * d + j) : zero;
    float inv = 1.0f;
    if ((is_q ? wq : wk) != nullptr || unit)
      inv = 1.0f / sqrtf(jb::warp_sum(x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w) / (float)d + eps);
    if (is_q) inv *= temp;
    const float4 g = is_q ? gq : gk;
    x = make_float4((x.x * inv) * g.x, (x.y * inv) * g.y, (x.z * inv) * g.z, (x.w * inv) * g.w);
    if (cs != nullptr) {
      const int other = j < half ? lane + half / 4 : lane - half / 4;
      const float4 y = make_float4(__shfl_sync(0xffffffffu, x.x, other), __shfl_sync(0xffffffffu, x.y, other),
                                   __shfl_sync(0xffffffffu, x.z, other), __shfl_sync(0xffffffffu, x.w, other));
      if (j < half)
        x = make_float4(x.x * c0.x - y.x * c0.y, x.y * c0.z - y.y * c0.w, x.z * c1.x - y.z * c1.y, x.w * c1.z - y.w * c1.w);
      else if (j < rot)
        x = make_float4(x.x * c0.x + y.x * c0.y, x.y * c0.z + y.y * c0.w, x.z * c1.x + y.z * c1.y, x.w * c1.z + y.w * c1.w);
    }
    TO* out = is_q ? q_out + ((size_t)t * H + head) * dp : k_cache + ((page * G + (head - H)) * page_size + prow) * dp;
    if (j < d) store4(out + j, x);
    if (is_q)
      for (int i = j < d ? j + 128 : j; i < dp; i += 128) store4(out + i, zero);
  }
}

// head_norm_rope_cache without norm, rotation and temperature: four numbers a thread (d, e, dp, ep and ld, ld_first whole
// groups of four at aligned addresses).  One block per token.
template <typename TO>
__global__ void __launch_bounds__(256) head_copy_cache_kernel(const float* __restrict__ proj, int ld, TO* __restrict__ q_out,
                                                              const int* __restrict__ dest, TO* __restrict__ k_cache,
                                                              TO* __restrict__ v_cache, int H, int G, int d, int e, int dp,
                                                              int ep, int page_size, int write_kv,
                                                              const float* __restrict__ first, int ld_first, float mix) {
  jb::pdl_launch_dependents();
  jb::pdl_wait();
  const int t = blockIdx.x;
  const float* pr = proj + (size_t)t * ld;
  size_t page = 0;
  int prow = 0;
  if (write_kv) {
    page = (size_t)(dest[t] / page_size);
    prow = dest[t] % page_size;
  }
  const int per_q = dp >> 2, per_k = d >> 2, per_v = e >> 2;
  const int nq = H * per_q, nk = write_kv ? G * per_k : 0, nv = write_kv ? G * per_v : 0;
#pragma unroll 4
  for (int i = threadIdx.x; i < nq + nk + nv; i += 256) {
    if (i < nq) {
      const int h = i / per_q, j = (i - h * per_q) << 2;
      const float4 x = j < d ? *reinterpret_cast<const float4*>(pr + (size_t)h * d + j) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      store4(q_out + ((size_t)t * H + h) * dp + j, x);
    } else if (i < nq + nk) {
      const int c = i - nq, g = c / per_k, j = (c - g * per_k) << 2;
      store4(k_cache + ((page * G + g) * page_size + prow) * dp + j,
             *reinterpret_cast<const float4*>(pr + (size_t)(H + g) * d + j));
    } else {
      const int c = i - nq - nk, g = c / per_v, j = (c - g * per_v) << 2;
      float4 x = *reinterpret_cast<const float4*>(pr + (size_t)(H + G) * d + (size_t)g * e + j);
      if (first != nullptr) {
        const float4 y = *reinterpret_cast<const float4*>(first + (size_t)t * ld_first + (size_t)g * e + j);
        const float own = 1.0f - mix;
        x = make_float4(own * x.x + mix * y.x, own * x.y + mix * y.y, own * x.z + mix * y.z, own * x.w + mix * y.w);
      }
      store4(v_cache + ((page * G + g) * page_size + prow) * ep + j, x);
    }
  }
}

}  // namespace

// proj: float32 [T, ld]; bq [H d], bk [G d] (either may be null), wq [H d], wk [G d] float32; table: float32
// [positions][rot/2][2] or null (no rotation); q_out [T, H dp] and the pages (rows of dp) in out_dtype.  write_kv = 0: q only
// (a place that reads the keys and values another place wrote).
JB_EXPORT int jb_qk_norm_rope_cache(const float* proj, int ld, const float* bq, const float* bk, const float* wq,
                                    const float* wk, float eps, const float* table, int rot, const int* positions,
                                    void* q_out, int out_dtype, const int* dest, void* k_cache, void* v_cache, int T,
                                    int H, int G, int d, int dp, int page_size, int write_kv, cudaStream_t stream) {
  if (T <= 0) return 0;
  JB_REFUSE(dp < d, "qk_norm_rope_cache: heads of %d cannot be stored in %d columns", d, dp);
  JB_REFUSE(rot < 0 || rot > d || (rot & 1), "qk_norm_rope_cache: %d rotated dimensions do not fit a head of %d", rot, d);
  JB_REFUSE(ld < (H + (write_kv ? G : 0)) * d, "qk_norm_rope_cache: rows of %d floats do not hold the projections", ld);
  const size_t smem = (size_t)(H + (write_kv ? G : 0)) * d * sizeof(float);
  JB_REFUSE(smem > 200 * 1024, "qk_norm_rope_cache: a token's projections (%zu bytes) do not fit shared memory", smem);
  cudaError_t e;
  const uintptr_t all = (uintptr_t)proj | (uintptr_t)bq | (uintptr_t)bk | (uintptr_t)wq | (uintptr_t)wk | (uintptr_t)table |
                        (uintptr_t)q_out | (uintptr_t)k_cache | (uintptr_t)v_cache;
  if (d == dp && ((d | ld) & 3) == 0 && (rot & 7) == 0 && (all & 15) == 0) {
    jb::Launch rows(dim3(T), dim3(QK_THREADS), smem, stream);
#define JB_GO(TO)                                                                                                      \
  do {                                                                                                                 \
    if (smem > 47 * 1024) {                                                                                            \
      e = cudaFuncSetAttribute(qk_norm_rope_rows_kernel<TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);  \
      if (e != cudaSuccess) return (int)e;                                                                             \
    }                                                                                                                  \
    return (int)cudaLaunchKernelEx(&rows.c, qk_norm_rope_rows_kernel<TO>, proj, ld, bq, bk, wq, wk, eps, table, rot,   \
                                   positions, (TO*)q_out, dest, (TO*)k_cache, (TO*)v_cache, H, G, d, page_size, write_kv); \
  } while (0)
    if (out_dtype == JB_F32) JB_GO(float);
    if (out_dtype == JB_BF16) JB_GO(bf16);
#undef JB_GO
  }
  jb::Launch cfg(dim3(T), dim3(QK_THREADS), smem, stream);
#define JB_LAUNCH_QK(TO)                                                                                               \
  do {                                                                                                                 \
    if (smem > 47 * 1024) {                                                                                            \
      e = cudaFuncSetAttribute(qk_norm_rope_cache_kernel<TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
      if (e != cudaSuccess) return (int)e;                                                                             \
    }                                                                                                                  \
    e = cudaLaunchKernelEx(&cfg.c, qk_norm_rope_cache_kernel<TO>, proj, ld, bq, bk, wq, wk, eps, table, rot,           \
                           positions, (TO*)q_out, dest, (TO*)k_cache, (TO*)v_cache, H, G, d, dp, page_size, write_kv);\
  } while (0)
  if (out_dtype == JB_F32) JB_LAUNCH_QK(float);
  else if (out_dtype == JB_BF16) JB_LAUNCH_QK(bf16);
  else return JB_ERR_BAD_DTYPE;
#undef JB_LAUNCH_QK
  return (int)e;
}

// proj: float32 [T, ld] with the queries in columns [0, Q) and the latent projection in [Q, Q + r); w [r] float32;
// q_out [T, Q] and the pages ([page][1][page_size][rp], rp >= r the size a row is stored with, extra columns never
// written) in out_dtype.  write_c = 0: queries only.
JB_EXPORT int jb_latent_prep(const float* proj, int ld, int Q, int r, int rp, const float* w, float eps, void* q_out,
                             int out_dtype, const int* dest, void* c_cache, int T, int write_c, cudaStream_t stream) {
  if (T <= 0) return 0;
  JB_REFUSE(ld < Q + (write_c ? r : 0) || rp < r, "latent_prep: rows of %d floats do not hold the projections", ld);
  cudaError_t e;
  const uintptr_t all = (uintptr_t)proj | (uintptr_t)w | (uintptr_t)q_out | (uintptr_t)c_cache;
  if (((ld | Q | r | rp) & 3) == 0 && r <= 4 * LP_THREADS && (all & 15) == 0) {
    const int slices = Q > 0 ? (Q + LP_SLICE - 1) / LP_SLICE : 1;
    jb::Launch rows(dim3(T, slices), dim3(LP_THREADS), 0, stream);
    if (slices <= 65535 && out_dtype == JB_F32)
      return (int)cudaLaunchKernelEx(&rows.c, latent_prep_rows_kernel<float>, proj, ld, Q, r, rp, w, eps, (float*)q_out, dest,
                                     (float*)c_cache, write_c);
    if (slices <= 65535 && out_dtype == JB_BF16)
      return (int)cudaLaunchKernelEx(&rows.c, latent_prep_rows_kernel<bf16>, proj, ld, Q, r, rp, w, eps, (bf16*)q_out, dest,
                                     (bf16*)c_cache, write_c);
  }
  jb::Launch cfg(dim3(T), dim3(256), 0, stream);
  if (out_dtype == JB_F32)
    e = cudaLaunchKernelEx(&cfg.c, latent_prep_kernel<float>, proj, ld, Q, r, rp, w, eps, (float*)q_out, dest,
                           (float*)c_cache, write_c);
  else if (out_dtype == JB_BF16)
    e = cudaLaunchKernelEx(&cfg.c, latent_prep_kernel<bf16>, proj, ld, Q, r, rp, w, eps, (bf16*)q_out, dest,
                           (bf16*)c_cache, write_c);
  else
    return JB_ERR_BAD_DTYPE;
  return (int)e;
}

// proj: float32 [T, ld] = [q: H d | k: G d | v: G e]; wq, wk: float32 [d] or null; table: float32 [positions][rot/2][2]
// or null; q_out [T, H dp] and the pages (rows of dp for keys, ep for values) in out_dtype.  write_kv = 0: q only.  unit = 1:
// heads are divided by their root mean square also without a weight.  temp_every > 0: the query temperature.  first
// (float32 rows of ld_first numbers, [G e] of each token, or null): values are mixed with it.
JB_EXPORT int jb_head_norm_rope_cache(const float* proj, int ld, const float* wq, const float* wk, float eps,
                                      const float* table, int rot, const int* positions, void* q_out, int out_dtype,
                                      const int* dest, void* k_cache, void* v_cache, int T, int H, int G, int d, int e,
                                      int dp, int ep, int page_size, int write_kv, int unit, float temp_coef,
                                      int temp_every, const float* first, int ld_first, float mix, cudaStream_t stream) {
  if (T <= 0) return 0;
  JB_REFUSE(dp < d || ep < e, "head_norm_rope_cache: heads of %d and %d cannot be stored in %d and %d columns", d, e, dp, ep);
  JB_REFUSE(rot < 0 || rot > d || (rot & 1), "head_norm_rope_cache: %d rotated dimensions do not fit a head of %d", rot, d);
  JB_REFUSE(ld < H * d + (write_kv ? G * (d + e) : 0), "head_norm_rope_cache: rows of %d floats do not hold the projections", ld);
  const bool plain = wq == nullptr && wk == nullptr && !unit && temp_every == 0 && (table == nullptr || rot == 0);
  if (plain && ((d | e | dp | ep | ld | ld_first) & 3) == 0 &&
      (((uintptr_t)proj | (uintptr_t)q_out | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)first) & 15) == 0) {
    jb::Launch pcfg(dim3(T), dim3(256), 0, stream);
    if (out_dtype == JB_F32)
      return (int)cudaLaunchKernelEx(&pcfg.c, head_copy_cache_kernel<float>, proj, ld, (float*)q_out, dest, (float*)k_cache,
                                     (float*)v_cache, H, G, d, e, dp, ep, page_size, write_kv, first, ld_first, mix);
    if (out_dtype == JB_BF16)
      return (int)cudaLaunchKernelEx(&pcfg.c, head_copy_cache_kernel<bf16>, proj, ld, (bf16*)q_out, dest, (bf16*)k_cache,
                                     (bf16*)v_cache, H, G, d, e, dp, ep, page_size, write_kv, first, ld_first, mix);
  }
  const int heads = H + (write_kv ? 2 * G : 0);
  cudaError_t err;
  const uintptr_t all = (uintptr_t)proj | (uintptr_t)wq | (uintptr_t)wk | (uintptr_t)table | (uintptr_t)q_out |
                        (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)first;
  if (d <= 128 && ((d | e | dp | ep | ld | (first != nullptr ? ld_first : 0)) & 3) == 0 && (rot & 7) == 0 && (all & 15) == 0) {
    // few tokens: a warp a head; many: eight warps a token, what an SM has in flight are its blocks
    const int warps = T <= 296 ? (heads < 32 ? heads : 32) : (heads < 8 ? heads : 8);
    jb::Launch rows(dim3(T), dim3(32 * warps), 0, stream);
    if (out_dtype == JB_F32)
      return (int)cudaLaunchKernelEx(&rows.c, head_norm_rope_rows_kernel<float>, proj, ld, wq, wk, eps, table, rot, positions,
                                     (float*)q_out, dest, (float*)k_cache, (float*)v_cache, H, G, d, e, dp, ep, page_size,
                                     write_kv, unit, temp_coef, temp_every, first, ld_first, mix);
    if (out_dtype == JB_BF16)
      return (int)cudaLaunchKernelEx(&rows.c, head_norm_rope_rows_kernel<bf16>, proj, ld, wq, wk, eps, table, rot, positions,
                                     (bf16*)q_out, dest, (bf16*)k_cache, (bf16*)v_cache, H, G, d, e, dp, ep, page_size,
                                     write_kv, unit, temp_coef, temp_every, first, ld_first, mix);
  }
  jb::Launch cfg(dim3(T), dim3(heads >= 8 ? 256 : heads >= 4 ? 128 : 64), 0, stream);
  if (out_dtype == JB_F32)
    err = cudaLaunchKernelEx(&cfg.c, head_norm_rope_cache_kernel<float>, proj, ld, wq, wk, eps, table, rot, positions,
                             (float*)q_out, dest, (float*)k_cache, (float*)v_cache, H, G, d, e, dp, ep, page_size,
                             write_kv, unit, temp_coef, temp_every, first, ld_first, mix);
  else if (out_dtype == JB_BF16)
    err = cudaLaunchKernelEx(&cfg.c, head_norm_rope_cache_kernel<bf16>, proj, ld, wq, wk, eps, table, rot, positions,
                             (bf16*)q_out, dest, (bf16*)k_cache, (bf16*)v_cache, H, G, d, e, dp, ep, page_size,
                             write_kv, unit, temp_coef, temp_every, first, ld_first, mix);
  else
    return JB_ERR_BAD_DTYPE;
  return (int)err;
}
