// One token of a recurrence with a matrix state per head, from the projections to the gated heads, in one launch: steps in
// which every sequence brings a single token.  A block owns a (sequence, head): the gates' numbers, the state's update and
// read-out, the head's norm and its output gate.  All arithmetic is float32; the formulas are those of delta_rule.cu,
// gated_linear.cu and of `head_norm_gate` in layer_norm.cu.
//   DELTA    S <- g S;  w = beta (v - S^T k);  S <- S + k w^T;  o = S^T q        (k, q unit vectors, q times d^-1/2)
//   MEMORY   S <- f S + i k v^T;  n <- f n + i k;  o = S^T q / max(|n . q|, exp(-m))    (gates with a running maximum m)
//   CHANNEL  S <- diag(a) S + k v^T;  o = S^T q            (a: a decay per key channel from a product of low rank)
//   out[h] = o / rms(o) * weight * act(gate[h])
// What bounds it: the state's bytes for many heads, else a chain of loads and sums, which the launches of its parts made three
// times.  In a captured step of 8 sequences, 16 heads of 128 x 128 (17 MB of state, 2.7 us): matrix memory, gates 3.0 +
// recurrence 4.1 + norm 4.1 us, here 6.9; channel decays 11.8 + 4.1 + 4.1 us, here 6.9.  One sequence of the delta rule is
// level with its walk and norm, a launch less.  Where many small heads lose by it is at `head_step_pays` in ops.py.  512 threads
// hold a head's state of up to 128 x 256 numbers in registers: a thread four columns of every ROWS-th row, all of its loads in
// flight before the gates are known.
#include <math_constants.h>
#include <stdio.h>

#include "common.cuh"

namespace {

typedef __nv_bfloat16 bf16;
constexpr int THREADS = 512, MAX_D = 128, MAX_E = 256;
constexpr float DEN_FLOOR = 1e-6f;
enum Kind { DELTA = 0, MEMORY = 1, CHANNEL = 2 };
enum Act { SILU = 0, SIGMOID = 1 };

__device__ __forceinline__ float log_sigmoid(float z) { return fminf(z, 0.0f) - log1pf(expf(-fabsf(z))); }

struct Args {
  const float* rows;       // [T][ld]: q, k and v (and what the gates come from, unless `raw` holds it)
  int ld, q_col, k_col, v_col;
  float q_scale;
  const float* raw;        // [T][ld_raw]: DELTA: b at col_a, a at col_b; MEMORY: i at col_a, f at col_b; CHANNEL: rank numbers at col_a
  int ld_raw, col_a, col_b;
  const float* p0;         // DELTA: A_log [H]; MEMORY: bias of i [H]; CHANNEL: the second matrix, transposed [rank][H d]
  const float* p1;         // DELTA: dt_bias [H]; MEMORY: bias of f [H]; CHANNEL: bias [H d]
  float scalar;            // DELTA: eps of the unit vectors; MEMORY: the gates' cap; CHANNEL: 1 / tau
  int rank;
  float* state;
  long long slot_stride, state_off, m_off;
  const float* gate;       // [T][ld_gate], head h at columns [h e, (h + 1) e)
  int ld_gate;
  const float* weight;
  int w_stride, act;       // a head's weight lies at w_stride h
  float eps;
  const int* q_start;
  const int* seq_slot;
  int H, G, d, e;
};

// CG: groups of four columns, CG * 4 >= e
template <int KIND, int CG, typename TO>
__global__ void __launch_bounds__(THREADS, CG <= 32 ? 2 : 1) head_step_kernel(const __grid_constant__ Args p, TO* __restrict__ out) {
  constexpr int ROWS = THREADS / CG, RI = MAX_D / ROWS, COLS = 4 * CG;
  __shared__ float q_s[MAX_D], k_s[MAX_D], a_s[MAX_D], parts_s[4][MAX_D];
  __shared__ __align__(16) float sums_s[KIND == DELTA ? 2 : 1][ROWS][COLS];
  __shared__ __align__(16) float w_s[COLS];
  __shared__ float o_s[COLS], nq_s[THREADS / 32];
  jb::pdl_launch_dependents();
  const int seq = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int d = p.d, e = p.e, ex = e + (KIND == MEMORY ? 1 : 0);
  const int col = tid % CG, row = tid / CG, j = 4 * col;
  const bool in = j < e;
  const float head0 = KIND == CHANNEL ? 0.0f : p.p0[h], head1 = KIND == CHANNEL ? 0.0f : p.p1[h];
  jb::pdl_wait();
  const size_t t = (size_t)p.q_start[seq];
  float* slot = p.state + (size_t)p.seq_slot[seq] * p.slot_stride;
  float* st = slot + p.state_off + (size_t)h * d * ex;
  float4 S[RI];
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const int r = row + ROWS * i;
    S[i] = in && r < d ? *reinterpret_cast<const float4*>(st + (size_t)r * e + j) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  const float* x = p.rows + t * p.ld;
  const float* raw = p.raw + t * p.ld_raw;
  const int kv = KIND == DELTA ? h / (p.H / p.G) : h;
  float n_r = 0.0f;
  if (tid < d) {
    q_s[tid] = x[p.q_col + (size_t)kv * d + tid];
    k_s[tid] = x[p.k_col + (size_t)kv * d + tid];
    if (KIND == MEMORY) n_r = st[(size_t)d * e + tid];
  }
  float v_c = 0.0f, z_c = 0.0f, w_c = 0.0f;                     // of column tid
  if (tid < e) {
    v_c = x[p.v_col + (size_t)h * e + tid];
    z_c = p.gate[t * p.ld_gate + (size_t)h * e + tid];
    w_c = p.weight[(size_t)h * p.w_stride + tid];
  }
  float keep = 0.0f, take = 0.0f, m_new = 0.0f;                 // MEMORY; DELTA: decay and beta
  if (KIND == MEMORY) {
    const float m = slot[p.m_off + h];
    const float gi = p.scalar * tanhf((raw[p.col_a + h] + head0) / p.scalar);
    const float gf = log_sigmoid(p.scalar * tanhf((raw[p.col_b + h] + head1) / p.scalar));
    m_new = fmaxf(gf + m, gi);
    keep = expf(gf + m - m_new), take = expf(gi - m_new);
  }
  if (KIND == DELTA) {
    const float z = raw[p.col_b + h] + head1;
    keep = expf(-expf(head0) * (z > 20.0f ? z : log1pf(expf(z))));
    take = 1.0f / (1.0f + expf(-raw[p.col_a + h]));
  }
  if (KIND == CHANNEL) {                                        // four threads a channel, each a quarter of the rank
    const int r = tid & (MAX_D - 1), part = tid / MAX_D, per = (p.rank + 3) / 4, C = p.H * d;
    float z = 0.0f;
    if (r < d) {
      const int last = min(p.rank, (part + 1) * per);
#pragma unroll 8
      for (int i = part * per; i < last; ++i) z = fmaf(p.p0[(size_t)i * C + (size_t)h * d + r], raw[p.col_a + i], z);
    }
    parts_s[part][r] = z;
    __syncthreads();
    if (tid < d) {
      z = p.p1[(size_t)h * d + tid] + ((parts_s[0][tid] + parts_s[1][tid]) + (parts_s[2][tid] + parts_s[3][tid]));
      a_s[tid] = expf(log_sigmoid(z) * p.scalar);
    }
  }
  if (KIND != DELTA && tid < e) w_s[tid] = v_c * (KIND == MEMORY ? take : 1.0f);
  __syncthreads();
  if (KIND == MEMORY && tid == 0) slot[p.m_off + h] = m_new;    // every thread has read the old one

  float iq = 1.0f, ik = 1.0f, qk = 0.0f;
  if (KIND == DELTA) {
    float sq = 0.0f, sk = 0.0f;
    for (int r = lane; r < d; r += 32) sq = fmaf(q_s[r], q_s[r], sq), sk = fmaf(k_s[r], k_s[r], sk), qk = fmaf(q_s[r], k_s[r], qk);
    iq = p.q_scale / sqrtf(jb::warp_sum(sq) + p.scalar);
    ik = 1.0f / sqrtf(jb::warp_sum(sk) + p.scalar);
    qk = jb::warp_sum(qk) * iq * ik;
  }
  float4 y = make_float4(0.0f, 0.0f, 0.0f, 0.0f), u = y;
  if (KIND == DELTA) {
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const int r = row + ROWS * i;
      if (r < d) {
        const float qr = q_s[r], kr = k_s[r];
        y.x = fmaf(S[i].x, qr, y.x), y.y = fmaf(S[i].y, qr, y.y), y.z = fmaf(S[i].z, qr, y.z), y.w = fmaf(S[i].w, qr, y.w);
        u.x = fmaf(S[i].x, kr, u.x), u.y = fmaf(S[i].y, kr, u.y), u.z = fmaf(S[i].z, kr, u.z), u.w = fmaf(S[i].w, kr, u.w);
      }
    }
    *reinterpret_cast<float4*>(&sums_s[KIND == DELTA ? 1 : 0][row][j]) = u;
  } else {
    const float4 v = in ? *reinterpret_cast<const float4*>(w_s + j) : y;
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const int r = row + ROWS * i;
      if (in && r < d) {
        const float ar = KIND == MEMORY ? keep : a_s[r], kr = k_s[r], qr = q_s[r];
        S[i] = make_float4(fmaf(ar, S[i].x, kr * v.x), fmaf(ar, S[i].y, kr * v.y), fmaf(ar, S[i].z, kr * v.z),
                           fmaf(ar, S[i].w, kr * v.w));
        *reinterpret_cast<float4*>(st + (size_t)r * e + j) = S[i];
        y.x = fmaf(S[i].x, qr, y.x), y.y = fmaf(S[i].y, qr, y.y), y.z = fmaf(S[i].z, qr, y.z), y.w = fmaf(S[i].w, qr, y.w);
      }
    }
  }
  *reinterpret_cast<float4*>(&sums_s[0][row][j]) = y;
  if (KIND == MEMORY && warp < MAX_D / 32) {
    float nq = 0.0f;
    if (tid < d) {
      n_r = fmaf(keep, n_r, k_s[tid] * take);
      st[(size_t)d * e + tid] = n_r;
      nq = n_r * q_s[tid];
    }
    nq = jb::warp_sum(nq);
    if (lane == 0) nq_s[warp] = nq;
  }
  __syncthreads();
  if (tid < COLS) {
    float o = 0.0f;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) o += sums_s[0][r][tid];
    if (KIND == DELTA) {
      float a = 0.0f;
#pragma unroll
      for (int r = 0; r < ROWS; ++r) a += sums_s[KIND == DELTA ? 1 : 0][r][tid];
      const float w = take * (v_c - keep * (a * ik));
      w_s[tid] = w;
      o = keep * (o * iq) + qk * w;
    } else if (KIND == MEMORY) {
      const float nq = (nq_s[0] + nq_s[1]) + (nq_s[2] + nq_s[3]);
      o = o * p.q_scale / (fmaxf(fabsf(nq * p.q_scale), expf(-m_new)) + DEN_FLOOR);
    } else {
      o = o * p.q_scale;
    }
    o_s[tid] = tid < e ? o : 0.0f;
  }
  __syncthreads();
  if (tid < COLS) {
    float ss = 0.0f;
#pragma unroll
    for (int c = lane; c < COLS; c += 32) ss = fmaf(o_s[c], o_s[c], ss);
    ss = jb::warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)e + p.eps), s = 1.0f / (1.0f + expf(-z_c));
    if (tid < e) out[(t * p.H + h) * e + tid] = jb::from_f32<TO>(((o_s[tid] * inv) * w_c) * (p.act == SILU ? z_c * s : s));
  }
  if (KIND == DELTA && in) {
    const float4 w = *reinterpret_cast<const float4*>(w_s + j);
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const int r = row + ROWS * i;
      if (r < d) {
        const float kr = k_s[r] * ik;
        *reinterpret_cast<float4*>(st + (size_t)r * e + j) =
            make_float4(fmaf(keep, S[i].x, kr * w.x), fmaf(keep, S[i].y, kr * w.y), fmaf(keep, S[i].z, kr * w.z),
                        fmaf(keep, S[i].w, kr * w.w));
      }
    }
  }
}

template <int KIND>
int launch(const Args& p, void* out, int out_dtype, int n_seqs, cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  const int ex = p.e + (KIND == MEMORY ? 1 : 0);
  JB_REFUSE(p.d < 1 || p.d > MAX_D || p.e < 4 || p.e > MAX_E || p.e % 4 || ((long long)p.d * ex) % 4 || p.slot_stride % 4 ||
                p.state_off % 4 || ((uintptr_t)p.state & 15),
            "head_step: heads of %d x %d are not whole 16-byte vectors of at most %d x %d", p.d, p.e, MAX_D, MAX_E);
  JB_REFUSE(p.H < 1 || p.H > 65535 || p.G < 1 || p.H % p.G || (KIND != DELTA && p.G != p.H), "head_step: %d heads of %d", p.H, p.G);
  const long long keys = (long long)p.G * p.d, values = (long long)p.H * p.e, from_a = KIND == CHANNEL ? p.rank : p.H;
  JB_REFUSE(p.q_col < 0 || p.k_col < 0 || p.v_col < 0 || p.q_col + keys > p.ld || p.k_col + keys > p.ld || p.v_col + values > p.ld ||
                p.col_a < 0 || from_a < 0 || p.col_a + from_a > p.ld_raw ||
                (KIND != CHANNEL && (p.col_b < 0 || p.col_b + (long long)p.H > p.ld_raw)),
            "head_step: columns %d, %d, %d of %d and %d, %d of %d do not hold %d heads of %d x %d", p.q_col, p.k_col, p.v_col, p.ld,
            p.col_a, p.col_b, p.ld_raw, p.H, p.d, p.e);
  JB_REFUSE(p.state_off < 0 || p.state_off + (long long)p.H * p.d * ex > p.slot_stride ||
                (KIND == MEMORY && (p.m_off < 0 || p.m_off + p.H > p.slot_stride)),
            "head_step: slots of %lld numbers do not hold the state", p.slot_stride);
  jb::Launch cfg(dim3(n_seqs, p.H), dim3(THREADS), 0, stream);
#define JB_GO(CG)                                                                                                 \
  return out_dtype == JB_F32 ? (int)cudaLaunchKernelEx(&cfg.c, head_step_kernel<KIND, CG, float>, p, (float*)out) \
                             : (int)cudaLaunchKernelEx(&cfg.c, head_step_kernel<KIND, CG, bf16>, p, (bf16*)out)
  if (out_dtype != JB_F32 && out_dtype != JB_BF16) return JB_ERR_BAD_DTYPE;
  if (p.e <= 64) JB_GO(16);
  if (p.e <= 128) JB_GO(32);
  JB_GO(64);
#undef JB_GO
}

}  // namespace

// Every sequence brings one token, row q_start[seq] of the matrices.  state: float32 rows of slot_stride floats, a slot's
// heads one after another at state_off, each [d][e] (MEMORY: then [d] of the normalizer; the heads' maxima at m_off).
// out: [T, H e] in out_dtype.  `kind`: 0 the delta rule, 1 the matrix memory, 2 decays per key channel; see Args.
JB_EXPORT int jb_head_step(int kind, const float* rows, int ld, int q_col, int k_col, int v_col, float q_scale, const float* raw,
                           int ld_raw, int col_a, int col_b, const float* p0, const float* p1, float scalar, int rank,
                           float* state, long long slot_stride, long long state_off, long long m_off, const float* gate,
                           int ld_gate, const float* weight, int w_stride, int act, float eps, void* out, int out_dtype,
                           const int* q_start, const int* seq_slot, int n_seqs, int H, int G, int d, int e,
                           cudaStream_t stream) {
  const Args p{rows, ld, q_col, k_col, v_col, q_scale, raw, ld_raw, col_a, col_b, p0, p1, scalar, rank, state, slot_stride,
               state_off, m_off, gate, ld_gate, weight, w_stride, act, eps, q_start, seq_slot, H, G, d, e};
  switch (kind) {
    case DELTA: return launch<DELTA>(p, out, out_dtype, n_seqs, stream);
    case MEMORY: return launch<MEMORY>(p, out, out_dtype, n_seqs, stream);
    case CHANNEL: return launch<CHANNEL>(p, out, out_dtype, n_seqs, stream);
    default: return JB_ERR_BAD_SIZE;
  }
}
