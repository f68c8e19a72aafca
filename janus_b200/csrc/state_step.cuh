// One token of a recurrence with a matrix state S [d][e] per head, S <- diag(a) S + k v^T, y = S^T q, for steps of one token
// a sequence: the state is read and written once and everything about it is in flight together.  A block of 256 threads
// owns 64 columns of a head: a thread four columns of every sixteenth row, RI rows.  Bound by the state's bytes; as a walk
// over one token the loads follow one another in rounds.
#pragma once
#include "common.cuh"

namespace jb {

constexpr int STEP_THREADS = 256, STEP_COLS = 64, STEP_ROWS = 16;

// Rows row, row + 16, ... of the four columns at `st` (in: they exist); a(r), k(r), q(r) are loaded for all rows first.
template <int RI, class A, class K, class Q>
__device__ __forceinline__ float4 state_step(float* __restrict__ st, int e, bool in, int d, int row, float4 v, A a, K k, Q q) {
  float4 S[RI], y = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float ar[RI], kr[RI], qr[RI];
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const int r = row + STEP_ROWS * i;
    if (in && r < d) {
      S[i] = *reinterpret_cast<const float4*>(st + (size_t)r * e);
      ar[i] = a(r), kr[i] = k(r), qr[i] = q(r);
    }
  }
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const int r = row + STEP_ROWS * i;
    if (in && r < d) {
      S[i] = make_float4(fmaf(ar[i], S[i].x, kr[i] * v.x), fmaf(ar[i], S[i].y, kr[i] * v.y), fmaf(ar[i], S[i].z, kr[i] * v.z),
                         fmaf(ar[i], S[i].w, kr[i] * v.w));
      *reinterpret_cast<float4*>(st + (size_t)r * e) = S[i];
      y.x = fmaf(S[i].x, qr[i], y.x), y.y = fmaf(S[i].y, qr[i], y.y);
      y.z = fmaf(S[i].z, qr[i], y.z), y.w = fmaf(S[i].w, qr[i], y.w);
    }
  }
  return y;
}

// The block's sums over its rows: column c of the 64 ends in thread c (others: 0).  Threads are (row, 16 groups of columns).
__device__ __forceinline__ float step_columns(float4 y, float4 (*sums)[STEP_COLS / 4]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  y.x += __shfl_xor_sync(0xffffffffu, y.x, 16), y.y += __shfl_xor_sync(0xffffffffu, y.y, 16);
  y.z += __shfl_xor_sync(0xffffffffu, y.z, 16), y.w += __shfl_xor_sync(0xffffffffu, y.w, 16);
  if (lane < 16) sums[warp][lane] = y;
  __syncthreads();
  float total = 0.0f;
  if (threadIdx.x < STEP_COLS) {
#pragma unroll
    for (int w = 0; w < STEP_THREADS / 32; ++w) total += reinterpret_cast<const float*>(sums[w])[threadIdx.x];
  }
  return total;
}

}  // namespace jb
