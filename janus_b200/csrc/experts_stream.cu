// Experts' feed-forwards for steps of up to 64 tokens, the weights streamed from their packed tiles: what every chosen expert
// makes of its tokens, for any choice, without the host.
//   z[pair] = [Wg_e; Wu_e] x[token]        (float32, slices of k meet by adds; z is zero before)
//   act[pair] = act(s z_gate) * (s z_up)   (bfloat16; s the pair's weight where it multiplies the input, else 1)
//   out[token] += s Wd_e act[pair]         (s where the weight multiplies the output, else 1)
// A pair is a token's choice, pair = token * top + choice; the weight on the input is applied to the float32 sums, which a
// product without a bias allows.
//
// What bounds both products is the chosen experts' bytes, so they are cut for even streams and nothing else: the tiles of
// 128 rows x 64 columns (16 KB each, as jb_pack_weight_bf16 lays them out) of all chosen experts are numbered expert by
// expert, row tile by row tile, k tile by k tile, and each of 148 CTAs takes one run of them, as long as every other's to a
// tile.  A run ends and begins in the middle of a row tile; the parts meet in z or out.  All tokens of the step are columns
// of every expert's product (16, 32 or 64 of them): a column that did not choose the expert is computed and left out.
// Blocks of 16 rows with mma.sync (expert_tc_kernel) read the weights row by row, for two tokens of 8 experts of 7,168 x 4,096
// in 6.05 waves.  Both products of a layer in a captured step, microseconds, by such blocks and here (the activation's launch
// included): these two tokens 114 and 106 (their experts' bytes at the copy rate: 99), 64 tokens 381 and 228 (215); of 4,096 x
// 2,048, one token 29 and 28 (15), 16 tokens 74 and 74 (61), 64 tokens 129 and 84; of 1,536 x 1,024, where start and end are the
// most of it, 8 tokens 19 and 23 (10): the callers' line is `experts_stream_pays` in ops.py.
#include <stdio.h>

#include "tc_common.cuh"

namespace {

typedef __nv_bfloat16 bf16;
constexpr int BM = 128, BK = 64, UMMA_K = 16, W_BYTES = BM * BK * 2;
constexpr int MAX_EXPERTS = 512, MAX_PLACES = 8192;              // experts; chosen experts x tokens
constexpr int THREADS = 192, RING_BYTES = 200 * 1024;

template <int BN>
struct Cfg {
  static constexpr int STAGE = W_BYTES + BN * BK * 2;
  static constexpr int STAGES = RING_BYTES / STAGE;
  static constexpr int TMEM = 2 * BN <= 32 ? 32 : 2 * BN <= 64 ? 64 : 128;
  static constexpr int BARS = 2 * STAGES + 4;
  static constexpr int smem(int places) { return 1024 + STAGES * STAGE + 8 * BARS + 16 + 2 * places; }
};

// The chosen experts in order: `slot_of` (in shared memory) becomes an expert's place among them, -1 where it was not chosen.
// Returns how many there are.  All threads of the block.
__device__ __forceinline__ int list_experts(const int* __restrict__ sel_e, int pairs, int E, short* slot_of, int* count) {
  for (int e = threadIdx.x; e < E; e += blockDim.x) slot_of[e] = -1;
  __syncthreads();
  for (int i = threadIdx.x; i < pairs; i += blockDim.x) slot_of[sel_e[i]] = 0;
  __syncthreads();
  if (threadIdx.x < 32) {
    int n = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + threadIdx.x;
      const bool used = e < E && slot_of[e] == 0;
      const unsigned mask = __ballot_sync(0xffffffffu, used);
      if (used) slot_of[e] = (short)(n + __popc(mask & ((1u << threadIdx.x) - 1u)));
      n += __popc(mask);
    }
    if (threadIdx.x == 0) *count = n;
  }
  __syncthreads();
  return *count;
}

// MATS = 2: Y = z [pairs][2 R] (gate rows, then up rows), the experts' input are the T rows of X; MATS = 1: Y = out [T][R],
// expert number s reads rows [s T, (s + 1) T) of X.  R: rows of one matrix, a multiple of 128.  up_tiles: where the up
// matrices' row tiles begin.  pair_slot (MATS = 2): block 0 leaves every pair's expert's place there.
template <int BN, int MATS>
__global__ void __launch_bounds__(THREADS, 1) experts_stream_kernel(
    const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const int* __restrict__ sel_e,
    const float* __restrict__ out_w, int T, int top, int E, int R, int k_tiles, int up_tiles, float* __restrict__ Y,
    int* __restrict__ pair_slot, int* __restrict__ status) {
  using C = Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ short slot_of[MAX_EXPERTS], expert_at[MAX_EXPERTS];
  __shared__ int count;
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + C::STAGES * C::STAGE);
  uint32_t* tmem_slot = (uint32_t*)(bars + C::BARS);
  short* pair_of = (short*)(tmem_slot + 4);                      // [chosen expert][token]: the pair, or -1
  const uint32_t base = jb::smem_u32(smem), full0 = jb::smem_u32(bars), empty0 = full0 + 8 * C::STAGES,
                 acc_full0 = full0 + 16 * C::STAGES, acc_empty0 = acc_full0 + 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, pairs = T * top;
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      jb::mbar_init(full0 + 8 * s, 1);
      jb::mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      jb::mbar_init(acc_full0 + 8 * b, 1);
      jb::mbar_init(acc_empty0 + 8 * b, 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) jb::tmem_alloc<C::TMEM>(jb::smem_u32(tmem_slot));
  jb::tc_fence_before();
  __syncthreads();
  jb::tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  jb::pdl_launch_dependents();          // not before: a block of the kernel behind this one may ask for TMEM columns too
  jb::pdl_wait();
  const int n = list_experts(sel_e, pairs, E, slot_of, &count);
  for (int e = threadIdx.x; e < E; e += THREADS)
    if (slot_of[e] >= 0) expert_at[slot_of[e]] = (short)e;
  for (int i = threadIdx.x; i < n * T; i += THREADS) pair_of[i] = -1;
  __syncthreads();
  for (int i = threadIdx.x; i < pairs; i += THREADS) {
    pair_of[slot_of[sel_e[i]] * T + i / top] = (short)i;
    if (MATS == 2 && blockIdx.x == 0) pair_slot[i] = slot_of[sel_e[i]];
  }
  __syncthreads();

  const int tiles_m = R / BM, row_tiles = MATS * tiles_m;        // of one matrix, of one expert
  const long long all = (long long)n * row_tiles * k_tiles;
  const int first = (int)(all * blockIdx.x / gridDim.x), last = (int)(all * (blockIdx.x + 1) / gridDim.x);   // this block's run
  if (warp == 0) {
    // ---------------- producer ----------------
    if (lane == 0) {
      const uint64_t policy = jb::read_once_policy();
      int rt = first / k_tiles, kt = first % k_tiles;
      for (int i = first, it = 0; i < last; ++i, ++it) {
        const int s = it % C::STAGES;
        if (it >= C::STAGES && !jb::mbar_wait(empty0 + 8 * s, (it / C::STAGES - 1) & 1, status, 41)) break;
        const int place = rt / row_tiles, m = rt % row_tiles, e = expert_at[place];
        const int tile = MATS == 2 && m >= tiles_m ? up_tiles + e * tiles_m + m - tiles_m : e * tiles_m + m;
        const uint32_t stage = base + s * C::STAGE, bar = full0 + 8 * s;
        jb::mbar_expect_tx(bar, C::STAGE);
        jb::tma_load_2d(stage, &map_w, bar, 0, (tile * k_tiles + kt) * BM, policy);
        jb::tma_load_2d(stage + W_BYTES, &map_x, bar, kt * BK, MATS == 2 ? 0 : place * T);
        if (++kt == k_tiles) kt = 0, ++rt;
      }
    }
  } else if (warp == 1) {
    // ---------------- products ----------------
    if (lane == 0) {
      int kt = first % k_tiles, j = 0;
      bool begins = true;
      for (int i = first, it = 0; i < last; ++i, ++it) {
        const int s = it % C::STAGES, buf = j & 1;
        if (begins && !jb::mbar_wait(acc_empty0 + 8 * buf, ((j >> 1) & 1) ^ 1, status, 42)) break;
        if (!jb::mbar_wait(full0 + 8 * s, (it / C::STAGES) & 1, status, 42)) break;
        jb::tc_fence_after();
        const uint32_t stage = base + s * C::STAGE;
        const uint64_t w_desc = jb::smem_desc_sw128(stage), x_desc = jb::smem_desc_sw128(stage + W_BYTES);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          jb::umma_bf16(tmem + buf * BN, w_desc + 2 * k, x_desc + 2 * k, jb::instr_desc_bf16(BN), begins && k == 0 ? 0u : 1u);
        jb::umma_commit(empty0 + 8 * s);
        begins = ++kt == k_tiles || i + 1 == last;               // the run leaves this row tile
        if (kt == k_tiles) kt = 0;
        if (begins) jb::umma_commit(acc_full0 + 8 * buf), ++j;
      }
    }
  } else {
    // ---------------- sums leave ----------------
    const int quarter = warp & 3;
    int j = 0;
    for (int i = first; i < last; ++j) {
      const int rt = i / k_tiles, place = rt / row_tiles, f = rt % row_tiles * BM + quarter * 32 + lane, buf = j & 1;
      i = min(last, (rt + 1) * k_tiles);
      if (!jb::mbar_wait(acc_full0 + 8 * buf, (j >> 1) & 1, status, 43)) break;
      jb::tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < BN && c < T; c += 8) {
        float r[8];
        jb::tmem_ld8(tmem + ((uint32_t)(quarter * 32) << 16) + buf * BN + c, r);
        jb::tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int t = c + q, pair = t < T ? pair_of[place * T + t] : -1;
          if (pair < 0) continue;
          if (MATS == 2) atomicAdd(Y + (size_t)pair * (2 * R) + f, r[q]);
          else atomicAdd(Y + (size_t)t * R + f, out_w != nullptr ? out_w[pair] * r[q] : r[q]);
        }
      }
      jb::tc_fence_before();
      __syncwarp();
      if (lane == 0) jb::mbar_arrive(acc_empty0 + 8 * buf);
    }
    jb::tc_fence_before();
  }
  __syncthreads();
  if (warp == 1) {
    jb::tc_fence_after();
    jb::tmem_dealloc<C::TMEM>(tmem);
  }
}

// act[place of the pair's expert * T + token][f], 4 f a thread
__global__ void __launch_bounds__(256) experts_activate_kernel(const float* __restrict__ z, const int* __restrict__ pair_slot,
                                                               const float* __restrict__ in_w, bf16* __restrict__ act, int T,
                                                               int top, int F, jb::Gate gate) {
  jb::pdl_launch_dependents();
  jb::pdl_wait();
  const int pair = blockIdx.y, f = (blockIdx.x * 256 + threadIdx.x) * 4;
  if (f >= F) return;
  const float s = in_w != nullptr ? in_w[pair] : 1.0f;
  const float4 g = *reinterpret_cast<const float4*>(z + (size_t)pair * 2 * F + f);
  const float4 u = *reinterpret_cast<const float4*>(z + (size_t)pair * 2 * F + F + f);
  const __nv_bfloat162 a = __floats2bfloat162_rn(jb::gated(s * g.x, s * u.x, gate), jb::gated(s * g.y, s * u.y, gate));
  const __nv_bfloat162 b = __floats2bfloat162_rn(jb::gated(s * g.z, s * u.z, gate), jb::gated(s * g.w, s * u.w, gate));
  const size_t row = (size_t)pair_slot[pair] * T + pair / top;
  *reinterpret_cast<uint2*>(act + row * F + f) =
      make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

template <int BN, int MATS>
int launch(const void* tiles, long long n_tiles, const void* X, long long x_rows, const int* sel_e, const float* out_w, int T,
           int top, int E, int R, int K, int up_tiles, float* Y, int* pair_slot, int places, int* status, cudaStream_t stream) {
  using C = Cfg<BN>;
  static int ready = -1, sms = 148;
  if (ready != 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    ready = (int)cudaFuncSetAttribute(experts_stream_kernel<BN, MATS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      C::smem(MAX_PLACES));
    if (ready != 0) return ready;
  }
  CUtensorMap mw, mx;
  if (!jb::make_map_64(&mw, tiles, (uint64_t)n_tiles * BM, BK, BM, false) || !jb::make_map_64(&mx, X, x_rows, K, BN, true))
    return JB_ERR_TENSORMAP;
  jb::Launch cfg(dim3(sms), dim3(THREADS), C::smem(places), stream);
  return (int)cudaLaunchKernelEx(&cfg.c, experts_stream_kernel<BN, MATS>, mw, mx, sel_e, out_w, T, top, E, R, K / BK, up_tiles, Y,
                                 pair_slot, status);
}

}  // namespace

// x: bfloat16 [T, W]; sel_e, sel_w [T, top]; gu: packed gate tiles of all experts' F rows, then from row tile `up_tiles` on the up
// tiles (gu_tiles tiles in all); dn: packed tiles of all experts' W rows; z: float32 [T top, 2 F], zero; act: bfloat16 scratch
// [min(E, T top) T, F]; pair_slot: int scratch [T top]; out: float32 [T, W], added to.  T <= 64, W and F multiples of 128.
// `status`: a device int that a wait that ran out sets to 41 (loads), 42 (products) or 43 (sums).
JB_EXPORT int jb_experts_stream(const void* x, const int* sel_e, const float* sel_w, int top, const void* gu, long long gu_tiles,
                                int up_tiles, const void* dn, long long dn_tiles, float* z, void* act, int* pair_slot, float* out,
                                int T, int W, int F, int E, float gate_limit, float gate_alpha, int weight_on_output, int* status,
                                cudaStream_t stream) {
  if (T <= 0) return 0;
  const int pairs = T * top, slots = pairs < E ? pairs : E;
  JB_REFUSE(T > 64 || top < 1 || E < 1 || E > MAX_EXPERTS || slots * T > MAX_PLACES, "experts_stream: %d tokens, %d of %d experts",
            T, top, E);
  JB_REFUSE(W % BM || F % BM || (((uintptr_t)x | (uintptr_t)gu | (uintptr_t)dn | (uintptr_t)z | (uintptr_t)act) & 15),
            "experts_stream: experts of %d x %d, or operands off a 16-byte boundary", F, W);
  JB_REFUSE(up_tiles < (long long)E * (F / BM) || gu_tiles < ((long long)up_tiles + (long long)E * (F / BM)) * (W / BK) ||
                dn_tiles < (long long)E * (W / BM) * (F / BK) || gu_tiles * BM > 0x7fffffffLL || dn_tiles * BM > 0x7fffffffLL ||
                (long long)slots * 2 * (F / BM) * (W / BK) > 0x7fffffffLL || (long long)slots * T > 0x7fffffffLL / F,
            "experts_stream: the packed weights hold %lld and %lld tiles", gu_tiles, dn_tiles);
  const float *in_w = weight_on_output ? nullptr : sel_w, *out_w = weight_on_output ? sel_w : nullptr;
  int e;
#define JB_GO(MATS, ...) \
  e = T <= 16 ? launch<16, MATS>(__VA_ARGS__) : T <= 32 ? launch<32, MATS>(__VA_ARGS__) : launch<64, MATS>(__VA_ARGS__)
  JB_GO(2, gu, gu_tiles, x, T, sel_e, nullptr, T, top, E, F, W, up_tiles, z, pair_slot, slots * T, status, stream);
  if (e != 0) return e;
  jb::Launch cfg(dim3((F + 1023) / 1024, pairs), dim3(256), 0, stream);
  e = (int)cudaLaunchKernelEx(&cfg.c, experts_activate_kernel, (const float*)z, (const int*)pair_slot, in_w, (bf16*)act, T, top, F,
                              jb::Gate{gate_limit, gate_alpha});
  if (e != 0) return e;
  JB_GO(1, dn, dn_tiles, act, (long long)slots * T, sel_e, out_w, T, top, E, W, F, 0, out, (int*)nullptr, slots * T, status, stream);
#undef JB_GO
  return e;
}
