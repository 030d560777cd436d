// The certified router's logits on the tensor cores (large batches), written for sm_100a.
//
// The certified pass (csk_kernels.cuh, above k_router_fast) needs, per (token, expert), a value close to the exact
// logit, the sum of the magnitudes of its prefixes, and a bound on its own error.  The FMA kernel is held by shared-
// memory operand delivery; here the products are INTEGER products on tcgen05.mma kind::f16, and the bound assumes of the
// tensor cores only that sums of integers are exact in their fp32 accumulators while every partial sum is below 2^24:
//   * per (row, block of 64 columns) x = 2^(e-8) (s0 + s1 2^-9 + s2 2^-18 + rest), 2^e the smallest power of two that
//     the block's largest magnitude m does not exceed, s0, s1, s2 integers of magnitude <= 256 (fp16 holds them
//     exactly), |rest| <= 2^-19: at most 2^-26 m is left out;
//   * three accumulators: s0 s0', s0 s1' + s1 s0', s0 s2' + s1 s1' + s2 s0'.  Each is a sum of at most 3 x 64 integer
//     products of magnitude <= 2^16, so below 2^24: exact in fp32 in any order.  The products left out (s1 s2', s2 s1'
//     and s2 s2') add up to at most 2^-18 m m' per block;
//   * per block the accumulators are added with weights 1, 2^-9, 2^-18, scaled (powers of two) and added to the running
//     prefix R in fp32.
// Distance from the exact logit S (u = 2^-24, h and w the token and gate rows, |.| their 2-norms, j a block): the rests
// cost 2^-26 (m |w_j|_1 + m' |h_j|_1) <= 4 u |h_j| |w_j| (|.|_1 <= 8 |.| over 64 columns), the products left out 64 u m m',
// the roundings u (|R_j| + 1.1 |h_j| |w_j|).  With 64-column blocks the chain's own distance from S is
// u (64 sum_j |R_j| + 65 |h| |w|).  Together, by Cauchy-Schwarz, u (65 sum_j |R_j| + 71 n n') with n^2 = |h|^2 + sum_j m^2
// and n' likewise: these norms and constants are what k_router_finish_many is given.
//
//   * work unit of a CTA: 64 tokens x 128 experts x one of `parts` runs of blocks.  MMAs are transposed (D[expert,
//     token]), M = 128; the token operand is the three digit matrices stacked, so s0' of the experts meets all of
//     them in one MMA of N = 192, s1' the first two (N = 128), s2' the first (N = 64): 208 tensor cycles per 16 columns;
//   * the gate rows' digits are laid out once, when the weights are set: 48 KB per block of columns, one bulk copy;
//   * eight warps turn token rows into digits (four threads a row, the next two blocks' loads in flight meanwhile) and
//     store them in the operand's swizzled layout; sixteen more keep R and sum |R| of 16 tokens x one expert per thread.
// 8192 tokens, 128 experts, 2880 columns: 66 us, then 30 us of selection and 38 us for the 2 % of the tokens that take the
// chain (the chain for all of them: 343 us).  Bound by instruction issue in conversion and read-out.
//
// Three stages of 72 KB and two sets of accumulators keep MMAs, conversion and read-out of neighbouring blocks apart.
//
// Waits are bounded as everywhere (csk_common.cuh); one that runs out sets kDevErrWaitTimeout in *status.
#pragma once

#include "csk_common.cuh"
#include "csk_tc.cuh"

namespace csk {

constexpr int kRtTokens = 64;
constexpr int kRtExperts = 128;
constexpr int kRtBlock = 64;                                  // columns of the hidden dimension per step
constexpr int kRtWBytes = 3 * kRtExperts * kRtBlock * 2;      // 48 KB: digits of 128 gate rows
constexpr int kRtXBytes = 3 * kRtTokens * kRtBlock * 2;       // 24 KB: digits of 64 token rows
constexpr int kRtStageBytes = kRtWBytes + kRtXBytes;
constexpr int kRtStages = 3;
constexpr int kRtScaleRing = 8;                               // blocks whose token scales are kept
constexpr int kRtReadWarps = 16;
constexpr int kRtThreads = (2 + 8 + kRtReadWarps) * 32;
constexpr int kRtSmem = kRtStages * kRtStageBytes + kRtScaleRing * kRtTokens * 4 + 512 + 1024;
constexpr float kRtPrefixCoef = 65.f, kRtNormCoef = 71.f;     // the bound's two constants (above)

inline int rt_blocks(int H) { return (H + kRtBlock - 1) / kRtBlock; }
inline int rt_groups(int E) { return (E + kRtExperts - 1) / kRtExperts; }
inline size_t rt_weight_bytes(int E, int H) { return (size_t)rt_groups(E) * rt_blocks(H) * kRtWBytes; }
inline size_t rt_scale_floats(int E, int H) { return (size_t)rt_groups(E) * rt_blocks(H) * kRtExperts; }

// 16-byte piece `piece` of row `r` in a K-major operand of 128-byte rows under the 128-byte swizzle
__host__ __device__ inline uint32_t rt_swizzled(int r, int piece) { return (uint32_t)r * 128u + (uint32_t)((piece ^ (r & 7)) << 4); }

// The scale of a block whose largest magnitude has the bits `amax`, and the factor that takes values to digit units.
// Blocks below 2^-107 are taken in units of that (what they lose is below the bound's absolute term); an infinity or
// NaN gives a NaN scale and no digits: nothing of that row is certified.
__device__ __forceinline__ float rt_scale_of(uint32_t amax, float& inv) {
  if (amax >= 0x7F800000u) {
    inv = 0.f;
    return __uint_as_float(0x7FC00000u);
  }
  const uint32_t e = max((amax + 0x7FFFFFu) >> 23, 20u);
  inv = __uint_as_float((262u - e) << 23);
  return __uint_as_float((e - 8u) << 23);
}
// Nearest integer of |y| <= 2^22 by two additions (the conversion instruction runs at an eighth of their rate).
__device__ __forceinline__ float rt_round(float y) { return __fsub_rn(__fadd_rn(y, 12582912.f), 12582912.f); }
__device__ __forceinline__ void rt_digits(float x, float inv, float (&d)[3]) {
  float y = inv == 0.f ? 0.f : x * inv;
  d[0] = rt_round(y);
  y = (y - d[0]) * 512.f;
  d[1] = rt_round(y);
  d[2] = rt_round((y - d[1]) * 512.f);
}
__device__ __forceinline__ uint32_t rt_pack(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Norms of the gate rows with their blocks' largest magnitudes (n' above), rounded up.  One warp per row.
__global__ void k_rt_wnorm(const float* __restrict__ wg, float* __restrict__ wnorm, int E, int H) {
  const int e = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (e >= E) return;
  float acc = 0.f;
  for (int b = 0; b < H; b += kRtBlock) {
    const float x = wg[(size_t)e * H + b + lane], y = b + 32 < H ? wg[(size_t)e * H + b + 32 + lane] : 0.f;
    acc = fmaf(x, x, fmaf(y, y, acc));
    const float m = __uint_as_float(__reduce_max_sync(0xffffffffu, max(__float_as_uint(x) & 0x7FFFFFFFu, __float_as_uint(y) & 0x7FFFFFFFu)));
    if (lane == 0) acc = fmaf(m, m, acc);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) wnorm[e] = sqrtf(acc) * 1.001f + kNormFloor;
}

// Gate rows as digits: one thread per (group, block, expert).
__global__ void k_rt_pack(const float* __restrict__ wg, uint8_t* __restrict__ dst, float* __restrict__ scales, int E, int H) {
  const int nb = (H + kRtBlock - 1) / kRtBlock;
  const int n = ((E + kRtExperts - 1) / kRtExperts) * nb * kRtExperts;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int r = i % kRtExperts, b = (i / kRtExperts) % nb, e = (i / (kRtExperts * nb)) * kRtExperts + r;
    const int cols = e < E ? min(kRtBlock, H - b * kRtBlock) : 0;
    const float* src = wg + (size_t)e * H + b * kRtBlock;
    uint32_t amax = 0;
    for (int c = 0; c < cols; ++c) amax = max(amax, __float_as_uint(src[c]) & 0x7FFFFFFFu);
    float inv;
    scales[i] = rt_scale_of(amax, inv);
    uint8_t* out = dst + (size_t)(i / kRtExperts) * kRtWBytes;
    for (int c = 0; c < kRtBlock; c += 2) {
      float d0[3], d1[3];
      rt_digits(c < cols ? src[c] : 0.f, inv, d0);
      rt_digits(c + 1 < cols ? src[c + 1] : 0.f, inv, d1);
      for (int p = 0; p < 3; ++p)
        *reinterpret_cast<uint32_t*>(out + (size_t)p * kRtExperts * 128 + rt_swizzled(r, c >> 3) + (c & 7) * 2) = rt_pack(d0[p], d1[p]);
    }
  }
}

struct RouterTcArgs {
  const float* hidden;    // [T,H], 16-byte aligned
  const uint8_t* w;       // k_rt_pack's digits
  const float* w_scale;
  float2* part;           // [T][parts][E]: (sum, sum of prefix magnitudes) of the part
  float* hn2;             // [T][parts]: the part's share of n^2
  int* status;
  int T, H, E;
  int stall;              // test hook: the copy role issues nothing, every wait of the other roles runs out
};

__global__ void __launch_bounds__(kRtThreads, 1) k_router_tc(const RouterTcArgs A) {
  extern __shared__ __align__(1024) uint8_t rt_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)rt_smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t smem_base = smem_u32(smem);
  float* s_scale = reinterpret_cast<float*>(smem + kRtStages * kRtStageBytes);
  uint8_t* ctrl = smem + kRtStages * kRtStageBytes + kRtScaleRing * kRtTokens * 4;
  const uint32_t bar_base = smem_u32(ctrl);
  auto bar_w = [&](int s) { return bar_base + 8u * s; };              // gate rows' digits landed
  auto bar_x = [&](int s) { return bar_base + 8u * (4 + s); };        // token rows' digits written
  auto bar_empty = [&](int s) { return bar_base + 8u * (8 + s); };    // the stage's MMAs retired
  auto bar_acc_full = [&](int b) { return bar_base + 8u * (12 + b); };
  auto bar_acc_empty = [&](int b) { return bar_base + 8u * (14 + b); };
  const uint32_t bar_drain = bar_base + 8u * 16;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(ctrl + 8 * 20);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(ctrl + 8 * 20 + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kRtStages; ++s) {
      mbar_init(bar_w(s), 1);
      mbar_init(bar_x(s), 8);
      mbar_init(bar_empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_acc_full(b), 1);
      mbar_init(bar_acc_empty(b), kRtReadWarps);
    }
    mbar_init(bar_drain, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int t0 = blockIdx.x * kRtTokens, group = blockIdx.y, parts = gridDim.z, part = blockIdx.z;
  const int nb = (A.H + kRtBlock - 1) / kRtBlock;
  const int b_begin = nb * part / parts, n = nb * (part + 1) / parts - b_begin;
  const size_t first = (size_t)group * nb + b_begin;  // this part's first block among the gate rows' digits

  if (warp == 0) {
    // ------------------------------ producer ------------------------------
    if (lane == 0) {
      int issued = 0;
      for (int i = 0; i < (A.stall ? 0 : n); ++i) {
        const int s = i % kRtStages;
        if (i >= kRtStages && !mbar_wait(bar_empty(s), (uint32_t)((i / kRtStages - 1) & 1), abort_flag)) break;
        mbar_expect_tx(bar_w(s), kRtWBytes);
        bulk_load(smem_base + (uint32_t)s * kRtStageBytes, A.w + (first + i) * kRtWBytes, kRtWBytes, bar_w(s));
        ++issued;
      }
      // copies whose MMAs never came (a wait ran out) still have to land before the CTA goes away
      for (int i = issued > kRtStages ? issued - kRtStages : 0; i < issued; ++i) {
        const long long c0 = clock64();
        while (!mbar_try(bar_w(i % kRtStages), (uint32_t)((i / kRtStages) & 1)) && clock64() - c0 < drain_budget()) {
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (warp-wide loop, one elected lane issues) ------------------------------
    const uint32_t tb = __shfl_sync(0xffffffffu, tmem_base, 0);
    bool ok = true;
    for (int i = 0; i < n; ++i) {
      const int s = i % kRtStages, buf = i & 1;
      ok = mbar_wait_warp(bar_acc_empty(buf), (uint32_t)((i >> 1) & 1) ^ 1u, abort_flag) &&
           mbar_wait_warp(bar_w(s), (uint32_t)((i / kRtStages) & 1), abort_flag) &&
           mbar_wait_warp(bar_x(s), (uint32_t)((i / kRtStages) & 1), abort_flag);
      if (!ok) break;
      tc_fence_after();
      const uint32_t st = smem_base + (uint32_t)s * kRtStageBytes;
      const uint64_t dw = umma_desc_sw128(st), dx = umma_desc_sw128(st + kRtWBytes);
      const uint32_t d = tb + (uint32_t)buf * 192u;
      if (elect_one()) {
#pragma unroll
        for (int k4 = 0; k4 < kRtBlock / 16; ++k4) {
#pragma unroll
          for (int p = 0; p < 3; ++p)
            umma_f16_ss(d + (uint32_t)p * kRtTokens, dw + (uint64_t)(p * (kRtExperts * 128 / 16) + k4 * 2), dx + (uint64_t)(k4 * 2),
                        umma_idesc_f16((3 - p) * kRtTokens), (k4 | p) ? 1u : 0u);
        }
        umma_commit(bar_empty(s));
        umma_commit(bar_acc_full(buf));
      }
      __syncwarp();
    }
    if (lane == 0) {
      umma_commit(bar_drain);
      const long long c0 = clock64();
      while (!mbar_try(bar_drain, 0) && clock64() - c0 < drain_budget()) {
      }
    }
    __syncwarp();
  } else if (warp < 10) {
    // ------------------------------ token rows to digits: four threads a row, every fourth 16-byte piece each ------------------------------
    const int x = threadIdx.x - 64, r = x >> 2, q = x & 3, t = t0 + r;
    griddep_wait();
    griddep_launch();
    const float* src = A.hidden + (size_t)min(t, A.T - 1) * A.H;
    float4 next[2][4];
    auto load = [&](int i, float4 (&to)[4]) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int col = (b_begin + i) * kRtBlock + (q + 4 * j) * 4;  // H is a multiple of 32: a piece is inside or outside
        to[j] = col < A.H ? __ldg(reinterpret_cast<const float4*>(src + col)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    float h2 = 0.f;
    auto step = [&](int i, float4 (&at_hand)[4]) {
      const int s = i % kRtStages;
      float v[16];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[4 * j] = at_hand[j].x;
        v[4 * j + 1] = at_hand[j].y;
        v[4 * j + 2] = at_hand[j].z;
        v[4 * j + 3] = at_hand[j].w;
      }
      if (i + 2 < n) load(i + 2, at_hand);
      uint32_t amax = 0;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        amax = max(amax, __float_as_uint(v[j]) & 0x7FFFFFFFu);
        h2 = fmaf(v[j], v[j], h2);
      }
      amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
      amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
      if (q == 0) h2 = fmaf(__uint_as_float(amax), __uint_as_float(amax), h2);
      float inv;
      const float scale = rt_scale_of(amax, inv);
      // (a wait that ran out must not part the lanes in front of the shuffles: they go on, every further wait ends at once
      // and nobody uses the digits)
      if (i >= kRtStages) mbar_wait(bar_empty(s), (uint32_t)((i / kRtStages - 1) & 1), abort_flag);
      uint8_t* out = smem + (size_t)s * kRtStageBytes + kRtWBytes;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float d[4][3];
#pragma unroll
        for (int c = 0; c < 4; ++c) rt_digits(v[4 * j + c], inv, d[c]);
        const uint32_t at = rt_swizzled(r, (q + 4 * j) >> 1) + (uint32_t)(q & 1) * 8u;
#pragma unroll
        for (int p = 0; p < 3; ++p)
          *reinterpret_cast<uint2*>(out + p * (kRtTokens * 128) + at) = make_uint2(rt_pack(d[0][p], d[1][p]), rt_pack(d[2][p], d[3][p]));
      }
      // the read-out of block i - 8 is over: block i - 3's MMAs were issued, so block i - 5 had been read out
      if (q == 0) s_scale[(i % kRtScaleRing) * kRtTokens + r] = scale;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_x(s));
    };
    if (n > 0) load(0, next[0]);
    if (n > 1) load(1, next[1]);
    for (int i = 0; i < n; i += 2) {
      step(i, next[0]);
      if (i + 1 < n) step(i + 1, next[1]);
    }
    __syncwarp();
    h2 += __shfl_xor_sync(0xffffffffu, h2, 1);
    h2 += __shfl_xor_sync(0xffffffffu, h2, 2);
    if (group == 0 && q == 0 && t < A.T) A.hn2[(size_t)t * parts + part] = h2;
  } else {
    // ------------------------------ read-out: lane = expert, 16 tokens a thread ------------------------------
    const int quarter = warp & 3, tok = (warp - 10) / 4 * 16;  // its tensor-memory lanes, its first token
    const int e = group * kRtExperts + quarter * 32 + lane;
    griddep_wait();  // the parts of an earlier call are read until then
    float R[16], aR[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) R[j] = aR[j] = 0.f;
    const float* ws = A.w_scale + first * kRtExperts + quarter * 32 + lane;
    bool ok = true;
    for (int i = 0; i < n; ++i) {
      const int buf = i & 1;
      const float sw = __ldg(ws + (size_t)i * kRtExperts);
      ok = mbar_wait_warp(bar_acc_full(buf), (uint32_t)((i >> 1) & 1), abort_flag);
      if (!ok) break;
      tc_fence_after();
      const uint32_t acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)buf * 192u + (uint32_t)tok;
      const float* sh = s_scale + (i % kRtScaleRing) * kRtTokens + tok;
#pragma unroll
      for (int c = 0; c < 16; c += 8) {
        uint32_t a0[8], a1[8], a2[8];
        tmem_ld8(acc + c, a0);
        tmem_ld8(acc + kRtTokens + c, a1);
        tmem_ld8(acc + 2 * kRtTokens + c, a2);
        float hs[8];
        *reinterpret_cast<float4*>(&hs[0]) = *reinterpret_cast<const float4*>(sh + c);
        *reinterpret_cast<float4*>(&hs[4]) = *reinterpret_cast<const float4*>(sh + c + 4);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float v = fmaf(__uint_as_float(a2[j]), 0x1p-9f, __uint_as_float(a1[j]));
          v = fmaf(v, 0x1p-9f, __uint_as_float(a0[j]));
          R[c + j] = fmaf(v * sw, hs[j], R[c + j]);
          aR[c + j] += fabsf(R[c + j]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_acc_empty(buf));
    }
    if (ok && e < A.E) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int t = t0 + tok + j;
        if (t < A.T) A.part[((size_t)t * parts + part) * A.E + e] = make_float2(R[j], aR[j]);
      }
    }
  }
  // ------------------------------ teardown ------------------------------
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag && A.status) atomicOr(A.status, kDevErrWaitTimeout);
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

inline cudaError_t rt_prepare_device() {
  return cudaFuncSetAttribute(k_router_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kRtSmem);
}

}  // namespace csk
