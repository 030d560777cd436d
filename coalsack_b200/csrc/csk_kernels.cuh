// The small kernels around the expert contractions: router, permutation by
// expert, gather to fp16 rows, weighted combine.
#pragma once

#include <algorithm>

#include "csk_common.cuh"

namespace csk {

// ---------------------------------------------------------------------------
// Router (moe_router_node::compute_impl, moe_router_node.h:140-214).
//
// The selected expert indices must equal the reference's bit for bit, and the
// reference accumulates each logit sequentially in fp32 with separate multiply
// and add.  So each (token, expert) logit is ONE thread's in-order chain of
// __fmul_rn / __fadd_rn over the hidden dimension (never contracted into an
// FMA, never reassociated).  Parallelism comes from the T*E independent chains.
// k_router_topk then selects per token: one warp, k rounds of arg-max by
// shuffles (ties -> lower expert id; the reference leaves ties unspecified),
// softmax over the selected logits (or sigmoid) exactly as the reference.
// ---------------------------------------------------------------------------
constexpr int kRouterPad = 4;       // row stride 4 mod 32 words: a quarter-warp's 128-bit loads hit distinct banks
// Columns of a stage: few / many tokens, and the ring's stages.  A stage costs a lone chain some 250 cycles: 192 columns and four stages 12.0 us
// (8 tokens, 32 experts, 2880 columns, back to back), 288 or 384 and three 11.2, 96 and six 13.9; of 256 two blocks fit an SM.
constexpr int kRouterChunkFew = 256, kRouterChunkMany = 128;
__host__ __device__ constexpr int router_stages(int ch) { return ch > 128 ? 3 : 4; }
constexpr int kMaxTopK = 16;
constexpr int kMaxExperts = 1024;
constexpr int kRouterClusterGroups = 8;  // groups of 32 experts up to which their blocks form a cluster (the portable size)

// ch = columns of the hidden dimension per pipeline stage; experts: of the logits that the blocks of a cluster exchange (twice), 0 without one
inline size_t router_smem_bytes(int tokens_per_block, int ch, int experts) {
  return ((size_t)router_stages(ch) * (32 + tokens_per_block) * (ch + kRouterPad) + 2 * (size_t)tokens_per_block * experts) * sizeof(float) + 128;
}

__device__ __forceinline__ void cp_async16(uint32_t smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_dst), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Router weights repacked for the logits kernel: [group of 32 experts][chunk of
// CH columns][32 rows][CH + pad] floats, so that a stage of the kernel's ring
// is ONE contiguous span (one bulk copy).  Rows past E and columns past H are 0.
inline size_t router_packed_floats(int E, int H, int ch) {
  return (size_t)((E + 31) / 32) * ((H + ch - 1) / ch) * 32 * (ch + kRouterPad);
}
__global__ void k_pack_router(const float* __restrict__ wg, float* __restrict__ packed, int E, int H, int ch) {
  const int ld = ch + kRouterPad, n_chunks = (H + ch - 1) / ch;
  const size_t n = (size_t)((E + 31) / 32) * n_chunks * 32 * ld;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % ld);
    const int r = (int)((i / ld) % 32);
    const int ci = (int)((i / ((size_t)ld * 32)) % n_chunks);
    const int g = (int)(i / ((size_t)ld * 32 * n_chunks));
    const int e = g * 32 + r, d = ci * ch + c;
    packed[i] = (c < ch && e < E && d < H) ? wg[(size_t)e * H + d] : 0.f;
  }
}

// Top-k of one token's logits by one warp, then softmax over the selected
// logits (or sigmoid) exactly as the reference (moe_router_node.h:165-214).
// The logits sit in registers (lane l holds experts l, l+32, ...); each of the
// k rounds is an arg-max over the warp (ties -> lower expert id; the reference
// leaves ties unspecified).  Lane j keeps the j-th selection: with all of them in one lane's arrays (local memory), ten
// shuffles a round and the softmax in one lane a token took 3 us more.
//
// With `bounds` (the logits then come from a fast kernel, see k_router_fast) the
// selection is CERTIFIED only if every gap between neighbours of the k best logits
// exceeds the sum of their error bounds, and the last of them less its bound exceeds
// every other logit plus ITS bound (not only the runner-up's: a gate row of large
// norm may have a larger bound than any).  The reference's own logits, which lie
// within those bounds, then order the same experts the same way.  Returns false (warp-uniform) when a gap is too
// small; the caller then sends the token through the order-faithful chain.
// CG: logits and bounds are global memory written by other blocks (read through L2); else
// they are the block's own shared memory.
// NV: logits per lane (E <= 32 * NV); the selection loops are unrolled over it.
template <bool CG, int NV>
__device__ __forceinline__ bool warp_topk_regs(float (&v)[NV], int E, int k, int sigmoid, float* __restrict__ out /* [k][2] */,
                                               const float* __restrict__ bounds) {
  const int lane = threadIdx.x & 31;
  float my_v = -INFINITY;
  int my_i = 0x7fffffff;
  uint32_t gone = 0;
  // With many logits a lane, its best is looked for again only when it was selected (1024 experts of 512 columns, 100 tokens 44.3 -> 37.1 us, 511
  // 78.0 -> 69.9; with eight a lane the branch costs as much).
  constexpr bool kKeepBest = NV > 16;
  float lane_v = -INFINITY;
  int lane_i = 0x7fffffff;
  bool look = true;
#pragma unroll 1
  for (int j = 0; j < k; ++j) {
    if (!kKeepBest || look) {
      lane_v = -INFINITY;
      lane_i = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        if (i * 32 < E) {  // warp-uniform
          const float x = v[i];
          if (x > lane_v && !(kKeepBest && (gone >> i & 1u))) {  // ascending expert id within the lane: '>' keeps the lowest on ties
            lane_v = x;
            lane_i = i * 32 + lane;
          }
        }
      }
    }
    // the lanes' bests as integers of the same order (both zeros alike), the lowest id of those that reach the maximum
    const uint32_t bits = __float_as_uint(lane_v + 0.f), key = bits ^ ((int)bits < 0 ? 0xffffffffu : 0x80000000u);
    const uint32_t top = __reduce_max_sync(0xffffffffu, key);
    const int bi = (int)__reduce_min_sync(0xffffffffu, key == top ? (uint32_t)lane_i : 0x7fffffffu);
    const float bv = __shfl_sync(0xffffffffu, lane_v, bi & 31);  // (nothing to choose from: -inf in every lane)
    if (lane == j) {
      my_v = bv;
      my_i = bi;
    }
    // the winner leaves the pool
    look = bi == lane_i && bi != 0x7fffffff;
    if (kKeepBest) {
      if (look) gone |= 1u << (bi >> 5);
      continue;
    }
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (i * 32 < E && bi == i * 32 + lane) {
        v[i] = __int_as_float(0xffc00000);  // NaN never wins a '>' test again
        gone |= 1u << i;
      }
  }
  bool certified = true;
  if (bounds) {
    float above = -INFINITY;  // what no logit left out exceeds
#pragma unroll
    for (int i = 0; i < NV; ++i)
      if (i * 32 < E && i * 32 + lane < E && !(gone >> i & 1u)) {
        const float x = v[i] + (CG ? __ldcg(bounds + i * 32 + lane) : bounds[i * 32 + lane]);
        above = x < INFINITY ? fmaxf(above, x) : INFINITY;  // (a NaN too)
      }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) above = fmaxf(above, __shfl_xor_sync(0xffffffffu, above, o));
    const float b = lane < k && my_i >= 0 && my_i < E ? (CG ? __ldcg(bounds + my_i) : bounds[my_i]) : INFINITY;
    const float next_v = __shfl_down_sync(0xffffffffu, my_v, 1), next_b = __shfl_down_sync(0xffffffffu, b, 1);
    const bool apart = lane + 1 < k ? my_v - next_v > b + next_b : my_v - b > above;  // false for NaN
    certified = __all_sync(0xffffffffu, lane >= k || apart);
  }
  float w;
  if (sigmoid) {
    w = 1.0f / (1.0f + expf(-my_v));
  } else {
    // one lane per selection; the sum in order
    float mx = __shfl_sync(0xffffffffu, my_v, 0);
    for (int j = 1; j < k; ++j) mx = fmaxf(mx, __shfl_sync(0xffffffffu, my_v, j));
    w = expf(my_v - mx);
    float se = 0.f;
    for (int j = 0; j < k; ++j) se += __shfl_sync(0xffffffffu, w, j);
    w *= se > 0.f ? 1.0f / se : 0.f;
  }
  if (lane < k) {
    out[2 * lane] = (float)my_i;
    out[2 * lane + 1] = w;
  }
  return certified;
}

template <bool CG, int NV>
__device__ __forceinline__ bool warp_topk_nv(const float* __restrict__ l, int E, int k, int sigmoid,
                                             float* __restrict__ out /* [k][2] */,
                                             const float* __restrict__ bounds) {
  const int lane = threadIdx.x & 31;
  float v[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i)
    v[i] = (i * 32 < E && i * 32 + lane < E) ? (CG ? __ldcg(l + i * 32 + lane) : l[i * 32 + lane]) : -INFINITY;
  return warp_topk_regs<CG, NV>(v, E, k, sigmoid, out, bounds);
}

// MAX_E: of the experts there may be.  Code that is never run makes kernels of a few microseconds longer: with the forms of 512 and 1024 experts the
// router of one token of 64 experts took 16.5 us, not 15.6 (cold code).
template <bool CG = true, int MAX_E = kMaxExperts, bool FORM_512 = true>
__device__ __forceinline__ bool warp_topk(const float* __restrict__ l, int E, int k, int sigmoid,
                                          float* __restrict__ out /* [k][2] */,
                                          const float* __restrict__ bounds = nullptr) {
  if (E <= 32) return warp_topk_nv<CG, 1>(l, E, k, sigmoid, out, bounds);
  if (E <= 64) return warp_topk_nv<CG, 2>(l, E, k, sigmoid, out, bounds);
  if (E <= 128) return warp_topk_nv<CG, 4>(l, E, k, sigmoid, out, bounds);
  if (MAX_E <= 256 || E <= 256) return warp_topk_nv<CG, 8>(l, E, k, sigmoid, out, bounds);
  if (FORM_512 && E <= 512) return warp_topk_nv<CG, 16>(l, E, k, sigmoid, out, bounds);
  return warp_topk_nv<CG, kMaxExperts / 32>(l, E, k, sigmoid, out, bounds);
}

struct RouterArgs {
  const float* hidden;   // [T,H], 16-byte aligned
  const float* wg;       // PACKED: router_packed layout for this CH; else [E,H], 16-byte aligned
  const float* bias;     // [E] or null
  float* logits;         // [T,E] scratch
  float* router_out;     // [T,k,2]; written when `counters` is given
  int* counters;         // one per token block, all zero between launches; null = logits only
  int* status;           // device status word or null
  int T, H, E, k, sigmoid;
  int cluster;           // the blocks of a token block's groups of experts form a cluster
  // order-faithful kernel over a token list (the fall-back pass): token_list[0 .. *n_list)
  const int* token_list;
  int* n_list;           // read at start; reset to zero, with fb_done, by the last block to finish
  int* fb_done;          // ticket of that reset
  unsigned long long* fb_total;  // running number of tokens that took the fall-back pass (statistics)
  int list_over, list_max;       // the launch takes a list of list_over < entries <= list_max, and leaves any other alone
};

// A block is one producer warp (four with plain weights) plus TW consumer warps.  A
// consumer warp owns TT tokens, its lanes 32 neighbouring experts: a thread runs TT chains.
//   * a ring of three or four stages of CH columns, filled by the producer alone: the expert rows by
//     bulk copies (cp.async.bulk; an SM starts only about one per 70-100 cycles, so with PACKED
//     weights a stage is one copy issued by one thread, with plain [E,H] weights a copy per
//     row), the token rows by cp.async; both count on the stage's mbarrier, the only thing a
//     consumer waits for.  Packed weights of the first stages are requested before the kernel
//     in front has ended;
//   * a lane reads its own expert row with 128-bit loads (conflict-free by the row padding)
//     and the token rows by broadcast, a batch of columns ahead; the products of the next four
//     columns are written between the additions of these, two to an instruction
//     (mul.rn.f32x2: the same rounding, half the issue slots);
//   * a chain costs one dependent addition per column, 4.3 cycles: TT = 1 runs one chain at
//     that speed (few tokens), larger TT has the additions of TT chains fill those cycles, up to
//     the 2 cycles a column and chain that product and sum take of the fp32 pipe;
//   * the logits of a token's other groups of 32 experts come from the blocks of the same
//     cluster (A.cluster: gridDim.y of them, through distributed shared memory; the tokens'
//     selections are dealt to its blocks), or, with more than eight groups, through global
//     memory: the last block to finish a token block's logits (an atomic ticket after a fence)
//     selects then.  With one group they are in the lanes already.  Without `counters` the
//     logits are all there is.
// Waits are bounded; a wait that runs out sets kDevErrWaitTimeout in *status (when given): every
// further wait of the block ends at once, and it goes through the rest of its loops with
// whatever it holds, so that the blocks of a cluster still meet.
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {  // arrives once this thread's cp.asyncs so far have landed
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ float4 lds128(uint32_t addr) {  // (volatile: it stays where the code asks for it, ahead of its use)
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
// Four products with the rounding of single multiplications; PACKED2: two to an instruction (half the issue slots, which a lone
// chain has to spare, while the pair's later result is in its way: 5.3 cycles a column, not 4.6).
template <bool PACKED2>
__device__ __forceinline__ float4 mul4_rn(const float4& a, const float4& b) {
  if (!PACKED2) return make_float4(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y), __fmul_rn(a.z, b.z), __fmul_rn(a.w, b.w));
  float4 r;
  asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%4, %5};\n\tmov.b64 q, {%8, %9};\n\tmul.rn.f32x2 p, p, q;\n\tmov.b64 {%0, %1}, p;\n\t"
      "mov.b64 p, {%6, %7};\n\tmov.b64 q, {%10, %11};\n\tmul.rn.f32x2 p, p, q;\n\tmov.b64 {%2, %3}, p;\n\t}"
      : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
      : "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w));
  return r;
}

// A batch of 4 G columns in registers: the lane's expert row and the warp's token rows.
// (two warps a scheduler hide the loads by themselves: 850 tokens of 128 experts 46.2 us with batches of eight columns, 47.5 with sixteen)
__host__ __device__ constexpr int router_groups(int tw, int tt) { return tw > 4 ? 2 : tt == 1 ? 8 : 4; }
template <int TT, int G>
struct ChainBatch {
  float4 w[G], h[G][TT];
  // w, h: where the rows' columns are in shared memory, the token rows ld_bytes apart
  __device__ __forceinline__ void load(int g, uint32_t wp, uint32_t hp, int ld_bytes) {
    w[g] = lds128(wp + 16 * g);
#pragma unroll
    for (int i = 0; i < TT; ++i) h[g][i] = lds128(hp + i * ld_bytes + 16 * g);
  }
  __device__ __forceinline__ void products(int g, float4 (&p)[TT]) const {
#pragma unroll
    for (int i = 0; i < TT; ++i) p[i] = mul4_rn<(TT > 1)>(h[g][i], w[g]);
  }
};
// Adds the batch's columns to the chains and loads the next batch, a group between each two groups' additions.  `now`: the products of
// the batch's first group; on return those of the next one's.
// Batches alternate between two sets of registers, across the chunks' borders too, so that a load is waited for a whole batch
// after it was asked for.  (With one ring of registers, refilled a group at a time, the additions of three chains waited for the
// latest loads: 2750 clocks per 128 columns, 333 tokens of 128 experts; now 1480.  One chain: 1445 per 256 columns, now 1355.)
template <int TT, int G>
__device__ __forceinline__ void chain_batch(const ChainBatch<TT, G>& b, ChainBatch<TT, G>& next_batch, uint32_t wp, uint32_t hp, int ld_bytes,
                                            float4 (&now)[TT], float (&acc)[TT]) {
#pragma unroll
  for (int g = 0; g < G; ++g) {
    next_batch.load(g, wp, hp, ld_bytes);
    float4 next[TT];
    if (g + 1 < G) b.products(g + 1, next);
    else next_batch.products(0, next);
#pragma unroll
    for (int i = 0; i < TT; ++i) acc[i] = __fadd_rn(acc[i], now[i].x);
#pragma unroll
    for (int i = 0; i < TT; ++i) acc[i] = __fadd_rn(acc[i], now[i].y);
#pragma unroll
    for (int i = 0; i < TT; ++i) acc[i] = __fadd_rn(acc[i], now[i].z);
#pragma unroll
    for (int i = 0; i < TT; ++i) acc[i] = __fadd_rn(acc[i], now[i].w);
#pragma unroll
    for (int i = 0; i < TT; ++i) now[i] = next[i];
  }
}

// Bounded wait that naps between polls, for a warp that shares its scheduler with a
// warp doing the real work.
__device__ __forceinline__ bool mbar_wait_nap(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (mbar_try(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
    __nanosleep(64);
    if (mbar_try(bar, parity)) return true;
    if (*abort_flag) return false;
    if (clock64() - t0 > wait_budget()) {
      *abort_flag = 1;
      return false;
    }
  }
}

__host__ __device__ constexpr int router_producer_warps(bool packed) { return packed ? 1 : 4; }

// PER_SM: blocks that an SM has to have registers for.  Two for blocks of 4 x 4 tokens in more than one wave (32 experts of 2880 columns, 8192 tokens
// 107 us with registers for one, 90 with two; plain weights 107 and 95).  In one wave an SM has one block anyhow, and registers for two take the
// second set of loads from it: 2000 tokens 29.3 us with two, 28.1 with one, plain weights 33.5 and 31.6; 512 tokens of 128 experts 28.2 and 27.0.
template <int TW, int TT, int CH, bool PACKED, int PER_SM = 1>
__global__ void __launch_bounds__((TW + router_producer_warps(PACKED)) * 32, PER_SM)
k_router_logits(const RouterArgs A) {
  extern __shared__ __align__(128) uint8_t router_smem_raw[];
  constexpr int LD = CH + kRouterPad;
  constexpr int NS = router_stages(CH), NP = router_producer_warps(PACKED);
  constexpr int BT = TW * TT;                   // tokens of the block
  constexpr int stage_floats = (32 + BT) * LD;  // ws[32][LD] then hs[BT][LD]
  const uint32_t stages = smem_u32(router_smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(router_smem_raw + (size_t)NS * stage_floats * sizeof(float));
  const uint32_t bar_base = smem_u32(bars);
  auto bar_full = [&](int s) { return bar_base + 8u * s; };
  auto bar_empty = [&](int s) { return bar_base + 8u * (NS + s); };
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * NS);
  volatile int* ticket = abort_flag + 1;
  float* const exchanged = reinterpret_cast<float*>(bars) + 32;  // two buffers of the block's tokens x E logits (with a cluster)

  const int T = A.T, H = A.H, E = A.E;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int e0 = blockIdx.y * 32;
  const int n_chunks = (H + CH - 1) / CH;

  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      mbar_init(bar_full(s), (PACKED ? 1 : NP) + 32 * NP);  // the copies' announcement, and every producer lane's token pieces
      mbar_init(bar_empty(s), TW);
    }
    *abort_flag = 0;
    *ticket = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (A.cluster) cluster_sync_all();  // (a block of the cluster may be written to only once it runs)
  else __syncthreads();
  const int* const list = A.token_list;
  const float* const packed = A.wg + (size_t)blockIdx.y * n_chunks * 32 * LD;
  auto packed_stage = [&](int ci, int st) {
    mbar_expect_tx(bar_full(st), 32 * LD * 4);
    bulk_load(stages + (uint32_t)st * stage_floats * 4, packed + (size_t)ci * 32 * LD, 32 * LD * 4, bar_full(st));
  };
  const int e = e0 + lane;
  const float bias = A.bias && warp >= NP && e < E ? __ldg(A.bias + e) : 0.f;  // (the router's own, older than any kernel of the step)
  const int ahead = PACKED && !list ? min(NS, n_chunks) : 0;  // (a list may turn out empty; T is not)
  if (warp == 0 && lane == 0)
    for (int ci = 0; ci < ahead; ++ci) packed_stage(ci, ci);
  griddep_wait();
  griddep_launch();
  // tokens of this launch: all T, or the entries of a list built by an earlier kernel
  const int n_list = list ? min(*reinterpret_cast<volatile int*>(A.n_list), T) : 0;
  const int n_tok = list ? (n_list > A.list_over && n_list <= A.list_max ? n_list : 0) : T;
  auto token_at = [&](int ti) { return ti < n_tok ? (list ? list[ti] : ti) : -1; };

  // A block takes the token blocks blockIdx.x, blockIdx.x + gridDim.x, ...  (one each unless the launch
  // is list-driven and the list turned out longer than the grid).  The ring's barriers carry on from
  // one token block to the next: cg = running number of the chunk.
  bool ok = true;
  int cg = 0;
  for (int tb = blockIdx.x, iter = 0; tb * BT < n_tok; tb += gridDim.x, ++iter) {
    const int t0 = tb * BT;
    if (warp < NP) {
      // ------------------------------ producers ------------------------------
      const int n_e = min(32, E - e0);
      const int row = warp + NP * lane;  // !PACKED: producer p moves expert rows p, p + NP, ...
      const int n_mine = __popc(__ballot_sync(0xffffffffu, row < n_e));
      constexpr int R = (BT + NP - 1) / NP;  // token rows p, p + NP, ... are a producer's
      const float* src[R];
      // Many rows: a lane looks up one, the others' come from their lanes.  With 32 look-ups one after the other, in code that runs for the first time,
      // the first stage came 6400 clocks after the wait, now 4500: 16 experts of 512 columns, 4096 tokens 16.0 us, now 15.0; 128 of 2880, 1000 tokens
      // 47.0, now 46.1.  Of 16 rows and fewer every lane looks up all of them: 200 tokens of 128 experts 18.4 us, with the exchange 23.9.
      constexpr bool kExchange = TW > 4;
      const int mine = kExchange && warp + NP * lane < BT ? token_at(t0 + warp + NP * lane) : -1;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int r = warp + NP * i, t = kExchange ? __shfl_sync(0xffffffffu, mine, i) : r < BT ? token_at(t0 + r) : -1;
        src[i] = t >= 0 ? A.hidden + (size_t)t * H + lane * 4 : nullptr;
      }
      for (int ci = 0; ci < n_chunks; ++ci, ++cg) {
        const int st = cg % NS, d0 = ci * CH, dc = min(CH, H - d0);
        if (ok && cg >= NS) ok = __all_sync(0xffffffffu, mbar_wait_nap(bar_empty(st), (uint32_t)((cg / NS - 1) & 1), abort_flag));
        if (!ok) break;
        const uint32_t dst = stages + (uint32_t)st * stage_floats * 4;
        if (PACKED) {
          if (lane == 0 && cg >= ahead) packed_stage(ci, st);
        } else {
          const uint32_t row_bytes = (uint32_t)dc * sizeof(float);  // H % 32 == 0: a multiple of 128
          if (lane == 0) mbar_expect_tx(bar_full(st), (uint32_t)n_mine * row_bytes);
          __syncwarp();
          if (row < n_e) bulk_load(dst + (uint32_t)row * LD * 4, A.wg + (size_t)(e0 + row) * H + d0, row_bytes, bar_full(st));
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
          if (src[i]) {
#pragma unroll
            for (int c = 0; c < CH; c += 128)
              if (c + lane * 4 < dc) cp_async16(dst + (uint32_t)((32 + warp + NP * i) * LD + c + lane * 4) * 4, src[i] + d0 + c);
          }
        }
        cp_async_arrive(bar_full(st));
      }
      __syncwarp();
    } else {
      // ------------------------------ consumers ------------------------------
      const int w = warp - NP;
      float acc[TT];
#pragma unroll
      for (int i = 0; i < TT; ++i) acc[i] = 0.f;
      constexpr int G = router_groups(TW, TT), BC = 4 * G, NB = CH / BC;  // columns of a batch, batches of a chunk
      static_assert(NB % 2 == 0 && 32 % BC == 0, "batches");
      ChainBatch<TT, G> even, odd;
      float4 now[TT];
      auto w_at = [&](int c) { return stages + (uint32_t)((c % NS) * stage_floats + lane * LD) * 4; };
      auto h_at = [&](int c) { return stages + (uint32_t)((c % NS) * stage_floats + (32 + w * TT) * LD) * 4; };
      ok = mbar_wait(bar_full(cg % NS), (uint32_t)((cg / NS) & 1), abort_flag) && ok;
      uint32_t wp = w_at(cg), hp = h_at(cg);
#pragma unroll
      for (int g = 0; g < G; ++g) even.load(g, wp, hp, LD * 4);
      even.products(0, now);
      const int full = H / CH;
#pragma unroll 1
      for (int ci = 0; ci < full; ++ci) {
        const int st = cg % NS;
        ++cg;
        const uint32_t parity = (uint32_t)((cg / NS) & 1);
        const bool more = ci + 1 < n_chunks;
        bool here = false;
#pragma unroll
        for (int b = 0; b < NB; b += 2) {
          chain_batch<TT, G>(even, odd, wp + (b + 1) * BC * 4, hp + (b + 1) * BC * 4, LD * 4, now, acc);
          if (b + 2 == NB && more) {  // the next chunk's first batch
            if (!here) ok = mbar_wait(bar_full(cg % NS), parity, abort_flag) && ok;
            wp = w_at(cg);
            hp = h_at(cg);
          }
          // (the answer is needed two batches on; the question alone costs 100 cycles in front of a chunk)
          if (b + 4 == NB) here = more && mbar_test(bar_full(cg % NS), parity);
          const int ahead_columns = b + 2 < NB ? (b + 2) * BC : 0;  // (without a next chunk: anything, not used)
          chain_batch<TT, G>(odd, even, wp + ahead_columns * 4, hp + ahead_columns * 4, LD * 4, now, acc);
        }
        __syncwarp();
        if (lane == 0 && ok) mbar_arrive(bar_empty(st));
      }
      if (full < n_chunks) {  // the rest of a row
        const int batches = (H - full * CH) / BC;
#pragma unroll 1
        for (int b = 0; b < batches; b += 2) {
          // (a batch past the row's end is in the stage too: anything, not used)
          chain_batch<TT, G>(even, odd, wp + (b + 1) * BC * 4, hp + (b + 1) * BC * 4, LD * 4, now, acc);
          if (b + 1 == batches) break;
          chain_batch<TT, G>(odd, even, wp + (b + 2) * BC * 4, hp + (b + 2) * BC * 4, LD * 4, now, acc);
        }
        const int st = cg++ % NS;
        __syncwarp();
        if (lane == 0 && ok) mbar_arrive(bar_empty(st));
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < TT; ++i) {
        const int j = w * TT + i, t = token_at(t0 + j);
        const float logit = e < E ? __fadd_rn(acc[i], bias) : -INFINITY;
        if (A.counters && gridDim.y == 1) {
          float v[1] = {logit};
          if (t >= 0) warp_topk_regs<false, 1>(v, E, A.k, A.sigmoid, A.router_out + (size_t)t * A.k * 2, nullptr);
        } else if (t >= 0 && e < E) {
          if (A.cluster) {
            const uint32_t to = map_to_cta(smem_u32(exchanged + ((size_t)(iter & 1) * BT + j) * E + e), (uint32_t)j % gridDim.y);
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to), "f"(logit) : "memory");
          } else {
            A.logits[(size_t)t * E + e] = logit;
          }
        }
      }
      if (A.counters && !A.cluster) __threadfence();  // the logits before the block's ticket below
    }
    if (A.counters == nullptr || gridDim.y == 1) continue;
    int first = 0, step = 1;
    if (A.cluster) {
      // (a block writes the next token block's logits into the other buffer, and the one after that only when all have come
      // past the next barrier, which is after they have read these)
      cluster_sync_all();
      first = blockIdx.y;
      step = gridDim.y;
    } else {
      // ---- the last block of this token block selects the top-k ----
      __syncthreads();
      if (tid == 0) {
        __threadfence();  // this block's logits before its ticket
        const int last = atomicAdd(&A.counters[tb], 1) == (int)gridDim.y - 1;
        if (last) {
          A.counters[tb] = 0;  // ready for the next launch
          __threadfence();     // the other blocks' logits after their tickets
        }
        *ticket = last;
      }
      __syncthreads();
      if (!*ticket) first = BT;
    }
    for (int j = first + step * warp; j < BT; j += step * (TW + NP)) {
      const int t = token_at(t0 + j);
      if (t < 0) continue;
      float* const to = A.router_out + (size_t)t * A.k * 2;
      if (A.cluster) warp_topk<false, 32 * kRouterClusterGroups>(exchanged + ((size_t)(iter & 1) * BT + j) * E, E, A.k, A.sigmoid, to);
      else warp_topk(A.logits + (size_t)t * E, E, A.k, A.sigmoid, to);
    }
    if (!A.cluster) __syncthreads();  // `ticket` is rewritten by the next token block
  }  // token blocks of this block

  if (warp < NP) {
    // let the copies still in flight land before the block goes away (they have, unless a wait ran out)
    const int issued = cg;
    for (int i = 0; lane == 0 && *abort_flag && i < NS && i < issued; ++i) {
      const int c = issued - 1 - i;
      const long long tc = clock64();
      while (!mbar_try(bar_full(c % NS), (uint32_t)((c / NS) & 1)) && clock64() - tc < drain_budget()) {
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  __syncthreads();
  if (tid == 0 && *abort_flag && A.status) atomicOr(A.status, kDevErrWaitTimeout);
  if (list && n_tok && tid == 0) {
    // every block of the launch that takes the list, busy or idle, has read its length by now: the last
    // one to get here clears it for the next step
    __threadfence();
    if (atomicAdd(A.fb_done, 1) == (int)(gridDim.x * gridDim.y) - 1) {
      if (A.fb_total) atomicAdd(A.fb_total, (unsigned long long)n_tok);
      *A.n_list = 0;
      *A.fb_done = 0;
      __threadfence();
    }
  }
}

template <int TW, int TT, int CH, bool PACKED, int PER_SM = 1>
cudaError_t router_prepare_one() {
  return cudaFuncSetAttribute(k_router_logits<TW, TT, CH, PACKED, PER_SM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)router_smem_bytes(TW * TT, CH, PACKED ? 32 * kRouterClusterGroups : 0));
}
template <bool PACKED>
cudaError_t router_prepare_set() {
  cudaError_t e = router_prepare_one<1, 1, kRouterChunkFew, PACKED>();
  if (e == cudaSuccess) e = router_prepare_one<2, 1, kRouterChunkFew, PACKED>();
  if (e == cudaSuccess) e = router_prepare_one<4, 1, kRouterChunkFew, PACKED>();
  if (e == cudaSuccess) e = router_prepare_one<4, 2, kRouterChunkMany, PACKED>();
  if (e == cudaSuccess) e = router_prepare_one<4, 3, kRouterChunkMany, PACKED>();
  if (e == cudaSuccess) e = router_prepare_one<4, 4, kRouterChunkMany, PACKED>();
  if (e == cudaSuccess) e = router_prepare_one<4, 4, kRouterChunkMany, PACKED, 2>();
  if (e == cudaSuccess) e = router_prepare_one<8, 3, kRouterChunkMany, PACKED>();
  if (e == cudaSuccess) e = router_prepare_one<8, 4, kRouterChunkMany, PACKED>();
  return e;
}
// Lets the router kernels use more than the default 48 KB of dynamic shared
// memory.  Once per device.
inline cudaError_t router_prepare_device();

// How the chain is launched for a number of groups of 32 experts: the blocks that are resident at once, and whether the blocks of a
// token block form a cluster (else they meet in global memory).
struct RouterWave {
  int blocks;
  bool clusters;
  int alone;  // blocks resident at once without clusters
};

template <int TW, int TT, int CH, bool PACKED, int PER_SM = 1>
void launch_router_one(RouterArgs a, int token_slots, RouterWave wave, cudaStream_t s, bool pdl) {
  const unsigned groups = (unsigned)((a.E + 31) / 32);
  constexpr int BT = TW * TT;
  a.cluster = PACKED && a.counters && wave.clusters;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)((token_slots + BT - 1) / BT), groups);
  cfg.blockDim = dim3((TW + router_producer_warps(PACKED)) * 32);
  cfg.dynamicSmemBytes = router_smem_bytes(BT, CH, a.cluster ? a.E : 0);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = a.cluster ? groups : 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  cudaLaunchKernelEx(&cfg, k_router_logits<TW, TT, CH, PACKED, PER_SM>, a);
}

// An SM each, but clusters leave some SMs of a GPC over (with a fixed nine tenths of the SMs, 64 tokens of 256 experts took two waves
// of clusters of eight, 30.5 us): the runtime is asked about the widest launch.  One group needs no cluster, more than
// kRouterClusterGroups of them can have none, and where no such cluster can be resident (a part of a device) there is none either.
// (Through global memory, with clusters / without, us: 128 experts of 2880 columns 8 tokens 14.5 / 15.7, 333 25.4 / 28.8; 64 experts 333 20.6 / 23.0.)
inline RouterWave router_wave(int groups, int sm_count) {
  if (groups < 2 || groups > kRouterClusterGroups) return {sm_count, false, sm_count};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(1024, (unsigned)groups);
  cfg.blockDim = dim3((8 + router_producer_warps(true)) * 32);
  cfg.dynamicSmemBytes = router_smem_bytes(32, kRouterChunkMany, 32 * groups);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = (unsigned)groups;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, k_router_logits<8, 4, kRouterChunkMany, true>, &cfg) != cudaSuccess || clusters < 1) {
    cudaGetLastError();
    return {sm_count, false, sm_count};
  }
  return {std::min(clusters * groups, sm_count), true, sm_count};
}

// The fewest tokens per block with which the blocks are one wave: a block's time goes by its chains per thread and, from four warps
// on, by its shared-memory reads (a row of weights per lane costs 4 cycles per four columns, a token row 2), so that a second
// wave is dearer than more chains in one.  `wave`: see router_wave.  A launch among others, us, 2880 columns, by the shape taken (warps x tokens
// of a warp): 128 experts, 8 tokens 1x1 11.8; 50 2x1 13.9; 100 4x1 14.4; 200 4x2 18.5; 333 4x3 22.3; 512 4x4 27.0; 700 8x3 38.3; 1000 8x4 46.1;
// 32 experts, 333 4x1 13.9; 1024 4x2 18.5; 2000 4x4 28.1; 4096 8x4 47.2; 6000 4x4 72.0 and 8192 4x4 90.2, two blocks an SM (8x4 95).  Other shapes: 100
// tokens 2x2 17.8; 592 8x2 38.3; 700 4x6 44.2; 1000 4x8 53.6.
// wg_few / wg_many: the weights packed for the two chunk widths (PACKED) or both the plain [E,H] matrix.  token_slots: tokens the
// grid is sized for (a.T, or for a list-driven launch the most entries the list can have).
template <bool PACKED>
inline void launch_router_logits(RouterArgs a, const float* wg_few, const float* wg_many, RouterWave wave, cudaStream_t s,
                                 bool pdl = false, int token_slots = -1) {
  if (token_slots < 0) token_slots = a.T;
  const int64_t groups = (a.E + 31) / 32;
  auto one_wave = [&](int tokens) { return (token_slots + tokens - 1) / tokens * groups <= wave.blocks; };
  if (wave.clusters && !one_wave(32) && a.H > 256) {
    // The SMs that clusters leave over may be what the last wave needs: without clusters then, unless a chain is so short that the
    // selection in one block per token block takes as long.  With / without, us: 2880 columns, 256 experts (120 blocks at once / 148), 511 tokens
    // 94.3 / 54.5, 1000 139.5 / 99.0; 224 experts, 560 tokens 94.3 / 55.0; 256 experts, 511 tokens, 1024 columns 43.2 / 30.9, 512 28.9 / 24.8, 128
    // 16.7 / 18.6.
    const int64_t blocks = (token_slots + 31) / 32 * groups;
    if ((blocks + wave.alone - 1) / wave.alone < (blocks + wave.blocks - 1) / wave.blocks) wave = {wave.alone, false, wave.alone};
  }
  a.wg = wg_few;
  if (one_wave(1)) return launch_router_one<1, 1, kRouterChunkFew, PACKED>(a, token_slots, wave, s, pdl);
  if (one_wave(2)) return launch_router_one<2, 1, kRouterChunkFew, PACKED>(a, token_slots, wave, s, pdl);
  if (one_wave(4)) return launch_router_one<4, 1, kRouterChunkFew, PACKED>(a, token_slots, wave, s, pdl);
  a.wg = wg_many;
  if (one_wave(8)) return launch_router_one<4, 2, kRouterChunkMany, PACKED>(a, token_slots, wave, s, pdl);
  if (one_wave(12)) return launch_router_one<4, 3, kRouterChunkMany, PACKED>(a, token_slots, wave, s, pdl);
  if (one_wave(16)) return launch_router_one<4, 4, kRouterChunkMany, PACKED>(a, token_slots, wave, s, pdl);
  if (!one_wave(32) && groups == 1) return launch_router_one<4, 4, kRouterChunkMany, PACKED, 2>(a, token_slots, wave, s, pdl);
  if (one_wave(24)) return launch_router_one<8, 3, kRouterChunkMany, PACKED>(a, token_slots, wave, s, pdl);
  launch_router_one<8, 4, kRouterChunkMany, PACKED>(a, token_slots, wave, s, pdl);
}

// ---------------------------------------------------------------------------
// Fast router with certified selection.
//
// The reference's logit is a sequential fp32 chain, which runs at the add latency and, for a
// handful of tokens, on a handful of SMs.  Here the logits are computed with fused
// multiply-adds, split over the hidden dimension across many CTAs, and every logit carries a
// rigorous bound on its distance from the reference's chain value C:
//   |C - S| <= u (sum_i |S_i| + A),  S_i the exact partial sums in column order, A = sum |h w|
//   (one rounding per product, one per addition; u = 2^-24), and for column i of 32-column
//   block j:  |S_i| <= |R_j| + A_j  (R_j the prefix at the block's start), so
//   sum_i |S_i| <= 32 sum_j |R_j| + 32 A;
//   the block-wise FMA sum itself is within u (17 A + sum_j |R_j|) of S;
//   A <= |h|_2 |w_e|_2 (Cauchy-Schwarz; |w_e|_2 precomputed, |h|_2 summed on the way).
// bound = 1.05 u (33 sum_j |R_j| + 50 |h| |w_e|) + 4 u |logit| covers both, the two roundings
// of the bias addition and the rounding of the bound's own arithmetic.  The top-k step accepts
// a selection only when the gaps between neighbours of the k best logits exceed the sum of
// their bounds and no expert left out can reach the last of them; every other token goes through the order-faithful chain (k_router_logits over
// the list of those tokens).  Expert indices are therefore the reference's in every case.
//
// k_router_fast: CTA = (block of 4*TPW tokens, group of 32 experts, part m of the hidden
// dimension).  A part is a run of 96-column slices; per slice the CTA stages the 32 x 96
// weight block and its tokens' 96 columns in shared memory, every lane takes ITS expert's 96
// weights into registers and runs its warp's TPW tokens against them (token values by
// broadcast loads: one shared-memory wavefront per four FMAs).  Per (token, expert, part) it
// leaves c = the part's sum and a = sum over the part's blocks of |prefix inside the part|.
// k_router_finish: a block per token, a thread per expert adds the parts in order (prefix P_m before part m:
// sum_j |R_j| <= sum_m (blocks_m |P_m| + a_m)), forms logits and bounds, selects and certifies.
// ---------------------------------------------------------------------------
constexpr int kFastSliceBlocks = 3;                     // 32-column blocks per slice
constexpr int kFastSliceCols = 32 * kFastSliceBlocks;   // 96
constexpr int kFastLdw = kFastSliceCols + 4;            // weight row stride in shared memory (16-byte multiple;
                                                        // a quarter-warp's 128-bit reads of one column group
                                                        // of eight neighbouring rows hit distinct banks)

struct FastRouterArgs {
  const float* hidden;  // [T,H], 16-byte aligned
  const float* wg;      // [E,H] plain, 16-byte aligned
  float2* part;         // [T][parts][E]: (c, a)
  float* hn2;           // [T][parts]: the part's share of the token row's sum of squares
  int T, H, E;
};

inline int fast_router_slices(int H) { return (H / 32 + kFastSliceBlocks - 1) / kFastSliceBlocks; }
inline size_t fast_router_smem(int tpw) { return 2 * (size_t)(32 * kFastLdw + 4 * tpw * kFastSliceCols) * sizeof(float); }

template <int TPW>
__global__ void __launch_bounds__(128) k_router_fast(const FastRouterArgs A) {
  constexpr int TB = 4 * TPW;
  constexpr int kStage = 32 * kFastLdw + TB * kFastSliceCols;  // floats: weight block, then token block
  extern __shared__ __align__(16) float fast_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int T = A.T, H = A.H, E = A.E;
  const int t_base = blockIdx.x * TB, e0 = blockIdx.y * 32;
  const int parts = gridDim.z, m = blockIdx.z;
  const int n_slices = (H / 32 + kFastSliceBlocks - 1) / kFastSliceBlocks;
  const int s_begin = n_slices * m / parts, s_end = n_slices * (m + 1) / parts;
  float R[TPW], aR[TPW], h2[TPW];
#pragma unroll
  for (int i = 0; i < TPW; ++i) R[i] = aR[i] = h2[i] = 0.f;
  griddep_wait();
  griddep_launch();
  // all 16-byte pieces of a slice are requested at once (cp.async); what lies outside the matrices is zero
  auto stage_slice = [&](int sl, int buf) {
    float* Ws = fast_smem + buf * kStage;
    float* Hs = Ws + 32 * kFastLdw;
    const int col0 = sl * kFastSliceCols;
    for (int idx = tid; idx < 32 * (kFastSliceCols / 4); idx += 128) {
      const int r = idx / (kFastSliceCols / 4), q = idx % (kFastSliceCols / 4);
      const int e = e0 + r, col = col0 + q * 4;  // H is a multiple of 32: col < H means the whole piece is inside
      float* d = Ws + r * kFastLdw + q * 4;
      if (e < E && col < H) cp_async16(smem_u32(d), A.wg + (size_t)e * H + col);
      else *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int idx = tid; idx < TB * (kFastSliceCols / 4); idx += 128) {
      const int r = idx / (kFastSliceCols / 4), q = idx % (kFastSliceCols / 4);
      const int t = t_base + r, col = col0 + q * 4;
      float* d = Hs + r * kFastSliceCols + q * 4;
      if (t < T && col < H) cp_async16(smem_u32(d), A.hidden + (size_t)t * H + col);
      else *reinterpret_cast<float4*>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    cp_async_commit();
  };
  if (s_begin < s_end) stage_slice(s_begin, 0);
  for (int sl = s_begin; sl < s_end; ++sl) {
    const int buf = (sl - s_begin) & 1;
    if (sl + 1 < s_end) {
      stage_slice(sl + 1, buf ^ 1);  // the other buffer's readers finished before the barrier that ended slice sl - 1
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const float* Ws = fast_smem + buf * kStage;
    const float* Hs = Ws + 32 * kFastLdw;
    float w[kFastSliceCols];
#pragma unroll
    for (int q = 0; q < kFastSliceCols / 4; ++q) {
      const float4 v = *reinterpret_cast<const float4*>(Ws + lane * kFastLdw + q * 4);
      w[q * 4 + 0] = v.x;
      w[q * 4 + 1] = v.y;
      w[q * 4 + 2] = v.z;
      w[q * 4 + 3] = v.w;
    }
    // TG tokens at a time: 2 * TG independent FMA chains and TG broadcast loads in flight per lane
    constexpr int TG = TPW < 4 ? TPW : 4;
#pragma unroll
    for (int i0 = 0; i0 < TPW; i0 += TG) {
      const float* hp = Hs + (warp * TPW + i0) * kFastSliceCols;
#pragma unroll
      for (int blk = 0; blk < kFastSliceBlocks; ++blk) {
        float b0[TG], b1[TG];
#pragma unroll
        for (int j = 0; j < TG; ++j) b0[j] = b1[j] = 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          float4 hv[TG];
#pragma unroll
          for (int j = 0; j < TG; ++j)
            hv[j] = *reinterpret_cast<const float4*>(hp + j * kFastSliceCols + blk * 32 + q * 4);
#pragma unroll
          for (int j = 0; j < TG; ++j) {
            b0[j] = fmaf(hv[j].x, w[blk * 32 + q * 4 + 0], b0[j]);
            b1[j] = fmaf(hv[j].y, w[blk * 32 + q * 4 + 1], b1[j]);
          }
#pragma unroll
          for (int j = 0; j < TG; ++j) {
            b0[j] = fmaf(hv[j].z, w[blk * 32 + q * 4 + 2], b0[j]);
            b1[j] = fmaf(hv[j].w, w[blk * 32 + q * 4 + 3], b1[j]);
          }
        }
#pragma unroll
        for (int j = 0; j < TG; ++j) {
          const float hx = hp[j * kFastSliceCols + blk * 32 + lane];  // the warp's lanes share the row's squares
          h2[i0 + j] = fmaf(hx, hx, h2[i0 + j]);
          R[i0 + j] += b0[j] + b1[j];
          aR[i0 + j] += fabsf(R[i0 + j]);
        }
      }
    }
    __syncthreads();  // this buffer is refilled during the next slice
  }
  const int e = e0 + lane;
#pragma unroll
  for (int i = 0; i < TPW; ++i) {
    const int t = t_base + warp * TPW + i;
    float q = h2[i];
    if (blockIdx.y == 0) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    }
    if (t < T) {
      if (e < E) A.part[((size_t)t * parts + m) * E + e] = make_float2(R[i], aR[i]);
      if (blockIdx.y == 0 && lane == 0) A.hn2[(size_t)t * parts + m] = q;
    }
  }
}

struct FinishRouterArgs {
  const float2* part;   // [T][parts][E]
  const float* hn2;     // [T][parts]
  const float* bias;    // [E] or null
  const float* wnorm;   // [E] upper bounds of the gate rows' 2-norms
  float* router_out;    // [T,k,2]
  int* fb_list;         // tokens whose selection is not certified ...
  int* fb_count;        // ... and how many (zero between steps)
  int T, H, E, k, sigmoid, parts;
  // k_router_finish_many: the blocks along H that the parts are made of, and the two constants of the logits' bound
  // u (coef_prefix * sum |prefix| + coef_norm * |h| |w|)
  int slices;
  float coef_prefix, coef_norm;
};

constexpr int kFastMaxParts = 32;
// Squares of values under 2^-75 vanish in fp32: 2^16 columns of them have a norm of at most this.
constexpr float kNormFloor = 0x1p-66f;

// One block per token, one thread per expert (more experts than threads take turns): the block brings the token's parts to shared
// memory, a thread adds its expert's in order; logits and bounds meet in shared memory, where warp 0 selects.  The code runs once a
// launch, cold, so its length counts: with the parts of an expert loaded by its thread, 32 of them unrolled, the sums took 5900
// clocks of the kernel's 9400 after the wait (30 parts, 128 experts).
constexpr int kFinishThreads = 256, kFinishMaxSmem = 96 * 1024;
inline size_t finish_smem_bytes(int parts, int E) { return sizeof(float2) * parts * E; }
__global__ void __launch_bounds__(kFinishThreads) k_router_finish(const FinishRouterArgs A) {
  extern __shared__ __align__(16) float2 finish_parts[];  // [parts][E]
  __shared__ float s_logit[kMaxExperts], s_bound[kMaxExperts];
  __shared__ float s_blocks[kFastMaxParts];
  const int tid = threadIdx.x, lane = tid & 31;
  const int t = blockIdx.x;
  const int parts = A.parts, E = A.E;
  const int n_slices = (A.H / 32 + kFastSliceBlocks - 1) / kFastSliceBlocks;
  // blocks of each part (a division each: by one thread)
  if (tid < parts) s_blocks[tid] = (float)(kFastSliceBlocks * (n_slices * (tid + 1) / parts - n_slices * tid / parts));
  // (the router's own, older than any kernel of the step)
  float bias = A.bias && tid < E ? __ldg(A.bias + tid) : 0.f, wn = tid < E ? __ldg(A.wnorm + tid) : 0.f;
  griddep_wait();
  griddep_launch();
  const float2* src = A.part + (size_t)t * parts * E;
  if (E % 2 == 0) {  // 16 bytes are two experts'
#pragma unroll 4
    for (int i = 2 * tid; i < parts * E; i += 2 * kFinishThreads) cp_async16(smem_u32(finish_parts + i), src + i);
    cp_async_commit();
  } else {
#pragma unroll 4
    for (int i = tid; i < parts * E; i += kFinishThreads) finish_parts[i] = __ldcg(src + i);
  }
  float h2 = lane < parts ? __ldcg(A.hn2 + (size_t)t * parts + lane) : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) h2 += __shfl_xor_sync(0xffffffffu, h2, o);  // every warp, all lanes
  const float hn = sqrtf(h2) * 1.001f + kNormFloor;
  cp_async_wait<0>();
  __syncthreads();
  for (int e = tid; e < E; e += kFinishThreads) {
    if (e >= kFinishThreads) {
      bias = A.bias ? __ldg(A.bias + e) : 0.f;
      wn = __ldg(A.wnorm + e);
    }
    float P = 0.f, sr = 0.f;
#pragma unroll 4
    for (int m = 0; m < parts; ++m) {
      const float2 v = finish_parts[m * E + e];
      sr += s_blocks[m] * fabsf(P) + v.y;
      P += v.x;
    }
    const float logit = __fadd_rn(P, bias);
    s_logit[e] = logit;
    s_bound[e] = 6.3e-8f * (33.f * sr + 50.f * hn * wn) + 2.4e-7f * fabsf(logit) + 1e-30f;
  }
  __syncthreads();
  if (tid >= 32) return;
  const bool sure = warp_topk<false, kMaxExperts, false>(s_logit, E, A.k, A.sigmoid, A.router_out + (size_t)t * A.k * 2, s_bound);
  if (!sure && lane == 0) A.fb_list[atomicAdd(A.fb_count, 1)] = t;  // at most one entry per token
}

// The same for many tokens: a warp per token, so that no warp waits while another selects (a block per token took 91 us
// of 8192 tokens).  Shared memory: logits and bounds of kFinishWarps tokens.
constexpr int kFinishWarps = 8;
// (two blocks an SM: left alone, the compiler takes 80 registers for three and spills in the loop over the parts, 256 experts of 1024 columns, 2048 tokens 50.5 -> 53.9 us)
__global__ void __launch_bounds__(32 * kFinishWarps, 2) k_router_finish_many(const FinishRouterArgs A) {
  extern __shared__ float finish_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = blockIdx.x * kFinishWarps + warp;
  const int parts = A.parts, E = A.E;
  float* s_logit = finish_smem + (size_t)warp * 2 * E;
  float* s_bound = s_logit + E;
  griddep_wait();
  griddep_launch();
  if (t >= A.T) return;
  float h2 = lane < parts ? __ldcg(A.hn2 + (size_t)t * parts + lane) : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) h2 += __shfl_xor_sync(0xffffffffu, h2, o);
  const float hn = sqrtf(h2) * 1.001f + kNormFloor;
  // four experts of a lane at a time, their loads in flight together (one after the other: 8192 tokens of 128 experts 24 us, now 15)
  constexpr int N = 4;
  for (int e0 = lane; e0 < E; e0 += 32 * N) {
    float P[N], sr[N], bias[N], wn[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int e = e0 + 32 * i;
      P[i] = sr[i] = 0.f;
      bias[i] = A.bias && e < E ? A.bias[e] : 0.f;
      wn[i] = e < E ? A.wnorm[e] : 0.f;
    }
    for (int m = 0; m < parts; ++m) {
      float2 v[N];
#pragma unroll
      for (int i = 0; i < N; ++i)
        if (e0 + 32 * i < E) v[i] = __ldcg(A.part + ((size_t)t * parts + m) * E + e0 + 32 * i);
      const float blocks = (float)(A.slices * (m + 1) / parts - A.slices * m / parts);
#pragma unroll
      for (int i = 0; i < N; ++i) {
        if (e0 + 32 * i >= E) continue;
        sr[i] += blocks * fabsf(P[i]) + v[i].y;
        P[i] += v[i].x;
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int e = e0 + 32 * i;
      if (e >= E) continue;
      const float logit = __fadd_rn(P[i], bias[i]);
      s_logit[e] = logit;
      s_bound[e] = 6.3e-8f * (A.coef_prefix * sr[i] + A.coef_norm * hn * wn[i]) + 2.4e-7f * fabsf(logit) + 1e-30f;
    }
  }
  __syncwarp();
  const bool sure = warp_topk<false>(s_logit, E, A.k, A.sigmoid, A.router_out + (size_t)t * A.k * 2, s_bound);
  if (!sure && lane == 0) A.fb_list[atomicAdd(A.fb_count, 1)] = t;  // at most one entry per token
}

inline cudaError_t router_prepare_device() {
  cudaError_t e = router_prepare_set<true>();
  if (e == cudaSuccess) e = router_prepare_set<false>();
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_router_finish_many, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(2 * kFinishWarps * kMaxExperts * sizeof(float)));
  // (Parts times groups of 32 experts are fewer than the SMs and the groups together, so the parts take at most 256 bytes an SM and 8 KB:
  // 45 KB on 148 SMs, with the arrays more than the 48 KB that need no leave; this is enough for 350.)
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_router_finish, cudaFuncAttributeMaxDynamicSharedMemorySize, kFinishMaxSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_router_fast<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fast_router_smem(8));
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_router_fast<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fast_router_smem(16));
  return e;
}

// 2-norm of every expert's gate row, rounded up (the fast router's Cauchy-Schwarz term).
__global__ void k_router_wnorm(const float* __restrict__ wg, float* __restrict__ wnorm, int E, int H) {
  const int e = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (e >= E) return;
  float acc = 0.f;
  for (int d = lane; d < H; d += 32) acc = fmaf(wg[(size_t)e * H + d], wg[(size_t)e * H + d], acc);
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) wnorm[e] = sqrtf(acc) * 1.001f + kNormFloor;
}

__global__ void __launch_bounds__(128)
k_router_topk(const float* __restrict__ logits, float* __restrict__ router_out, int T, int E, int k, int sigmoid) {
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (t >= T) return;
  warp_topk(logits + (size_t)t * E, E, k, sigmoid, router_out + (size_t)t * k * 2);
}

// ---------------------------------------------------------------------------
// Permutation by expert ("dispatch").  The reference's dispatch
// (moe_weight_fetch_node::extract_selected_experts, moe_weight_fetch_node.h:31-60,
// and the per-expert membership scans of expert_mlp_node.h:784-822) only finds
// WHICH experts were selected; grouping the (token, expert) rows by expert is
// what lets every expert's weights be read once.
//
// meta layout (int32): [0] row tiles, [1] total rows, [2] distinct experts,
//                      [3] device status word (or-ed kDevErr*), [4] rows of the tallest row tile, [5..7] spare.
// ---------------------------------------------------------------------------
//
// k_hist: rows per expert of a batch that is planned by two launches.  With `partial` every block leaves its own counts,
// partial[block][E + 1], the last of them whether it met an id outside [0, E), and nothing has to be cleared beforehand;
// else they are added to `counts` (zero at first) and the status word.
constexpr int kHistBlocks = 32;
__global__ void k_hist(const float* __restrict__ router_out, int n_pairs, int E, int only_expert,
                       int* __restrict__ counts, int* __restrict__ meta, int* __restrict__ partial = nullptr) {
  extern __shared__ int sc[];
  for (int e = threadIdx.x; e <= E; e += blockDim.x) sc[e] = 0;
  __syncthreads();
  griddep_wait();
  griddep_launch();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pairs; i += gridDim.x * blockDim.x) {
    const int e = (int)router_out[2 * (size_t)i];
    if (e < 0 || e >= E) {
      sc[E] = 1;
      continue;
    }
    if (only_expert >= 0 && e != only_expert) continue;
    atomicAdd(&sc[e], 1);
  }
  __syncthreads();
  if (partial) {
    for (int e = threadIdx.x; e <= E; e += blockDim.x) partial[(size_t)blockIdx.x * (E + 1) + e] = sc[e];
    return;
  }
  for (int e = threadIdx.x; e < E; e += blockDim.x)
    if (sc[e]) atomicAdd(&counts[e], sc[e]);
  if (threadIdx.x == 0 && sc[E]) atomicOr(&meta[3], kDevErrExpertRange);
}

// An expert with several tiles gets them equally tall instead of full ones and a short rest: for the block-scaled kernel always (its
// time goes by the tile's rows), for the CTA-pair kernels, whose tiles of 256 rows take MMAs of a multiple of 32, with two to four
// tiles (with more only the last one would change).  Full and rest / even, us: 8 experts of 2880 x 2880 (MXFP4) with 257 rows each 141 / 111, 330
// 147 / 127, 480 166 / 166, 513 224 / 184, 800 292 / 269, 1000 326 / 326; 32 experts 257 rows 452 / 397, 480 617 / 616 (637 with heights of a multiple of
// 16), 700 892 / 897 (955); fp16, one of 2880 x 2880, 257 43.8 / 33.5, 480 45.0 / 45.0, 800 54.0 / 51.5.
__device__ __forceinline__ int even_tile_height(int cnt, int tile_rows, bool block_scaled) {
  const int ntl = (cnt + tile_rows - 1) / tile_rows;
  if (ntl < 2) return tile_rows;
  const int even = (cnt + ntl - 1) / ntl;
  if (block_scaled) return even;
  return tile_rows >= 64 && ntl <= 4 ? min(tile_rows, (even + 31) & ~31) : tile_rows;
}

// Exclusive scan of the per-expert row counts, row-tile list for tiles of
// `tile_rows` rows, cursor reset.  One block of whole warps, a thread for every expert.
// counts are indexed by GLOBAL expert id; tiles carry the id local to this
// device (e - e_begin); rows of experts outside [e_begin, e_begin+e_count) get
// offsets but no tiles (under expert parallelism they belong to other devices).
//
// The counts come from `counts` or, with `partial`, from k_hist's blocks; with router_out given (small batches: at most
// kScanPairs pairs a thread) the block builds the histogram itself, and the whole plan is one launch.  In both cases counts
// and the status word need no clearing beforehand.
//
// With row_of_pair given as well the block also places every pair: row_of_pair[i] = its row in
// the grouped order (-1: not placed).  Which row of its expert's segment a pair gets is what the histogram's atomic returned;
// a row's value does not depend on it.
//
// Bound by its barriers and the latency of the routing's loads: 32 pairs, 128 experts 6.3 us with 1024 threads, a second
// pass of loads and atomics for the places and a search of the offsets for every tile, now 5.3 (profiler, cold caches).
constexpr int kScanPairs = 8;
struct ScanArgs {
  int *counts, *offsets, *cursor, *meta;
  int E, e_begin, e_count, tile_rows, max_rows, max_tiles;
  const uint8_t* resident;
  RowTile* tiles;
  const int* partial;           // or null
  int n_partial;
  const float* router_out;      // or null
  int n_pairs, only_expert;
  int* row_of_pair;             // or null
  ExpertTiles* expert_tiles;    // block-scaled kernel: where the experts' tiles are, the tiles' words to clear, the pairs' places
  uint32_t* tile_words;
  int words_per_tile;
  int4* places;
};
// Threads of the block.
inline int scan_threads(int E, int n_pairs) { return std::min(1024, std::max(ceil_div(E, 32), ceil_div(n_pairs, 32)) * 32); }

__global__ void __launch_bounds__(1024) k_scan(const ScanArgs A) {
  __shared__ int s_row_off[1024], s_tile_off[1024], s_count[1024];
  __shared__ int s_warp[2][32];
  __shared__ int s_distinct, s_tallest, s_status;
  const int e = threadIdx.x, lane = e & 31, warp = e >> 5, B = blockDim.x, E = A.E;
  if (e == 0) s_distinct = s_tallest = s_status = 0;
  s_count[e] = 0;
  const bool local = e >= A.e_begin && e < A.e_begin + A.e_count;
  const bool missing = local && A.resident && !A.resident[e - A.e_begin];  // (older than the kernel in front)
  __syncthreads();
  griddep_wait();
  griddep_launch();
  int x[kScanPairs], r[kScanPairs];  // the pairs of this thread: expert (-1: none, or not placed), row among the expert's
  if (A.router_out) {
#pragma unroll
    for (int j = 0; j < kScanPairs; ++j) x[j] = e + j * B < A.n_pairs ? (int)A.router_out[2 * (size_t)(e + j * B)] : 0;
#pragma unroll
    for (int j = 0; j < kScanPairs; ++j) {
      if (e + j * B >= A.n_pairs) {
        x[j] = -1;
      } else if (x[j] < 0 || x[j] >= E) {
        x[j] = -1;
        atomicOr(&s_status, kDevErrExpertRange);
      } else if (A.only_expert >= 0 && x[j] != A.only_expert) {
        x[j] = -1;
      }
      if (x[j] >= 0) r[j] = atomicAdd(&s_count[x[j]], 1);
    }
    __syncthreads();
  } else if (e < E) {
    int n = 0;
    if (A.partial)
      for (int b = 0; b < A.n_partial; ++b) n += A.partial[(size_t)b * (E + 1) + e];
    else
      n = A.counts[e];
    s_count[e] = n;
  }
  if (A.partial && e < A.n_partial && A.partial[(size_t)e * (E + 1) + E]) atomicOr(&s_status, kDevErrExpertRange);
  const int c = e < E ? s_count[e] : 0;
  const int nt = local ? (c + A.tile_rows - 1) / A.tile_rows : 0;
  auto tile_height = [&](int cnt) { return even_tile_height(cnt, A.tile_rows, A.expert_tiles != nullptr); };
  if (c > 0) {
    atomicAdd(&s_distinct, 1);
    if (missing) atomicOr(&s_status, kDevErrNotResident);
  }
  // block-wide inclusive scans of (c, nt)
  int rc = c, rt = nt;
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, rc, o), b = __shfl_up_sync(0xffffffffu, rt, o);
    if (lane >= o) {
      rc += a;
      rt += b;
    }
  }
  if (lane == 31) {
    s_warp[0][warp] = rc;
    s_warp[1][warp] = rt;
  }
  __syncthreads();
  // every warp adds up the warps before it and all of them
  int wc = lane < B / 32 ? s_warp[0][lane] : 0, wt = lane < B / 32 ? s_warp[1][lane] : 0;
  const int total_rows = __reduce_add_sync(0xffffffffu, wc), total_tiles = __reduce_add_sync(0xffffffffu, wt);
  if (lane >= warp) wc = wt = 0;
  const int row_off = __reduce_add_sync(0xffffffffu, wc) + rc - c, tile_off = __reduce_add_sync(0xffffffffu, wt) + rt - nt;
  s_row_off[e] = row_off;
  s_tile_off[e] = tile_off;
  const bool over = total_rows > A.max_rows || total_tiles > A.max_tiles;
  const int height = tile_height(c);
  if (e < E) {
    if (A.router_out || A.partial) A.counts[e] = c;
    A.offsets[e] = row_off;
    A.cursor[e] = 0;
    if (A.expert_tiles) A.expert_tiles[e] = ExpertTiles{tile_off, height};
  }
  if (nt && !over) {
    for (int q = 0; q < nt; ++q) A.tiles[tile_off + q] = RowTile{e - A.e_begin, row_off + q * height, min(height, c - q * height), 0};
    atomicMax(&s_tallest, min(height, c));
  }
  __syncthreads();
  if (e == 0) {
    A.offsets[E] = total_rows;
    A.meta[0] = over ? 0 : total_tiles;
    A.meta[1] = total_rows;
    A.meta[2] = s_distinct;
    const int st = s_status | (over ? kDevErrCapacity : 0);
    if (A.router_out || A.partial) A.meta[3] = st;
    else if (st) atomicOr(&A.meta[3], st);
    A.meta[4] = s_tallest;
    A.meta[5] = A.meta[6] = 0;
  }
  if (A.router_out && A.row_of_pair) {
#pragma unroll
    for (int j = 0; j < kScanPairs; ++j) {
      const int i = e + j * B;
      if (i >= A.n_pairs) break;
      int pos = -1;
      if (!over && x[j] >= 0) {
        pos = s_row_off[x[j]] + r[j];
        if (pos >= A.max_rows) pos = -1;
      }
      A.row_of_pair[i] = pos;
      if (A.places) {
        // the pair's row tile (number, first row, rows) and its row in it, or -1: one load for the kernel that writes the rows
        // where it would chase expert, tile number and tile
        int4 at = make_int4(0, 0, 0, -1);
        if (pos >= 0 && x[j] >= A.e_begin && x[j] < A.e_begin + A.e_count) {
          const int cnt = s_count[x[j]], per = tile_height(cnt), q = r[j] / per;
          at = make_int4(s_tile_off[x[j]] + q, s_row_off[x[j]] + q * per, min(per, cnt - q * per), r[j] - q * per);
        }
        A.places[i] = at;
      }
    }
  }
  if (A.tile_words && !over)  // the block-scaled kernel's record masks and counts: nothing marked or done yet
    for (int i = e; i < total_tiles * A.words_per_tile; i += B) A.tile_words[i] = 0;
}

// The same plan for a batch of up to kPlanPairs pairs, a thread each, whose rows stay on this device: nothing needs the experts in order, so
// an expert's first pair takes the next rows and tiles for all of them, without a scan over the experts and a thread for each.
// `offsets`, `cursor` and `expert_tiles` are not written: nothing reads them where the pairs' rows are given.  The flags of the loaded
// experts, older than the kernel in front, are read before the wait.  Bound by the latency of the routing's loads: 4 to 256 pairs of 128
// experts 2.3 -> 1.9 us in a step (16 tokens of eight slots 62.2 -> 61.8 us, 100 89.6 -> 88.2, block of 5 tokens with a shared expert 54.7 -> 53.7;
// with four pairs a thread 4000 pairs were no quicker than by k_scan).
constexpr int kPlanPairs = 1024;
__global__ void __launch_bounds__(kPlanPairs) k_plan(const ScanArgs A) {
  __shared__ int s_count[kMaxExperts], s_row[kMaxExperts], s_tile[kMaxExperts];
  __shared__ uint8_t s_missing[kMaxExperts];
  __shared__ uint32_t s_next;  // rows, and in the low half row tiles, given out
  __shared__ int s_distinct, s_tallest, s_status;
  const int i = threadIdx.x, lane = i & 31, B = blockDim.x, E = A.E;
  if (i == 0) s_next = 0u, s_distinct = s_tallest = s_status = 0;
  for (int e = i; e < E; e += B) {
    s_count[e] = 0;
    s_missing[e] = A.resident && e >= A.e_begin && e < A.e_begin + A.e_count && !A.resident[e - A.e_begin];
  }
  __syncthreads();
  griddep_wait();
  griddep_launch();
  const bool pair = i < A.n_pairs;
  int x = pair ? (int)A.router_out[2 * (size_t)i] : -1, r = -1;  // expert (-1: none, or not placed), row among the expert's
  if (x < 0 || x >= E) {
    if (pair) atomicOr(&s_status, kDevErrExpertRange);
    x = -1;
  } else if (A.only_expert >= 0 && x != A.only_expert) {
    x = -1;
  }
  if (x >= 0) r = atomicAdd(&s_count[x], 1);
  __syncthreads();
  const bool local = x >= A.e_begin && x < A.e_begin + A.e_count && x >= 0;
  const int count = x >= 0 ? s_count[x] : 0, height = even_tile_height(count, A.tile_rows, A.expert_tiles != nullptr);
  {
    // the experts whose first pair a lane has: the warp's lanes one after the other, the warps as they come
    const bool first = r == 0;
    const int nt = first && local ? (count + A.tile_rows - 1) / A.tile_rows : 0;
    const uint32_t mine = first ? (uint32_t)count << 16 | (uint32_t)nt : 0u;
    uint32_t upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += u;
    }
    uint32_t base = 0;
    if (lane == 31 && upto) base = atomicAdd(&s_next, upto);
    const uint32_t at = __shfl_sync(0xffffffffu, base, 31) + upto - mine;
    if (first) {
      const int row0 = (int)(at >> 16), tile0 = (int)(at & 0xffffu);
      s_row[x] = row0;
      s_tile[x] = tile0;
      atomicAdd(&s_distinct, 1);
      if (s_missing[x]) atomicOr(&s_status, kDevErrNotResident);
      if (nt) atomicMax(&s_tallest, min(height, count));
      for (int q = 0; q < nt && tile0 + q < A.max_tiles; ++q)
        A.tiles[tile0 + q] = RowTile{x - A.e_begin, row0 + q * height, min(height, count - q * height), 0};
    }
  }
  __syncthreads();
  const int rows = (int)(s_next >> 16), tiles = (int)(s_next & 0xffffu);
  const bool over = rows > A.max_rows || tiles > A.max_tiles;
  if (pair) {
    const bool placed = x >= 0 && !over;
    A.row_of_pair[i] = placed ? s_row[x] + r : -1;
    if (A.places) {
      int4 p = make_int4(0, 0, 0, -1);
      if (placed && local) {
        const int q = r / height;
        p = make_int4(s_tile[x] + q, s_row[x] + q * height, min(height, count - q * height), r - q * height);
      }
      A.places[i] = p;
    }
  }
  if (i == 0) {
    A.meta[0] = over ? 0 : tiles;
    A.meta[1] = rows;
    A.meta[2] = s_distinct;
    A.meta[3] = s_status | (over ? kDevErrCapacity : 0);
    A.meta[4] = s_tallest;
    A.meta[5] = A.meta[6] = 0;
  }
  for (int e = i; e < E; e += B) A.counts[e] = s_count[e];
  if (A.tile_words && !over)  // the block-scaled kernel's record masks: nothing marked yet
    for (int w = i; w < tiles * A.words_per_tile; w += B) A.tile_words[w] = 0;
}

// One block per token: its hidden row goes to the token's rows as fp16 (times the routing weight when it is applied before the
// expert).  The rows are given (cursor null) or claimed here, in the experts' segments.  The hidden states are older than the
// kernel before this one and are on their way while that ends; a row is read once and stored k times, 16 bytes a thread.
// Bound by HBM (4 H bytes in, 2 k H out): 4096 tokens x 4 slots x 2880 columns, 141 MB, 19.5 us (a warp per pair,
// eight bytes a lane: 38).
// V: what a store moves, uint4, or uint2 where the rows (a caller's, who sends them) lie at a multiple of 8 bytes only.
constexpr int kScatterThreads = 128, kScatterKept = 3;  // columns of a row in registers: 8 x 128 x 3
template <typename V>
__global__ void __launch_bounds__(kScatterThreads) k_scatter(const float* __restrict__ router_out, const float* __restrict__ hidden,
                                                             int k, int H, int E, int only_expert, const int* __restrict__ offsets,
                                                             int* __restrict__ cursor, int* __restrict__ row_of_pair,
                                                             __half* __restrict__ x16, int ldx, int max_rows, int weight_before_ffn) {
  __shared__ int s_pos[kMaxTopK];
  __shared__ float s_w[kMaxTopK];
  const int t = blockIdx.x;
  const float* src = hidden + (size_t)t * H;
  float4 v[kScatterKept][2];
#pragma unroll
  for (int i = 0; i < kScatterKept; ++i) {
    const int d = (threadIdx.x + i * kScatterThreads) * 8;
    if (d < H) {
      v[i][0] = __ldg(reinterpret_cast<const float4*>(src + d));
      v[i][1] = __ldg(reinterpret_cast<const float4*>(src + d + 4));
    }
  }
  griddep_wait();
  griddep_launch();
  if ((int)threadIdx.x < k) {
    const size_t i = (size_t)t * k + threadIdx.x;
    int pos = -1;
    if (!cursor) {
      pos = row_of_pair[i];
    } else {
      const int e = (int)router_out[2 * i];
      if (e >= 0 && e < E && (only_expert < 0 || e == only_expert)) {
        pos = offsets[e] + atomicAdd(&cursor[e], 1);
        if (pos >= max_rows) pos = -1;
      }
      row_of_pair[i] = pos;
    }
    s_pos[threadIdx.x] = pos;
    s_w[threadIdx.x] = weight_before_ffn ? router_out[2 * i + 1] : 1.0f;
  }
  __syncthreads();
  auto store = [&](int d, const float4& a, const float4& b) {
    for (int j = 0; j < k; ++j) {
      if (s_pos[j] < 0) continue;
      const float m = s_w[j];
      const __align__(16) __half2 h[4] = {__floats2half2_rn(a.x * m, a.y * m), __floats2half2_rn(a.z * m, a.w * m),
                                          __floats2half2_rn(b.x * m, b.y * m), __floats2half2_rn(b.z * m, b.w * m)};
#pragma unroll
      for (int i = 0; i < (int)(16 / sizeof(V)); ++i)
        reinterpret_cast<V*>(x16 + (size_t)s_pos[j] * ldx + d)[i] = reinterpret_cast<const V*>(h)[i];
    }
  };
#pragma unroll
  for (int i = 0; i < kScatterKept; ++i) {
    const int d = (threadIdx.x + i * kScatterThreads) * 8;
    if (d < H) store(d, v[i][0], v[i][1]);
  }
  for (int d = (threadIdx.x + kScatterKept * kScatterThreads) * 8; d < H; d += 8 * kScatterThreads)
    store(d, __ldg(reinterpret_cast<const float4*>(src + d)), __ldg(reinterpret_cast<const float4*>(src + d + 4)));
}

// The whole plan of a dense FFN (one expert, every token in order): rows to fp16, and by block 0 what k_scan leaves for
// one expert.  The down projection's rows are the tokens' then, so no combine follows.
__global__ void __launch_bounds__(256) k_dense_rows(const float* __restrict__ hidden, __half* __restrict__ x16, int ldx, int T, int H,
                                                    int tile_rows, const uint8_t* __restrict__ resident, int* __restrict__ counts,
                                                    int* __restrict__ offsets, RowTile* __restrict__ tiles, int* __restrict__ meta) {
  griddep_wait();
  griddep_launch();
  if (blockIdx.x == 0) {
    const int nt = (T + tile_rows - 1) / tile_rows;
    const int per = even_tile_height(T, tile_rows, false);
    for (int i = threadIdx.x; i < nt; i += blockDim.x) tiles[i] = RowTile{0, i * per, min(per, T - i * per), 0};
    if (threadIdx.x == 0) {
      counts[0] = offsets[1] = meta[1] = T;
      offsets[0] = 0;
      meta[0] = nt;
      meta[2] = 1;
      meta[3] = resident[0] ? 0 : kDevErrNotResident;
      meta[4] = min(per, T);
    }
  }
  const int per_row = H / 8;  // H is a multiple of 32, a row of x16 of 64
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)T * per_row; i += (size_t)gridDim.x * blockDim.x) {
    const int t = (int)(i / per_row), d = (int)(i % per_row) * 8;
    const float4 a = *reinterpret_cast<const float4*>(hidden + (size_t)t * H + d), b = *reinterpret_cast<const float4*>(hidden + (size_t)t * H + d + 4);
    const __half2 h[4] = {__floats2half2_rn(a.x, a.y), __floats2half2_rn(a.z, a.w), __floats2half2_rn(b.x, b.y), __floats2half2_rn(b.z, b.w)};
    *reinterpret_cast<uint4*>(x16 + (size_t)t * ldx + d) = *reinterpret_cast<const uint4*>(h);
  }
}

// ---------------------------------------------------------------------------
// Weighted combine (expert_merge_node::compute, expert_merge_node.h:88-131):
// out[t] = sum over slots j = 0..k-1, in that order, of w[t,j] * y[row(t,j)],
// a separate multiply and add per term as the reference does.  mode 1 is the
// dense single-expert output of expert_mlp_node (expert_mlp_node.h:503-529):
// the token's row unweighted, or zeros.
// ---------------------------------------------------------------------------
//
// Bound by HBM (k rows of y in, one out).  AT_ONCE slots' rows are requested at once: one at a time a
// step of 8192 tokens took 2046 us, with four 2011; 2048 tokens of eight slots 318 and 306.
// Few tokens (FEW) are bound by the latency of their loads: up to eight slots' rows are requested at once, and the shared expert's and the
// residual row with them (16 tokens of eight slots, a step: four at once and those two rows after them 64.0 us, now 62.5); of fewer than four an
// SM a row is dealt to several blocks (gridDim.y), so that a thread has one round of loads (8 tokens of 2880 columns 7.9 -> 4.5 us, profiler).
// Many tokens need blocks on an SM more than loads of a block: eight of them, with 32 registers a thread (profiler, cold caches; in
// brackets with the few tokens' form, whose registers leave room for six or four): 8192 tokens, four slots of 512 columns 16.5 us (18.5); 4096, two
// of 1024 11.2 (12.5); 2048, one of 2048 8.5 (9.7); 2048, eight of 2048 23.9 (25.1).  Their barrier stands behind the wait, where the next kernel has been let in already (in front, with the
// test for page-locked results: 16 experts of 2048 x 2048, top-1, 2048 tokens 92.8 -> 98.5 for the step, 64 of 1024 x 512, top-2, 77.6 -> 80.3).
// The rows are read for the last time, so they are the first to leave L2 (a step of 2048 tokens of eight slots 244.5 -> 240.6, of 4096
// of four level; this kernel alone, 4096 tokens, eight slots of 2048 columns 57 -> 47, 8192 tokens, four of 2880 82 -> 76).
//
// carry (optional; the host entry point that runs a batch in several passes): block 0 folds this
// pass's status word into a sticky one and adds its per-expert row counts to running totals --
// layout: carry[0] = sticky status, carry[1 .. E] = rows per expert.
//
// host_router, host_meta (optional, FEW only): page-locked memory that the routing and the 16 words of `meta` go to beside the results, which
// `out` may be in then, too.
template <int AT_ONCE, bool FEW>
__global__ void __launch_bounds__(256, !FEW ? 8 : AT_ONCE > 4 ? 4 : 6) k_combine(const float* __restrict__ router_out, const int* __restrict__ row_of_pair,
                          const float* __restrict__ y, int ldy, float* __restrict__ out, int T,
                          int k, int H, int unweighted, int dense_single,
                          const int* __restrict__ meta, const int* __restrict__ counts, int* __restrict__ carry, int E,
                          const float* residual, const float* shared_out, float* host_router, int* host_meta) {
  __shared__ int s_row[kMaxTopK];
  __shared__ float s_w[kMaxTopK];
  const int t = blockIdx.x;
  // (the routing and the rows' places are older than the kernel in front)
  if (t < T && (int)threadIdx.x < k) {
    s_row[threadIdx.x] = row_of_pair[(size_t)t * k + threadIdx.x];
    s_w[threadIdx.x] = unweighted ? 1.f : router_out[((size_t)t * k + threadIdx.x) * 2 + 1];  // 1 * v is v
  }
  if (FEW) __syncthreads();
  griddep_wait();
  griddep_launch();
  if (carry && t == 0 && blockIdx.y == 0) {
    if (threadIdx.x == 0 && meta[3]) atomicOr(&carry[0], meta[3]);
    for (int e = threadIdx.x; e < E; e += blockDim.x) carry[1 + e] += counts[e];
  }
  if (t >= T) return;
  if (!FEW) __syncthreads();
  if (FEW && blockIdx.y == 0) {
    if (host_router && (int)threadIdx.x < 2 * k) host_router[(size_t)t * k * 2 + threadIdx.x] = router_out[(size_t)t * k * 2 + threadIdx.x];
    if (host_meta && t == 0 && threadIdx.x < 16) host_meta[threadIdx.x] = meta[threadIdx.x];
  }
  for (int d = (blockIdx.y * blockDim.x + threadIdx.x) * 4; d < H; d += gridDim.y * blockDim.x * 4) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    // (FEW: on their way with the rows)
    float4 sh, r;
    if (FEW && shared_out) sh = *reinterpret_cast<const float4*>(shared_out + (size_t)t * H + d);
    if (FEW && residual) r = *reinterpret_cast<const float4*>(residual + (size_t)t * H + d);
    bool done = false;
    for (int j0 = 0; j0 < k && !done; j0 += AT_ONCE) {
      float4 v[AT_ONCE];
#pragma unroll
      for (int j = 0; j < AT_ONCE; ++j)
        if (j0 + j < k && s_row[j0 + j] >= 0) v[j] = __ldcs(reinterpret_cast<const float4*>(y + (size_t)s_row[j0 + j] * ldy + d));
#pragma unroll
      for (int j = 0; j < AT_ONCE; ++j) {
        if (j0 + j >= k || s_row[j0 + j] < 0 || done) continue;
        if (dense_single) {
          acc = v[j];
          done = true;
        } else {
          const float w = s_w[j0 + j];
          acc.x = __fadd_rn(acc.x, __fmul_rn(w, v[j].x));
          acc.y = __fadd_rn(acc.y, __fmul_rn(w, v[j].y));
          acc.z = __fadd_rn(acc.z, __fmul_rn(w, v[j].z));
          acc.w = __fadd_rn(acc.w, __fmul_rn(w, v[j].w));
        }
      }
    }
    if (shared_out) {
      if (!FEW) sh = *reinterpret_cast<const float4*>(shared_out + (size_t)t * H + d);
      // the shared expert's dense FFN on the same rows: add(merge output, shared output), llm_engine.cpp:766-769
      acc.x = __fadd_rn(acc.x, sh.x);
      acc.y = __fadd_rn(acc.y, sh.y);
      acc.z = __fadd_rn(acc.z, sh.z);
      acc.w = __fadd_rn(acc.w, sh.w);
    }
    if (residual) {
      if (!FEW) r = *reinterpret_cast<const float4*>(residual + (size_t)t * H + d);
      // the residual connection around the layer: add(residual, merge output), llm_engine.cpp:773-777
      acc.x = __fadd_rn(r.x, acc.x);
      acc.y = __fadd_rn(r.y, acc.y);
      acc.z = __fadd_rn(r.z, acc.z);
      acc.w = __fadd_rn(r.w, acc.w);
    }
    *reinterpret_cast<float4*>(out + (size_t)t * H + d) = acc;
  }
}

// ---------------------------------------------------------------------------
// RMSNorm in front of the router (rmsnorm_node::compute_impl, rmsnorm_node.h:60-82):
// out = (x / sqrt(sum(x^2) / H + eps)) * w.  The router's expert indices must equal the
// reference's bit for bit, so its INPUT must too: the sum of squares is the reference's
// sequential fp32 chain of separate multiplies and adds, division, square root and products are the
// IEEE round-to-nearest operations the reference's scalar code performs.
//
// A block per token: all its threads square the row into shared memory, one walks the squares, 32 columns of them in registers
// ahead, all of them scale the row.  Bound by that chain, 4.3 cycles a column.
//
// A few tokens: 256 threads, which keep the row and its weights in registers (the rest of a row of more than 4096 columns is
// read again); 8 tokens x 2880 columns 14.1 -> 10.2 us (profiler, cold caches; 16 columns ahead and the row read twice before).  An SM
// holds three such blocks, and of many tokens the other chains wait: then 128 threads that read the row twice, twelve blocks.
// The line is where a fourth block an SM would have to wait, and a little beyond.  256 / 128 threads, what the norm adds to a step, us: 2880
// columns, 333 tokens 16.4 / 18.8, 444 16.1 / 18.0, 480 22.4 / 17.7, 1200 39 / 29, 2048 52 / 35, 8192 183 / 110; 512, 444 4.8 / 5.1, 480 7.1 / 6.1, 8192
// 43 / 18; 4096, 444 19.1 / 24.3, 480 31.9 / 24.2, 8192 250 / 143; 8192, 333 47.5 / 44.9, 8192 507 / 348.
// ---------------------------------------------------------------------------
constexpr int kNormThreadsFew = 256, kNormKeptFew = 4, kNormThreadsMany = 128;
inline bool norm_few(int64_t T, int sm_count) { return 5 * T <= 16 * (int64_t)sm_count; }
template <int N>
__device__ __forceinline__ float add_columns(float s, uint32_t at) {
  constexpr int G = N / 4, A = 8;
  float4 v[A];
#pragma unroll
  for (int g = 0; g < A; ++g) v[g] = lds128(at + 16 * g);
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const float4 u = v[g % A];
    if (g + A < G) v[g % A] = lds128(at + 16 * (g + A));
    s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, u.x), u.y), u.z), u.w);
  }
  return s;
}
// THREADS of a block, of whose columns KEPT runs of four are in registers
template <int THREADS, int KEPT>
__global__ void __launch_bounds__(THREADS) k_rmsnorm(const float* __restrict__ x, const float* __restrict__ w, float eps,
                                                     float* __restrict__ out, int T, int H) {
  extern __shared__ __align__(16) float rms_sq[];
  __shared__ float s_rms;
  float4 g[KEPT + 1];
#pragma unroll
  for (int i = 0; i < KEPT; ++i) {
    const int d = (threadIdx.x + i * THREADS) * 4;
    if (d < H) g[i] = __ldg(reinterpret_cast<const float4*>(w + d));
  }
  griddep_wait();
  griddep_launch();
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    const float* src = x + (size_t)t * H;
    auto square = [&](int d, const float4& v) {
      *reinterpret_cast<float4*>(rms_sq + d) = make_float4(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y), __fmul_rn(v.z, v.z), __fmul_rn(v.w, v.w));
    };
    auto scale = [&](int d, const float4& v, const float4& f, float rms) {
      *reinterpret_cast<float4*>(out + (size_t)t * H + d) =
          make_float4(__fmul_rn(__fdiv_rn(v.x, rms), f.x), __fmul_rn(__fdiv_rn(v.y, rms), f.y), __fmul_rn(__fdiv_rn(v.z, rms), f.z),
                      __fmul_rn(__fdiv_rn(v.w, rms), f.w));
    };
    float4 kept[KEPT + 1];
#pragma unroll
    for (int i = 0; i < KEPT; ++i) {
      const int d = (threadIdx.x + i * THREADS) * 4;
      if (d < H) kept[i] = __ldg(reinterpret_cast<const float4*>(src + d));
    }
#pragma unroll
    for (int i = 0; i < KEPT; ++i) {
      const int d = (threadIdx.x + i * THREADS) * 4;
      if (d < H) square(d, kept[i]);
    }
    for (int d = (threadIdx.x + KEPT * THREADS) * 4; d < H; d += 4 * THREADS) square(d, __ldg(reinterpret_cast<const float4*>(src + d)));
    __syncthreads();
    if (threadIdx.x == 0) {
      const uint32_t at = smem_u32(rms_sq);
      float s = 0.f;
      int d = 0;
#pragma unroll 1
      for (; d + 192 <= H; d += 192) s = add_columns<192>(s, at + 4 * d);
#pragma unroll 1
      for (; d < H; d += 32) s = add_columns<32>(s, at + 4 * d);  // H is a multiple of 32
      s_rms = __fsqrt_rn(__fadd_rn(__fdiv_rn(s, (float)H), eps));
    }
    __syncthreads();
    const float rms = s_rms;
#pragma unroll
    for (int i = 0; i < KEPT; ++i) {
      const int d = (threadIdx.x + i * THREADS) * 4;
      if (d < H) scale(d, kept[i], g[i], rms);
    }
    for (int d = (threadIdx.x + KEPT * THREADS) * 4; d < H; d += 4 * THREADS)
      scale(d, __ldg(reinterpret_cast<const float4*>(src + d)), __ldg(reinterpret_cast<const float4*>(w + d)), rms);
    __syncthreads();  // s_rms and the squares are rewritten for the block's next token
  }
}

// Router output with logical expert ids replaced by the slots their rows are grouped
// under: the primary slot, or for odd-numbered tokens the slot of the expert's second copy.
__global__ void k_ep_slots(const float* __restrict__ router, float* __restrict__ out, int n_pairs, int k, int E_logical,
                           const int* __restrict__ primary, const int* __restrict__ replica) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_pairs; i += gridDim.x * blockDim.x) {
    const float ef = router[2 * i];
    const int e = (int)ef;
    const int t = i / k;
    float o = -1.f;  // an id the permutation reports as out of range
    if (e >= 0 && e < E_logical) {
      const int r = replica[e];
      o = (float)((r >= 0 && (t & 1)) ? r : primary[e]);
    }
    out[2 * i] = o;
    out[2 * i + 1] = router[2 * i + 1];
  }
}

// ---------------------------------------------------------------------------
// Expert-parallel receive side.  Rows arrive as n_src segments (one per source
// device), each ordered by local expert; the contractions want them grouped by
// expert.  seg layout (int32): [0..1024] exclusive offsets of the (src, expert)
// segments in arrival order, [1025..2048] rows of the same expert that arrive
// from lower-numbered sources.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024)
k_ep_plan(const int* __restrict__ recv_counts, int n_src, int e_count, int e_begin,
          int* __restrict__ counts, int* __restrict__ seg) {
  __shared__ int s_warp[32];
  const int i = threadIdx.x, lane = i & 31, warp = i >> 5;
  const int n_seg = n_src * e_count;
  const int c = i < n_seg ? recv_counts[i] : 0;
  int r = c;
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, r, o);
    if (lane >= o) r += a;
  }
  if (lane == 31) s_warp[warp] = r;
  __syncthreads();
  if (warp == 0) {
    int a = s_warp[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, a, o);
      if (lane >= o) a += u;
    }
    s_warp[lane] = a;
  }
  __syncthreads();
  const int base = warp ? s_warp[warp - 1] : 0;
  seg[i] = base + r - c;
  if (i == 0) seg[1024] = s_warp[31];
  if (i < n_seg) {
    const int src = i / e_count, e = i % e_count;
    int before = 0;
    for (int s2 = 0; s2 < src; ++s2) before += recv_counts[s2 * e_count + e];
    seg[1025 + i] = before;
    if (src == 0) {
      int tot = 0;
      for (int s2 = 0; s2 < n_src; ++s2) tot += recv_counts[s2 * e_count + e];
      counts[e_begin + e] = tot;
    }
  }
}

// Blocks (x = segment, y = row slice): copy the segment's rows to their
// expert-major place and remember where each came from.  A row is ldx/8 16-byte
// words, so every thread has only a couple of independent loads per row and
// many rows are in flight across the y dimension.
__global__ void k_ep_regroup(const __half* __restrict__ recv, __half* __restrict__ x16, int ldx,
                             const int* __restrict__ seg, const int* __restrict__ offsets, int n_src,
                             int e_count, int e_begin, int* __restrict__ out_row_map) {
  const int b = blockIdx.x;
  const int e = b % e_count;
  const int src_row0 = seg[b], n = seg[b + 1] - seg[b];
  const int dst_row0 = offsets[e_begin + e] + seg[1025 + b];
  const int w16 = ldx / 8;
  for (int r = blockIdx.y; r < n; r += gridDim.y) {
    const uint4* s = reinterpret_cast<const uint4*>(recv + (size_t)(src_row0 + r) * ldx);
    uint4* d = reinterpret_cast<uint4*>(x16 + (size_t)(dst_row0 + r) * ldx);
    for (int i = threadIdx.x; i < w16; i += blockDim.x) d[i] = s[i];
    if (threadIdx.x == 0) out_row_map[dst_row0 + r] = src_row0 + r;
  }
}

// Stream path only: rows computed in expert-major order go back to arrival order.
__global__ void k_ep_ungroup(const float* __restrict__ y, float* __restrict__ ret, int H,
                             const int* __restrict__ out_row_map, int rows) {
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < rows; r += gridDim.x * wpb) {
    const float4* s = reinterpret_cast<const float4*>(y + (size_t)r * H);
    float4* d = reinterpret_cast<float4*>(ret + (size_t)out_row_map[r] * H);
    for (int i = lane; i < H / 4; i += 32) d[i] = s[i];
  }
}

// ---------------------------------------------------------------------------
// Expert parallelism over peer memory (NVLink): the dispatch writes every row
// straight into the row buffer of the rank that owns its expert slot, at its
// final expert-grouped position, and the down projection's epilogue writes
// every output row straight into the return buffer of the rank that owns the
// token.  The only collectives left are the (tiny) exchange of row counts and
// two barriers.  All cross-GPU traffic is plain stores to peer pointers.
//
// Layout of a destination's row buffer: slot-major, within a slot the rows of
// source rank 0, then 1, ...  Every rank derives all positions from the full
// count table all_counts[source][slot].
// ---------------------------------------------------------------------------
struct RowOrigin {
  int src;   // rank that sent the row
  int pair;  // index of the (token, k) pair there = row of its return buffer
};

// One block of 1024 threads, E <= 1024.  base[e] = first row, in the buffer of the
// rank owning slot e, of the rows THIS rank sends to e; cursor[e] = 0.
__global__ void __launch_bounds__(1024)
k_ep_p2p_base(const int* __restrict__ all_counts, int world, int me, int E, int e_per_rank, int max_rows,
              int* __restrict__ base, int* __restrict__ cursor, int* __restrict__ meta) {
  __shared__ int s_scan[1024];
  __shared__ int s_warp[32];
  const int e = threadIdx.x, lane = e & 31, warp = e >> 5;
  int tot = 0, before = 0;
  if (e < E)
    for (int s = 0; s < world; ++s) {
      const int c = all_counts[s * E + e];
      tot += c;
      if (s < me) before += c;
    }
  int r = tot;
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, r, o);
    if (lane >= o) r += a;
  }
  if (lane == 31) s_warp[warp] = r;
  __syncthreads();
  if (warp == 0) {
    int a = s_warp[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, a, o);
      if (lane >= o) a += u;
    }
    s_warp[lane] = a;
  }
  __syncthreads();
  s_scan[e] = (warp ? s_warp[warp - 1] : 0) + r - tot;  // exclusive prefix over all slots
  __syncthreads();
  if (e < E) {
    const int first = (e / e_per_rank) * e_per_rank;  // first slot of the owning rank
    const int in_rank = s_scan[e] - s_scan[first];    // rows of that rank's earlier slots
    base[e] = in_rank + before;
    cursor[e] = 0;
    if (in_rank + tot > max_rows) atomicOr(&meta[3], kDevErrCapacity);
  }
}

// One warp per (token, slot) pair: claim the next row of this rank's share of the slot on
// the owning rank, write the token's hidden row there as fp16 (peer store) with its origin.
__global__ void k_ep_p2p_scatter(const float* __restrict__ router_out, const float* __restrict__ hidden,
                                 int n_pairs, int k, int H, int E, int e_per_rank, int me,
                                 const int* __restrict__ base, int* __restrict__ cursor,
                                 __half* const* __restrict__ peer_x16, RowOrigin* const* __restrict__ peer_info,
                                 int ldx, int max_rows, int weight_before_ffn, int* __restrict__ row_of_pair,
                                 int* __restrict__ meta) {
  const int lane = threadIdx.x & 31;
  const int warps_per_block = blockDim.x >> 5;
  for (int i = blockIdx.x * warps_per_block + (threadIdx.x >> 5); i < n_pairs; i += gridDim.x * warps_per_block) {
    const int e = (int)router_out[2 * (size_t)i];
    const float w = router_out[2 * (size_t)i + 1];
    int pos = -1;
    if (e >= 0 && e < E) {
      if (lane == 0) pos = base[e] + atomicAdd(&cursor[e], 1);
      pos = __shfl_sync(0xffffffffu, pos, 0);
      if (pos >= max_rows) pos = -1;
    } else if (lane == 0) {
      atomicOr(&meta[3], kDevErrExpertRange);
    }
    if (lane == 0) row_of_pair[i] = pos < 0 ? -1 : i;  // the return buffer is indexed by pair
    if (pos < 0) continue;
    const int dst_rank = e / e_per_rank;
    const float* src = hidden + (size_t)(i / k) * H;
    __half* dst = peer_x16[dst_rank] + (size_t)pos * ldx;
    if (lane == 0) peer_info[dst_rank][pos] = RowOrigin{me, i};
    const float mul = weight_before_ffn ? w : 1.0f;
    for (int d = lane * 8; d < H; d += 256) {
      const float4 v0 = *reinterpret_cast<const float4*>(src + d);
      const float4 v1 = *reinterpret_cast<const float4*>(src + d + 4);
      __half2 a = __floats2half2_rn(v0.x * mul, v0.y * mul), b = __floats2half2_rn(v0.z * mul, v0.w * mul);
      __half2 c = __floats2half2_rn(v1.x * mul, v1.y * mul), f = __floats2half2_rn(v1.z * mul, v1.w * mul);
      uint4 o;
      o.x = *reinterpret_cast<uint32_t*>(&a);
      o.y = *reinterpret_cast<uint32_t*>(&b);
      o.z = *reinterpret_cast<uint32_t*>(&c);
      o.w = *reinterpret_cast<uint32_t*>(&f);
      *reinterpret_cast<uint4*>(dst + d) = o;
    }
  }
  __threadfence_system();  // the peer stores before whatever signals their arrival
}

// counts[e] of the slots this rank owns = rows it received (all sources); zero elsewhere.
__global__ void k_ep_p2p_local_counts(const int* __restrict__ all_counts, int world, int E, int e_begin, int e_count,
                                      int* __restrict__ counts) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= E) return;
  int tot = 0;
  if (e >= e_begin && e < e_begin + e_count)
    for (int s = 0; s < world; ++s) tot += all_counts[s * E + e];
  counts[e] = tot;
}

// Where each received row's output goes: the pair's row of the sender's return buffer.
// Nothing is derived when the row plan overran the buffers (the expert kernels then have no
// tiles either), and a row whose origin record is not a valid (rank, pair) gets a null
// pointer, which every consumer skips, plus kDevErrPeerRow in the status word.
__global__ void k_ep_p2p_rowptr(const RowOrigin* __restrict__ info, int* __restrict__ meta,
                                float* const* __restrict__ peer_back, int H, float** __restrict__ row_ptr, int max_rows,
                                int world, int max_pairs) {
  if (meta[3] & kDevErrCapacity) return;
  const int rows = min(meta[1], max_rows);
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
    const RowOrigin o = info[r];
    const bool ok = o.src >= 0 && o.src < world && o.pair >= 0 && o.pair < max_pairs;
    row_ptr[r] = ok ? peer_back[o.src] + (size_t)o.pair * H : nullptr;
    if (!ok) atomicOr(&meta[3], kDevErrPeerRow);
  }
}

// Output rows computed into a local buffer (streaming path) -> their owners' return buffers.
__global__ void k_ep_p2p_return(const float* __restrict__ y, int H, float* const* __restrict__ row_ptr,
                                const int* __restrict__ meta, int max_rows) {
  if (meta[3] & kDevErrCapacity) return;
  const int rows = min(meta[1], max_rows);
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < rows; r += gridDim.x * wpb) {
    const float4* s = reinterpret_cast<const float4*>(y + (size_t)r * H);
    float4* d = reinterpret_cast<float4*>(row_ptr[r]);
    if (!d) continue;
    for (int i = lane; i < H / 4; i += 32) d[i] = s[i];
  }
  __threadfence_system();
}

// ---------------------------------------------------------------------------
// Barrier (and, with a payload, the exchange of the per-slot row counts) between the ranks of
// the peer-memory step, without a collective library: every rank owns a small sync area at
// the tail of its return buffer, which all peers can write --
//   flags[3][64]         flags[b][r] = last epoch of barrier b that rank r has reached
//   all_counts[64][E]    all_counts[r][.] = rank r's row counts of this step
// A rank stores its payload into every peer's area, fences (system scope), stores the epoch
// into its flag on every peer, then waits until all of its own flags show the epoch.  Flags only
// grow, nothing is reset.  The wait is bounded (clock budget); when it runs out the kernel sets
// kDevErrWaitTimeout and returns.  One block; ranks run on different GPUs, so no rank's wait
// depends on a kernel queued behind it on the same device.
// ---------------------------------------------------------------------------
constexpr int kEpMaxWorld = 64;
__host__ __device__ inline size_t ep_sync_ints(int E) { return (size_t)3 * kEpMaxWorld + (size_t)kEpMaxWorld * E; }

__global__ void __launch_bounds__(1024)
k_ep_p2p_sync(float* const* __restrict__ peer_back, size_t tail_floats, int me, int world, int which,
              int* __restrict__ epochs, const int* __restrict__ my_counts, int E, int* __restrict__ all_counts_out,
              int* __restrict__ meta) {
  __shared__ int s_timeout, s_epoch;
  const int tid = threadIdx.x;
  // The barrier's generation lives on the device and every launch advances its own rank's copy: all
  // ranks launch the same sequence, so their copies agree, and a captured launch sequence can be
  // replayed (a generation passed from the host would be frozen into the graph).
  if (tid == 0) {
    s_timeout = 0;
    s_epoch = ++epochs[which];
  }
  __syncthreads();
  const int epoch = s_epoch;
  if (my_counts) {
    for (int idx = tid; idx < world * E; idx += blockDim.x) {
      const int r = idx / E, e = idx % E;
      int* tail = reinterpret_cast<int*>(peer_back[r] + tail_floats);
      tail[3 * kEpMaxWorld + (size_t)me * E + e] = my_counts[e];
    }
  }
  __threadfence_system();
  __syncthreads();
  if (tid < world) {
    volatile int* theirs = reinterpret_cast<volatile int*>(peer_back[tid] + tail_floats);
    theirs[which * kEpMaxWorld + me] = epoch;
    volatile int* mine = reinterpret_cast<volatile int*>(peer_back[me] + tail_floats);
    const long long t0 = clock64();
    while (mine[which * kEpMaxWorld + tid] < epoch) {
      if (clock64() - t0 > 4 * wait_budget()) {
        s_timeout = 1;
        break;
      }
    }
  }
  __threadfence_system();
  __syncthreads();
  if (s_timeout) {
    if (tid == 0) atomicOr(&meta[8], kDevErrWaitTimeout);  // the sticky word: later stages do not clear it
    return;
  }
  if (all_counts_out) {
    const volatile int* mine = reinterpret_cast<const volatile int*>(peer_back[me] + tail_floats);
    for (int idx = tid; idx < world * E; idx += blockDim.x) all_counts_out[idx] = mine[3 * kEpMaxWorld + idx];
  }
}

}  // namespace csk
