// Shared definitions of the MoE library: code conversion, activations, barriers, launches and work lists.
// sm_100a only.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "csk_moe.h"

namespace csk {

constexpr int kTileK = 64;  // columns of K per step of the fp16 tensor-core kernels

inline int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Two packed E2M1 codes (one byte) -> half2, low nibble in the low half.
__device__ __forceinline__ uint32_t e2m1x2_to_h2(uint32_t byte) {
  uint32_t r;
  asm("{\n\t.reg .b8 b;\n\tcvt.u8.u32 b, %1;\n\tcvt.rn.f16x2.e2m1x2 %0, b;\n\t}" : "=r"(r) : "r"(byte));
  return r;
}

// A word of eight codes -> four half2 (columns 0-1, 2-3, 4-5, 6-7).
__device__ __forceinline__ void dequant_word(uint32_t w, uint32_t (&h)[4]) {
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
      "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
      "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
      : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
      : "r"(w));
}

// x limited to [-lim, lim]; a NaN stays one, as the reference's comparisons leave it (fminf and fmaxf would make it a limit,
// and a row that holds an infinity or a NaN would come out finite).
__device__ __forceinline__ float limit_keep_nan(float x, float lim) {
  float r;
  asm("{\n\t.reg .f32 t;\n\tmax.NaN.f32 t, %1, %2;\n\tmin.NaN.f32 %0, t, %3;\n\t}" : "=f"(r) : "f"(x), "f"(-lim), "f"(lim));
  return r;
}

// The same activations with the hardware's approximate exp2 and reciprocal (one MUFU
// operation each, relative error around 2^-22, far below the fp16 rounding of the stored
// result).  Used in the tensor-core kernel's epilogue, which sits on the critical path.
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float gated_act_fast(float gate, float up, int act) {
  constexpr float kLog2e = 1.4426950408889634f;
  if (act == CSK_ACT_MODIFIED_SWIGLU) {
    const float lim = 7.0f, alpha = 1.702f;
    const float g = fminf(gate, lim);
    const float u = limit_keep_nan(up, lim);
    return g * rcp_approx(1.0f + ex2_approx(-alpha * kLog2e * g)) * (u + 1.0f);
  }
  return gate * rcp_approx(1.0f + ex2_approx(-kLog2e * gate)) * up;
}

// Gated activations of the reference (expert_mlp_node.h:657-658, 699-707).
__device__ __forceinline__ float gated_act(float gate, float up, int act) {
  if (act == CSK_ACT_MODIFIED_SWIGLU) {
    const float lim = 7.0f, alpha = 1.702f;
    float g = fminf(gate, lim);
    float u = limit_keep_nan(up, lim);
    float glu = g / (1.0f + expf(alpha * (-g)));
    return glu * (u + 1.0f);
  }
  float silu = gate / (1.0f + expf(-gate));
  return silu * up;
}

// ---- mbarrier and bulk-copy helpers shared by the two expert kernels -----------
// Clock cycles before a bounded wait gives up (about one second at full clock).  A device
// variable rather than a constant so that a test can shorten it and watch a wait run out
// without hanging anything (csk_moe_debug_set, key 0).  Read only on the slow path of a wait.
__device__ long long g_wait_budget = 2000000000LL;
__device__ __forceinline__ long long wait_budget() { return *(volatile long long*)&g_wait_budget; }
// Waits for copies or MMAs that are already in flight (teardown after a wait ran out) keep a
// floor of a few milliseconds however short the budget was made: what is in flight must land.
__device__ __forceinline__ long long drain_budget() { return wait_budget() + 8000000LL; }

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// CLUSTER: threads of the other CTA of a cluster arrive on this barrier, too (without a qualifier the wait acquires from its own CTA
// only; no dearer in k_tile2: 8192 tokens of the 128-expert layer 1.58 ms either way)
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  if (CLUSTER)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  return ok != 0;
}
// Has the phase completed?  (Never suspends the thread.)
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait.  Returns false (and raises the CTA's abort flag) when the clock budget ran out or another role already aborted.  All but
// the first test is in one function that every wait of a kernel shares: kernels of many roles and waits have the less code to fetch
// (k_tile2 on 2048 tokens of the 128-expert 2048 x 768 layer 97 -> 93 us, k_mx on 16 tokens of it 81 -> 79 for the step).
template <bool CLUSTER = false>
static __device__ __noinline__ bool mbar_wait_more(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  const long long t0 = clock64();
#pragma unroll 1
  for (;;) {
    if (*abort_flag) return false;
#pragma unroll 1
    for (int i = 0; i < 32; ++i)
      if (mbar_try<CLUSTER>(bar, parity)) return true;
    if (clock64() - t0 > wait_budget()) {
      *abort_flag = 1;
      return false;
    }
  }
}
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return mbar_try<CLUSTER>(bar, parity) || mbar_wait_more<CLUSTER>(bar, parity, abort_flag);
}
// The same for a whole warp that goes on to warp-wide instructions: its lanes agree on whether the wait ran out (each lane
// reads the clock and the flag for itself).
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of `local_addr` (a shared::cta address of this CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
  return r;
}

// Programmatic dependent launch: a kernel launched with `pdl` may become resident while
// the kernel before it in the stream is still running.  Every kernel of the layer therefore
// calls griddep_wait() before it touches global memory that an earlier kernel may still be
// writing or reading (a no-op for an ordinary launch), and griddep_launch() to let its own
// successor start early.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Bulk and tensor copies read global memory through the async proxy.  A kernel that is already running when its predecessor ends has
// no kernel boundary in front of what that wrote with ordinary stores: the threads that issue such copies of it call this after
// griddep_wait().
__device__ __forceinline__ void fence_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_k(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, bool pdl,
                            A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, P(std::forward<A>(args))...);
}

// Work item lists built on the device by the permutation step.
struct RowTile {
  int expert;  // expert index local to this device
  int row0;    // first row of the tile in the grouped activation buffer
  int rows;    // rows in the tile (1 .. tile height)
  int pad;
};

// Where an expert's rows are among the row tiles: its first tile and the height of its tiles (the last may be shorter).
struct ExpertTiles {
  int tile0, height;
};

// Device-side status word values (or-ed).
enum : int {
  kDevErrExpertRange = 1,   // router output names an expert outside [0, E)
  kDevErrCapacity = 2,      // more rows than the scratch buffers hold
  kDevErrWaitTimeout = 4,   // a bounded wait in a kernel ran out
  kDevErrNotResident = 8,   // rows were routed to an expert that is not loaded
  kDevErrPeerRow = 16,      // a row received from a peer carries no valid origin record
};

}  // namespace csk
