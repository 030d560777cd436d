// Grouped contraction over fp16 weights for FEW token rows (the dense FFN and fp16 experts in decode), written for sm_100a.
//
// Every weight is read once and meets at most 64 token rows, so its bytes count.  k_pair16 gives a CTA pair 256 weight rows and all of
// K, which leaves most SMs without work (a 2880 x 2880 matrix is 23 items) and each of the others with one stream.  Here a block
// of eight warps has 16 weight rows (gate/up: 16 gate and the same features' 16 up rows); its warps take the k-tiles in turn
// and their sums are added in warp order at the end, so a matrix is some hundred blocks that are all resident at once.
//
// Weights go from global memory straight to the operand registers of mma.sync (m16n8k16: at these rates the legacy tensor path
// is far from its limit): within a k-tile the order of the columns is free as long as both operands agree on it, so a
// thread's 16-byte piece of a weight row is its part of two MMAs, and the same piece of a token row is the other operand's.
// Two k-tiles of weights are in flight per warp (8 KB for gate/up); the first are asked for before griddepcontrol.wait.
//
// What bounds it: the bytes in flight.  Five of 16 experts of 2048 x 2048: gate/up reads its 84 MB in 23.8 us, down 42 MB in 15.7 (3.5
// and 2.7 TB/s, 44 and 33 % of the DRAM peak, cold caches); sixteen warps an SM, and 640 blocks are 2.2 rounds whose starts
// and ends nothing covers.
#pragma once

#include "csk_tile.cuh"

namespace csk {

constexpr int kFewWarps = 8;
constexpr int kFewMaxRows = 32;        // tokens of a batch: the layer holds one expert ...
constexpr int kFewMaxRowsWave = 64;    // ... of which all blocks are resident at once, one an SM ...
constexpr int kFewMaxRowsRouted = 16;  // ... or several experts

inline size_t few_smem_bytes(int groups, bool gated) { return (size_t)kFewWarps * 32 * 4 * groups * (gated ? 2 : 1) * sizeof(float); }

__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct FewArgs {
  TileArgs t;
  const __half* x;  // grouped rows [rows, ldx]
  int ldx;
  int one_expert;   // the layer holds a single expert: the tile list may be one launch old
};

// NT = groups of eight token rows.  blockIdx.x: 16 weight rows (features), blockIdx.y: row tile.  TURNS: the tile may have more
// than 8 NT rows, which are taken 8 NT after another (the loop's registers cost the others up to 5 %: 128 experts of 2048 x 768, 16
// tokens of eight slots 224 -> 236 us).
// Two blocks an SM up to 32 rows (in 128 registers; three blocks of 80 were slower, 62 -> 70 us for a block of 5 tokens).
template <bool GATED, int NT, bool TURNS>
__global__ void __launch_bounds__(kFewWarps * 32, NT <= 4 ? 2 : 1) k_few16(const FewArgs F) {
  extern __shared__ float few_sums[];
  const TileArgs& A = F.t;
  const TileLayout& L = A.L;
  constexpr int M = GATED ? 2 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int n0 = blockIdx.x * 16;
  // (the tile list is two launches old, unless there is one expert only)
  const int expert = !F.one_expert && (int)blockIdx.y < *A.n_tiles_ptr ? A.tiles[blockIdx.y].expert : 0;
  const uint8_t* ebase = A.weights + (size_t)expert * A.expert_stride;
  // row g of the block's 16 in the tile layout (gate/up: the up rows 16 rows behind), its pieces stored at piece ^ (row & 7)
  constexpr int kUp = 16 * 128;
  const int nt = n0 / L.feats_per_tile(), half = L.half_of(n0), r0 = L.row_of(n0 % L.feats_per_tile(), 0);
  const uint8_t* wt = ebase + A.mat_offset + (size_t)nt * L.k_tiles * kTile16 + (size_t)half * kHalf16 + (size_t)(r0 + g) * 128;
  const int p0 = (q ^ g) << 4, p1 = ((q + 4) ^ g) << 4;  // (row & 7 = g for rows g and g + 8)
  uint4 w[2][M][2][2];  // [buffer][matrix][row g, g + 8][piece q, q + 4]
  auto load_w = [&](int kt, uint4 (&d)[M][2][2]) {
    const uint8_t* base = wt + (size_t)kt * kTile16;
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        d[m][h][0] = __ldg(reinterpret_cast<const uint4*>(base + m * kUp + h * 1024 + p0));
        d[m][h][1] = __ldg(reinterpret_cast<const uint4*>(base + m * kUp + h * 1024 + p1));
      }
  };
  if (warp < L.k_tiles) load_w(warp, w[0]);
  if (warp + kFewWarps < L.k_tiles) load_w(warp + kFewWarps, w[1]);
  griddep_wait();
  griddep_launch();
  if ((int)blockIdx.y >= *A.n_tiles_ptr) return;
  RowTile rt = A.tiles[blockIdx.y];
  for (;;) {
    float acc[M][NT][4];
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[m][t][c] = 0.f;
    const __half* x = F.x + (size_t)(rt.row0 + g) * F.ldx + q * 8;
    auto step = [&](int kt, const uint4 (&d)[M][2][2]) {
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        if (t && 8 * t >= rt.rows) continue;
        const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)(8 * t) * F.ldx + kt * kTileK);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          const uint4 b = xr[4 * p];
#pragma unroll
          for (int m = 0; m < M; ++m) {
            const uint4 lo = d[m][0][p], hi = d[m][1][p];
            mma_16816(acc[m][t], lo.x, hi.x, lo.y, hi.y, b.x, b.y);
            mma_16816(acc[m][t], lo.z, hi.z, lo.w, hi.w, b.z, b.w);
          }
        }
      }
    };
    for (int kt = warp; kt < L.k_tiles; kt += 2 * kFewWarps) {
      step(kt, w[0]);
      if (kt + 2 * kFewWarps < L.k_tiles) load_w(kt + 2 * kFewWarps, w[0]);
      if (kt + kFewWarps < L.k_tiles) {
        step(kt + kFewWarps, w[1]);
        if (kt + 3 * kFewWarps < L.k_tiles) load_w(kt + 3 * kFewWarps, w[1]);
      }
    }
    // [warp][matrix][group][register][lane]
    constexpr int kPer = M * NT * 4 * 32;
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int c = 0; c < 4; ++c) few_sums[warp * kPer + ((m * NT + t) * 4 + c) * 32 + lane] = acc[m][t][c];
    __syncthreads();
    const float* bias = reinterpret_cast<const float*>(ebase + A.bias_offset);
    for (int i = threadIdx.x; i < NT * 128; i += kFewWarps * 32) {
      // sixteen neighbouring threads: sixteen features of one token
      const int row = i & 15, token = i >> 4, n = n0 + row;
      const int at = ((token >> 3) * 4 + (row >> 3) * 2 + (token & 1)) * 32 + (row & 7) * 4 + (token >> 1 & 3);
      float s[M];
#pragma unroll
      for (int m = 0; m < M; ++m) {
        s[m] = few_sums[m * NT * 128 + at];
#pragma unroll
        for (int v = 1; v < kFewWarps; ++v) s[m] += few_sums[v * kPer + m * NT * 128 + at];
      }
      if (token >= rt.rows) continue;
      if (GATED) {
        const float gate = s[0] + (A.has_bias ? bias[A.F + n] : 0.f), up = s[M - 1] + (A.has_bias ? bias[n] : 0.f);
        A.a_out[(size_t)(rt.row0 + token) * A.lda + n] = __float2half_rn(gated_act_fast(gate, up, A.act));
      } else {
        A.y_out[(size_t)(rt.row0 + token) * A.ldy + n] = s[0] + (A.has_bias ? bias[2 * A.F + n] : 0.f);
      }
    }
    rt.row0 += 8 * NT;
    rt.rows -= 8 * NT;
    if (!TURNS || rt.rows <= 0) break;
    __syncthreads();  // the sums have been read
    if (warp < L.k_tiles) load_w(warp, w[0]);
    if (warp + kFewWarps < L.k_tiles) load_w(warp + kFewWarps, w[1]);
  }
}

template <bool GATED, bool TURNS>
inline cudaError_t few_launch_turns(const FewArgs& f, int features, int tiles, int rows, cudaStream_t s, bool pdl) {
  const int groups = rows <= 8 ? 1 : rows <= 16 ? 2 : rows <= 32 || TURNS ? 4 : 8;
  const dim3 grid((unsigned)(features / 16), (unsigned)tiles), block(kFewWarps * 32);
  const size_t smem = few_smem_bytes(groups, GATED);
  switch (groups) {
    case 1: return launch_k(k_few16<GATED, 1, TURNS>, grid, block, smem, s, pdl, f);
    case 2: return launch_k(k_few16<GATED, 2, TURNS>, grid, block, smem, s, pdl, f);
    case 4: return launch_k(k_few16<GATED, 4, TURNS>, grid, block, smem, s, pdl, f);
    default: return launch_k(k_few16<GATED, TURNS ? 4 : 8, TURNS>, grid, block, smem, s, pdl, f);
  }
}

// `tiles`: no fewer than the list may have; `rows`: of an expert, unless the routing may name it twice in a token
template <bool GATED>
inline cudaError_t few_launch_one(const FewArgs& f, int features, int tiles, int rows, bool repeats, cudaStream_t s, bool pdl) {
  return repeats ? few_launch_turns<GATED, true>(f, features, tiles, rows, s, pdl)
                 : few_launch_turns<GATED, false>(f, features, tiles, rows, s, pdl);
}

inline cudaError_t few_prepare_device() {
  return cudaFuncSetAttribute(k_few16<true, 8, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)few_smem_bytes(8, true));
}

}  // namespace csk
