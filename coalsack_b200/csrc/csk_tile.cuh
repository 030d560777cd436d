// Weight layouts, their repacks, and what both CTA-pair kernels (csk_tile2.cuh: MXFP4 weights, csk_pair16.cuh: fp16 weights) are given.
#pragma once

#include <cuda.h>

#include <functional>
#include <string>

#include "csk_common.cuh"
#include "csk_tc.cuh"

namespace csk {

constexpr int kTileW = 128;          // weight rows of half a weight tile (tensor-memory lanes of a CTA)
constexpr int kHalfPacked = 4352;                           // packed half tile: 4096 codes + 256 scales
constexpr int kTilePacked = 2 * kHalfPacked;                // packed weight tile (two halves)
// fp16 weights (dense FFN, fp16 expert slices): a half tile is 128 rows x 64 fp16 = 16 KB, rows of 128 bytes whose eight 16-byte
// pieces are stored at piece ^ (row & 7): the MMA's operand under the 128-byte swizzle
constexpr int kHalf16 = 128 * 128;
constexpr int kTile16 = 2 * kHalf16;
constexpr int kPairBoxes = 8;                               // the CTA-pair kernel's half tiles: boxes of 16, 32, ... 128 rows
struct PairMaps {
  CUtensorMap m[kPairBoxes];
};
constexpr uint32_t kTmemCols = 512;

// Device layout of a matrix for the fp16 tensor-core kernels: tiles of 256 rows x 64 columns, as two halves of 128 rows.
//
// MXFP4 (the CTA-pair kernel, csk_tile2.cuh): [n_tile][half][k_tile], so that a CTA's half runs on along K; a half tile is
// 4352 bytes,
//   bytes    0..4095  codes: [column block 0/1][row 0..127][16 bytes = 32 codes, nibble i of
//                     word w = column 8w + i]
//   bytes 4096..4351  E8M0 scales: [column block][row]
// Gate/up: half c holds the features 64c .. 64c+63 of the tile's 128, in groups of 16 gate and 16 up rows (a warp's lanes).
//
// fp16 (csk_pair16.cuh): [n_tile][k_tile][half], a half tile is 128 rows of 128 bytes.  Gate/up: the same features in the same
// order as MXFP4's halves.
//
// The file images have their own order of tiles and rows (k_reorder_tile).
struct TileLayout {
  int N, K, paired, n_tiles, k_tiles, w16;
  __host__ __device__ int half_bytes() const { return w16 ? kHalf16 : kHalfPacked; }
  __host__ __device__ int tile_bytes() const { return 2 * half_bytes(); }
  __host__ __device__ int feats_per_tile() const { return paired ? kTileW : 2 * kTileW; }
  // halves of tile nt that hold any real row (the last tile of a plain matrix may need only one)
  __host__ __device__ int halves(int nt) const { return paired || nt * 2 * kTileW + kTileW < N ? 2 : 1; }
  __host__ __device__ size_t bytes() const { return (size_t)n_tiles * k_tiles * tile_bytes(); }
  __host__ __device__ int k_pad() const { return k_tiles * kTileK; }
  // where half tiles of MXFP4 codes lie, and which half and which of its rows row `feat` of the matrix (of its gate or,
  // which = 1, its up matrix) is
  __host__ __device__ size_t half_at(int nt, int half, int kt) const { return (((size_t)nt * 2 + half) * k_tiles + kt) * kHalfPacked; }
  __host__ __device__ int half_of(int feat) const { return feat / (paired ? kTileW / 2 : kTileW) & 1; }
  __host__ __device__ int row_of(int feat, int which) const {
    return paired ? (feat % (kTileW / 2) & ~15) * 2 + which * 16 + (feat & 15) : feat % kTileW;
  }
};
inline TileLayout make_tile_layout(int N, int K, bool paired, bool w16 = false) {
  TileLayout L{};
  L.w16 = w16 ? 1 : 0;
  L.N = N;
  L.K = K;
  L.paired = paired ? 1 : 0;
  L.n_tiles = ceil_div(N, L.feats_per_tile());
  L.k_tiles = ceil_div(K, kTileK);
  return L;
}

// Repack of 17-byte blocks into the layout above (src1 = up matrix when paired).
__global__ void k_repack_tile(const uint8_t* __restrict__ src0, const uint8_t* __restrict__ src1,
                              uint8_t* __restrict__ dst, TileLayout L) {
  const size_t n_words = L.bytes() / 4;
  constexpr int WPT = kHalfPacked / 4;  // 1088 words per half tile
  for (size_t w = (size_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words; w += (size_t)gridDim.x * blockDim.x) {
    const size_t half_idx = w / WPT;
    const int wi = (int)(w % WPT);
    const int kt = (int)(half_idx % L.k_tiles), half = (int)(half_idx / L.k_tiles & 1), nt = (int)(half_idx / (2 * L.k_tiles));
    uint32_t out = 0;
    auto source = [&](int trow, const uint8_t*& src, int& feat) {
      if (L.paired) {
        src = trow & 16 ? src1 : src0;
        feat = nt * kTileW + half * (kTileW / 2) + (trow >> 5) * 16 + (trow & 15);
      } else {
        src = src0;
        feat = nt * 2 * kTileW + half * kTileW + trow;
      }
    };
    if (wi < 1024) {
      const int blk = wi >> 9, trow = (wi & 511) >> 2, q = wi & 3;
      const int col = kt * kTileK + blk * 32 + q * 8;
      const uint8_t* src;
      int feat;
      source(trow, src, feat);
      if (feat < L.N && col < L.K) {
        const uint8_t* b = src + ((size_t)feat * (L.K / 32) + col / 32) * 17;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int j = q * 8 + i;
          const uint32_t code = j < 16 ? (b[1 + j] & 0xF) : (b[1 + j - 16] >> 4);
          out |= code << (4 * i);
        }
      }
    } else {
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int bi = (wi - 1024) * 4 + t;
        const int blk = bi >> 7, trow = bi & 127;
        const int col = kt * kTileK + blk * 32;
        const uint8_t* src;
        int feat;
        source(trow, src, feat);
        uint32_t e = 0;  // padding: zero codes under the smallest scale
        if (feat < L.N && col < L.K) e = src[((size_t)feat * (L.K / 32) + col / 32) * 17];
        out |= e << (8 * t);
      }
    }
    reinterpret_cast<uint32_t*>(dst)[w] = out;
  }
}

// fp16 weights, row-major [N,K] (src1 = up matrix when paired), into the fp16 tile layout.  One thread
// per 16-byte piece (eight columns of one row).
__global__ void k_repack_tile_f16(const __half* __restrict__ src0, const __half* __restrict__ src1,
                                  uint8_t* __restrict__ dst, TileLayout L) {
  const size_t n_pieces = L.bytes() / 16;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_pieces; i += (size_t)gridDim.x * blockDim.x) {
    const size_t half_idx = i >> 10;  // 1024 pieces per half tile
    const int pi = (int)(i & 1023);
    const int trow = pi >> 3, piece = (pi & 7) ^ (trow & 7);  // the piece stored here
    const int half = (int)(half_idx & 1);
    const size_t tile = half_idx >> 1;
    const int kt = (int)(tile % L.k_tiles), nt = (int)(tile / L.k_tiles);
    const __half* src = L.paired && (trow & 16) ? src1 : src0;
    const int feat = L.paired ? nt * kTileW + half * (kTileW / 2) + (trow >> 5) * 16 + (trow & 15) : nt * 2 * kTileW + half * kTileW + trow;
    const int col = kt * kTileK + piece * 8;
    uint4 out = make_uint4(0u, 0u, 0u, 0u);
    if (feat < L.N && col < L.K) {  // K is a multiple of 32: a piece is inside or outside as a whole
      const __half* p = src + (size_t)feat * L.K + col;
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        w[e] = (uint32_t)__half_as_ushort(p[2 * e]) | ((uint32_t)__half_as_ushort(p[2 * e + 1]) << 16);
      out = make_uint4(w[0], w[1], w[2], w[3]);
    }
    reinterpret_cast<uint4*>(dst)[i] = out;
  }
}

// Inverse of k_repack_tile for one source matrix (which_half: 0 = the matrix
// itself or the gate rows, 1 = the up rows).  One thread per 17-byte block.
__global__ void k_unpack_tile(const uint8_t* __restrict__ packed, uint8_t* __restrict__ out, TileLayout L,
                              int which_half) {
  const int kb = L.K / 32;
  const size_t n_blocks = (size_t)L.N * kb;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_blocks; i += (size_t)gridDim.x * blockDim.x) {
    const int feat = (int)(i / kb), blk_g = (int)(i % kb);
    const int nt = feat / L.feats_per_tile(), trow = L.row_of(feat, which_half);
    const int kt = blk_g / 2, blk = blk_g & 1;
    const uint8_t* tile = packed + L.half_at(nt, L.half_of(feat), kt);
    uint8_t* o = out + i * 17;
    o[0] = tile[4096 + blk * 128 + trow];
    const uint32_t* words = reinterpret_cast<const uint32_t*>(tile + ((size_t)blk * 128 + trow) * 16);
    uint32_t codes[32];
    for (int q = 0; q < 4; ++q)
      for (int t = 0; t < 8; ++t) codes[q * 8 + t] = (words[q] >> (4 * t)) & 0xF;
    for (int j = 0; j < 16; ++j) o[1 + j] = (uint8_t)(codes[j] | (codes[j + 16] << 4));
  }
}

// From the device's order of tiles and rows to that of the file images ([n_tile][k_tile][half]; gate/up: half 0 the gate, half 1 the up
// rows of 128 features) or back.  One thread per row of a half tile.
__global__ void k_reorder_tile(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, TileLayout L, int to_file) {
  const size_t n = (size_t)L.n_tiles * 2 * L.k_tiles * kTileW;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int r = (int)(i % kTileW), kt = (int)(i / kTileW % L.k_tiles);
    const int half = (int)(i / ((size_t)kTileW * L.k_tiles) & 1), nt = (int)(i / ((size_t)2 * kTileW * L.k_tiles));
    const int file_half = L.paired ? r >> 4 & 1 : half, file_row = L.paired ? half * 64 + (r >> 5) * 16 + (r & 15) : r;
    const size_t tile = (size_t)nt * L.k_tiles + kt;
    const size_t here = L.w16 ? (tile * 2 + half) * kHalf16 : L.half_at(nt, half, kt), file = (tile * 2 + file_half) * L.half_bytes();
    const uint8_t* s = src + (to_file ? here : file);
    uint8_t* d = dst + (to_file ? file : here);
    const int sr = to_file ? r : file_row, dr = to_file ? file_row : r;
    if (L.w16) {  // (a row's pieces stay where they are: r and file_row agree modulo 8)
#pragma unroll
      for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(d + dr * 128 + c * 16) = *reinterpret_cast<const uint4*>(s + sr * 128 + c * 16);
      continue;
    }
#pragma unroll
    for (int blk = 0; blk < 2; ++blk) {
      *reinterpret_cast<uint4*>(d + (blk * 128 + dr) * 16) = *reinterpret_cast<const uint4*>(s + (blk * 128 + sr) * 16);
      d[4096 + blk * 128 + dr] = s[4096 + blk * 128 + sr];
    }
  }
}

struct TileState {
  bool available = false;
  std::string err;
  PairMaps pair_x{};      // grouped input rows  [rows, ldx] fp16, a map for every height of a CTA's half of a row tile
  PairMaps pair_a{};      // activated rows      [rows, lda] fp16
  CUtensorMap weights{};  // fp16 weights as rows of 128 bytes, boxes of a half tile
  bool maps_ready = false;
  void* encode_fn = nullptr;
};

// fp16 bit pattern (in both halves) of 2^s for s in [-24, 15]; 0 below, 2^15 above.
__device__ __forceinline__ uint32_t h2_pow2(int s) {
  s = s > 15 ? 15 : s;
  uint32_t b = s >= -14 ? (uint32_t)(s + 15) << 10 : (s >= -24 ? 1u << (s + 24) : 0u);
  return b | (b << 16);
}
__device__ __forceinline__ uint32_t hmul2_u32(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("mul.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

struct TileArgs {
  const uint8_t* weights;
  size_t expert_stride, mat_offset, bias_offset, meta_offset;
  TileLayout L;
  __half* a_out;          // GATED: activated rows [rows, lda]
  int lda;
  float* y_out;           // !GATED: output rows [rows, ldy]
  int ldy;
  const int* out_row_map; // optional indirection of output rows (!GATED)
  float* const* out_row_ptr;  // or: where each output row goes (possibly another GPU's memory); wins over the map
  const RowTile* tiles;
  const int* n_tiles_ptr;
  int* meta;              // meta[3] = device status word
  int has_bias, act, F, meta_slot;
  int stall;              // test hook: the copy role issues nothing, so every other role's wait runs out
};

// ---- host side ------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline int tile_init(TileState& st, int device) {
  (void)device;
  st.available = false;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn) {
    cudaGetLastError();
    st.err = "cuTensorMapEncodeTiled not found in the driver";
    return CSK_ERR_CUDA;
  }
  st.encode_fn = fn;
  st.available = true;
  return CSK_OK;
}
inline void tile_destroy(TileState&) {}

// [rows, ld] fp16 row-major, boxes of box_rows rows x 64 columns; in shared memory under the 128-byte swizzle, or as they are.
inline int tile_make_map(TileState& st, CUtensorMap* map, const void* base, size_t rows, int ld, int box_rows, bool swizzle = true) {
  const cuuint64_t dims[2] = {(cuuint64_t)ld, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(__half)};
  const cuuint32_t box[2] = {(cuuint32_t)kTileK, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  CUresult r = ((EncodeTiledFn)st.encode_fn)(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)base, dims, strides, box,
                                             estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                             swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    st.err = "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r);
    return CSK_ERR_CUDA;
  }
  return CSK_OK;
}

// weights16: the layer's weights, weight_bytes of them (a multiple of 128), if they are fp16
inline int tile_set_buffers(TileState& st, const __half* x16, int ldx, const __half* a16, int lda, size_t rows_alloc, const uint8_t* weights16,
                            size_t weight_bytes) {
  if (!st.available) return CSK_OK;
  int rc = CSK_OK;
  if (weights16) rc = tile_make_map(st, &st.weights, weights16, weight_bytes / 128, kTileK, kTileW, false);
  for (int b = 0; b < kPairBoxes && !rc; ++b) {
    rc = tile_make_map(st, &st.pair_x.m[b], x16, rows_alloc, ldx, 16 * (b + 1));
    if (!rc) rc = tile_make_map(st, &st.pair_a.m[b], a16, rows_alloc, lda, 16 * (b + 1));
  }
  if (rc) return rc;
  st.maps_ready = true;
  return CSK_OK;
}

}  // namespace csk
