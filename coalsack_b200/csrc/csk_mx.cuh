// Block-scaled grouped contraction over MXFP4 weights (the decode-side kernel), written for sm_100a.
//
// The weights go to the tensor cores AS THEY ARE: tcgen05.mma kind::mxf4 multiplies E2M1 codes under E8M0 block
// scales, so no weight is ever converted, and the kernel's only bulk work is moving the packed bytes from HBM to
// shared memory.  Its other operand has to be E2M1 codes under E8M0 scales too, so every activation row is written
// as several rows of such codes (the "digits" of a radix-8 expansion, below), which are as many columns of the same
// MMA; the accumulators of the digits are added with weights 8^-p in the epilogue.
//
// Digits.  For a block of 32 values with largest magnitude m the scale is the power of two 2^e with m <= 4.5 * 2^e.
// Digit 0 is v / 2^e rounded to E2M1 (0, 0.5, 1, 1.5, 2, 3, 4, 6): the remainder of a value of magnitude up to 4.5 is
// at most 0.5, so eight times the remainder is again at most 4: the other digits repeat the step.  n digits leave at
// most 0.5 * 8^(1-n) * 2^e of every value (rms measured: 0.15 * 8^(1-n) * 2^e), the SAME amount of a large and of a small
// one.  An fp16 operand leaves a share of each value (rms 2.07e-4 of it).  Token rows get five digits, activated rows,
// whose values spread further, six: measured 2.9e-5 of the norm for normal values in five, 4.6e-6 to 5.8e-6 for gated
// products of normal values in six, fp16 2.1e-4 for both.  Products of codes are exact and the sums are fp32.
//
// Wide blocks.  Where a few values of a block are far above the others, the digits' absolute error may be more than fp16
// would leave of those others, and the weights of the few may be zero.  Such a block gets as many digits again,
// continuing the expansion (at most 2^-29 of the block's largest value is then left), in a second image of the same
// geometry; the records of a row tile that hold any are run twice, once per image, into the same accumulators, and
// everywhere else the second image holds zeros.  A block is taken as it is only if, WHICHEVER t of its values are left
// out, the digits' error over the others is no larger than that of an fp16 operand (mx_wide_limit; t = 8 of 32 for
// token rows, 4 for activated rows).  That costs nothing for normal values (none of 400,000 blocks is wide) and little for gated
// products of them (7e-4 of the blocks and fewer).
//
//   * a work unit is (row tile of up to 40 grouped token rows of one expert) x (256 weight rows, as two halves of
//     128: gate and up rows of the same 128 features, or 256 rows of a plain matrix); units are dealt to one
//     persistent CTA per SM;
//   * along K the unit is a run of records of 128 columns: 2 x 8192 bytes of codes and 2 x 512 bytes of scales,
//     contiguous in memory, moved with ONE bulk copy each; a second bulk copy brings the same columns of the token
//     rows' image.  A ring of 6 (40 rows a tile) to 12 (3 rows) such stages keeps 105-210 KB of weights per SM in flight;
//   * the MMA warp copies the record's scales to tensor memory (tcgen05.cp) and issues two K=64 MMAs per half;
//   * eight epilogue warps add up the digits' accumulators, add the bias and either apply the gated activation and
//     write the result as digits again (a warp's 32 lanes are the 32 features of one block), in the images the down
//     projection reads, or (plain matrix) store fp32 output rows.  Accumulators of even units grow from the bottom of
//     tensor memory, those of odd units from the top: the epilogue of one unit runs under the MMAs of the next unless
//     the two need more than 480 columns together (gate/up: two tiles of 22 rows fit; down: of 18).
//
// The producer asks for weights before griddepcontrol.wait: the tile list comes from a kernel two launches back.
//
// Every wait is bounded (csk_common.cuh); when one runs out the CTA records kDevErrWaitTimeout, all roles leave
// their loops, copies and MMAs in flight are waited for (bounded again), tensor memory is freed.
//
// Follows the arithmetic of expert_mlp_node::compute_token_mxfp4
// (include/coalsack/nn/nn_ops/expert_mlp_node.h:651-732): up/gate projections + bias, gated activation, down
// projection + bias.
#pragma once

#include "csk_common.cuh"
#include "csk_tc.cuh"

namespace csk {

constexpr int kMxDigitsX = 5, kMxDigitsA = 6;      // digits of a token row, of an activated row
constexpr int kMxTileRows = 40;                    // token rows of a row tile: 6 * 40 = 240 MMA columns, twice in tensor memory
constexpr int kMxRecBlocks = 4;                    // 32-column blocks per record
constexpr int kMxSfAtom = 512;                     // scales of 128 rows x 4 blocks: [row % 32][row / 32][block]
constexpr int kMxARecMax = kMxRecBlocks * 256 * 16 + 2 * kMxSfAtom;
constexpr int kMxEpilogueWarps = 8;
constexpr int kMxThreads = (2 + kMxEpilogueWarps) * 32;
constexpr int kMxMaxStages = 12;
constexpr int kMxSmem = 227 * 1024;
constexpr int kMxCtrl = 512;
constexpr int kMxSlack = 4096;      // a half of fewer than 128 rows lets the MMA read past its codes
constexpr uint32_t kMxTmemCols = 512;
constexpr uint32_t kMxTmemSf = 480;                // two sets of 16 columns: SF of half 0, of half 1, of the rows (8)

// Device layout of a matrix for this kernel: units of 256 rows (paired: 128 gate + 128 up rows of the same features)
// in order; a unit is `recs` records along K; a record of nb (4, the last one 2 or 4) 32-column blocks is
//   for each pair of blocks: [half 0: 2 blocks x r0 rows x 16 bytes][half 1: 2 blocks x r1 rows x 16 bytes],
//   then per half one 512-byte atom of scales.
// 16 bytes are a row's 32 codes, column 2i in the low nibble of byte i.  r0, r1 are the half's real rows (the last
// unit may have fewer than 128); columns past K are zero codes, scales of absent rows and columns 0.
struct MxLayout {
  int N, K, paired;
  int n_units, blocks /* even */, recs;
  __host__ __device__ int rows(int nt, int half) const {
    const int left = paired ? N - nt * 128 : N - nt * 256 - half * 128;
    return left < 0 ? 0 : left > 128 ? 128 : left;
  }
  __host__ __device__ int halves(int nt) const { return rows(nt, 1) > 0 ? 2 : 1; }
  __host__ __device__ int rec_blocks(int rec) const { return blocks - rec * kMxRecBlocks < kMxRecBlocks ? blocks - rec * kMxRecBlocks : kMxRecBlocks; }
  __host__ __device__ int rec_bytes(int nt, int nb) const {
    return nb * (rows(nt, 0) + rows(nt, 1)) * 16 + halves(nt) * kMxSfAtom;
  }
  __host__ __device__ size_t unit_bytes(int nt) const {
    return (size_t)blocks * (rows(nt, 0) + rows(nt, 1)) * 16 + (size_t)recs * halves(nt) * kMxSfAtom;
  }
  __host__ __device__ size_t bytes() const { return (size_t)(n_units - 1) * unit_bytes(0) + unit_bytes(n_units - 1); }
};
inline MxLayout make_mx_layout(int N, int K, bool paired) {
  MxLayout L{};
  L.N = N;
  L.K = K;
  L.paired = paired ? 1 : 0;
  L.n_units = ceil_div(N, paired ? 128 : 256);
  L.blocks = 2 * ceil_div(K, 64);
  L.recs = ceil_div(L.blocks, kMxRecBlocks);
  return L;
}

// The image of a row tile of `rows` rows of n digits (n * rows MMA columns, padded to a multiple of 16): per record
// [scale atoms][4 blocks x npad x 16 bytes of codes]; column n r + p is digit p of row r.  Tiles lie one after the
// other in row order; `col0` and `atom0` bound what the tiles before this one take.
struct MxTileImage {
  int npad, atoms;
  size_t offset;      // of the tile's image
  size_t rec_stride;
};
template <int D>
__host__ __device__ inline int mx_npad(int rows) { return (D * rows + 15) / 16 * 16; }
template <int D>
__host__ __device__ inline MxTileImage mx_tile_image(int tile, int row0, int rows, int recs) {
  MxTileImage t;
  t.npad = mx_npad<D>(rows);
  t.atoms = t.npad > 128 ? 2 : 1;
  const size_t col0 = (size_t)D * row0 + 16 * (size_t)tile;
  const size_t atom0 = (size_t)D * row0 / 128 + 2 * (size_t)tile;
  t.offset = (size_t)recs * (col0 * (kMxRecBlocks * 16) + atom0 * kMxSfAtom);
  t.rec_stride = (size_t)t.atoms * kMxSfAtom + (size_t)t.npad * (kMxRecBlocks * 16);
  return t;
}
inline size_t mx_image_bytes(int digits, size_t rows, size_t tiles, int recs) {
  return (size_t)recs * ((digits * rows + 16 * tiles) * (kMxRecBlocks * 16) + (digits * rows / 128 + 2 * tiles + 2) * kMxSfAtom);
}
// Words of a row tile's record mask (a bit per record: some row's block in it is wide).
__host__ __device__ inline int mx_mask_words(int recs) { return (recs + 31) / 32; }
__device__ __forceinline__ size_t mx_sf_pos(int n, int kb) {  // column n's scale of block kb inside a record's atoms
  return (size_t)(n >> 7) * kMxSfAtom + (n & 31) * 16 + ((n & 127) >> 5) * 4 + (kb & 3);
}

// ---- repack and its inverse ---------------------------------------------------------------------------------------
// One thread per (row, block): 17 raw bytes -> 16 bytes of codes and a scale byte; then one thread per absent row's
// scale.  src1 = up matrix when paired.  A raw block holds column j in the low and column j + 16 in the high nibble
// of byte j.  Scale byte 255 (NaN in the OCP MX specification) is stored as 254, so that a block of zero codes stays
// zero under any scale byte, as in the reference.
__global__ void k_mx_repack(const uint8_t* __restrict__ src0, const uint8_t* __restrict__ src1, uint8_t* __restrict__ dst,
                            MxLayout L, int* __restrict__ emax_out) {
  int emax = -1;
  const int halves_all = 2 * L.n_units;
  const size_t n = (size_t)halves_all * L.recs * kMxRecBlocks * 128;
  const size_t unit0 = L.unit_bytes(0);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int kb = (int)(i % (L.recs * kMxRecBlocks));  // neighbouring threads: neighbouring raw blocks of one row
    const size_t rest = i / (L.recs * kMxRecBlocks);
    const int r = (int)(rest % 128), half = (int)((rest / 128) & 1), nt = (int)(rest / 256);
    if (half >= L.halves(nt)) continue;
    const int rec = kb / kMxRecBlocks, nb = L.rec_blocks(rec), kbl = kb % kMxRecBlocks;
    const int r0 = L.rows(nt, 0), r1 = L.rows(nt, 1), rh = half ? r1 : r0;
    uint8_t* record = dst + nt * unit0 + (size_t)rec * L.rec_bytes(nt, kMxRecBlocks);
    const int row = L.paired ? nt * 128 + r : nt * 256 + half * 128 + r;
    const bool real = r < rh && kb * 32 < L.K;
    uint32_t e = 0;
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    if (real) {
      const uint8_t* b = (L.paired && half ? src1 : src0) + ((size_t)row * (L.K / 32) + kb) * 17;
      e = min((uint32_t)b[0], 254u);
      // a block of zero codes is zero under any scale: it does not widen the matrix's exponent range
      uint32_t any = 0;
#pragma unroll
      for (int j = 1; j < 17; ++j) any |= b[j];
      if (any) emax = max(emax, (int)e);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const uint32_t x = b[1 + 2 * q], y = b[2 + 2 * q];
        const uint32_t lo = (x & 0xFu) | (y & 0xFu) << 4, hi = x >> 4 | (y >> 4) << 4;
        w[q >> 2] |= lo << (8 * (q & 3));
        w[2 + (q >> 2)] |= hi << (8 * (q & 3));
      }
    }
    if (r < rh && kbl < nb)
      *reinterpret_cast<uint4*>(record + (kbl >> 1) * 32 * (r0 + r1) + half * 32 * r0 + (size_t)(kbl & 1) * 16 * rh +
                                (size_t)r * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    record[nb * (r0 + r1) * 16 + half * kMxSfAtom + (r & 31) * 16 + (r >> 5) * 4 + kbl] = (uint8_t)e;
  }
  emax = __reduce_max_sync(0xffffffffu, emax);
  if ((threadIdx.x & 31) == 0 && emax >= 0) atomicMax(emax_out, emax);  // largest scale exponent of the non-zero blocks
}
// which_half: 0 = the matrix itself or the gate rows, 1 = the up rows.  One thread per 17-byte block.
__global__ void k_mx_unpack(const uint8_t* __restrict__ packed, uint8_t* __restrict__ out, MxLayout L, int which_half) {
  const int kbs = L.K / 32;
  const size_t n = (size_t)L.N * kbs;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const int row = (int)(i / kbs), kb = (int)(i % kbs);
    const int nt = row / (L.paired ? 128 : 256), half = L.paired ? which_half : row / 128 % 2, r = row % 128;
    const int rec = kb / kMxRecBlocks, nb = L.rec_blocks(rec), kbl = kb % kMxRecBlocks;
    const int r0 = L.rows(nt, 0), r1 = L.rows(nt, 1), rh = half ? r1 : r0;
    const uint8_t* record = packed + nt * L.unit_bytes(0) + (size_t)rec * L.rec_bytes(nt, kMxRecBlocks);
    const uint8_t* c = record + (kbl >> 1) * 32 * (r0 + r1) + half * 32 * r0 + (kbl & 1) * 16 * rh + r * 16;
    uint8_t* o = out + i * 17;
    o[0] = record[nb * (r0 + r1) * 16 + half * kMxSfAtom + (r & 31) * 16 + (r >> 5) * 4 + kbl];
    for (int j = 0; j < 16; ++j) {
      const uint32_t lo = c[j / 2] >> (4 * (j & 1)) & 0xFu, hi = c[8 + j / 2] >> (4 * (j & 1)) & 0xFu;
      o[1 + j] = (uint8_t)(lo | hi << 4);
    }
  }
}

// ---- digits ---------------------------------------------------------------------------------------------------------
// Two values to a byte of E2M1 codes (a in the low nibble), round to nearest even.
__device__ __forceinline__ uint32_t f32x2_to_e2m1(float a, float b) {
  uint32_t r;
  asm("{\n\t.reg .b8 t;\n\tcvt.rn.satfinite.e2m1x2.f32 t, %2, %1;\n\tcvt.u32.u8 %0, t;\n\t}" : "=r"(r) : "f"(a), "f"(b));
  return r;
}
// The scale byte of a block whose largest magnitude has the bit pattern `amax`, and the factor that takes values to
// digit units: 2^(sf - 127) is the smallest power of two with amax <= 4.5 of it.  A block that holds an infinity or
// a NaN gets the NaN scale: its row's results are NaN, no other row's.
__device__ __forceinline__ uint32_t mx_scale_of(uint32_t amax, float& inv) {
  if (amax >= 0x7F800000u) {
    inv = 0.f;
    return 255u;
  }
  const uint32_t sf = (__float_as_uint(__uint_as_float(amax) * (1.0f / 4.5f)) + 0x7FFFFFu) >> 23;
  inv = __uint_as_float((254u - sf) << 23);
  return sf;
}
// One digit of two values; a and b become eight times the remainder.
__device__ __forceinline__ uint32_t mx_digit(float& a, float& b) {
  const uint32_t d = f32x2_to_e2m1(a, b);
  const uint32_t h = e2m1x2_to_h2(d);
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
  a = (a - f.x) * 8.0f;
  b = (b - f.y) * 8.0f;
  return d;
}
// Clip and limit of the test for wide blocks.  With values in units of 2^e, digits leave an rms of 0.15 * 8^(1-n) of
// each, fp16 2.07e-4 of each value: over any set of values whose rms is at least kappa = 0.15 * 8^(1-n) / 2.07e-4 (0.177 for
// five digits, 0.0221 for six) the digits are the better operand.  The sum over the block of min(v^2, clip^2) loses at most
// t clip^2 with any t of the values, so a sum of t clip^2 + (32 - t) kappa^2 leaves rms kappa for the rest.  Clip and t:
// five digits 1/2 and 8 (2 + 0.752), six 1/8 and 4 (0.0625 + 0.0137); rounded up.
template <int D>
__host__ __device__ constexpr float mx_wide_clip2() { return D == kMxDigitsX ? 0.25f : 1.0f / 64.0f; }
template <int D>
__host__ __device__ constexpr float mx_wide_limit() { return D == kMxDigitsX ? 2.76f : 0.077f; }
__host__ __device__ constexpr uint32_t mx_rest_shift(int digits) { return 3u * (uint32_t)digits; }  // the digits' scale over that of the digits after them

// A block by four neighbouring lanes, eight values each: `d` the digits (a word of digit p's codes), `rest` the digits
// after them (zeros unless the block is wide), the scale byte.  All lanes of the warp call it.
struct MxEncoded {
  uint32_t d[kMxDigitsX], rest[kMxDigitsX], sf;
  bool wide;
};
__device__ __forceinline__ void mx_digits(float (&v)[8], uint32_t (&d)[kMxDigitsX]) {
#pragma unroll
  for (int p = 0; p < kMxDigitsX; ++p) {
    d[p] = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) d[p] |= mx_digit(v[2 * q], v[2 * q + 1]) << (8 * q);
  }
}
__device__ __forceinline__ MxEncoded mx_encode_block(float (&v)[8]) {
  MxEncoded e;
  uint32_t amax = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = max(amax, __float_as_uint(v[i]) & 0x7FFFFFFFu);
  amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
  amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
  float inv, q = 0.f;
  e.sf = mx_scale_of(amax, inv);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[i] *= inv;
    q += fminf(v[i] * v[i], mx_wide_clip2<kMxDigitsX>());
  }
  q += __shfl_xor_sync(0xffffffffu, q, 1);  // (both sums are the same in every lane of the four)
  q += __shfl_xor_sync(0xffffffffu, q, 2);
  mx_digits(v, e.d);
  e.wide = q < mx_wide_limit<kMxDigitsX>() && e.sf >= mx_rest_shift(kMxDigitsX) && e.sf != 255u;
#pragma unroll
  for (int p = 0; p < kMxDigitsX; ++p) e.rest[p] = 0;
  if (e.wide) mx_digits(v, e.rest);
  uint32_t left = 0;
#pragma unroll
  for (int p = 0; p < kMxDigitsX; ++p) left |= e.rest[p];
  // a power of two among zeros: nothing is left (sign bits alone are digits of zero too)
  e.wide = __ballot_sync(0xffffffffu, (left & 0x77777777u) != 0) >> (threadIdx.x & 28) & 0xFu;
  return e;
}
// The four lanes' words of the digits to their columns of row r (word q = lane & 3 of each 16 bytes); the scale bytes
// unless sf < 0: zeros are zero under any scale but NaN, and the second image never holds that.
__device__ __forceinline__ void mx_store_block(uint8_t* image, const MxTileImage& g, int r, int kb, int q, const uint32_t (&d)[kMxDigitsX],
                                               int sf) {
  uint8_t* rec = image + g.offset + (size_t)(kb / kMxRecBlocks) * g.rec_stride;
  const int n = kMxDigitsX * r;
  uint8_t* codes = rec + g.atoms * kMxSfAtom + ((size_t)(kb & 3) * g.npad + n) * 16 + 4 * q;
#pragma unroll
  for (int p = 0; p < kMxDigitsX; ++p) *reinterpret_cast<uint32_t*>(codes + 16 * p) = d[p];
  if (sf >= 0)
    for (int p = q; p < kMxDigitsX; p += 4) rec[mx_sf_pos(n + p, kb)] = (uint8_t)sf;
}
// Columns past K inside the last pair of blocks: the weights' codes are zero there, so any scale but NaN will do.
__device__ __forceinline__ void mx_store_pad(uint8_t* image, const MxTileImage& g, int r, int kb, int q) {
  uint8_t* rec = image + g.offset + (size_t)(kb / kMxRecBlocks) * g.rec_stride;
  for (int p = q; p < kMxDigitsX; p += 4) rec[mx_sf_pos(kMxDigitsX * r + p, kb)] = 0;
}
__device__ __forceinline__ void mx_mark_wide(uint32_t* tile_mask, int kb) {
  atomicOr(tile_mask + kb / (32 * kMxRecBlocks), 1u << (kb / kMxRecBlocks & 31));
}

struct MxQuantArgs {
  const float* hidden;       // [T,H]
  const float* router;       // [T,k,2]
  const int* offsets;        // [E+1] first row of each expert
  const ExpertTiles* et;     // [E]
  int* cursor;               // null: the places are given; else rows are claimed here and row_of_pair is written
  int* row_of_pair;          // [T*k]
  const int4* places;        // [T*k] the pairs' places by k_scan (cursor null), see there
  const RowTile* tiles;
  const int* n_tiles_ptr;
  uint8_t *image, *rest;     // digits, and the digits after them
  uint32_t* wide;            // record masks of the row tiles, wide_stride words each
  int wide_stride;
  int T, H, E, k, e_begin, e_count, only_expert, max_rows, weight_before_ffn, blocks, recs;
};
// What four neighbouring lanes hold of a block, a word of each digit, as whole digits: lane q has digit q in `own` and all have the fifth.
struct MxColumns {
  uint4 own, fifth;
};
__device__ __forceinline__ MxColumns mx_columns(const uint32_t (&d)[kMxDigitsX], int q) {
  const bool odd = q & 1, high = q & 2;
  const uint32_t a = __shfl_xor_sync(0xffffffffu, odd ? d[0] : d[1], 1), b = __shfl_xor_sync(0xffffffffu, odd ? d[2] : d[3], 1);
  const uint32_t l0 = odd ? a : d[0], l1 = odd ? d[1] : a, h0 = odd ? b : d[2], h1 = odd ? d[3] : b;  // two words of digits q & 1, 2 + (q & 1)
  const uint32_t r0 = __shfl_xor_sync(0xffffffffu, high ? l0 : h0, 2), r1 = __shfl_xor_sync(0xffffffffu, high ? l1 : h1, 2);
  MxColumns c;
  c.own = high ? make_uint4(r0, r1, h0, h1) : make_uint4(l0, l1, r0, r1);
  const int first = threadIdx.x & 28;
  c.fifth = make_uint4(__shfl_sync(0xffffffffu, d[4], first), __shfl_sync(0xffffffffu, d[4], first + 1),
                       __shfl_sync(0xffffffffu, d[4], first + 2), __shfl_sync(0xffffffffu, d[4], first + 3));
  return c;
}

// Token rows to digits, into the images of the row tiles they were placed in.  A CTA per token and 32 of its 32-column blocks, four threads
// per block: a token is encoded once and stored k times (with the routing weight applied before the expert it is
// encoded per pair).  What a token costs is its stores (one CTA a token and a word a store: 1 token of 2880 columns 5500 of the
// kernel's 6100 clocks after the wait): a lane stores whole digits, 16 bytes, sixteen lanes a record's scales as words, and
// the blocks of a token are on several SMs (one CTA where the rows are claimed here).
constexpr int kMxQuantThreads = 384, kMxQuantPart = 128;
static_assert(kMxDigitsX == 5, "four lanes' digits and a fifth");
__global__ void __launch_bounds__(kMxQuantThreads) k_mx_quant(const MxQuantArgs A) {
  __shared__ MxTileImage s_img[16];
  __shared__ int s_r[16], s_tile[16];
  __shared__ float s_w[16];
  const int t = blockIdx.x, kbs = A.H / 32, q = threadIdx.x & 3, step = (gridDim.y * blockDim.x) >> 2;
  int kb = (blockIdx.y * blockDim.x + threadIdx.x) >> 2;
  float v[8];
  MxEncoded e;
  auto load = [&](float w) {  // the eight values of this thread times w (zeros past the row)
    const float4* src = reinterpret_cast<const float4*>(A.hidden + (size_t)t * A.H + kb * 32 + q * 8);
    const float4 x = kb < kbs ? __ldg(src) : make_float4(0.f, 0.f, 0.f, 0.f), y = kb < kbs ? __ldg(src + 1) : x;
    v[0] = x.x * w, v[1] = x.y * w, v[2] = x.z * w, v[3] = x.w * w;
    v[4] = y.x * w, v[5] = y.y * w, v[6] = y.z * w, v[7] = y.w * w;
  };
  MxColumns c, rest;
  uint32_t scales = 0;  // of the record's four blocks
  bool any_wide = false;
  auto encode = [&](float w) {
    load(w);
    e = mx_encode_block(v);
    c = mx_columns(e.d, q);
    any_wide = __any_sync(0xffffffffu, e.wide);
    if (any_wide) rest = mx_columns(e.rest, q);
    else rest.own = rest.fifth = make_uint4(0, 0, 0, 0);
    // (columns past K inside the last blocks: the weights' codes are zero there, so any scale but NaN will do)
    scales = kb < kbs ? e.sf << (8 * (kb & 3)) : 0u;
    scales |= __shfl_xor_sync(0xffffffffu, scales, 4);
    scales |= __shfl_xor_sync(0xffffffffu, scales, 8);
  };
  // the hidden states are older than the kernel before this one: encode while it is still placing rows
  if (!A.weight_before_ffn) encode(1.f);
  griddep_wait();
  griddep_launch();
  if ((int)threadIdx.x < A.k) {
    const int j = threadIdx.x, pair = t * A.k + j;
    if (!A.cursor) {
      const int4 at = A.places[pair];
      s_img[j] = mx_tile_image<kMxDigitsX>(at.x, at.y, at.z, A.recs);
      s_tile[j] = at.x;
      s_r[j] = at.w;
      s_w[j] = A.router[2 * (size_t)pair + 1];
    } else {
      const int x = (int)A.router[2 * (size_t)pair];
      int pos = -1;
      if (x >= 0 && x < A.E && (A.only_expert < 0 || x == A.only_expert)) pos = A.offsets[x] + atomicAdd(&A.cursor[x], 1);
      if (pos >= A.max_rows) pos = -1;
      A.row_of_pair[pair] = pos;
      s_r[j] = -1;
      if (pos >= 0 && x >= A.e_begin && x < A.e_begin + A.e_count && *A.n_tiles_ptr > 0) {
        const ExpertTiles et = A.et[x];
        const int r = pos - A.offsets[x], tile = et.tile0 + r / et.height;
        const RowTile rt = A.tiles[tile];
        s_img[j] = mx_tile_image<kMxDigitsX>(tile, rt.row0, rt.rows, A.recs);
        s_tile[j] = tile;
        s_r[j] = r % et.height;
        s_w[j] = A.router[2 * (size_t)pair + 1];
      }
    }
  }
  __syncthreads();
  // (whole warps: the lanes of a block past the row's end take part in the exchanges)
  for (bool first = true; (kb & ~7) < A.blocks; kb += step, first = false) {
    if (!first && !A.weight_before_ffn) encode(1.f);
    for (int j = 0; j < A.k; ++j) {
      if (s_r[j] < 0) continue;
      if (A.weight_before_ffn) encode(s_w[j]);
      if ((kb & ~3) >= A.blocks) continue;
      const MxTileImage& g = s_img[j];
      const int n = kMxDigitsX * s_r[j];
      const size_t rec = g.offset + (size_t)(kb / kMxRecBlocks) * g.rec_stride;
      const size_t codes = rec + g.atoms * kMxSfAtom + ((size_t)(kb & 3) * g.npad + n) * 16;
      if (kb < kbs) {
        *reinterpret_cast<uint4*>(A.image + codes + 16 * q) = c.own;
        *reinterpret_cast<uint4*>(A.rest + codes + 16 * q) = rest.own;
        if (q == (j & 3)) {
          *reinterpret_cast<uint4*>(A.image + codes + 64) = c.fifth;
          *reinterpret_cast<uint4*>(A.rest + codes + 64) = rest.fifth;
        }
      }
      const int l = threadIdx.x & 15;
      if (l < kMxDigitsX) *reinterpret_cast<uint32_t*>(A.image + rec + mx_sf_pos(n + l, 0)) = scales;
      if (any_wide && e.wide && kb < kbs) {
        // (zeros are zero under any scale but NaN, and the second image never holds that)
        for (int p = q; p < kMxDigitsX; p += 4) A.rest[rec + mx_sf_pos(n + p, kb)] = (uint8_t)(e.sf - mx_rest_shift(kMxDigitsX));
        if (q == 0) mx_mark_wide(A.wide + (size_t)s_tile[j] * A.wide_stride, kb);
      }
    }
  }
}
// The same from grouped fp16 rows (the expert-parallel receive side): a CTA per row tile.
__global__ void __launch_bounds__(128) k_mx_quant_rows(const __half* __restrict__ x16, int ldx, const RowTile* __restrict__ tiles,
                                                       const int* __restrict__ n_tiles_ptr, uint8_t* __restrict__ image,
                                                       uint8_t* __restrict__ rest_image, uint32_t* __restrict__ wide_masks, int wide_stride,
                                                       int K, int blocks, int recs) {
  const int n_tiles = *n_tiles_ptr, kbs = K / 32, q = threadIdx.x & 3;
  for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const RowTile rt = tiles[tile];
    const MxTileImage g = mx_tile_image<kMxDigitsX>(tile, rt.row0, rt.rows, recs);
    for (int base = 0; base < rt.rows * blocks; base += blockDim.x >> 2) {
      const int i = base + (threadIdx.x >> 2);
      const int r = i / blocks, kb = i % blocks;
      const bool real = i < rt.rows * blocks && kb < kbs;
      float v[8];
      const uint4 x = real ? *reinterpret_cast<const uint4*>(x16 + (size_t)(rt.row0 + r) * ldx + kb * 32 + q * 8) : make_uint4(0, 0, 0, 0);
      const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[c]));
        v[2 * c] = f.x;
        v[2 * c + 1] = f.y;
      }
      const MxEncoded e = mx_encode_block(v);
      if (real) {
        mx_store_block(image, g, r, kb, q, e.d, (int)e.sf);
        mx_store_block(rest_image, g, r, kb, q, e.rest, e.wide ? (int)(e.sf - mx_rest_shift(kMxDigitsX)) : -1);
        if (e.wide && q == 0) mx_mark_wide(wide_masks + (size_t)tile * wide_stride, kb);
      } else if (i < rt.rows * blocks) {
        mx_store_pad(image, g, r, kb, q);
      }
    }
  }
}

// ---- the contraction ------------------------------------------------------------------------------------------------
struct MxArgs {
  const uint8_t* weights;
  size_t expert_stride, mat_offset, bias_offset;
  MxLayout L;
  const uint8_t *x_img, *x_rest;  // the operand rows' images (digits, the digits after them), L.recs records
  const uint32_t* x_wide;         // record masks, wide_stride words per row tile
  uint8_t *a_img, *a_rest;        // GATED: the activated rows' images for the down projection ...
  uint32_t* a_wide;
  int a_blocks, a_recs;           // ... and its blocks and records
  int wide_stride;
  float* y;               // !GATED: output rows [rows, ldy]
  int ldy;
  const RowTile* tiles;
  const int* n_tiles_ptr;
  int max_tiles;          // places in `tiles`
  int* meta;              // meta[3] = device status word
  int has_bias, act, F;
  int stall;              // test hook: the copy role issues nothing, every wait of the other roles runs out
};

template <int D>
__device__ __forceinline__ float mx_sum(const uint32_t* d) {  // the digits' accumulators, radix 8
  float v = __uint_as_float(d[D - 1]);
#pragma unroll
  for (int p = D - 2; p >= 0; --p) v = fmaf(v, 0.125f, __uint_as_float(d[p]));
  return v;
}
// Eight rows' accumulators.  With a tile's last group of rows this reads up to 32 columns past the tile's own (of the other
// accumulators, or of the scales: not used).
template <int D>
__device__ __forceinline__ void mx_ld_group(uint32_t taddr, uint32_t (&r)[8 * D]) {
  tmem_ld32(taddr, *reinterpret_cast<uint32_t(*)[32]>(&r[0]));
  if constexpr (D == 5) tmem_ld8(taddr + 32, *reinterpret_cast<uint32_t(*)[8]>(&r[32]));
  else tmem_ld16(taddr + 32, *reinterpret_cast<uint32_t(*)[16]>(&r[32]));
}

// Is any record of the unit's row tile marked as holding wide blocks?  (After the kernel that writes the masks.)
__device__ __forceinline__ uint32_t mx_any_wide(const MxArgs& A, int tile) {
  uint32_t any = 0;
  for (int w = 0; w < mx_mask_words(A.L.recs); ++w) any |= __ldcg(A.x_wide + (size_t)tile * A.wide_stride + w);
  return any;
}

template <bool GATED>
__global__ void __launch_bounds__(kMxThreads, 1) k_mx(const MxArgs A) {
  extern __shared__ __align__(128) uint8_t mx_smem[];
  const MxLayout& L = A.L;
  constexpr int D = GATED ? kMxDigitsX : kMxDigitsA;
  // What the copies wait for is asked for at once, in front of the barriers and tensor memory: the list's length, its tallest tile, this
  // CTA's first tile (past the list's end: anything, not used).  One after the other, with the barriers between them, a step of 1
  // token took 0.6 us more, 16 tokens of the 128-expert 2048 x 768 layer 1.0.
  const int n_tiles = *A.n_tiles_ptr, tallest = A.meta[4];
  const RowTile first_tile = A.tiles[min((int)blockIdx.x / L.n_units, A.max_tiles - 1)];
  // How many columns the launch's tallest row tile takes decides the stage size: the tile list knows, the host does not.
  const int n_max = mx_npad<D>(max(1, tallest));
  const int stage_bytes = kMxARecMax + (n_max > 128 ? 2 : 1) * kMxSfAtom + (n_max * kMxRecBlocks * 16 + 127) / 128 * 128;
  const int NS = min(kMxMaxStages, (kMxSmem - kMxCtrl - kMxSlack) / stage_bytes);
  uint8_t* ctrl = mx_smem + kMxSmem - kMxCtrl;
  uint64_t* bars = reinterpret_cast<uint64_t*>(ctrl);
  const uint32_t smem_base = smem_u32(mx_smem), bar_base = smem_u32(bars);
  auto bar_full = [&](int s) { return bar_base + 8u * s; };
  auto bar_empty = [&](int s) { return bar_base + 8u * (kMxMaxStages + s); };
  auto bar_acc_full = [&](int b) { return bar_base + 8u * (2 * kMxMaxStages + b); };
  auto bar_acc_empty = [&](int b) { return bar_base + 8u * (2 * kMxMaxStages + 2 + b); };
  const uint32_t bar_drain = bar_base + 8u * (2 * kMxMaxStages + 4);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(ctrl + 8 * 32);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(ctrl + 8 * 32 + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kMxMaxStages; ++s) {
      mbar_init(bar_full(s), 1);
      mbar_init(bar_empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_acc_full(b), 1);
      mbar_init(bar_acc_empty(b), kMxEpilogueWarps);
    }
    mbar_init(bar_drain, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)),
                 "r"(kMxTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // The tile list is two launches old: only the token rows' image has to be waited for.
  const long n_items = (long)n_tiles * L.n_units;

  if (warp == 0) {
    // ------------------------------ producer ------------------------------
    if (lane == 0) {
      const int n = A.stall ? 0 : (int)n_items;
      bool ok = true;
      // What does not change over a unit's records is worked out once (twelve rows' copies after the wait: 0.9 us with the addresses worked out
      // for each, now 0.67).
      const int last = L.recs - 1, nb_last = L.rec_blocks(last);
      const uint8_t *w_src = nullptr, *x_src = nullptr;
      uint32_t w_full = 0, w_last = 0, x_full = 0, x_last = 0;
      MxTileImage g{};
      auto unit = [&](int item, const RowTile& rt) {
        const int tile = item / L.n_units, nt = item % L.n_units;
        g = mx_tile_image<D>(tile, rt.row0, rt.rows, L.recs);
        w_src = A.weights + (size_t)rt.expert * A.expert_stride + A.mat_offset + (size_t)nt * L.unit_bytes(0);
        w_full = (uint32_t)L.rec_bytes(nt, kMxRecBlocks);
        w_last = (uint32_t)L.rec_bytes(nt, nb_last);
        x_src = A.x_img + g.offset;
        x_full = (uint32_t)g.rec_stride;
        x_last = (uint32_t)(g.atoms * kMxSfAtom + nb_last * g.npad * 16);
      };
      // a stage's weights, and (separately) its token rows; both count on the stage's barrier
      auto weights = [&](int rec, int s) {
        const uint32_t bytes = rec == last ? w_last : w_full;
        mbar_expect_tx(bar_full(s), bytes + (rec == last ? x_last : x_full));
        bulk_load(smem_base + (uint32_t)s * stage_bytes, w_src + (size_t)rec * w_full, bytes, bar_full(s));
      };
      auto rows = [&](const uint8_t* image, int rec, int s) {
        bulk_load(smem_base + (uint32_t)s * stage_bytes + kMxARecMax, image + (size_t)rec * x_full, rec == last ? x_last : x_full, bar_full(s));
      };
      // as many records of the first unit as the ring holds are requested before the rows' images are complete
      int first = 0;
      if ((int)blockIdx.x < n) {
        unit(blockIdx.x, first_tile);
        for (; first < NS && first < L.recs; ++first) weights(first, first);
        griddep_wait();
        fence_async_global();  // the images were written by ordinary stores
        for (int rec = 0; rec < first; ++rec) rows(x_src, rec, rec);
      }
      int s = first == NS ? 0 : first, issued = first;
      uint32_t ph = first == NS ? 0u : 1u;  // a stage's first use waits for nothing
      auto put = [&](const uint8_t* image, int rec) {
        if (!mbar_wait(bar_empty(s), ph, abort_flag)) return false;
        weights(rec, s);
        rows(image, rec, s);
        ++issued;
        if (++s == NS) {
          s = 0;
          ph ^= 1u;
        }
        return true;
      };
      for (int item = blockIdx.x; ok && item < n; item += gridDim.x) {
        if (item != (int)blockIdx.x) unit(item, A.tiles[item / L.n_units]);
        // (the first word of the marks is on its way while the unit's records are asked for)
        const uint32_t* marks = A.x_wide + (size_t)(item / L.n_units) * A.wide_stride;
        uint32_t any_wide = __ldcg(marks);
        int rec = first;
        {
          // full records in a loop without a branch but the wait's
          bool here = false;
          const uint32_t bytes = w_full + x_full;
#pragma unroll 2
          for (; rec < last; ++rec) {
            if (!here && !mbar_wait(bar_empty(s), ph, abort_flag)) {
              ok = false;
              break;
            }
            const uint32_t bar = bar_full(s), dst = smem_base + (uint32_t)s * stage_bytes;
            ++s;
            ++issued;
            const bool wrap = s == NS;
            s = wrap ? 0 : s;
            ph ^= wrap ? 1u : 0u;
            here = mbar_test(bar_empty(s), ph);
            mbar_expect_tx(bar, bytes);
            bulk_load(dst, w_src + (size_t)rec * w_full, w_full, bar);
            bulk_load(dst + kMxARecMax, x_src + (size_t)rec * x_full, x_full, bar);
          }
        }
        for (; ok && rec < L.recs; ++rec) ok = put(x_src, rec);
        first = 0;
        // (Put together in front of the records, the wait for the words stood between two units, which shows where units are short: 512 experts of
        // 2048 x 256, 1000 tokens 160.8 us, now 156.7; 128 experts, 64 tokens of eight slots 51.3, now 50.4.)
        for (int w = 1; w < mx_mask_words(L.recs); ++w) any_wide |= __ldcg(marks + w);
        if (any_wide) {  // the records with wide blocks once more
          for (int w = 0; ok && w < mx_mask_words(L.recs); ++w)
            for (uint32_t bits = __ldcg(marks + w); ok && bits; bits &= bits - 1)
              ok = put(A.x_rest + g.offset, 32 * w + __ffs((int)bits) - 1);
        }
      }
      if (!ok) {
        // let the copies still in flight land before the CTA goes away
        for (int i = issued > NS ? issued - NS : 0; i < issued; ++i) {
          const long long t0 = clock64();
          while (!mbar_try(bar_full(i % NS), (uint32_t)((i / NS) & 1)) && clock64() - t0 < drain_budget()) {
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (warp-wide loop, one elected lane issues) ------------------------------
    const uint32_t tb = __shfl_sync(0xffffffffu, tmem_base, 0);
    uint32_t c = 0, it = 0;  // records, units so far
    bool ok = true;
    griddep_wait();  // this kernel's successor may count on everything before this kernel's predecessor being complete
    griddep_launch();
    int npad_before = 0, ahead_rows = 0;
    uint32_t ahead_wide = 0;
    const uint32_t stage16 = (uint32_t)stage_bytes >> 4, base16 = smem_base >> 4;
    for (long item = blockIdx.x; ok && item < n_items; item += gridDim.x, ++it) {
      const int tile = (int)(item / L.n_units), nt = (int)(item % L.n_units);
      if (!(it & 31u)) {
        // what it needs to know of the next 32 units, one per lane (with a load in front of every unit, 16 tokens of the
        // 128-expert 2048 x 768 layer took 2 us more)
        const long ahead = item + (long)lane * gridDim.x;
        if (ahead < n_items) {
          ahead_rows = A.tiles[ahead / L.n_units].rows;
          ahead_wide = mx_any_wide(A, (int)(ahead / L.n_units));
        }
      }
      const int rows = __shfl_sync(0xffffffffu, ahead_rows, (int)(it & 31u));
      const uint32_t any_wide = __shfl_sync(0xffffffffu, ahead_wide, (int)(it & 31u));
      const int npad = mx_npad<D>(rows), atoms = npad > 128 ? 2 : 1;
      const int r0 = L.rows(nt, 0), r1 = L.rows(nt, 1);
      const uint32_t buf = it & 1u, use = it >> 1;
      const uint32_t d0 = tb + (buf ? kMxTmemSf - 2u * (uint32_t)npad : 0u), d1 = d0 + (uint32_t)npad;
      ok = mbar_wait_warp(bar_acc_empty(buf), (use & 1u) ^ 1u, abort_flag);
      if (ok && it && npad_before + npad > (int)kMxTmemSf / 2)  // the unit before this one lies in the way
        ok = mbar_wait_warp(bar_acc_empty(buf ^ 1u), ((it - 1u) >> 1) & 1u, abort_flag);
      if (!ok) break;
      npad_before = npad;
      tc_fence_after();
      int s = (int)(c % (uint32_t)NS);
      uint32_t ph = c / (uint32_t)NS & 1u;
      // One lane takes the unit's records by itself.  Its instructions are what a record takes once the stages are full (the tensor cores
      // wait for it), so the operands' descriptors are worked out per unit and a record adds its stage's address, which is their
      // low bits.  Records of the ordinary form (both halves, one atom of row scales, four blocks) have a loop without any
      // branch but the wait's, which asks for the next stage beforehand: 430 -> 230 clocks a record.
      if (elect_one()) {
        const uint32_t all = (uint32_t)(r0 + r1), idesc0 = umma_idesc_mxf4(npad, 0), idesc1 = umma_idesc_mxf4(npad, 2);
        const uint32_t a0 = (uint32_t)r0 << 16, a1 = (uint32_t)(2 * r0) | (uint32_t)r1 << 16;
        const uint32_t b0 = (uint32_t)(kMxARecMax / 16 + atoms * (kMxSfAtom / 16)) | (uint32_t)npad << 16;
        constexpr uint32_t kSf = 8u << 16, kHi = 8u | 1u << 14;  // groups of 8 rows 128 bytes apart; descriptor version
        auto desc = [](uint32_t lo) { return (uint64_t)kHi << 32 | lo; };
        uint32_t at = base16 + (uint32_t)s * stage16, sf = tb + kMxTmemSf + (c & 1u) * 16u;
        auto advance = [&]() {
          at += stage16;
          ++s;
          const bool wrap = s == NS;
          s = wrap ? 0 : s;
          at = wrap ? base16 : at;
          ph ^= wrap ? 1u : 0u;
          sf ^= 16u;
        };
        // the MMAs of a record in stage s (`add` 0: the accumulators start here)
        auto record = [&](int rec, uint32_t add) {
          if (!mbar_wait(bar_full(s), ph, abort_flag)) return false;
          tc_fence_after();
          const int nb = L.rec_blocks(rec);
          const uint32_t a_sf = at + (uint32_t)nb * all + kSf, b_sf = at + kMxARecMax / 16 + kSf;
          tmem_cp_scales(sf, desc(a_sf));
          if (r1) tmem_cp_scales(sf + 4, desc(a_sf + kMxSfAtom / 16));
          tmem_cp_scales(sf + 8, desc(b_sf));
          if (atoms > 1) tmem_cp_scales(sf + 12, desc(b_sf + kMxSfAtom / 16));
          umma_mxf4_ss(d0, desc(at + a0), desc(at + b0), idesc0, sf, sf + 8, add);
          if (r1) umma_mxf4_ss(d1, desc(at + a1), desc(at + b0), idesc0, sf + 4, sf + 8, add);
          if (nb > 2) {
            const uint32_t a = at + 2 * all, b = at + b0 + 2 * (uint32_t)npad;
            umma_mxf4_ss(d0, desc(a + a0), desc(b), idesc1, sf, sf + 8, 1u);
            if (r1) umma_mxf4_ss(d1, desc(a + a1), desc(b), idesc1, sf + 4, sf + 8, 1u);
          }
          umma_commit(bar_empty(s));
          advance();
          return true;
        };
        int rec = 0;
        if (r1 && atoms == 1) {
          const int ordinary = L.rec_blocks(L.recs - 1) == kMxRecBlocks ? L.recs : L.recs - 1;
          const uint32_t a_sf = kMxRecBlocks * all + kSf, b_sf = kMxARecMax / 16 + kSf;
          const uint32_t a2 = a0 + 2 * all, a3 = a1 + 2 * all, b2 = b0 + 2 * (uint32_t)npad;
          bool here = false;
#pragma unroll 2
          for (; rec < ordinary; ++rec) {
            if (!here && !mbar_wait(bar_full(s), ph, abort_flag)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t now = at, sf_now = sf, bar_now = bar_empty(s);
            advance();
            here = mbar_test(bar_full(s), ph);  // (of a stage that nobody fills any more: not used)
            tmem_cp_scales(sf_now, desc(now + a_sf));
            tmem_cp_scales(sf_now + 4, desc(now + a_sf + kMxSfAtom / 16));
            tmem_cp_scales(sf_now + 8, desc(now + b_sf));
            umma_mxf4_ss(d0, desc(now + a0), desc(now + b0), idesc0, sf_now, sf_now + 8, rec ? 1u : 0u);
            umma_mxf4_ss(d1, desc(now + a1), desc(now + b0), idesc0, sf_now + 4, sf_now + 8, rec ? 1u : 0u);
            umma_mxf4_ss(d0, desc(now + a2), desc(now + b2), idesc1, sf_now, sf_now + 8, 1u);
            umma_mxf4_ss(d1, desc(now + a3), desc(now + b2), idesc1, sf_now + 4, sf_now + 8, 1u);
            umma_commit(bar_now);
          }
        }
        for (; ok && rec < L.recs; ++rec) ok = record(rec, rec ? 1u : 0u);
        if (any_wide)  // the records with wide blocks once more
          for (int w = 0; ok && w < mx_mask_words(L.recs); ++w)
            for (uint32_t bits = __ldcg(A.x_wide + (size_t)tile * A.wide_stride + w); ok && bits; bits &= bits - 1)
              ok = record(32 * w + __ffs((int)bits) - 1, 1u);
        if (ok) umma_commit(bar_acc_full(buf));
      }
      ok = __all_sync(0xffffffffu, ok);
      c += (uint32_t)L.recs;
      if (any_wide)
        for (int w = 0; w < mx_mask_words(L.recs); ++w) c += (uint32_t)__popc(__ldcg(A.x_wide + (size_t)tile * A.wide_stride + w));
    }
    // everything issued has to retire before tensor memory is freed
    if (lane == 0) {
      umma_commit(bar_drain);
      const long long t0 = clock64();
      while (!mbar_try(bar_drain, 0) && clock64() - t0 < drain_budget()) {
      }
    }
    __syncwarp();
  } else {
    // ------------------------------ epilogue ------------------------------
    const int quarter = warp & 3, grp = (warp - 2) >> 2;  // tensor-memory lanes 32 * quarter ..; every second group of 8 rows
    griddep_wait();  // output rows of an earlier launch of this step are read until then
    uint32_t it = 0;
    for (long item = blockIdx.x; item < n_items; item += gridDim.x, ++it) {
      const int tile = (int)(item / L.n_units), nt = (int)(item % L.n_units);
      const RowTile rt = A.tiles[tile];
      const int halves = L.halves(nt);
      const float* bias = reinterpret_cast<const float*>(A.weights + (size_t)rt.expert * A.expert_stride + A.bias_offset);
      const uint32_t buf = it & 1u, use = it >> 1;
      const uint32_t npad = (uint32_t)mx_npad<D>(rt.rows);
      const uint32_t t_acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (buf ? kMxTmemSf - 2u * npad : 0u);
      const int groups = (rt.rows + 7) >> 3;
      const int n = (GATED ? nt * 128 : nt * 256) + quarter * 32 + lane;
      float b0 = 0.f, b1 = 0.f;
      if (A.has_bias) {
        if (GATED) {
          if (n < L.N) {
            b0 = bias[A.F + n];
            b1 = bias[n];
          }
        } else {
          if (n < L.N) b0 = bias[2 * A.F + n];
          if (n + 128 < L.N) b1 = bias[2 * A.F + n + 128];
        }
      }
      if (!mbar_wait_warp(bar_acc_full(buf), use & 1u, abort_flag)) break;
      tc_fence_after();
      if (GATED) {
        const bool live = nt * 128 + quarter * 32 < L.N;  // N is a multiple of 32: a warp's features are real or not as one
        constexpr int DA = kMxDigitsA;
        const MxTileImage g = mx_tile_image<DA>(tile, rt.row0, rt.rows, A.a_recs);
        const int kb = nt * 4 + quarter;
        const size_t rec_at = g.offset + (size_t)(kb / kMxRecBlocks) * g.rec_stride;
        uint8_t *rec = A.a_img + rec_at, *rest = A.a_rest + rec_at;
        const size_t codes_at = g.atoms * kMxSfAtom + (size_t)(kb & 3) * g.npad * 16;
        const bool odd = lane & 1;
        // neighbouring lanes hold neighbouring columns: the even one packs the even row's bytes, the odd one the odd row's
        auto pack = [&](uint32_t w) {
          const uint32_t o = __shfl_xor_sync(0xffffffffu, w, 1);
          return odd ? ((o >> 4) & 0x0F0F0F0Fu) | (w & 0xF0F0F0F0u) : (w & 0x0F0F0F0Fu) | ((o & 0x0F0F0F0Fu) << 4);
        };
        // the next six digits of two rows, into the columns of row `to` (nothing when it is past the tile)
        auto digits = [&](float (&v)[2], uint8_t* codes, int to) {
          uint32_t w = 0, w2 = 0;  // byte p: digit p of both rows (low nibble: the even one)
#pragma unroll
          for (int p = 0; p < 4; ++p) w |= mx_digit(v[0], v[1]) << (8 * p);
#pragma unroll
          for (int p = 0; p < DA - 4; ++p) w2 |= mx_digit(v[0], v[1]) << (8 * p);
          w = pack(w);
          w2 = pack(w2);
          if (to < rt.rows) {
            uint8_t* dst = codes + (size_t)DA * to * 16 + (lane >> 1);
#pragma unroll
            for (int p = 0; p < 4; ++p) dst[16 * p] = (uint8_t)(w >> (8 * p));
#pragma unroll
            for (int p = 0; p < DA - 4; ++p) dst[16 * (4 + p)] = (uint8_t)(w2 >> (8 * p));
          }
        };
        for (int gr = grp; gr < groups; gr += 2) {
          uint32_t rg[8 * D], ru[8 * D];
          mx_ld_group<D>(t_acc + (uint32_t)gr * 8 * D, rg);
          mx_ld_group<D>(t_acc + npad + (uint32_t)gr * 8 * D, ru);
          tmem_ld_wait();
          if (!live) continue;
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            const int r = gr * 8 + i;
            if (r >= rt.rows) break;
            float v[2];
            uint32_t sf[2];
            bool wide[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              v[j] = gated_act(mx_sum<D>(rg + D * (i + j)) + b0, mx_sum<D>(ru + D * (i + j)) + b1, A.act);
              float inv;
              sf[j] = mx_scale_of(__reduce_max_sync(0xffffffffu, __float_as_uint(v[j]) & 0x7FFFFFFFu), inv);
              v[j] *= inv;
              constexpr float kFixed = 1048576.f;  // the sum in fixed point: one instruction over the warp
              const uint32_t q = (uint32_t)(fminf(v[j] * v[j], mx_wide_clip2<DA>()) * kFixed);
              wide[j] = __reduce_add_sync(0xffffffffu, q) < (uint32_t)(mx_wide_limit<DA>() * kFixed) && r + j < rt.rows &&
                        sf[j] >= mx_rest_shift(DA) && sf[j] != 255u;
            }
            const int my = r + (odd ? 1 : 0);
            digits(v, rec + codes_at, my);
            if (my < rt.rows && lane < 2 * DA) {
              const int col = DA * my + (lane >> 1);
              rec[mx_sf_pos(col, kb)] = (uint8_t)(odd ? sf[1] : sf[0]);
              if (kb + 1 < A.a_blocks && (kb + 1) * 32 >= A.F) rec[mx_sf_pos(col, kb + 1)] = 0;  // the padding block
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)  // a power of two, zeros: nothing is left
              wide[j] = wide[j] && __ballot_sync(0xffffffffu, (__float_as_uint(v[j]) & 0x7FFFFFFFu) != 0) != 0;
            if (lane < 2 * DA && r + lane / DA < rt.rows)
              *reinterpret_cast<uint4*>(rest + codes_at + (size_t)(DA * r + lane) * 16) = make_uint4(0, 0, 0, 0);
            if (wide[0] || wide[1]) {
              const bool mine = odd ? wide[1] : wide[0];
              __syncwarp();
              digits(v, rest + codes_at, mine ? my : rt.rows);
              if (mine && lane < 2 * DA) rest[mx_sf_pos(DA * my + (lane >> 1), kb)] = (uint8_t)((odd ? sf[1] : sf[0]) - mx_rest_shift(DA));
              if (lane == 0) mx_mark_wide(A.a_wide + (size_t)tile * A.wide_stride, kb);
            }
          }
        }
      } else {
        for (int w = grp; w < halves * groups; w += 2) {
          const int half = w >= groups ? 1 : 0, gr = w - half * groups;
          uint32_t rd[8 * D];
          mx_ld_group<D>(t_acc + (half ? npad : 0u) + (uint32_t)gr * 8 * D, rd);
          tmem_ld_wait();
          const int col = n + 128 * half;
          if (col >= L.N) continue;
          float* out = A.y + (size_t)(rt.row0 + gr * 8) * A.ldy + col;
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (gr * 8 + i < rt.rows) out[(size_t)i * A.ldy] = mx_sum<D>(rd + D * i) + (half ? b1 : b0);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_acc_empty(buf));
    }
  }

  // ------------------------------ teardown ------------------------------
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) atomicOr(&A.meta[3], kDevErrWaitTimeout);
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kMxTmemCols) : "memory");
  }
}

inline cudaError_t mx_prepare_device() {
  cudaError_t e = cudaFuncSetAttribute(k_mx<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMxSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_mx<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMxSmem);
  return e;
}

}  // namespace csk
