// C ABI of the MoE layer (see include/csk_moe.h): handle, weight repack,
// host- and device-buffer entry points, expert-parallel stages.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <new>

#include "csk_common.cuh"
#include "csk_kernels.cuh"
#include "csk_few16.cuh"
#include "csk_kquant.cuh"
#include "csk_mx.cuh"
#include "csk_router_tc.cuh"
#include "csk_tile.cuh"
#include "csk_tile2.cuh"
#include "csk_pair16.cuh"

using namespace csk;

namespace {
std::mutex g_err_mu;
std::string g_create_error;
}  // namespace

struct csk_moe_layer {
  csk_moe_config cfg{};
  int E = 0, k = 0, H = 0, F = 0, e0 = 0, Eloc = 0;
  MxLayout Lgu{}, Ld{};     // block-scaled kernel's layout
  TileLayout Tgu{}, Td{};   // tensor-core kernel's layout (a second copy of the codes)
  size_t off_gu = 0, off_d = 0, off_tgu = 0, off_td = 0, off_bias = 0, off_meta = 0, expert_stride = 0;
  uint8_t* d_weights = nullptr;
  uint8_t* d_resident = nullptr;  // [Eloc] flags on the device
  std::vector<uint8_t> resident;
  uint8_t* d_stage = nullptr;     // raw 17-byte blocks during load / unpack
  uint8_t* d_stage2 = nullptr;    // second staging area (bulk load)
  size_t stage_bytes = 0;
  bool w16 = false;            // fp16 weights: tensor-core kernel only, no streaming layout
  float* d_unit_router = nullptr;  // dense FFN (E = k = 1): (expert 0, weight 1) for every token

  float* d_wg = nullptr;   // [E,H]
  float* d_wg_few = nullptr;   // the same repacked for the router kernel's two chunk widths
  float* d_wg_many = nullptr;
  int* d_route_cnt = nullptr;  // [max_T] tickets of the router's token blocks (zero between launches)
  float2* d_part = nullptr;    // [part_rows,E] partial sums of the fast router, one row per (token, part of H)
  float* d_hn2 = nullptr;      // [part_rows] the parts' shares of the token rows' sums of squares
  int64_t part_rows = 0;
  float* d_wnorm = nullptr;    // [E] 2-norms of the gate rows
  int* d_fb_list = nullptr;    // [max_T] tokens the fast router could not certify
  int* d_fb = nullptr;         // [0] entries of d_fb_list, [1] ticket of its reset, [2..3] 64-bit running total
  uint8_t* d_wg_tc = nullptr;      // gate rows as digits for the tensor-core router, their scales and norms
  float* d_wg_tc_scale = nullptr;
  float* d_wnorm_tc = nullptr;
  int router_mode = CSK_ROUTER_AUTO;
  RouterWave router_waves[kMaxExperts / 32 + 1] = {};  // by groups of 32 experts
  int64_t routed_tokens = 0;   // tokens routed in certified mode since creation
  float* d_logits = nullptr;  // [max_T,E] router scratch
  float* d_rbias = nullptr;
  bool router_set = false, has_rbias = false;
  // expert parallelism over peer memory
  int p2p_rank = -1, p2p_world = 0;
  size_t back_tail = 0;               // floats of d_back in front of its sync area
  int* d_p2p_epoch = nullptr;         // device: generations of the three flag barriers of a step
  RowOrigin* d_info = nullptr;        // [max_rows] origin of every received row
  float* d_back = nullptr;            // [max_T*k, H] output rows returned for this rank's pairs
  float** d_row_ptr = nullptr;        // [max_rows] where each received row's output goes
  int* d_p2p_base = nullptr;          // [E]
  __half** d_peer_x16 = nullptr;      // [world] every rank's row buffer (own entry: d_x16)
  RowOrigin** d_peer_info = nullptr;  // [world]
  float** d_peer_back = nullptr;      // [world]
  std::vector<void*> ipc_opened;      // peer mappings to close
  bool pdl = false;  // launch the kernels with programmatic dependent launch (unless they are timed one by one)
  bool debug_stall = false;  // test hooks: the next expert (router) launch's copy role issues nothing (one shot)
  bool debug_stall_router = false;

  float* d_norm_w = nullptr;   // [H] weight of the RMSNorm in front of the router (csk_moe_set_ffn_norm)
  float* d_normed = nullptr;   // [max_T,H] its output
  float* d_shared_out = nullptr;  // [max_T,H] the shared expert's rows of a block forward
  cudaEvent_t ev_shared_fork = nullptr, ev_shared_join = nullptr;
  float norm_eps = 1e-5f;
  int64_t max_T = 0, max_rows = 0;
  int max_tiles = 0;
  float* d_hidden = nullptr;  // [max_T,H] staging for the host entry points
  float* d_router = nullptr;  // [max_T,k,2]
  float* d_router_phys = nullptr;  // the same with logical expert ids replaced by slots (expert-parallel dispatch)
  int* d_slot_map = nullptr;       // [2][E]: primary slot, replica slot (or -1) of each logical expert
  bool has_slot_map = false;
  int E_router = 0;                // experts the router scores (= E without a slot map)
  float* d_out = nullptr;     // [max_T,H]
  __half* d_x16 = nullptr;    // [max_rows+pad, ldx]
  __half* d_a16 = nullptr;    // [max_rows+pad, lda]
  float* d_y = nullptr;       // [max_rows, H]
  int ldx = 0, lda = 0;
  int* d_hist = nullptr;       // [kHistBlocks][E + 1] row counts of a large batch's plan
  int* d_counts = nullptr;       // [E]
  int* d_offsets = nullptr;      // [E+1]
  int* d_cursor = nullptr;       // [E]
  int* d_row_of_pair = nullptr;  // [max_rows]
  int4* d_places = nullptr;      // [min(max_rows, kOneBlockPairs)] where the pairs of a small batch go (block-scaled kernel)
  ExpertTiles* d_expert_tiles = nullptr;  // [E] where the experts' row tiles are (block-scaled kernel)
  uint8_t* d_ximg = nullptr;     // the block-scaled kernel's operands: token rows and activated rows as digit images
  uint8_t* d_aimg = nullptr;
  size_t ximg_rest = 0, aimg_rest = 0;  // where the images of the digits after the first begin
  int64_t mx_rows = 0;           // rows the images hold
  uint32_t* d_wide = nullptr;    // [max_tiles][mask words of token rows, of activated rows]
  std::vector<uint8_t*> mx_outgrown;
  int* d_out_row_map = nullptr;  // [max_rows] (expert-parallel receive side)
  int* d_seg = nullptr;          // [2*1024+2] segment plan (expert-parallel receive side)
  RowTile* d_tiles = nullptr;
  int* d_meta = nullptr;  // 16 ints: [0..7] rewritten by every permutation, [8] the router's status word
  int* h_meta = nullptr;  // pinned mirror
  int64_t* h_counts64 = nullptr;
  float* h_staged = nullptr;       // page-locked staging of small host batches, of h_staged_bytes: first in, then out
  size_t h_staged_bytes = 0;

  cudaStream_t stream = nullptr;
  // the host entry point's pipeline: copy-in and copy-out streams beside `stream`, one event pair per pass
  cudaStream_t stream_in = nullptr, stream_out = nullptr;
  static constexpr int kMaxPasses = 8;
  cudaEvent_t ev_in[kMaxPasses]{}, ev_done[kMaxPasses]{}, ev_free = nullptr;
  int* d_carry = nullptr;      // [1 + E]: sticky status and per-expert row totals over the passes of one call
  bool carry_active = false;   // the combine kernel folds each pass into d_carry
  bool counts_in_carry = false;  // the last call's counters are the totals in d_carry
  cudaEvent_t ev[8]{};
  bool timing = false;
  csk_moe_timings last{};
  int path = CSK_PATH_AUTO;
  int sm_count = 148;
  TileState tile;  // tensor maps and launch state of the tensor-core path
  PairState pair;  // the CTA-pair kernel, where clusters of two can be launched

  // Small batches are launch-bound: their kernel sequence is captured once per
  // (T, buffers, stream) into a CUDA graph and replayed.
  struct GraphEntry {
    int64_t T;
    const void *hidden, *router_in;
    void *router_out, *out;
    const void* host_router;
    cudaStream_t stream;
    cudaGraphExec_t exec;
  };
  std::vector<GraphEntry> graphs;
  bool use_graphs = true;

  std::string err;
  int64_t last_T = 0;
  int n_marks = 0;
  bool last_routed = false;
  cudaStream_t last_stream = nullptr;
};

namespace {

// Host buffers of at most so many bytes each way go through page-locked staging of the handle's own if they are pageable.  32
// tokens of the 32-expert layer: 200 -> 169 us a call, 80 (0.9 MB) 277 -> 268 (copies of pageable memory wait for the device, and the status had a
// wait of its own).  One area for both ways: with two, creating a layer of 8192 tokens took 13.5 ms, with one 11.1.
// The last kernel writes results, routing and status word there itself: copies by the driver, three of them behind the kernels, cost 13 to
// 18 us more (1 token of that layer 72 -> 56, 4 95 -> 78, 16 140 -> 127, 32 182 -> 167, 80 280 -> 262).
constexpr size_t kStagedMax = 1 << 20;
// On the way in the driver takes up to 64 KB itself without a wait, and a second piece, whose host copy runs beside the first one's way
// to the device, costs a launch.  By the driver / one piece / two, us: 2 tokens of that layer (22 KB) 76 / 78 / 89, 4 (45 KB) 97.5 / 103 / 107, 8 (90
// KB) 134 / 129 / 131, 16 (180 KB) 155 / 148 / 151, 32 (360 KB) 176 / 173 / 169; 8 experts of 512 x 512, 8 tokens (16 KB) 51 / 51 / 63, 32 (64 KB)
// 60 / 65 / 67, 80 (160 KB) 80 / 73 / 77, 200 (400 KB) 101 / 99 / 92.
constexpr size_t kStagedInMin = 64 << 10, kStagedTwoPieces = 256 << 10;
// Page-locked buffers need none on the way in (32 tokens 160 without, 173 with).  On the way out a copy into them has to wait for the status
// word, so that a call that fails leaves them alone: up to so many bytes that wait, and the copies, are dearer than a host copy.
// The layer above, direct / staged, us: 1 token (11 KB) 62.6 / 47.0, 8 (90 KB) 114.7 / 101.1, 16 (180 KB) 134.0 / 121.9, 24 (270 KB) 139.0 / 130.9, 32
// (361 KB) 145.5 / 139.5, 50 (564 KB) 155 / 166, 80 175 / 206; 128 experts of 2048 x 768, 30 tokens (240 KB) 122.4 / 111.0, 100 (800 KB) 159 / 186.
// A row of 24 handles called in turn, whose staging areas are cold, as a model's layers are: 8 experts of 2880 x 2880, top-4, 16 tokens 97 / 89, 24 100 / 97, 28
// (324 KB) 101 / 101, 32 102 and 111 / 107 (two runs); 32 of 2048 x 768, top-8, 32 tokens (266 KB) 92 / 89, 42 (350 KB) 101 / 95.5, 47 (392 KB) 104 / 106.
constexpr size_t kStagedLockedMax = 384 << 10;

int wide_stride(const csk_moe_layer* L) { return mx_mask_words(L->Lgu.recs) + mx_mask_words(L->Ld.recs); }

int fail(csk_moe_layer* L, int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (L) {
    L->err = buf;
  } else {
    std::lock_guard<std::mutex> lk(g_err_mu);
    g_create_error = buf;
  }
  return code;
}

#define CSK_CUDA(L, call)                                                                    \
  do {                                                                                       \
    cudaError_t _e = (call);                                                                 \
    if (_e != cudaSuccess)                                                                   \
      return fail(L, CSK_ERR_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(_e),   \
                  __FILE__, __LINE__);                                                       \
  } while (0)

// Bytes of an expert's tensor-core tiles in the order of the file images.  The first staging area holds them, so that images can be
// written and read when the device is full.
size_t image_part_bytes(const csk_moe_layer* L) { return L->off_bias - L->off_tgu; }

int grid_for(size_t work_items, int threads, int cap) {
  size_t b = (work_items + threads - 1) / threads;
  return (int)std::max<size_t>(1, std::min<size_t>(b, (size_t)cap));
}

cudaStream_t pick(csk_moe_layer* L, void* s) { return s ? (cudaStream_t)s : L->stream; }

// Launches of the handle are programmatic dependents for as long as this lives (unless they are timed one by one).
struct PdlScope {
  csk_moe_layer* L;
  explicit PdlScope(csk_moe_layer* l) : L(l) { L->pdl = !L->timing; }
  ~PdlScope() { L->pdl = false; }
};

struct StageTimer {
  csk_moe_layer* L;
  cudaStream_t s;
  int n = 0;
  StageTimer(csk_moe_layer* l, cudaStream_t st) : L(l), s(st) {}
  void mark() {
    if (L->timing && n < 8) cudaEventRecord(L->ev[n++], s);
  }
};

// ---- the stages ----------------------------------------------------------

int launch_router(csk_moe_layer* L, const float* d_hidden, int64_t T, float* d_router,
                  cudaStream_t s) {
  if (!L->router_set) return fail(L, CSK_ERR_INVALID, "router weights were never set");
  if (reinterpret_cast<uintptr_t>(d_hidden) % 16)
    return fail(L, CSK_ERR_INVALID, "hidden states must be 16-byte aligned");
  RouterArgs a{};
  a.hidden = d_hidden;
  a.bias = L->has_rbias ? L->d_rbias : nullptr;
  a.logits = L->d_logits;
  a.router_out = d_router;
  a.counters = L->d_route_cnt;
  a.status = L->d_meta + 8;
  a.T = (int)T;
  a.H = L->H;
  a.E = L->E_router;
  a.k = L->k;
  a.sigmoid = L->cfg.sigmoid_gating;
  // Of a handful of tokens the certified pass (three launches: sliced FMA logits, certification, chain over the few tokens it
  // could not separate) spreads the columns over the machine, where a chain is alone.  A layer's step over fresh inputs, chain / certified, us: 128
  // experts, 2880 columns, 1 token 35.4 / 30.9, 2 43.3 / 38.9, 4 59.1 / 55.9, 8 84.8 / 83.6, 16 126.8 / 127.3; 128 x 2048, 1 26.8 / 24.2, 4 35.9 / 36.3, 6
  // 40.0 / 41.1.  (Rows that it cannot separate, like rows of zeros without a bias, cost both.)
  constexpr int64_t kCertifiedMaxTokens = 4;
  // With many tokens the chain is held by its arithmetic, token x expert; the certified pass on the tensor cores costs
  // little per token, but four launches and the chain of the few percent it cannot separate.  Chain / certified, us, normal
  // rows: 128 experts, 2880 columns: 64 tokens 13 / (FMA pass) 25, 512 26 / 34, 1024 47 / 35, 2048 95 / 43; 128 x 2048: 600 29 / 32, 1000 36 / 32; 64 x 2880:
  // 1024 26 / 34, 2048 48 / 44, 3000 96 / 49; 256 x 2880: 256 38 / 39, 512 54 / 39; 512 x 2048: 256 45 / (FMA) 95, 512 79 / 44; 128 x 512: 1000 14 /
  // 21; 32 x 2880: 4096 47 / 104, 8192 90 / 146
  // (a digit matrix has 128 rows whatever the experts).  The line is a compromise over the columns, by which a chain goes and the certified pass hardly:
  // at 1024 tokens of 128 experts the chain costs 12 us more of 2880 columns, 4 of 2048, and 7 less of 512, so that the two meet below the line (700
  // tokens) for wide layers and beyond it for narrow ones; with 256 experts of 2880 columns they meet at half of it.  From 512 experts on (few
  // tokens, many digit matrices) it is at twice as many pairs, where the chain is 35 us behind (512 x 2048, 512 tokens).  Below the line the certified
  // mode takes the FMA pass, which is slower than the chain everywhere.
  const int groups = (L->E_router + 31) / 32;
  const int64_t tensor_min_work = groups >= 16 ? 8192 : 4096;  // tokens x groups of 32 experts
  const bool few = T <= kCertifiedMaxTokens, many = groups > 1 && T * groups >= tensor_min_work;
  const RouterWave router_wave = L->router_waves[groups];
  if (L->router_mode == CSK_ROUTER_CHAIN || (L->router_mode == CSK_ROUTER_AUTO && !few && !many)) {
    launch_router_logits<true>(a, L->d_wg_few, L->d_wg_many, router_wave, s, L->pdl);
    CSK_CUDA(L, cudaGetLastError());
    L->last.launches += 1;
    return CSK_OK;
  }
  // (the kernels of a large batch's pass start while the one before them ends, too: the second launch for the list is then
  // nearly free, 5 us otherwise)
  const bool pdl = L->pdl || (many && !L->timing);
  // fast logits with error bounds; tokens whose selection the bounds do not certify are listed ...
  FinishRouterArgs g{};
  g.part = L->d_part;
  g.hn2 = L->d_hn2;
  g.bias = a.bias;
  g.router_out = d_router;
  g.fb_list = L->d_fb_list;
  g.fb_count = L->d_fb;
  g.T = (int)T;
  g.H = L->H;
  g.E = L->E_router;
  g.k = L->k;
  g.sigmoid = L->cfg.sigmoid_gating;
  if (many) {
    RouterTcArgs f{};
    f.hidden = d_hidden;
    f.w = L->d_wg_tc;
    f.w_scale = L->d_wg_tc_scale;
    f.part = L->d_part;
    f.hn2 = L->d_hn2;
    f.status = a.status;
    f.T = (int)T;
    f.H = L->H;
    f.E = L->E_router;
    f.stall = L->debug_stall_router;
    L->debug_stall_router = false;
    const int token_tiles = ceil_div((int)T, kRtTokens), rg = rt_groups(L->E_router);
    // one CTA fits an SM: as many parts of the hidden dimension as one wave holds
    int parts = std::min(std::min(rt_blocks(L->H), kFastMaxParts), std::max(1, L->sm_count / (token_tiles * rg)));
    while (parts > 1 && T * parts > L->part_rows) --parts;
    launch_k(k_router_tc, dim3((unsigned)token_tiles, (unsigned)rg, (unsigned)parts), dim3(kRtThreads), kRtSmem, s, pdl, f);
    g.wnorm = L->d_wnorm_tc;
    g.parts = parts;
    g.slices = rt_blocks(L->H);
    g.coef_prefix = kRtPrefixCoef;
    g.coef_norm = kRtNormCoef;
    launch_k(k_router_finish_many, dim3((unsigned)ceil_div((int)T, kFinishWarps)), dim3(32 * kFinishWarps),
             sizeof(float) * 2 * kFinishWarps * L->E_router, s, pdl, g);
  } else {
    FastRouterArgs f{};
    f.hidden = d_hidden;
    f.wg = L->d_wg;
    f.part = L->d_part;
    f.hn2 = L->d_hn2;
    f.T = (int)T;
    f.H = L->H;
    f.E = L->E_router;
    const int tpw = T <= 4 ? 1 : T <= 8 ? 2 : T <= 16 ? 4 : T <= 32 ? 8 : 16;
    const int token_blocks = (int)((T + 4 * tpw - 1) / (4 * tpw));
    // enough parts of the hidden dimension to put a CTA on every SM (few tokens); one part once
    // the token blocks alone fill the machine
    int parts = std::min(std::min(fast_router_slices(L->H), kFastMaxParts),
                         std::max(1, (L->sm_count + token_blocks * groups - 1) / (token_blocks * groups)));
    while (parts > 1 && T * parts > L->part_rows) --parts;
    const dim3 grid((unsigned)token_blocks, (unsigned)groups, (unsigned)parts);
    const size_t smem = fast_router_smem(tpw);
    switch (tpw) {
      case 1: launch_k(k_router_fast<1>, grid, dim3(128), smem, s, pdl, f); break;
      case 2: launch_k(k_router_fast<2>, grid, dim3(128), smem, s, pdl, f); break;
      case 4: launch_k(k_router_fast<4>, grid, dim3(128), smem, s, pdl, f); break;
      case 8: launch_k(k_router_fast<8>, grid, dim3(128), smem, s, pdl, f); break;
      default: launch_k(k_router_fast<16>, grid, dim3(128), smem, s, pdl, f); break;
    }
    g.wnorm = L->d_wnorm;
    g.parts = parts;
    launch_k(k_router_finish, dim3((unsigned)T), dim3(kFinishThreads), finish_smem_bytes(parts, L->E_router), s, pdl, g);
  }
  // ... and go through the order-faithful chain: its blocks walk the list and leave at once when it is empty
  RouterArgs b = a;
  b.token_list = L->d_fb_list;
  b.n_list = L->d_fb;
  b.fb_done = L->d_fb + 1;
  b.fb_total = reinterpret_cast<unsigned long long*>(L->d_fb + 2);
  b.list_max = INT32_MAX;
  const int64_t wave = std::max(1, 4 * (router_wave.blocks / groups));  // tokens of one wave of four-token blocks
  if (many) {
    // How long the list is the data decide: 2 % of the tokens of normal rows, half of them with a few channels at 1000 times
    // the others, all where rows repeat a value (padding).  Blocks of few tokens are quicker for a short list: the first
    // launch has them for a 32nd of the tokens (at least one wave of four-token blocks, at most two) and takes up to two rounds of
    // that.  The second has up to 32 tokens a block and takes any longer list; each leaves the other's lists alone.  2880 columns, one
    // launch / two (the chain of all tokens), us: 128 experts, 8192 normal rows 105 / 107 (326), nine channels at 1000 times the others 120 / 123,
    // every tenth row zero 197 / 138, every second 564 / 277, every row 990 / 463; 2048 normal rows 43.6 / 46.5 (92), every row zero 241 / 126;
    // 1024 35.5 / 39.0 (47), every row zero 128 / 72; 256 experts, 2048 normal rows 73 / 75 (185), every tenth zero 161 / 96, every row 965 / 281.  (With room
    // for a quarter of a wave: 2048 tokens of eight slots, whose lists are longer, 284 -> 291 for the step.)
    const int few_slots = (int)std::min(2 * wave, std::max(wave, T / 32));
    b.list_max = 2 * few_slots;
    launch_router_logits<true>(b, L->d_wg_few, L->d_wg_many, router_wave, s, pdl, few_slots);
    if (T > b.list_max) {
      b.list_over = b.list_max;
      b.list_max = INT32_MAX;
      launch_router_logits<true>(b, L->d_wg_few, L->d_wg_many, router_wave, s, pdl, (int)std::min(T, 8 * wave));
      L->last.launches += 1;
    }
  } else {
    launch_router_logits<true>(b, L->d_wg_few, L->d_wg_many, router_wave, s, pdl, (int)std::min(T, wave));
  }
  CSK_CUDA(L, cudaGetLastError());
  L->last.launches += 3;
  L->routed_tokens += T;
  return CSK_OK;
}

ScanArgs scan_args(csk_moe_layer* L, int tile_rows, int e_begin, int e_count, const uint8_t* resident, int64_t max_rows, bool digits) {
  ScanArgs p{};
  p.counts = L->d_counts;
  p.offsets = L->d_offsets;
  p.cursor = L->d_cursor;
  p.meta = L->d_meta;
  p.E = L->E;
  p.e_begin = e_begin;
  p.e_count = e_count;
  p.tile_rows = tile_rows;
  p.max_rows = (int)max_rows;
  p.max_tiles = L->max_tiles;
  p.resident = resident;
  p.tiles = L->d_tiles;
  p.only_expert = -1;
  if (digits) {
    p.expert_tiles = L->d_expert_tiles;
    p.tile_words = L->d_wide;
    p.words_per_tile = wide_stride(L);
  }
  return p;
}

// histogram -> scan (+ row tiles of `tile_rows`) -> token rows: as fp16 rows into x16, or (x16 null) as digits into
// the block-scaled kernel's image
constexpr int kOneBlockPairs = 8192;  // up to here histogram, scan and tile list are one single-block launch

int launch_permute(csk_moe_layer* L, const float* d_hidden, const float* d_router, int64_t T, int only_expert,
                   int tile_rows, int e_begin, int e_count, __half* x16, int ldx, int64_t max_rows, cudaStream_t s) {
  const int n_pairs = (int)(T * L->k);
  const uint8_t* res = e_count ? L->d_resident : nullptr;
  const bool digits = x16 == nullptr;
  const bool one_block = n_pairs <= kOneBlockPairs;
  ScanArgs p = scan_args(L, tile_rows, e_begin, e_count, res, max_rows, digits);
  if (one_block) {
    // small batch: histogram, scan, tile list (and, for digits, the rows' places) in one single-block launch
    p.router_out = d_router;
    p.n_pairs = n_pairs;
    p.only_expert = only_expert;
    p.row_of_pair = L->d_row_of_pair;
    p.places = digits ? L->d_places : nullptr;
    L->last.launches += 1;
  } else {
    launch_k(k_hist, dim3(kHistBlocks), dim3(512), sizeof(int) * (L->E + 1), s, L->pdl, d_router, n_pairs, L->E, only_expert, L->d_counts,
             L->d_meta, L->d_hist);
    p.partial = L->d_hist;
    p.n_partial = kHistBlocks;
    L->last.launches += 2;
  }
  if (e_count && n_pairs <= kPlanPairs)  // (rows to send have to be in the order of the slots)
    launch_k(k_plan, dim3(1), dim3(ceil_div(n_pairs, 32) * 32), 0, s, L->pdl, p);
  else
    launch_k(k_scan, dim3(1), dim3(scan_threads(L->E, one_block ? n_pairs : 0)), 0, s, L->pdl, p);
  if (digits) {
    MxQuantArgs a{};
    a.hidden = d_hidden;
    a.router = d_router;
    a.offsets = L->d_offsets;
    a.et = L->d_expert_tiles;
    a.cursor = one_block ? nullptr : L->d_cursor;
    a.row_of_pair = L->d_row_of_pair;
    a.places = L->d_places;
    a.tiles = L->d_tiles;
    a.n_tiles_ptr = L->d_meta;
    a.image = L->d_ximg;
    a.rest = L->d_ximg + L->ximg_rest;
    a.wide = L->d_wide;
    a.wide_stride = wide_stride(L);
    a.T = (int)T;
    a.H = L->H;
    a.E = L->E;
    a.k = L->k;
    a.e_begin = e_begin;
    a.e_count = e_count;
    a.only_expert = only_expert;
    a.max_rows = (int)max_rows;
    a.weight_before_ffn = L->cfg.weight_before_ffn;
    a.blocks = L->Lgu.blocks;
    a.recs = L->Lgu.recs;
    const int threads = ceil_div(L->Lgu.blocks, 8) * 32, part = one_block ? kMxQuantPart : kMxQuantThreads;
    launch_k(k_mx_quant, dim3((unsigned)T, one_block ? ceil_div(threads, part) : 1), dim3(std::min(part, threads)), 0, s, L->pdl, a);
  } else {
    launch_k(reinterpret_cast<uintptr_t>(x16) % 16 ? k_scatter<uint2> : k_scatter<uint4>, dim3((unsigned)T), dim3(kScatterThreads), 0, s, L->pdl,
             d_router, d_hidden, L->k, L->H, L->E, only_expert, L->d_offsets, one_block ? (int*)nullptr : L->d_cursor, L->d_row_of_pair, x16, ldx,
             (int)max_rows, L->cfg.weight_before_ffn);
  }
  CSK_CUDA(L, cudaGetLastError());
  L->last.launches += 1;
  return CSK_OK;
}

// Images for `rows` grouped rows (row tiles of full height plus one shorter one per expert).  Called when the layer is
// created, when a path is chosen and when peers are set up, never from a stage: those may run under a caller's capture.  Images that were
// outgrown live as long as the layer, because graphs captured before (the handle's or a caller's) still name them.
int mx_reserve(csk_moe_layer* L, int64_t rows) {
  if (L->w16 || rows <= L->mx_rows) return CSK_OK;
  const size_t tiles = (size_t)rows / kMxTileRows + L->Eloc + 1;
  const size_t x1 = (mx_image_bytes(kMxDigitsX, rows, tiles, L->Lgu.recs) + 255) / 256 * 256, xb = 2 * x1;
  const size_t a1 = (mx_image_bytes(kMxDigitsA, rows, tiles, L->Ld.recs) + 255) / 256 * 256, ab = 2 * a1;
  uint8_t *x = nullptr, *a = nullptr;
  cudaError_t e = cudaMalloc(&x, xb);
  if (e == cudaSuccess) e = cudaMalloc(&a, ab);
  if (e == cudaSuccess) e = cudaMemsetAsync(x, 0, xb, L->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(a, 0, ab, L->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(L->stream);
  if (e != cudaSuccess) {
    cudaFree(x);
    cudaFree(a);
    cudaGetLastError();
    return fail(L, e == cudaErrorMemoryAllocation ? CSK_ERR_NOMEM : CSK_ERR_CUDA, "row images: %s", cudaGetErrorString(e));
  }
  if (L->d_ximg) {  // at most once: the images grow from their first size to max_rows
    L->mx_outgrown.push_back(L->d_ximg);
    L->mx_outgrown.push_back(L->d_aimg);
  }
  L->d_ximg = x;
  L->d_aimg = a;
  L->ximg_rest = x1;
  L->aimg_rest = a1;
  L->mx_rows = rows;
  return CSK_OK;
}

// The grouped fp16 rows of the expert-parallel receive side as digits.
void mx_quant_rows(csk_moe_layer* L, cudaStream_t s) {
  k_mx_quant_rows<<<4 * L->sm_count, 128, 0, s>>>(L->d_x16, L->ldx, L->d_tiles, L->d_meta, L->d_ximg, L->d_ximg + L->ximg_rest,
                                                  L->d_wide, wide_stride(L), L->H, L->Lgu.blocks, L->Lgu.recs);
}

void launch_mx_pair(csk_moe_layer* L, float* y, int ldy, cudaStream_t s, StageTimer& tm) {
  MxArgs a{};
  a.weights = L->d_weights;
  a.expert_stride = L->expert_stride;
  a.bias_offset = L->off_bias;
  a.tiles = L->d_tiles;
  a.n_tiles_ptr = L->d_meta;
  a.max_tiles = L->max_tiles;
  a.has_bias = L->cfg.has_bias;
  a.act = L->cfg.activation;
  a.F = L->F;
  a.meta = L->d_meta;
  // gate/up + activation
  a.mat_offset = L->off_gu;
  a.L = L->Lgu;
  a.x_img = L->d_ximg;
  a.x_rest = L->d_ximg + L->ximg_rest;
  a.x_wide = L->d_wide;
  a.a_img = L->d_aimg;
  a.a_rest = L->d_aimg + L->aimg_rest;
  a.a_wide = L->d_wide + mx_mask_words(L->Lgu.recs);
  a.wide_stride = wide_stride(L);
  a.a_blocks = L->Ld.blocks;
  a.a_recs = L->Ld.recs;
  a.stall = L->debug_stall;
  L->debug_stall = false;
  launch_k(k_mx<true>, dim3(L->sm_count), dim3(kMxThreads), kMxSmem, s, L->pdl, a);
  a.stall = 0;
  tm.mark();
  // down
  a.mat_offset = L->off_d;
  a.L = L->Ld;
  a.x_img = a.a_img;
  a.x_rest = a.a_rest;
  a.x_wide = a.a_wide;
  a.y = y;
  a.ldy = ldy;
  launch_k(k_mx<false>, dim3(L->sm_count), dim3(kMxThreads), kMxSmem, s, L->pdl, a);
  tm.mark();
  L->last.launches += 2;
}

// Rows per resident expert from which the fp16 tensor-core kernel takes over: the block-scaled one's time goes by the rows
// (digit columns; from 40 on it reads weights twice), the other's hardly, and short contractions leave its units' epilogues
// exposed.  Whole layer, block-scaled / fp16 kernel, us: 128 experts of 2880 x 2880 at 32 rows 565 / 670, at 40 667 / 684, at 48
// 826 / 705; 32 experts of 2880 x 2880 at 32 171 / 192, at 40 208 / 198 (Zipf load: 199 / 205); 8 experts of 1728 x 1728 at 32
// 48 / 54, at 40 58 / 54; 128 experts of 2048 x 768 at 24 191 / 197, at 32 216 / 203.
int64_t mx_rows_per_expert(const csk_moe_layer* L) { return std::min(kMxTileRows, 20 + std::min(L->H, L->F) / 128); }

// Rows the block-scaled kernel's images have to hold when a layer is created: the batches the kernel takes by itself, or every
// batch where no cluster of two CTAs can be resident (an MXFP4 layer has no other kernel then, whatever path is asked for).
int64_t mx_rows_own(const csk_moe_layer* L) {
  return L->pair.available ? std::min(L->max_rows, mx_rows_per_expert(L) * L->Eloc) : L->max_rows;
}

int choose_path(const csk_moe_layer* L, int64_t rows) {
  if (L->w16) return CSK_PATH_TILE;  // fp16 weights exist in the tensor-core layout only
  if (L->path == CSK_PATH_STREAM || !L->pair.available) return CSK_PATH_STREAM;
  if (L->path == CSK_PATH_TILE || L->path == CSK_PATH_TILE_PAIR) return CSK_PATH_TILE;
  return (rows >= mx_rows_per_expert(L) * std::max(1, L->Eloc)) ? CSK_PATH_TILE : CSK_PATH_STREAM;
}

// The expert-parallel receive side: the block-scaled kernel needs images for every row that may come (`most`).
int choose_path_received(const csk_moe_layer* L, int64_t rows, int64_t most) {
  const int path = choose_path(L, rows);
  return path == CSK_PATH_STREAM && L->mx_rows < most ? CSK_PATH_TILE : path;
}

int tile_rows_for(int path) { return path == CSK_PATH_TILE ? kPairN : kMxTileRows; }

// What is known of the tokens whose rows are listed (nothing of rows received from peers).
struct Batch {
  int64_t tokens = INT64_MAX;
  bool repeats = false;     // a token's slots may name an expert more than once
  bool one_expert = false;  // only one expert's rows are listed
};

// fp16 weights: the kernel for few rows (csk_few16.cuh) takes a batch of so many tokens.  The weights' bytes are all that counts
// there.  Step, k_pair16 / k_few16, us: dense FFN of 2880 x 2880 (weights in L2) 1 token 26.8 / 14.4, 16 27.8 / 16.5, 32 28.4 / 24.7, 48 28.8 /
// 40.1; 2048 x 8192 16 43.4 / 29.3, 24 44.7 / 43.7, 32 45.0 / 46.9; 512 x 512 32 12.5 / 10.4.  Of 33 to 64 rows a block has an SM to itself, and a
// second round of blocks costs more than it saves: 33 and 64 rows, 256 x 256 12.4 / 10.3 and 12.4 / 10.3, 1024 x 1024 16.5 / 14.4 and 16.5 / 14.8, 2368 x
// 2368 (148 blocks) 26.7 / 20.6 and 26.4 / 22.7, 2400 x 2400 24.7 / 32.9 and 26.3 / 36.1, 2048 x 2880 26.7 / 27.2 and 26.7 / 29.8.
// Of several experts its time goes by the row tiles, most of which hold a row or two, k_pair16's by the rounds of its items (128
// features of an expert) on the SMs.  The line is half an item per SM, for evenly spread routing (in brackets): 16 of 2048 x 2048, top-1, 1 token
// (0.11) 36.0 / 25.6, 5 (0.47) 51.3 / 51.3, 16 (1.1) 70.8 / 81.5; top-2, 1 (0.22) 37.0 / 28.3, 4 (0.70) 55.2 / 61.7; top-4, 1 (0.39) 42.0 / 41.6;
// 2 of 2880 x 2880, 1 (0.16) 40.7 / 26.9, 8 (0.31) 47.6 / 43.3; 4, top-2, 1 (0.27) 45.2 / 44.7; 128 of 2048 x 768, top-8, 1 (0.32) 39.0 / 43.1, 2 (0.61)
// 53.5 / 58.6; 64 of 512 x 512, top-8, 1 (0.21) 25.8 / 21.0, 4 (0.69) 32.2 / 35.0; beside a shared expert 16 of 2048 x 2048, top-1, 5 tokens level (60.4 / 59.2 of a block that takes 55 now).  And 24 MB of
// weights, where launches and latencies are what is left: 64 of 256 x 512, top-8, 2 (0.37, 11 MB) 22.7 / 20.6, 4 (0.68, 20 MB) 24.2 / 24.7, 8 (1.1, 32 MB)
// 24.8 / 30.9.
bool few_rows(const csk_moe_layer* L, const Batch& b) {
  if (L->Eloc == 1) return b.tokens <= (std::max(L->F, L->H) / 16 <= L->sm_count ? kFewMaxRowsWave : kFewMaxRows);
  if (b.tokens > kFewMaxRowsRouted) return false;
  if (b.one_expert) return true;
  const double hit = L->Eloc * (1.0 - std::pow(1.0 - 1.0 / L->E, (double)(b.tokens * L->k)));
  return hit * L->Tgu.n_tiles <= 0.5 * L->sm_count || hit * (3.0 * sizeof(__half) * L->H * L->F) <= 24e6;
}

// grouped gate/up + activation + down over the row tiles listed in d_tiles; the grouped rows are in d_x16 (tensor-core
// path) or in d_ximg (streaming path); output rows go to y (through out_row_map or out_row_ptr if set)
int launch_experts(csk_moe_layer* L, int path, float* y, int ldy, const int* out_row_map, cudaStream_t s, StageTimer& tm,
                   float* const* out_row_ptr = nullptr, const Batch& batch = {}) {
  if (path == CSK_PATH_TILE && L->w16 && few_rows(L, batch) && !L->debug_stall) {
    FewArgs f{};
    f.x = L->d_x16;
    f.ldx = L->ldx;
    f.one_expert = L->Eloc == 1;
    TileArgs& a = f.t;
    a.weights = L->d_weights;
    a.expert_stride = L->expert_stride;
    a.bias_offset = L->off_bias;
    a.tiles = L->d_tiles;
    a.n_tiles_ptr = a.meta = L->d_meta;
    a.has_bias = L->cfg.has_bias;
    a.act = L->cfg.activation;
    a.F = L->F;
    a.mat_offset = L->off_tgu;
    a.L = L->Tgu;
    a.a_out = L->d_a16;
    a.lda = L->lda;
    // (where a token's slots may all name one expert, its rows may need several tiles)
    const int64_t pairs = batch.tokens * L->k;
    const int tiles = (int)std::min(pairs, batch.repeats ? L->Eloc + pairs / kPairN : (int64_t)L->Eloc);
    CSK_CUDA(L, few_launch_one<true>(f, L->F, tiles, (int)batch.tokens, batch.repeats, s, L->pdl));
    tm.mark();
    f.x = L->d_a16;
    f.ldx = L->lda;
    a.mat_offset = L->off_td;
    a.L = L->Td;
    a.y_out = y;
    a.ldy = ldy;
    CSK_CUDA(L, few_launch_one<false>(f, L->H, tiles, (int)batch.tokens, batch.repeats, s, L->pdl));
    tm.mark();
    L->last.launches += 2;
  } else if (path == CSK_PATH_TILE) {
    const int rc =
        pair_launch(L->pair, L->tile, L->tile.pair_x, L->tile.pair_a, L->d_weights, L->expert_stride, L->off_tgu,
                       L->off_td, L->off_bias, L->off_meta, L->Tgu, L->Td, L->d_a16, L->lda, y, ldy, out_row_map,
                       out_row_ptr, L->d_tiles, L->d_meta, L->cfg.has_bias, L->cfg.activation, L->F, s, L->pdl,
                       [&]() { tm.mark(); }, L->debug_stall);
    L->debug_stall = false;
    if (rc) return fail(L, rc, "tensor-core path: %s", L->tile.err.c_str());
    L->last.launches += 2;
  } else {
    if (out_row_map || out_row_ptr) return fail(L, CSK_ERR_INVALID, "row maps need the tile path");
    launch_mx_pair(L, y, ldy, s, tm);
  }
  CSK_CUDA(L, cudaGetLastError());
  L->last.path = path;
  return CSK_OK;
}

int report_status(csk_moe_layer* L, int st, cudaStream_t s);

int check_device_status(csk_moe_layer* L, cudaStream_t s) {
  CSK_CUDA(L, cudaMemcpyAsync(L->h_meta, L->d_meta, sizeof(int) * 16, cudaMemcpyDeviceToHost, s));
  CSK_CUDA(L, cudaStreamSynchronize(s));
  return report_status(L, L->h_meta[3] | L->h_meta[8], s);
}

// The host's view of a status word (h_meta holds the copy it came from).
int report_status(csk_moe_layer* L, int st, cudaStream_t s) {
  if (L->h_meta[8]) cudaMemsetAsync(L->d_meta + 8, 0, sizeof(int), s);
  if (st & kDevErrExpertRange)
    return fail(L, CSK_ERR_INVALID, "expert_idx out of range in router output");
  if (st & kDevErrCapacity)
    return fail(L, CSK_ERR_NOMEM, "more rows than max_tokens allows (%d rows)", L->h_meta[1]);
  if (st & kDevErrNotResident)
    return fail(L, CSK_ERR_MISSING, "tokens were routed to an expert whose weights are not loaded");
  if (st & kDevErrPeerRow)
    return fail(L, CSK_ERR_DEVICE, "a row received from a peer carries no valid origin (rank, pair)");
  if (st & kDevErrWaitTimeout)
    return fail(L, CSK_ERR_DEVICE, "a bounded device-side wait ran out");
  return CSK_OK;
}

void finish_timings(csk_moe_layer* L, int n_marks, bool routed) {
  if (!L->timing) return;
  float ms[8] = {0};
  for (int i = 0; i + 1 < n_marks; ++i) cudaEventElapsedTime(&ms[i], L->ev[i], L->ev[i + 1]);
  int i = 0;
  L->last.route_ms = routed ? ms[i++] : 0.f;
  L->last.permute_ms = ms[i++];
  L->last.gate_up_ms = ms[i++];
  L->last.down_ms = ms[i++];
  L->last.combine_ms = ms[i++];
  cudaEventElapsedTime(&L->last.total_ms, L->ev[0], L->ev[n_marks - 1]);
}

// Page-locked memory that the last kernel writes the routing (or null) and the words of d_meta to.
struct HostResult {
  float* router = nullptr;
  int* meta = nullptr;
};

// What k_combine does beside the sums, see there.
struct CombineArgs {
  bool dense_single = false;
  const int *meta = nullptr, *counts = nullptr;
  int* carry = nullptr;
  const float *residual = nullptr, *shared = nullptr;
  HostResult host;
};

// The rows of y (places in d_row_of_pair) to the tokens' results: of the layer, of the merge node, of expert parallelism.
void launch_combine(csk_moe_layer* L, const float* router, const float* y, int64_t T, float* out, cudaStream_t s, bool pdl,
                    const CombineArgs& c = {}) {
  const unsigned row_blocks = T < 4 * L->sm_count ? (unsigned)ceil_div(L->H, 1024) : 1u;
  // As long as its blocks are resident at once (of eight slots a little longer) the form for few tokens is the quicker one.  Few / many, a step, us:
  // four slots of 2880 columns, 600 tokens 60.2 / 62.3, 740 63.9 / 66.1, 820 67.9 / 69.3, 1000 74.4 / 74.2; eight of 2048, 600 60.1 / 61.6, 740 65.4 / 66.1,
  // 900 71.8 / 71.7, 1000 72.9 / 72.4; eight of 512, 740 36.1 / 35.5.
  const bool few = c.host.meta || T <= (L->k > 4 ? 5 : 6) * L->sm_count;  // (page-locked results are small ones)
  launch_k(!few ? k_combine<4, false> : L->k > 4 ? k_combine<8, true> : k_combine<4, true>, dim3((unsigned)T, row_blocks), dim3(256), 0, s, pdl, router,
           L->d_row_of_pair, y, L->H, out, (int)T, L->k, L->H, (int)L->cfg.weight_before_ffn, (int)c.dense_single, c.meta, c.counts, c.carry,
           L->E, c.residual, c.shared, c.host.router, c.host.meta);
}

// The whole layer on device buffers.  only_expert >= 0 gives the dense output
// of that single expert node.
int forward_dev(csk_moe_layer* L, const float* d_hidden, int64_t T, const float* d_router_in,
                float* d_router_out, float* d_out, int only_expert, cudaStream_t s, bool sync_check,
                const float* d_residual = nullptr, const float* d_shared = nullptr, cudaEvent_t shared_ready = nullptr, const HostResult& host = {}) {
  if (T <= 0 || T > L->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld outside (0, max_tokens=%lld]",
                                          (long long)T, (long long)L->max_T);
  if (L->has_slot_map)
    return fail(L, CSK_ERR_INVALID, "the layer has an expert-parallel slot map: use the csk_moe_ep_* stages");
  L->last = csk_moe_timings{};
  L->last_T = T;
  if (!L->carry_active) L->counts_in_carry = false;
  // each kernel may become resident while its predecessor drains
  const PdlScope pdl_scope(L);
  StageTimer tm(L, s);
  tm.mark();
  const float* router = d_router_in;
  const bool routed = d_router_in == nullptr;
  if (routed) {
    // the routing is written where the caller wants it (else into the handle's buffer) and read from there
    float* route_to = d_router_out ? d_router_out : L->d_router;
    int rc = launch_router(L, d_hidden, T, route_to, s);
    if (rc) return rc;
    router = route_to;
    tm.mark();
  } else if (d_router_out && d_router_out != router) {
    CSK_CUDA(L, cudaMemcpyAsync(d_router_out, router, sizeof(float) * T * L->k * 2,
                                cudaMemcpyDeviceToDevice, s));
  }
  const int64_t rows = only_expert >= 0 ? T : T * L->k;
  const int path = choose_path(L, only_expert >= 0 ? rows * std::max(1, L->Eloc) : rows);
  const int tile_rows = tile_rows_for(path);
  if (reinterpret_cast<uintptr_t>(d_hidden) % 16) return fail(L, CSK_ERR_INVALID, "hidden states must be 16-byte aligned");
  const bool mx = path == CSK_PATH_STREAM;
  if (router == L->d_unit_router && router && !mx && only_expert < 0 && !d_router_out && !d_residual && !d_shared && !L->carry_active &&
      !host.meta) {
    // a dense FFN on the tensor-core kernel: the token rows are the grouped rows, and the down projection's the result
    // (8192 tokens, 2880 x 2880: 498 -> 450 us for a scan, a scatter and a combine less)
    launch_k(k_dense_rows, dim3(grid_for((size_t)T * (L->H / 8), 256, 8 * L->sm_count)), dim3(256), 0, s, L->pdl, d_hidden, L->d_x16, L->ldx,
             (int)T, L->H, tile_rows, (const uint8_t*)L->d_resident, L->d_counts, L->d_offsets, L->d_tiles, L->d_meta);
    CSK_CUDA(L, cudaGetLastError());
    L->last.launches++;
    tm.mark();
    int rc = launch_experts(L, path, d_out, L->H, nullptr, s, tm, nullptr, Batch{T});
    if (rc) return rc;
    tm.mark();  // nothing to combine
    L->n_marks = tm.n;
    L->last_routed = false;
    L->last_stream = s;
    if (!sync_check) return CSK_OK;
    rc = check_device_status(L, s);
    if (rc) return rc;
    finish_timings(L, tm.n, false);
    return CSK_OK;
  }
  int rc = launch_permute(L, d_hidden, router, T, only_expert, tile_rows, L->e0, L->Eloc, mx ? nullptr : L->d_x16, L->ldx,
                          mx ? L->mx_rows : L->max_rows, s);
  if (rc) return rc;
  tm.mark();
  rc = launch_experts(L, path, L->d_y, L->H, nullptr, s, tm, nullptr, Batch{T, !routed && L->k > 1, only_expert >= 0});
  if (rc) return rc;
  // the shared expert's rows come from another stream: the combine is the first kernel that reads them
  if (shared_ready) CSK_CUDA(L, cudaStreamWaitEvent(s, shared_ready, 0));
  CombineArgs c;
  c.dense_single = only_expert >= 0;
  c.meta = L->d_meta;
  c.counts = L->d_counts;
  c.carry = L->carry_active ? L->d_carry : nullptr;
  c.residual = d_residual;
  c.shared = d_shared;
  c.host = host;
  launch_combine(L, router, L->d_y, T, d_out, s, L->pdl && !shared_ready, c);
  CSK_CUDA(L, cudaGetLastError());
  L->last.launches++;
  tm.mark();
  L->n_marks = tm.n;
  L->last_routed = routed;
  L->last_stream = s;
  if (!sync_check) return CSK_OK;
  rc = check_device_status(L, s);
  if (rc) return rc;
  finish_timings(L, tm.n, routed);
  return CSK_OK;
}

int check_layer(csk_moe_layer* L) { return L ? CSK_OK : CSK_ERR_INVALID; }

// Captured launch sequences embed kernel arguments (which router bias, which path, which
// slot map): whatever changes one of those drops them.
void drop_graphs(csk_moe_layer* L) {
  for (auto& g : L->graphs)
    if (g.exec) cudaGraphExecDestroy(g.exec);
  L->graphs.clear();
}

}  // namespace

// ===========================================================================
extern "C" {

int csk_moe_device_ok(int device) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) {
    cudaGetLastError();
    return 0;
  }
  cudaDeviceProp p{};
  if (cudaGetDeviceProperties(&p, device) != cudaSuccess) return 0;
  return p.major == 10 ? 1 : 0;
}

const char* csk_moe_last_error(const csk_moe_layer* layer) {
  if (layer) return layer->err.c_str();
  std::lock_guard<std::mutex> lk(g_err_mu);
  return g_create_error.c_str();
}

int csk_moe_create(const csk_moe_config* cfg, csk_moe_layer** out) {
  if (!cfg || !out) return fail(nullptr, CSK_ERR_INVALID, "null argument");
  *out = nullptr;
  if (cfg->num_experts <= 0 || cfg->num_experts > 1024)
    return fail(nullptr, CSK_ERR_INVALID, "num_experts must be in [1,1024], got %d", cfg->num_experts);
  if (cfg->top_k <= 0 || cfg->top_k > kMaxTopK || cfg->top_k > cfg->num_experts)
    return fail(nullptr, CSK_ERR_INVALID, "top_k must be in [1,%d] and <= num_experts, got %d",
                kMaxTopK, cfg->top_k);
  if (cfg->hidden <= 0 || cfg->hidden % 32)
    return fail(nullptr, CSK_ERR_INVALID,
                "expert_mlp: hidden_dim must be a multiple of 32 for MXFP4, got %d", cfg->hidden);
  if (cfg->ffn <= 0 || cfg->ffn % 32)
    return fail(nullptr, CSK_ERR_INVALID,
                "expert_mlp: expert_ffn_dim must be a multiple of 32 for MXFP4, got %d", cfg->ffn);
  if (cfg->weight_format != CSK_WEIGHTS_MXFP4 && cfg->weight_format != CSK_WEIGHTS_F16)
    return fail(nullptr, CSK_ERR_INVALID, "unknown weight format %d", cfg->weight_format);
  if (cfg->activation != CSK_ACT_MODIFIED_SWIGLU && cfg->activation != CSK_ACT_STANDARD_SWIGLU)
    return fail(nullptr, CSK_ERR_INVALID, "unknown activation %d", cfg->activation);
  if (cfg->max_tokens <= 0 || cfg->max_tokens * cfg->top_k > (1 << 28))
    return fail(nullptr, CSK_ERR_INVALID, "max_tokens out of range");
  const int eloc = cfg->expert_count ? cfg->expert_count : cfg->num_experts;
  const int e0 = cfg->expert_count ? cfg->expert_begin : 0;
  if (e0 < 0 || eloc <= 0 || e0 + eloc > cfg->num_experts)
    return fail(nullptr, CSK_ERR_INVALID, "expert range [%d,%d) outside [0,%d)", e0, e0 + eloc,
                cfg->num_experts);
  if (!csk_moe_device_ok(cfg->device))
    return fail(nullptr, CSK_ERR_CUDA, "device %d is not a usable sm_100 GPU (no CPU fallback exists)",
                cfg->device);

  csk_moe_layer* L = new (std::nothrow) csk_moe_layer();
  if (!L) return fail(nullptr, CSK_ERR_NOMEM, "out of host memory");
  L->cfg = *cfg;
  L->E = cfg->num_experts;
  L->k = cfg->top_k;
  L->H = cfg->hidden;
  L->F = cfg->ffn;
  L->e0 = e0;
  L->Eloc = eloc;
  L->w16 = cfg->weight_format == CSK_WEIGHTS_F16;
  L->Lgu = make_mx_layout(L->F, L->H, true);
  L->Ld = make_mx_layout(L->H, L->F, false);
  L->Tgu = make_tile_layout(L->F, L->H, true, L->w16);
  L->Td = make_tile_layout(L->H, L->F, false, L->w16);
  auto up256 = [](size_t v) { return (v + 255) / 256 * 256; };
  L->off_gu = 0;
  L->off_d = L->w16 ? 0 : up256(L->Lgu.bytes());                  // fp16 weights have no streaming layout
  L->off_tgu = L->w16 ? 0 : L->off_d + up256(L->Ld.bytes());
  L->off_td = L->off_tgu + up256(L->Tgu.bytes());
  L->off_bias = L->off_td + up256(L->Td.bytes());
  L->off_meta = L->off_bias + sizeof(float) * (2 * (size_t)L->F + L->H);  // int[4]: e_max of gate/up, of down
  L->expert_stride = (L->off_meta + 16 + 255) / 256 * 256;
  L->resident.assign(eloc, 0);
  L->max_T = cfg->max_tokens;
  L->max_rows = cfg->max_tokens * cfg->top_k;
  L->ldx = L->Tgu.k_pad();
  L->lda = L->Td.k_pad();
  L->max_tiles = (int)(L->max_rows / 8 + eloc + 8);

#define CK(call)                                                                              \
  do {                                                                                        \
    cudaError_t _e = (call);                                                                  \
    if (_e != cudaSuccess) {                                                                  \
      int rc = fail(nullptr, _e == cudaErrorMemoryAllocation ? CSK_ERR_NOMEM : CSK_ERR_CUDA,  \
                    "%s failed: %s", #call, cudaGetErrorString(_e));                          \
      csk_moe_destroy(L);                                                                     \
      return rc;                                                                              \
    }                                                                                         \
  } while (0)

  CK(cudaSetDevice(cfg->device));
  cudaDeviceProp prop{};
  CK(cudaGetDeviceProperties(&prop, cfg->device));
  L->sm_count = prop.multiProcessorCount;
  CK(cudaStreamCreateWithFlags(&L->stream, cudaStreamNonBlocking));
  CK(cudaStreamCreateWithFlags(&L->stream_in, cudaStreamNonBlocking));
  CK(cudaStreamCreateWithFlags(&L->stream_out, cudaStreamNonBlocking));
  for (auto& e : L->ev) CK(cudaEventCreate(&e));
  for (auto& e : L->ev_in) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  for (auto& e : L->ev_done) CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  CK(cudaEventCreateWithFlags(&L->ev_free, cudaEventDisableTiming));
  CK(cudaMalloc(&L->d_carry, sizeof(int) * (1 + L->E)));
  CK(cudaMemset(L->d_carry, 0, sizeof(int) * (1 + L->E)));
  CK(cudaMalloc(&L->d_weights, L->expert_stride * eloc));
  CK(cudaMemset(L->d_weights, 0, L->expert_stride * eloc));
  CK(cudaMalloc(&L->d_resident, eloc));
  CK(cudaMemset(L->d_resident, 0, eloc));
  L->stage_bytes = L->w16 ? (size_t)L->H * L->F * 2 : (size_t)L->H * L->F / 32 * 17;
  CK(cudaMalloc(&L->d_stage, std::max(3 * L->stage_bytes, image_part_bytes(L))));
  CK(cudaMalloc(&L->d_wg, sizeof(float) * L->E * L->H));
  CK(cudaMalloc(&L->d_wg_few, sizeof(float) * router_packed_floats(L->E, L->H, kRouterChunkFew)));
  CK(cudaMalloc(&L->d_wg_many, sizeof(float) * router_packed_floats(L->E, L->H, kRouterChunkMany)));
  CK(cudaMalloc(&L->d_route_cnt, sizeof(int) * L->max_T));
  CK(cudaMemset(L->d_route_cnt, 0, sizeof(int) * L->max_T));
  CK(cudaMalloc(&L->d_logits, sizeof(float) * L->max_T * L->E));
  CK(cudaMalloc(&L->d_wnorm, sizeof(float) * L->E));
  CK(cudaMalloc(&L->d_wg_tc, rt_weight_bytes(L->E, L->H)));
  CK(cudaMalloc(&L->d_wg_tc_scale, sizeof(float) * rt_scale_floats(L->E, L->H)));
  CK(cudaMalloc(&L->d_wnorm_tc, sizeof(float) * L->E));
  L->part_rows = L->max_T + 64 * (int64_t)(L->sm_count + fast_router_slices(L->H));
  CK(cudaMalloc(&L->d_part, sizeof(float2) * L->part_rows * L->E));
  CK(cudaMalloc(&L->d_hn2, sizeof(float) * L->part_rows));
  CK(cudaMalloc(&L->d_fb_list, sizeof(int) * L->max_T));
  CK(cudaMalloc(&L->d_fb, sizeof(int) * 4));
  CK(cudaMemset(L->d_fb, 0, sizeof(int) * 4));
  CK(cudaMalloc(&L->d_rbias, sizeof(float) * L->E));
  CK(cudaMalloc(&L->d_hidden, sizeof(float) * L->max_T * L->H));
  CK(cudaMalloc(&L->d_router, sizeof(float) * L->max_T * L->k * 2));
  CK(cudaMalloc(&L->d_router_phys, sizeof(float) * L->max_T * L->k * 2));
  CK(cudaMalloc(&L->d_p2p_epoch, sizeof(int) * 4));
  CK(cudaMemset(L->d_p2p_epoch, 0, sizeof(int) * 4));
  if (L->E == 1 && L->k == 1) {  // a dense FFN: every token goes to expert 0 with weight 1
    std::vector<float> unit(2 * (size_t)L->max_T);
    for (int64_t t = 0; t < L->max_T; ++t) {
      unit[2 * t] = 0.0f;
      unit[2 * t + 1] = 1.0f;
    }
    CK(cudaMalloc(&L->d_unit_router, sizeof(float) * unit.size()));
    CK(cudaMemcpy(L->d_unit_router, unit.data(), sizeof(float) * unit.size(), cudaMemcpyHostToDevice));
  }
  CK(cudaMalloc(&L->d_slot_map, sizeof(int) * 2 * L->E));
  CK(cudaMalloc(&L->d_p2p_base, sizeof(int) * L->E));
  L->E_router = L->E;
  CK(cudaMalloc(&L->d_out, sizeof(float) * L->max_T * L->H));
  const size_t pad_rows = 32;  // a row tile's loads may reach this far past the last row (its MMAs' rows are a multiple of 32)
  CK(cudaMalloc(&L->d_x16, sizeof(__half) * (L->max_rows + pad_rows) * L->ldx));
  CK(cudaMemset(L->d_x16, 0, sizeof(__half) * (L->max_rows + pad_rows) * L->ldx));
  CK(cudaMalloc(&L->d_a16, sizeof(__half) * (L->max_rows + pad_rows) * L->lda));
  CK(cudaMemset(L->d_a16, 0, sizeof(__half) * (L->max_rows + pad_rows) * L->lda));
  CK(cudaMalloc(&L->d_y, sizeof(float) * L->max_rows * L->H));
  CK(cudaMalloc(&L->d_counts, sizeof(int) * L->E));
  CK(cudaMalloc(&L->d_hist, sizeof(int) * kHistBlocks * (L->E + 1)));
  CK(cudaMalloc(&L->d_offsets, sizeof(int) * (L->E + 1)));
  CK(cudaMalloc(&L->d_cursor, sizeof(int) * L->E));
  CK(cudaMalloc(&L->d_row_of_pair, sizeof(int) * L->max_rows));
  CK(cudaMalloc(&L->d_places, sizeof(int4) * std::min<int64_t>(L->max_rows, kOneBlockPairs)));
  CK(cudaMalloc(&L->d_expert_tiles, sizeof(ExpertTiles) * L->E));
  CK(cudaMalloc(&L->d_out_row_map, sizeof(int) * L->max_rows));
  CK(cudaMalloc(&L->d_seg, sizeof(int) * (3 * 1024 + 8)));
  CK(cudaMalloc(&L->d_tiles, sizeof(RowTile) * L->max_tiles));
  CK(cudaMalloc(&L->d_wide, sizeof(uint32_t) * L->max_tiles * wide_stride(L)));
  CK(cudaMalloc(&L->d_meta, sizeof(int) * 16));
  CK(cudaMemset(L->d_meta, 0, sizeof(int) * 16));
  CK(cudaMallocHost(&L->h_meta, sizeof(int) * 16));
  CK(cudaMallocHost(&L->h_counts64, sizeof(int64_t) * L->E));
  L->h_staged_bytes = std::min<size_t>(kStagedMax, sizeof(float) * L->max_T * (L->H + 2 * L->k));
  CK(cudaMallocHost(&L->h_staged, L->h_staged_bytes));
  CK(router_prepare_device());
  for (int g = 1; g <= kMaxExperts / 32; ++g) L->router_waves[g] = router_wave(g, L->sm_count);
  CK(mx_prepare_device());
  CK(few_prepare_device());
  CK(rt_prepare_device());
  {
    int rc = tile_init(L->tile, cfg->device);
    if (!rc)
      rc = tile_set_buffers(L->tile, L->d_x16, L->ldx, L->d_a16, L->lda, (size_t)L->max_rows + pad_rows, L->w16 ? L->d_weights : nullptr,
                            L->expert_stride * L->Eloc);
    if (!rc) rc = pair_init(L->pair, L->tile, L->sm_count);
    if (rc) {
      rc = fail(nullptr, rc, "tensor-core path setup: %s", L->tile.err.c_str());
      csk_moe_destroy(L);
      return rc;
    }
  }
  if (mx_reserve(L, mx_rows_own(L))) {
    fail(nullptr, CSK_ERR_NOMEM, "%s", L->err.c_str());
    csk_moe_destroy(L);
    return CSK_ERR_NOMEM;
  }
  CK(cudaDeviceSynchronize());
#undef CK
  *out = L;
  return CSK_OK;
}

int csk_moe_destroy(csk_moe_layer* L) {
  if (!L) return CSK_OK;
  cudaSetDevice(L->cfg.device);
  if (L->stream) cudaStreamSynchronize(L->stream);
  for (auto& g : L->graphs)
    if (g.exec) cudaGraphExecDestroy(g.exec);
  tile_destroy(L->tile);
  for (void* p : L->ipc_opened) cudaIpcCloseMemHandle(p);
  void* dev[] = {L->d_shared_out, L->d_p2p_epoch, L->d_unit_router, L->d_stage2, L->d_norm_w, L->d_normed, L->d_part, L->d_hn2, L->d_wnorm, L->d_wg_tc, L->d_wg_tc_scale, L->d_wnorm_tc, L->d_fb_list, L->d_fb, L->d_info, L->d_back, L->d_row_ptr, L->d_p2p_base, L->d_peer_x16, L->d_peer_info, L->d_peer_back,
                 L->d_router_phys, L->d_slot_map, L->d_weights, L->d_resident, L->d_stage, L->d_wg, L->d_wg_few, L->d_wg_many, L->d_route_cnt, L->d_logits, L->d_rbias, L->d_hidden,
                 L->d_router, L->d_out, L->d_x16, L->d_a16, L->d_y, L->d_counts, L->d_hist, L->d_offsets,
                 L->d_cursor, L->d_row_of_pair, L->d_places, L->d_expert_tiles, L->d_ximg, L->d_aimg, L->d_wide, L->d_out_row_map, L->d_seg, L->d_tiles, L->d_meta};
  for (void* p : dev)
    if (p) cudaFree(p);
  for (uint8_t* p : L->mx_outgrown) cudaFree(p);
  if (L->h_meta) cudaFreeHost(L->h_meta);
  if (L->h_counts64) cudaFreeHost(L->h_counts64);
  if (L->h_staged) cudaFreeHost(L->h_staged);
  for (auto& e : L->ev)
    if (e) cudaEventDestroy(e);
  for (auto& e : L->ev_in)
    if (e) cudaEventDestroy(e);
  for (auto& e : L->ev_done)
    if (e) cudaEventDestroy(e);
  if (L->ev_free) cudaEventDestroy(L->ev_free);
  if (L->ev_shared_fork) cudaEventDestroy(L->ev_shared_fork);
  if (L->ev_shared_join) cudaEventDestroy(L->ev_shared_join);
  if (L->d_carry) cudaFree(L->d_carry);
  if (L->stream_in) cudaStreamDestroy(L->stream_in);
  if (L->stream_out) cudaStreamDestroy(L->stream_out);
  if (L->stream) cudaStreamDestroy(L->stream);
  delete L;
  return CSK_OK;
}

int csk_moe_set_router(csk_moe_layer* L, const float* gate_w, const float* gate_bias) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!gate_w) return fail(L, CSK_ERR_INVALID, "gate_weights is null");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  CSK_CUDA(L, cudaMemcpyAsync(L->d_wg, gate_w, sizeof(float) * L->E_router * L->H, cudaMemcpyHostToDevice,
                              L->stream));
  k_pack_router<<<grid_for(router_packed_floats(L->E_router, L->H, kRouterChunkFew), 256, 1024), 256, 0, L->stream>>>(
      L->d_wg, L->d_wg_few, L->E_router, L->H, kRouterChunkFew);
  k_pack_router<<<grid_for(router_packed_floats(L->E_router, L->H, kRouterChunkMany), 256, 1024), 256, 0, L->stream>>>(
      L->d_wg, L->d_wg_many, L->E_router, L->H, kRouterChunkMany);
  k_router_wnorm<<<(L->E_router + 7) / 8, 256, 0, L->stream>>>(L->d_wg, L->d_wnorm, L->E_router, L->H);
  k_rt_wnorm<<<(L->E_router + 7) / 8, 256, 0, L->stream>>>(L->d_wg, L->d_wnorm_tc, L->E_router, L->H);
  k_rt_pack<<<grid_for(rt_scale_floats(L->E_router, L->H), 64, 1024), 64, 0, L->stream>>>(L->d_wg, L->d_wg_tc, L->d_wg_tc_scale,
                                                                                       L->E_router, L->H);
  CSK_CUDA(L, cudaGetLastError());
  L->has_rbias = gate_bias != nullptr;
  if (gate_bias)
    CSK_CUDA(L, cudaMemcpyAsync(L->d_rbias, gate_bias, sizeof(float) * L->E_router, cudaMemcpyHostToDevice,
                                L->stream));
  CSK_CUDA(L, cudaStreamSynchronize(L->stream));
  L->router_set = true;
  drop_graphs(L);
  return CSK_OK;
}

namespace {
// One expert: raw blocks to a staging area, the four repacks, biases.  Enqueue only; `stage` is one
// of the handle's two staging areas (3 * stage_bytes each).  With null weight pointers the staging
// area already holds the three matrices (decoded there by the caller).
int load_expert_enqueue(csk_moe_layer* L, int le, const uint8_t* w_up, const uint8_t* w_gate, const uint8_t* w_down,
                        const float* b_up, const float* b_gate, const float* b_down, uint8_t* stage, cudaStream_t s) {
  uint8_t* base = L->d_weights + (size_t)le * L->expert_stride;
  uint8_t *s_up = stage, *s_gate = stage + L->stage_bytes, *s_down = stage + 2 * L->stage_bytes;
  if (w_up) {
    CSK_CUDA(L, cudaMemcpyAsync(s_up, w_up, L->stage_bytes, cudaMemcpyHostToDevice, s));
    CSK_CUDA(L, cudaMemcpyAsync(s_gate, w_gate, L->stage_bytes, cudaMemcpyHostToDevice, s));
    CSK_CUDA(L, cudaMemcpyAsync(s_down, w_down, L->stage_bytes, cudaMemcpyHostToDevice, s));
  }
  int* emeta = reinterpret_cast<int*>(base + L->off_meta);
  CSK_CUDA(L, cudaMemsetAsync(emeta, 0, 16, s));
  if (L->w16) {
    const __half *h_up = reinterpret_cast<const __half*>(s_up), *h_gate = reinterpret_cast<const __half*>(s_gate),
                 *h_down = reinterpret_cast<const __half*>(s_down);
    k_repack_tile_f16<<<grid_for(L->Tgu.bytes() / 16, 256, 4096), 256, 0, s>>>(h_gate, h_up, base + L->off_tgu, L->Tgu);
    k_repack_tile_f16<<<grid_for(L->Td.bytes() / 16, 256, 4096), 256, 0, s>>>(h_down, nullptr, base + L->off_td, L->Td);
  } else {
  k_mx_repack<<<grid_for(L->Lgu.bytes() / 16, 256, 4096), 256, 0, s>>>(s_gate, s_up, base + L->off_gu, L->Lgu, emeta);
  k_mx_repack<<<grid_for(L->Ld.bytes() / 16, 256, 4096), 256, 0, s>>>(s_down, nullptr, base + L->off_d, L->Ld, emeta + 1);
  k_repack_tile<<<grid_for(L->Tgu.bytes() / 4, 256, 4096), 256, 0, s>>>(s_gate, s_up, base + L->off_tgu, L->Tgu);
  k_repack_tile<<<grid_for(L->Td.bytes() / 4, 256, 4096), 256, 0, s>>>(s_down, nullptr, base + L->off_td, L->Td);
  }
  CSK_CUDA(L, cudaGetLastError());
  if (L->cfg.has_bias) {
    float* b = reinterpret_cast<float*>(base + L->off_bias);
    CSK_CUDA(L, cudaMemcpyAsync(b, b_up, sizeof(float) * L->F, cudaMemcpyHostToDevice, s));
    CSK_CUDA(L, cudaMemcpyAsync(b + L->F, b_gate, sizeof(float) * L->F, cudaMemcpyHostToDevice, s));
    CSK_CUDA(L, cudaMemcpyAsync(b + 2 * L->F, b_down, sizeof(float) * L->H, cudaMemcpyHostToDevice, s));
  }
  CSK_CUDA(L, cudaMemsetAsync(L->d_resident + le, 1, 1, s));
  return CSK_OK;
}
}  // namespace

int csk_moe_load_expert_mxfp4(csk_moe_layer* L, int32_t expert_id, const uint8_t* w_up,
                              const uint8_t* w_gate, const uint8_t* w_down, const float* b_up,
                              const float* b_gate, const float* b_down) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (expert_id < L->e0 || expert_id >= L->e0 + L->Eloc)
    return fail(L, CSK_ERR_INVALID, "expert %d is not resident on this device (range [%d,%d))",
                expert_id, L->e0, L->e0 + L->Eloc);
  if (!w_up || !w_gate || !w_down) return fail(L, CSK_ERR_INVALID, "null weight pointer");
  if (L->cfg.has_bias && (!b_up || !b_gate || !b_down))
    return fail(L, CSK_ERR_INVALID, "layer has biases but a bias pointer is null");
  if (L->w16) return fail(L, CSK_ERR_INVALID, "this layer holds fp16 weights: use csk_moe_load_expert_f16");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  const int le = expert_id - L->e0;
  int rc = load_expert_enqueue(L, le, w_up, w_gate, w_down, b_up, b_gate, b_down, L->d_stage, L->stream);
  if (rc) return rc;
  CSK_CUDA(L, cudaStreamSynchronize(L->stream));
  L->resident[le] = 1;
  return CSK_OK;
}

int csk_moe_load_expert_f16(csk_moe_layer* L, int32_t expert_id, const uint16_t* w_up, const uint16_t* w_gate,
                            const uint16_t* w_down, const float* b_up, const float* b_gate, const float* b_down) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!L->w16) return fail(L, CSK_ERR_INVALID, "this layer holds MXFP4 weights: use csk_moe_load_expert_mxfp4");
  if (expert_id < L->e0 || expert_id >= L->e0 + L->Eloc)
    return fail(L, CSK_ERR_INVALID, "expert %d is not resident on this device (range [%d,%d))",
                expert_id, L->e0, L->e0 + L->Eloc);
  if (!w_up || !w_gate || !w_down) return fail(L, CSK_ERR_INVALID, "null weight pointer");
  if (L->cfg.has_bias && (!b_up || !b_gate || !b_down))
    return fail(L, CSK_ERR_INVALID, "layer has biases but a bias pointer is null");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  const int le = expert_id - L->e0;
  int rc = load_expert_enqueue(L, le, reinterpret_cast<const uint8_t*>(w_up), reinterpret_cast<const uint8_t*>(w_gate),
                               reinterpret_cast<const uint8_t*>(w_down), b_up, b_gate, b_down, L->d_stage, L->stream);
  if (rc) return rc;
  CSK_CUDA(L, cudaStreamSynchronize(L->stream));
  L->resident[le] = 1;
  return CSK_OK;
}

namespace {
size_t ggml_bytes(int32_t type, int64_t n) {
  switch (type) {
    case CSK_GGML_F16: return (size_t)n * 2;
    case CSK_GGML_Q4_K: return (size_t)(n / kQkK) * kQ4kBytes;
    case CSK_GGML_Q6_K: return (size_t)(n / kQkK) * kQ6kBytes;
  }
  return 0;
}
// Raw blocks of one matrix (device) to fp16 (device).  Enqueue only.
void ggml_decode_enqueue(int32_t type, const uint8_t* d_raw, unsigned short* d_f16, int64_t n, bool nearest,
                         cudaStream_t s) {
  const int64_t nb = n / kQkK;
  if (type == CSK_GGML_Q4_K) {
    const int grid = grid_for((size_t)nb * 4 * 32, 256, 8192);
    if (nearest) k_dequant_q4k<true><<<grid, 256, 0, s>>>(d_raw, d_f16, nb);
    else k_dequant_q4k<false><<<grid, 256, 0, s>>>(d_raw, d_f16, nb);
  } else {
    const int grid = grid_for((size_t)nb * 2 * 32, 256, 8192);
    if (nearest) k_dequant_q6k<true><<<grid, 256, 0, s>>>(d_raw, d_f16, nb);
    else k_dequant_q6k<false><<<grid, 256, 0, s>>>(d_raw, d_f16, nb);
  }
}
}  // namespace

int csk_moe_load_expert_ggml(csk_moe_layer* L, int32_t expert_id, int32_t type_up, const void* w_up,
                             int32_t type_gate, const void* w_gate, int32_t type_down, const void* w_down,
                             const float* b_up, const float* b_gate, const float* b_down, int32_t f16_rounding) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!L->w16)
    return fail(L, CSK_ERR_INVALID, "this layer holds MXFP4 weights: Q4_K / Q6_K / F16 slices need a layer created "
                                    "with CSK_WEIGHTS_F16");
  if (expert_id < L->e0 || expert_id >= L->e0 + L->Eloc)
    return fail(L, CSK_ERR_INVALID, "expert %d is not resident on this device (range [%d,%d))",
                expert_id, L->e0, L->e0 + L->Eloc);
  if (!w_up || !w_gate || !w_down) return fail(L, CSK_ERR_INVALID, "null weight pointer");
  if (L->cfg.has_bias && (!b_up || !b_gate || !b_down))
    return fail(L, CSK_ERR_INVALID, "layer has biases but a bias pointer is null");
  if (f16_rounding != CSK_F16_TRUNCATE && f16_rounding != CSK_F16_NEAREST)
    return fail(L, CSK_ERR_INVALID, "f16_rounding must be CSK_F16_TRUNCATE or CSK_F16_NEAREST, got %d", f16_rounding);
  const int32_t types[3] = {type_up, type_gate, type_down};
  const void* src[3] = {w_up, w_gate, w_down};
  const int64_t n = (int64_t)L->H * L->F;  // a multiple of 1024: whole super-blocks
  for (int i = 0; i < 3; ++i)
    if (types[i] != CSK_GGML_F16 && types[i] != CSK_GGML_Q4_K && types[i] != CSK_GGML_Q6_K)
      return fail(L, CSK_ERR_INVALID, "ggml type %d is not handled (F16 = %d, Q4_K = %d, Q6_K = %d)", types[i],
                  CSK_GGML_F16, CSK_GGML_Q4_K, CSK_GGML_Q6_K);
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  if (!L->d_stage2) {
    cudaError_t e = cudaMalloc(&L->d_stage2, 3 * L->stage_bytes);
    if (e != cudaSuccess) return fail(L, CSK_ERR_NOMEM, "cudaMalloc failed: %s", cudaGetErrorString(e));
  }
  cudaStream_t s = L->stream;
  for (int i = 0; i < 3; ++i) {
    uint8_t* f16 = L->d_stage + (size_t)i * L->stage_bytes;
    if (types[i] == CSK_GGML_F16) {
      CSK_CUDA(L, cudaMemcpyAsync(f16, src[i], L->stage_bytes, cudaMemcpyHostToDevice, s));
    } else {
      // the blocks are smaller than the fp16 matrix: they fit the second staging area's slot
      uint8_t* raw = L->d_stage2 + (size_t)i * L->stage_bytes;
      CSK_CUDA(L, cudaMemcpyAsync(raw, src[i], ggml_bytes(types[i], n), cudaMemcpyHostToDevice, s));
      ggml_decode_enqueue(types[i], raw, reinterpret_cast<unsigned short*>(f16), n, f16_rounding == CSK_F16_NEAREST, s);
    }
  }
  CSK_CUDA(L, cudaGetLastError());
  const int le = expert_id - L->e0;
  int rc = load_expert_enqueue(L, le, nullptr, nullptr, nullptr, b_up, b_gate, b_down, L->d_stage, s);
  if (rc) return rc;
  CSK_CUDA(L, cudaStreamSynchronize(s));
  L->resident[le] = 1;
  return CSK_OK;
}

int csk_moe_load_expert_f32(csk_moe_layer* L, int32_t expert_id, const float* w_up, const float* w_gate,
                            const float* w_down, const float* b_up, const float* b_gate, const float* b_down) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!L->w16)
    return fail(L, CSK_ERR_INVALID, "this layer holds MXFP4 weights: fp32 matrices need a layer created with CSK_WEIGHTS_F16");
  if (expert_id < L->e0 || expert_id >= L->e0 + L->Eloc)
    return fail(L, CSK_ERR_INVALID, "expert %d is not resident on this device (range [%d,%d))",
                expert_id, L->e0, L->e0 + L->Eloc);
  if (!w_up || !w_gate || !w_down) return fail(L, CSK_ERR_INVALID, "null weight pointer");
  if (L->cfg.has_bias && (!b_up || !b_gate || !b_down))
    return fail(L, CSK_ERR_INVALID, "layer has biases but a bias pointer is null");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  const int64_t n = (int64_t)L->H * L->F;
  // one fp32 matrix at a time through a temporary of its size (load time only), plus the overflow counter
  uint8_t* tmp = nullptr;
  cudaError_t e = cudaMalloc(&tmp, (size_t)n * 4 + 16);
  if (e != cudaSuccess) return fail(L, CSK_ERR_NOMEM, "cudaMalloc failed: %s", cudaGetErrorString(e));
  int* d_over = reinterpret_cast<int*>(tmp + (size_t)n * 4);
  cudaStream_t s = L->stream;
  const float* src[3] = {w_up, w_gate, w_down};
  int over = 0;
  e = cudaMemsetAsync(d_over, 0, 4, s);
  for (int i = 0; i < 3 && e == cudaSuccess; ++i) {
    e = cudaMemcpyAsync(tmp, src[i], (size_t)n * 4, cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) break;
    k_f32_to_f16<<<grid_for((size_t)n, 256, 4096), 256, 0, s>>>(
        reinterpret_cast<const float*>(tmp), reinterpret_cast<unsigned short*>(L->d_stage + (size_t)i * L->stage_bytes), n, d_over);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(&over, d_over, 4, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFree(tmp);
  if (e != cudaSuccess) return fail(L, CSK_ERR_CUDA, "load_expert_f32: %s", cudaGetErrorString(e));
  if (over)
    return fail(L, CSK_ERR_INVALID, "load_expert_f32: a weight lies beyond the fp16 range (|w| > 65504); the tensor-core "
                                    "kernel's operands are fp16");
  const int le = expert_id - L->e0;
  int rc = load_expert_enqueue(L, le, nullptr, nullptr, nullptr, b_up, b_gate, b_down, L->d_stage, s);
  if (rc) return rc;
  CSK_CUDA(L, cudaStreamSynchronize(s));
  L->resident[le] = 1;
  return CSK_OK;
}

int csk_moe_dequant_ggml_f16(int32_t device, int32_t ggml_type, const void* blocks, int64_t n_elements, uint16_t* out_f16,
                         int32_t f16_rounding) {
  if (!blocks || !out_f16) return fail(nullptr, CSK_ERR_INVALID, "dequant_ggml: null argument");
  if (ggml_type != CSK_GGML_Q4_K && ggml_type != CSK_GGML_Q6_K)
    return fail(nullptr, CSK_ERR_INVALID, "dequant_ggml: ggml type %d is not handled (Q4_K = %d, Q6_K = %d)", ggml_type,
                CSK_GGML_Q4_K, CSK_GGML_Q6_K);
  if (n_elements <= 0 || n_elements % kQkK)
    return fail(nullptr, CSK_ERR_INVALID, "dequant_ggml: the element count must be a positive multiple of %d, got %lld",
                kQkK, (long long)n_elements);
  if (f16_rounding != CSK_F16_TRUNCATE && f16_rounding != CSK_F16_NEAREST)
    return fail(nullptr, CSK_ERR_INVALID, "dequant_ggml: f16_rounding must be CSK_F16_TRUNCATE or CSK_F16_NEAREST");
  if (!csk_moe_device_ok(device)) return fail(nullptr, CSK_ERR_CUDA, "dequant_ggml: device %d is not an sm_100 GPU; no CPU fallback exists", device);
  CSK_CUDA(nullptr, cudaSetDevice(device));
  const size_t qb = ggml_bytes(ggml_type, n_elements);
  uint8_t* d_raw = nullptr;
  unsigned short* d_out = nullptr;
  cudaError_t e = cudaMalloc(&d_raw, qb);
  if (e == cudaSuccess) e = cudaMalloc(&d_out, (size_t)n_elements * 2);
  if (e != cudaSuccess) {
    cudaFree(d_raw);
    return fail(nullptr, CSK_ERR_NOMEM, "dequant_ggml: cudaMalloc failed: %s", cudaGetErrorString(e));
  }
  e = cudaMemcpy(d_raw, blocks, qb, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    ggml_decode_enqueue(ggml_type, d_raw, d_out, n_elements, f16_rounding == CSK_F16_NEAREST, 0);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out_f16, d_out, (size_t)n_elements * 2, cudaMemcpyDeviceToHost);
  cudaFree(d_raw);
  cudaFree(d_out);
  if (e != cudaSuccess) return fail(nullptr, CSK_ERR_CUDA, "dequant_ggml: %s", cudaGetErrorString(e));
  return CSK_OK;
}

int csk_moe_load_experts_mxfp4(csk_moe_layer* L, int32_t first_expert, int32_t count, const uint8_t* w_up,
                               const uint8_t* w_gate, const uint8_t* w_down, const float* b_up, const float* b_gate,
                               const float* b_down) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (L->w16) return fail(L, CSK_ERR_INVALID, "this layer holds fp16 weights: use csk_moe_load_expert_f16");
  if (count <= 0 || first_expert < L->e0 || first_expert + count > L->e0 + L->Eloc)
    return fail(L, CSK_ERR_INVALID, "experts [%d,%d) are not all resident on this device (range [%d,%d))", first_expert,
                first_expert + count, L->e0, L->e0 + L->Eloc);
  if (!w_up || !w_gate || !w_down) return fail(L, CSK_ERR_INVALID, "null weight pointer");
  if (L->cfg.has_bias && (!b_up || !b_gate || !b_down))
    return fail(L, CSK_ERR_INVALID, "layer has biases but a bias pointer is null");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  if (!L->d_stage2) {
    cudaError_t e = cudaMalloc(&L->d_stage2, 3 * L->stage_bytes);
    if (e != cudaSuccess) return fail(L, CSK_ERR_NOMEM, "cudaMalloc failed: %s", cudaGetErrorString(e));
  }
  // two staging areas: the copies of expert i+1 run while expert i is repacked
  cudaStream_t s = L->stream, s2 = L->stream_in;
  for (int i = 0; i < count; ++i) {
    const int le = first_expert - L->e0 + i;
    cudaStream_t st = (i & 1) ? s2 : s;
    uint8_t* stage = (i & 1) ? L->d_stage2 : L->d_stage;
    const size_t wb = L->stage_bytes;
    int rc = load_expert_enqueue(L, le, w_up + (size_t)i * wb, w_gate + (size_t)i * wb, w_down + (size_t)i * wb,
                                 b_up ? b_up + (size_t)i * L->F : nullptr, b_gate ? b_gate + (size_t)i * L->F : nullptr,
                                 b_down ? b_down + (size_t)i * L->H : nullptr, stage, st);
    if (rc) return rc;
  }
  CSK_CUDA(L, cudaStreamSynchronize(s));
  CSK_CUDA(L, cudaStreamSynchronize(s2));
  for (int i = 0; i < count; ++i) L->resident[first_expert - L->e0 + i] = 1;
  return CSK_OK;
}

namespace {
struct ImageHeader {
  char magic[8];
  int32_t E, k, H, F, has_bias, e0, eloc, reserved;
  uint64_t expert_stride, off_gu, off_d, off_tgu, off_td, off_bias, off_meta;
};
ImageHeader image_header_of(const csk_moe_layer* L) {
  ImageHeader h{};
  memcpy(h.magic, "CSKMOE03", 8);  // 03: the block-scaled kernel's layout; it stores scale byte 255 as 254
  h.E = L->E; h.k = L->k; h.H = L->H; h.F = L->F; h.has_bias = L->cfg.has_bias; h.e0 = L->e0; h.eloc = L->Eloc;
  h.expert_stride = L->expert_stride; h.off_gu = L->off_gu; h.off_d = L->off_d; h.off_tgu = L->off_tgu;
  h.off_td = L->off_td; h.off_bias = L->off_bias; h.off_meta = L->off_meta;
  return h;
}
// The header of an image of the layout before this one (02).  It differs in the first part of an expert's record only: the
// decode kernel's copy of the codes was cut into records of 544 bytes, 16 rows x 64 columns.  What follows, from the other
// kernel's tiles on, is the same.
ImageHeader image_header_02(const csk_moe_layer* L) {
  ImageHeader h = image_header_of(L);
  memcpy(h.magic, "CSKMOE02", 8);
  if (L->w16) return h;  // fp16 weights have no such copy
  auto bytes = [](int N, int K, int parts) {
    return ((size_t)ceil_div(N, 16) * ceil_div(K, 64) * parts * 544 + 255) / 256 * 256;
  };
  h.off_d = bytes(L->F, L->H, 2);
  const uint64_t off_tgu = h.off_d + bytes(L->H, L->F, 1);
  for (uint64_t* o : {&h.off_td, &h.off_bias, &h.off_meta}) *o = *o - h.off_tgu + off_tgu;
  h.off_tgu = off_tgu;
  h.expert_stride = (h.off_meta + 16 + 255) / 256 * 256;
  return h;
}
// An expert's tensor-core codes to the file's order (from the device into the staging area) or from it (and back).
int reorder_tiles_enqueue(csk_moe_layer* L, int le, bool to_file, cudaStream_t s) {
  uint8_t* base = L->d_weights + (size_t)le * L->expert_stride + L->off_tgu;
  uint8_t* part = L->d_stage;
  for (const auto& [lay, at] : {std::pair{L->Tgu, (size_t)0}, std::pair{L->Td, L->off_td - L->off_tgu}})
    k_reorder_tile<<<grid_for(lay.bytes() / (lay.w16 ? 128 : 34), 256, 4096), 256, 0, s>>>(to_file ? base + at : part + at, to_file ? part + at : base + at, lay,
                                                                       to_file);
  CSK_CUDA(L, cudaGetLastError());
  return CSK_OK;
}
// The decode kernel's copy of a resident expert's codes from the other kernel's tiles (which hold the blocks losslessly).
int rebuild_mx_enqueue(csk_moe_layer* L, int le, cudaStream_t s) {
  uint8_t* base = L->d_weights + (size_t)le * L->expert_stride;
  uint8_t *s_up = L->d_stage, *s_gate = L->d_stage + L->stage_bytes, *s_down = L->d_stage + 2 * L->stage_bytes;
  int* emeta = reinterpret_cast<int*>(base + L->off_meta);
  const int grid = grid_for((size_t)L->F * (L->H / 32), 128, 4096);
  k_unpack_tile<<<grid, 128, 0, s>>>(base + L->off_tgu, s_gate, L->Tgu, 0);
  k_unpack_tile<<<grid, 128, 0, s>>>(base + L->off_tgu, s_up, L->Tgu, 1);
  k_unpack_tile<<<grid, 128, 0, s>>>(base + L->off_td, s_down, L->Td, 0);
  k_mx_repack<<<grid_for(L->Lgu.bytes() / 16, 256, 4096), 256, 0, s>>>(s_gate, s_up, base + L->off_gu, L->Lgu, emeta);
  k_mx_repack<<<grid_for(L->Ld.bytes() / 16, 256, 4096), 256, 0, s>>>(s_down, nullptr, base + L->off_d, L->Ld, emeta + 1);
  CSK_CUDA(L, cudaGetLastError());
  return CSK_OK;
}
}  // namespace

int csk_moe_save_image(csk_moe_layer* L, const char* path) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!path) return fail(L, CSK_ERR_INVALID, "null path");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  const size_t part = image_part_bytes(L);
  FILE* f = fopen(path, "wb");
  if (!f) return fail(L, CSK_ERR_INVALID, "cannot open %s for writing", path);
  const ImageHeader h = image_header_of(L);
  bool ok = fwrite(&h, sizeof h, 1, f) == 1 && fwrite(L->resident.data(), 1, L->Eloc, f) == (size_t)L->Eloc;
  std::vector<uint8_t> buf(L->expert_stride);
  for (int e = 0; ok && e < L->Eloc; ++e) {
    if (cudaMemcpy(buf.data(), L->d_weights + (size_t)e * L->expert_stride, L->expert_stride, cudaMemcpyDeviceToHost) != cudaSuccess) ok = false;
    if (ok && part) {
      ok = reorder_tiles_enqueue(L, e, true, L->stream) == CSK_OK && cudaStreamSynchronize(L->stream) == cudaSuccess &&
           cudaMemcpy(buf.data() + L->off_tgu, L->d_stage, part, cudaMemcpyDeviceToHost) == cudaSuccess;
    }
    ok = ok && fwrite(buf.data(), 1, buf.size(), f) == buf.size();
  }
  ok = fclose(f) == 0 && ok;
  if (!ok) return fail(L, CSK_ERR_CUDA, "writing the weight image to %s failed", path);
  return CSK_OK;
}

int csk_moe_load_image(csk_moe_layer* L, const char* path) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!path) return fail(L, CSK_ERR_INVALID, "null path");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  const size_t part = image_part_bytes(L);
  FILE* f = fopen(path, "rb");
  if (!f) return fail(L, CSK_ERR_INVALID, "cannot open %s", path);
  ImageHeader h{};
  const ImageHeader want = image_header_of(L), before = image_header_02(L);
  std::vector<uint8_t> res(L->Eloc);
  bool ok = fread(&h, sizeof h, 1, f) == 1;
  const bool older = ok && memcmp(&h, &before, sizeof h) == 0;
  if (ok && !older && memcmp(&h, &want, sizeof h) != 0) {
    fclose(f);
    return fail(L, CSK_ERR_INVALID, "%s was written for another layer shape, expert range or library layout", path);
  }
  ok = ok && fread(res.data(), 1, L->Eloc, f) == (size_t)L->Eloc;
  const bool rebuild = older && !L->w16;
  const size_t from = rebuild ? h.off_tgu : 0, to = rebuild ? L->off_tgu : 0;
  std::vector<uint8_t> buf(h.expert_stride);
  for (int e = 0; ok && e < L->Eloc; ++e) {
    uint8_t* base = L->d_weights + (size_t)e * L->expert_stride;
    ok = fread(buf.data(), 1, buf.size(), f) == buf.size();
    // (on the handle's stream, which does not wait for the default one: a plain copy may still be landing when it returns)
    ok = ok && cudaMemcpyAsync(base + to, buf.data() + from, h.off_meta + 16 - from, cudaMemcpyHostToDevice, L->stream) == cudaSuccess;
    if (ok && part)
      ok = cudaMemcpyAsync(L->d_stage, base + L->off_tgu, part, cudaMemcpyDeviceToDevice, L->stream) == cudaSuccess &&
           reorder_tiles_enqueue(L, e, false, L->stream) == CSK_OK;
    if (ok && rebuild && res[e]) ok = rebuild_mx_enqueue(L, e, L->stream) == CSK_OK;
    ok = cudaStreamSynchronize(L->stream) == cudaSuccess && ok;
  }
  fclose(f);
  if (!ok) return fail(L, CSK_ERR_CUDA, "reading the weight image from %s failed", path);
  CSK_CUDA(L, cudaMemcpy(L->d_resident, res.data(), L->Eloc, cudaMemcpyHostToDevice));
  L->resident = res;
  return CSK_OK;
}

int csk_moe_unpack_expert_mxfp4(csk_moe_layer* L, int32_t expert_id, int32_t which, uint8_t* out) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (expert_id < L->e0 || expert_id >= L->e0 + L->Eloc || !L->resident[expert_id - L->e0])
    return fail(L, CSK_ERR_MISSING, "expert %d is not loaded", expert_id);
  if (which < 0 || which > 5 || !out) return fail(L, CSK_ERR_INVALID, "bad argument");
  if (L->w16) return fail(L, CSK_ERR_INVALID, "this layer holds fp16 weights, not MXFP4 blocks");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  const uint8_t* base = L->d_weights + (size_t)(expert_id - L->e0) * L->expert_stride;
  if (which < 3) {
    const MxLayout& lay = which == 2 ? L->Ld : L->Lgu;
    const uint8_t* packed = base + (which == 2 ? L->off_d : L->off_gu);
    k_mx_unpack<<<grid_for((size_t)lay.N * (lay.K / 32), 128, 4096), 128, 0, L->stream>>>(
        packed, L->d_stage, lay, which == 0 ? 1 : 0);
  } else {
    const int w = which - 3;
    const TileLayout& lay = w == 2 ? L->Td : L->Tgu;
    const uint8_t* packed = base + (w == 2 ? L->off_td : L->off_tgu);
    k_unpack_tile<<<grid_for((size_t)lay.N * (lay.K / 32), 128, 4096), 128, 0, L->stream>>>(
        packed, L->d_stage, lay, w == 0 ? 1 : 0);
  }
  CSK_CUDA(L, cudaGetLastError());
  CSK_CUDA(L, cudaMemcpyAsync(out, L->d_stage, L->stage_bytes, cudaMemcpyDeviceToHost, L->stream));
  CSK_CUDA(L, cudaStreamSynchronize(L->stream));
  return CSK_OK;
}

int csk_moe_expert_resident(const csk_moe_layer* L, int32_t expert_id) {
  if (!L || expert_id < L->e0 || expert_id >= L->e0 + L->Eloc) return 0;
  return L->resident[expert_id - L->e0];
}

int csk_moe_set_path(csk_moe_layer* L, int32_t path) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (path < CSK_PATH_AUTO || path > CSK_PATH_TILE_PAIR) return fail(L, CSK_ERR_INVALID, "unknown path %d", path);
  if (L->w16 && (path == CSK_PATH_STREAM || path == CSK_PATH_TILE_PAIR))
    return fail(L, CSK_ERR_INVALID, "fp16 weights have no weight-streaming kernel, and their CTA-pair kernel is not chosen by name");
  if (path == CSK_PATH_TILE_PAIR && !L->pair.available)
    return fail(L, CSK_ERR_INVALID, "the CTA-pair kernel is not available on this device: %s", L->pair.err.c_str());
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  if (path == CSK_PATH_STREAM) {  // any batch may come: images for all of it
    int rc = mx_reserve(L, L->max_rows);
    if (rc) return rc;
  }
  L->path = path;
  drop_graphs(L);
  return CSK_OK;
}

int csk_moe_set_activation(csk_moe_layer* L, int32_t activation, int32_t weight_before_ffn) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (activation != CSK_ACT_MODIFIED_SWIGLU && activation != CSK_ACT_STANDARD_SWIGLU)
    return fail(L, CSK_ERR_INVALID, "unknown activation %d", activation);
  if (L->cfg.activation == activation && (L->cfg.weight_before_ffn != 0) == (weight_before_ffn != 0)) return CSK_OK;
  L->cfg.activation = activation;
  L->cfg.weight_before_ffn = weight_before_ffn != 0;
  drop_graphs(L);
  return CSK_OK;
}

int csk_moe_set_router_mode(csk_moe_layer* L, int32_t mode) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (mode < CSK_ROUTER_AUTO || mode > CSK_ROUTER_CERTIFIED) return fail(L, CSK_ERR_INVALID, "unknown router mode %d", mode);
  L->router_mode = mode;
  drop_graphs(L);
  return CSK_OK;
}

int csk_moe_get_router_stats(csk_moe_layer* L, int64_t* routed_tokens, int64_t* chain_tokens) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  unsigned long long fb = 0;
  CSK_CUDA(L, cudaMemcpy(&fb, L->d_fb + 2, sizeof(fb), cudaMemcpyDeviceToHost));
  if (routed_tokens) *routed_tokens = L->routed_tokens;
  if (chain_tokens) *chain_tokens = (int64_t)fb;
  return CSK_OK;
}

int csk_moe_enable_timing(csk_moe_layer* L, int32_t on) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  L->timing = on != 0;
  return CSK_OK;
}

int csk_moe_sync(csk_moe_layer* L) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  int rc = check_device_status(L, L->last_stream ? L->last_stream : L->stream);
  if (rc) return rc;
  if (L->timing && L->n_marks > 1) finish_timings(L, L->n_marks, L->last_routed);
  return CSK_OK;
}

int csk_moe_get_timings(csk_moe_layer* L, csk_moe_timings* out) {
  if (check_layer(L) || !out) return CSK_ERR_INVALID;
  *out = L->last;
  return CSK_OK;
}

int csk_moe_get_counters(csk_moe_layer* L, int64_t* rows_per_expert, int64_t* distinct,
                         int64_t* weight_bytes) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  std::vector<int> c(L->E);
  CSK_CUDA(L, cudaMemcpy(c.data(), L->counts_in_carry ? L->d_carry + 1 : L->d_counts, sizeof(int) * L->E,
                         cudaMemcpyDeviceToHost));
  int64_t d = 0;
  for (int e = 0; e < L->E; ++e) {
    if (rows_per_expert) rows_per_expert[e] = c[e];
    if (c[e] > 0) ++d;
  }
  if (distinct) *distinct = d;
  if (weight_bytes) {
    const int64_t per = (int64_t)3 * L->H * L->F / 32 * 17 +
                        (L->cfg.has_bias ? (int64_t)sizeof(float) * (2 * L->F + L->H) : 0);
    *weight_bytes = d * per;
  }
  return CSK_OK;
}

// ---- device-buffer entry points -------------------------------------------
int csk_moe_route_dev(csk_moe_layer* L, const float* d_hidden, int64_t T, float* d_router_out, void* stream) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!d_hidden || !d_router_out) return fail(L, CSK_ERR_INVALID, "null argument");
  if (T <= 0 || T > L->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld outside (0, max_tokens]", (long long)T);
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  L->last = csk_moe_timings{};
  const PdlScope pdl_scope(L);
  return launch_router(L, d_hidden, T, d_router_out, pick(L, stream));
}

// forward_dev, small batches as captured sequences
static int forward_replayed(csk_moe_layer* L, const float* d_hidden, int64_t T, const float* d_router_in, float* d_router_out, float* d_out,
                            cudaStream_t s, const HostResult& host = {}) {
  auto enqueue = [&]() { return forward_dev(L, d_hidden, T, d_router_in, d_router_out, d_out, -1, s, false, nullptr, nullptr, nullptr, host); };
  constexpr int64_t kGraphMaxTokens = 512;
  if (!L->use_graphs || L->timing || L->debug_stall || L->debug_stall_router || T > kGraphMaxTokens || T <= 0 || T > L->max_T)
    return enqueue();
  for (auto& g : L->graphs)
    if (g.T == T && g.hidden == d_hidden && g.router_in == d_router_in && g.router_out == d_router_out &&
        g.out == d_out && g.host_router == host.router && g.stream == s) {
      CSK_CUDA(L, cudaGraphLaunch(g.exec, s));
      L->last_T = T;
      L->last_stream = s;
      L->n_marks = 0;
      return CSK_OK;
    }
  // first call with these arguments: capture the sequence, then replay it
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone) {
    cudaGetLastError();  // the caller is capturing this stream itself: just enqueue
    return enqueue();
  }
  if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    cudaGetLastError();
    return enqueue();
  }
  int rc = enqueue();
  cudaGraph_t graph = nullptr;
  cudaError_t ce = cudaStreamEndCapture(s, &graph);
  if (rc || ce != cudaSuccess || !graph) {
    cudaGetLastError();
    if (graph) cudaGraphDestroy(graph);
    if (rc) return rc;
    L->use_graphs = false;  // capture is not possible here: fall back to plain launches for good
    return enqueue();
  }
  cudaGraphExec_t exec = nullptr;
  ce = cudaGraphInstantiate(&exec, graph, 0);
  cudaGraphDestroy(graph);
  if (ce != cudaSuccess || !exec) {
    cudaGetLastError();
    L->use_graphs = false;
    return enqueue();
  }
  if (L->graphs.size() >= 32) {
    cudaGraphExecDestroy(L->graphs.front().exec);
    L->graphs.erase(L->graphs.begin());
  }
  L->graphs.push_back({T, d_hidden, d_router_in, d_router_out, d_out, host.router, s, exec});
  CSK_CUDA(L, cudaGraphLaunch(exec, s));
  return CSK_OK;
}

int csk_moe_forward_dev(csk_moe_layer* L, const float* d_hidden, int64_t T, const float* d_router_in,
                        float* d_router_out, float* d_out, void* stream) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!d_hidden || !d_out) return fail(L, CSK_ERR_INVALID, "null argument");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  return forward_replayed(L, d_hidden, T, d_router_in, d_router_out, d_out, pick(L, stream));
}

// ---- the layer with the steps either side of it ------------------------------
int csk_moe_set_ffn_norm(csk_moe_layer* L, const float* weight, float eps) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!weight) return fail(L, CSK_ERR_INVALID, "norm weight is null");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  if (!L->d_norm_w) {
    cudaError_t e = cudaMalloc(&L->d_norm_w, sizeof(float) * L->H);
    if (e == cudaSuccess) e = cudaMalloc(&L->d_normed, sizeof(float) * L->max_T * L->H);
    if (e != cudaSuccess) return fail(L, CSK_ERR_NOMEM, "cudaMalloc failed: %s", cudaGetErrorString(e));
    // any layer's row: the attribute is the function's, not the layer's
    CSK_CUDA(L, cudaFuncSetAttribute(k_rmsnorm<kNormThreadsFew, kNormKeptFew>, cudaFuncAttributeMaxDynamicSharedMemorySize, 50 * 1024));
    CSK_CUDA(L, cudaFuncSetAttribute(k_rmsnorm<kNormThreadsMany, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 50 * 1024));
  }
  CSK_CUDA(L, cudaMemcpyAsync(L->d_norm_w, weight, sizeof(float) * L->H, cudaMemcpyHostToDevice, L->stream));
  CSK_CUDA(L, cudaStreamSynchronize(L->stream));
  L->norm_eps = eps;
  return CSK_OK;
}

static cudaError_t launch_norm(csk_moe_layer* L, const float* d_x, int64_t T, cudaStream_t s) {
  const bool few = norm_few(T, L->sm_count);
  return launch_k(few ? k_rmsnorm<kNormThreadsFew, kNormKeptFew> : k_rmsnorm<kNormThreadsMany, 0>,
                  dim3((unsigned)std::min<int64_t>(T, 16 * (int64_t)L->sm_count)), dim3(few ? kNormThreadsFew : kNormThreadsMany),
                  sizeof(float) * L->H, s, !L->timing, d_x, (const float*)L->d_norm_w, L->norm_eps, L->d_normed, (int)T, L->H);
}

int csk_moe_block_forward_dev(csk_moe_layer* L, const float* d_x, int64_t T, float* d_router_out, float* d_out,
                              void* stream) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!d_x || !d_out) return fail(L, CSK_ERR_INVALID, "null argument");
  if (!L->d_norm_w) return fail(L, CSK_ERR_INVALID, "the norm weight was never set (csk_moe_set_ffn_norm)");
  if (T <= 0 || T > L->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld outside (0, max_tokens]", (long long)T);
  if (reinterpret_cast<uintptr_t>(d_x) % 16 || reinterpret_cast<uintptr_t>(d_out) % 16)
    return fail(L, CSK_ERR_INVALID, "activations must be 16-byte aligned");
  if ((size_t)L->H * sizeof(float) * 4 > 200 * 1024) return fail(L, CSK_ERR_NOMEM, "hidden dimension too large for the norm kernel's row buffer");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = pick(L, stream);
  CSK_CUDA(L, launch_norm(L, d_x, T, s));
  return forward_dev(L, L->d_normed, T, nullptr, d_router_out, d_out, -1, s, false, d_x);
}

int csk_moe_block_forward_shared_dev(csk_moe_layer* L, csk_moe_layer* S, const float* d_x, int64_t T,
                                     float* d_router_out, float* d_out, void* stream) {
  if (!S) return csk_moe_block_forward_dev(L, d_x, T, d_router_out, d_out, stream);
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!d_x || !d_out) return fail(L, CSK_ERR_INVALID, "null argument");
  if (!L->d_norm_w) return fail(L, CSK_ERR_INVALID, "the norm weight was never set (csk_moe_set_ffn_norm)");
  if (T <= 0 || T > L->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld outside (0, max_tokens]", (long long)T);
  if (S == L || !S->d_unit_router || S->H != L->H || S->cfg.device != L->cfg.device)
    return fail(L, CSK_ERR_INVALID, "the shared expert must be another layer on the same device with num_experts = top_k = 1 "
                                    "and the same hidden size");
  if (T > S->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld exceeds the shared expert's max_tokens", (long long)T);
  if (!S->resident[0]) return fail(L, CSK_ERR_MISSING, "the shared expert's weights are not loaded");
  if (reinterpret_cast<uintptr_t>(d_x) % 16 || reinterpret_cast<uintptr_t>(d_out) % 16)
    return fail(L, CSK_ERR_INVALID, "activations must be 16-byte aligned");
  if ((size_t)L->H * sizeof(float) * 4 > 200 * 1024) return fail(L, CSK_ERR_NOMEM, "hidden dimension too large for the norm kernel's row buffer");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  if (!L->d_shared_out) {
    cudaError_t e = cudaMalloc(&L->d_shared_out, sizeof(float) * L->max_T * L->H);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&L->ev_shared_fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&L->ev_shared_join, cudaEventDisableTiming);
    if (e != cudaSuccess) return fail(L, CSK_ERR_NOMEM, "shared-expert buffers: %s", cudaGetErrorString(e));
  }
  cudaStream_t s = pick(L, stream);
  CSK_CUDA(L, launch_norm(L, d_x, T, s));
  // the shared expert reads the normed rows on its own stream, next to the routed experts; the combine joins them
  CSK_CUDA(L, cudaEventRecord(L->ev_shared_fork, s));
  CSK_CUDA(L, cudaStreamWaitEvent(S->stream, L->ev_shared_fork, 0));
  int rc = csk_moe_dense_forward_dev(S, L->d_normed, T, L->d_shared_out, S->stream);
  if (rc) return fail(L, rc, "shared expert: %s", S->err.c_str());
  CSK_CUDA(L, cudaEventRecord(L->ev_shared_join, S->stream));
  return forward_dev(L, L->d_normed, T, nullptr, d_router_out, d_out, -1, s, false, d_x, L->d_shared_out, L->ev_shared_join);
}

int csk_moe_block_forward_shared(csk_moe_layer* L, csk_moe_layer* S, const float* x, int64_t T, float* router_out,
                                 float* out) {
  if (!S) return csk_moe_block_forward(L, x, T, router_out, out);
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!x || !out) return fail(L, CSK_ERR_INVALID, "null argument");
  if (T <= 0 || T > L->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld outside (0, max_tokens]", (long long)T);
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = L->stream;
  CSK_CUDA(L, cudaMemcpyAsync(L->d_hidden, x, sizeof(float) * T * L->H, cudaMemcpyHostToDevice, s));
  int rc = csk_moe_block_forward_shared_dev(L, S, L->d_hidden, T, L->d_router, L->d_out, s);
  if (rc) return rc;
  rc = check_device_status(L, s);
  if (rc) return rc;
  rc = check_device_status(S, S->stream);
  if (rc) return fail(L, rc, "shared expert: %s", S->err.c_str());
  CSK_CUDA(L, cudaMemcpyAsync(out, L->d_out, sizeof(float) * T * L->H, cudaMemcpyDeviceToHost, s));
  if (router_out)
    CSK_CUDA(L, cudaMemcpyAsync(router_out, L->d_router, sizeof(float) * T * L->k * 2, cudaMemcpyDeviceToHost, s));
  CSK_CUDA(L, cudaStreamSynchronize(s));
  return CSK_OK;
}

int csk_moe_block_forward(csk_moe_layer* L, const float* x, int64_t T, float* router_out, float* out) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!x || !out) return fail(L, CSK_ERR_INVALID, "null argument");
  if (T <= 0 || T > L->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld outside (0, max_tokens]", (long long)T);
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = L->stream;
  CSK_CUDA(L, cudaMemcpyAsync(L->d_hidden, x, sizeof(float) * T * L->H, cudaMemcpyHostToDevice, s));
  int rc = csk_moe_block_forward_dev(L, L->d_hidden, T, L->d_router, L->d_out, s);
  if (rc) return rc;
  rc = check_device_status(L, s);
  if (rc) return rc;
  CSK_CUDA(L, cudaMemcpyAsync(out, L->d_out, sizeof(float) * T * L->H, cudaMemcpyDeviceToHost, s));
  if (router_out)
    CSK_CUDA(L, cudaMemcpyAsync(router_out, L->d_router, sizeof(float) * T * L->k * 2, cudaMemcpyDeviceToHost, s));
  CSK_CUDA(L, cudaStreamSynchronize(s));
  return CSK_OK;
}

// ---- host-buffer entry points ----------------------------------------------
int csk_moe_route(csk_moe_layer* L, const float* hidden, int64_t T, float* router_out) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!hidden || !router_out) return fail(L, CSK_ERR_INVALID, "null argument");
  if (T <= 0 || T > L->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld outside (0, max_tokens]", (long long)T);
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = L->stream;
  L->last = csk_moe_timings{};
  CSK_CUDA(L, cudaMemcpyAsync(L->d_hidden, hidden, sizeof(float) * T * L->H, cudaMemcpyHostToDevice, s));
  const PdlScope pdl_scope(L);
  int rc = launch_router(L, L->d_hidden, T, L->d_router, s);
  if (rc) return rc;
  CSK_CUDA(L, cudaMemcpyAsync(router_out, L->d_router, sizeof(float) * T * L->k * 2, cudaMemcpyDeviceToHost, s));
  CSK_CUDA(L, cudaStreamSynchronize(s));
  return CSK_OK;
}

namespace {
// What memory a buffer is in: page-locked (Host), pageable (Unregistered), or the device's or managed.
cudaMemoryType memory_of(const void* p) {
  cudaPointerAttributes at{};
  if (cudaPointerGetAttributes(&at, p) == cudaSuccess) return at.type;
  cudaGetLastError();
  return cudaMemoryTypeManaged;
}
// Whether every buffer of a call (null: not given) is page-locked.
bool page_locked(std::initializer_list<const void*> buffers) {
  for (const void* p : buffers)
    if (p && memory_of(p) != cudaMemoryTypeHost) return false;
  return true;
}

// How many equal passes the host entry point cuts a batch into so that the copies of one pass overlap the kernels of another.
// Pageable buffers: two from 600 rows per expert on.  Their copies block the caller, so a pass is enqueued only when the one before
// it has been copied out.  1 / 2 / 4 / 8 passes, ms: 128 experts of 2880 x 2880, 4096 tokens (128 rows per expert) 7.57 / 7.59 / 7.91 / 8.99, 8192
// (256) 14.7 / 15.4 / 15.9 / 18.0; 32 experts, 2048 (256) 2.92 / 3.12 / 3.67 / 4.56, 3000 (375) 4.46 / 4.41 / 5.09 / 5.95, 8192 (1024) 13.5 / 13.4 /
// 15.2 / 15.3; 8 of 1728 x 1728, top-2, 2000 (500) 1.68 / 1.80 / 2.02 / 2.39; fp16, 32 of 2880 x 2880, 4096 (512) 6.10 / 6.32 / 6.88 / 8.35.
// Page-locked buffers: two from 128 rows per expert on, and one for every 120.  What stays exposed is the first copy in and the last
// copy out; what passes cost is kernel time, the less the more rows an expert has (a row tile's cost is nearly flat below 100
// rows).  1 / 2 / 3 / 4 / 8 passes, ms: 128 experts of 2880 x 2880, 4096 tokens 2.58 / 2.20 / 2.46 / 2.74 / 3.18; 32 experts, 1500 (187) 0.95 / 0.77 /
// 0.82 / 0.93 / 1.29, 3000 1.80 / 1.30 / 1.14 / 1.18 / 1.66, 8192 4.76 / 3.39 / 2.97 / 2.76 / 2.49; fp16, 32 of 2880 x 2880, 1500 1.03 / 1.01 / 1.16 / 1.39 /
// 2.44, 8192 4.98 / 3.47 / 3.02 / 2.80 / 3.14.  From 240 rows on three may be quicker already: the third hides a sixth of both copies and
// reads the weights once more, with 30 us of launches; the two meet where a copy has 6 MB and a 21st of the weights' bytes.  2 / 3 passes, ms
// (copy of that sum): 128 of 2880 x 2880, 240 rows 3.32 / 3.23 (1.02), 256 3.47 / 3.33 (1.09); 64, 240 1.69 / 1.69 (0.95), 256 1.78 / 1.75 (1.02), 320
// 2.17 / 1.97 (1.27); 32, 240 0.87 / 0.91 (0.85), 256 0.91 / 0.94 (0.90), 290 1.02 / 0.98 (1.02), 359 1.24 / 1.11; 8 of 1728 x 1728, 240 0.281 / 0.279 (0.85), 300
// 0.36 / 0.33 (1.06); 128 of 2048 x 768, top-8, 256 1.23 / 1.10 (1.58); 16 of 2048 x 2880, top-8, 240 0.30 / 0.34 (0.30), 300 0.33 / 0.37; 32 of 1024 x 1024, 240 0.32 /
// 0.32 (0.92), 300 0.40 / 0.35 (1.15); fp16, 16 of 2048 x 2048, 256 1.12 / 1.07 (1.33); 32 of 2880 x 2880, 300 1.23 / 1.36 (0.34); 1 of 2880 x 2880, 240 0.18 / 0.22 (0.33).  But no more than leave a pass items (a row
// tile x 128 features) for a third of the SMs: below, its kernels take as long as the whole batch's (one fp16 expert of 2880 x 2880, 150
// tokens 0.15 / 0.16 / 0.20 / 0.24 / 0.37, 1024 0.56 / 0.46 / 0.42 / 0.43 / 0.50).
// (Shorter first and last passes were up to 5 % quicker still, but the certified router adds a token's parts in an order that goes
// by the pass's size: the low bits of its weights would depend on where in the batch it stands.)
int host_passes(const csk_moe_layer* L, int64_t T, std::initializer_list<const void*> buffers) {
  if (L->timing || L->path == CSK_PATH_STREAM) return 1;
  const int64_t rows = T * L->k / std::max(1, L->Eloc);  // per expert
  if (rows < 128) return 1;
  // (a copy to or from other than page-locked memory returns when it is done)
  if (!page_locked(buffers)) return rows < 600 ? 1 : 2;
  const int least = rows < 256 ? 1 : 2;
  const int tile_rows = tile_rows_for(CSK_PATH_TILE);
  auto items = [&](int passes) { return (rows / passes + tile_rows - 1) / tile_rows * L->Eloc * L->Tgu.n_tiles; };
  int passes = (int)std::max<int64_t>(2, std::min<int64_t>(csk_moe_layer::kMaxPasses, rows / 120));
  const double weights = (L->w16 ? 2.0 : 17.0 / 32) * 3 * L->H * L->F * L->Eloc;
  if (rows >= 240 && passes == 2 && (double)sizeof(float) * T * L->H >= 6e6 + weights / 21) passes = 3;
  while (passes > least && 3 * items(passes) < L->sm_count) --passes;
  return passes;
}
// Whether a pass's results start on their way with the copy in of the pass after next (all copies in are enqueued in front then).  A copy
// out that starts in the middle of a copy in leaves the two some 65 GB/s between them, where both starting together have 80: in passes of 4
// to 12 MB that is worth the wait (smaller ones are over too soon, larger ones wait too long) if the kernels take less than a third of a
// copy's time (they take about 7.5e-5 k F of it).  At once / in step, ms (MB of a pass, k F): 8 experts of 1728 x 1024, top-4, 8192 tokens in 8 passes 1.69 / 1.48
// (7.1, 4096); 8 of 2048 x 1024, top-1, 8192 in 8 1.87 / 1.71 (8.4, 1024), 4096 in 4 1.02 / 1.00; 8 of 1024 x 2048, top-1, 8192 in 8 1.13 / 0.95 (4.2, 2048),
// 4096 in 4 0.61 / 0.54; 16 of 2048 x 2048, top-2, 4096 in 4 1.06 / 1.02 (8.4, 4096); fp16, 1 of 2880 x 2880, 4096 in 7 1.43 / 1.31 (6.7, 2880); but 8 of 512 x 512, 8192 in
// 8 0.53 / 0.59 (2.1); 16 of 2880 x 1024, top-1, 8192 in 4 2.51 / 2.69 (23.6); 16 of 2880 x 768, top-8, 4096 in 8 1.26 / 1.29 (5.9, 6144); 32 of 2880 x 2880, top-4, 8192
// in 8 2.39 / 2.44 (11.8, 11520).
bool copies_in_step(const csk_moe_layer* L, int64_t T, int passes) {
  const double mb = 1e-6 * sizeof(float) * T * L->H / passes;
  return passes >= 4 && mb >= 4 && mb <= 12 && (int64_t)L->k * L->F <= 4096;
}
}  // namespace

int csk_moe_forward(csk_moe_layer* L, const float* hidden, int64_t T, const float* router_in,
                    float* router_out, float* out) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!hidden || !out) return fail(L, CSK_ERR_INVALID, "null argument");
  if (T <= 0 || T > L->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld outside (0, max_tokens]", (long long)T);
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = L->stream;
  const int passes = host_passes(L, T, {hidden, router_in, router_out, out});
  const size_t row_bytes = sizeof(float) * T * L->H, route_bytes = sizeof(float) * T * L->k * 2;
  if (passes == 1) {
    // Through the handle's staging area a batch's status word comes back with its results, and nothing waits for a copy that the driver stages.
    const size_t bytes = row_bytes + route_bytes;
    const bool fits = bytes <= L->h_staged_bytes;
    // (a buffer that the host may copy: pageable, or page-locked where asked for; null: not given)
    auto to_copy = [](const void* p, bool locked) {
      const cudaMemoryType m = p ? memory_of(p) : cudaMemoryTypeUnregistered;
      return m == cudaMemoryTypeUnregistered || (locked && m == cudaMemoryTypeHost);
    };
    const bool staged_in = fits && row_bytes > kStagedInMin && to_copy(hidden, false) && to_copy(router_in, true);
    float* staged_route = L->h_staged + T * L->H;
    if (staged_in) {
      const int64_t half = row_bytes < kStagedTwoPieces ? 0 : T / 2 * L->H;
      for (const auto& [at, n] : {std::pair{(int64_t)0, half}, std::pair{half, T * L->H - half}}) {
        if (!n) continue;
        memcpy(L->h_staged + at, hidden + at, sizeof(float) * n);
        CSK_CUDA(L, cudaMemcpyAsync(L->d_hidden + at, L->h_staged + at, sizeof(float) * n, cudaMemcpyHostToDevice, s));
      }
      if (router_in) memcpy(staged_route, router_in, route_bytes);
    } else {
      CSK_CUDA(L, cudaMemcpyAsync(L->d_hidden, hidden, row_bytes, cudaMemcpyHostToDevice, s));
    }
    if (router_in) CSK_CUDA(L, cudaMemcpyAsync(L->d_router, staged_in ? staged_route : router_in, route_bytes, cudaMemcpyHostToDevice, s));
    // Results that the host copies are written to the staging area by the last kernel (where the inputs went out from, too: the stream has
    // taken those first), with the routing and the status word.
    const bool locked = bytes <= kStagedLockedMax;
    const bool staged_out = fits && to_copy(out, locked) && to_copy(router_out, true);
    HostResult host;
    if (staged_out) host = {router_out ? staged_route : nullptr, L->h_meta};
    int rc = forward_replayed(L, L->d_hidden, T, router_in ? L->d_router : nullptr, nullptr, staged_out ? L->h_staged : L->d_out, s, host);
    if (rc) {
      if (staged_in) cudaStreamSynchronize(s);  // the copies in have left the staging area
      return rc;
    }
    if (staged_out) {
      CSK_CUDA(L, cudaStreamSynchronize(s));
      rc = report_status(L, L->h_meta[3] | L->h_meta[8], s);
    } else {
      rc = check_device_status(L, s);
    }
    if (rc) return rc;
    if (L->timing && L->n_marks > 1) finish_timings(L, L->n_marks, L->last_routed);
    if (staged_out) {
      memcpy(out, L->h_staged, row_bytes);
      if (router_out) memcpy(router_out, staged_route, route_bytes);
      return CSK_OK;
    }
    CSK_CUDA(L, cudaMemcpyAsync(out, L->d_out, row_bytes, cudaMemcpyDeviceToHost, s));
    if (router_out) CSK_CUDA(L, cudaMemcpyAsync(router_out, L->d_router, route_bytes, cudaMemcpyDeviceToHost, s));
    CSK_CUDA(L, cudaStreamSynchronize(s));
    return CSK_OK;
  }
  // Several passes over token ranges, three streams: the rows of pass i+1 arrive and the results of
  // pass i-1 leave while the kernels of pass i run (tokens are independent, so the passes give the
  // same rows as one pass would).  One cudaMemcpyAsync per range and direction.  The status word of
  // every pass is folded into a sticky one that is read once, at the end.
  CSK_CUDA(L, cudaMemsetAsync(L->d_carry, 0, sizeof(int) * (1 + L->E), s));
  CSK_CUDA(L, cudaEventRecord(L->ev_free, s));  // earlier work on this handle is done before the copies overwrite d_hidden
  CSK_CUDA(L, cudaStreamWaitEvent(L->stream_in, L->ev_free, 0));
  struct CarryScope {
    csk_moe_layer* l;
    ~CarryScope() { l->carry_active = false; }
  } carry_scope{L};
  L->carry_active = true;
  const int k2 = L->k * 2;
  auto copy_in = [&](int p) -> int {
    const int64_t t0 = T * p / passes, n = T * (p + 1) / passes - t0;
    CSK_CUDA(L, cudaMemcpyAsync(L->d_hidden + t0 * L->H, hidden + t0 * L->H, sizeof(float) * n * L->H,
                                cudaMemcpyHostToDevice, L->stream_in));
    if (router_in)
      CSK_CUDA(L, cudaMemcpyAsync(L->d_router + t0 * k2, router_in + t0 * k2, sizeof(float) * n * k2,
                                  cudaMemcpyHostToDevice, L->stream_in));
    CSK_CUDA(L, cudaEventRecord(L->ev_in[p], L->stream_in));
    return CSK_OK;
  };
  const bool in_step = copies_in_step(L, T, passes);
  int rc = CSK_OK;
  for (int p = 0; in_step && p < passes && !rc; ++p) rc = copy_in(p);
  for (int p = 0; p < passes && !rc; ++p) {
    const int64_t t0 = T * p / passes, t1 = T * (p + 1) / passes, n = t1 - t0;
    if (!in_step) rc = copy_in(p);
    if (rc) break;
    CSK_CUDA(L, cudaStreamWaitEvent(s, L->ev_in[p], 0));
    // the router writes the pass's routing to its place in d_router (kept for router_out and for the counters)
    rc = forward_dev(L, L->d_hidden + t0 * L->H, n, router_in ? L->d_router + t0 * k2 : nullptr,
                     router_in ? nullptr : L->d_router + t0 * k2, L->d_out + t0 * L->H, -1, s, false);
    if (rc) break;
    CSK_CUDA(L, cudaEventRecord(L->ev_done[p], s));
    CSK_CUDA(L, cudaStreamWaitEvent(L->stream_out, L->ev_done[p], 0));
    if (in_step && p + 1 < passes) CSK_CUDA(L, cudaStreamWaitEvent(L->stream_out, L->ev_in[p + 1], 0));
    CSK_CUDA(L, cudaMemcpyAsync(out + t0 * L->H, L->d_out + t0 * L->H, sizeof(float) * n * L->H,
                                cudaMemcpyDeviceToHost, L->stream_out));
    if (router_out)
      CSK_CUDA(L, cudaMemcpyAsync(router_out + t0 * k2, L->d_router + t0 * k2, sizeof(float) * n * k2,
                                  cudaMemcpyDeviceToHost, L->stream_out));
  }
  L->counts_in_carry = true;
  L->last_T = T;
  // the sticky status word travels with the last results
  cudaMemcpyAsync(L->h_meta, L->d_meta, sizeof(int) * 16, cudaMemcpyDeviceToHost, L->stream_out);
  cudaMemcpyAsync(L->h_meta + 3, L->d_carry, sizeof(int), cudaMemcpyDeviceToHost, L->stream_out);
  cudaError_t e1 = cudaStreamSynchronize(L->stream_in), e2 = cudaStreamSynchronize(s), e3 = cudaStreamSynchronize(L->stream_out);
  if (rc) return rc;
  if (e1 != cudaSuccess || e2 != cudaSuccess || e3 != cudaSuccess)
    return fail(L, CSK_ERR_CUDA, "pipelined forward: %s", cudaGetErrorString(e1 != cudaSuccess ? e1 : e2 != cudaSuccess ? e2 : e3));
  return report_status(L, L->h_meta[3] | L->h_meta[8], s);
}

int csk_moe_dense_forward_dev(csk_moe_layer* L, const float* d_hidden, int64_t T, float* d_out, void* stream) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!L->d_unit_router) return fail(L, CSK_ERR_INVALID, "dense forward needs a layer with num_experts = top_k = 1");
  return csk_moe_forward_dev(L, d_hidden, T, L->d_unit_router, nullptr, d_out, stream);
}

int csk_moe_dense_forward(csk_moe_layer* L, const float* hidden, int64_t T, float* out) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!L->d_unit_router) return fail(L, CSK_ERR_INVALID, "dense forward needs a layer with num_experts = top_k = 1");
  if (!hidden || !out) return fail(L, CSK_ERR_INVALID, "null argument");
  if (T <= 0 || T > L->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld outside (0, max_tokens]", (long long)T);
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = L->stream;
  CSK_CUDA(L, cudaMemcpyAsync(L->d_hidden, hidden, sizeof(float) * T * L->H, cudaMemcpyHostToDevice, s));
  int rc = forward_dev(L, L->d_hidden, T, L->d_unit_router, nullptr, L->d_out, -1, s, true);
  if (rc) return rc;
  CSK_CUDA(L, cudaMemcpyAsync(out, L->d_out, sizeof(float) * T * L->H, cudaMemcpyDeviceToHost, s));
  CSK_CUDA(L, cudaStreamSynchronize(s));
  return CSK_OK;
}

int csk_moe_expert_forward(csk_moe_layer* L, int32_t expert_id, const float* hidden, int64_t T,
                           const float* router_out, float* out, int32_t* selected) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!hidden || !router_out || !out || !selected) return fail(L, CSK_ERR_INVALID, "null argument");
  if (T <= 0 || T > L->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld outside (0, max_tokens]", (long long)T);
  if (expert_id < L->e0 || expert_id >= L->e0 + L->Eloc || !L->resident[expert_id - L->e0])
    return fail(L, CSK_ERR_MISSING, "expert %d is not loaded", expert_id);
  // the reference's early return: no token selected this expert (expert_mlp_node.h:441-443)
  bool any = false;
  for (int64_t i = 0; i < T * L->k && !any; ++i) any = (int)router_out[2 * i] == expert_id;
  *selected = any ? 1 : 0;
  if (!any) return CSK_OK;
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = L->stream;
  CSK_CUDA(L, cudaMemcpyAsync(L->d_hidden, hidden, sizeof(float) * T * L->H, cudaMemcpyHostToDevice, s));
  CSK_CUDA(L, cudaMemcpyAsync(L->d_router, router_out, sizeof(float) * T * L->k * 2, cudaMemcpyHostToDevice, s));
  int rc = forward_dev(L, L->d_hidden, T, L->d_router, nullptr, L->d_out, expert_id, s, true);
  if (rc) return rc;
  CSK_CUDA(L, cudaMemcpyAsync(out, L->d_out, sizeof(float) * T * L->H, cudaMemcpyDeviceToHost, s));
  CSK_CUDA(L, cudaStreamSynchronize(s));
  return CSK_OK;
}

int csk_moe_merge(csk_moe_layer* L, const float* router_out, int64_t T, const float* const* expert_outs,
                  float* out) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!router_out || !expert_outs || !out) return fail(L, CSK_ERR_INVALID, "null argument");
  if (T <= 0 || T > L->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld outside (0, max_tokens]", (long long)T);
  bool any = false;
  for (int e = 0; e < L->E; ++e) any = any || expert_outs[e];
  if (!any) return fail(L, CSK_ERR_INVALID, "expert_merge: no non-empty expert outputs found");
  // Only the k rows each token actually uses travel to the device: row (t,j)
  // of expert e(t,j), or nothing when that expert's output is the empty tensor.
  std::vector<int> rows((size_t)T * L->k, -1);
  std::vector<float> packed;
  packed.reserve((size_t)T * L->k * L->H);
  int n = 0;
  for (int64_t t = 0; t < T; ++t)
    for (int j = 0; j < L->k; ++j) {
      const int e = (int)router_out[(t * L->k + j) * 2];
      if (e < 0 || e >= L->E)
        return fail(L, CSK_ERR_INVALID, "expert_merge: expert_idx out of range: %d", e);
      if (!expert_outs[e]) continue;
      rows[t * L->k + j] = n++;
      const float* src = expert_outs[e] + t * L->H;
      packed.insert(packed.end(), src, src + L->H);
    }
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = L->stream;
  CSK_CUDA(L, cudaMemcpyAsync(L->d_y, packed.data(), sizeof(float) * packed.size(), cudaMemcpyHostToDevice, s));
  CSK_CUDA(L, cudaMemcpyAsync(L->d_row_of_pair, rows.data(), sizeof(int) * rows.size(), cudaMemcpyHostToDevice, s));
  CSK_CUDA(L, cudaMemcpyAsync(L->d_router, router_out, sizeof(float) * T * L->k * 2, cudaMemcpyHostToDevice, s));
  launch_combine(L, L->d_router, L->d_y, T, L->d_out, s, false);
  CSK_CUDA(L, cudaGetLastError());
  CSK_CUDA(L, cudaMemcpyAsync(out, L->d_out, sizeof(float) * T * L->H, cudaMemcpyDeviceToHost, s));
  CSK_CUDA(L, cudaStreamSynchronize(s));
  return CSK_OK;
}

// ---- expert parallelism -------------------------------------------------------
int csk_moe_ep_row_pitch(const csk_moe_layer* L) { return L ? L->ldx : CSK_ERR_INVALID; }

int csk_moe_ep_dispatch_dev(csk_moe_layer* L, const float* d_hidden, int64_t T, const float* d_router_in,
                            void* d_send_f16, int32_t* d_counts, void* stream) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!d_hidden || !d_send_f16 || !d_counts) return fail(L, CSK_ERR_INVALID, "null argument");
  if (T <= 0 || T > L->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld outside (0, max_tokens]", (long long)T);
  if (reinterpret_cast<uintptr_t>(d_hidden) % 16) return fail(L, CSK_ERR_INVALID, "hidden states must be 16-byte aligned");
  if (reinterpret_cast<uintptr_t>(d_send_f16) % 8) return fail(L, CSK_ERR_INVALID, "the rows to send must be 8-byte aligned");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = pick(L, stream);
  const PdlScope pdl_scope(L);  // (the kernels are those of a layer's plan)
  L->last = csk_moe_timings{};
  L->last_T = T;
  if (!d_router_in) {
    int rc = launch_router(L, d_hidden, T, L->d_router, s);
    if (rc) return rc;
  } else if (d_router_in != L->d_router) {
    CSK_CUDA(L, cudaMemcpyAsync(L->d_router, d_router_in, sizeof(float) * T * L->k * 2,
                                cudaMemcpyDeviceToDevice, s));
  }
  const float* router = L->d_router;
  if (L->has_slot_map) {
    k_ep_slots<<<grid_for((size_t)T * L->k, 256, 4 * L->sm_count), 256, 0, s>>>(
        L->d_router, L->d_router_phys, (int)(T * L->k), L->k, L->E_router, L->d_slot_map, L->d_slot_map + L->E);
    CSK_CUDA(L, cudaGetLastError());
    router = L->d_router_phys;
  }
  // group by global expert id; no tiles are built here (e_count = 0)
  int rc = launch_permute(L, d_hidden, router, T, -1, 8, 0, 0, (__half*)d_send_f16, L->ldx,
                          T * L->k, s);
  if (rc) return rc;
  CSK_CUDA(L, cudaMemcpyAsync(d_counts, L->d_counts, sizeof(int) * L->E, cudaMemcpyDeviceToDevice, s));
  return CSK_OK;
}

int csk_moe_ep_set_slot_map(csk_moe_layer* L, int32_t n_logical, const int32_t* primary_slot,
                            const int32_t* replica_slot) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  drop_graphs(L);
  if (n_logical == 0) {
    if (L->has_slot_map) L->router_set = false;
    L->has_slot_map = false;
    L->E_router = L->E;
    return CSK_OK;
  }
  if (n_logical < L->k || n_logical > L->E || !primary_slot)
    return fail(L, CSK_ERR_INVALID, "slot map: need top_k <= n_logical <= num_experts (%d) and a primary_slot array, got %d",
                L->E, n_logical);
  std::vector<int> map(2 * (size_t)L->E, -1);
  std::vector<char> used(L->E, 0);
  for (int e = 0; e < n_logical; ++e) {
    for (int c = 0; c < 2; ++c) {
      const int s = c == 0 ? primary_slot[e] : (replica_slot ? replica_slot[e] : -1);
      if (c == 1 && s == -1) continue;
      if (s < 0 || s >= L->E) return fail(L, CSK_ERR_INVALID, "slot map: slot %d of expert %d is outside [0,%d)", s, e, L->E);
      if (used[s]) return fail(L, CSK_ERR_INVALID, "slot map: slot %d is used twice", s);
      used[s] = 1;
      map[(size_t)c * L->E + e] = s;
    }
  }
  CSK_CUDA(L, cudaMemcpyAsync(L->d_slot_map, map.data(), sizeof(int) * map.size(), cudaMemcpyHostToDevice, L->stream));
  CSK_CUDA(L, cudaStreamSynchronize(L->stream));
  L->has_slot_map = true;
  L->E_router = n_logical;
  L->router_set = false;  // the router's weights are per logical expert from here on
  return CSK_OK;
}

// ---- expert parallelism over peer memory ----------------------------------------
namespace {
// End of an experts stage: enqueue only, unless timing is on (then wait, check the status word, read the events).
int ep_finish(csk_moe_layer* L, cudaStream_t s, int n_marks) {
  L->last_stream = s;
  if (!L->timing) return CSK_OK;  // csk_moe_sync reports what the kernels found
  int rc = check_device_status(L, s);
  if (rc) return rc;
  if (n_marks == 3) {  // the status check above already waited for the stream
    cudaEventElapsedTime(&L->last.gate_up_ms, L->ev[0], L->ev[1]);
    cudaEventElapsedTime(&L->last.down_ms, L->ev[1], L->ev[2]);
    L->last.total_ms = L->last.gate_up_ms + L->last.down_ms;
  }
  return CSK_OK;
}
int p2p_alloc_local(csk_moe_layer* L) {
  if (L->d_info) return CSK_OK;
  int rc = mx_reserve(L, L->max_rows);  // how many rows the peers will send is not known on the host
  if (rc) return rc;
  CSK_CUDA(L, cudaMalloc(&L->d_info, sizeof(RowOrigin) * (size_t)L->max_rows));
  // 0xFF bytes: (-1, -1), which no reader accepts as an origin (rows a sender had to skip stay that way)
  CSK_CUDA(L, cudaMemset(L->d_info, 0xFF, sizeof(RowOrigin) * (size_t)L->max_rows));
  // the return buffer carries the sync area of the flag barriers at its tail (peers can write both)
  L->back_tail = (size_t)L->max_T * L->k * L->H;
  const size_t back_bytes = sizeof(float) * L->back_tail + sizeof(int) * ep_sync_ints(L->E);
  CSK_CUDA(L, cudaMalloc(&L->d_back, back_bytes));
  CSK_CUDA(L, cudaMemset(reinterpret_cast<uint8_t*>(L->d_back) + sizeof(float) * L->back_tail, 0, sizeof(int) * ep_sync_ints(L->E)));
  CSK_CUDA(L, cudaMalloc(&L->d_row_ptr, sizeof(float*) * (size_t)L->max_rows));
  return CSK_OK;
}
int p2p_set_peers(csk_moe_layer* L, int rank, int world, void* const* x16, void* const* info, void* const* back) {
  if (world < 1 || world > 64 || rank < 0 || rank >= world) return fail(L, CSK_ERR_INVALID, "p2p: bad rank/world %d/%d", rank, world);
  if (L->E % world || L->Eloc != L->E / world || L->e0 != rank * L->Eloc)
    return fail(L, CSK_ERR_INVALID, "p2p: rank %d of %d must own expert slots [%d, %d)", rank, world,
                rank * (L->E / std::max(1, world)), (rank + 1) * (L->E / std::max(1, world)));
  for (void** p : {(void**)&L->d_peer_x16, (void**)&L->d_peer_info, (void**)&L->d_peer_back}) {
    if (*p) cudaFree(*p);
    *p = nullptr;
  }
  CSK_CUDA(L, cudaMalloc(&L->d_peer_x16, sizeof(void*) * world));
  CSK_CUDA(L, cudaMalloc(&L->d_peer_info, sizeof(void*) * world));
  CSK_CUDA(L, cudaMalloc(&L->d_peer_back, sizeof(void*) * world));
  CSK_CUDA(L, cudaMemcpy(L->d_peer_x16, x16, sizeof(void*) * world, cudaMemcpyHostToDevice));
  CSK_CUDA(L, cudaMemcpy(L->d_peer_info, info, sizeof(void*) * world, cudaMemcpyHostToDevice));
  CSK_CUDA(L, cudaMemcpy(L->d_peer_back, back, sizeof(void*) * world, cudaMemcpyHostToDevice));
  L->p2p_rank = rank;
  L->p2p_world = world;
  return CSK_OK;
}
}  // namespace

int csk_moe_ep_p2p_local_ptrs(csk_moe_layer* L, void** x16, void** info, void** back) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  int rc = p2p_alloc_local(L);
  if (rc) return rc;
  if (x16) *x16 = L->d_x16;
  if (info) *info = L->d_info;
  if (back) *back = L->d_back;
  return CSK_OK;
}

int csk_moe_ep_p2p_export(csk_moe_layer* L, uint8_t* handles) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!handles) return fail(L, CSK_ERR_INVALID, "null argument");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  int rc = p2p_alloc_local(L);
  if (rc) return rc;
  static_assert(sizeof(cudaIpcMemHandle_t) + sizeof(uint64_t) == CSK_IPC_HANDLE_BYTES, "handle size");
  // the driver entry point is looked up at run time: the library has no link-time dependency on libcuda
  typedef CUresult (*GetRangeFn)(CUdeviceptr*, size_t*, CUdeviceptr);
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuMemGetAddressRange", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn) {
    cudaGetLastError();
    return fail(L, CSK_ERR_CUDA, "p2p: cuMemGetAddressRange not found in the driver");
  }
  const GetRangeFn get_range = (GetRangeFn)fn;
  void* bufs[3] = {L->d_x16, L->d_info, L->d_back};
  for (int i = 0; i < 3; ++i) {
    // a handle names the whole allocation a pointer lies in (small buffers share one): ship the offset too
    cudaIpcMemHandle_t h;
    CSK_CUDA(L, cudaIpcGetMemHandle(&h, bufs[i]));
    CUdeviceptr base = 0;
    size_t size = 0;
    if (get_range(&base, &size, (CUdeviceptr)bufs[i]) != CUDA_SUCCESS)
      return fail(L, CSK_ERR_CUDA, "p2p: cuMemGetAddressRange failed");
    const uint64_t off = (uint64_t)((CUdeviceptr)bufs[i] - base);
    memcpy(handles + (size_t)i * CSK_IPC_HANDLE_BYTES, &h, sizeof(h));
    memcpy(handles + (size_t)i * CSK_IPC_HANDLE_BYTES + sizeof(h), &off, sizeof(off));
  }
  return CSK_OK;
}

int csk_moe_ep_p2p_import(csk_moe_layer* L, int32_t rank, int32_t world, const uint8_t* all_handles) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!all_handles) return fail(L, CSK_ERR_INVALID, "null argument");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  int rc = p2p_alloc_local(L);
  if (rc) return rc;
  if (world < 1 || world > 64 || rank < 0 || rank >= world) return fail(L, CSK_ERR_INVALID, "p2p: bad rank/world %d/%d", rank, world);
  std::vector<void*> ptr(3 * (size_t)world, nullptr);
  std::vector<cudaIpcMemHandle_t> opened_handles;
  std::vector<void*> opened_ptrs;
  void* own[3] = {L->d_x16, L->d_info, L->d_back};
  for (int r = 0; r < world; ++r)
    for (int i = 0; i < 3; ++i) {
      if (r == rank) {
        ptr[(size_t)i * world + r] = own[i];
        continue;
      }
      cudaIpcMemHandle_t h;
      uint64_t off = 0;
      const uint8_t* rec = all_handles + ((size_t)r * 3 + i) * CSK_IPC_HANDLE_BYTES;
      memcpy(&h, rec, sizeof(h));
      memcpy(&off, rec + sizeof(h), sizeof(off));
      // two of a peer's buffers may lie in one allocation: open each allocation once
      void* p = nullptr;
      for (size_t j = 0; j < opened_handles.size(); ++j)
        if (!memcmp(&opened_handles[j], &h, sizeof(h))) p = opened_ptrs[j];
      if (!p) {
        CSK_CUDA(L, cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess));
        L->ipc_opened.push_back(p);
        opened_handles.push_back(h);
        opened_ptrs.push_back(p);
      }
      ptr[(size_t)i * world + r] = static_cast<uint8_t*>(p) + off;
    }
  return p2p_set_peers(L, rank, world, ptr.data(), ptr.data() + world, ptr.data() + 2 * (size_t)world);
}

int csk_moe_ep_p2p_import_ptrs(csk_moe_layer* L, int32_t rank, int32_t world, void* const* x16, void* const* info,
                               void* const* back) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!x16 || !info || !back) return fail(L, CSK_ERR_INVALID, "null argument");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  int rc = p2p_alloc_local(L);
  if (rc) return rc;
  return p2p_set_peers(L, rank, world, x16, info, back);
}

// Stage 1: route, map to slots, count this rank's rows per slot.
int csk_moe_ep_p2p_counts_dev(csk_moe_layer* L, const float* d_hidden, int64_t T, const float* d_router_in,
                              int32_t* d_counts, void* stream) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!d_hidden || !d_counts) return fail(L, CSK_ERR_INVALID, "null argument");
  if (L->p2p_world <= 0) return fail(L, CSK_ERR_INVALID, "p2p: peers were never imported");
  if (T <= 0 || T > L->max_T) return fail(L, CSK_ERR_NOMEM, "T=%lld outside (0, max_tokens]", (long long)T);
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = pick(L, stream);
  L->last = csk_moe_timings{};
  L->last_T = T;
  if (!d_router_in) {
    int rc = launch_router(L, d_hidden, T, L->d_router, s);
    if (rc) return rc;
  } else if (d_router_in != L->d_router) {
    CSK_CUDA(L, cudaMemcpyAsync(L->d_router, d_router_in, sizeof(float) * T * L->k * 2, cudaMemcpyDeviceToDevice, s));
  }
  const int n_pairs = (int)(T * L->k);
  const float* router = L->d_router;
  if (L->has_slot_map) {
    k_ep_slots<<<grid_for((size_t)n_pairs, 256, 4 * L->sm_count), 256, 0, s>>>(
        L->d_router, L->d_router_phys, n_pairs, L->k, L->E_router, L->d_slot_map, L->d_slot_map + L->E);
    router = L->d_router_phys;
  }
  CSK_CUDA(L, cudaMemsetAsync(L->d_counts, 0, sizeof(int) * L->E, s));
  CSK_CUDA(L, cudaMemsetAsync(L->d_meta, 0, sizeof(int) * 8, s));
  k_hist<<<grid_for(n_pairs, 256, 2 * L->sm_count), 256, sizeof(int) * (L->E + 1), s>>>(router, n_pairs, L->E, -1, L->d_counts,
                                                                                 L->d_meta);
  CSK_CUDA(L, cudaGetLastError());
  CSK_CUDA(L, cudaMemcpyAsync(d_counts, L->d_counts, sizeof(int) * L->E, cudaMemcpyDeviceToDevice, s));
  return CSK_OK;
}

// Barrier `which` (0: counts, 1: rows landed, 2: outputs landed) between the ranks, by flags in peer
// memory; with d_counts / d_all_counts it also exchanges the per-slot row counts (the all-gather).
int csk_moe_ep_p2p_sync_dev(csk_moe_layer* L, int32_t which, const int32_t* d_counts, int32_t* d_all_counts, void* stream) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (L->p2p_world <= 0) return fail(L, CSK_ERR_INVALID, "p2p: peers were never imported");
  if (which < 0 || which > 2 || (d_counts == nullptr) != (d_all_counts == nullptr))
    return fail(L, CSK_ERR_INVALID, "p2p sync: which must be 0..2, counts and all_counts go together");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = pick(L, stream);
  k_ep_p2p_sync<<<1, 1024, 0, s>>>(L->d_peer_back, L->back_tail, L->p2p_rank, L->p2p_world, which, L->d_p2p_epoch,
                                   d_counts, L->E, d_all_counts, L->d_meta);
  CSK_CUDA(L, cudaGetLastError());
  L->last_stream = s;
  return CSK_OK;
}

// Stage 2 (after the all-gather of the counts): rows to the ranks that own their slots.
int csk_moe_ep_p2p_scatter_dev(csk_moe_layer* L, const float* d_hidden, int64_t T, const int32_t* d_all_counts,
                               void* stream) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!d_hidden || !d_all_counts) return fail(L, CSK_ERR_INVALID, "null argument");
  if (L->p2p_world <= 0) return fail(L, CSK_ERR_INVALID, "p2p: peers were never imported");
  if (T != L->last_T) return fail(L, CSK_ERR_INVALID, "p2p: scatter must follow counts of the same batch");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = pick(L, stream);
  const int n_pairs = (int)(T * L->k);
  const float* router = L->has_slot_map ? L->d_router_phys : L->d_router;
  k_ep_p2p_base<<<1, 1024, 0, s>>>(d_all_counts, L->p2p_world, L->p2p_rank, L->E, L->Eloc, (int)L->max_rows,
                                   L->d_p2p_base, L->d_cursor, L->d_meta);
  k_ep_p2p_scatter<<<grid_for(n_pairs, 8, 8 * L->sm_count), 256, 0, s>>>(
      router, d_hidden, n_pairs, L->k, L->H, L->E, L->Eloc, L->p2p_rank, L->d_p2p_base, L->d_cursor, L->d_peer_x16,
      L->d_peer_info, L->ldx, (int)L->max_rows, L->cfg.weight_before_ffn, L->d_row_of_pair, L->d_meta);
  CSK_CUDA(L, cudaGetLastError());
  return CSK_OK;
}

// Stage 3 (after a barrier: every rank's rows have landed): the resident experts over the
// received rows; output rows go straight to their owners' return buffers.
int csk_moe_ep_p2p_experts_dev(csk_moe_layer* L, const int32_t* d_all_counts, int64_t rows_hint, void* stream) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!d_all_counts) return fail(L, CSK_ERR_INVALID, "null argument");
  if (L->p2p_world <= 0) return fail(L, CSK_ERR_INVALID, "p2p: peers were never imported");
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = pick(L, stream);
  rows_hint = std::max<int64_t>(1, std::min<int64_t>(rows_hint, L->max_rows));
  const int path = choose_path_received(L, rows_hint, L->max_rows);  // (a hint is no bound)
  const int tile_rows = tile_rows_for(path);
  const bool mx = path == CSK_PATH_STREAM;
  // the status word of the dispatch stays; the tile list is rebuilt from the received counts
  k_ep_p2p_local_counts<<<(L->E + 255) / 256, 256, 0, s>>>(d_all_counts, L->p2p_world, L->E, L->e0, L->Eloc, L->d_counts);
  k_scan<<<1, scan_threads(L->E, 0), 0, s>>>(scan_args(L, tile_rows, L->e0, L->Eloc, L->d_resident, mx ? L->mx_rows : L->max_rows, mx));
  k_ep_p2p_rowptr<<<4 * L->sm_count, 256, 0, s>>>(L->d_info, L->d_meta, L->d_peer_back, L->H, L->d_row_ptr,
                                                  (int)L->max_rows, L->p2p_world, (int)L->max_rows);
  CSK_CUDA(L, cudaGetLastError());
  StageTimer tm(L, s);
  tm.mark();
  int rc;
  if (path == CSK_PATH_TILE) {
    rc = launch_experts(L, path, nullptr, L->H, nullptr, s, tm, L->d_row_ptr);
  } else {
    mx_quant_rows(L, s);
    rc = launch_experts(L, path, L->d_y, L->H, nullptr, s, tm);
    if (!rc) {
      k_ep_p2p_return<<<8 * L->sm_count, 256, 0, s>>>(L->d_y, L->H, L->d_row_ptr, L->d_meta, (int)L->max_rows);
      CSK_CUDA(L, cudaGetLastError());
    }
  }
  if (rc) return rc;
  return ep_finish(L, s, tm.n);
}

// Stage 4 (after a second barrier: every output row of this rank's pairs has landed).
int csk_moe_ep_p2p_combine_dev(csk_moe_layer* L, int64_t T, float* d_out, float* d_router_out, void* stream) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (L->p2p_world <= 0) return fail(L, CSK_ERR_INVALID, "p2p: peers were never imported");
  return csk_moe_ep_combine_dev(L, L->d_back, T, d_out, d_router_out, stream);
}

int csk_moe_ep_experts_dev(csk_moe_layer* L, const void* d_recv_f16, const int32_t* d_recv_counts,
                           int32_t n_src, int64_t total_rows, float* d_ret, void* stream) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!d_recv_f16 || !d_recv_counts || !d_ret) return fail(L, CSK_ERR_INVALID, "null argument");
  if (n_src <= 0 || (int64_t)n_src * L->Eloc > 1024)
    return fail(L, CSK_ERR_INVALID, "n_src * local experts must be in [1,1024]");
  if (total_rows < 0 || total_rows > L->max_rows)
    return fail(L, CSK_ERR_NOMEM, "%lld received rows exceed max_tokens*top_k = %lld",
                (long long)total_rows, (long long)L->max_rows);
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = pick(L, stream);
  if (total_rows == 0) return CSK_OK;
  const int path = choose_path_received(L, total_rows, total_rows);
  const int tile_rows = tile_rows_for(path);
  const bool mx = path == CSK_PATH_STREAM;
  CSK_CUDA(L, cudaMemsetAsync(L->d_meta, 0, sizeof(int) * 8, s));
  CSK_CUDA(L, cudaMemsetAsync(L->d_counts, 0, sizeof(int) * L->E, s));
  k_ep_plan<<<1, 1024, 0, s>>>(d_recv_counts, n_src, L->Eloc, L->e0, L->d_counts, L->d_seg);
  k_scan<<<1, scan_threads(L->E, 0), 0, s>>>(scan_args(L, tile_rows, L->e0, L->Eloc, L->d_resident, mx ? L->mx_rows : L->max_rows, mx));
  k_ep_regroup<<<dim3((unsigned)(n_src * L->Eloc), (unsigned)std::max(1, 16 * L->sm_count / (n_src * L->Eloc))), 128, 0, s>>>((const __half*)d_recv_f16, L->d_x16, L->ldx, L->d_seg,
                                               L->d_offsets, n_src, L->Eloc, L->e0, L->d_out_row_map);
  CSK_CUDA(L, cudaGetLastError());
  StageTimer tm(L, s);
  tm.mark();
  int rc;
  if (path == CSK_PATH_TILE) {
    rc = launch_experts(L, path, d_ret, L->H, L->d_out_row_map, s, tm);
  } else {
    mx_quant_rows(L, s);
    rc = launch_experts(L, path, L->d_y, L->H, nullptr, s, tm);
    if (!rc) {
      k_ep_ungroup<<<grid_for((size_t)total_rows, 8, 8 * L->sm_count), 256, 0, s>>>(
          L->d_y, d_ret, L->H, L->d_out_row_map, (int)total_rows);
      CSK_CUDA(L, cudaGetLastError());
    }
  }
  if (rc) return rc;
  return ep_finish(L, s, tm.n);
}

int csk_moe_ep_combine_dev(csk_moe_layer* L, const float* d_back, int64_t T, float* d_out,
                           float* d_router_out, void* stream) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!d_back || !d_out) return fail(L, CSK_ERR_INVALID, "null argument");
  if (T != L->last_T) return fail(L, CSK_ERR_INVALID, "combine T=%lld does not match dispatch T=%lld",
                                  (long long)T, (long long)L->last_T);
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  cudaStream_t s = pick(L, stream);
  launch_combine(L, L->d_router, d_back, T, d_out, s, false);
  CSK_CUDA(L, cudaGetLastError());
  if (d_router_out)
    CSK_CUDA(L, cudaMemcpyAsync(d_router_out, L->d_router, sizeof(float) * T * L->k * 2,
                                cudaMemcpyDeviceToDevice, s));
  return CSK_OK;
}

// ---- routing without any allocation ---------------------------------------------
// Scratch for csk_moe_route_static: the [T,E] logits between its two kernels.
// File-scope device memory, so every GPU that loads this library carries these
// 1 MiB until the process exits.  In host code `g_static_logits` is only a
// stand-in for the symbol; the device address comes from cudaGetSymbolAddress.
constexpr int64_t kStaticLogitsMax = 256 * 1024;  // floats: T * E may not exceed this
static __device__ __align__(256) float g_static_logits[kStaticLogitsMax];
// Status word of the same entry point (kDevErr* bits or-ed by its kernels), read and cleared by
// csk_moe_route_static_status.
static __device__ int g_static_status;

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_static_mu;
float* g_static_logits_addr[kMaxDevices] = {nullptr};
int* g_static_status_addr[kMaxDevices] = {nullptr};
}  // namespace

int csk_moe_route_static(const float* d_hidden, int64_t T, int32_t H, const float* d_gate_w,
                         const float* d_gate_bias, int32_t E, int32_t k, int32_t sigmoid_gating,
                         float* d_router_out, void* stream) {
  if (!d_hidden || !d_gate_w || !d_router_out) return fail(nullptr, CSK_ERR_INVALID, "route_static: null argument");
  if (T <= 0 || H <= 0 || H % 32 || E <= 0 || E > 1024 || k <= 0 || k > kMaxTopK || k > E)
    return fail(nullptr, CSK_ERR_INVALID,
                "route_static: need T > 0, H a positive multiple of 32, 1 <= E <= 1024, 1 <= k <= min(E, %d); "
                "got T=%lld H=%d E=%d k=%d", kMaxTopK, (long long)T, H, E, k);
  if (T * (int64_t)E > kStaticLogitsMax)
    return fail(nullptr, CSK_ERR_NOMEM,
                "route_static: T*E = %lld exceeds the built-in scratch of %lld logits; split the batch or use "
                "csk_moe_route_dev on a handle", (long long)(T * (int64_t)E), (long long)kStaticLogitsMax);
  int dev = -1;
  cudaError_t ce = cudaGetDevice(&dev);
  if (ce != cudaSuccess) return fail(nullptr, CSK_ERR_CUDA, "route_static: cudaGetDevice: %s", cudaGetErrorString(ce));
  if (dev < 0 || dev >= kMaxDevices) return fail(nullptr, CSK_ERR_INVALID, "route_static: device ordinal %d not supported", dev);
  float* logits = nullptr;
  {
    // once per device, with that device current: resolve the symbol to its address there
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (!g_static_logits_addr[dev]) {
      void* p = nullptr;
      ce = cudaGetSymbolAddress(&p, g_static_logits);
      if (ce != cudaSuccess || !p)
        return fail(nullptr, CSK_ERR_CUDA, "route_static: cudaGetSymbolAddress: %s", cudaGetErrorString(ce));
      void* ps = nullptr;
      ce = cudaGetSymbolAddress(&ps, g_static_status);
      if (ce != cudaSuccess || !ps)
        return fail(nullptr, CSK_ERR_CUDA, "route_static: cudaGetSymbolAddress: %s", cudaGetErrorString(ce));
      ce = router_prepare_device();
      if (ce != cudaSuccess)
        return fail(nullptr, CSK_ERR_CUDA, "route_static: cudaFuncSetAttribute: %s", cudaGetErrorString(ce));
      g_static_status_addr[dev] = static_cast<int*>(ps);
      g_static_logits_addr[dev] = static_cast<float*>(p);
    }
    logits = g_static_logits_addr[dev];
  }
  cudaStream_t s = (cudaStream_t)stream;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (reinterpret_cast<uintptr_t>(d_hidden) % 16 || reinterpret_cast<uintptr_t>(d_gate_w) % 16)
    return fail(nullptr, CSK_ERR_INVALID, "route_static: hidden states and gate weights must be 16-byte aligned");
  RouterArgs a{};
  a.hidden = d_hidden;
  a.bias = d_gate_bias;
  a.logits = logits;
  a.status = g_static_status_addr[dev];
  a.T = (int)T;
  a.H = H;
  a.E = E;
  launch_router_logits<false>(a, d_gate_w, d_gate_w, RouterWave{sms, false, sms}, s);
  k_router_topk<<<(unsigned)((T + 3) / 4), 128, 0, s>>>(logits, d_router_out, (int)T, E, k, sigmoid_gating);
  ce = cudaGetLastError();
  if (ce != cudaSuccess) return fail(nullptr, CSK_ERR_CUDA, "route_static: launch failed: %s", cudaGetErrorString(ce));
  return CSK_OK;
}

int csk_moe_route_static_status(void) {
  int dev = -1;
  cudaError_t ce = cudaGetDevice(&dev);
  if (ce != cudaSuccess) return fail(nullptr, CSK_ERR_CUDA, "route_static_status: cudaGetDevice: %s", cudaGetErrorString(ce));
  int* addr = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (dev >= 0 && dev < kMaxDevices) addr = g_static_status_addr[dev];
  }
  if (!addr) return CSK_OK;  // csk_moe_route_static never ran on this device
  int st = 0;
  ce = cudaMemcpy(&st, addr, sizeof(int), cudaMemcpyDeviceToHost);
  if (ce != cudaSuccess) return fail(nullptr, CSK_ERR_CUDA, "route_static_status: %s", cudaGetErrorString(ce));
  if (!st) return CSK_OK;
  ce = cudaMemset(addr, 0, sizeof(int));
  if (ce != cudaSuccess) return fail(nullptr, CSK_ERR_CUDA, "route_static_status: %s", cudaGetErrorString(ce));
  return fail(nullptr, CSK_ERR_DEVICE, "route_static: a bounded device-side wait ran out; the routing output of that call is not valid");
}

// ---- test hooks ---------------------------------------------------------------------
int csk_moe_debug_set(csk_moe_layer* L, int32_t key, int64_t value) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  CSK_CUDA(L, cudaSetDevice(L->cfg.device));
  if (key == CSK_DEBUG_WAIT_BUDGET) {
    if (value < 1000) return fail(L, CSK_ERR_INVALID, "debug: the wait budget must be at least 1000 cycles");
    const long long v = value;
    CSK_CUDA(L, cudaStreamSynchronize(L->stream));
    CSK_CUDA(L, cudaMemcpyToSymbol(g_wait_budget, &v, sizeof(v)));
    return CSK_OK;
  }
  if (key == CSK_DEBUG_STALL_TILE_PRODUCER) {
    L->debug_stall = value != 0;
    return CSK_OK;
  }
  if (key == CSK_DEBUG_STALL_ROUTER) {
    L->debug_stall_router = value != 0;
    return CSK_OK;
  }
  if (key == CSK_DEBUG_NO_CLUSTERS) {
    if (!value) return fail(L, CSK_ERR_INVALID, "debug: clusters do not come back");
    L->pair.available = false;
    L->pair.err = "turned off by a test";
    for (RouterWave& w : L->router_waves) w = RouterWave{L->sm_count, false, L->sm_count};
    drop_graphs(L);
    return mx_reserve(L, mx_rows_own(L));
  }
  return fail(L, CSK_ERR_INVALID, "debug: unknown key %d", key);
}

int csk_moe_debug_get(csk_moe_layer* L, int32_t key, int64_t* value) {
  if (check_layer(L)) return CSK_ERR_INVALID;
  if (!value) return fail(L, CSK_ERR_INVALID, "null argument");
  const RouterWave w = L->router_waves[(L->E_router + 31) / 32];
  if (key == CSK_DEBUG_ROUTER_WAVE) {
    *value = w.blocks;
    return CSK_OK;
  }
  if (key == CSK_DEBUG_ROUTER_CLUSTERS) {
    *value = w.clusters ? 1 : 0;
    return CSK_OK;
  }
  return fail(L, CSK_ERR_INVALID, "debug: unknown key %d", key);
}

}  // extern "C"
