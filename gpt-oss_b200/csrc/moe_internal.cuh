// Internal structures shared by the host API and the kernels of the MoE block.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/moe_b200.h"

namespace moe {

// ---- tiling constants of the expert GEMM (expert_gemm_sm100.cu) -------------
constexpr int kBlockRows = 240;    // weight rows per work item; divides 5760 and 2880
constexpr int kHalfRows = kBlockRows / 2;  // weight rows per CTA of a pair: a weight tile
constexpr int kChunkK = 128;       // reduction elements per slice (4 MMA k-steps of 32)
constexpr int kMaxTileTok = 96;    // tokens per token tile, at most
constexpr int kTileRows = 2 * kMaxTileTok;  // each token contributes a high and a low e4m3 row
constexpr int kPairBytes = kTileRows * 2 * kChunkK;  // two k slices of a token tile: 49152 bytes
constexpr int kSfAtomBytes = 512;  // scale factors of 128 rows x 4 k-blocks, tensor-memory order
constexpr int kSfbTileBytes = 2 * kSfAtomBytes;   // token scales of one tile (192 rows in two atoms)
constexpr int kWTileCodes = kHalfRows * kChunkK / 2;  // 7680 bytes of packed codes per weight tile
constexpr int kWTileBytes = kWTileCodes + kSfAtomBytes;  // 8192: codes and scales
static_assert(kMaxTileTok % 8 == 0, "token tiles are cut in steps of 8 tokens");

// Tokens per tile of an expert with cnt rows: as few tiles as hold them, of equal size in steps of 8 tokens (the
// instruction's N moves in steps of 16 rows), so that no tile is a small rest.  No tile is empty: one less would
// hold at most kMaxTileTok * (tiles - 1) < cnt rows.
__host__ __device__ inline int expert_tiles(int cnt) { return (cnt + kMaxTileTok - 1) / kMaxTileTok; }
__host__ __device__ inline int tokens_per_tile(int cnt) {
  const int n = expert_tiles(cnt);
  return n == 0 ? kMaxTileTok : ((cnt + n - 1) / n + 7) / 8 * 8;
}
// Most tiles that `pairs` (token, expert) pairs over E experts can need: ceil(cnt / max) is at most 1 + (cnt - 1) / max for
// each expert with rows, and there are at most min(E, pairs) of those.  (All experts get 97 rows: exactly this many.)
inline int max_token_tiles(int pairs, int E) {
  const int experts = std::min(pairs, E);
  return experts + (pairs - experts) / kMaxTileTok;
}
__host__ __device__ inline int slice_pairs(int n_slices) { return (n_slices + 1) / 2; }

// Token rows of a tile: [pair of k slices][CTA][8-row group][slice of the pair][8 rows][128 bytes].  Four tokens make
// a group of 8 rows (high and low term each); even groups belong to the even CTA of the pair that works on the tile,
// odd ones to the odd CTA, so that what one CTA needs of both slices is one contiguous run whatever the number of
// tokens.  The eight 16-byte pieces of a row are permuted by the row (the 128-byte swizzle the tensor core reads).
// Byte of (token, low term?, element) inside a tile's pair of slices; k is the element's position in the pair.
__host__ __device__ inline int x_pair_offset(int tok, int low, int k) {
  const int row = (tok & 3) * 2 + low;
  return ((tok >> 2) & 1) * (kPairBytes / 2) + (tok >> 3) * 2048 + (k >> 7) * 1024 + row * kChunkK +
         ((((k >> 4) ^ row) & 7) << 4) + (k & 15);
}
// Row of the instruction's N operand that holds the token's high term (the low term follows) in a tile with N = n:
// the even CTA's groups come first.  The accumulator column and the scale row have the same number.
__host__ __device__ inline int x_operand_row(int tok, int n) { return ((tok >> 2) & 1) * (n / 2) + (tok >> 3) * 8 + (tok & 3) * 2; }
// Instruction N for a tile of ntok tokens: two rows per token, in the steps of 16 that M = 256 allows.
__host__ __device__ inline int tile_n(int ntok) { return (2 * ntok + 15) & ~15; }

// Weight tiles of one 120-row half of a block: pairs of k slices of 16 KB, [codes, 2 x 7680][scale atoms, 2 x 512],
// then a single slice of 8 KB, [codes][scale atom], where their number is odd.  Byte of slice kc's codes and scales:
__host__ __device__ inline size_t w_codes_offset(int kc) {
  return static_cast<size_t>(kc >> 1) * 2 * kWTileBytes + (kc & 1) * kWTileCodes;
}
__host__ __device__ inline size_t w_scales_offset(int kc, int n_kc) {
  const int in_pair = (kc | 1) < n_kc ? 2 : 1;   // slices stored together with this one
  return static_cast<size_t>(kc >> 1) * 2 * kWTileBytes + in_pair * kWTileCodes + (kc & 1) * kSfAtomBytes;
}

// Device status bits (MOE_DBG_STATUS).
enum : unsigned {
  ST_WAIT_FULL = 1u,      // expert GEMM: TMA data never arrived
  ST_WAIT_EMPTY = 2u,     // expert GEMM: stage never released
  ST_WAIT_AREADY = 4u,    // expert GEMM: dequantised tile never published
  ST_WAIT_AFREE = 8u,     // expert GEMM: tensor-memory A buffer never released
  ST_WAIT_DFULL = 16u,    // expert GEMM: accumulator never completed
  ST_WAIT_DEMPTY = 32u,   // expert GEMM: accumulator never drained
  ST_BAD_INDEX = 64u,     // routing produced an out-of-range row
  ST_WAIT_PEER = 128u,    // TP collective: a peer's flag never arrived
  ST_Y_RANGE = 256u,      // expert GEMM: an MLP2 output does not fit fp16 (|y| > 65504)
};

// Error code for a non-zero device status word.
inline int status_error(unsigned st) {
  return (st & ST_BAD_INDEX) ? MOE_ERR_STATE : (st & ST_Y_RANGE) ? MOE_ERR_Y_RANGE : MOE_ERR_TIMEOUT;
}

constexpr int kMaxTp = 8;  // MAX_TP of getp-csrc/nccl.hpp:6
// Symmetric buffers of a tensor-parallel group as seen from one rank: entry r is rank r's buffer
// (a peer mapping, or this rank's own memory for r == rank).
struct TpPeers {
  void *gather[kMaxTp];       // bf16 [max_rows, H]: all-gather destination (gather_x_g)
  void *partial[kMaxTp];      // bf16 [max_rows, H]: this rank's partial block output (e_agg_g)
  uint32_t *flags[kMaxTp];    // [kTpPhases][kMaxTp] epoch words
  void *topk_idx[kMaxTp];     // i32 [max_rows, K]: every rank routes its own rows and writes them to all (topk_i_g)
  void *topk_w[kMaxTp];       // f32 [max_rows, K]                                                  (topk_v_g)
};
constexpr int kTpBufs = 5;
// Hand-shakes of a tensor-parallel call, each with its own row of epoch words: the gathered rows are in
// place, the partial outputs are in place, the expert selections are in place.
enum { kTpPhaseGather = 0, kTpPhaseScatter = 1, kTpPhaseSelection = 2, kTpPhases = 3 };

// One call in flight through moe_forward_host_submit: its own input and output staging, so that the copies of
// neighbouring calls overlap the block of this one.
constexpr int kHostSlots = 3;
struct HostSlot {
  __nv_bfloat16 *in = nullptr, *out = nullptr;   // [max_rows, H] each
  unsigned int *status_dev = nullptr;            // status word of the call that owns the slot (cleared in stream order)
  unsigned int *status_host = nullptr;           // pinned copy of it, taken after the block
  cudaEvent_t in_ready = nullptr, out_ready = nullptr, done = nullptr;
  long long ticket = -1;                         // call that owns the slot; -1: free
};

// One work item of the grouped GEMM: one token tile against one kBlockRows-row block of the expert's weight matrix.
struct __align__(16) WorkItem {
  int expert;  // expert index
  int ntile;   // kBlockRows-row block of that expert's weight matrix
  int tile;    // global token-tile index
  int row0;    // first permuted row of the token tile
  int ntok;    // token rows in the tile (1..kMaxTileTok)
  int lead;    // 1 for the one item of its weight block (the expert has one token tile): the block is brought into L2 ahead
  int pad[2];
};

struct GemmArgs {
  const WorkItem *work;
  const int *n_work;
  int K;          // reduction length in elements (multiple of 32)
  int R;          // weight rows per expert on this rank
  int n_kchunks;  // ceil(K / kChunkK)
  int n_ntiles;   // ceil(R / kBlockRows)
  const uint8_t *w_tiles;     // weight tiles [E][n_ntiles][2][n_kchunks * kWTileBytes], see LayerWeights::w1_tiles
  int x_half0;                // token rows, e4m3 [tile][slice_pairs(n_kchunks)][2 halves]: the first half's place in TokenMaps
  int sfb_tile0, sfb_step;    // their scales: place of tile 0 in TokenMaps, and of the next one (0: shared by all tiles)
  const __nv_bfloat16 *bias;  // [E][R]
  int add_bias;               // MLP2 on TP ranks other than 0 leaves the bias out
  uint8_t *hq_out;            // MLP1: quantised SwiGLU output, tiled like xq
  int hq_joff, hq_nkc;        //       column of the shard's first output inside MLP2's k window; its k slices
  __half *y_out;              // MLP2: [P, ld_out] fp16
  int ld_out;
  int h_exp;                  // MLP1: SwiGLU outputs are stored as e4m3(h * 2^-h_exp)
  float limit, alpha;
  unsigned int *status;
};

// How one launch of the expert GEMM kernel runs: which phases (0 = MLP1, 1 = MLP2), and where the MLP1 items
// of a token tile are counted so that the tile's MLP2 items, in the same launch, know when its SwiGLU rows
// are complete.
struct MlpFuse {
  int phase_begin, phase_end;
  unsigned int *tile_done;   // [total_slot + 1], zeroed by build_index_kernel; nullptr: phases in separate launches
  int total_slot;            // the last word counts the MLP1 items of all tiles
  int done_per_tile;         // CTAs of a pair x MLP1 weight blocks
};

// Tensor maps of the quantised token rows, xq and hq as one array of halves (what one CTA of a pair reads of a pair of k
// slices, kPairBytes / 2) and their scales as one array of kSfbTileBytes.  rows[g - 1]: a box is the first g 8-row groups
// of both slices, 2 KB each, for tiles of tile_n = 16 g rows.
struct TokenMaps {
  CUtensorMap rows[kMaxTileTok / 8];
  CUtensorMap scales;
};
// Tensor maps of a weight matrix: codes and scale atoms of a pair of k slices, and of the single last slice.
struct WeightMaps {
  CUtensorMap codes, scales, codes_last, scales_last;
};

struct LayerWeights {
  bool loaded = false;
  // MLP1 weights as the GEMM streams them, 8 KB per (expert, 240-row block, 120-row half, 128-wide slice of k):
  // 120 rows x 64 bytes of packed e2m1 codes and one 512-byte E8M0 scale atom in the order tcgen05.cp wants, two
  // slices stored together (w_codes_offset, w_scales_offset).  Rows or k beyond the matrix hold zero codes and
  // scale 1 (byte 127).
  uint8_t *w1_tiles = nullptr;
  __nv_bfloat16 *b1 = nullptr;   // [E, R1]
  uint8_t *w2_tiles = nullptr;   // MLP2 weights [E, H, Kw], same tiling
  __nv_bfloat16 *b2 = nullptr;   // [E, H]
  // raw (row-major, unpadded) scales for the validation GEMM
  uint8_t *w1_scales_raw = nullptr;  // [E, R1, H/32]
  uint8_t *w2_scales_raw = nullptr;  // [E, H, Dl/32]
  __nv_bfloat16 *router_w3 = nullptr;  // [3][E][H] exact 3-way bf16 split of the fp32 router weight
  float *router_b = nullptr;           // [E]
  WeightMaps tm_w1, tm_w2;
  CUtensorMap tm_router;
};

}  // namespace moe

struct moe_ctx {
  moe_config cfg;
  int H, D, E, K, L;
  int d0, Dl;     // this rank's slice of the intermediate dimension
  int R1;         // 2*Dl
  int k0, Kw;     // MLP2 reads intermediate columns [k0, k0+Kw): the whole scale blocks around the shard
  int joff;       // d0 - k0: column of the shard's first SwiGLU output inside that window
  int max_rows, max_pairs;
  int sm_count;
  int gemm_grid = 0;        // CTAs of the expert GEMM (two per pair) the device keeps resident at once
  int router_cluster = 0;   // largest thread-block cluster the fused router kernel can use on this device (0: none)
  cudaStream_t stream = nullptr;  // used by moe_forward_host
  std::vector<moe::LayerWeights> layers;

  // run state (names of the reference's GPURunState fields in comments)
  __nv_bfloat16 *t_in = nullptr;    // gather_x_g          [max_rows, H]
  __nv_bfloat16 *t_norm = nullptr;  // t                   [max_rows, H]  RMS-normalised rows of moe_block()
  float *logits = nullptr;          // router_score_g      [max_rows, E]
  float *router_part = nullptr;     // split-k partial sums of the router [splits, rows, E]
  int *topk_idx = nullptr;          // topk_i_g            [max_rows, K]
  float *topk_w = nullptr;          // topk_v_g            [max_rows, K]
  int *hist = nullptr;              // selections per expert of the running call [E]; zero between calls (combine clears it,
                                    // or the failing call itself)
  int *counts = nullptr;            // d_expert_counts     [E]   hist of the last call, kept
  int *offsets = nullptr;           // d_expert_offsets    [E+1]
  int *pair_row = nullptr;          // local_ids_g         [max_rows, K]
  int *row_token = nullptr;         // expert_row_token_g  [max_pairs]
  int2 *pair_slot = nullptr;        // place of (token, k) in xq: tile * kMaxTileTok + token, scale row [max_rows, K]
  unsigned int *tile_done = nullptr;   // [max_tiles + 1] MlpFuse::tile_done
  __half *xperm = nullptr;          // expert_input_buffer [max_pairs, H]   fp16 (validation GEMM only)
  __half *hbuf = nullptr;           // gate_up             [max_pairs, Dl]  fp16 (validation GEMM only)
  uint8_t *xq = nullptr;            // expert_input_buffer as e4m3 high/low rows, [max_tiles][pairs of k slices][kPairBytes]
  uint8_t *hq = nullptr;            // gate_up as e4m3 high/low rows, same tiling over MLP2's k window (behind xq, one allocation)
  uint8_t *sfb_x = nullptr;         // per-tile scale atoms of xq [max_tiles][1024], then those of hq, the same for every tile
  moe::TokenMaps tm_x;              // of xq, hq and their scales
  int *tile_base = nullptr;         // first token tile of each expert [E+1]
  int max_tiles = 0;
  int h_exp = 0;                    // hq holds e4m3(h * 2^-h_exp)
  __half *ybuf = nullptr;           // expert_output_partial [max_pairs, H] fp16
  float *out_f32 = nullptr;         // fp32 block output   [max_rows, H] (debug / TP partial)
  __nv_bfloat16 *out_bf16 = nullptr;// e_agg_g             [max_rows, H]
  moe::WorkItem *work1 = nullptr, *work2 = nullptr;
  int *n_work = nullptr;            // [2]
  int max_work1 = 0, max_work2 = 0;
  unsigned int *status = nullptr;
  int last_rows = 0;
  long long launches = 0;
  moe::TpPeers peers = {};          // TP group view; own entries are set at creation
  __nv_bfloat16 *tp_partial = nullptr;  // this rank's bf16 partial output [max_rows, H]
  uint32_t *tp_flags = nullptr;     // [kTpPhases][kMaxTp], written by the peers
  uint64_t tp_attached = 0;         // bit (kTpBufs*r + which) set once rank r's buffer `which` is known
  moe::HostSlot host_slots[moe::kHostSlots];
  cudaStream_t h2d_stream = nullptr, d2h_stream = nullptr;
  long long host_submitted = 0;
  cudaStream_t aux_stream = nullptr;  // the all-gather push runs beside the router
  cudaEvent_t ev_fork = nullptr, ev_fork2 = nullptr, ev_join = nullptr;
  uint32_t tp_epoch = 0, tp_epoch_rs = 0;  // all-gather / reduce-scatter call counters
  std::vector<void *> ipc_opened;   // mappings to close at destroy
  bool profiling = false;
  std::vector<cudaEvent_t> prof_events;  // MOE_N_STAGES + 1 per profiled call
  std::vector<cudaEvent_t> prof_pool;    // recycled events
  std::string err;
};

namespace moe {

// cuTensorMapEncodeTiled through the runtime's driver entry point table (no link against libcuda).
typedef CUresult (*TensorMapEncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                      const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                      CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline TensorMapEncodeFn tensor_map_encoder() {
  static TensorMapEncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<TensorMapEncodeFn>(p);
  });
  return fn;
}

// Programmatic dependent launch.  The kernels of a block run one after the other and the small ones are mostly launch
// latency and set-up; launched with chained = true a kernel may start while its predecessor in the stream still runs.
// Every kernel of the chain therefore begins with grid_dep_sync(): it lets the successor start in turn, and waits until
// the predecessor has completed and its writes are visible.  Before it only parameters, barriers and tensor memory
// are touched (the router also fetches its weights).  Since every grid waits for the one before it, a completed grid
// means that all earlier ones are complete.  Without the attribute the wait returns at once.
// What such a kernel reads is still being written while it is resident: results of its predecessors, rows and gain of the
// caller, buffers that the kernels of the call before are still using.  It reads them with ordinary loads, behind the wait:
// the read-only path (__ldg, or const __restrict__, which lets the compiler take it) promises data that nobody writes
// during the kernel's life, and a load of such data may be moved above the wait.  Only what moe_load_layer wrote is constant.
// Measured, whole calls: 1 row 54.4 -> 47.3 us, 64 rows of 32 experts 114.5 -> 104.8, 256 rows (block) 343 -> 338.
__device__ __forceinline__ void grid_dep_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_sync() {
  grid_dep_release();
  grid_dep_wait();
}
template <class... Params, class... Args>
cudaError_t launch_kernel(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s, bool chained,
                          unsigned cluster_y, Args &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  unsigned n = 0;
  if (chained) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster_y > 0) {   // thread-block clusters of cluster_y CTAs along y
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = 1;
    at[n].val.clusterDim.y = cluster_y;
    at[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(std::forward<Args>(args))...);
}

// What the fused router kernel writes: logits [rows, E], and the selection, weights and expert histogram
// exactly as topk_softmax_kernel does (to every rank's top-k buffers when tp > 0, at row_offset).
struct RouteOut {
  float *logits;
  const float *bias;
  int K;
  int *idx;
  float *w;
  int *counts;
  int tp;
  int row_offset;
  TpPeers peers;
};

// router_sm100.cu
cudaError_t router_init(int *max_cluster);   // per-device kernel attributes; call with the device current
int router_fused_slices(int T, int H, int E, int sm_count, int max_cluster);
bool launch_router_fused(const __nv_bfloat16 *t, const CUtensorMap &tm_w, int T, int H, int E, int slices,
                         const RouteOut &ro, unsigned int *status, cudaStream_t s, bool chained);
int router_splits(int T, int H, int sm_count);
int router_chunks(int H);
bool make_router_weight_map(CUtensorMap *m, const __nv_bfloat16 *w3, int E, int H);
bool launch_router_partials(const __nv_bfloat16 *t, const CUtensorMap &tm_w, float *partial, int T, int H, int E,
                            int splits, unsigned int *status, cudaStream_t s, bool chained = false);
// route.cu
void launch_topk_softmax(float *logits, const float *partial, int splits, const float *bias, int T, int E, int K,
                         int *idx, float *w, int *counts, cudaStream_t s, int tp = 0, const TpPeers *peers = nullptr,
                         int row_offset = 0, bool chained = false);
void launch_count_experts(const int *idx, int n, int E, int *counts, cudaStream_t s);
void launch_build_index(const int *topk_idx, const int *hist, int *counts, int T, int E, int K, int n_ntiles1, int n_ntiles2,
                        int *offsets, int *tile_base, int *pair_row, int *row_token, int2 *pair_slot, unsigned int *tile_done, int tile_done_total_slot, WorkItem *work1,
                        WorkItem *work2, int *n_work, int max_work1, int max_work2, unsigned int *status,
                        cudaStream_t s, bool chained);
void launch_quantize_rows(const __nv_bfloat16 *t, const int2 *pair_slot, int T, int K, uint8_t *xq, uint8_t *sfb, int H,
                          cudaStream_t s, bool chained);
int quantize_rows_max_hidden();
void launch_gather_rows(const __nv_bfloat16 *t, const int *row_token, const int *offsets, int E, __half *xperm,
                        int H, int max_pairs, cudaStream_t s);
void launch_combine(const __half *y, const int *topk_idx, const float *topk_w, const int *pair_row, int T, int H,
                    int K, __nv_bfloat16 *out_bf16, float *out_f32, int *hist, int E, cudaStream_t s, bool chained, int tp = 0,
                    const TpPeers *peers = nullptr, int rows_local = 0, int rank = 0,
                    const __nv_bfloat16 *residual = nullptr);
void launch_rmsnorm_rows(const __nv_bfloat16 *x, const __nv_bfloat16 *w, __nv_bfloat16 *t, int rows, int H,
                         cudaStream_t s, bool chained);

// expert_gemm_sm100.cu
cudaError_t expert_gemm_init(int *grid);   // per-device kernel attributes; call with the device current
void launch_expert_mlp(const WeightMaps &tm_w1, const GemmArgs &a, const WeightMaps &tm_w2, const GemmArgs &b,
                       const TokenMaps &tm_x, const MlpFuse &f, int grid, cudaStream_t s, bool chained);
int expert_mlp_done_per_tile(int n_ntiles1);

// tp_collectives.cu
// Both pushes send rows [row0, row0 + n_rows) of this rank's rows_local rows (n_rows < 0: all of them).
void launch_tp_allgather_push(const __nv_bfloat16 *src, int rows_local, int H, const TpPeers &peers, int tp, int rank,
                              cudaStream_t s, int row0 = 0, int n_rows = -1);
void launch_tp_rmsnorm_push(const __nv_bfloat16 *x, const __nv_bfloat16 *w, int rows_local, int H, const TpPeers &peers,
                            int tp, int rank, cudaStream_t s, int row0 = 0, int n_rows = -1);
void launch_tp_signal_wait(const TpPeers &peers, uint32_t *my_flags, int tp, int rank, int phase, uint32_t epoch,
                           unsigned int *status, cudaStream_t s);
void launch_tp_sum_slots(const __nv_bfloat16 *landing, int tp, int rows_local, int H, __nv_bfloat16 *out, int sm_count,
                         cudaStream_t s, const __nv_bfloat16 *residual = nullptr);
void launch_tp_reduce_scatter_pull(const TpPeers &peers, int tp, int rank, int rows_local, int H, __nv_bfloat16 *out,
                                   int sm_count, cudaStream_t s);
void launch_tp_sum_all(const TpPeers &peers, int tp, size_t n_elems, __nv_bfloat16 *out, int sm_count, cudaStream_t s);

// expert_gemm_simt.cu (validation path)
void launch_simt_mlp1(const uint8_t *w_tiles, const uint8_t *scales_raw, const __nv_bfloat16 *bias,
                      const __half *x, const int *offsets, int E, int H, int R1, __half *h_out, int ld_h,
                      float limit, float alpha, int n_rows, cudaStream_t s);
void launch_simt_mlp2(const uint8_t *w_tiles, const uint8_t *scales_raw, const __nv_bfloat16 *bias,
                      int add_bias, const __half *h, const int *offsets, int E, int Dl, int H, __half *y_out,
                      int n_rows, cudaStream_t s);

// moe_tp_api.cu: argument and group checks shared by the calls of a tensor-parallel group.
int check_tp_call(moe_ctx *c, int rows_local, const char *who);

// moe_api.cu: the block itself.  With tp_rows_local > 0 this is a call of a tensor-parallel group: t is the
// gather buffer, t_local this rank's rows; routing is computed for the local rows only and exchanged, the
// combine pushes each row's partial to the rank that owns it, and out_dev receives this rank's summed rows.
// With norm_gain set (moe_block) `residual` holds the rows of the residual stream and the call starts with
// their RMSNorm: into c->t_norm, which then replaces t (one GPU) or t_local (TP group; the all-gather push
// normalises on the fly).
int forward_impl(moe_ctx *c, int layer, const __nv_bfloat16 *t, int T, __nv_bfloat16 *out_dev, unsigned flags,
                 cudaStream_t s, const __nv_bfloat16 *t_local, int tp_rows_local,
                 const __nv_bfloat16 *residual = nullptr, unsigned int *status = nullptr,
                 const __nv_bfloat16 *norm_gain = nullptr);

}  // namespace moe
