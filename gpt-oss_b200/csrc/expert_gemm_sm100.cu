// Grouped expert GEMM for sm_100a: block-scaled tcgen05 MMA (kind::mxf8f6f4)
// that consumes the MXFP4 expert weights exactly as they lie in HBM, for MLP1
// (+bias, clamped SwiGLU) and MLP2 (+bias).
//
// Reference counterparts: grouped_mlp1_bf16_bias_kernel_tiled_optimized_outbf16
// and grouped_mlp2_... (getp-csrc/kernels/moe.hpp:2651, :2923, :3197) with
// swiglu_epilogue_kernel_bf16_mlp_in_bf16 (:1472) between them, fed by weights
// that the reference first expands to bf16 in a staging buffer
// (getp_run.cpp:1019-1086).  Here the packed 4-bit codes and their E8M0 scales
// go from HBM through TMA straight into the tensor core; no thread touches a
// weight.
//
// There is no bf16 x fp4 instruction, so every bf16 activation is split into two e4m3
// terms (high + low, exact for bf16 inputs): row 2i of a token tile is the high term of its
// token i, row 2i+1 the low term, whose block scale carries the extra 2^-4.  The two partial
// sums land in adjacent columns of the accumulator and are added in the epilogue.
//
// Why this shape.  Two CTAs (a cluster, one TPC) work on one item: 240 weight rows
// against up to 96 tokens of one expert, M256 (120 of 128 rows used in each CTA; 240 divides
// both 5760 and 2880) x N x K32 instructions of cta_group::2.  The weights are the M operand,
// so that N follows the number of tokens in steps of 8 and an expert with a few rows pays for
// a few rows; each CTA holds its own 120 weight rows and HALF of the token rows, which its
// tensor core shares with the peer's, so the token tile crosses L2 -> SM and the shared-memory
// port once per pair.
//
// Per 128-element slice of k (two to a shared-memory stage) each CTA loads: weight codes
// [120 rows x 128] (TMA, 16U4_ALIGN16B: 4-bit codes are expanded to the 8-bit containers the
// MMA reads, 128-byte swizzle), their 512-byte scale atom (pre-tiled at load time), and its
// half of the token rows.  The weights of both slices are one TMA box, and so are the token rows (the
// quantiser and the SwiGLU epilogue write them interleaved by slice and with the 128-byte
// swizzle already applied): what a role spends per stage is issue time, ~150 cycles per copy, ~110
// per wait, ~35 per commit, and it was that time that bounded earlier forms with one slice per stage.
// Two producer warps (weights and their scales; tokens) keep kStages stages in flight.  The MMA warp
// of the even CTA copies the scales of both CTAs to tensor memory (tcgen05.cp) and issues four
// instructions per slice for the pair.  The copies of both CTAs complete on the even CTA's barrier (loads of
// cta_group::2, whose completion is a release at cluster scope), where its MMA warp acquires them at cluster scope.
// (The odd CTA used to report what had landed with an arrival of CTA scope, which promises nothing across CTAs; with
// release at cluster scope such a report costs 0.9 us a stage.  Whole calls, us, report of CTA scope / now: 1 row 39.3 /
// 39.0, 32 rows 185.8 / 185.9, 64 rows of 32 experts 102.8 / 103.1, 256 rows (block) 330 / 331, larger ones within the spread
// of the runs.)
// Issuing warps stay converged and elect one lane, so that descriptors and
// tensor-memory addresses live in uniform registers.  Sixteen epilogue warps per CTA drain the
// fp32 accumulator (double buffered: 2 x 192 columns).
// One more warp counts finished MLP1 items for the MLP2 items that wait for them.
// No multicast: every CTA fetches its own tiles.
//
// Measured (B200, one launch of both phases, us, layer of 128 experts, hidden and intermediate size 2880; before: one CTA
// per item of 64 tokens x 240 rows, tokens on the fixed M = 128 axis), without the L2 prefetch further down: 32 rows
// 179 -> 174, 256 rows 324 -> 299, 1856 rows 412 -> 396, 8192 rows 1459 -> 1403.  Bound by HBM up to ~16 tokens per
// expert, by the tensor pipe at 8192 rows (86 % of the cycles, at the 1.29 GHz that the power cap leaves).  In between no
// single bound is shown: at 1856 rows (~58 tokens per expert) a stage takes 773 cycles, the tensor pipe 492 of them and HBM
// ~550.  A count of all bytes through the shared-memory port at 128 a cycle gives 734, but the same count at 8192 rows
// asks for more than what is measured there (~420 against 388 cycles per slice), so the port is not it as counted.
#include <cuda_fp8.h>

#include "moe_internal.cuh"
#include "sm100_ptx.cuh"
#include "swiglu.cuh"

namespace moe {

using namespace sm100;

constexpr int kStages = 4;
constexpr int kSlices = 2;                        // k slices per stage: one wait and one commit for eight MMAs
constexpr int kWBytes = kHalfRows * kChunkK;      // 15360: 120 rows x 128 containers
// the transaction count of a 16U4_ALIGN16B copy is the PACKED size: 120 rows x 64 bytes
constexpr int kWLoadBytes = kWTileCodes;
// the M = 128 rows of a weight slice are read 8 rows into what follows it: rows 120..127 of the accumulator are
// never used
constexpr int kXOff = kSlices * kWBytes;
constexpr int kSfaOff = kXOff + kPairBytes / 2;             // 24576: this CTA's half of the token rows, at most
constexpr int kSfbOff = kSfaOff + kSlices * kSfAtomBytes;   // token scales, loaded with the first stage of an item
constexpr int kStageBytes = kSfbOff + kSfbTileBytes;        // 57344
constexpr int kBarOff = kStages * kStageBytes;
constexpr int kNumBars = 2 * kStages + 4;         // full, empty, d_full[2], d_empty[2]
constexpr int kProgOff = kBarOff + 8 * kNumBars + 16;       // MLP1 items finished by each epilogue warp
constexpr int kSmemBytes = kProgOff + 16 * 4 + 1024 /*alignment slack*/;

constexpr int kEpiWarps = 16;             // four per tensor-memory lane quadrant
constexpr int kWProducerWarp = 16, kXProducerWarp = 17, kMmaWarp = 18, kDoneWarp = 19;
constexpr int kThreads = 20 * 32;

constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kAccBufCols = kTileRows;       // accumulator buffer d at columns d*192
constexpr uint32_t kSfbCol0 = 2 * kAccBufCols;    // + 8*(item & 1): token scales
constexpr uint32_t kSfaCol0 = kSfbCol0 + 16;      // + 4*(slice & 3): weight scales

static_assert(kSfaCol0 + 16 <= kTmemCols, "tensor memory");
static_assert(kWBytes % 1024 == 0 && kPairBytes % 2048 == 0 && kStageBytes % 1024 == 0, "swizzled tiles keep 1024-byte alignment");
static_assert(kSmemBytes <= 227 * 1024, "shared memory budget");

// Two fp32 values -> two e4m3 bytes (first value in the low byte), and back.
__device__ __forceinline__ uint32_t pack_e4m3x2(float a, float b) {
  return __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ float2 unpack_e4m3x2(uint32_t v) {
  const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(v), __NV_E4M3);
  return __half22float2(__half2(h));
}

__device__ __forceinline__ void st_release_cta(uint32_t saddr, uint32_t v) {
  asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(saddr), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_cta(uint32_t saddr) {
  uint32_t v;
  asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(saddr) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_acquire_gpu(const unsigned int *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// 4 x 4 byte transposes of two words across the four lanes that differ in bits 1 and 2: before, lane q holds four
// tokens of feature q, afterwards four features of token q.
__device__ __forceinline__ void transpose_pair(uint32_t &w0, uint32_t &w1, int q) {
  const bool b1 = (q & 2) != 0, b0 = (q & 1) != 0;
  uint32_t r = __shfl_xor_sync(0xffffffffu, __byte_perm(w0, w1, b1 ? 0x5410 : 0x7632), 4);
  const uint32_t y0 = __byte_perm(w0, r, b1 ? 0x3254 : 0x5410), y1 = __byte_perm(w1, r, b1 ? 0x3276 : 0x7610);
  r = __shfl_xor_sync(0xffffffffu, __byte_perm(y0, y1, b0 ? 0x6420 : 0x7531), 2);
  w0 = __byte_perm(y0, r, b0 ? 0x3514 : 0x5240);
  w1 = __byte_perm(y1, r, b0 ? 0x3716 : 0x7260);
}

// One launch runs the phases [f.phase_begin, f.phase_end): phase 0 = MLP1 (bias + SwiGLU -> e4m3 high/low
// rows, args pa), phase 1 = MLP2 (bias -> fp16, args pb).  Run together, the pipeline state (stage ring,
// accumulator buffers) simply carries over from the last MLP1 item of a CTA pair to its first MLP2
// item: no drain, no second prologue, and pairs that are out of MLP1 items start on MLP2 while the others
// finish.  An MLP2 item reads the SwiGLU rows of its token tile, which the MLP1 items of that tile (on any
// SM) have written: kDoneWarp counts a finished MLP1 item of its CTA into tile_done[tile] behind a fence, and
// the token producers wait (bounded) for the tile's count before they request the tile's rows; the weight
// producers run ahead of that wait.  MLP1 items wait for nothing and every pair is resident (the grid is
// what the device places at once), so the MLP2 waits always end.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
expert_gemm_kernel(const __grid_constant__ WeightMaps tm_w1, const __grid_constant__ WeightMaps tm_w2,
                   const __grid_constant__ TokenMaps tm_x, const GemmArgs pa, const GemmArgs pb, const MlpFuse f) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + kBarOff;
  volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(smem_gen + kBarOff + 8 * kNumBars);
  uint32_t *tmem_slot = const_cast<uint32_t *>(abort_flag) + 1;
  const uint32_t prog_base = smem_base + kProgOff;

  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kStages + s); };
  auto dfull_bar = [&](int d) { return bar_base + 8u * (2 * kStages + d); };
  auto dempty_bar = [&](int d) { return bar_base + 8u * (2 * kStages + 2 + d); };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());   // 0 issues the MMAs of the pair

  if (threadIdx.x == 0) {
    // full (used in the even CTA only): its producers, which announce the bytes of both CTAs
    for (int s = 0; s < kStages; ++s) { mbar_init(full_bar(s), 2); mbar_init(empty_bar(s), 1); }
    for (int d = 0; d < 2; ++d) {
      mbar_init(dfull_bar(d), 1);
      mbar_init(dempty_bar(d), 2 * kEpiWarps);   // the epilogue warps of both CTAs (even CTA's copy only)
    }
    *abort_flag = 0u;
    for (int w = 0; w < kEpiWarps; ++w) st_release_cta(prog_base + 4u * w, 0u);
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == kMmaWarp) {
    tmem_alloc_pair(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish_pair();
  }
  if (warp == kWProducerWarp && lane == 0) {
    const WeightMaps *m = f.phase_begin == 0 ? &tm_w1 : &tm_w2;
    prefetch_tensormap(&m->codes);
    prefetch_tensormap(&m->scales);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_dep_sync();   // from here on the work lists and the token rows are read

  // Items of a phase are dealt round-robin to the pairs.  In a fused launch the MLP2 deal starts where the MLP1
  // deal ended, so that the pairs with one MLP1 item more are not also the ones with one MLP2 item more.
  const int n_work1 = *pa.n_work;
  const int pairs = static_cast<int>(gridDim.x) >> 1, pair = static_cast<int>(blockIdx.x) >> 1;
  auto first_item = [&](int phase) -> int {
    if (phase == 0 || f.phase_begin != 0) return pair;
    return (pair + pairs - n_work1 % pairs) % pairs;
  };
  unsigned int *status = pa.status;
  bool ok = true;
  // The even CTA's full barriers.  A copy of the odd CTA for the next use of a stage cannot come early: it waits for the
  // MMAs of the present one, which wait for the barrier's phase.
  const uint32_t full0 = map_to_cta(full_bar(0), 0);

  if (warp == kWProducerWarp) {
    // ------------------------------------------------------------- weight producer
    uint32_t s = 0, e_par = 1u;   // a fresh stage passes the first wait
    const uint64_t w_policy = l2_policy_evict_first();
   for (int phase = f.phase_begin; ok && phase < f.phase_end; ++phase) {
    const bool second = phase != 0;
    const WeightMaps *tm_w = second ? &tm_w2 : &tm_w1;
    const WorkItem *work = second ? pb.work : pa.work;
    const int n_work = second ? *pb.n_work : n_work1;
    const int nkc = second ? pb.n_kchunks : pa.n_kchunks, n_ntiles = second ? pb.n_ntiles : pa.n_ntiles;
    const uint8_t *w_tiles = second ? pb.w_tiles : pa.w_tiles;
    const int first = first_item(phase);
    WorkItem w_next = {};
    if (first < n_work) w_next = work[first];
    for (int wi = first; ok && wi < n_work; wi += pairs) {
      const WorkItem w = w_next;
      // the weights of the item after this one (the first of MLP2 after the last of MLP1)
      const uint8_t *ahead = nullptr;
      int ahead_nkc = nkc;
      if (wi + pairs < n_work) {
        w_next = work[wi + pairs];
        if (w_next.lead) ahead = w_tiles + static_cast<size_t>((w_next.expert * n_ntiles + w_next.ntile) * 2 + rank) * nkc * kWTileBytes;
      } else if (phase + 1 < f.phase_end) {
        const int wi2 = first_item(1);
        if (wi2 < *pb.n_work) {
          const WorkItem w2 = pb.work[wi2];
          ahead_nkc = pb.n_kchunks;
          if (w2.lead) ahead = pb.w_tiles + static_cast<size_t>((w2.expert * pb.n_ntiles + w2.ntile) * 2 + rank) * ahead_nkc * kWTileBytes;
        }
      }
      const int half = (w.expert * n_ntiles + w.ntile) * 2 + rank;
      // weights pass through once per step: the loads leave them first in line to go, before activations and results
      for (int kc = 0; kc < nkc; kc += kSlices) {
        if (!mbar_wait_warp<Wait::kClusterRelaxed>(empty_bar(s), e_par, abort_flag, status, ST_WAIT_EMPTY)) { ok = false; break; }
        const uint32_t stage = smem_base + s * kStageBytes;
        if (elect_one()) {
          // The ring alone holds less than HBM's latency takes at full rate (four stages turn round in ~2800 cycles):
          // while one item streams, the next one's weights come into L2.  It pays where HBM is the bound, that is for
          // experts with a single token tile (WorkItem::lead).  Whole calls, us, without it / for experts of one tile /
          // for the first tile of every expert: 1 row 41.6 / 39.2 / 39.3, 32 rows 195.5 / 185.1 / 184.9, 256 rows (block)
          // 338 / 328 / 327, 1856 rows 528 / 520 / 523; two tiles (32 experts, 1536 rows, block) 344 / 344 / 361; three
          // (8192 rows) 1824 / 1816 / 1895.  Experts of up to two tiles: 354 at two.  The evict-first policy of the
          // loads changes nothing here, neither the times nor the ~5 MB more that DRAM is written (464 rows, 32 experts).
          if (ahead != nullptr && kc < ahead_nkc)
            bulk_prefetch_l2(ahead + static_cast<size_t>(kc) * kWTileBytes, min(2, ahead_nkc - kc) * kWTileBytes);
          if (rank == 0) mbar_arrive_expect_tx(full_bar(s), 2 * min(2, nkc - kc) * (kWLoadBytes + kSfAtomBytes));
          const uint32_t bar = full0 + 8u * s;
          if (kc + 1 < nkc) {
            tma_load_5d_pair_hint(stage, &tm_w->codes, 0, 0, 0, kc >> 1, half, bar, w_policy);
            tma_load_3d_pair_hint(stage + kSfaOff, &tm_w->scales, 0, kc >> 1, half, bar, w_policy);
          } else {
            tma_load_3d_pair_hint(stage, &tm_w->codes_last, 0, 0, half, bar, w_policy);
            tma_load_2d_pair_hint(stage + kSfaOff, &tm_w->scales_last, 0, half, bar, w_policy);
          }
        }
        if (++s == kStages) { s = 0; e_par ^= 1u; }
      }
    }
   }
  } else if (warp == kXProducerWarp) {
    // ------------------------------------------------------------- token producer
    uint32_t s = 0, e_par = 1u;
    bool all_done = f.tile_done == nullptr;   // every MLP1 item of the launch is finished: no more checks
   for (int phase = f.phase_begin; ok && phase < f.phase_end; ++phase) {
    const bool second = phase != 0;
    const WorkItem *work = second ? pb.work : pa.work;
    const int n_work = second ? *pb.n_work : n_work1;
    const int nkc = second ? pb.n_kchunks : pa.n_kchunks;
    const int x_half0 = second ? pb.x_half0 : pa.x_half0;
    const int sfb_tile0 = second ? pb.sfb_tile0 : pa.sfb_tile0, sfb_step = second ? pb.sfb_step : pa.sfb_step;
    const int first = first_item(phase);
    WorkItem w_next = {};
    if (first < n_work) w_next = work[first];
    for (int wi = first; ok && wi < n_work; wi += pairs) {
      const WorkItem w = w_next;
      if (wi + pairs < n_work) w_next = work[wi + pairs];
      if (second && !all_done) {
        // the SwiGLU rows of this token tile: all MLP1 items of the tile (one per weight block) must have been
        // counted in by both CTAs of their pair
        const long long t0 = clock64();
        for (uint32_t spin = 0;; ++spin) {
          const uint32_t total = __shfl_sync(0xffffffffu, ld_acquire_gpu(f.tile_done + f.total_slot), 0);
          if (total >= 2u * static_cast<uint32_t>(n_work1)) { all_done = true; break; }
          const uint32_t mine = __shfl_sync(0xffffffffu, ld_acquire_gpu(f.tile_done + w.tile), 0);
          if (mine >= static_cast<uint32_t>(f.done_per_tile)) break;
          if ((spin & 15u) == 15u) {
            const bool late = __any_sync(0xffffffffu, clock64() - t0 > kWaitCycles);
            if (late || __any_sync(0xffffffffu, *abort_flag != 0u)) {
              if (late && lane == 0) { *abort_flag = 1u; atomicOr(status, ST_WAIT_AREADY); }
              ok = false;
              break;
            }
          }
        }
        if (!ok) break;
        // written with ordinary stores on other SMs, read by the copy engine here
        asm volatile("fence.proxy.async;" ::: "memory");
      }
      // this CTA's half of the tile's rows (both slices of a pair; of a single last slice the unused other half too)
      const int n_rows = tile_n(w.ntok);
      const uint32_t bytes = static_cast<uint32_t>(n_rows) * kChunkK;
      const CUtensorMap *tm_rows = &tm_x.rows[n_rows / 16 - 1];
      const int half = x_half0 + w.tile * slice_pairs(nkc) * 2 + rank;
      for (int kc = 0; kc < nkc; kc += kSlices) {
        if (!mbar_wait_warp<Wait::kClusterRelaxed>(empty_bar(s), e_par, abort_flag, status, ST_WAIT_EMPTY)) { ok = false; break; }
        const uint32_t stage = smem_base + s * kStageBytes;
        if (elect_one()) {
          if (rank == 0) mbar_arrive_expect_tx(full_bar(s), 2 * (bytes + (kc == 0 ? kSfbTileBytes : 0)));
          const uint32_t bar = full0 + 8u * s;
          if (kc == 0) tma_load_2d_pair(stage + kSfbOff, &tm_x.scales, 0, sfb_tile0 + w.tile * sfb_step, bar);
          tma_load_3d_pair(stage + kXOff, tm_rows, 0, 0, half + kc, bar);   // a pair of slices has two halves
        }
        if (++s == kStages) { s = 0; e_par ^= 1u; }
      }
    }
   }
  } else if (warp == kMmaWarp && rank != 0) {
    // the even CTA's warp issues for both
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------- even CTA: MMA issuer of the pair
    // The warp stays converged and one elected lane issues the tcgen05 instructions, so that their operands
    // live in uniform registers.  The weights and activations need no tcgen05 fence after their wait (copy
    // engine and tensor core meet through the mbarrier); the accumulator hand-over from the epilogue does.
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem_base, 0);
    uint32_t item = 0, s = 0, f_par = 0, sfa_sel = 0;
    const uint64_t desc_w = smem_desc_sw128(0), desc_x = smem_desc_sw128(0, 2048);   // slices alternate in the token rows
   for (int phase = f.phase_begin; ok && phase < f.phase_end; ++phase) {
    const bool second = phase != 0;
    const WorkItem *work = second ? pb.work : pa.work;
    const int n_work = second ? *pb.n_work : n_work1;
    const int K = second ? pb.K : pa.K, nkc = second ? pb.n_kchunks : pa.n_kchunks;
    const int full_chunks = K / kChunkK, tail_steps = (K % kChunkK) / 32;
    const int first = first_item(phase);
    int ntok_next = 0;
    if (first < n_work) ntok_next = work[first].ntok;
    for (int wi = first; ok && wi < n_work; wi += pairs, ++item) {
      const uint32_t n = __shfl_sync(0xffffffffu, static_cast<uint32_t>(tile_n(ntok_next)), 0);
      if (wi + pairs < n_work) ntok_next = work[wi + pairs].ntok;
      const uint32_t d = item & 1u;
      if (!mbar_wait_warp<Wait::kClusterRelaxed>(dempty_bar(d), ((item >> 1) & 1u) ^ 1u, abort_flag, status, ST_WAIT_DEMPTY)) { ok = false; break; }
      tc_fence_after();
      const uint32_t sfb_t = tm + kSfbCol0 + 8 * d;
      const uint32_t d_addr = tm + d * kAccBufCols;
      const uint32_t idesc = idesc_mxf8f6f4_m256(n, 0);
      auto mma_slice = [&](uint32_t sl, uint32_t stage, int steps, bool first) {   // one elected lane
        const uint32_t sfa_t = tm + kSfaCol0 + 4 * (sfa_sel + sl);
        const uint64_t adesc = desc_w | ((stage + sl * kWBytes) >> 4);
        const uint64_t bdesc = desc_x | ((stage + kXOff + sl * 1024) >> 4);
        tmem_cp_sf_atom_pair(sfa_t, stage + kSfaOff + sl * kSfAtomBytes);
        if (steps == 4) {
          mma_mxf8f6f4_pair(d_addr, adesc, bdesc, idesc, first ? 0u : 1u, sfa_t, sfb_t);
          mma_mxf8f6f4_pair(d_addr, adesc + 2, bdesc + 2, idesc | idesc_sf_id(1), 1u, sfa_t, sfb_t);
          mma_mxf8f6f4_pair(d_addr, adesc + 4, bdesc + 4, idesc | idesc_sf_id(2), 1u, sfa_t, sfb_t);
          mma_mxf8f6f4_pair(d_addr, adesc + 6, bdesc + 6, idesc | idesc_sf_id(3), 1u, sfa_t, sfb_t);
        } else {
          for (int kb = 0; kb < steps; ++kb)
            mma_mxf8f6f4_pair(d_addr, adesc + 2 * kb, bdesc + 2 * kb, idesc | idesc_sf_id(kb), first && kb == 0 ? 0u : 1u, sfa_t, sfb_t);
        }
      };
      for (int kc = 0; kc < nkc; kc += kSlices) {
        if (!mbar_wait_warp<Wait::kCluster>(full_bar(s), f_par, abort_flag, status, ST_WAIT_FULL)) { ok = false; break; }
        const uint32_t stage = smem_base + s * kStageBytes;
        if (elect_one()) {
          if (kc == 0) {
            tmem_cp_sf_atom_pair(sfb_t, stage + kSfbOff);
            tmem_cp_sf_atom_pair(sfb_t + 4, stage + kSfbOff + kSfAtomBytes);
          }
          if (kc + kSlices <= full_chunks) {
            mma_slice(0, stage, 4, kc == 0);
            mma_slice(1, stage, 4, false);
          } else {
            for (int k = kc; k < min(nkc, kc + kSlices); ++k) mma_slice(k - kc, stage, k < full_chunks ? 4 : tail_steps, k == 0);
          }
          mma_commit_pair(empty_bar(s));
        }
        if (++s == kStages) { s = 0; f_par ^= 1u; }
        sfa_sel ^= 2u;
      }
      if (ok && elect_one()) mma_commit_pair(dfull_bar(d));
    }
   }
  } else if (warp == kDoneWarp) {
    // ------------------------------------------------------------- counts finished MLP1 items
    // A fence takes about as long as a small item: here it stays out of the epilogue warps' way, and one fence
    // serves all items that every one of them has finished since the last.
    if (f.phase_begin == 0 && f.tile_done != nullptr) {
      uint32_t published = 0;
      const uint32_t mine = pair < n_work1 ? static_cast<uint32_t>((n_work1 - 1 - pair) / pairs + 1) : 0u;
      long long t0 = clock64();
      for (uint32_t spin = 0; published < mine; ++spin) {
        const uint32_t done = __reduce_min_sync(0xffffffffu, ld_acquire_cta(prog_base + 4u * (lane % kEpiWarps)));
        if (done > published) {
          // Each lane has acquired the progress of one epilogue warp; the warp barrier puts all sixteen before every
          // lane's fence, and the fence before the counts that the lane adds: whoever acquires a count sees all rows.
          __syncwarp();
          __threadfence();
          for (uint32_t i = published + lane; i < done; i += 32)
            atomicAdd(f.tile_done + pa.work[pair + static_cast<int>(i) * pairs].tile, 1u);
          if (lane == 0) atomicAdd(f.tile_done + f.total_slot, done - published);
          published = done;
          t0 = clock64();
          spin = 0;
        } else {
          if ((spin & 63u) == 63u) {   // the MMA and copy roles record what went wrong; this one only leaves
            if (__any_sync(0xffffffffu, *abort_flag != 0u || clock64() - t0 > 2 * kWaitCycles)) break;
          }
          __nanosleep(100);
        }
      }
    }
  } else {
    // ------------------------------------------------------------- epilogue warps
    // Warp w reads tensor-memory lanes 32*(w%4)..: lane l of quadrant q is weight row 32q + l of this CTA's 120;
    // neighbouring columns are the high and the low term of a token (x_operand_row).  Warps 4g..4g+3 take every
    // fourth chunk of 16 columns; the next chunk's load is in flight while one is processed.
    const int quad = warp & 3, grp = warp >> 2;
    const uint32_t lane_field = static_cast<uint32_t>(quad * 32) << 16;
    const int odd = lane & 1;
    const int lrow = quad * 32 + lane, q4 = (lane >> 1) & 3;
    const float h_scale = exp2f(static_cast<float>(-pa.h_exp));
    const uint32_t dempty0 = map_to_cta(dempty_bar(0), 0);
    uint32_t item = 0;
   for (int phase = f.phase_begin; ok && phase < f.phase_end; ++phase) {
    const bool second = phase != 0;
    const WorkItem *work = second ? pb.work : pa.work;
    const int n_work = second ? *pb.n_work : n_work1;
    const int R = second ? pb.R : pa.R;
    const bool add_bias = !second || pb.add_bias;
    const __nv_bfloat16 *bias = second ? pb.bias : pa.bias;
    const int first = first_item(phase);
    WorkItem w_next = {};
    if (first < n_work) w_next = work[first];
    for (int wi = first; ok && wi < n_work; wi += pairs, ++item) {
      const WorkItem w = w_next;
      if (wi + pairs < n_work) w_next = work[wi + pairs];  // in flight during the wait below
      const uint32_t d = item & 1u;
      const int n0 = w.ntile * kBlockRows + rank * kHalfRows;   // first weight row of this CTA's half
      const bool row_ok = lrow < kHalfRows && n0 + lrow < R;
      const float b = row_ok && add_bias ? __bfloat162float(bias[static_cast<size_t>(w.expert) * R + n0 + lrow]) : 0.f;
      const int n_chunks = tile_n(w.ntok) / 16;   // 8 tokens each, and as many 4-token groups per CTA
      if (!mbar_wait_warp<Wait::kClusterRelaxed>(dfull_bar(d), (item >> 1) & 1u, abort_flag, status, ST_WAIT_DFULL)) { ok = false; break; }
      tc_fence_after();
      const uint32_t acc = tmem_base + lane_field + d * kAccBufCols;
      auto release = [&]() {   // the accumulator is in registers (or not this warp's business): the MMAs may go on
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_relaxed_cluster(dempty0 + 8u * d);
      };
      auto process = [&](const uint32_t (&v)[16], int c) {
        // Sum of the high and low partial products, plus the bias of this lane's row.  Of a pair of lanes (rows
        // 2j, 2j+1) the even one finishes the first four tokens of the chunk, the odd one the others.
        const int grp4 = 2 * c + odd;   // the lane's group of 8 columns; the even CTA's groups come first
        const int t0 = (grp4 < n_chunks ? 2 * grp4 : 2 * (grp4 - n_chunks) + 1) * 4;
        float even_row[4], odd_row[4];   // MLP1: gate, up; MLP2: two neighbouring outputs
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float lo = __uint_as_float(v[2 * i]) + __uint_as_float(v[2 * i + 1]) + b;
          const float hi = __uint_as_float(v[2 * i + 8]) + __uint_as_float(v[2 * i + 9]) + b;
          const float got = __shfl_xor_sync(0xffffffffu, odd ? lo : hi, 1);
          even_row[i] = odd ? got : lo;
          odd_row[i] = odd ? hi : got;
        }
        if (!second) {
          float hs[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) hs[i] = swiglu_clamped(even_row[i], odd_row[i], pa.limit, pa.alpha) * h_scale;
          const uint32_t h0 = pack_e4m3x2(hs[0], hs[1]), h1 = pack_e4m3x2(hs[2], hs[3]);
          const float2 f0 = unpack_e4m3x2(h0), f1 = unpack_e4m3x2(h1);
          const uint32_t l0 = pack_e4m3x2((hs[0] - f0.x) * 16.0f, (hs[1] - f0.y) * 16.0f);
          const uint32_t l1 = pack_e4m3x2((hs[2] - f1.x) * 16.0f, (hs[3] - f1.y) * 16.0f);
          uint32_t hi4 = h0 | (h1 << 16), lo4 = l0 | (l1 << 16);
          transpose_pair(hi4, lo4, q4);   // four tokens of one feature per word -> four features of one token
          const int grow = quad * 32 + (lane & 24);   // first weight row of the lane group: 4 intermediate features
          if (grow < kHalfRows && n0 + grow < R && t0 + q4 < w.ntok) {
            const int j = pa.hq_joff + (n0 + grow) / 2;   // their column in MLP2's k window
            uint8_t *pr = pa.hq_out + (static_cast<size_t>(w.tile) * slice_pairs(pa.hq_nkc) + (j >> 8)) * kPairBytes;
            *reinterpret_cast<uint32_t *>(pr + x_pair_offset(t0 + q4, 0, j & 255)) = hi4;
            *reinterpret_cast<uint32_t *>(pr + x_pair_offset(t0 + q4, 1, j & 255)) = lo4;
          }
        } else if (row_ok) {   // R is a multiple of 32 here: both rows of a lane pair exist or neither does
          // fp16 keeps 11 significant bits of a value that the combine will round to 8; what it cannot hold
          // is a magnitude above 65504, which is reported, not stored silently as infinity
          float big = 0.f;
          __half *dst = pb.y_out + static_cast<size_t>(w.row0 + t0) * pb.ld_out + n0 + (lrow & ~1);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (t0 + i < w.ntok) {
              big = fmaxf(big, fmaxf(fabsf(even_row[i]), fabsf(odd_row[i])));
              *reinterpret_cast<__half2 *>(dst + static_cast<size_t>(i) * pb.ld_out) = __floats2half2_rn(even_row[i], odd_row[i]);
            }
          }
          if (big > 65504.f) atomicOr(status, ST_Y_RANGE);
        }
      };
      constexpr int kStep = kEpiWarps / 4;
      uint32_t va[16], vb[16];
      if (grp < n_chunks) tmem_ld16(acc + grp * 16, va);
      else release();
      for (int c = grp; c < n_chunks; c += 2 * kStep) {
        tmem_wait_ld();
        if (c + kStep < n_chunks) tmem_ld16(acc + (c + kStep) * 16, vb);
        else release();
        process(va, c);
        if (c + kStep >= n_chunks) break;
        tmem_wait_ld();
        if (c + 2 * kStep < n_chunks) tmem_ld16(acc + (c + 2 * kStep) * 16, va);
        else release();
        process(vb, c + kStep);
      }
      if (!second && f.tile_done != nullptr) {   // this warp's SwiGLU rows of the item are written
        __syncwarp();
        if (lane == 0) st_release_cta(prog_base + 4u * warp, item + 1u);
      }
    }
   }
  }

  if (!ok && warp >= kWProducerWarp) {  // give copies in flight time to land before shared memory is released
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // neither CTA leaves while the pair's MMAs, copies or reports may still touch its memory
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

// Per-device attributes; *grid receives the CTAs (two per pair) the device keeps resident at once, which the
// waits of MLP2 items on MLP1 items rely on.
cudaError_t expert_gemm_init(int *grid) {
  cudaError_t e = cudaFuncSetAttribute(expert_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmemBytes;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int pairs = 0;
  e = cudaOccupancyMaxActiveClusters(&pairs, expert_gemm_kernel, &cfg);
  if (e != cudaSuccess) return e;
  if (pairs < 1) return cudaErrorLaunchOutOfResources;
  *grid = 2 * pairs;
  return cudaSuccess;
}

// Phases [f.phase_begin, f.phase_end) of the expert MLP in one launch: both in the usual call, one at a
// time (two launches, f.tile_done = nullptr) on request.
void launch_expert_mlp(const WeightMaps &tm_w1, const GemmArgs &a, const WeightMaps &tm_w2, const GemmArgs &b,
                       const TokenMaps &tm_x, const MlpFuse &f, int grid, cudaStream_t s, bool chained) {
  launch_kernel(expert_gemm_kernel, dim3(grid), kThreads, kSmemBytes, s, chained, 0, tm_w1, tm_w2, tm_x, a, b, f);
}

int expert_mlp_done_per_tile(int n_ntiles1) { return 2 * n_ntiles1; }

}  // namespace moe
