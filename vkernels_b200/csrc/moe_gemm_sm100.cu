// moe_gemm_sm100.cu - the two grouped GEMMs of the fused MXFP4 MoE layer on
// tcgen05 tensor cores (sm_100a only).
//
// Orientation: the WEIGHTS are the M operand. One work item is 128 weight rows
// (gate/up GEMM: 64 gate rows + the 64 matching up rows; down GEMM: 128 rows)
// against up to 256 tokens of ONE expert (320 for a CTA pair, see below). A thread of a dequant warp owns one
// weight row = one TMEM lane: it reads the row's packed nibbles (K-contiguous,
// exactly the memory layout of the weights), expands them to bf16 with the
// exact table (common.cuh) and stores them with tcgen05.st as the A operand in
// tensor memory; the scale of a 32-element group is a per-thread scalar. The
// tokens are the N operand (any multiple of 16 up to 256), staged in shared
// memory by TMA with the 128-byte swizzle, so a ragged expert costs at most 15
// padded columns and a decode batch with a handful of tokens per expert still
// fills all 128 tensor-core rows. Accumulators D[weight row, token] stay in
// tensor memory (fp32) until the epilogue:
//   gate/up : bias, activation, ONE rounding to bf16, act[row, feature] store
//   down    : bias, routing weight, red.global.add.f32 into out[token, h]
//             (the weighted un-permute/combine, fused)
//
// Warp roles (640 threads, one persistent CTA per SM):
//   warp 0      TMA producer: packed weights (2 boxes of 64 rows x 128 B per
//               256-K stage) and scale bytes (bulk copy per item)
//   warp 1      tcgen05.mma issuer + tensor-memory allocation
//   warp 2      TMA producer: token tiles
//   warps 4-19  sixteen workers in sets of four (one warp per tensor-memory lane quarter):
//               dequant sets (shared memory -> registers -> tensor memory, a stage each in
//               turn) and epilogue sets (tensor memory -> registers -> global, a 32-token round
//               each in turn) - two + two for a CTA pair, three + one for a lone CTA
//
// Batches of up to a few dozen tokens an expert run moe_gemm_fp4.cu instead. Two forms here, chosen by the largest token
// tile of the launch:
//   lone CTA (the stage split of tensor parallelism, VK_MOE_SMALL=bf16, VK_MOE_PAIR=0, and reductions too long for a
//     pair): stages of 256 K-elements for tiles of up to 64 tokens, because the issuer's per-stage
//     handshake costs a few hundred cycles whatever the stage holds, and of 64 for tiles of up to 256;
//   CTA pair (larger tiles, the prefill regime): a cluster of two CTAs works on one item of
//     256 weight rows x up to 320 tokens with cta_group::2 MMAs. Each CTA dequantises its own
//     128 rows and stages HALF of the token rows, which halves the token bytes an SM pulls
//     from L2 per flop. Tensor memory: columns 0..255 main accumulator, 256..319 a second
//     accumulator for tokens 256..319 (fed by a second MMA per K block), 320..511 three A
//     slots of 128 K-elements. One ring serves A slots and token slots: the token bytes are
//     expected on the barrier the dequant warps arrive on.
//
// Every wait on an mbarrier is bounded; a wait that runs out raises a flag all
// roles observe, the CTA frees its tensor memory and returns, and the launcher
// reports the failure through the device-side status word.
//
// Reference behaviour replaced: gateup_swiglu_kernel* and down_combine_kernel*
// (src/c/vkernels/kernels/moe_fused.hip:681-1436) and their launcher
// (moe_fused.hip:1448-1663).
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <mutex>
#include <string>
#include <vector>

#include "common.cuh"
#include "moe_fused.hpp"
#include "moe_gemm_fp4.hpp"
#include "sm100.cuh"

namespace vkernels::kernels::cuda {

namespace {

// ---------------------------------------------------------------------------
// geometry
// ---------------------------------------------------------------------------
constexpr int kMaxTok = 256;        // tokens (MMA N) per work item of a lone CTA
// A CTA pair takes up to 320 tokens per item: a 256-column accumulator plus a 64-column one
// fed by a second MMA per K block. An expert whose token count is a little over 256 (the common
// case when tokens spread evenly) then costs one pass over its weights instead of two.
constexpr int kPairMainTok = 256;
constexpr int kPairMaxTok = 320;
constexpr int kRows = 128;          // weight rows (MMA M) per work item
constexpr int kWStageK = 256;       // K elements per packed-weight stage (128 B per row)
constexpr int kMaxWStages = 8;    // packed-weight ring depth is chosen per launch (3..8)
constexpr int kMaxAStages = 8;
constexpr int kMaxBStages = 8;
constexpr int kWStageBytes = kRows * 128;          // 16 KB
// 16 worker warps after the four control warps, split by form: a CTA pair (prefill) runs two
// dequant sets and two epilogue sets (the accumulator drains twice as fast, which is what its
// MMA issuer waits for); a lone CTA (decode) runs three dequant sets and one epilogue set (its
// epilogue is a few rounds, its bound is the expansion).
constexpr int dequant_sets(int ctas) { return ctas == 2 ? 2 : 3; }   // dequant warps per TMEM lane quarter
constexpr int epi_sets(int ctas) { return ctas == 2 ? 2 : 1; }       // epilogue warps per lane quarter
constexpr int block_threads(int ctas) { return (4 + 4 * (dequant_sets(ctas) + epi_sets(ctas))) * 32; }
constexpr int kPackedSfBytes = kRows * 8;   // prepacked scale factors of a 128-row, 256-K stage
constexpr int kTmemCols = 512;
constexpr int kEpiPitch = 72;                     // bf16 per staged token row: 64 features + 16 bytes against bank conflicts
// epilogue staging: gate/up two rounds of 32 tokens per set, down one 16 x 32 fp32 block per warp
constexpr int epi_stage_bytes(bool gateup, int ctas) { return epi_sets(ctas) * (gateup ? 2 * 32 * kEpiPitch * 2 : 4 * 16 * 32 * 4); }
// Lone-CTA form: byte -> bf16 pair lookup table in shared memory, one copy per bank (lane l reads
// word 32 * byte + l), so a warp's 32 lookups of different bytes are one conflict-free access.
constexpr int kLutBytes = 256 * 32 * 4;

// Device status word of the tensor-core kernels: 0, or 100 + the code of the wait that ran out.
// It lives in the library image (one per GPU that loads the library), so no launch needs a
// buffer for it and nothing but an expired wait writes it.
__device__ int g_kernel_status;

struct GemmParams {
  const uint8_t* w_scale;     // [E, n_wrows, K/32]
  const float* bias;          // gate/up: [E, 2*n_feat]; down: [E, n_feat]; or null
  const float* topk_w;        // down only
  const int32_t* sorted_ids;  // [EM]
  uint16_t* act;              // gate/up output [EM, n_feat]
  float* out;                 // down output [M, n_feat]
  float* const* out_rows;     // optional: address of each token's output row (may be another GPU's memory)
  int store_rows;             // with out_rows: out_rows[m] is a [top_k, n_feat] block; slot j's row (act @ w2^T + b2,
                              // unweighted) is STORED at row j instead of being added, weighted, into one row
  float* raw;                 // optional: plain fp32 result rows [EM, raw_ld] instead of the fused epilogue
  int raw_ld;                 //   (the tensor-parallel stage split: the caller reduces across ranks first)
  int k_base;                 // first column of the token rows this launch reduces over (K-sharded weights)
  const TokTile* tiles;
  const int* n_tiles;
  int K;                      // reduction length (hidden for gate/up, ispp for down)
  int n_feat;                 // gate/up: ispp; down: hidden
  int n_ftiles;
  int N;                      // M * top_k (sentinel of padded rows)
  int top_k;
  int w_sorted;
  int b_stages;
  int b_stage_bytes;          // max_tok * 128
  int w_stages;
  int max_tok;                // largest token tile of this launch (multiple of 16, <= 256)
  int scale_bufs;
  int scale_buf_bytes;
  int activation;
  float limit, beta, linear_beta;
};

// ---------------------------------------------------------------------------
// shared-memory carve-up
// ---------------------------------------------------------------------------
// Accumulator columns: a lone CTA sizes them by the stage length (long stages serve small token
// tiles), a pair always holds up to kPairMaxTok tokens.
constexpr int acc_cols(int ks, int ctas) { return ctas == 2 ? kPairMaxTok : (ks == 64 ? 256 : 64); }

struct Barriers {
  uint64_t w_full[kMaxWStages], w_empty[kMaxWStages];
  uint64_t a_full[kMaxAStages];    // dequant warps -> MMA issuer (4 arrivals, one per TMEM lane quarter)
  uint64_t stage_done[kMaxAStages];  // MMA completion of a stage: frees its A slot AND its token slot
  uint64_t b_full[kMaxBStages];
  uint64_t sc_full[2], sc_empty[2];
  uint64_t acc_full, acc_empty;
  uint32_t tmem_base;
  int abort_flag;
  // per token column of the current item: gate/up 1 for a real row, 0 for padding;
  // down: address of the token's output row, 0 for padding
  unsigned long long tile_ref[kPairMaxTok];
  float tile_w[kPairMaxTok];
};

// Tensor maps of the token rows. Pair form: m[i] has boxes of 16 (i + 1) rows x 128 K (two 64-K slices, one after the
// other in shared memory), so that a stage is one copy per CTA - two with extension rows - whatever the tile: a copy costs
// its issuing thread 200 clocks and more, and with four to eight boxes of 16 or 64 rows a stage that thread was what the
// kernel waited for. Lone CTA: m[0] and m[1] have boxes of 16 and 64 rows x 64 K.
struct TokMaps {
  CUtensorMap m[8];
};

// ---------------------------------------------------------------------------
// the kernel
// ---------------------------------------------------------------------------
// KS = K elements per pipeline stage (one A slot in tensor memory, one token
// slot in shared memory, one handshake of the MMA issuer). The issuer's
// per-stage latency (barrier polls + commit) is a few hundred cycles whatever
// the stage holds, so small token tiles, whose MMAs are short, take long
// stages: lone CTA, KS = 64 for tiles up to 256 tokens, 256 up to 64; pair, KS = 128.
template <bool GATEUP, int KS, int CTAS>
__global__ void __launch_bounds__(block_threads(CTAS), 1)
moe_gemm_sm100_kernel(const __grid_constant__ CUtensorMap tmap_w,
                      const __grid_constant__ TokMaps tok_maps, const GemmParams p) {
  constexpr int kThreads = block_threads(CTAS);
  constexpr int kAccCols = acc_cols(KS, CTAS);
  constexpr int kACols = KS / 2;                                      // columns of one A slot
  constexpr int kAStages = (kTmemCols - kAccCols) / kACols;           // lone CTA: 3 of 256, 8 of 64; pair: 3 of 128
  constexpr int kSubPerW = kWStageK / KS;                             // stages per packed-weight stage
  constexpr int kPieces = KS / 64;                                    // 64-K pieces of a stage
  static_assert(kAStages <= kMaxAStages, "A ring too deep for the barrier arrays");
  static_assert(CTAS == 1 || KS == 128, "the CTA-pair form takes 128-K stages");
  // CTAS == 2: two CTAs of a cluster work on one item - 256 weight rows (128 per CTA, each CTA
  // dequantises its own) against ONE token tile of up to 256 tokens, of which each CTA stages only
  // half. The leader (even) CTA issues cta_group::2 MMAs that read both halves; every CTA keeps
  // its 128 accumulator rows in its own tensor memory. This halves the token bytes a CTA pulls
  // from L2 per flop and doubles the depth of the token ring that fits in shared memory.
  // A pair keeps ONE ring: token slot i lives and dies with A slot i, and the token bytes are
  // expected on the same barrier the dequant warps arrive on, so the MMA issuer polls a single
  // barrier per stage.
  constexpr bool kMerged = CTAS == 2;
  constexpr int kDequantSets = dequant_sets(CTAS), kEpiSets = epi_sets(CTAS);
  constexpr int kEpiWarp0 = 4 + 4 * kDequantSets;   // first epilogue warp
  static_assert((kEpiWarp0 + 4 * kEpiSets) * 32 == kThreads, "the role split must use every warp");
  const uint32_t cta_rank = CTAS == 2 ? cluster_ctarank() : 0u;
  const bool leader = cta_rank == 0;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  uint8_t* w_smem = smem;                                      // w_stages x 16 KB
  uint8_t* b_smem = w_smem + p.w_stages * kWStageBytes;        // b_stages x b_stage_bytes
  uint8_t* sc_smem = b_smem + p.b_stages * p.b_stage_bytes;    // scale_bufs x scale_buf_bytes
  Barriers* bars = reinterpret_cast<Barriers*>(sc_smem + p.scale_bufs * p.scale_buf_bytes);
  // gate/up epilogue staging: 2 x (32 tokens x 64 features) bf16, 16-byte aligned
  uint16_t* epi_stage = reinterpret_cast<uint16_t*>(reinterpret_cast<uint8_t*>(bars) + ((sizeof(Barriers) + 127) & ~size_t(127)));
  constexpr bool kUseLut = CTAS == 1;
  uint32_t* lut = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(epi_stage) +
                                              epi_stage_bytes(GATEUP, CTAS));

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int* abort_flag = &bars->abort_flag;

  if (kUseLut) fill_dequant_lut(lut, tid, kThreads);
  if (tid == 0) {
    for (int i = 0; i < kMaxWStages; ++i) {
      mbar_init(smem_u32(&bars->w_full[i]), 1);
      mbar_init(smem_u32(&bars->w_empty[i]), 4 * kDequantSets);
    }
    for (int i = 0; i < kMaxAStages; ++i) {
      mbar_init(smem_u32(&bars->a_full[i]), kMerged ? 4 * CTAS + 1 : 4);
      mbar_init(smem_u32(&bars->stage_done[i]), 1);
    }
    for (int i = 0; i < kMaxBStages; ++i) mbar_init(smem_u32(&bars->b_full[i]), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&bars->sc_full[i]), 1);
      mbar_init(smem_u32(&bars->sc_empty[i]), 4 * kDequantSets);
    }
    mbar_init(smem_u32(&bars->acc_full), 1);
    mbar_init(smem_u32(&bars->acc_empty), 4 * kEpiSets * CTAS);
    bars->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    if (CTAS == 2) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_u32(&bars->tmem_base)),
                   "r"((uint32_t)kTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_u32(&bars->tmem_base)),
                   "r"((uint32_t)kTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (CTAS == 2) cluster_sync_all();   // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;

  const int n_tok_tiles = *p.n_tiles;
  const int unit = CTAS == 2 ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;      // CTA (pair) index
  const int n_units = CTAS == 2 ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int n_fgroups = (p.n_ftiles + CTAS - 1) / CTAS;   // feature tiles per token tile, in units of CTAS
  const int n_items = n_tok_tiles * n_fgroups;
  // feature tile of this CTA inside an item; with an odd tile count the last pair's second CTA idles
  auto item_f = [&](int item) { return (item % n_fgroups) * CTAS + (int)cta_rank; };
  const int n_kw = (p.K + kWStageK - 1) / kWStageK;   // packed-weight stages per item
  const int n_stages = (p.K + KS - 1) / KS;           // pipeline stages per item (last may be short)
  const int pitch = p.K / 32;                         // scale bytes per weight row
  const int n_wrows = GATEUP ? 2 * p.n_feat : p.n_feat;
  const int slice_bytes = p.max_tok * 128;            // lone CTA: one 64-K slice of a token stage

  if (warp == 0) {
    // ------------------- TMA producer: packed weights + scales ---------------
    // Runs ahead by the depth of its own ring, independent of the token stages,
    // so the weight stream (the HBM-bound part) is never held back by them.
    if (lane == 0) {
      Ring w;
      uint32_t sc_it = 0;
      bool ok = true;
      for (int item = unit; item < n_items && ok; item += n_units) {
        const TokTile tt = p.tiles[item / n_fgroups];
        const int f = item_f(item);
        int row_a, row_b, rows_valid;   // two boxes of 64 weight rows
        if (GATEUP) {
          row_a = tt.expert * n_wrows + f * 64;
          row_b = row_a + p.n_feat;
          rows_valid = 128;
        } else {
          row_a = tt.expert * n_wrows + f * 128;
          row_b = row_a + 64;
          rows_valid = min(128, p.n_feat - f * 128);
        }
        if (f >= p.n_ftiles) rows_valid = 0;   // idle half of the last pair: nothing to load
        {
          const int sb = sc_it % p.scale_bufs;
          const uint32_t par = ((sc_it / p.scale_bufs) & 1u) ^ 1u;
          if (!mbar_wait(smem_u32(&bars->sc_empty[sb]), par, abort_flag, 1, 128)) break;
          const uint32_t bar = smem_u32(&bars->sc_full[sb]);
          const uint32_t dst = smem_u32(sc_smem + sb * p.scale_buf_bytes);
          const uint32_t half = 64u * pitch;
          if (rows_valid == 0) {
            mbar_arrive(bar);
          } else {
            mbar_expect_tx(bar, rows_valid == 128 ? 2 * half : half);
            bulk_load_1d(dst, p.w_scale + (size_t)row_a * pitch, half, bar);
            if (rows_valid == 128)
              bulk_load_1d(dst + half, p.w_scale + (size_t)row_b * pitch, half, bar);
          }
          ++sc_it;
        }
        for (int kw = 0; kw < n_kw; ++kw) {
          if (!mbar_wait(smem_u32(&bars->w_empty[w.slot]), w.phase ^ 1u, abort_flag, 2, 128)) {
            ok = false;
            break;
          }
          const uint32_t bar = smem_u32(&bars->w_full[w.slot]);
          const uint32_t dst = smem_u32(w_smem + w.slot * kWStageBytes);
          if (rows_valid == 0) {
            mbar_arrive(bar);
          } else {
            mbar_expect_tx(bar, rows_valid == 128 ? kWStageBytes : kWStageBytes / 2);
            tma_load_2d(dst, &tmap_w, kw * (kWStageK / 2), row_a, bar);
            if (rows_valid == 128)
              tma_load_2d(dst + kWStageBytes / 2, &tmap_w, kw * (kWStageK / 2), row_b, bar);
          }
          w.advance(p.w_stages);
        }
      }
    }
  } else if (warp == 2) {
    // ------------------- TMA producer: token tiles ---------------------------
    // Token slot of stage s is free once the MMAs of stage s - b_stages are done;
    // that event is stage_done of the A slot that stage used (b_stages <= kAStages,
    // so the barrier cannot have moved on to a later phase yet).
    if (kMerged) {
      if (lane == 0) {
        Ring a;
        bool ok = true;
        for (int item = unit; item < n_items && ok; item += n_units) {
          const TokTile tt = p.tiles[item / n_fgroups];
          // The tile, rounded up to 32 rows, is split into a main part (<= 256 rows, first MMA)
          // and an extension (<= 64 rows, second MMA); this CTA stages half of each. Rows past
          // the tile are someone else's (or zero fill past the tensor): their columns are never
          // read back.
          const int n32 = (tt.n_rows + 31) & ~31;
          const int h0 = min(n32, kPairMainTok) >> 1, h1 = (n32 >> 1) - h0;
          const int row_main = tt.row0 + (int)cta_rank * h0;
          const int row_ext = tt.row0 + 2 * h0 + (int)cta_rank * h1;
          const CUtensorMap* map0 = &tok_maps.m[(h0 >> 4) - 1];
          const CUtensorMap* map1 = &tok_maps.m[h1 != 0 ? (h1 >> 4) - 1 : 0];
          for (int st = 0; st < n_stages; ++st) {
            if (!mbar_wait(smem_u32(&bars->stage_done[a.slot]), a.phase ^ 1u, abort_flag, 3, 64)) {
              ok = false;
              break;
            }
            const uint32_t bar = smem_u32(&bars->a_full[a.slot]);
            const uint32_t dst = smem_u32(b_smem + a.slot * p.b_stage_bytes);
            // (a slice past the end of K, or past the shard, is zero fill or other columns: it counts, and no MMA reads it)
            const int c2 = (p.k_base + st * KS) / 64;
            if (leader) mbar_expect_tx(bar, 2 * (h0 + h1) * 128 * kPieces);
            tma_load_3d_pair(dst, map0, 0, row_main, c2, bar);
            if (h1 != 0) tma_load_3d_pair(dst + kPieces * h0 * 128, map1, 0, row_ext, c2, bar);
            a.advance(kAStages);
          }
        }
      }
    } else if (lane == 0) {
      Ring b, lag;           // lag trails b by b_stages stages, on the A ring
      int issued = 0;        // stages issued so far (all items)
      bool ok = true;
      for (int item = unit; item < n_items && ok; item += n_units) {
        const TokTile tt = p.tiles[item / n_fgroups];
        for (int st = 0; st < n_stages; ++st, ++issued) {
          if (issued >= p.b_stages) {
            if (!mbar_wait(smem_u32(&bars->stage_done[lag.slot]), lag.phase, abort_flag, 3, 64)) {
              ok = false;
              break;
            }
            lag.advance(kAStages);
          }
          const uint32_t bar = smem_u32(&bars->b_full[b.slot]);
          const uint32_t dst = smem_u32(b_smem + b.slot * p.b_stage_bytes);
          const int k0 = st * KS;
          const int n_slices = min(kPieces, (p.K - k0) / 64);
          mbar_expect_tx(bar, tt.n_rows * 128 * n_slices);
          for (int sl = 0; sl < n_slices; ++sl) {
            int r = 0;
            for (; r + 64 <= tt.n_rows; r += 64)
              tma_load_2d(dst + sl * slice_bytes + r * 128, &tok_maps.m[1], p.k_base + k0 + sl * 64, tt.row0 + r, bar);
            for (; r < tt.n_rows; r += 16)
              tma_load_2d(dst + sl * slice_bytes + r * 128, &tok_maps.m[0], p.k_base + k0 + sl * 64, tt.row0 + r, bar);
          }
          b.advance(p.b_stages);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer -----------------------------
    // The whole warp stays converged: lanes 0 and 1 poll the A-ready and the
    // tokens-ready barrier of the stage in the SAME instruction (one poll latency
    // instead of two), lane 0 issues the MMAs and one commit per stage.
    uint32_t acc_phase = 0;
    bool ok = true;
    const uint32_t tmem_u = __shfl_sync(0xFFFFFFFFu, tmem_base, 0);
    if (kMerged) {
      // One thread's dependent instructions are the clock of this loop, so everything a stage
      // needs (barrier addresses, tensor-memory column, token descriptor) is carried along and
      // bumped per stage instead of being recomputed from the slot index.
      const uint32_t ready0 = smem_u32(&bars->a_full[0]), done0 = smem_u32(&bars->stage_done[0]);
      const uint32_t acc_full_bar = smem_u32(&bars->acc_full);
      const uint32_t a0 = tmem_u + kAccCols;
      const uint64_t desc_first = make_b_desc(smem_u32(b_smem));
      const uint32_t desc_step = (uint32_t)p.b_stage_bytes >> 4;
      uint32_t ready = ready0, done = done0, a_addr = a0, phase = 0;
      uint64_t desc = desc_first;
      int slot = 0;
      for (int item = unit; item < n_items && ok && leader; item += n_units) {
        const int n_rows_u = __shfl_sync(0xFFFFFFFFu, p.tiles[item / n_fgroups].n_rows, 0);
        const int n32 = (n_rows_u + 31) & ~31;
        const int n_main = min(n32, kPairMainTok), n_ext = n32 - n_main;
        const uint32_t idesc = make_idesc(n_main, 256), idesc_ext = make_idesc(n_ext, 256);
        // descriptor distances (16-byte units): slice to slice, main to extension rows
        const uint32_t slice16 = (uint32_t)(n_main >> 1) * 8u, ext16 = kPieces * slice16, slice16_ext = (uint32_t)(n_ext >> 1) * 8u;
        if (!mbar_wait(smem_u32(&bars->acc_empty), acc_phase ^ 1u, abort_flag, 4)) break;
        tc_fence_after();
        for (int st = 0; st < n_stages; ++st) {
          if (!mbar_wait(ready, phase, abort_flag, 5)) {
            ok = false;
            break;
          }
          tc_fence_after();
          if (elect_one()) {
            const int n_slices = min(kPieces, (p.K - st * KS) / 64);
#pragma unroll
            for (int sl = 0; sl < kPieces; ++sl) {
              if (sl < n_slices) {
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                  const uint32_t acc = (sl | kk) != 0 ? 1u : (st != 0 ? 1u : 0u);
                  tc_mma_ts_pair(tmem_u, a_addr + sl * 32 + kk * 8, desc + sl * slice16 + kk * 2, idesc, acc);
                  if (n_ext != 0)
                    tc_mma_ts_pair(tmem_u + kPairMainTok, a_addr + sl * 32 + kk * 8,
                                   desc + ext16 + sl * slice16_ext + kk * 2, idesc_ext, acc);
                }
              }
            }
            tc_commit_pair(done);   // completion is announced in both CTAs of the pair
            if (st == n_stages - 1) tc_commit_pair(acc_full_bar);
          }
          ready += 8;
          done += 8;
          a_addr += kACols;
          desc += desc_step;
          if (++slot == kAStages) {
            slot = 0;
            phase ^= 1u;
            ready = ready0;
            done = done0;
            a_addr = a0;
            desc = desc_first;
          }
        }
        acc_phase ^= 1u;
      }
    }
    Ring a, b;
    uint32_t acc_free = 1u;
    for (int item = unit; item < n_items && ok && !kMerged; item += n_units) {
      const int n_rows_u = __shfl_sync(0xFFFFFFFFu, p.tiles[item / n_fgroups].n_rows, 0);
      const uint32_t idesc = make_idesc(n_rows_u);
      if (!mbar_wait(smem_u32(&bars->acc_empty), acc_free, abort_flag, 4)) break;
      acc_free ^= 1u;
      tc_fence_after();
      for (int st = 0; st < n_stages; ++st) {
        const uint32_t bar = lane == 0 ? smem_u32(&bars->a_full[a.slot]) : smem_u32(&bars->b_full[b.slot]);
        if (!mbar_wait_lanes(bar, lane == 0 ? a.phase : b.phase, lane < 2, abort_flag, 5)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (elect_one()) {
          const uint32_t a_addr = tmem_u + kAccCols + a.slot * kACols;
          const uint64_t desc0 = make_b_desc(smem_u32(b_smem + b.slot * p.b_stage_bytes));
          const uint32_t slice16 = (uint32_t)slice_bytes >> 4;
          const int n_slices = min(kPieces, (p.K - st * KS) / 64);
#pragma unroll
          for (int sl = 0; sl < kPieces; ++sl) {
            if (sl < n_slices) {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                tc_mma_ts(tmem_u, a_addr + sl * 32 + kk * 8, desc0 + sl * slice16 + kk * 2, idesc,
                          (st | sl | kk) != 0 ? 1u : 0u);
            }
          }
          tc_commit(smem_u32(&bars->stage_done[a.slot]));
          if (st == n_stages - 1) tc_commit(smem_u32(&bars->acc_full));
        }
        __syncwarp();
        a.advance(kAStages);
        b.advance(p.b_stages);
      }
    }
  } else if (warp >= 4 && warp < kEpiWarp0) {
    // ------------------------------ dequant --------------------------------
    // Warp (q, h): TMEM lane quarter q; set h takes every kDequantSets-th stage of the
    // running stage sequence. A stage is decoded 64 K-elements (32 columns) at a time:
    // two 16-byte chunks of the thread's row -> 32 registers -> one tcgen05.st.
    // With 64-K stages the store of a stage stays in flight while the warp's next
    // stage is decoded; longer stages overlap their own pieces instead.
    const int q = warp & 3, h = (warp - 4) >> 2;
    const int row = q * 32 + lane;                 // TMEM lane of this thread
    // gate/up items interleave the two halves in groups of 16 lanes: lanes 0-7 of a group hold
    // the gate rows of eight features, lanes 8-15 the matching up rows, so a 16x256b read of
    // the accumulator hands one thread the gate and the up value of the same (feature, token).
    const int srow = GATEUP ? (((row >> 3) & 1) * 64 + (row >> 4) * 8 + (row & 7)) : row;   // row inside the staged tile
    const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + kAccCols;
    const uint32_t lut_lane = smem_u32(lut) + (uint32_t)lane * 4u;
    Ring w, a;
    uint32_t sc_it = 0;
    int turn = 0;   // which dequant set takes the coming stage, running over all items
    int pending = -1;   // A slot whose stores are not yet handed to the MMA issuer
    bool ok = true;
    auto retire = [&]() {
      if (pending >= 0) {
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (CTAS == 2 && !leader) mbar_arrive_cta(smem_u32(&bars->a_full[pending]), 0);
          else mbar_arrive(smem_u32(&bars->a_full[pending]));
        }
        pending = -1;
      }
    };
    for (int item = unit; item < n_items && ok; item += n_units) {
      const int f = item_f(item);
      const int rows_valid = f >= p.n_ftiles ? 0 : (GATEUP ? 128 : min(128, p.n_feat - f * 128));
      const int sbuf = sc_it % p.scale_bufs;
      if (!mbar_wait(smem_u32(&bars->sc_full[sbuf]), (sc_it / p.scale_bufs) & 1u, abort_flag, 7)) {
        ok = false;
        break;
      }
      const uint8_t* my_scales = sc_smem + sbuf * p.scale_buf_bytes + srow * pitch;
      for (int kw = 0; kw < n_kw && ok; ++kw) {
        if (!mbar_wait(smem_u32(&bars->w_full[w.slot]), w.phase, abort_flag, 8)) {
          ok = false;
          break;
        }
        const uint8_t* my_row = w_smem + w.slot * kWStageBytes + (srow >> 6) * (kWStageBytes / 2) +
                                (srow & 63) * 128;
        const int k_left = p.K - kw * kWStageK;                       // K elements from this W stage on
        const int n_sub = min(kSubPerW, (k_left + KS - 1) / KS);      // pipeline stages in this W stage
        for (int j = 0; j < n_sub; ++j, turn = (turn + 1 == kDequantSets ? 0 : turn + 1), a.advance(kAStages)) {
          if (turn != h) continue;
          if (!mbar_wait(smem_u32(&bars->stage_done[a.slot]), a.phase ^ 1u, abort_flag, 9)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const int n_pieces = min(kPieces, (k_left - j * KS) / 64);
#pragma unroll
          for (int pc = 0; pc < kPieces; ++pc) {
            if (pc < n_pieces) {
              uint32_t v[32];
              if (srow < rows_valid) {
                const int c0 = (j * kPieces + pc) * 2;   // two 16-byte chunks = two scale groups
                const uint4 p0 = *reinterpret_cast<const uint4*>(my_row + (((c0) ^ (srow & 7)) << 4));
                const uint4 p1 = *reinterpret_cast<const uint4*>(my_row + (((c0 + 1) ^ (srow & 7)) << 4));
                const uint32_t s0 = ue8m0_to_bf16x2(my_scales[kw * 8 + c0]);
                const uint32_t s1 = ue8m0_to_bf16x2(my_scales[kw * 8 + c0 + 1]);
                if (kUseLut) {
                  dequant64_lut(p0, p1, s0, s1, lut_lane, v);
                } else {
                  dequant8(p0.x, s0, v + 0);
                  dequant8(p0.y, s0, v + 4);
                  dequant8(p0.z, s0, v + 8);
                  dequant8(p0.w, s0, v + 12);
                  dequant8(p1.x, s1, v + 16);
                  dequant8(p1.y, s1, v + 20);
                  dequant8(p1.z, s1, v + 24);
                  dequant8(p1.w, s1, v + 28);
                }
              } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = 0u;
              }
              if (KS == 64) retire();   // previous stage of this warp: its store had a stage time to land
              tc_st32(t_row + a.slot * kACols + pc * 32, v);
            }
          }
          pending = a.slot;
          if (KS != 64) retire();
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bars->w_empty[w.slot]));
        w.advance(p.w_stages);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bars->sc_empty[sbuf]));
      ++sc_it;
    }
    retire();
  } else if (warp >= kEpiWarp0) {
    // ------------------------------ epilogue -------------------------------
    // Two sets of four warps (one per lane quarter): the gate/up rounds of 32 tokens alternate
    // between them, and so do the rounds of the down epilogue, which halves the time the MMA
    // issuer waits for the accumulator.
    const int q = warp & 3;
    const int es = (warp - kEpiWarp0) >> 2;          // epilogue set
    const int etid = tid - kEpiWarp0 * 32;           // 0 .. 128 * kEpiSets - 1
    const int ltid = etid & 127;                     // thread inside the set = TMEM lane
    uint32_t acc_phase = 0u;
    int round = 0;   // gate/up staging buffer parity of this set, running over all items
    for (int item = unit; item < n_items; item += n_units) {
      const TokTile tt = p.tiles[item / n_fgroups];
      const int f = item_f(item);
      // per-token info of this item (previous item's readers are past the barrier below)
      named_bar_sync(1, 128 * kEpiSets);
      for (int j = etid; j < tt.n_rows; j += 128 * kEpiSets) {
        const int flat = p.sorted_ids[tt.row0 + j];
        const bool real = flat >= 0 && flat < p.N;
        if (GATEUP) {
          bars->tile_ref[j] = real ? 1ull : 0ull;
        } else {
          const int token = real ? flat / p.top_k : 0;
          float* orow = p.out_rows ? p.out_rows[token] : p.out + (size_t)token * p.n_feat;
          if (p.store_rows && real) orow += (size_t)(flat - token * p.top_k) * p.n_feat;
          bars->tile_ref[j] = real ? reinterpret_cast<unsigned long long>(orow) : 0ull;
        }
        if (!GATEUP) bars->tile_w[j] = (real && p.topk_w != nullptr) ? p.topk_w[p.w_sorted ? tt.row0 + j : flat] : 0.0f;
      }
      // The wait's outcome is shared by all epilogue warps before anyone acts on it: a warp that
      // gave up must not leave the others standing at a later named barrier.
      const bool gave_up = !mbar_wait(smem_u32(&bars->acc_full), acc_phase, abort_flag, 10, 256);
      acc_phase ^= 1u;
      if (named_bar_or(1, 128 * kEpiSets, gave_up)) break;
      tc_fence_after();
      const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16);
      auto release_acc = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (CTAS == 2 && !leader) mbar_arrive_cta(smem_u32(&bars->acc_empty), 0);
          else mbar_arrive(smem_u32(&bars->acc_empty));
        }
      };
      if (f >= p.n_ftiles || es * 32 >= tt.n_rows || (!GATEUP && (p.n_feat & 3) != 0 && es != 0)) {
        release_acc();   // idle half of the last pair, or a set with no round in this item
        continue;
      }
      if (GATEUP) {
        // Per 32 token columns the warp reads its two 16-lane groups in the 16x256b shape:
        // a thread then holds gate and up of (feature lane / 4 [+ 8], tokens 8i + 2 * (lane % 4)
        // and the next one), so the activation needs no exchange between lanes.
        const bool situ = p.activation == 1;   // uniform across the launch
        const float clamp = p.limit > 0.0f ? p.limit : INFINITY;
        const int fl = q * 16 + (lane >> 2);   // feature inside the item's 64, first lane group
        const int tk = (lane & 3) * 2;
        float bg[2] = {0.f, 0.f}, bu[2] = {0.f, 0.f};
        if (p.bias) {
          const float* bp = p.bias + (size_t)tt.expert * 2 * p.n_feat + f * 64 + fl;
          bg[0] = bp[0]; bg[1] = bp[8]; bu[0] = bp[p.n_feat]; bu[1] = bp[p.n_feat + 8];
        }
        uint16_t* const my_stage = epi_stage + es * (2 * 32 * kEpiPitch);
        for (int c0 = es * 32; c0 < tt.n_rows; c0 += 32 * kEpiSets, ++round) {
          uint32_t va[16], vb[16];
          tc_ld_16x256b_x4(t_lane + c0, va);
          tc_ld_16x256b_x4(t_lane + (16u << 16) + c0, vb);
          tc_wait_ld();
          if (c0 + 32 * kEpiSets >= tt.n_rows) release_acc();   // this warp's last read of the accumulator
          if (p.raw != nullptr) {   // stage split: pre-activation sums, gate columns then up columns
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const int t = c0 + 8 * i + tk + e;
                if (t < tt.n_rows) {
                  float* d = p.raw + (size_t)(tt.row0 + t) * p.raw_ld + f * 64 + fl;
                  d[0] = __uint_as_float(va[4 * i + e]);
                  d[p.n_feat] = __uint_as_float(va[4 * i + 2 + e]);
                  d[8] = __uint_as_float(vb[4 * i + e]);
                  d[p.n_feat + 8] = __uint_as_float(vb[4 * i + 2 + e]);
                }
              }
            }
            continue;
          }
          // which of the round's 32 tokens are real rows: one shared-memory read per lane and
          // a ballot, so the stores below depend on no load
          const int my_t = c0 + lane;
          const unsigned real = __ballot_sync(0xFFFFFFFFu, my_t < tt.n_rows && bars->tile_ref[my_t] != 0ull);
          // activation -> bf16 into the staging tile [token][feature] of this round ... (one straight line of sixteen
          // independent elements: a warp alone on its scheduler's slot is bound by their latency)
          uint16_t* stg = my_stage + (round & 1) * (32 * kEpiPitch) + tk * kEpiPitch + fl;
          uint16_t act[4][2][2];
          if (!situ) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                act[i][e][0] = f32_to_bf16_bits(swiglu_fast(__uint_as_float(va[4 * i + e]) + bg[0], __uint_as_float(va[4 * i + 2 + e]) + bu[0], clamp));
                act[i][e][1] = f32_to_bf16_bits(swiglu_fast(__uint_as_float(vb[4 * i + e]) + bg[1], __uint_as_float(vb[4 * i + 2 + e]) + bu[1], clamp));
              }
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                act[i][e][0] = f32_to_bf16_bits(moe_act_value(1, __uint_as_float(va[4 * i + e]) + bg[0], __uint_as_float(va[4 * i + 2 + e]) + bu[0],
                                                              p.limit, p.beta, p.linear_beta));
                act[i][e][1] = f32_to_bf16_bits(moe_act_value(1, __uint_as_float(vb[4 * i + e]) + bg[1], __uint_as_float(vb[4 * i + 2 + e]) + bu[1],
                                                              p.limit, p.beta, p.linear_beta));
              }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              stg[(8 * i + e) * kEpiPitch] = act[i][e][0];
              stg[(8 * i + e) * kEpiPitch + 8] = act[i][e][1];
            }
          // ... then rows leave as 16-byte pieces: 8 consecutive threads write one 128-byte act row.
          // One barrier per round: a buffer is rewritten two rounds later, after the barrier of
          // the round in between, which every reader of this round has passed by then.
          named_bar_sync(2 + es, 128);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int piece = ltid + i * 128;           // 256 pieces of 16 bytes
            const int tok = piece >> 3, ch = piece & 7;
            if ((real >> tok) & 1u) {
              const uint4 val = *reinterpret_cast<const uint4*>(my_stage + (round & 1) * (32 * kEpiPitch) + tok * kEpiPitch + ch * 8);
              *reinterpret_cast<uint4*>(p.act + (size_t)(tt.row0 + c0 + tok) * p.n_feat + f * 64 + ch * 8) = val;
            }
          }
        }
      } else {
        const int rows_valid = min(128, p.n_feat - f * 128);
        if ((p.n_feat & 3) == 0) {
          // 16-byte reductions: the warp turns its 32 rows x 32 tokens block around through
          // shared memory, so a lane holds four consecutive output features of one token and
          // adds them with one red.v4 (a quarter of the reduction instructions, which are what
          // this epilogue is bound by). Lane l: features 4 * (l % 8).., tokens l / 8 + 4 * i.
          // The two warp sets take the 32-token rounds in turn; a warp's block is 16 tokens wide,
          // so a round goes through it in two halves.
          float* stage = reinterpret_cast<float*>(epi_stage) + (es * 4 + q) * (16 * 32);
          const int hq = (lane & 7) * 4;                 // feature quad inside the warp's 32 rows
          const int h0 = f * 128 + q * 32 + hq;
          const bool quad_ok = q * 32 + hq < rows_valid;
          float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
          if (p.bias && quad_ok) b4 = *reinterpret_cast<const float4*>(p.bias + (size_t)tt.expert * p.n_feat + h0);
          for (int c0 = es * 32; c0 < tt.n_rows; c0 += 32 * kEpiSets) {
            uint32_t v[32];
            tc_ld32(t_lane + c0, v);
            tc_wait_ld();
            if (c0 + 32 * kEpiSets >= tt.n_rows) release_acc();   // this warp's last read of the accumulator
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              // this lane's four tokens of the half, looked up before the block turns around
              unsigned long long ref[4];
              float wgt[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int t = c0 + half * 16 + (lane >> 3) + 4 * i;
                const bool in = t < tt.n_rows && quad_ok;
                ref[i] = in ? (p.raw != nullptr ? 1ull : bars->tile_ref[t]) : 0ull;
                wgt[i] = in ? bars->tile_w[t] : 0.0f;
              }
              __syncwarp();   // the previous block has been read
#pragma unroll
              for (int j = 0; j < 16; ++j) stage[j * 32 + lane] = __uint_as_float(v[half * 16 + j]);
              __syncwarp();
              float4 a[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                a[i] = *reinterpret_cast<const float4*>(stage + ((lane >> 3) + 4 * i) * 32 + hq);
                // plain rows leave as they are: whoever combines them (combine_rows_kernel, the ranks' reduction) adds the bias
                if (p.raw == nullptr) { a[i].x += b4.x; a[i].y += b4.y; a[i].z += b4.z; a[i].w += b4.w; }
              }
              if (p.raw != nullptr) {   // plain partial rows, no bias, no routing weight
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  if (ref[i] != 0ull)
                    *reinterpret_cast<float4*>(p.raw + (size_t)(tt.row0 + c0 + half * 16 + (lane >> 3) + 4 * i) * p.raw_ld + h0) = a[i];
              } else if (p.store_rows) {   // plain 16-byte store of the slot's row; the home rank adds its slots in order
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  if (ref[i] != 0ull) *reinterpret_cast<float4*>(reinterpret_cast<float*>(ref[i]) + h0) = a[i];
              } else if (p.out_rows != nullptr) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  if (ref[i] != 0ull)
                    red_add_v4_sys(reinterpret_cast<float*>(ref[i]) + h0, a[i].x * wgt[i], a[i].y * wgt[i], a[i].z * wgt[i], a[i].w * wgt[i]);
              } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                  if (ref[i] != 0ull)
                    red_add_v4(reinterpret_cast<float*>(ref[i]) + h0, a[i].x * wgt[i], a[i].y * wgt[i], a[i].z * wgt[i], a[i].w * wgt[i]);
              }
            }
          }
        } else {
          const int hcol = f * 128 + etid;
          const bool row_ok = etid < rows_valid;
          const float b = (p.bias && row_ok) ? p.bias[(size_t)tt.expert * p.n_feat + hcol] : 0.0f;
          for (int c0 = 0; c0 < tt.n_rows; c0 += 32) {
            uint32_t v[32];
            tc_ld32(t_lane + c0, v);
            tc_wait_ld();
            if (c0 + 32 >= tt.n_rows) release_acc();
#pragma unroll 4
            for (int j = 0; j < 32; ++j) {
              const int t = c0 + j;
              float* orow = t < tt.n_rows ? reinterpret_cast<float*>(bars->tile_ref[t]) : nullptr;
              if (orow != nullptr && row_ok)
                atomicAdd(orow + hcol, (__uint_as_float(v[j]) + b) * bars->tile_w[t]);
            }
          }
        }
      }
    }
  }

  // ------------------------------ teardown ---------------------------------
  tc_fence_before();
  __syncthreads();
  if (CTAS == 2) cluster_sync_all();   // the peer no longer touches this CTA's barriers or tensor memory
  if (warp == 1) {
    tc_fence_after();
    if (CTAS == 2)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                   "r"((uint32_t)kTmemCols)
                   : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                   "r"((uint32_t)kTmemCols)
                   : "memory");
  }
  if (tid == 0 && bars->abort_flag != 0) atomicExch(&g_kernel_status, 100 + bars->abort_flag);
}

// One warp waits, with the kernels' own bounded wait, on a barrier nobody arrives on, and
// reports the expiry through the status word like a GEMM kernel would: the way to exercise the
// give-up path without starving a real launch.
__global__ void wait_timeout_probe_kernel(long long limit_clocks) {
  __shared__ uint64_t bar;
  __shared__ int abort_flag;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar), 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  if (threadIdx.x == 0) {
    const bool ok = mbar_wait(smem_u32(&bar), 0, &abort_flag, 99, 0, limit_clocks);
    if (!ok) atomicExch(&g_kernel_status, 100 + abort_flag);
  }
}

// ---------------------------------------------------------------------------
// pre-pass kernels
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(1024)
build_tiles_kernel(const int32_t* __restrict__ expert_ids, int n_blocks, int block_size, int max_tok,
                   TokTile* __restrict__ tiles, int* __restrict__ n_tiles, int max_tiles) {
  __shared__ int warp_sums[32];
  build_tiles_block<1024>(expert_ids, n_blocks, block_size, max_tok, tiles, n_tiles, max_tiles, warp_sums);
}

// A_sorted[r, :] = A[sorted_ids[r] / top_k, :] (or the row at A_rows[sorted_ids[r] / top_k]) for real rows; padding rows
// become zeros if `zero_pad` (the plain-result GEMM writes its results for them) and are left alone otherwise: a padding
// column's results are never read. A warp per row with four 16-byte vectors a lane in flight: the copy is bound by the
// bytes in flight (8192 tokens x 4 x 5760 bytes: 104 us with one vector a thread in flight, 256 threads a row). CTA 0
// builds the token-tile list instead (tiles != nullptr), so that the list costs no launch of its own and is ready
// when the rows are.
constexpr int kGatherWarps = 8;
__global__ void __launch_bounds__(32 * kGatherWarps)
gather_rows_kernel(const uint16_t* __restrict__ A, const uint16_t* const* __restrict__ A_rows,
                   const int32_t* __restrict__ sorted_ids,
                   const int32_t* __restrict__ expert_ids, int block_size, int EM, int N, int top_k,
                   int H, uint16_t* __restrict__ dst, int32_t* __restrict__ inv, int zero_pad, int max_tok,
                   TokTile* __restrict__ tiles, int* __restrict__ n_tiles, int max_tiles) {
  if (blockIdx.x == 0) {
    __shared__ int warp_sums[kGatherWarps];
    if (tiles != nullptr)
      build_tiles_block<32 * kGatherWarps>(expert_ids, EM / block_size, block_size, max_tok, tiles, n_tiles, max_tiles, warp_sums);
    return;
  }
  const int lane = threadIdx.x & 31;
  const int r = ((int)blockIdx.x - 1) * kGatherWarps + (threadIdx.x >> 5);
  if (r >= EM) return;
  if (expert_ids[r / block_size] < 0) return;  // never read by any tile
  const int flat = sorted_ids[r];
  const bool real = flat >= 0 && flat < N;
  if (!real && zero_pad == 0) return;
  const int token = real ? flat / top_k : 0;
  if (real && inv != nullptr && lane == 0) inv[flat] = r;
  // a row address from A_rows may lie in another GPU's memory (peer load over NVLink)
  const uint4* src = reinterpret_cast<const uint4*>(
      A_rows != nullptr ? (real ? A_rows[token] : nullptr) : A + (size_t)token * H);
  uint4* d = reinterpret_cast<uint4*>(dst + (size_t)r * H);
  const int n_vec = H / 8;  // 16-byte vectors
  constexpr int kFlight = 4;
  for (int i0 = lane; i0 < n_vec; i0 += 32 * kFlight) {
    uint4 v[kFlight];
#pragma unroll
    for (int j = 0; j < kFlight; ++j)
      v[j] = real && i0 + 32 * j < n_vec ? src[i0 + 32 * j] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int j = 0; j < kFlight; ++j)
      if (i0 + 32 * j < n_vec) d[i0 + 32 * j] = v[j];
  }
}

// Ordered combine: y[t, :] = bf16( sum over the token's routed slots, in ascending sorted-row
// order - for one token that is ascending expert order, the order in which the CPU definition
// adds (reference moe_fused.cpp:539-562) - of (partial[r, :] + b2[e, :]) * w ). No atomics: the
// result does not depend on which CTA finished first, and the fp32 accumulator never travels
// through memory. inv[flat] = sorted row of routed slot `flat`; an entry is trusted only if
// sorted_ids[inv[flat]] == flat (slots that were not routed leave stale entries behind).
// A CTA per token and 1024 columns, a thread per four of them with the loads of up to eight slots in flight: with the
// whole row per CTA the kernel was a chain of loads (32 tokens x 9 slots x 7168: 21 us).
constexpr int kMaxCombineSlots = 32;
__global__ void __launch_bounds__(256)
combine_rows_kernel(const float* __restrict__ partial, const float* __restrict__ b2, const float* __restrict__ topk_w,
                    int w_sorted, const int32_t* __restrict__ sorted_ids, const int32_t* __restrict__ expert_ids,
                    const int32_t* __restrict__ inv, int block_size, int EM, int top_k, int H,
                    uint16_t* __restrict__ y_bf16, float* __restrict__ out_f32) {
  __shared__ int s_row[kMaxCombineSlots];
  __shared__ int s_exp[kMaxCombineSlots];
  __shared__ float s_w[kMaxCombineSlots];
  __shared__ int s_n;
  const int t = blockIdx.x;
  if (threadIdx.x < 32) {
    // lane j looks slot j up (three dependent loads, all slots at once); a valid slot's place in
    // the order is the number of valid slots on smaller rows
    const int j = threadIdx.x;
    int r = -1, e = -1;
    float w = 0.0f;
    if (j < top_k) {
      const int flat = t * top_k + j;
      const int cand = inv[flat];
      if (cand >= 0 && cand < EM && sorted_ids[cand] == flat) {
        e = expert_ids[cand / block_size];
        if (e >= 0) {
          r = cand;
          w = topk_w[w_sorted ? cand : flat];
        }
      }
    }
    const unsigned valid = __ballot_sync(0xFFFFFFFFu, r >= 0);
    int rank = 0;
    for (int o = 0; o < top_k; ++o) {
      const int ro = __shfl_sync(0xFFFFFFFFu, r, o);
      if (ro >= 0 && ro < r) ++rank;
    }
    if (r >= 0) {
      s_row[rank] = r;
      s_exp[rank] = e;
      s_w[rank] = w;
    }
    if (j == 0) s_n = __popc(valid);
  }
  __syncthreads();
  const int n = s_n;
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
  if (c < H) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    constexpr int kFlight = 8;
    for (int i0 = 0; i0 < n; i0 += kFlight) {
      float4 v[kFlight];
#pragma unroll
      for (int j = 0; j < kFlight; ++j)
        v[j] = i0 + j < n ? *reinterpret_cast<const float4*>(partial + (size_t)s_row[i0 + j] * H + c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int j = 0; j < kFlight; ++j) {
        if (i0 + j >= n) break;
        if (b2 != nullptr) {
          const float4 b = *reinterpret_cast<const float4*>(b2 + (size_t)s_exp[i0 + j] * H + c);
          v[j].x += b.x; v[j].y += b.y; v[j].z += b.z; v[j].w += b.w;
        }
        const float w = s_w[i0 + j];
        acc.x += v[j].x * w; acc.y += v[j].y * w; acc.z += v[j].z * w; acc.w += v[j].w * w;
      }
    }
    if (out_f32 != nullptr) *reinterpret_cast<float4*>(out_f32 + (size_t)t * H + c) = acc;
    if (y_bf16 != nullptr) {
      uint2 o;
      o.x = (uint32_t)f32_to_bf16_bits(acc.x) | ((uint32_t)f32_to_bf16_bits(acc.y) << 16);
      o.y = (uint32_t)f32_to_bf16_bits(acc.z) | ((uint32_t)f32_to_bf16_bits(acc.w) << 16);
      *reinterpret_cast<uint2*>(y_bf16 + (size_t)t * H + c) = o;
    }
  }
}

// ---------------------------------------------------------------------------
// prepack: checkpoint-layout MXFP4 -> the form the prepacked fp4 GEMM (moe_gemm_fp4.cu) reads
// ---------------------------------------------------------------------------
// Codes. The layer's table {0, .25, 1, 1.5, 2, 3} (magnitude codes 0..5) times two is
// {0, .5, 2, 3, 4, 6}: e2m1 codes 0, 1, 4, 5, 6, 7 - every code from 2 on moves up by two. Codes
// 6 and 7 (inf, NaN in this layer) have no e2m1 counterpart: they are counted, and a caller
// that finds a non-zero count keeps such weights on the checkpoint-layout path. A group whose
// scale byte is 0xFF (zero weights in this layer, NaN to the tensor core) becomes zero codes.
// One thread per 32-element group (16 bytes).
__global__ void prepack_codes_kernel(const uint4* __restrict__ w, const uint8_t* __restrict__ scale, long long n_groups,
                                     uint4* __restrict__ out, int* __restrict__ nonfinite) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n_groups) return;
  uint4 v = w[g];
  uint32_t x[4] = {v.x, v.y, v.z, v.w}, bad = 0u;
  const bool zero = scale[g] == 0xFFu;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t b1 = x[i] >> 1, b2 = x[i] >> 2;
    bad |= b1 & b2 & 0x11111111u;
    x[i] = zero ? 0u : x[i] + (((b1 | b2) & 0x11111111u) << 1);
  }
  if (bad != 0u && !zero) atomicAdd(nonfinite, 1);
  out[g] = make_uint4(x[0], x[1], x[2], x[3]);
}

// Scale factors, regrouped per (expert, 128-row work item, 256-K stage) as [128 accumulator
// rows][8 groups] so that a stage's kilobyte is one contiguous copy; rows and groups past the
// end read as 1.0 (0x7F), and so does the 0xFF of a zeroed group. One thread per byte.
__global__ void prepack_scales_kernel(const uint8_t* __restrict__ scale, int gateup, int n_feat, int K, int n_ftiles,
                                      int n_kw, long long total, uint8_t* __restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int b = (int)(i & 7), L = (int)((i >> 3) & 127);
  long long r = i >> 10;
  const int kw = (int)(r % n_kw);  r /= n_kw;
  const int f = (int)(r % n_ftiles);
  const long long e = r / n_ftiles;
  const int kb = kw * 8 + b, pitch = K / 32;
  long long row = -1;
  if (gateup) {
    const int sr = ((L >> 3) & 1) * 64 + (L >> 4) * 8 + (L & 7);   // accumulator row -> staged row (gate rows, then up rows)
    row = e * 2 * n_feat + (sr < 64 ? f * 64 + sr : n_feat + f * 64 + sr - 64);
  } else if (f * 128 + L < n_feat) {
    row = e * n_feat + f * 128 + L;
  }
  uint8_t v = 0x7Fu;
  if (row >= 0 && kb < pitch) {
    v = scale[row * pitch + kb];
    if (v == 0xFFu) v = 0x7Fu;
  }
  out[i] = v;
}

// ---------------------------------------------------------------------------
// host side: tensor maps, workspace layout, launch
// ---------------------------------------------------------------------------
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                              CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);

EncodeFn get_encode_fn() {
  static EncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    VK_CUDA_CHECK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres));
    if (p == nullptr || qres != cudaDriverEntryPointSuccess)
      throw std::runtime_error("cuTensorMapEncodeTiled is not available from the driver");
    return reinterpret_cast<EncodeFn>(p);
  }();
  return fn;
}

// Row-major tensor of up to four dimensions, innermost first, 128-byte swizzle; zero fill outside. Encoded anew for every
// launch: an encode is arithmetic on the host and takes 0.05 us, and a list of encoded maps costs more than that to search as
// soon as the batch sizes of a server fill it (256 entries, 24 layers' weights, every call another size: 65 us of host time
// a call in the pair form with the list, 32 without; the same size again and again: 32 both).
CUtensorMap make_map_nd(const void* ptr, CUtensorMapDataType dt, int elem_bytes, int rank, const uint64_t* dims,
                        const uint64_t* strides, const uint32_t* box) {
  CUtensorMap m;
  cuuint64_t d[4], st[3];
  cuuint32_t bx[4], estr[4] = {1, 1, 1, 1};
  for (int i = 0; i < rank; ++i) {
    d[i] = dims[i];
    bx[i] = box[i];
    if (i + 1 < rank) st[i] = strides[i];
  }
  expects(box[0] * elem_bytes == 128, "tensor map: the box must be 128 bytes wide");
  const CUresult r = get_encode_fn()(&m, dt, (cuuint32_t)rank, const_cast<void*>(ptr), d, st, bx, estr,
                                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    throw std::runtime_error("cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
  return m;
}

CUtensorMap make_map(const void* ptr, CUtensorMapDataType dt, int elem_bytes, uint64_t inner,
                     uint64_t outer, uint64_t pitch_bytes, uint32_t box_inner, uint32_t box_outer) {
  const uint64_t dims[2] = {inner, outer}, strides[1] = {pitch_bytes};
  const uint32_t box[2] = {box_inner, box_outer};
  return make_map_nd(ptr, dt, elem_bytes, 2, dims, strides, box);
}

// Token operand: bf16 rows [EM, K], K a multiple of 64.
TokMaps token_maps(const void* rows, int K, int EM, bool pair) {
  TokMaps t{};
  if (pair) {
    const uint64_t dims[3] = {64, (uint64_t)EM, (uint64_t)K / 64}, strides[2] = {(uint64_t)K * 2, 128};
    for (uint32_t i = 0; i < 8; ++i) {
      const uint32_t box[3] = {64, 16 * (i + 1), 2};
      t.m[i] = make_map_nd(rows, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, 3, dims, strides, box);
    }
  } else {
    t.m[0] = make_map(rows, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, K, EM, (uint64_t)K * 2, 64, 16);
    t.m[1] = make_map(rows, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, K, EM, (uint64_t)K * 2, 64, 64);
  }
  return t;
}

int max_tok_tiles(int EM) { return EM / 16 + 1; }

// Scratch of one layer call. bf16 forms: the gathered rows [EM, hidden] bf16. fp4 form: the six digit planes of the token rows
// [6][EM, hidden / 2] and of the activation rows [6][EM, ispp / 2], one fp32 scale per row each. The token planes are dead when
// the activation planes are written (the gate/up GEMM lies between them on the stream), so the two share their place -
// or, in the ordered form, the token planes lie where the down GEMM puts its partial rows later.
// ordered = the bf16-output form: + the inverse permutation [N] and the fp32 partial rows [EM, hidden] of the down GEMM.
struct WsLayout {
  size_t tiles_off, count_off, rows_off, act4_off, scale_x_off, scale_a_off, inv_off, partial_off, total;
};
WsLayout ws_layout(bool fp4, int EM, int hidden, int ispp, bool ordered = false, int N = 0) {
  WsLayout l{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = (off + bytes + 1023) & ~size_t(1023);
    return at;
  };
  l.count_off = off;  off += 256;
  l.tiles_off = take((size_t)max_tok_tiles(EM) * sizeof(TokTile));
  if (ordered) {
    l.inv_off = take((size_t)N * sizeof(int32_t));
    l.partial_off = take((size_t)EM * hidden * sizeof(float));
  }
  const size_t x4 = (size_t)EM * hidden * 3, a4 = (size_t)EM * ispp * 3;
  if (!fp4) {
    l.rows_off = take((size_t)EM * hidden * sizeof(uint16_t));
  } else {
    l.scale_x_off = take((size_t)EM * sizeof(float));
    l.scale_a_off = take((size_t)EM * sizeof(float));
    l.rows_off = ordered ? l.partial_off : off;
    l.act4_off = take(ordered ? a4 : std::max(x4, a4));
  }
  l.total = off;
  return l;
}


// Small token tiles (up to 64 rows) run the fp4 form (moe_gemm_fp4.cu); VK_MOE_SMALL=bf16 keeps them on the bf16
// table form (which also propagates an infinite activation as inf rather than NaN).
bool small_fp4_mode() {
  static const bool on = [] {
    const char* e = std::getenv("VK_MOE_SMALL");
    return e == nullptr || std::string(e) != "bf16";
  }();
  return on;
}

// Large token tiles run on CTA pairs; VK_MOE_PAIR=0 keeps every launch on single CTAs.
bool pair_mode() {
  static const bool on = [] {
    const char* e = std::getenv("VK_MOE_PAIR");
    return e == nullptr || std::atoi(e) != 0;
  }();
  return on;
}

// Whether the CTA-pair form fits shared memory: one token slot per A slot, one scale buffer,
// at least two packed-weight stages.
bool pair_fits(const GemmParams& p, bool gateup) {
  const int scale_tile = (128 * (p.K / 32) + 127) & ~127;
  const int fixed = 1024 + (((int)sizeof(Barriers) + 127) & ~127) + epi_stage_bytes(gateup, 2) + 128;
  const int tokens = 6 * (((p.max_tok + 31) >> 5) << 4) * 128;   // 6 x 64-K or 3 x 128-K slots
  return 227 * 1024 - fixed - scale_tile - tokens >= 2 * kWStageBytes;
}

template <bool GATEUP, int KS, int CTAS>
void launch_gemm_ks(const CUtensorMap& tw, const TokMaps& tb, GemmParams p,
                    cudaStream_t stream) {
  // Shared memory: token stages (this CTA's rows x KS), scales (double-buffered when they fit),
  // barriers, epilogue staging; what is left becomes the packed-weight ring (3..8 stages of
  // 16 KB): the deeper it is, the more weight bytes are in flight, which is what a decode-size
  // batch is bound by.
  constexpr int kAccCols = acc_cols(KS, CTAS);
  constexpr int kAStages = (kTmemCols - kAccCols) / (KS / 2);
  constexpr int kThreads = block_threads(CTAS);
  const int max_smem = 227 * 1024;
  const int scale_tile = (128 * (p.K / 32) + 127) & ~127;
  const int fixed = 1024 + (((int)sizeof(Barriers) + 127) & ~127) + epi_stage_bytes(GATEUP, CTAS) + 128 +
                    (CTAS == 1 ? kLutBytes : 0);
  // a pair's MMA N is the tile rounded up to 32 rows, half of them staged by each CTA
  p.b_stage_bytes = (CTAS == 2 ? (((p.max_tok + 31) >> 5) << 4) : p.max_tok) * 128 * (KS / 64);
  // token ring: 4 slots for a lone CTA; a pair has one token slot per A slot
  int b_stages = CTAS == 2 ? kAStages : (kAStages < 4 ? kAStages : 4), scale_bufs = 2;
  auto w_room = [&]() {
    return (max_smem - fixed - scale_bufs * scale_tile - b_stages * p.b_stage_bytes) / kWStageBytes;
  };
  if (w_room() < 4) scale_bufs = 1;
  while (CTAS == 1 && w_room() < 3 && b_stages > 2) --b_stages;
  expects(w_room() >= 2, "fused_moe_mxfp4: reduction dimension too large for shared memory");
  p.w_stages = w_room() > kMaxWStages ? kMaxWStages : w_room();
  if (CTAS == 1 && p.w_stages == kMaxWStages) {   // spare room: deepen the token ring
    const int keep_w = kMaxWStages;
    while (b_stages < kAStages && b_stages < kMaxBStages &&
           (max_smem - fixed - scale_bufs * scale_tile - (b_stages + 1) * p.b_stage_bytes) / kWStageBytes >= keep_w)
      ++b_stages;
    p.w_stages = w_room() > kMaxWStages ? kMaxWStages : w_room();
  }
  p.b_stages = b_stages;
  p.scale_bufs = scale_bufs;
  p.scale_buf_bytes = scale_tile;
  const int smem = fixed + scale_bufs * scale_tile + b_stages * p.b_stage_bytes + p.w_stages * kWStageBytes;
  // the attribute belongs to the device's context: once per device and instantiation
  static std::atomic<bool> configured[64];
  int dev = 0;
  VK_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev].load()) {
    VK_CUDA_CHECK(cudaFuncSetAttribute(moe_gemm_sm100_kernel<GATEUP, KS, CTAS>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
    if (dev >= 0 && dev < 64) configured[dev].store(true);
  }
  if (CTAS == 1) {
    moe_gemm_sm100_kernel<GATEUP, KS, CTAS><<<sm_count(), kThreads, smem, stream>>>(tw, tb, p);
  } else {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(sm_count() & ~1));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    VK_CUDA_CHECK(cudaLaunchKernelEx(&cfg, moe_gemm_sm100_kernel<GATEUP, KS, CTAS>, tw, tb, p));
  }
}

// Stage length and CTA grouping by the largest token tile of the launch (see the kernel's comment; choose_tiles makes none of
// 65 to 128 tokens).
template <bool GATEUP>
void launch_gemm(const CUtensorMap& tw, const TokMaps& tb, GemmParams p,
                 bool use_pair, cudaStream_t stream) {
  if (p.max_tok <= 64) launch_gemm_ks<GATEUP, 256, 1>(tw, tb, p, stream);
  else if (use_pair) launch_gemm_ks<GATEUP, 128, 2>(tw, tb, p, stream);
  else launch_gemm_ks<GATEUP, 64, 1>(tw, tb, p, stream);
}

}  // namespace

// What a call on EM sorted rows may take, whichever form it runs.
size_t sm100_workspace_bytes(int EM, int hidden, int ispp) {
  return std::max(ws_layout(false, EM, hidden, ispp).total, ws_layout(true, EM, hidden, ispp).total);
}
size_t sm100_workspace_bytes_ordered(int EM, int hidden, int ispp, int N) {
  return std::max(ws_layout(false, EM, hidden, ispp, true, N).total, ws_layout(true, EM, hidden, ispp, true, N).total);
}

// Sizes of the prepacked form of one weight set. which = 0: w13 [E, 2 * ispp, hidden / 2];
// 1: w2 [E, hidden, ispp / 2]. The code buffer carries 128 rows + 64 bytes of zero padding: a
// work item's box always spans 128 rows and a row's last 128-K box may reach past the row.
void prepack_sizes(int which, int E, int hidden, int ispp, size_t* w_bytes, size_t* sf_bytes) {
  expects(which == 0 || which == 1, "prepack: which must be 0 (w13) or 1 (w2)");
  expects(E > 0 && hidden > 0 && ispp > 0 && hidden % 64 == 0 && ispp % 64 == 0, "prepack: hidden and ispp must be multiples of 64");
  const long long rows = which == 0 ? 2ll * ispp : hidden;
  const int K = which == 0 ? hidden : ispp;
  const int n_ftiles = which == 0 ? ispp / 64 : (hidden + 127) / 128;
  const int n_kw = (K + kWStageK - 1) / kWStageK;
  if (w_bytes) *w_bytes = (size_t)(E * rows + 128) * (K / 2) + 256;
  if (sf_bytes) *sf_bytes = (size_t)E * n_ftiles * n_kw * kPackedSfBytes;
}

void prepack_weights(int which, const uint8_t* w, const uint8_t* scale, int E, int hidden, int ispp, uint8_t* w_out,
                     uint8_t* sf_out, int* nonfinite, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  size_t w_bytes = 0, sf_bytes = 0;
  prepack_sizes(which, E, hidden, ispp, &w_bytes, &sf_bytes);
  expects(w && scale && w_out && sf_out && nonfinite, "prepack: buffers must not be null");
  auto aligned = [](const void* p, unsigned a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; };
  expects(aligned(w, 16) && aligned(w_out, 32) && aligned(sf_out, 16), "prepack: w 16-byte, w_out 32-byte, sf_out 16-byte aligned");
  const long long rows = which == 0 ? 2ll * ispp : hidden;
  const int K = which == 0 ? hidden : ispp;
  const int n_feat = which == 0 ? ispp : hidden;
  const int n_ftiles = which == 0 ? ispp / 64 : (hidden + 127) / 128;
  const int n_kw = (K + kWStageK - 1) / kWStageK;
  const long long n_groups = (long long)E * rows * (K / 32);
  VK_CUDA_CHECK(cudaMemsetAsync(nonfinite, 0, sizeof(int), stream));
  VK_CUDA_CHECK(cudaMemsetAsync(w_out + (size_t)n_groups * 16, 0, w_bytes - (size_t)n_groups * 16, stream));
  prepack_codes_kernel<<<(unsigned)((n_groups + 255) / 256), 256, 0, stream>>>(
      reinterpret_cast<const uint4*>(w), scale, n_groups, reinterpret_cast<uint4*>(w_out), nonfinite);
  const long long total = (long long)sf_bytes;
  prepack_scales_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(scale, which == 0 ? 1 : 0, n_feat, K, n_ftiles,
                                                                           n_kw, total, sf_out);
  VK_CUDA_CHECK(cudaGetLastError());
}
// ---------------------------------------------------------------------------
// optional per-kernel timing: CUDA events recorded around the two GEMM kernels
// on the launch stream (no synchronisation while recording), summed on demand.
// The counterpart of the reference's VK_MOE_KTIME switch
// (src/c/vkernels/kernels/moe_fused.hip:1482-1493), without serialising stages.
// ---------------------------------------------------------------------------
namespace {
struct KernelTimer {
  bool on = false;
  std::vector<cudaEvent_t> ev;  // 3 per call: before gate/up, between, after down
  size_t used = 0;
} g_timer;
std::mutex g_timer_mu;
}  // namespace

void timing_begin(int max_calls) {
  std::lock_guard<std::mutex> lock(g_timer_mu);
  while (g_timer.ev.size() < (size_t)max_calls * 3) {
    cudaEvent_t e;
    VK_CUDA_CHECK(cudaEventCreate(&e));
    g_timer.ev.push_back(e);
  }
  g_timer.used = 0;
  g_timer.on = true;
}

void timing_end(float* gateup_ms, float* down_ms, int* calls) {
  std::lock_guard<std::mutex> lock(g_timer_mu);
  g_timer.on = false;
  float g = 0.f, d = 0.f;
  const size_t n = g_timer.used / 3;
  if (n > 0) VK_CUDA_CHECK(cudaEventSynchronize(g_timer.ev[n * 3 - 1]));
  for (size_t i = 0; i < n; ++i) {
    float a = 0.f, b = 0.f;
    VK_CUDA_CHECK(cudaEventElapsedTime(&a, g_timer.ev[3 * i], g_timer.ev[3 * i + 1]));
    VK_CUDA_CHECK(cudaEventElapsedTime(&b, g_timer.ev[3 * i + 1], g_timer.ev[3 * i + 2]));
    g += a;
    d += b;
  }
  if (gateup_ms) *gateup_ms = g;
  if (down_ms) *down_ms = d;
  if (calls) *calls = (int)n;
}

namespace {
// Records event `which` (0, 1, 2) of the current call when timing is on.
void timer_mark(int which, cudaStream_t stream) {
  if (!g_timer.on) return;
  std::lock_guard<std::mutex> lock(g_timer_mu);
  if (!g_timer.on) return;
  // used counts recorded events; a call's three events are consecutive
  if (g_timer.used % 3 != (size_t)which || g_timer.used >= g_timer.ev.size()) return;
  cudaEventRecord(g_timer.ev[g_timer.used], stream);
  g_timer.used += 1;
}
}  // namespace


// For the other tcgen05 kernel of the library (the router GEMM, moe_route.cu): a bf16 tensor map
// [outer, inner] with a byte pitch and a 128-byte-wide box, and the device address of the
// status word, so that its bounded waits report through the same word.
CUtensorMap sm100_make_map_bf16(const void* ptr, uint64_t inner, uint64_t outer, uint64_t pitch_bytes, uint32_t box_outer) {
  return make_map(ptr, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, inner, outer, pitch_bytes, 64, box_outer);
}
CUtensorMap sm100_make_map_u8(const void* ptr, int rank, const uint64_t* dims, const uint64_t* strides, const uint32_t* box) {
  return make_map_nd(ptr, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, rank, dims, strides, box);
}
int* sm100_status_address() {
  int* p = nullptr;
  VK_CUDA_CHECK(cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_kernel_status));
  return p;
}

// Status of the tcgen05 launches on the current device since the last reset: 0, or
// 100 + the code of the wait that ran out. Synchronises the device.
int sm100_last_status() {
  int v = 0;
  VK_CUDA_CHECK(cudaDeviceSynchronize());
  VK_CUDA_CHECK(cudaMemcpyFromSymbol(&v, g_kernel_status, sizeof(int)));
  return v;
}

// Clears the status word of the current device (after the failure has been dealt with).
void sm100_reset_status() {
  const int zero = 0;
  VK_CUDA_CHECK(cudaDeviceSynchronize());
  VK_CUDA_CHECK(cudaMemcpyToSymbol(g_kernel_status, &zero, sizeof(int)));
}

// Launches the one-warp probe whose bounded wait is certain to run out after `limit_clocks`.
void launch_wait_timeout_probe(long long limit_clocks, cudaStream_t stream) {
  expects(limit_clocks > 0 && limit_clocks <= 2000000000ll, "wait probe: limit must be in (0, 2e9] clocks");
  wait_timeout_probe_kernel<<<1, 32, 0, stream>>>(limit_clocks);
  VK_CUDA_CHECK(cudaGetLastError());
}


namespace {
// Largest token tile of a launch and whether the CTA-pair form runs it.
struct TileChoice {
  int max_tok;
  bool use_pair;
};
// The expert count is not an argument of the layer: callers size EM as N + E * (block - 1), which gives a lower bound of E
// (an exact EM only makes the estimate more conservative).
long long experts_estimate(int M, int top_k, int EM, int block_size) {
  return std::max<long long>(1, ((long long)EM - (long long)M * top_k) / (block_size - 1));
}
TileChoice choose_tiles(int M, int top_k, int EM, int block_size, int k_gateup, int k_down) {
  // A token meets an expert once as a rule, so an expert holds at most M rows (+ padding); one that holds more gets more tiles.
  int max_tok = ((M + block_size - 1) / block_size) * block_size;
  max_tok = ((max_tok + 15) / 16) * 16;
  // When an expert sees a few dozen tokens at most, tiles are capped at 64 rows so that the launch
  // takes the long-stage form built for small tiles (an expert with more rows is split into
  // several items); the crossover against the CTA-pair form, about 48 tokens per expert, was measured with the byte form that
  // ran small tiles before the fp4 form.
  {
    const long long n_slots = (long long)M * top_k;
    if ((M <= 256 || n_slots <= 48 * experts_estimate(M, top_k, EM, block_size)) && max_tok > 64) max_tok = 64;
  }
  // Tiles over 128 tokens go to CTA pairs when both GEMMs fit shared memory in that form.
  bool use_pair = false;
  if (max_tok > 128 && pair_mode()) {
    GemmParams probe{};
    probe.max_tok = max_tok > kPairMaxTok ? kPairMaxTok : ((max_tok + 31) & ~31);
    probe.K = k_gateup;
    use_pair = pair_fits(probe, true);
    probe.K = k_down;
    use_pair = use_pair && pair_fits(probe, false);
    if (use_pair) max_tok = probe.max_tok;   // a CTA pair stages half of the rows each
  }
  if (!use_pair && max_tok > kMaxTok) max_tok = kMaxTok;
  return TileChoice{max_tok, use_pair};
}

// moe_gemm_fp4.cu takes tiles of up to 32 tokens. Where an expert sees eight on average or fewer, tiles end at 16 (a few
// experts in a thousand hold more): the token slots are sized for the largest tile, and what they do not take holds weights -
// or, with a very long reduction, its scale bytes.
int fp4_tile_limit(int M, int top_k, int EM, int block_size, int max_k) {
  return M <= 16 || max_k > 32768 || (long long)M * top_k <= 8 * experts_estimate(M, top_k, EM, block_size) ? 16 : 32;
}

// The form of a layer call: fp4 (small tiles) or bf16 (lone CTAs or pairs), and the limit its tile list is built with.
struct Form {
  bool fp4, use_pair;
  int max_tok;
};
Form choose_form(int M, int top_k, int EM, int block_size, int hidden, int ispp, bool packed) {
  const TileChoice c = choose_tiles(M, top_k, EM, block_size, hidden, ispp);
  const bool fp4 = c.max_tok <= 64 && (small_fp4_mode() || packed);
  return Form{fp4, c.use_pair, fp4 ? fp4_tile_limit(M, top_k, EM, block_size, std::max(hidden, ispp)) : c.max_tok};
}
}  // namespace

// Scratch with which every layer call of up to max_tokens tokens fits whose EM is the host bound of its alignment
// (min(N, experts) experts with one row each, the other rows in one more), in the fp32 form and, up to ordered_tokens, in
// the ordered one.
size_t sm100_workspace_bytes_upto(int max_tokens, int top_k, int n_experts, int hidden, int ispp, int block_size,
                                  int ordered_tokens) {
  size_t most = 0;
  for (int M = 1; M <= max_tokens; ++M) {
    const long long N = (long long)M * top_k, head = std::min<long long>(N, n_experts);
    const int EM = (int)(head * block_size + (N - head + block_size - 1) / block_size * block_size);
    const bool fp4 = choose_form(M, top_k, EM, block_size, hidden, ispp, false).fp4;
    most = std::max(most, ws_layout(fp4, EM, hidden, ispp).total);
    if (M <= ordered_tokens) most = std::max(most, ws_layout(fp4, EM, hidden, ispp, true, (int)N).total);
    // (prepacked weights run the fp4 form even where VK_MOE_SMALL keeps the others off it)
    if (M <= ordered_tokens) most = std::max(most, ws_layout(true, EM, hidden, ispp, true, (int)N).total);
  }
  return most;
}

// Test hook: {whether the fp4 form runs, its tile limit, tokens that a slot of the gate/up and of the down GEMM holds}.
void sm100_test_form(int M, int top_k, int EM, int block_size, int hidden, int ispp, bool packed, int* out) {
  expects(M > 0 && top_k > 0 && EM > 0 && block_size >= 16 && block_size % 16 == 0 && out != nullptr, "test_form: bad arguments");
  const Form form = choose_form(M, top_k, EM, block_size, hidden, ispp, packed);
  out[0] = form.fp4 ? 1 : 0;
  out[1] = form.max_tok;
  out[2] = out[3] = 0;
  if (!form.fp4) return;
  out[2] = fp4_plan(packed, hidden, form.max_tok).b_stage_bytes / (6 * 128);
  out[3] = fp4_plan(packed, ispp, form.max_tok).b_stage_bytes / (6 * 128);
}

// moe_gemv.cu
bool moe_tiny_eligible(int M, int hidden, int ispp, int top_k);
void launch_moe_tiny(const uint16_t* A, const uint8_t* w13, const uint8_t* w13_scale, const uint8_t* w2,
                     const uint8_t* w2_scale, const float* topk_w, uint16_t* act, uint16_t* y, int M, int hidden, int ispp,
                     int top_k, const int32_t* sorted_ids, const int32_t* expert_ids, int EM, float swiglu_limit,
                     int activation, float beta, float linear_beta, const float* b13, const float* b2, int block_size,
                     int32_t* slot_expert, cudaStream_t stream);

void launch_moe_sm100(const uint16_t* A, const uint8_t* w13, const uint8_t* w13_scale,
                      const uint8_t* w2, const uint8_t* w2_scale, const float* topk_w,
                      int w_sorted, uint16_t* act_scratch, float* out, int M, int hidden, int ispp,
                      int top_k, const int32_t* sorted_ids, const int32_t* expert_ids, int EM,
                      float swiglu_limit, int activation, float beta, float linear_beta,
                      const float* b13, const float* b2, int block_size, cudaStream_t stream,
                      const RowPtrs* rows, uint16_t* y_bf16, bool w4) {
  const bool store_rows = rows != nullptr && rows->store_slots;
  auto aligned16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  const uint16_t* const* a_rows = rows ? rows->a_rows : nullptr;
  float* const* out_rows = rows ? rows->out_rows : nullptr;
  expects(aligned16(A) && aligned16(w13) && aligned16(w13_scale) && aligned16(w2) &&
              aligned16(w2_scale) && aligned16(act_scratch),
          "fused_moe_mxfp4: A, weights, scales and act_scratch must be 16-byte aligned");
  // y_bf16 != nullptr: the down GEMM leaves plain partial rows and an ordered combine writes the
  // bf16 result (no atomics, no fp32 output buffer to zero and convert)
  const bool ordered = y_bf16 != nullptr;
  const Form form = choose_form(M, top_k, EM, block_size, hidden, ispp, w4);
  const bool mx = form.fp4;
  expects(!w4 || mx, "fused_moe_mxfp4: prepacked weights serve decode-size batches only (token tiles of up to 64 rows); "
                     "larger batches take the checkpoint-layout weights");
  const WsLayout l = ws_layout(mx, EM, hidden, ispp, ordered, M * top_k);
  uint8_t* ws = static_cast<uint8_t*>(workspace_get(l.total, stream));
  TokTile* tiles = reinterpret_cast<TokTile*>(ws + l.tiles_off);
  int* n_tiles = reinterpret_cast<int*>(ws + l.count_off);
  uint16_t* gathered = reinterpret_cast<uint16_t*>(ws + l.rows_off);
  int32_t* inv = ordered ? reinterpret_cast<int32_t*>(ws + l.inv_off) : nullptr;
  float* partial = ordered ? reinterpret_cast<float*>(ws + l.partial_off) : nullptr;

  // One or two decode tokens: two flat kernels instead of the grouped GEMMs and their helpers.
  if (ordered && rows == nullptr && !w4 && w_sorted == 0 && moe_tiny_eligible(M, hidden, ispp, top_k)) {
    timer_mark(0, stream);
    launch_moe_tiny(A, w13, w13_scale, w2, w2_scale, topk_w, act_scratch, y_bf16, M, hidden, ispp, top_k, sorted_ids,
                    expert_ids, EM, swiglu_limit, activation, beta, linear_beta, b13, b2, block_size,
                    reinterpret_cast<int32_t*>(ws + l.count_off + 64), stream);
    timer_mark(1, stream);
    timer_mark(2, stream);
    return;
  }

  // The number of experts is not an argument of the layer; the tensor maps
  // cover the rows of every expert id that fits an int32 row index.
  const uint64_t w13_rows_cap = (uint64_t)1 << 31;
  const int max_tok = form.max_tok;
  const bool use_pair = form.use_pair;
  if (mx) {
    // Small tiles: the fp4 form. The tile list is built by an extra CTA of the row pre-pass.
    uint8_t* x4 = reinterpret_cast<uint8_t*>(gathered);   // digit planes of the token rows
    uint8_t* a4 = ws + l.act4_off;                        //              of the activation rows
    float* scale_x = reinterpret_cast<float*>(ws + l.scale_x_off);
    float* scale_a = reinterpret_cast<float*>(ws + l.scale_a_off);
    launch_digit_rows(true, A, a_rows, sorted_ids, expert_ids, block_size, EM, M * top_k, top_k, hidden, x4, scale_x, inv,
                      max_tok, tiles, n_tiles, max_tok_tiles(EM), stream);
    Fp4Params f{};
    f.sorted_ids = sorted_ids; f.tiles = tiles; f.n_tiles = n_tiles;
    f.N = M * top_k; f.top_k = top_k; f.w_sorted = w_sorted; f.activation = activation;
    f.limit = swiglu_limit; f.beta = beta; f.linear_beta = linear_beta; f.tile_tok = max_tok;
    Fp4Params p = f;
    p.w = w13; p.w_scale = w13_scale; p.x = A; p.x_rows = a_rows; p.tok_scale = scale_x; p.bias = b13; p.act = act_scratch;
    p.K = hidden; p.n_feat = ispp; p.n_ftiles = ispp / 64;
    timer_mark(0, stream);
    launch_gemm_fp4(true, w4, p, x4, EM, stream);
    timer_mark(1, stream);
    launch_digit_rows(false, act_scratch, nullptr, sorted_ids, expert_ids, block_size, EM, M * top_k, top_k, ispp, a4, scale_a,
                      nullptr, 0, nullptr, nullptr, 0, stream);
    p = f;
    p.w = w2; p.w_scale = w2_scale; p.x = act_scratch; p.tok_scale = scale_a; p.bias = b2; p.topk_w = topk_w; p.out = out;
    p.out_rows = out_rows; p.store_rows = store_rows ? 1 : 0; p.raw = partial;
    p.K = ispp; p.n_feat = hidden; p.n_ftiles = (hidden + 127) / 128;
    launch_gemm_fp4(false, w4, p, a4, EM, stream);
    timer_mark(2, stream);
    if (ordered)
      combine_rows_kernel<<<dim3((unsigned)M, (unsigned)((hidden + 1023) / 1024)), 256, 0, stream>>>(partial, b2, topk_w, w_sorted, sorted_ids, expert_ids, inv, block_size, EM,
                                                 top_k, hidden, y_bf16, out);
    VK_CUDA_CHECK(cudaGetLastError());
    return;
  }
  // (a large one's by an extra CTA of the row gather)
  gather_rows_kernel<<<(EM + kGatherWarps - 1) / kGatherWarps + 1, 32 * kGatherWarps, 0, stream>>>(
      A, a_rows, sorted_ids, expert_ids, block_size, EM, M * top_k, top_k, hidden, gathered, inv, 0, max_tok, tiles, n_tiles,
      max_tok_tiles(EM));

  GemmParams g{};
  g.sorted_ids = sorted_ids; g.tiles = tiles; g.n_tiles = n_tiles;
  g.N = M * top_k; g.top_k = top_k; g.w_sorted = w_sorted; g.activation = activation;
  g.limit = swiglu_limit; g.beta = beta; g.linear_beta = linear_beta; g.max_tok = max_tok;
  {  // gate/up
    GemmParams p = g;
    p.w_scale = w13_scale; p.bias = b13; p.act = act_scratch;
    p.K = hidden; p.n_feat = ispp; p.n_ftiles = ispp / 64;
    const CUtensorMap tw = make_map(w13, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, hidden / 2, w13_rows_cap, hidden / 2, 128, 64);
    const TokMaps tb = token_maps(gathered, hidden, EM, use_pair);
    timer_mark(0, stream);
    launch_gemm<true>(tw, tb, p, use_pair, stream);
    timer_mark(1, stream);
  }
  {  // down + combine
    GemmParams p = g;
    p.w_scale = w2_scale; p.bias = b2; p.topk_w = topk_w; p.out = out; p.out_rows = out_rows;
    p.store_rows = store_rows ? 1 : 0;
    p.K = ispp; p.n_feat = hidden; p.n_ftiles = (hidden + 127) / 128;
    if (ordered) {
      p.raw = partial;
      p.raw_ld = hidden;
    }
    const CUtensorMap tw = make_map(w2, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, ispp / 2, w13_rows_cap, ispp / 2, 128, 64);
    const TokMaps tb = token_maps(act_scratch, ispp, EM, use_pair);
    launch_gemm<false>(tw, tb, p, use_pair, stream);
    timer_mark(2, stream);
  }
  if (ordered)
    combine_rows_kernel<<<dim3((unsigned)M, (unsigned)((hidden + 1023) / 1024)), 256, 0, stream>>>(partial, b2, topk_w, w_sorted, sorted_ids, expert_ids, inv, block_size, EM,
                                               top_k, hidden, y_bf16, out);
  VK_CUDA_CHECK(cudaGetLastError());
}

// One GEMM of the tensor-parallel stage split (reference moe_fused.hpp:265-286): this rank's
// weights are a K-shard ([E, rows, k_shard/2] packed, [E, rows, k_shard/32] scales), the token
// rows are full width and are read from column k_base on; the result is the plain fp32 partial
// sum (no bias, activation or routing weight), which the caller all-reduces over the ranks.
//   which = 0: gate_up[EM, 2*n_out] = gather(A[M, k_full]) @ w13_shard^T     (n_out = ispp)
//   which = 1: partial[EM, n_out]   = act[EM, k_full]      @ w2_shard^T      (n_out = hidden)
// Rows of blocks with expert_ids < 0 are left untouched, padding rows of real blocks become 0.
void launch_moe_stage_gemm(int which, const uint16_t* rows_in, const uint8_t* w, const uint8_t* w_scale,
                           const int32_t* sorted_ids, const int32_t* expert_ids, float* raw, int M,
                           int k_full, int n_out, int top_k, int EM, int k_base, int k_shard,
                           cudaStream_t stream) {
  constexpr int block_size = 16;
  auto aligned16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  expects(which == 0 || which == 1, "moe stage: unknown stage");
  expects(M >= 0 && EM >= 0 && top_k > 0 && EM % block_size == 0, "moe stage: bad M / EM / top_k");
  expects(k_full > 0 && k_full % 64 == 0 && n_out > 0 && n_out % 64 == 0, "moe stage: dimensions must be multiples of 64");
  expects(k_shard > 0 && k_shard % 64 == 0 && k_base >= 0 && k_base % 64 == 0 && k_base + k_shard <= k_full,
          "moe stage: the K shard must be a multiple of 64 inside the full reduction length");
  if (M == 0 || EM == 0) return;
  expects(rows_in && w && w_scale && sorted_ids && expert_ids && raw, "moe stage: buffers must not be null");
  expects(aligned16(rows_in) && aligned16(w) && aligned16(w_scale) && aligned16(raw),
          "moe stage: buffers must be 16-byte aligned");
  const WsLayout l = ws_layout(false, EM, which == 0 ? k_full : 64, 0);
  uint8_t* ws = static_cast<uint8_t*>(workspace_get(l.total, stream));
  TokTile* tiles = reinterpret_cast<TokTile*>(ws + l.tiles_off);
  int* n_tiles = reinterpret_cast<int*>(ws + l.count_off);
  uint16_t* gathered = reinterpret_cast<uint16_t*>(ws + l.rows_off);
  const TileChoice choice = choose_tiles(M, top_k, EM, block_size, k_shard, k_shard);
  build_tiles_kernel<<<1, 1024, 0, stream>>>(expert_ids, EM / block_size, block_size, choice.max_tok, tiles,
                                             n_tiles, max_tok_tiles(EM));
  const uint16_t* token_rows = rows_in;
  if (which == 0) {
    gather_rows_kernel<<<(EM + kGatherWarps - 1) / kGatherWarps + 1, 32 * kGatherWarps, 0, stream>>>(
        rows_in, nullptr, sorted_ids, expert_ids, block_size, EM, M * top_k, top_k, k_full, gathered, nullptr, 1, 0, nullptr,
        nullptr, 0);
    token_rows = gathered;
  }
  GemmParams p{};
  p.sorted_ids = sorted_ids; p.tiles = tiles; p.n_tiles = n_tiles;
  p.N = M * top_k; p.top_k = top_k; p.max_tok = choice.max_tok;
  p.w_scale = w_scale; p.K = k_shard; p.k_base = k_base; p.raw = raw;
  p.n_feat = n_out;
  const uint64_t rows_cap = (uint64_t)1 << 31;
  const CUtensorMap tw = make_map(w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, k_shard / 2, rows_cap, k_shard / 2, 128, 64);
  const TokMaps tb = token_maps(token_rows, k_full, EM, choice.use_pair);
  if (which == 0) {
    p.n_ftiles = n_out / 64;
    p.raw_ld = 2 * n_out;
    launch_gemm<true>(tw, tb, p, choice.use_pair, stream);
  } else {
    p.n_ftiles = (n_out + 127) / 128;
    p.raw_ld = n_out;
    launch_gemm<false>(tw, tb, p, choice.use_pair, stream);
  }
  VK_CUDA_CHECK(cudaGetLastError());
}

}  // namespace vkernels::kernels::cuda
