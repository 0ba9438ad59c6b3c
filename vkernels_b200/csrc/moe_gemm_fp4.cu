// moe_gemm_fp4.cu - the two grouped GEMMs for small token tiles (decode, and batches of up to a few
// dozen tokens an expert) on block-scaled FP4 tensor-core instructions (tcgen05.mma.kind::mxf4).
//
// A small batch is bound by the weight stream, so the weights should reach the tensor core as the
// four bits they are. The layer's table {0, .25, 1, 1.5, 2, 3} times two, {0, .5, 2, 3, 4, 6}, is a
// subset of what the hardware reads as e2m1: moving every magnitude code c >= 2 up by two makes a
// packed word of the checkpoint a packed word of MMA operand (five integer instructions per eight
// weights and no growth; the epilogue halves the sums, which is exact), and the ue8m0 byte of a
// 32-element group is the instruction's own scale factor. Expanding to one byte a weight, as
// kind::mxf8f6f4 wants it, takes twice the integer work and twice the tensor-memory stores, and the
// padded form the copy engine can unpack to takes twice the shared memory and its bandwidth.
//
// kind::mxf4 wants four-bit tokens too. A bf16 row is written as x = s * v with s a power of two
// and v a 17-bit integer (|v| < 2^17: exact unless an element lies more than 2^9 below the row's leading
// power of two, then off by at most half a unit, 2^-17 of that power), and v as six balanced base-8 digits
// -4..4, each of which is an e2m1 value. The six digit planes of a tile lie side by side along N:
// an MMA of K = 64 takes 48 clocks at N = 96 and 96 at N = 192 (measured, the unit's full rate), its issue about 40, so
// sixteen tokens cost little more than one. The epilogue adds the planes' sums, times 8^d s / 2, in fp32.
//
// What bounds it: the weight bytes. Per 128 rows x 256 K (17 KB) an SM gets its share of HBM in about 700 clocks. A
// stage takes about 720 prepacked and 950 to 1000 from the checkpoint layout (the code warps' latency); with one byte a
// weight it took 1100 and 1700. Whole decode steps of the gpt-oss-20b shape: 8 tokens prepacked 105 -> 84 us, 64
// prepacked 142 -> 117, 128 from the checkpoint layout 203 -> 148; 48 tokens of 16 experts each (hidden 7168, ispp
// 512) 719 -> 379.
//
// Warp roles (one persistent CTA per SM; the (token tile, feature tile) items are dealt out one after the
// other):
//   warp 0      TMA producer: packed weights (128 rows x 256 K a stage)
//   warp 1      tcgen05.mma issuer + tensor-memory allocation
//   warp 2      TMA producer: digit planes of the token tile
//   warp 3      checkpoint layout: the items' scale bytes (bulk copies)
//   warps 4..   checkpoint layout: three teams of four warps (one per tensor-memory lane quarter),
//               a stage each in turn: shared memory -> code rewrite -> tensor memory, scale factors
//               prepacked weights: one team that only copies scale factors, the MMA reads the codes
//               from shared memory
//   last eight  epilogue in two sets of four: tensor memory -> registers -> global
//
// Tensor memory: columns 0..191 accumulators - two of 96 columns for tiles of up to 16 tokens, so
// that the next item's MMAs run under this item's epilogue, or one of 192; 192..199 unit scale
// factors of the tokens; then the ring of A slots (32 columns of codes and 8 of scale factors).
//
// Weights that hold the layer's inf / NaN codes (6, 7) are not expressible: the rewrite notices
// them, and the epilogue of such an item adds inf * x or NaN to the rows concerned by a scan of the
// item's codes (add_nonfinite below). A group whose scale byte is 0xFF (zero weights here, NaN to
// the tensor core) becomes scale 1 with zero codes. A token row that holds an inf or a NaN gets a
// NaN scale: every output it touches is NaN.
//
// Every wait on an mbarrier is bounded, as in moe_gemm_sm100.cu.
//
// Reference behaviour replaced: gateup_swiglu_kernel* and down_combine_kernel*
// (src/c/vkernels/kernels/moe_fused.hip:681-1436).
#include "moe_gemm_fp4.hpp"

#include <algorithm>
#include <atomic>

#include "sm100.cuh"

namespace vkernels::kernels::cuda {

namespace {

constexpr int kStageK = 256;             // K elements per stage: 128 bytes of a weight row or digit plane
constexpr int kRows = 128;               // weight rows (MMA M) per item
constexpr int kDigits = 6;
constexpr int kWBytes = kRows * 128;     // one slot of the weight ring
constexpr int kSfBytes = kRows * 8;      // prepacked scale factors of a stage
constexpr int kUnitCols = 16 * kDigits;  // accumulator columns of up to 16 tokens
constexpr int kSfbCol = 2 * kUnitCols;
constexpr int kSlot0 = kSfbCol + 8;
constexpr int kMaxW = 8, kMaxSc = 8;   // weight slots (prepacked: all eight), scale buffers
constexpr int kBadRing = 16;
constexpr int kEpiSets = 2;
constexpr int kEpiPitch = 72;            // bf16 per staged token row: 64 features + 16 bytes against bank conflicts
constexpr int kEpiBytes = 8 * 8 * 32 * 4;   // staging: down, a 1 KB block per epilogue warp; gate/up, 16 rows per set
static_assert(kEpiSets * 16 * kEpiPitch * 2 <= kEpiBytes, "gate/up staging");
constexpr int a_cols(bool packed) { return packed ? 8 : 40; }
constexpr int a_slots(bool packed) { return packed ? 8 : 7; }
constexpr int teams(bool packed) { return packed ? 1 : 3; }
constexpr int n_threads(bool packed) { return (4 + 4 * teams(packed) + 4 * kEpiSets) * 32; }
static_assert(kSlot0 + a_cols(false) * a_slots(false) <= 512 && kSlot0 + a_cols(true) * a_slots(true) <= 512, "tensor memory");

struct Bars {
  uint64_t w_full[kMaxW], w_empty[kMaxW];
  // A stage's operands, one barrier for all of them (indexed by the A slot): the code / scale-factor warps arrive, the
  // producers of the tokens - and, prepacked, of the weights - expect their bytes on it.
  uint64_t ready[8];
  uint64_t stage_done[8];   // MMA completion of a stage: frees its A slot and its token slot
  uint64_t sc_full[kMaxSc], sc_empty[kMaxSc];
  uint64_t acc_full[2], acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  int bad_item[kBadRing];   // 1 + running number of an item whose weights hold inf / NaN codes
  // per token of an epilogue set: gate/up 1 for a real row; down: address of its output row; 0 for padding
  unsigned long long tile_ref[kEpiSets][16];
  float tile_w[kEpiSets][16], tile_s[kEpiSets][16];
  int tile_flat[kEpiSets][16];
};

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}
// D[tmem] (+)= (A x 2^sfa) * (B[smem] x 2^sfb), e2m1 x e2m1, one ue8m0 factor per 32 K, K = 64.
__device__ __forceinline__ void mma_fp4_ts(uint32_t d, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t sfa,
                                           uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], %2, %3, [%5], [%6], p;\n"
      "}\n" ::"r"(d),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
      : "memory");
}
__device__ __forceinline__ void mma_fp4_ss(uint32_t d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t sfa,
                                           uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%5], [%6], p;\n"
      "}\n" ::"r"(d),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(sfa), "r"(sfb)
      : "memory");
}
// Instruction descriptor: A and B e2m1 (format 1 of this kind), ue8m0 scale factors, M = 128; which pair of
// the four scale bytes a K block takes goes to bits 29-30 (A) and 4-5 (B) per instruction.
__device__ __forceinline__ uint32_t make_idesc_fp4(int n) {
  return (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | ((uint32_t)(kRows >> 4) << 24);
}
// thread t: rows t / 4 (registers 0, 1) and t / 4 + 8 (2, 3) of 16 lanes, columns 2 (t % 4) and the next one
__device__ __forceinline__ void tc_ld_16x256b_x1(uint32_t taddr, float (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tc_ld_32x32b_x8(uint32_t taddr, float (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
               : "r"(taddr)
               : "memory");
}

// Eight packed codes of the layer -> the e2m1 codes of twice their value; *bad collects, in bit 0 of every
// nibble, the codes that have none (6 and 7: inf and NaN).
__device__ __forceinline__ uint32_t rewrite8(uint32_t w, uint32_t& bad) {
  const uint32_t b1 = w >> 1, b2 = w >> 2;
  bad |= b1 & b2;
  return w + ((b1 | b2) & 0x11111111u) * 2u;
}

// What the inf / NaN codes of one weight row add to its dot product with one token row: 0, +-inf or NaN.
__device__ __noinline__ float nonfinite_part(const uint8_t* __restrict__ w, const uint8_t* __restrict__ scale,
                                             const uint16_t* __restrict__ x, int K) {
  float sum = 0.0f;
  for (int k0 = 0; k0 < K; k0 += 8) {
    const uint32_t v = *reinterpret_cast<const uint32_t*>(w + (k0 >> 1));
    if (((v >> 1) & (v >> 2) & 0x11111111u) == 0u) continue;
    const bool zero = scale[k0 >> 5] == 0xFFu;   // inf * 0 = NaN
    for (int i = 0; i < 8; ++i) {
      const uint32_t c = (v >> (4 * i)) & 15u;
      if ((c & 6u) != 6u) continue;
      if (zero || (c & 1u)) return __int_as_float(0x7FC00000);
      sum += ((c & 8u) ? -INFINITY : INFINITY) * bf16_bits_to_f32(x[k0 + i]);
      if (sum != sum) return sum;
    }
  }
  return sum;
}

// This CTA's walk over its share of the items: every gridDim.x-th, so that the CTAs are at a few neighbouring tiles at any time
// and their reads of a tile's planes (3 K bytes a token, once per feature tile), and of an expert's weights for its next tile, come
// out of L2. With a contiguous range per CTA, which looks a tile up once for many items, the planes of as many tiles as there are CTAs
// are in use beside the weight stream: 3760 us a layer at 1024 tokens of hidden 7168, ispp 2048, 256 + 1 experts for 3068 this way, 841 for
// 748 at 1024 tokens of hidden = ispp = 2880 and 128 experts, 751 for 694 at 32 tokens of the wide shape prepacked; nowhere less. The tile is
// looked up when it changes.
struct Walk {
  const Fp4Params& p;
  int left, f, t;
  TokTile tt;
  __device__ __forceinline__ explicit Walk(const Fp4Params& p_) : p(p_) {
    const long long n = (long long)*p.n_tiles * p.n_ftiles;
    const int first = (int)blockIdx.x;
    left = (int)((n - first + gridDim.x - 1) / gridDim.x);   // (not below 0: first < gridDim.x)
    t = first / p.n_ftiles;
    f = first - t * p.n_ftiles;
    if (left > 0) tt = p.tiles[t];
  }
  __device__ __forceinline__ void next() {
    --left;
    const int was = t;
    t += p.step_t;
    f += p.step_f;
    if (f >= p.n_ftiles) {
      f -= p.n_ftiles;
      ++t;
    }
    if (t != was && left > 0) tt = p.tiles[t];
  }
};
// Tokens of a tile per MMA column block (8 or 16) and how many such blocks.
struct TileShape {
  int unit, subs;
  __device__ __forceinline__ explicit TileShape(const TokTile& tt) {
    unit = tt.n_real <= 8 ? 8 : 16;
    subs = tt.n_real <= 16 ? 1 : 2;
  }
};

template <bool GATEUP, bool PACKED>
__global__ void __launch_bounds__(n_threads(PACKED), 1)
moe_gemm_fp4_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x8,
                    const __grid_constant__ CUtensorMap tmap_x16, const Fp4Params p) {
  constexpr int kTeams = teams(PACKED), kACols = a_cols(PACKED), kASlots = a_slots(PACKED);
  constexpr int kSfCol = PACKED ? 0 : 32;   // scale-factor columns inside an A slot
  constexpr int kEpiWarp0 = 4 + 4 * kTeams;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* w_smem = smem;
  uint8_t* b_smem = w_smem + p.w_stages * kWBytes;
  uint8_t* sc_smem = b_smem + p.b_stages * p.b_stage_bytes;
  Bars* bars = reinterpret_cast<Bars*>(sc_smem + p.scale_bufs * p.scale_buf_bytes);
  uint8_t* epi_smem = reinterpret_cast<uint8_t*>(bars) + ((sizeof(Bars) + 127) & ~size_t(127));

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile int* abort_flag = &bars->abort_flag;

  if (tid == 0) {
    for (int i = 0; i < kMaxW; ++i) {
      mbar_init(smem_u32(&bars->w_full[i]), 1);
      mbar_init(smem_u32(&bars->w_empty[i]), PACKED ? 1 : 4);   // released by the stage's MMAs, or by its team
    }
    for (int i = 0; i < 8; ++i) {
      mbar_init(smem_u32(&bars->ready[i]), PACKED ? 6 : 5);
      mbar_init(smem_u32(&bars->stage_done[i]), 1);
    }
    for (int i = 0; i < kMaxSc; ++i) {
      mbar_init(smem_u32(&bars->sc_full[i]), 1);
      mbar_init(smem_u32(&bars->sc_empty[i]), 4 * p.teams);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&bars->acc_full[i]), 1);
      mbar_init(smem_u32(&bars->acc_empty[i]), 4);
    }
    bars->abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (tid < kBadRing) bars->bad_item[tid] = 0;
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;

  const int n_wrows = GATEUP ? 2 * p.n_feat : p.n_feat;
  const int n_kw = (p.K + kStageK - 1) / kStageK;
  const int pitch = p.K / 32;   // scale bytes per weight row
  Walk wk(p);

  if (warp == 0) {
    // ------------------- TMA producer: packed weights -----------------------
    if (lane == 0) {
      Ring w, a;
      bool ok = true;
      for (; wk.left > 0 && ok; wk.next()) {
        if (PACKED) {
          // one 4-D box per stage lands the item's rows in accumulator order
          const int g0 = GATEUP ? (wk.tt.expert * n_wrows + wk.f * 64) >> 3 : (wk.tt.expert * n_wrows + wk.f * 128) >> 4;
          for (int kw = 0; kw < n_kw; ++kw) {
            if (!mbar_wait(smem_u32(&bars->w_empty[w.slot]), w.phase ^ 1u, abort_flag, 2)) {
              ok = false;
              break;
            }
            // (w_stages <= kASlots: the barrier is in this stage's phase, as for the tokens below)
            const uint32_t bar = smem_u32(&bars->ready[a.slot]);
            mbar_expect_tx(bar, kWBytes);
            tma_load_4d(smem_u32(w_smem + w.slot * kWBytes), &tmap_w, kw * 128, 0, 0, g0, bar);
            w.advance(p.w_stages);
            a.advance(kASlots);
          }
        } else {
          const int row_a = GATEUP ? wk.tt.expert * n_wrows + wk.f * 64 : wk.tt.expert * n_wrows + wk.f * 128;
          const int row_b = GATEUP ? row_a + p.n_feat : row_a + 64;
          const bool both = GATEUP || p.n_feat - wk.f * 128 > 64;
          for (int kw = 0; kw < n_kw; ++kw) {
            if (!mbar_wait(smem_u32(&bars->w_empty[w.slot]), w.phase ^ 1u, abort_flag, 2)) {
              ok = false;
              break;
            }
            const uint32_t bar = smem_u32(&bars->w_full[w.slot]);
            const uint32_t dst = smem_u32(w_smem + w.slot * kWBytes);
            mbar_expect_tx(bar, both ? kWBytes : kWBytes / 2);
            tma_load_2d(dst, &tmap_w, kw * 128, row_a, bar);
            if (both) tma_load_2d(dst + kWBytes / 2, &tmap_w, kw * 128, row_b, bar);
            w.advance(p.w_stages);
          }
        }
      }
    }
  } else if (!PACKED && warp == 3) {
    // ------------------- scale bytes, an item at a time ----------------------
    // (a thread of its own: with one buffer, long K, the weights of the next item do not wait for it)
    if (lane == 0) {
      Ring sc;
      for (; wk.left > 0; wk.next()) {
        const int row_a = GATEUP ? wk.tt.expert * n_wrows + wk.f * 64 : wk.tt.expert * n_wrows + wk.f * 128;
        const int row_b = GATEUP ? row_a + p.n_feat : row_a + 64;
        const bool both = GATEUP || p.n_feat - wk.f * 128 > 64;
        if (!mbar_wait(smem_u32(&bars->sc_empty[sc.slot]), sc.phase ^ 1u, abort_flag, 1)) break;
        const uint32_t bar = smem_u32(&bars->sc_full[sc.slot]);
        const uint32_t dst = smem_u32(sc_smem + sc.slot * p.scale_buf_bytes);
        const uint32_t half = 64u * pitch;
        mbar_expect_tx(bar, both ? 2 * half : half);
        bulk_load_1d(dst, p.w_scale + (size_t)row_a * pitch, half, bar);
        if (both) bulk_load_1d(dst + half, p.w_scale + (size_t)row_b * pitch, half, bar);
        sc.advance(p.scale_bufs);
      }
    }
  } else if (warp == 2) {
    // ------------------- TMA producer: digit planes of the tokens ------------
    // Token slot of stage s is free once the MMAs of stage s - b_stages are done: stage_done of the A slot that stage used
    // (b_stages <= kASlots, so that barrier cannot have moved on to a later phase yet, and the MMAs of the stage that
    // used this A slot before have waited for its `ready` phase).
    if (lane == 0) {
      Ring a, b, lag;
      int issued = 0;
      bool ok = true;
      for (; wk.left > 0 && ok; wk.next()) {
        const TileShape sh(wk.tt);
        const uint32_t sub_bytes = (uint32_t)sh.unit * kDigits * 128;
        const CUtensorMap* map = sh.unit == 8 ? &tmap_x8 : &tmap_x16;
        for (int kw = 0; kw < n_kw; ++kw) {
          if (issued >= p.b_stages) {
            if (!mbar_wait(smem_u32(&bars->stage_done[lag.slot]), lag.phase, abort_flag, 3)) {
              ok = false;
              break;
            }
            lag.advance(kASlots);
          } else {
            ++issued;
          }
          const uint32_t bar = smem_u32(&bars->ready[a.slot]);
          const uint32_t dst = smem_u32(b_smem + b.slot * p.b_stage_bytes);
          mbar_expect_tx(bar, sub_bytes * sh.subs);
          for (int s = 0; s < sh.subs; ++s) tma_load_3d(dst + s * sub_bytes, map, kw * 128, wk.tt.row0 + 16 * s, 0, bar);
          a.advance(kASlots);
          b.advance(p.b_stages);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer -----------------------------
    // What a stage costs this warp decides the kernel's pace: a poll of a barrier takes some 120 clocks even when the
    // phase is complete, as long as all four MMAs of a 16-token tile. So a stage has ONE barrier, and the next stage's
    // is polled before this stage's MMAs are issued, under which the poll's latency disappears (three polls a
    // stage, each waited for: 1000 clocks a stage; now 400 to 450, and the loads are what is waited for).
    Ring a, b, w;
    uint32_t empty_phase = 3u;   // bit h: parity that says "free" for half h of the accumulator columns
    int half = 0;
    bool ok = true;
    bool ready = false;   // the coming stage's barrier has been seen complete
    const uint32_t tmem_u = __shfl_sync(0xFFFFFFFFu, tmem_base, 0);
    for (; wk.left > 0 && ok; wk.next()) {
      const TileShape sh(wk.tt);
      const int subs = __shfl_sync(0xFFFFFFFFu, sh.subs, 0), unit = __shfl_sync(0xFFFFFFFFu, sh.unit, 0);
      if (subs == 2) half = 0;
      const uint32_t idesc = make_idesc_fp4(unit * subs * kDigits);
      const uint32_t d_addr = tmem_u + half * kUnitCols;
      for (int h = half; h < half + subs && ok; ++h) {
        ok = mbar_wait(smem_u32(&bars->acc_empty[h]), (empty_phase >> h) & 1u, abort_flag, 4);
        empty_phase ^= 1u << h;
      }
      if (!ok) break;
      tc_fence_after();
      for (int kw = 0; kw < n_kw; ++kw) {
        if (!ready) ok = mbar_wait(smem_u32(&bars->ready[a.slot]), a.phase, abort_flag, 5);
        if (!__all_sync(0xFFFFFFFFu, ok)) {
          ok = false;
          break;
        }
        Ring nx = a;
        nx.advance(kASlots);
        ready = mbar_test(smem_u32(&bars->ready[nx.slot]), nx.phase);
        tc_fence_after();
        if (elect_one()) {
          const uint32_t a_addr = tmem_u + kSlot0 + a.slot * kACols;
          const uint64_t bdesc = make_b_desc(smem_u32(b_smem + b.slot * p.b_stage_bytes));
          const uint64_t adesc = make_b_desc(smem_u32(w_smem + w.slot * kWBytes));
          const int n_kb = min(4, (p.K - kw * kStageK) / 64);
#pragma unroll
          for (int kb = 0; kb < 4; ++kb) {
            if (kb < n_kb) {
              const uint32_t id = idesc | ((uint32_t)(2 * (kb & 1)) << 29) | ((uint32_t)(2 * (kb & 1)) << 4);
              const uint32_t sfa = a_addr + kSfCol + (kb >> 1) * 4, acc = (kw | kb) != 0 ? 1u : 0u;
              if (PACKED) mma_fp4_ss(d_addr, adesc + kb * 2, bdesc + kb * 2, id, sfa, tmem_u + kSfbCol, acc);
              else mma_fp4_ts(d_addr, a_addr + kb * 8, bdesc + kb * 2, id, sfa, tmem_u + kSfbCol, acc);
            }
          }
          tc_commit(smem_u32(&bars->stage_done[a.slot]));
          if (PACKED) tc_commit(smem_u32(&bars->w_empty[w.slot]));
          if (kw == n_kw - 1) {
            tc_commit(smem_u32(&bars->acc_full[half]));
            if (subs == 2) tc_commit(smem_u32(&bars->acc_full[1]));
          }
        }
        __syncwarp();
        a = nx;
        b.advance(p.b_stages);
        if (PACKED) w.advance(p.w_stages);
      }
      half = subs == 2 ? 0 : half ^ 1;
    }
  } else if (warp >= 4 && warp < kEpiWarp0) {
    // ------------------------------ codes / scale factors -------------------
    const int q = warp & 3, team = (warp - 4) >> 2;
    const int row = q * 32 + lane;   // tensor-memory lane of this thread
    const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + kSlot0;
    if (team == 0) {
      // unit scale factors of the digits (rows carry their scale to the epilogue), written once; the first
      // stage's hand-over to the MMA issuer orders them before any MMA
      const uint32_t one[8] = {0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu};
      tc_st8(tmem_base + ((uint32_t)(q * 32) << 16) + kSfbCol, one);
    }
    // Scale factors: column 4 h + i, byte b = tensor-memory row 32 i + lane, group 4 h + b; every lane quarter keeps a copy.
    if (PACKED) {
      // Read straight from global memory ([stage][accumulator row][8 groups]) into registers one stage ahead of
      // their use; one lane pulls them into L2 kAhead stages ahead of that (a load that went to HBM would take
      // longer than a stage lasts).
      constexpr int kAhead = 6;
      auto item_sf = [&](const Walk& v) { return p.w_scale + ((size_t)v.tt.expert * p.n_ftiles + v.f) * n_kw * kSfBytes; };
      Walk pf = wk, nx = wk;
      int pf_kw = 0, nx_kw = 0;
      auto prefetch_stage = [&]() {
        if (pf.left <= 0) return;
        bulk_prefetch_l2(item_sf(pf) + (size_t)pf_kw * kSfBytes, kSfBytes);
        if (++pf_kw == n_kw) {
          pf_kw = 0;
          pf.next();
        }
      };
      const bool pf_lane = warp == 4 && lane == 0;
      if (pf_lane)
        for (int i = 0; i < kAhead; ++i) prefetch_stage();
      uint2 nxt[4];
      auto load_next = [&]() {
        if (nx.left <= 0) return;
        const uint8_t* sf = item_sf(nx) + (size_t)nx_kw * kSfBytes;
#pragma unroll
        for (int i = 0; i < 4; ++i) nxt[i] = __ldg(reinterpret_cast<const uint2*>(sf + (32 * i + lane) * 8));
        if (++nx_kw == n_kw) {
          nx_kw = 0;
          nx.next();
        }
      };
      load_next();
      Ring sa;
      long long stages = (long long)wk.left * n_kw;
      for (; stages > 0; --stages) {
        uint32_t sf[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          sf[i] = nxt[i].x;
          sf[4 + i] = nxt[i].y;
        }
        load_next();
        if (pf_lane) prefetch_stage();
        if (!mbar_wait(smem_u32(&bars->stage_done[sa.slot]), sa.phase ^ 1u, abort_flag, 9)) break;
        __syncwarp();
        tc_fence_after();
        tc_st8(t_row + sa.slot * kACols, sf);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bars->ready[sa.slot]));
        sa.advance(kASlots);
      }
    } else if (team < p.teams) {
      // A team takes every teams-th stage of the CTA's running stage sequence: its ring positions advance by
      // that, and a weight slot is released by its team alone. The weight ring's depth is a multiple of the teams, so that
      // a slot always belongs to one team: a barrier's parity tells a phase from the next one only to a waiter that has seen
      // the phase before, and copies complete out of order - the team of stage i cannot conclude from its own stages that
      // another team's load into the slot of i has landed.
      const int srow = GATEUP ? (((row >> 3) & 1) * 64 + (row >> 4) * 8 + (row & 7)) : row;   // row inside the staged tile
      int sf_row[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int L = 32 * i + lane;
        sf_row[i] = GATEUP ? (((L >> 3) & 1) * 64 + (L >> 4) * 8 + (L & 7)) : L;
      }
      const int n_teams = p.teams;
      int w_slot = team, a_slot = team;
      uint32_t w_phase = 0, a_phase = 0;
      int kw = team, seq = 0;   // stage inside the item; running number of the item
      // A poll of a barrier costs over a hundred clocks even when its phase is complete, and these warps are bound by their
      // latency: the coming stage's codes and this stage's slot are polled ahead of the work that hides it.
      bool codes_seen = false;
      Ring sc;
      bool ok = true;
      for (; wk.left > 0 && ok; wk.next(), ++seq) {
        const int rows_valid = GATEUP ? 128 : min(128, p.n_feat - wk.f * 128);
        if (!mbar_wait(smem_u32(&bars->sc_full[sc.slot]), sc.phase, abort_flag, 7)) break;
        const uint8_t* sc_tile = sc_smem + sc.slot * p.scale_buf_bytes;
        for (; kw < n_kw; kw += n_teams) {
          if (!codes_seen && !mbar_wait(smem_u32(&bars->w_full[w_slot]), w_phase, abort_flag, 8)) {
            ok = false;
            break;
          }
          const bool slot_seen = mbar_test(smem_u32(&bars->stage_done[a_slot]), a_phase ^ 1u);
          const uint8_t* my_row = w_smem + w_slot * kWBytes + srow * 128;
          uint32_t v[32];
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const uint4 t = *reinterpret_cast<const uint4*>(my_row + ((c ^ (srow & 7)) << 4));
            v[4 * c + 0] = t.x;
            v[4 * c + 1] = t.y;
            v[4 * c + 2] = t.z;
            v[4 * c + 3] = t.w;
          }
          // the scale bytes of my four accumulator rows' eight groups (rows of the tile are 2 n bytes long)
          uint32_t sf[8];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint16_t* sp = reinterpret_cast<const uint16_t*>(sc_tile + sf_row[i] * pitch + kw * 8);
            sf[i] = (uint32_t)sp[0] | ((uint32_t)sp[1] << 16);
            sf[4 + i] = (uint32_t)sp[2] | ((uint32_t)sp[3] << 16);
          }
          uint32_t bad = 0u;
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = rewrite8(v[i], bad);
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bars->w_empty[w_slot]));   // every lane has read its codes
          if (__any_sync(0xFFFFFFFFu, (bad & 0x11111111u) != 0u && srow < rows_valid) && lane == 0)
            *reinterpret_cast<volatile int*>(&bars->bad_item[seq % kBadRing]) = seq + 1;
          // a scale byte of 0xFF anywhere (rare): zero codes and scale 1 for the group
          if (((sf[0] | sf[1] | sf[2] | sf[3] | sf[4] | sf[5] | sf[6] | sf[7]) & 0x80808080u) != 0u) {   // (none of 0x80 or more)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint32_t own = q == 0 ? sf[4 * h] : q == 1 ? sf[4 * h + 1] : q == 2 ? sf[4 * h + 2] : sf[4 * h + 3];
              const uint32_t ff = ((own & 0x7F7F7F7Fu) + 0x01010101u) & own & 0x80808080u;
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if ((ff >> (8 * (i >> 2) + 7)) & 1u) v[16 * h + i] = 0u;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) sf[i] ^= ((sf[i] & 0x7F7F7F7Fu) + 0x01010101u) & sf[i] & 0x80808080u;   // 0xFF -> 0x7F
          }
          if (!slot_seen && !mbar_wait(smem_u32(&bars->stage_done[a_slot]), a_phase ^ 1u, abort_flag, 9)) {
            ok = false;
            break;
          }
          __syncwarp();   // the tensor-memory stores are warp-aligned; the lanes may have left the wait one by one
          tc_fence_after();
          const uint32_t slot_col = t_row + a_slot * kACols;
          tc_st32(slot_col, v);
          tc_st8(slot_col + kSfCol, sf);
          w_slot += n_teams;
          if (w_slot >= p.w_stages) { w_slot -= p.w_stages; w_phase ^= 1u; }
          codes_seen = mbar_test(smem_u32(&bars->w_full[w_slot]), w_phase);
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&bars->ready[a_slot]));
          a_slot += n_teams;
          if (a_slot >= kASlots) { a_slot -= kASlots; a_phase ^= 1u; }
        }
        kw -= n_kw;
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bars->sc_empty[sc.slot]));
        sc.advance(p.scale_bufs);
      }
    }
  } else if (warp >= kEpiWarp0) {
    // ------------------------------ epilogue -------------------------------
    // Two sets of four warps (one per lane quarter), one for each half of the accumulator columns: the tiles of up to 16
    // tokens alternate between them, a larger tile gives each its 16.
    const int q = warp & 3, es = (warp - kEpiWarp0) >> 2;
    const int etid = (tid - kEpiWarp0 * 32) & 127;
    const int bar_a = 1 + es, bar_b = 3 + es;   // named barriers of the set
    unsigned long long* const tile_ref = bars->tile_ref[es];
    float* const tile_s = bars->tile_s[es];
    uint32_t phase = 0u;
    int half = 0, seq = 0, known_tile = -1;
    const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16) + es * kUnitCols;
    for (; wk.left > 0; wk.next(), ++seq) {
      const TileShape sh(wk.tt);
      const bool mine = sh.subs == 2 || half == es;
      half = sh.subs == 2 ? 0 : half ^ 1;
      if (!mine) continue;
      const int f = wk.f, row0 = wk.tt.row0 + (sh.subs == 2 ? 16 * es : 0);
      const int n_tok = sh.unit;
      if (wk.t != known_tile) {
        // per-token info of the tile (the previous tile's readers are past this barrier)
        known_tile = wk.t;
        named_bar_sync(bar_a, 128);
        if (etid < 16) {
          const int flat = row0 + etid < wk.tt.row0 + wk.tt.n_real ? p.sorted_ids[row0 + etid] : p.N;
          const bool real = flat >= 0 && flat < p.N;
          const int token = real ? flat / p.top_k : 0;
          bars->tile_flat[es][etid] = flat;
          if (GATEUP || p.raw != nullptr) {
            tile_ref[etid] = real ? 1ull : 0ull;
          } else {
            float* orow = p.out_rows ? p.out_rows[token] : p.out + (size_t)token * p.n_feat;
            if (p.store_rows && real) orow += (size_t)(flat - token * p.top_k) * p.n_feat;
            tile_ref[etid] = real ? reinterpret_cast<unsigned long long>(orow) : 0ull;
            bars->tile_w[es][etid] = (real && p.topk_w != nullptr) ? p.topk_w[p.w_sorted ? row0 + etid : flat] : 0.0f;
          }
          tile_s[etid] = real ? p.tok_scale[row0 + etid] : 0.0f;
        }
      }
      // The wait's outcome is shared by the set before anyone acts on it: a warp that gave up must not leave the others
      // standing at a later named barrier. (The barrier also publishes the tile's info and frees the staging tile of the
      // previous item.)
      const bool gave_up = !mbar_wait(smem_u32(&bars->acc_full[es]), phase, abort_flag, 10);
      phase ^= 1u;
      if (named_bar_or(bar_a, 128, gave_up)) break;
      __syncwarp();
      tc_fence_after();
      const bool bad = !PACKED && *reinterpret_cast<volatile int*>(&bars->bad_item[seq % kBadRing]) == seq + 1;
      auto release_acc = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&bars->acc_empty[es]));
      };
      // what the inf / NaN codes of weight row `wrow` add for token t of the set (cold path)
      auto nonfinite = [&](size_t wrow, int t) {
        const uint16_t* x;
        if (GATEUP) {
          const int token = bars->tile_flat[es][t] / p.top_k;
          x = p.x_rows ? p.x_rows[token] : p.x + (size_t)token * p.K;
        } else {
          x = p.x + (size_t)(row0 + t) * p.K;
        }
        return nonfinite_part(p.w + wrow * (size_t)(p.K / 2), p.w_scale + wrow * pitch, x, p.K);
      };
      if (GATEUP) {
        // Per 8 token columns the warp reads its two 16-lane groups in the 16x256b shape: a thread then holds gate and
        // up of (feature lane / 4 [+ 8], tokens 2 (lane % 4) and the next one).
        const bool situ = p.activation == 1;   // uniform across the launch
        const float clamp = p.limit > 0.0f ? p.limit : INFINITY;
        const int fl = q * 16 + (lane >> 2);
        const int tk = (lane & 3) * 2;
        float bg[2] = {0.f, 0.f}, bu[2] = {0.f, 0.f};
        if (p.bias) {
          const float* bp = p.bias + (size_t)wk.tt.expert * 2 * p.n_feat + f * 64 + fl;
          bg[0] = bp[0]; bg[1] = bp[8]; bu[0] = bp[p.n_feat]; bu[1] = bp[p.n_feat + 8];
        }
        uint16_t* const stage = reinterpret_cast<uint16_t*>(epi_smem) + es * (16 * kEpiPitch);
        for (int c0 = 0; c0 < n_tok; c0 += 8) {
          float acc[2][4];   // [lane group][gate, gate, up, up] of two tokens
#pragma unroll
          for (int d0 = 0; d0 < kDigits; d0 += 3) {   // three planes at a time, for the registers' sake
            float v[3][2][4];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
              const uint32_t col = t_lane + c0 + (d0 + d) * sh.unit;
              tc_ld_16x256b_x1(col, v[d][0]);
              tc_ld_16x256b_x1(col + (16u << 16), v[d][1]);
            }
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i) {   // digit planes: 8^d each, the largest last
              float& s = acc[i >> 2][i & 3];
              s = d0 == 0 ? v[0][i >> 2][i & 3] : s * 0.125f + v[0][i >> 2][i & 3];
              s = s * 0.125f + v[1][i >> 2][i & 3];
              s = s * 0.125f + v[2][i >> 2][i & 3];
            }
          }
          if (c0 + 8 >= n_tok) release_acc();   // this warp's last read of the accumulator
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int t = c0 + tk + e;
            const float ts = tile_s[t];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              acc[h][e] *= ts;
              acc[h][2 + e] *= ts;
            }
            if (bad && tile_ref[t] != 0ull) {
              for (int h = 0; h < 2; ++h) {
                const size_t r = (size_t)wk.tt.expert * n_wrows + f * 64 + fl + 8 * h;
                acc[h][e] += nonfinite(r, t);
                acc[h][2 + e] += nonfinite(r + p.n_feat, t);
              }
            }
          }
          uint16_t* const d = stage + (c0 + tk) * kEpiPitch + fl;
          if (!situ) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int e = 0; e < 2; ++e)
                d[e * kEpiPitch + 8 * h] = f32_to_bf16_bits(swiglu_fast(acc[h][e] + bg[h], acc[h][2 + e] + bu[h], clamp));
          } else {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int e = 0; e < 2; ++e)
                d[e * kEpiPitch + 8 * h] = f32_to_bf16_bits(moe_act_value(1, acc[h][e] + bg[h], acc[h][2 + e] + bu[h], p.limit, p.beta, p.linear_beta));
          }
        }
        // rows leave as 16-byte pieces: 8 consecutive threads write one 128-byte act row
        named_bar_sync(bar_b, 128);
        const int tok = etid >> 3, ch = etid & 7;
        if (tok < n_tok && tile_ref[tok] != 0ull)
          *reinterpret_cast<uint4*>(p.act + (size_t)(row0 + tok) * p.n_feat + f * 64 + ch * 8) =
              *reinterpret_cast<const uint4*>(stage + tok * kEpiPitch + ch * 8);
      } else {
        // The warp turns its 32 rows x 8 tokens around through shared memory, so that a lane holds four consecutive
        // output features of one token: 16-byte stores or reductions.
        const int rows_valid = min(128, p.n_feat - f * 128);
        float* stage = reinterpret_cast<float*>(epi_smem) + (es * 4 + q) * (8 * 32);
        const int hq = (lane & 7) * 4, h0 = f * 128 + q * 32 + hq;
        const bool quad_ok = q * 32 + hq < rows_valid;
        float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (p.bias && quad_ok) b4 = *reinterpret_cast<const float4*>(p.bias + (size_t)wk.tt.expert * p.n_feat + h0);
        for (int c0 = 0; c0 < n_tok; c0 += 8) {
          float a[8];
#pragma unroll
          for (int d0 = 0; d0 < kDigits; d0 += 3) {
            float v[3][8];
#pragma unroll
            for (int d = 0; d < 3; ++d) tc_ld_32x32b_x8(t_lane + c0 + (d0 + d) * sh.unit, v[d]);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              a[j] = d0 == 0 ? v[0][j] : a[j] * 0.125f + v[0][j];
              a[j] = a[j] * 0.125f + v[1][j];
              a[j] = a[j] * 0.125f + v[2][j];
            }
          }
          if (c0 + 8 >= n_tok) release_acc();
          __syncwarp();   // the previous block has been read
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float s = a[j] * tile_s[c0 + j];
            if (bad && q * 32 + lane < rows_valid && tile_ref[c0 + j] != 0ull)
              s += nonfinite((size_t)wk.tt.expert * n_wrows + f * 128 + q * 32 + lane, c0 + j);
            stage[j * 32 + lane] = s;
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int tl = (lane >> 3) + 4 * i, t = c0 + tl;
            const float4 r = *reinterpret_cast<const float4*>(stage + tl * 32 + hq);
            if (tile_ref[t] == 0ull || !quad_ok) continue;
            if (p.raw != nullptr) {   // plain partial rows, no bias, no routing weight
              *reinterpret_cast<float4*>(p.raw + (size_t)(row0 + t) * p.n_feat + h0) = r;
              continue;
            }
            float* orow = reinterpret_cast<float*>(tile_ref[t]);
            const float wgt = bars->tile_w[es][t];
            if (p.store_rows)   // plain 16-byte store of the slot's row; the home rank adds its slots in order
              *reinterpret_cast<float4*>(orow + h0) = make_float4(r.x + b4.x, r.y + b4.y, r.z + b4.z, r.w + b4.w);
            else if (p.out_rows != nullptr)
              red_add_v4_sys(orow + h0, (r.x + b4.x) * wgt, (r.y + b4.y) * wgt, (r.z + b4.z) * wgt, (r.w + b4.w) * wgt);
            else
              red_add_v4(orow + h0, (r.x + b4.x) * wgt, (r.y + b4.y) * wgt, (r.z + b4.z) * wgt, (r.w + b4.w) * wgt);
          }
        }
      }
    }
  }

  // ------------------------------ teardown ---------------------------------
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
  if (tid == 0 && bars->abort_flag != 0) atomicExch(p.status, 100 + bars->abort_flag);
}

// ---------------------------------------------------------------------------
// digit planes of the token rows
// ---------------------------------------------------------------------------

// Eight 17-bit integers -> one packed word per digit plane (plane d: digit of 8^d as an e2m1 code).
// Adding 4 (8^0 + .. + 8^4) makes the lower five digits plain base-8 fields f = digit + 4; the code of
// f is a Boolean function of its three bits, evaluated for eight nibbles at once:
//   f     0  1  2  3  4  5  6  7        digit -4 -3 -2 -1 0 1 2 3
//   code 14 13 12 10  0  2  4  5
__device__ __forceinline__ void digits8(const int (&v)[8], uint32_t (&out)[kDigits]) {
  uint32_t top = 0u;
  uint32_t u[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int s = v[i] + 18724;           // 44444 in base 8
    u[i] = (uint32_t)s;
    const int d5 = s >> 15;               // -4 .. 4
    const int m = abs(d5);
    const uint32_t c = (uint32_t)(m + min(m, 2)) | (d5 < 0 ? 8u : 0u);   // 0 2 4 5 6
    top |= c << (4 * i);
  }
  out[5] = top;
#pragma unroll
  for (int d = 0; d < 5; ++d) {
    uint32_t w = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) w |= ((u[i] >> (3 * d)) & 7u) << (4 * i);
    const uint32_t f0 = w, f1 = w >> 1, f2 = w >> 2, one = 0x11111111u;
    const uint32_t sign = ~f2 & one;
    const uint32_t c2 = ((f2 & f1) | (~f2 & ~(f1 & f0))) & one;
    const uint32_t c1 = ((f2 & ~f1 & f0) | (~f2 & ~(f1 ^ f0))) & one;
    const uint32_t c0 = (f0 & ~(f1 ^ f2)) & one;
    out[d] = (sign << 3) | (c2 << 2) | (c1 << 1) | c0;
  }
}

// Row r of the sorted order (gate/up: the activation row of token sorted_ids[r] / top_k, or the row
// at src_rows[token]; down: row r of `src` itself) -> six digit planes [6][EM][K / 2] and the row's
// scale. One CTA per row, the row held in registers between its two passes (largest magnitude,
// digits) while it has at most kHeld vectors a thread. Padding rows are left alone: their columns
// are never read back. The gather variant also does two small jobs of the layer's front end: CTA 0
// builds the token-tile list (tiles != nullptr), and every real row records where its routed slot
// went (inv[flat] = r, when inv != nullptr).
constexpr int kSplitThreads = 256;   // (128: the tile list of 240 tiles 4 us longer)
constexpr int kHeld = 4;
template <bool GATHER>
__global__ void __launch_bounds__(kSplitThreads)
digit_rows_kernel(const uint16_t* __restrict__ src, const uint16_t* const* __restrict__ src_rows,
                  const int32_t* __restrict__ sorted_ids, const int32_t* __restrict__ expert_ids, int block_size, int EM,
                  int N, int top_k, int K, uint8_t* __restrict__ planes, float* __restrict__ tok_scale,
                  int32_t* __restrict__ inv, int max_tok, TokTile* __restrict__ tiles, int* __restrict__ n_tiles,
                  int max_tiles) {
  __shared__ int s_red[kSplitThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (GATHER && blockIdx.x == 0) {
    build_tiles_block<kSplitThreads>(expert_ids, EM / block_size, block_size, max_tok, tiles, n_tiles, max_tiles, s_red,
                                     sorted_ids, N);
    return;
  }
  const int r = (int)blockIdx.x - (GATHER ? 1 : 0);
  if (expert_ids[r / block_size] < 0) return;   // never read by any tile
  const int flat = sorted_ids[r];
  if (flat < 0 || flat >= N) return;
  if (GATHER && inv != nullptr && tid == 0) inv[flat] = r;
  const uint4* row;
  if (GATHER) {
    const int token = flat / top_k;
    row = reinterpret_cast<const uint4*>(src_rows != nullptr ? src_rows[token] : src + (size_t)token * K);
  } else {
    row = reinterpret_cast<const uint4*>(src + (size_t)r * K);
  }
  const int n_vec = K / 8;
  uint4 held[kHeld];
#pragma unroll
  for (int i = 0; i < kHeld; ++i) held[i] = tid + i * kSplitThreads < n_vec ? row[tid + i * kSplitThreads] : make_uint4(0u, 0u, 0u, 0u);
  // pass 1: largest magnitude (bf16 bit patterns order like their magnitudes; inf and NaN come out on top)
  uint32_t mx = 0u;
  auto largest = [&](const uint4& v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) mx = max(mx, max(w[j] & 0x7FFFu, (w[j] >> 16) & 0x7FFFu));
  };
#pragma unroll
  for (int i = 0; i < kHeld; ++i) largest(held[i]);
  for (int i = tid + kHeld * kSplitThreads; i < n_vec; i += kSplitThreads) largest(row[i]);
  mx = __reduce_max_sync(0xFFFFFFFFu, mx);
  if (lane == 0) s_red[warp] = (int)mx;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kSplitThreads / 32; ++w) mx = max(mx, (uint32_t)s_red[w]);
  // e = floor(log2 of the largest magnitude): v = x * 2^(16 - e) lies below 2^17
  int e = mx >= 0x80u ? (int)(mx >> 7) - 127 : (mx == 0u ? 0 : 31 - __clz((int)mx) - 133);
  const bool finite = mx < 0x7F80u;
  // (in two factors: 2^(16 - e) alone leaves the fp32 range at either end)
  const float s_lo = e < 0 ? 18446744073709551616.0f : 1.0f;                 // 2^64
  const float s_hi = scalbnf(1.0f, e < 0 ? 16 - e - 64 : 16 - e);
  if (tid == 0) tok_scale[r] = finite ? scalbnf(1.0f, e - 2) : __int_as_float(0x7FC00000);   // 2^(e - 16) * 8^5 / 2
  const size_t plane = (size_t)EM * (K / 2);
  uint8_t* dst = planes + (size_t)r * (K / 2);
  auto convert = [&](const uint4& x, int i) {
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
    int v[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[2 * j] = finite ? __float2int_rn(bf16_bits_to_f32(w[j] & 0xFFFFu) * s_lo * s_hi) : 0;
      v[2 * j + 1] = finite ? __float2int_rn(bf16_bits_to_f32(w[j] >> 16) * s_lo * s_hi) : 0;
    }
    uint32_t o[kDigits];
    digits8(v, o);
#pragma unroll
    for (int d = 0; d < kDigits; ++d) *reinterpret_cast<uint32_t*>(dst + d * plane + (size_t)i * 4) = o[d];
  };
#pragma unroll
  for (int i = 0; i < kHeld; ++i)
    if (tid + i * kSplitThreads < n_vec) convert(held[i], tid + i * kSplitThreads);
  for (int i = tid + kHeld * kSplitThreads; i < n_vec; i += kSplitThreads) convert(row[i], i);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
constexpr int kMaxSmem = 227 * 1024;

template <bool GATEUP, bool PACKED>
void launch_one(const CUtensorMap& tw, const CUtensorMap& tx8, const CUtensorMap& tx16, Fp4Params p, cudaStream_t stream) {
  const Fp4Plan plan = fp4_plan(PACKED, p.K, p.tile_tok);
  p.b_stages = plan.b_stages; p.b_stage_bytes = plan.b_stage_bytes; p.w_stages = plan.w_stages;
  p.scale_bufs = plan.scale_bufs; p.scale_buf_bytes = plan.scale_buf_bytes; p.teams = plan.teams;
  static std::atomic<bool> configured[64];   // the attribute belongs to the device's context
  int dev = 0;
  VK_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev].load()) {
    VK_CUDA_CHECK(cudaFuncSetAttribute(moe_gemm_fp4_kernel<GATEUP, PACKED>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
    if (dev >= 0 && dev < 64) configured[dev].store(true);
  }
  moe_gemm_fp4_kernel<GATEUP, PACKED><<<sm_count(), n_threads(PACKED), plan.smem, stream>>>(tw, tx8, tx16, p);
}

}  // namespace

Fp4Plan fp4_plan(bool packed, int K, int tile_tok) {
  expects(tile_tok == 16 || tile_tok == 32, "fused_moe_mxfp4: the fp4 form takes tiles of up to 16 or 32 tokens");
  const int fixed = 1024 + (((int)sizeof(Bars) + 127) & ~127) + kEpiBytes + 128;
  Fp4Plan p{};
  p.b_stage_bytes = tile_tok * kDigits * 128;
  p.scale_buf_bytes = packed ? 0 : (kRows * (K / 32) + 16 + 127) & ~127;
  // Enough scale buffers that short items do not hold the code warps back (a buffer lasts an item), four token slots of the
  // largest tiles or five of the small ones (they come from L2 with its full latency), six weight slots (96 KB an SM are what
  // HBM takes to run at its rate; fewer where K is so long that its scale bytes fill the rest), and what is left for tokens
  // again. The checkpoint layout wants a multiple of the teams (see the code warps): three, or with K beyond some 40 000, where
  // the scale bytes leave room for two slots only, two.
  const int n_kw = (K + kStageK - 1) / kStageK;
  p.teams = teams(packed);
  p.scale_bufs = packed ? 0 : std::min(kMaxSc, 2 + (kMaxW - 1) / n_kw);
  p.b_stages = tile_tok == 16 || packed ? 5 : 4;
  auto room = [&]() { return (kMaxSmem - fixed - p.scale_bufs * p.scale_buf_bytes - p.b_stages * p.b_stage_bytes) / kWBytes; };
  while (room() < 6 && p.scale_bufs > 2) --p.scale_bufs;
  while (room() < 6 && p.b_stages > 4) --p.b_stages;
  while (room() < 6 && p.scale_bufs > 1) --p.scale_bufs;
  while (room() < 6 && p.b_stages > 3) --p.b_stages;
  while (room() < 3 && p.b_stages > 1) --p.b_stages;
  if (!packed && room() < 3) p.teams = 2;
  expects(room() >= p.teams, "fused_moe_mxfp4: reduction dimension too large for shared memory");
  p.w_stages = std::min(room(), packed ? kMaxW : 2 * p.teams);
  p.w_stages -= p.w_stages % p.teams;
  while (p.b_stages < a_slots(packed) && (kMaxSmem - fixed - p.scale_bufs * p.scale_buf_bytes - (p.b_stages + 1) * p.b_stage_bytes) / kWBytes >= p.w_stages)
    ++p.b_stages;
  p.smem = fixed + p.scale_bufs * p.scale_buf_bytes + p.b_stages * p.b_stage_bytes + p.w_stages * kWBytes;
  return p;
}

void launch_gemm_fp4(bool gateup, bool packed, Fp4Params p, const uint8_t* planes, int EM, cudaStream_t stream) {
  p.status = sm100_status_address();
  p.step_t = sm_count() / p.n_ftiles;   // (the grid is one CTA per SM)
  p.step_f = sm_count() % p.n_ftiles;
  const uint64_t half = (uint64_t)p.K / 2;
  const uint64_t xdims[3] = {half, (uint64_t)EM, kDigits}, xstr[2] = {half, half * EM};
  const uint32_t box8[3] = {128, 8, kDigits}, box16[3] = {128, 16, kDigits};
  const CUtensorMap tx8 = sm100_make_map_u8(planes, 3, xdims, xstr, box8);
  const CUtensorMap tx16 = sm100_make_map_u8(planes, 3, xdims, xstr, box16);
  CUtensorMap tw;
  if (packed) {
    expects((reinterpret_cast<uintptr_t>(p.w) & 31u) == 0, "prepacked weights: 32-byte alignment, K a multiple of 64");
    // Accumulator row 16 g + 8 u + j: gate/up j = feature inside a group of 8, u = gate / up half, g = group; down: plain order.
    const uint64_t n_feat = (uint64_t)p.n_feat;
    const uint64_t dims[4] = {half, 8, 2, 1ull << 27};
    const uint64_t str[3] = {half, gateup ? n_feat * half : 8 * half, gateup ? 8 * half : 16 * half};
    const uint32_t box[4] = {128, 8, 2, 8};
    tw = sm100_make_map_u8(p.w, 4, dims, str, box);
  } else {
    const uint64_t dims[2] = {half, 1ull << 31}, str[1] = {half};
    const uint32_t box[2] = {128, 64};
    tw = sm100_make_map_u8(p.w, 2, dims, str, box);
  }
  if (gateup)
    packed ? launch_one<true, true>(tw, tx8, tx16, p, stream) : launch_one<true, false>(tw, tx8, tx16, p, stream);
  else
    packed ? launch_one<false, true>(tw, tx8, tx16, p, stream) : launch_one<false, false>(tw, tx8, tx16, p, stream);
}

void launch_digit_rows(bool gather, const uint16_t* src, const uint16_t* const* src_rows, const int32_t* sorted_ids,
                       const int32_t* expert_ids, int block_size, int EM, int N, int top_k, int K, uint8_t* planes,
                       float* tok_scale, int32_t* inv, int max_tok, TokTile* tiles, int* n_tiles, int max_tiles,
                       cudaStream_t stream) {
  if (gather)
    digit_rows_kernel<true><<<EM + 1, kSplitThreads, 0, stream>>>(src, src_rows, sorted_ids, expert_ids, block_size, EM, N, top_k,
                                                                  K, planes, tok_scale, inv, max_tok, tiles, n_tiles, max_tiles);
  else
    digit_rows_kernel<false><<<EM, kSplitThreads, 0, stream>>>(src, nullptr, sorted_ids, expert_ids, block_size, EM, N, top_k, K,
                                                               planes, tok_scale, nullptr, 0, nullptr, nullptr, 0);
}

}  // namespace vkernels::kernels::cuda
