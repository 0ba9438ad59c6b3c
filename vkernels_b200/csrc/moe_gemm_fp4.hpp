// moe_gemm_fp4.hpp - launchers of the small-tile GEMM form (moe_gemm_fp4.cu).
#pragma once

#include <cuda.h>

#include "moe_tiles.cuh"

namespace vkernels::kernels::cuda {

struct Fp4Params {
  const uint8_t* w;           // packed codes: checkpoint layout or prepacked
  const uint8_t* w_scale;     // scale bytes: [E, rows, K / 32], or prepacked [E][item][stage][128 rows][8]
  const uint16_t* x;          // bf16 source rows: gate/up A (by token), down act (by sorted row)
  const uint16_t* const* x_rows;   // gate/up: optional address of every token's row
  const float* tok_scale;     // [EM]
  const float* bias;          // gate/up: [E, 2 * n_feat]; down: [E, n_feat]; or null
  const float* topk_w;        // down
  const int32_t* sorted_ids;  // [EM]
  uint16_t* act;              // gate/up output [EM, n_feat]
  float* out;                 // down output [M, n_feat]
  float* const* out_rows;     // optional: address of each token's output row (may be another GPU's memory)
  float* raw;                 // optional: plain fp32 result rows [EM, n_feat] instead of the fused combine
  int* status;
  const TokTile* tiles;
  const int* n_tiles;
  int store_rows;             // with out_rows: slot j's unweighted row is stored at row j of the token's block
  int tile_tok;               // the tile list's limit (16 or 32): what a token slot holds
  int K, n_feat, n_ftiles;
  int step_t, step_f;         // from one item of a CTA to its next (grid size items on) in tiles and feature tiles (launch_gemm_fp4)
  int N, top_k, w_sorted;
  int b_stages, b_stage_bytes, w_stages, scale_bufs, scale_buf_bytes, teams;   // (launch_gemm_fp4 fills these in)
  int activation;
  float limit, beta, linear_beta;
};

// Shared-memory plan of a launch for reduction length K over tiles of up to tile_tok tokens (16 or 32); throws where K does
// not fit. A slot takes whatever tile the list may hold: how many rows an expert has is the list's matter, not the batch's -
// a token may name an expert twice, and the real rows of a block need not be its first.
struct Fp4Plan {
  int b_stages, b_stage_bytes, w_stages, scale_bufs, scale_buf_bytes, teams, smem;
};
Fp4Plan fp4_plan(bool packed, int K, int tile_tok);

// planes: [6][EM][K / 2] digit planes of the sorted token rows (launch_digit_rows with the same tile_tok).
void launch_gemm_fp4(bool gateup, bool packed, Fp4Params p, const uint8_t* planes, int EM, cudaStream_t stream);
void launch_digit_rows(bool gather, const uint16_t* src, const uint16_t* const* src_rows, const int32_t* sorted_ids,
                       const int32_t* expert_ids, int block_size, int EM, int N, int top_k, int K, uint8_t* planes,
                       float* tok_scale, int32_t* inv, int max_tok, TokTile* tiles, int* n_tiles, int max_tiles,
                       cudaStream_t stream);

// moe_gemm_sm100.cu: a byte tensor map (128-byte swizzle, boxes 128 bytes wide; dims and box
// innermost first, strides of the outer dimensions in bytes) and the device address of the status word.
CUtensorMap sm100_make_map_u8(const void* ptr, int rank, const uint64_t* dims, const uint64_t* strides, const uint32_t* box);
int* sm100_status_address();

}  // namespace vkernels::kernels::cuda
