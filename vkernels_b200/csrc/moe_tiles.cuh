// moe_tiles.cuh - the token-tile list of the grouped GEMMs, built from the alignment's expert_ids.
#pragma once

#include "common.cuh"

namespace vkernels::kernels::cuda {

struct TokTile {
  int expert;
  int row0;
  int n_rows;  // multiple of 16, at most the launch's tile limit
  int n_real;  // fp4 form: rows up to and including the last real one (0 when there is none)
};

namespace {

// A run of consecutive blocks with the same non-negative expert becomes ceil(rows / max_tok) tiles
// of (almost) equal size, each a multiple of 16 rows. With `sorted_ids` (tiles of up to 32 rows)
// every tile also learns where its last real row is, so that padding is neither fetched nor
// multiplied. One CTA of NT threads.
template <int NT>
__device__ __forceinline__ void build_tiles_block(const int32_t* __restrict__ expert_ids, int n_blocks, int block_size,
                                                  int max_tok, TokTile* __restrict__ tiles, int* __restrict__ n_tiles,
                                                  int max_tiles, int* warp_sums /* [NT / 32] shared */,
                                                  const int32_t* __restrict__ sorted_ids = nullptr, int N = 0) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int base = 0;   // tiles of the blocks before this round, the same in every thread
  for (int b0 = 0; b0 < n_blocks; b0 += NT) {
    const int b = b0 + tid;
    int e = -1, run_blocks = 0;
    if (b < n_blocks) {
      e = expert_ids[b];
      const bool start = e >= 0 && (b == 0 || expert_ids[b - 1] != e);
      if (start) {
        run_blocks = 1;
        while (b + run_blocks < n_blocks && expert_ids[b + run_blocks] == e) ++run_blocks;
      }
    }
    const int rows = run_blocks * block_size;
    const int nt = (rows + max_tok - 1) / max_tok;
    int incl = nt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
      if (lane >= d) incl += v;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    int before = 0, total = 0;
    for (int w = 0; w < NT / 32; ++w) {
      const int v = warp_sums[w];
      if (w < warp) before += v;
      total += v;
    }
    if (nt > 0) {
      int at = base + before + incl - nt;
      // equal split, rounded up to 16 rows
      const int per = (((rows + nt - 1) / nt) + 15) & ~15;
      int r = 0;
      for (int i = 0; i < nt; ++i, ++at) {
        const int n = min(per, rows - r);
        if (at < max_tiles && n > 0) tiles[at] = TokTile{e, b * block_size + r, n, n};
        r += n;
      }
    }
    base += total;
    __syncthreads();
  }
  const int n = min(base, max_tiles);
  if (tid == 0) *n_tiles = n;
  if (sorted_ids != nullptr) {
    // a thread per tile, its loads all in flight at once: with a warp per tile this pass was most of the row pre-pass's time
    // (240 tiles: 60 dependent round trips)
    for (int t = tid; t < n; t += NT) {
      const int row0 = tiles[t].row0, n_rows = tiles[t].n_rows;
      int last = 0;
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const int flat = j < n_rows ? sorted_ids[row0 + j] : N;
        if (flat >= 0 && flat < N) last = j + 1;
      }
      tiles[t].n_real = last;
    }
  }
}

}  // namespace

}  // namespace vkernels::kernels::cuda
