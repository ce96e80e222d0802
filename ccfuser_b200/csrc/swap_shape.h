// Tile geometry of the swapped grouped GEMM (gemm_swap.cu), host-callable so that it can be checked without a GPU.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "gemm_args.h"

namespace ccf {

struct SwapShape {
  int f_tiles;        // 256-feature tiles
  int total_tiles;
  int total_rows;
  int width;          // accumulator columns = most rows of one part
  int bufs;           // accumulators
  int buf_cols;       // TMEM columns of one
  int kblocks;        // k-blocks of a tile (both segments)
  int stages;         // of the pipeline, one k-block each
  uint32_t stage_bytes;
};

__host__ __device__ inline int swap_round16(int x) { return (x + 15) & ~15; }
// SwiGLU holds two accumulators of 128 columns twice; else 2 x 256, or 3 x 160 when a group has more than 256 rows and tiles
// have two parts: of three buffers one is free when a tile of two parts ends
__host__ __device__ inline int swap_width(int max_rows, bool wide) { return wide ? 128 : max_rows <= 256 ? 256 : 160; }
__host__ __device__ inline int swap_cap(int max_rows, bool wide) { return wide ? 128 : max_rows <= 256 ? 256 : 320; }
// rows of tokens that a CTA holds per stage for a tile of `tokens` rows: half of every part, in boxes of 16
__host__ __device__ inline int swap_half_rows(int tokens, int width) {
  const int parts = tokens > width ? 2 : 1;
  const int np = swap_round16((tokens + parts - 1) / parts);
  return parts * (((np >> 1) + 15) & ~15);
}

// The last round: `whole` tiles fill the rounds before it, each of the others comes in `pieces` parts of its rows, so that no pair has
// more than one. A piece streams the tile's weights again, from L2, and its MMAs take no less than a turn of the issuing thread (377
// clocks a k-block up to 128 rows, 512 with 256 rows), so pieces have 64 rows or more: `tile_rows` is the most that a tile holds.
struct SwapRound {
  int whole, pieces, items;
};
__host__ __device__ inline SwapRound swap_last_round(int tiles, int pairs, int tile_rows) {
  SwapRound r = {tiles, 1, tiles};
  if (tile_rows < 128) return r;
  // quotients below 2^16 of integers, half a unit above a multiple at most: exact in fp32, and a few instructions
  const int rest = tiles - pairs * static_cast<int>((static_cast<float>(tiles) + 0.5f) / static_cast<float>(pairs));
  if (2 * rest > pairs || rest < 1) return r;
  const int fit = static_cast<int>((static_cast<float>(pairs) + 0.5f) / static_cast<float>(rest)), most = tile_rows >> 6;
  r.whole = tiles - rest;
  r.pieces = fit < most ? fit : most;
  r.items = r.whole + rest * r.pieces;
  return r;
}

__host__ __device__ inline SwapShape swap_shape(const CcfGemmArgs& a, int row_tiles, int total_rows, int half_rows, int width, bool wide,
                                                int pipe_bytes, int max_stages) {
  SwapShape s;
  s.f_tiles = (a.n + 255) / 256;
  s.total_tiles = row_tiles * s.f_tiles;
  s.total_rows = total_rows;
  s.width = width;
  s.bufs = width == 160 ? 3 : 2;
  s.buf_cols = width == 160 ? 160 : 256;
  s.kblocks = a.kseg * ((a.k + 63) / 64);
  s.stage_bytes = static_cast<uint32_t>((wide ? 2 : 1) * 16384 + half_rows * 128);
  s.stages = pipe_bytes / static_cast<int>(s.stage_bytes);
  if (s.stages > max_stages) s.stages = max_stages;
  return s;
}

}  // namespace ccf
