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
__host__ __device__ inline int swap_min(int a, int b) { return a < b ? a : b; }
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

// The last round: `whole` tiles fill the rounds before it, each of the others comes in up to `pieces` parts of its rows, so that no pair
// has more than one. A piece streams the tile's weights again, from L2, and its MMAs take no less than a turn of the issuing thread (377
// clocks a k-block up to 128 rows, 512 with 256 rows), so pieces have 64 rows or more: `tile_rows` is the most that a tile holds, and a
// tile of fewer rows takes fewer of its items (decode_swap_item).
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

struct SwapTile {
  int g;
  int row0;       // first row (absolute)
  int tokens;     // rows of the tile
  int zero_rows;  // rows behind them that get zeros where a reduction over rows reads the output
  int n0;         // first feature of the pair
  int parts;
  int np;         // columns of a part, a multiple of 16
};

// Work item w: a whole tile or, in the last round, a piece of one (an item without rows is nobody's work).
// `c` holds the launch's tables: shape, round, and of every group mt_prefix (row tiles in front of it), base and rows.
template <typename Tables>
__host__ __device__ __forceinline__ SwapTile decode_swap_item(int w, const Tables* c, int num_groups) {
  SwapTile ti;
  const SwapShape& s = c->shape;
  int t = w, piece = 0, pieces = 1;
  if (w >= c->round.whole) {
    pieces = c->round.pieces;
    const int u = w - c->round.whole;
    t = c->round.whole + u / pieces;
    piece = u % pieces;
  }
  int lo = 0, hi = num_groups;   // largest g with f_tiles * mt_prefix[g] <= t
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (s.f_tiles * c->mt_prefix[mid] <= t) lo = mid; else hi = mid;
  }
  ti.g = lo;
  const int mt = c->mt_prefix[lo + 1] - c->mt_prefix[lo];
  const int local = t - s.f_tiles * c->mt_prefix[lo];
  const int rows = c->rows[lo];
  // the row tiles of one block of features side by side: they share its weights. Mostly there is one, and no division to wait for
  int j = local, i = 0, per = rows;
  if (mt > 1) {
    j = local / mt;
    i = local - j * mt;
    per = swap_round16((rows + mt - 1) / mt);
  }
  ti.row0 = c->base[lo] + i * per;
  ti.tokens = swap_min(per, rows - i * per);
  ti.zero_rows = i == mt - 1 ? ((rows + 63) & ~63) - rows : 0;
  if (pieces > 1) {
    // as many as have 64 rows, in whole units of 16 rows: with at least four units to a piece the last one, whose last unit need not be
    // full, has 64 rows too. The other items of a tile are empty. Second projection of 256, 40 and 17 rows, 1024 x 4096: 30.2 -> 29.7 us
    // against one number of pieces for every tile; groups that are alike 0.1 us either way.
    const int all = ti.tokens, units = (all + 15) >> 4, most = all >> 6, of = most < 1 ? 1 : swap_min(pieces, most);
    const int at = swap_min(units * swap_min(piece, of) / of * 16, all);
    ti.tokens = swap_min(units * swap_min(piece + 1, of) / of * 16, all) - at;
    ti.row0 += at;
    if (ti.tokens == 0 || at + ti.tokens < all) ti.zero_rows = 0;   // they lie behind the tile's last row
  }
  ti.n0 = j * 256;
  ti.parts = ti.tokens > s.width ? 2 : 1;
  ti.np = swap_round16(ti.parts > 1 ? (ti.tokens + 1) >> 1 : ti.tokens);
  return ti;
}

}  // namespace ccf
