// Tile geometry and work split of the swapped grouped GEMM (gemm_swap.cu), host-callable so that it can be checked without a GPU.
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
  int dp_tiles;       // tiles before this one belong to one pair each; the k-blocks of the others are shared
  int sharers;        // pairs that share them
  int share_floats;   // one warp's share of a part of a sum
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

// Shortest run of k-blocks that a pair takes of a shared tile, and how close to a tile's end a run may end: a shorter one costs
// more in exchanged parts than it moves.
constexpr int kSwMinRun = 8, kSwSnap = 2;

__host__ __device__ inline SwapShape swap_shape(const CcfGemmArgs& a, int row_tiles, int total_rows, int half_rows, int width, bool wide,
                                                int n_pairs, int pipe_bytes, int max_stages) {
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
  s.share_floats = wide ? 4096 : width == 160 ? 3072 : 4096;
  s.dp_tiles = s.total_tiles;
  s.sharers = n_pairs;
  const int full = s.total_tiles / n_pairs, rem = s.total_tiles - full * n_pairs;
  // Sharing pays when the k-blocks that idle pairs would have done are worth the exchange: about 16 per pair.
  if (a.split_ws != nullptr && rem != 0 && n_pairs <= CCF_SPLIT_PAIRS && (n_pairs - rem) * s.kblocks > 16 * n_pairs) {
    s.dp_tiles = full > 1 ? (full - 1) * n_pairs : 0;
    const int runs = (s.total_tiles - s.dp_tiles) * s.kblocks / kSwMinRun;
    if (runs < s.sharers) s.sharers = runs > 0 ? runs : 1;
  }
  return s;
}

struct SwapSegment {
  int tile, kb0, kb1;
};

// The work of one CTA pair: whole tiles, then its run of the shared k-blocks, cut at the tiles' ends.
struct SwapSegments {
  const SwapShape& s;
  int t, step, pos, end;
  __host__ __device__ int bound(int p) const {
    const int kb = s.kblocks, b = static_cast<int>(static_cast<long long>(p) * (s.total_tiles - s.dp_tiles) * kb / s.sharers);
    const int r = b % kb;
    return r <= kSwSnap ? b - r : kb - r <= kSwSnap ? b + kb - r : b;
  }
  __host__ __device__ SwapSegments(const SwapShape& shape, int pair, int n_pairs) : s(shape), t(pair), step(n_pairs), pos(0), end(0) {
    if (s.dp_tiles < s.total_tiles && pair < s.sharers) {
      pos = bound(pair);
      end = bound(pair + 1);
    }
  }
  __host__ __device__ SwapSegments(const SwapShape& shape, int t_now, int pos_now, int end_now, int n_pairs)
      : s(shape), t(t_now), step(n_pairs), pos(pos_now), end(end_now) {}
  __host__ __device__ bool next(SwapSegment& g) {
    if (t < s.dp_tiles) {
      g.tile = t;
      g.kb0 = 0;
      g.kb1 = s.kblocks;
      t += step;
      return true;
    }
    if (pos >= end) return false;
    const int i = pos / s.kblocks;
    g.tile = s.dp_tiles + i;
    g.kb0 = pos - i * s.kblocks;
    const int left = end - pos, room = s.kblocks - g.kb0;
    g.kb1 = g.kb0 + (left < room ? left : room);
    pos += g.kb1 - g.kb0;
    return true;
  }
  // the pairs first .. first + n - 1 share this segment's tile, in the order of its k-blocks
  __host__ __device__ void contributors(const SwapSegment& g, int pair, int& first, int& n) const {
    const int begin = (g.tile - s.dp_tiles) * s.kblocks, stop = begin + s.kblocks;
    int last = pair;
    first = pair;
    while (bound(first) > begin) --first;
    while (bound(last + 1) < stop) ++last;
    n = last - first + 1;
  }
};

}  // namespace ccf
