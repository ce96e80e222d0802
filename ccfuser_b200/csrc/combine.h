// Last kernels of a pass over one layer (combine.cu): slot reduction, and the router's part of the backward pass. Also the rule
// by which the grouped row sums (router_dw_kernel, colsum_grouped_kernel) share the rows of a group among a cluster.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ccf {

// Cluster size of a launch with `blocks` blocks per split: as many as keep the launch resident at once (five blocks of these kernels
// fit on an SM; clusters of four and eight no longer pack from 704 blocks on). Column sums, us with 1024 rows per group at
// 1 / 2 / 4 / 8 blocks per group: 32 blocks 13.4 / 8.7 / 6.5 / 5.6; 128 blocks 14.3 / 10.4 / 9.0 / 11.7; with 1 and 2 368 blocks
// 18.9 / 17.5, 384 blocks 19.2 / 24.1; with 2 and 4 160 blocks 11.1 / 10.1, 176 blocks 11.4 / 14.2. `rows`: expected rows per group,
// 0 = not known; blocks that will hardly find work are not launched (0.5 to 0.8 us for a launch of 96 to 128 blocks).
constexpr int kRowsPerSplit = 128;
inline int group_splits(int blocks, int rows) {
  int splits = 1;
  while (splits < 8 && 2 * splits * blocks <= (splits == 1 ? 5 * 148 : 640) && (rows <= 0 || rows >= 2 * splits * kRowsPerSplit)) splits *= 2;
  return splits;
}
// Of those, the ones that have work: every block keeps at least two passes of 64 rows. The count is read on the device, group by
// group; the other blocks leave at once (a cluster barrier waits for blocks that have not left). 128 blocks, 188 rows: 4.6 us
// with one block per group, 4.9 with two, 4.8 with four; 256 rows: 5.3 / 5.1 / 5.1; 512 rows: 8.4 / 6.9 / 6.4.
__device__ __forceinline__ int splits_with_work(int rows, int splits) {
  while (splits > 1 && rows < kRowsPerSplit * splits) splits >>= 1;
  return splits;
}

}  // namespace ccf

// One launch of the slot reduction y[t] = sum of the kept slots' rows of token t (+ the router's share of an input
// gradient). The optional parts are off where their first pointer is null.
struct CcfReduceArgs {
  const void* comb;          // [tokens * top_k, d] rows returned by the owners
  const int* slot_row;       // [tokens * top_k] negative = slot was not dispatched
  void* y;                   // [tokens, d]
  // completion check of a single-rank layer (with peers ccf_combine_wait comes first): the launch that fills `comb`
  // precedes this one on the stream, so one thread only has to verify and consume its count
  const int* done;
  int* cum;
  const int* sent_rows;
  int* status;
  unsigned long long wait_limit_ns;
  int* zero_words;           // the layer's arrival counters, returned to zero for the next pass
  int n_tiles, zero_count;
  // router: y[t] += sum_j g_j * Wg[idx_j],  g_j = w_j (dw_j - sum_i w_i dw_i); g [tokens * top_k] is written
  const int* idx;
  const float* w;
  const float* dw;           // gradient arriving for the weights; taken as zero for slots that were not dispatched
  const void* wg;            // [e, d]
  float* g;
  int tokens, top_k, d, e, fp16;
  int early;                 // 1: may be set up while the kernel in front of it still runs (sm100.cuh)
};

extern "C" int ccf_reduce(const CcfReduceArgs* a, void* stream);

// dWg[e, :] = sum over the slots routed to e (dropped ones too) of g * x[token, :], db[e] = sum of those g. `raw_order` is
// the list that the routing kernel wrote ([CCF_MAX_GROUPS] starts, then slots by expert), count_raw [e] its lengths.
extern "C" int ccf_router_dw(const int* raw_order, const int* count_raw, const float* g, const void* x, void* dwg, void* db,
                             int slots, int d, int e, int top_k, int fp16, void* stream);
