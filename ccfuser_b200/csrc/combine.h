// Last kernels of a pass over one layer (combine.cu): slot reduction, and the router's part of the backward pass.
#pragma once
#include <stdint.h>

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
};

extern "C" int ccf_reduce(const CcfReduceArgs* a, void* stream);

// dWg[e, :] = sum over the slots routed to e (dropped ones too) of g * x[token, :], db[e] = sum of those g. `raw_order` is
// the list that the routing kernel wrote ([CCF_MAX_GROUPS] starts, then slots by expert), count_raw [e] its lengths.
extern "C" int ccf_router_dw(const int* raw_order, const int* count_raw, const float* g, const void* x, void* dwg, void* db,
                             int slots, int d, int e, int top_k, int fp16, void* stream);
