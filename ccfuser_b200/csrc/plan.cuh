// Count exchange + row layout, shared by the stand-alone plan kernels (moe_kernels.cu) and the kernel that also computes
// the routing positions (route.cu). One CTA. Every rank writes its kept counts into every rank's table (peer stores +
// release flag carrying the step epoch), waits (bounded) for all rows of its own table, then computes the row layout of
// every owner's receive buffer:
//   rows of expert e start at base[e] (multiple of 128) on owner e / E_loc,
//   rows sent by source r start at base[e] + sum_{r' < r} count[r'][e].
// Replaces the NCCL all-gather + .cpu() + Python block planner of the reference
// (mix_moe/csrc/cuda/global_exchange.cpp:139-177, mix_moe/mix_moe/transformer.py:150-250).
#pragma once
#include "dispatch.cuh"
#include "gemm_args.h"
#include "sm100.cuh"

namespace ccf {

// `kept`: this rank's kept rows per expert, readable by every thread of the block (global or shared memory).
// A single rank skips the exchange: its own counts are the table. The prefix sums run one thread per expert over the
// experts in front of it on the same owner (independent shared-memory reads) instead of one thread per owner over all of
// them.
__device__ __forceinline__ void plan_body(const CcfPlanArgs& a, const int epoch, const int* kept) {
  __shared__ int rows[CCF_MAX_GROUPS];
  __shared__ int myoff[CCF_MAX_GROUPS];
  __shared__ int base[CCF_MAX_GROUPS];
  __shared__ int sent[CCF_MAX_RANKS];
  __shared__ int failed;
  const int tid = threadIdx.x;
  if (tid == 0) failed = 0;
  if (tid < CCF_MAX_RANKS) sent[tid] = 0;
  if (a.world > 1) {
    // 1. publish my counts
    for (int i = tid; i < a.world * a.e_total; i += blockDim.x) {
      const int p = i / a.e_total, e = i - p * a.e_total;
      a.peer_table[p][a.my_rank * a.e_total + e] = kept[e];
    }
    __threadfence_system();
    __syncthreads();
    if (tid < a.world) st_release_sys(a.peer_flag[tid] + a.my_rank, epoch);
    // 2. wait for everyone's counts (my own table, local memory)
    if (tid < a.world) {
      if (!wait_flag_ge(a.peer_flag[a.my_rank] + tid, epoch, fail_fast_limit(a.status, a.wait_limit_ns))) {
        report_status(a.status, CCF_ERR_FLAG_TIMEOUT, 0x800000 | tid);
        failed = 1;
      }
    }
  }
  __syncthreads();
  if (failed) {
    for (int e = tid; e < a.e_total; e += blockDim.x) a.dst_base[e] = 0;
    for (int e = tid; e < a.e_loc; e += blockDim.x) {
      a.group_base[e] = 0;
      a.group_rows[e] = 0;
      if (a.local_begin != nullptr) { a.local_begin[e] = 0; a.local_rows[e] = 0; }
    }
    if (tid < a.world) a.sent_rows[tid] = 0;
    return;
  }
  // 3. plan
  const int* table = a.peer_table[a.my_rank];
  for (int e = tid; e < a.e_total; e += blockDim.x) {
    int tot = 0, off = 0;
    for (int r = 0; r < a.world; ++r) {
      const int c = a.world > 1 ? ld_relaxed_sys(table + r * a.e_total + e) : kept[e];
      if (a.table_copy) a.table_copy[r * a.e_total + e] = c;
      if (r < a.my_rank) off += c;
      tot += c;
    }
    rows[e] = tot;
    myoff[e] = off;
  }
  __syncthreads();
  for (int e = tid; e < a.e_total; e += blockDim.x) {
    const int owner = e / a.e_loc, first_e = owner * a.e_loc;
    int run = 0;
    for (int i = first_e; i < e; ++i) run += (rows[i] + 127) & ~127;
    base[e] = run;
    // rows of mine that fit into the owner's buffer: the rest is rejected by the dispatch role and must not be
    // waited for (source and owner derive the same limit from the same table)
    const int fit = max(0, min(kept[e], a.max_rows - (run + myoff[e])));
    if (fit > 0) atomicAdd(&sent[owner], fit);
    if (e - first_e == a.e_loc - 1 && run + ((rows[e] + 127) & ~127) > a.max_rows) report_status(a.status, CCF_ERR_OVERFLOW, owner);
    a.dst_base[e] = run + myoff[e];
  }
  __syncthreads();
  if (tid < a.world) a.sent_rows[tid] = sent[tid];
  for (int i = tid; i < a.e_loc; i += blockDim.x) {
    const int e = a.my_rank * a.e_loc + i;
    a.group_base[i] = base[e];
    a.group_rows[i] = min(rows[e], max(0, a.max_rows - base[e]));
    if (a.local_begin != nullptr) {
      a.local_begin[i] = myoff[e];
      a.local_rows[i] = max(0, min(kept[e], a.max_rows - (base[e] + myoff[e])));
    }
  }
}

}  // namespace ccf
