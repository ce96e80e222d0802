// Routing positions, counts, destination order and row-layout plan of one call in one kernel.
//
// What bounds it is latency, not bandwidth: a few hundred kilobytes at most pass through it, but as three kernels
// (histogram, plan, positions) every call paid three launches and three chains of dependent global reads in front of the
// first GEMM: 15.4 us at 32 slots, 20-24 us at 16384, now 4.6 and 8-10 us. One cluster of up to eight CTAs (co-scheduled by
// definition, so its barrier cannot wait for a CTA that has no SM) holds all slots of a call in registers: counts per warp in
// shared memory, counts per CTA exchanged over distributed shared memory, positions written once. Calls with
// more than CCF_ROUTE_CLUSTER_SLOTS slots use the three kernels of moe_kernels.cu, whose grid is not limited.
#include <cuda_runtime.h>
#include <stdint.h>

#include "plan.cuh"
#include "route.h"

namespace ccf {

constexpr int kRouteThreads = 1024;
constexpr int kRouteWarps = kRouteThreads / 32;
constexpr int kRouteMaxCtas = 8;

struct RouteArgs {
  const int* expert;   // [slots] expert id of each slot in token-major order; outside [0, E): not routed
  int slots, e_total, cap, first_expert;
  int* pos;            // [slots] position inside the expert (before the capacity clamp)
  int* count_raw;      // [E]
  int* count_kept;     // [E]
  int* order_off;      // [E + 1] start of each expert in the destination order
  int* sorted_slot;    // kept slots in destination order
  int* slot_row;       // [slots] -1 for slots that will not be dispatched
  int* raw_order;      // optional: [CCF_MAX_GROUPS] start of each expert, then all routed slots (dropped ones too) by expert
};

__device__ __forceinline__ int ld_cluster_s32(uint32_t cluster_addr) {
  int v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(cluster_addr) : "memory");
  return v;
}

// kL slots per thread: warp w of CTA c owns the 32 * kL consecutive slots that start at ((c * 32 + w) * kL) * 32.
template <int kL>
__global__ void __launch_bounds__(kRouteThreads) route_plan_kernel(const __grid_constant__ RouteArgs a,
                                                                   const __grid_constant__ CcfPlanArgs p, int* epoch_counter) {
  __shared__ int wh[kRouteWarps][CCF_MAX_GROUPS];   // per warp: rows per expert, then their exclusive prefix over the warps
  __shared__ int cnt[CCF_MAX_GROUPS];               // this CTA's rows per expert (read by the other CTAs of the cluster)
  __shared__ int off[CCF_MAX_GROUPS];               // rows of each expert in front of this CTA's
  __shared__ int kept[CCF_MAX_GROUPS];
  __shared__ int raw[CCF_MAX_GROUPS];
  __shared__ int order[CCF_MAX_GROUPS];             // destination order: start of each expert's kept rows
  __shared__ int order_raw[CCF_MAX_GROUPS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = static_cast<int>(blockIdx.x), ctas = static_cast<int>(gridDim.x);
  const int E = a.e_total;
  const int s0 = (rank * kRouteWarps + warp) * kL * 32 + lane;
  int e[kL], r[kL];
  after_previous();
  const int* const expert = behind(a.expert);
  for (int i = lane; i < E; i += 32) wh[warp][i] = 0;
#pragma unroll
  for (int l = 0; l < kL; ++l) {
    const int s = s0 + 32 * l;
    e[l] = s < a.slots ? expert[s] : -1;
  }
  __syncwarp();
#pragma unroll
  for (int l = 0; l < kL; ++l) {
    if (e[l] < 0 || e[l] >= E) e[l] = -1;
    const unsigned m = __match_any_sync(0xffffffffu, e[l]);
    const int below = __popc(m & ((1u << lane) - 1u));
    const int before = e[l] >= 0 ? wh[warp][e[l]] : 0;
    __syncwarp();
    if (e[l] >= 0 && below == 0) wh[warp][e[l]] = before + __popc(m);
    __syncwarp();
    r[l] = before + below;
  }
  __syncthreads();
  if (tid < E) {
    int run = 0;
#pragma unroll 8
    for (int w = 0; w < kRouteWarps; ++w) {
      const int c = wh[w][tid];
      wh[w][tid] = run;
      run += c;
    }
    cnt[tid] = run;
  }
  if (ctas > 1) cluster_sync_all(); else __syncthreads();
  if (tid < E) {
    int before = 0, tot = 0;
    const uint32_t mine = smem_u32(&cnt[tid]);
    for (int c = 0; c < ctas; ++c) {
      const int v = c == rank ? cnt[tid] : ld_cluster_s32(map_to_cta(mine, c));
      if (c < rank) before += v;
      tot += v;
    }
    off[tid] = before;
    raw[tid] = tot;
    kept[tid] = min(tot, a.cap);
  }
  __syncthreads();
  if (tid < E) {
    // destination order of this rank's kept rows: experts starting with this rank's own (first_expert), then the next
    // owner's, ... so that local rows are pushed first and every source starts with a different owner
    const int turn = (tid - a.first_expert + E) % E;
    int o = 0, o_raw = 0, x = a.first_expert;
    for (int k = 0; k < turn; ++k) {
      o += kept[x];
      o_raw += raw[x];
      if (++x == E) x = 0;
    }
    order[tid] = o;
    order_raw[tid] = o_raw;
    if (rank == 0) {
      a.count_raw[tid] = raw[tid];
      a.count_kept[tid] = kept[tid];
      a.order_off[tid] = o;
      if (turn == E - 1) a.order_off[E] = o + kept[tid];   // kept rows in total
      if (a.raw_order != nullptr) a.raw_order[tid] = o_raw;
    }
  }
  __syncthreads();
#pragma unroll
  for (int l = 0; l < kL; ++l) {
    const int s = s0 + 32 * l;
    if (s >= a.slots) continue;
    if (e[l] < 0) {
      a.pos[s] = 0x3fffffff;
      a.slot_row[s] = -1;
      continue;
    }
    const int q = off[e[l]] + wh[warp][e[l]] + r[l];
    a.pos[s] = q;
    if (q < a.cap) a.sorted_slot[order[e[l]] + q] = s;
    else a.slot_row[s] = -1;                       // dropped slots are never dispatched
    if (a.raw_order != nullptr) a.raw_order[CCF_MAX_GROUPS + order_raw[e[l]] + q] = s;
  }
  if (rank == 0) {
    int epoch = p.epoch;
    if (epoch_counter != nullptr) epoch = *epoch_counter + 1;   // a replayed graph has frozen arguments
    __syncthreads();
    plan_body(p, epoch, kept);
    if (epoch_counter != nullptr && tid == 0) *epoch_counter = epoch;
  }
  if (ctas > 1) cluster_sync_all();   // no CTA leaves while its counts may still be read
}

}  // namespace ccf

extern "C" {

// Routing (as ccf_route_ordered) and plan (as ccf_plan, or ccf_plan_dev_epoch when epoch_counter is not null) of one call.
// Returns 1 without launching anything when the call has no slots or more than this kernel holds: use the separate
// entry points then.
int ccf_route_plan(const int* expert, int S, int E, int cap, int* pos, int* count_raw, int* count_kept, int* order_off,
                   int* sorted_slot, int* slot_row, int first_expert, int* raw_order, const CcfPlanArgs* plan,
                   int* epoch_counter, void* stream) {
  using namespace ccf;
  if (E < 1 || E > CCF_MAX_GROUPS || plan->world < 1 || plan->world > CCF_MAX_RANKS || plan->e_total != E) return -2;
  if (S < 1 || S > CCF_ROUTE_CLUSTER_SLOTS) return 1;
  int ctas = 1;
  while (ctas < kRouteMaxCtas && ctas * kRouteThreads < S) ctas *= 2;
  int per = 1;
  while (ctas * kRouteThreads * per < S) per *= 2;
  RouteArgs a = {expert, S, E, cap, first_expert, pos, count_raw, count_kept, order_off, sorted_slot, slot_row, raw_order};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kRouteThreads);
  cfg.stream = reinterpret_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[2] = {cluster_attribute(ctas, 1, 1), early_attribute()};
  cfg.attrs = attr;
  cfg.numAttrs = 1 + (plan->world == 1 ? early_launches(S, cfg.stream) : 0);
  auto kern = per == 1 ? route_plan_kernel<1> : per == 2 ? route_plan_kernel<2> : per == 4 ? route_plan_kernel<4> : route_plan_kernel<8>;
  cudaError_t err = cudaLaunchKernelEx(&cfg, kern, a, *plan, epoch_counter);
  return err == cudaSuccess ? 0 : -static_cast<int>(err);
}

}  // extern "C"
