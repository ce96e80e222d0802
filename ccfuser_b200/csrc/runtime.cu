// Native runtime of one fused MoE layer (see runtime.h): ccf_layer_forward / ccf_layer_backward issue the launches of a pass in
// order and on one stream: routing, count exchange + plan, dispatch fused with GEMM-1, GEMM-2 fused with combine, wait +
// reduce; and for backward the dy dispatch fused with dgrad-2, both weight-gradient GEMMs, the bias-gradient column sums,
// dgrad-1 fused with combine, wait + reduce and, where the call included the router, its gradients. The GEMM launches are
// those that ops/fused.py issues call by call from Python (tests/test_native_runtime.py compares the launch blocks); around
// them that path keeps the kernels apart that are one here: routing and plan, completion wait, clearing of the arrival
// counters and reduce.
#include <cuda_runtime.h>
#include <string.h>

#include "combine.h"
#include "route.h"
#include "runtime.h"
#include "sm100.cuh"

extern "C" {
int ccf_gemm_launch(const CcfGemmLaunch* L, void* stream);
int ccf_route_ordered(const int* expert, int S, int E, int cap, int* pos, int* block_hist, int* block_off,
                      int* count_raw, int* count_kept, int* ticket, int* order_off, int* sorted_slot, int* slot_row,
                      int first_expert, void* stream);
int ccf_plan(const CcfPlanArgs* a, void* stream);
int ccf_plan_dev_epoch(const CcfPlanArgs* a, int* epoch_counter, void* stream);
int ccf_combine_wait(const int* done, int* cum, const int* sent_rows, int n_tiles, int world,
                     unsigned long long limit_ns, int* status, void* stream);
int ccf_colsum_grouped_hint(const void* x, long long ld, int n, int groups, const int* group_base, const int* group_rows,
                            void* out, int fp16, int rows_hint, void* stream);
}

namespace {

constexpr int kMajK = 0, kMajMN = 1;

struct Dry {
  CcfGemmLaunch* out;
  int cap;
  int n;
};

// completion-counter increments per row of a COMBINE GEMM with n columns: one per 32 columns, whatever kernel stores them
int combine_units(int n) { return n / 32; }

// Kernel of a row-grouped launch (row_kernel below)
struct RowKernel {
  int few_rows, two_cta, a_rows, bn;
};

// Bound on the rows of any expert of a single-rank call (its capacity, at most all slots of the call; other ranks may bring
// any number of rows), rounded up to a pipeline geometry of the one-CTA kernel: 32, 64, or 0 for no bound.
int row_bound(int capacity, int world) { return world != 1 || capacity > 64 ? 0 : capacity > 32 ? 64 : 32; }

// The kernel of a row-grouped launch of a call that expects `rows` rows for each of `experts` experts of this rank:
// at most small_rows: weights on the M side (gemm_swap.cu); more: CTA pairs (gemm2.cu). Without CTA pairs (CCFUSER_TWO_CTA=0) the
// one-CTA kernel, with the pipeline that the capacity allows, and with 128-column tiles for a second projection whose 256-column
// tiles would leave most of the 148 SMs without one. Every rank of a group may come to another choice: what it counts for
// the others does not depend on the kernel (combine_units).
RowKernel row_kernel(int epi, int b_major, long long rows, int experts, int n, int capacity, int world, int small_rows, int two_cta) {
  if (rows <= small_rows && two_cta) return {1, 0, 0, 0};
  if (two_cta) return {0, 1, 0, 0};
  const long long tiles = experts * (rows > 128 ? (rows + 127) / 128 : 1) * ((n + 255) / 256);
  return {0, 0, row_bound(capacity, world), epi == CCF_EPI_COMBINE && b_major == kMajK && tiles < 148 ? 128 : 0};
}

void set_row_kernel(CcfGemmLaunch& g, const CcfLayer* L, int tokens, int capacity) {
  const long long rows = static_cast<long long>(tokens) * L->top_k * L->world / (L->e_total > 0 ? L->e_total : 1);
  const RowKernel r = row_kernel(g.epi, g.b_major, rows, L->e_loc, g.args.n, capacity, L->world, L->small_rows, L->two_cta);
  g.few_rows = r.few_rows;
  g.two_cta = r.two_cta;
  g.args.a_rows = r.a_rows;
  g.args.bn = r.bn;
}

// Whether a weight-gradient launch of a call that expects `rows` rows per expert runs on gemm_wgrad.cu, which moves its result by TMA,
// or on the pair kernel: with few rows the reduction is only a handful of k-blocks, and moving the weights decides. In place the
// weights are read as well as written, and the line lies higher. The lines were drawn when gemm_wgrad.cu held three stages, and
// tests/test_row_kernel.py holds them there. With four stages it is the faster one beyond them too; gemm_wgrad.cu over pair kernel, time of
// single launches, both in alternation:
//   plain     1024 x 4096, 64 experts: 0.94 at 512 rows, 0.94 at 640, 1.01 at 768; 2048 x 8192, 16: 0.93, 0.95, 1.00, and 1.05 at 1024;
//             768 x 3072, 16: 0.92, 0.95, 1.02, 1.05; 4096 x 14336, 8: 0.93, 0.92, 0.99
//   in place  1024 x 4096, 64 experts: 0.83 at 512 rows, 0.94 at 640, 0.99 at 768; 2048 x 8192, 16: 0.79, 0.90, 0.94, and 1.03 at 1024;
//             4096 x 14336, 8: 0.79, 0.91, 0.97
// Whole training passes, two runs each, of which those of a millisecond differ by up to 5 % among themselves:
//   plain     at 400, 450, 512, 580 and 640 rows: 1024 x 4096, 64 experts 0.99, 1.00, 0.96, 1.02, 0.98; 16 experts 0.99 at all five;
//             2048 x 8192, 16: 1.03, 0.99, 0.95, 1.05, 0.99; 768 x 3072, 16: 0.99, 0.99, 0.99, 1.00, 1.00. About 1 % lies between the lines
//   in place  at 560, 640 and 768 rows: 1024 x 4096, 64 experts 0.95, 0.98, 0.96; 16 experts 0.96, 0.97, 0.99; 2048 x 8192, 16: 0.92, 0.97,
//             0.94; 768 x 3072, 16: 0.97, 0.98, 0.99. Here the line at 512 costs a pass 1 to 8 %
bool wgrad_few(long long rows, bool in_place, int two_cta) { return two_cta && rows <= (in_place ? 512 : 384); }

// Whether the launches of a call may overlap with the end of the ones in front of them (sm100.cuh). A group of ranks leaves it: there a
// clearing of counters lies between its kernels.
int early_of(const CcfLayer* L, int tokens, const Dry* dry, void* stream) {
  return dry == nullptr && L->world == 1 ? ccf::early_launches(static_cast<long long>(tokens) * L->top_k, reinterpret_cast<cudaStream_t>(stream)) : 0;
}

// fields every launch of this layer shares
CcfGemmLaunch base_launch(const CcfLayer* L, int early) {
  CcfGemmLaunch g;
  memset(&g, 0, sizeof(g));
  g.args.group_base = L->group_base;
  g.args.group_rows = L->group_rows;
  g.args.sched = L->sched;
  g.args.status = L->status;
  g.args.wait_limit_ns = L->wait_limit_ns;
  g.args.num_groups = L->e_loc;
  g.args.kseg = 1;
  g.args.fp16 = L->fp16;
  g.args.world = 1;
  g.args.count_rows = 1;
  g.args.total_index = -1;
  g.args.comm_warps = L->comm_warps;
  g.device = L->device;
  g.two_cta = L->two_cta;
  g.early = early;
  return g;
}

void set_a(CcfGemmLaunch& g, const void* a0, long long rows, long long cols, int major) {
  g.a0 = a0;
  g.a_rows = rows;
  g.a_cols = cols;
  g.a_major = major;
}
void set_b(CcfGemmLaunch& g, const void* b0, long long rows, long long cols, int major) {
  g.b0 = b0;
  g.b_rows = rows;
  g.b_cols = cols;
  g.b_major = major;
}

// the dispatch role's arguments (forward: x rows into the owners' xrecv; backward: g * dy rows into their grecv)
void set_dispatch(CcfGemmLaunch& g, const CcfLayer* L, const void* src, const int* idx, const float* gate_w, int tokens,
                  int capacity, int backward, float* dgate) {
  CcfDispatchArgs& a = g.args.disp;
  a.x = src;
  a.slot_expert = idx;
  a.slot_pos = L->slot_pos;
  a.dst_base = L->dst_base;
  a.slot_gate = gate_w;
  a.saved_comb = backward ? L->comb : nullptr;
  a.dgate = dgate;
  a.slot_row = L->slot_row;
  a.sorted_slot = L->sorted_slot;
  a.order_off = L->order_off;
  for (int r = 0; r < L->world; ++r) {
    a.peer_recv[r] = backward ? L->peer_grecv[r] : L->peer_xrecv[r];
    a.peer_row_src[r] = L->peer_row_src[r];
    a.peer_row_gate[r] = L->peer_row_gate[r];
    a.peer_tile_flags[r] = L->peer_tile_flags[r];
  }
  a.work_counter = L->sched + 2;
  a.tokens = tokens;
  a.top_k = L->top_k;
  a.d = L->d_model;
  a.capacity = capacity;
  a.experts_per_rank = L->e_loc;
  a.my_rank = L->rank;
  a.backward = backward;
  a.fp16 = L->fp16;
  a.max_rows = L->max_rows;
  a.total_index = L->max_rows / 128;
  a.e_total = L->e_total;
  // the GEMM side of the same kernel: tiles gated on the arrival counters, local-source tiles first
  g.args.tile_flags = L->tile_flags;
  g.args.local_begin = L->local_begin;
  g.args.local_rows = L->local_rows;
  g.args.n_comm_ctas = L->n_comm_ctas;
  g.args.total_index = L->max_rows / 128;
}

void set_combine(CcfGemmLaunch& g, const CcfLayer* L, void* const* peer_comb, const float* row_gate) {
  g.args.row_src = L->row_src;
  g.args.row_gate = row_gate;
  for (int r = 0; r < L->world; ++r) {
    g.args.peer_comb[r] = peer_comb[r];
    g.args.peer_done[r] = L->peer_done[r];
  }
  g.args.world = L->world;
  g.args.send_finish = 1;
  g.args.count_rows = L->world > 1;
  g.args.max_slots = L->max_slots;
}

int issue(CcfGemmLaunch& g, Dry* dry, void* stream) {
  // the kernels on CTA pairs need 256-row output tiles in k-grouped mode
  if (g.kgroup && g.args.m_per_group % 256 != 0) g.two_cta = g.few_rows = 0;
  if (g.args.ld_out == 0) g.args.ld_out = g.args.n;
  if (dry != nullptr) {
    if (dry->n < dry->cap) dry->out[dry->n] = g;
    ++dry->n;
    return 0;
  }
  return ccf_gemm_launch(&g, stream);
}

// Wait for the owners and sum the k slots of each token. With G (backward) and a router in the call, the sum also carries
// the gradient through the gate weights.
int wait_and_reduce(const CcfLayer* L, const void* comb, void* out, int tokens, const CcfLayerGrads* G, const int* idx,
                    const float* gate_w, int early, Dry* dry, void* stream) {
  if (dry != nullptr) return 0;
  CcfReduceArgs r;
  memset(&r, 0, sizeof(r));
  r.comb = comb;
  r.slot_row = L->slot_row;
  r.y = out;
  r.tokens = tokens;
  r.top_k = L->top_k;
  r.d = L->d_model;
  r.fp16 = L->fp16;
  r.early = early;
  if (L->world == 1) {
    r.done = L->done;
    r.cum = L->done_cum;
    r.sent_rows = L->sent_rows;
    r.n_tiles = 0;   // the rows of a single rank are not counted
    r.status = L->status;
    r.wait_limit_ns = L->wait_limit_ns;
    r.zero_words = L->tile_flags;
    r.zero_count = L->max_rows / 128 + 1;
  } else {
    const int rc = ccf_combine_wait(L->done, L->done_cum, L->sent_rows, combine_units(L->d_model), L->world,
                                    L->wait_limit_ns, L->status, stream);
    if (rc) return rc;
  }
  if (G != nullptr && G->router_w != nullptr) {
    r.idx = idx;
    r.w = gate_w;
    r.dw = G->dgate;
    r.wg = G->router_w;
    r.g = G->slot_grad;
    r.e = L->e_total;
  }
  return ccf_reduce(&r, stream);
}

int clear_arrivals(const CcfLayer* L, void* stream) {
  cudaError_t e = cudaMemsetAsync(L->tile_flags, 0, sizeof(int) * (L->max_rows / 128 + 1),
                                  reinterpret_cast<cudaStream_t>(stream));
  return e == cudaSuccess ? 0 : -static_cast<int>(e);
}

// The arrival counters return to zero between the kernel that waits on them and this rank's finish token: peers push the
// next pass's rows only after that token. A single rank has no peers, and its reduce kernel, the last of the pass, does it.
int zero_tile_flags(const CcfLayer* L, Dry* dry, void* stream) {
  if (dry != nullptr || L->world == 1) return 0;
  return clear_arrivals(L, stream);
}

// Result of a pass that ends with `rc`. A pass of a single rank that is given up at one of its launches never reaches the reduce
// kernel: with the counters left full, every tile of the group's next pass would go through its gate before its rows have
// arrived.
int end_of_pass(const CcfLayer* L, int rc, Dry* dry, void* stream) {
  if (rc != 0 && dry == nullptr && L->world == 1) clear_arrivals(L, stream);
  return rc;
}

int forward_pass(const CcfLayer* L, const void* x, const int* idx, const float* gate_w, void* y, int tokens, int capacity,
                 int save_pre, int epoch, void* stream, Dry* dry) {
  const int d = L->d_model, f = L->d_ffn, e_loc = L->e_loc, early = early_of(L, tokens, dry, stream);
  int rc = 0;
  if (dry == nullptr) {
    if (L->device >= 0 && cudaSetDevice(L->device) != cudaSuccess) return -7;
    // 1. positions, kept counts, destination order of this rank's slots; count exchange with all ranks + row layout
    CcfPlanArgs p;
    memset(&p, 0, sizeof(p));
    p.count_kept = L->count_kept;
    for (int r = 0; r < L->world; ++r) {
      p.peer_table[r] = L->peer_cnt_table[r];
      p.peer_flag[r] = L->peer_cnt_flag[r];
    }
    p.dst_base = L->dst_base;
    p.group_base = L->group_base;
    p.group_rows = L->group_rows;
    p.sent_rows = L->sent_rows;
    p.table_copy = L->table_copy;
    p.local_begin = L->local_begin;
    p.local_rows = L->local_rows;
    p.status = L->status;
    p.wait_limit_ns = L->wait_limit_ns;
    p.world = L->world;
    p.my_rank = L->rank;
    p.e_total = L->e_total;
    p.e_loc = e_loc;
    p.epoch = epoch;
    p.max_rows = L->max_rows;
    int* epoch_dev = epoch >= 0 ? nullptr : L->epoch_dev;
    rc = ccf_route_plan(idx, tokens * L->top_k, L->e_total, capacity, L->slot_pos, L->count_raw, L->count_kept, L->order_off,
                        L->sorted_slot, L->slot_row, L->rank * e_loc, save_pre ? L->raw_order : nullptr, &p, epoch_dev, stream);
    if (rc == 1) {   // no slots, or more than the one-kernel form holds
      rc = ccf_route_ordered(idx, tokens * L->top_k, L->e_total, capacity, L->slot_pos, L->block_hist, L->block_off,
                             L->count_raw, L->count_kept, L->ticket, L->order_off, L->sorted_slot, L->slot_row,
                             L->rank * e_loc, stream);
      if (rc) return rc;
      rc = epoch_dev == nullptr ? ccf_plan(&p, stream) : ccf_plan_dev_epoch(&p, epoch_dev, stream);
    }
    if (rc) return rc;
  }
  // 3. dispatch + GEMM-1 (+ bias + activation)
  {
    CcfGemmLaunch g = base_launch(L, early);
    set_a(g, L->xrecv, L->max_rows, d, kMajK);
    set_b(g, L->w1, static_cast<long long>(e_loc) * f, d, kMajK);
    g.args.n = f;
    g.args.k = d;
    g.args.b_group_rows = f;
    g.args.out0 = L->h_act;
    g.out_rows = L->max_rows;
    g.args.out1 = save_pre ? L->h_pre : nullptr;
    g.args.bias0 = L->b1;
    if (L->swiglu) {
      g.epi = CCF_EPI_SWIGLU;
      g.b1 = L->wg;
      g.args.out2 = save_pre ? L->h_pre2 : nullptr;
      g.args.bias1 = L->bg;
    } else {
      g.epi = CCF_EPI_BIAS_ACT;
      g.args.act = L->act;
    }
    set_dispatch(g, L, x, idx, gate_w, tokens, capacity, 0, nullptr);
    set_row_kernel(g, L, tokens, capacity);
    if ((rc = issue(g, dry, stream))) return rc;
    if ((rc = zero_tile_flags(L, dry, stream))) return rc;
  }
  // 4. GEMM-2 + combine into the source ranks
  {
    CcfGemmLaunch g = base_launch(L, early);
    set_a(g, L->h_act, L->max_rows, f, kMajK);
    set_b(g, L->w2, static_cast<long long>(e_loc) * d, f, kMajK);
    g.epi = CCF_EPI_COMBINE;
    g.args.n = d;
    g.args.k = f;
    g.args.b_group_rows = d;
    g.args.bias0 = L->b2;
    g.args.ld_out = d;
    set_combine(g, L, L->peer_comb, L->row_gate);
    set_row_kernel(g, L, tokens, capacity);
    if ((rc = issue(g, dry, stream))) return rc;
  }
  // 5. wait for every owner, sum the k slots of each token
  return wait_and_reduce(L, L->comb, y, tokens, nullptr, nullptr, nullptr, early, dry, stream);
}

int backward_pass(const CcfLayer* L, const void* dy, const int* idx, const float* gate_w, const CcfLayerGrads* G, int tokens,
                  int capacity, void* stream, Dry* dry) {
  const int d = L->d_model, f = L->d_ffn, e_loc = L->e_loc, early = early_of(L, tokens, dry, stream);
  int rc = 0;
  if (dry == nullptr && L->device >= 0 && cudaSetDevice(L->device) != cudaSuccess) return -7;
  const long long rows_per_expert = static_cast<long long>(tokens) * L->top_k * L->world / (L->e_total > 0 ? L->e_total : 1);
  const int rows_hint = static_cast<int>(rows_per_expert > 0 ? rows_per_expert : 1);
  // In-place SGD (sgd_lr != 0), matrix by matrix: a weight whose gradient pointer is null is updated by its weight-gradient
  // GEMM. w2 may be at any group size (dgrad-2 above it is its last reader). w1 / wg only on a single rank: dgrad-1 reads
  // them and, with peers, has to stay the last owner-side kernel of the pass.
  const bool sgd2 = G->sgd_lr != 0.f && G->dw2 == nullptr;
  const bool sgd = G->sgd_lr != 0.f && G->dw1 == nullptr;     // w1 (and wg) in place: dgrad-1 moves in front of wgrad-1
  if (sgd && L->world != 1) return -2;
  if (sgd && L->swiglu && G->dwg != nullptr) return -2;
  // 1 + 2. push g * dy rows + dgrad-2 with the activation derivative
  {
    CcfGemmLaunch g = base_launch(L, early);
    set_a(g, L->grecv, L->max_rows, d, kMajK);
    set_b(g, L->w2, static_cast<long long>(e_loc) * d, f, kMajMN);
    g.args.n = f;
    g.args.k = d;
    g.args.b_group_rows = d;
    g.args.out0 = G->dh;
    g.out_rows = L->max_rows;
    g.args.aux0 = L->h_pre;
    if (L->swiglu) {
      g.epi = CCF_EPI_DSWIGLU;
      g.args.out1 = G->dh2;
      g.args.aux1 = L->h_pre2;
    } else {
      g.epi = CCF_EPI_DACT;
      g.args.act = L->act;
    }
    set_dispatch(g, L, dy, idx, gate_w, tokens, capacity, 1, G->dgate);
    set_row_kernel(g, L, tokens, capacity);
    if ((rc = issue(g, dry, stream))) return rc;
    if ((rc = zero_tile_flags(L, dry, stream))) return rc;
  }
  // 3. wgrad-2: dW2[e] = (g dy)^T h_act  [d, f]
  {
    CcfGemmLaunch g = base_launch(L, early);
    set_a(g, L->grecv, L->max_rows, d, kMajMN);
    set_b(g, L->h_act, L->max_rows, f, kMajMN);
    g.epi = CCF_EPI_STORE;
    g.kgroup = 1;
    g.args.n = f;
    g.args.m_per_group = d;
    g.args.out0 = sgd2 ? const_cast<void*>(L->w2) : G->dw2;   // dgrad-2 above was the last reader of the old w2
    g.args.sgd_lr = sgd2 ? G->sgd_lr : 0.f;
    g.args.sgd_wd = sgd2 ? G->sgd_wd : 0.f;
    g.args.ld_out = f;
    g.few_rows = wgrad_few(rows_per_expert, g.args.sgd_lr != 0.f, L->two_cta);
    if ((rc = issue(g, dry, stream))) return rc;
  }
  if (G->db2 != nullptr && dry == nullptr) {
    if ((rc = ccf_colsum_grouped_hint(L->grecv, d, d, e_loc, L->group_base, L->group_rows, G->db2, L->fp16, rows_hint, stream))) return rc;
  }
  // 4. wgrad-1: dW1[e] = dh^T x_e  [f, d]  (SwiGLU: gate projection from dh, up projection from dh2)
  auto wgrad1 = [&](const void* a0, void* out) {
    CcfGemmLaunch g = base_launch(L, early);
    set_a(g, a0, L->max_rows, f, kMajMN);
    set_b(g, L->xrecv, L->max_rows, d, kMajMN);
    g.epi = CCF_EPI_STORE;
    g.kgroup = 1;
    g.args.n = d;
    g.args.m_per_group = f;
    g.args.out0 = out;
    g.args.sgd_lr = sgd ? G->sgd_lr : 0.f;
    g.args.sgd_wd = sgd ? G->sgd_wd : 0.f;
    g.args.ld_out = d;
    g.few_rows = wgrad_few(rows_per_expert, g.args.sgd_lr != 0.f, L->two_cta);
    return issue(g, dry, stream);
  };
  // 5. dgrad-1 + combine: dx rows go back to the ranks the tokens came from. Issued after the weight gradients (its
  // finish token then tells the sources that every buffer of this call is free), except when those update w1 / wg in
  // place: then it must read them first.
  auto dgrad1 = [&]() {
    CcfGemmLaunch g = base_launch(L, early);
    set_a(g, G->dh, L->max_rows, f, kMajK);
    g.epi = CCF_EPI_COMBINE;
    g.args.n = d;
    g.args.k = f;
    g.args.b_group_rows = f;
    g.args.ld_out = d;
    if (L->swiglu) {
      g.a1 = G->dh2;
      set_b(g, L->wg, static_cast<long long>(e_loc) * f, d, kMajMN);
      g.b1 = L->w1;
      g.args.kseg = 2;
    } else {
      set_b(g, L->w1, static_cast<long long>(e_loc) * f, d, kMajMN);
    }
    set_combine(g, L, L->peer_gcomb, nullptr);
    set_row_kernel(g, L, tokens, capacity);
    return issue(g, dry, stream);
  };
  if (sgd && (rc = dgrad1())) return rc;
  if (L->swiglu) {
    if ((rc = wgrad1(G->dh, sgd ? const_cast<void*>(L->wg) : G->dwg))) return rc;
    if ((rc = wgrad1(G->dh2, sgd ? const_cast<void*>(L->w1) : G->dw1))) return rc;
    if (dry == nullptr) {
      if (G->db1 != nullptr &&
          (rc = ccf_colsum_grouped_hint(G->dh2, f, f, e_loc, L->group_base, L->group_rows, G->db1, L->fp16, rows_hint, stream)))
        return rc;
      if (G->dbg != nullptr &&
          (rc = ccf_colsum_grouped_hint(G->dh, f, f, e_loc, L->group_base, L->group_rows, G->dbg, L->fp16, rows_hint, stream)))
        return rc;
    }
  } else {
    if ((rc = wgrad1(G->dh, sgd ? const_cast<void*>(L->w1) : G->dw1))) return rc;
    if (dry == nullptr && G->db1 != nullptr &&
        (rc = ccf_colsum_grouped_hint(G->dh, f, f, e_loc, L->group_base, L->group_rows, G->db1, L->fp16, rows_hint, stream)))
      return rc;
  }
  if (!sgd && (rc = dgrad1())) return rc;
  if ((rc = wait_and_reduce(L, L->gcomb, G->dx, tokens, G, idx, gate_w, early, dry, stream))) return rc;
  if (G->router_dw != nullptr && dry == nullptr)
    rc = ccf_router_dw(L->raw_order, L->count_raw, G->slot_grad, G->x, G->router_dw, G->router_db, tokens * L->top_k, d,
                       L->e_total, L->top_k, L->fp16, stream);
  return rc;
}

}  // namespace

extern "C" {

// The rule of row_kernel for a caller that issues the launches itself: out = {few_rows, two_cta, a_rows, bn}
int ccf_row_kernel(int epi, int b_major, int rows, int experts, int n, int capacity, int world, int small_rows, int two_cta, int* out) {
  const RowKernel r = row_kernel(epi, b_major, rows, experts, n, capacity, world, small_rows, two_cta);
  out[0] = r.few_rows;
  out[1] = r.two_cta;
  out[2] = r.a_rows;
  out[3] = r.bn;
  return 0;
}

int ccf_wgrad_few(int rows, int in_place, int two_cta) { return wgrad_few(rows, in_place != 0, two_cta); }

int ccf_sizeof_layer() { return static_cast<int>(sizeof(CcfLayer)); }
int ccf_sizeof_layer_grads() { return static_cast<int>(sizeof(CcfLayerGrads)); }

int ccf_layer_forward(const CcfLayer* L, const void* x, const int* idx, const float* gate_w, void* y, int tokens,
                      int capacity, int save_pre, int epoch, void* stream, CcfGemmLaunch* dry_gemms, int dry_cap,
                      int* dry_count) {
  if (L == nullptr || L->world < 1 || L->world > CCF_MAX_RANKS || L->e_total > CCF_MAX_GROUPS) return -2;
  Dry dry_state = {dry_gemms, dry_cap, 0};
  Dry* dry = dry_gemms != nullptr ? &dry_state : nullptr;
  const int rc = forward_pass(L, x, idx, gate_w, y, tokens, capacity, save_pre, epoch, stream, dry);
  if (dry_count != nullptr) *dry_count = dry_state.n;
  return end_of_pass(L, rc, dry, stream);
}

int ccf_layer_backward(const CcfLayer* L, const void* dy, const int* idx, const float* gate_w, const CcfLayerGrads* G,
                       int tokens, int capacity, void* stream, CcfGemmLaunch* dry_gemms, int dry_cap, int* dry_count) {
  if (L == nullptr || G == nullptr || L->world < 1 || L->world > CCF_MAX_RANKS) return -2;
  Dry dry_state = {dry_gemms, dry_cap, 0};
  Dry* dry = dry_gemms != nullptr ? &dry_state : nullptr;
  const int rc = backward_pass(L, dy, idx, gate_w, G, tokens, capacity, stream, dry);
  if (dry_count != nullptr) *dry_count = dry_state.n;
  return end_of_pass(L, rc, dry, stream);
}

}  // extern "C"
