// Last kernels of a pass over one layer: the slot reduction (forward output, input gradient) and the router's backward.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "combine.h"
#include "dispatch.cuh"
#include "gemm_args.h"
#include "sm100.cuh"

namespace ccf {

constexpr int kMaxK = 8;
constexpr int kReduceThreads = 256;
// 16-byte pieces of the result per thread: with one slot per token a single row read would not cover the memory latency
__host__ __device__ constexpr int reduce_pieces(int k) { return k == 1 ? 2 : 1; }

__device__ __forceinline__ void add_piece(float (&acc)[8], const uint4& x, float scale, int fp16) {
  const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 f = unpack2(w[q], fp16);
    acc[2 * q] = fmaf(scale, f.x, acc[2 * q]);
    acc[2 * q + 1] = fmaf(scale, f.y, acc[2 * q + 1]);
  }
}

// y[t, :] = sum_j keep(t, j) * comb[t * k + j, :] in fp32, one rounding. Bound by reading k rows and writing one per token. kK is
// the number of slots per token (0: more than eight, eight at a time), so that all rows of a piece are requested before the first
// is used, and none besides. 8192 x 4096, us with 1 / 2 / 3 / 4 / 8 slots: 30 / 41 / 76 / 79 / 99 with whole tokens per block and one
// form for three to eight slots, now 23 / 36 / 42 / 49 / 91; one token of 8192 columns, two slots: 3.2, now 1.9. With kRouter the
// same pass adds the router's share of the input gradient, sum_j g_j Wg[idx_j, :] (Wg is small and stays in L2), which as a kernel
// of its own wrote and re-read a [T, d] matrix: 16384 x 4096, top-2: 91 us, from 81 + 42 + 59 us (reduce, router dx, addition of
// the two gradients).
template <int kK, bool kRouter>
__global__ void __launch_bounds__(kReduceThreads) combine_reduce_kernel(const __grid_constant__ CcfReduceArgs a) {
  const int vecs = a.d >> 3, K = kK > 0 ? kK : a.top_k, fp16 = a.fp16;
  after_previous();
  if (blockIdx.x == 0 && a.done != nullptr) {
    if (threadIdx.x == 0) {
      const int target = *a.cum + *a.sent_rows * a.n_tiles + 1;
      if (!wait_flag_ge(a.done, target, fail_fast_limit(a.status, a.wait_limit_ns)))
        report_status(a.status, CCF_ERR_FLAG_TIMEOUT, 0x400000);
      *a.cum = target;
    }
    for (int i = threadIdx.x; i < a.zero_count; i += kReduceThreads) a.zero_words[i] = 0;
  }
  const uint4* comb = behind(reinterpret_cast<const uint4*>(a.comb));
  const uint4* wg = behind(reinterpret_cast<const uint4*>(a.wg));
  const int *const slot_row = behind(a.slot_row), *const idx = behind(a.idx);
  const float* const gate_w = behind(a.w);
  constexpr int kP = reduce_pieces(kK), kSpan = kReduceThreads * kP, kN = kK > 0 ? kK : kMaxK;
  // pieces kSpan * block + thread (+ 256, ...) of [tokens, vecs], without a product that may not fit 32 bits: `vecs` blocks are
  // kSpan tokens
  const int i0 = static_cast<int>(blockIdx.x % vecs) * kSpan + threadIdx.x, tb = static_cast<int>(blockIdx.x / vecs) * kSpan;
  uint4 x[kP][kN];
  bool on[kP][kN];
  auto fetch = [&](int p, int j0) {
    const int i = i0 + p * kReduceThreads, t = tb + i / vecs, v = i % vecs;
    const size_t s0 = static_cast<size_t>(t) * K + j0;
#pragma unroll
    for (int j = 0; j < kN; ++j) {
      on[p][j] = t < a.tokens && j0 + j < K && __ldg(slot_row + s0 + j) >= 0;
      x[p][j] = make_uint4(0u, 0u, 0u, 0u);
      if (on[p][j]) x[p][j] = comb[(s0 + j) * vecs + v];
    }
  };
  if constexpr (kK > 0) {
#pragma unroll
    for (int p = 0; p < kP; ++p) fetch(p, 0);
  }
#pragma unroll
  for (int p = 0; p < kP; ++p) {
    const int i = i0 + p * kReduceThreads, t = tb + i / vecs, v = i % vecs;
    if (t >= a.tokens) break;
    const size_t s0 = static_cast<size_t>(t) * K;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int j0 = 0; j0 < K; j0 += kN) {   // once, except for more than kMaxK slots per token
      if constexpr (kK == 0) fetch(p, j0);
#pragma unroll
      for (int j = 0; j < kN; ++j)
        if (on[p][j]) add_piece(acc, x[p][j], 1.f, fp16);
    }
    if constexpr (kRouter) {
      float w[kN], dw[kN];
      float dot = 0.f;
#pragma unroll
      for (int j = 0; j < kN; ++j) {
        w[j] = j < K ? __ldg(gate_w + s0 + j) : 0.f;
        dw[j] = on[p][j] ? a.dw[s0 + j] : 0.f;
        dot = fmaf(w[j], dw[j], dot);
      }
#pragma unroll
      for (int j = 0; j < kN; ++j) {
        if (j >= K) continue;
        const int e = __ldg(idx + s0 + j);
        const bool routed = e >= 0 && e < a.e;
        const float g = routed ? w[j] * (dw[j] - dot) : 0.f;
        if (v == 0) a.g[s0 + j] = g;
        if (routed) add_piece(acc, __ldg(wg + static_cast<size_t>(e) * vecs + v), g, fp16);
      }
    }
    uint4 o;
    o.x = pack2(acc[0], acc[1], fp16);
    o.y = pack2(acc[2], acc[3], fp16);
    o.z = pack2(acc[4], acc[5], fp16);
    o.w = pack2(acc[6], acc[7], fp16);
    reinterpret_cast<uint4*>(a.y)[static_cast<size_t>(t) * vecs + v] = o;
  }
}

// The gradient of the logits is non-zero only in the k selected columns, so dWg is a sum of scaled token rows per expert.
// The routing kernel left the slots listed by expert: a block sums 128 columns over one expert's list (16 row lanes, four
// rows in flight per thread), and a cluster of up to 8 blocks shares a long list, its first block adding their partial sums
// in a fixed order. x is read top_k times, from L2 after the first; products and sums are fp32 and the result is
// rounded once, where scattering into shared memory needed atomics, a zeroed fp32 result and a conversion pass, and the
// dense [T, 128] gradient for a tensor-core product needed ten small launches around it.
__global__ void __launch_bounds__(256) router_dw_kernel(const int* __restrict__ raw_order, const int* __restrict__ count_raw,
                                                        const float* __restrict__ g_slot, const void* __restrict__ x, void* dwg,
                                                        void* db, int d, int top_k, int fp16) {
  __shared__ float red[16][128];
  __shared__ float redg[16];
  __shared__ float part[128];
  __shared__ float partg;
  const int e = blockIdx.y, nr = count_raw[e];
  const int* list = raw_order + CCF_MAX_GROUPS + __ldg(raw_order + e);   // both reads on their way before either is needed
  const int split = blockIdx.z, splits = splits_with_work(nr, gridDim.z);
  if (split >= splits) return;
  const int cx = threadIdx.x & 15, ry = threadIdx.x >> 4;
  const int col = blockIdx.x * 128 + cx * 8;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  float sum_g = 0.f;
  const uint16_t* base = reinterpret_cast<const uint16_t*>(x) + col;
  // the slot ids are read one pass ahead: otherwise every pass waits for two dependent reads
  int s_next[4];
  auto fetch = [&](int r) {
#pragma unroll
    for (int u = 0; u < 4; ++u) s_next[u] = r + 16 * u < nr ? __ldg(list + r + 16 * u) : -1;
  };
  fetch(split * 64 + ry);
  for (int r = split * 64 + ry; r < nr; r += 64 * splits) {
    float g[4];
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int s = s_next[u];
      g[u] = s >= 0 ? __ldg(g_slot + s) : 0.f;
      v[u] = s >= 0 && col < d ? __ldg(reinterpret_cast<const uint4*>(base + static_cast<size_t>(s / top_k) * d))
                               : make_uint4(0u, 0u, 0u, 0u);
    }
    fetch(r + 64 * splits);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      add_piece(acc, v[u], g[u], fp16);
      sum_g += g[u];
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) red[ry][cx * 8 + i] = acc[i];
  if (cx == 0) redg[ry] = sum_g;
  __syncthreads();
  float s = 0.f, sg = 0.f;
  if (threadIdx.x < 128) {
#pragma unroll
    for (int i = 0; i < 16; ++i) { s += red[i][threadIdx.x]; sg += redg[i]; }
    part[threadIdx.x] = s;
    if (threadIdx.x == 0) partg = sg;
  }
  if (splits > 1) {
    cluster_sync_all();
    if (split == 0 && threadIdx.x < 128) {
      const uint32_t mine = smem_u32(&part[threadIdx.x]), mineg = smem_u32(&partg);
      for (int r = 1; r < splits; ++r) {
        s += ld_cluster_f32(map_to_cta(mine, r));
        if (threadIdx.x == 0) sg += ld_cluster_f32(map_to_cta(mineg, r));
      }
    }
    cluster_sync_all();   // no block leaves while its partial sums may still be read
  }
  if (split != 0 || threadIdx.x >= 128) return;
  const int c = blockIdx.x * 128 + threadIdx.x;
  if (c < d) {
    if (fp16) reinterpret_cast<__half*>(dwg)[static_cast<size_t>(e) * d + c] = __float2half(s);
    else reinterpret_cast<__nv_bfloat16*>(dwg)[static_cast<size_t>(e) * d + c] = __float2bfloat16(s);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && db != nullptr) {
    if (fp16) reinterpret_cast<__half*>(db)[e] = __float2half(sg);
    else reinterpret_cast<__nv_bfloat16*>(db)[e] = __float2bfloat16(sg);
  }
}

}  // namespace ccf

extern "C" {

int ccf_reduce(const CcfReduceArgs* a, void* stream) {
  using namespace ccf;
  if (a->d < 8 || a->d % 8 != 0 || a->top_k < 0) return -2;
  if (a->wg != nullptr && (a->top_k > kMaxK || a->top_k < 1)) return -2;
  if (a->tokens == 0 && a->done == nullptr) return 0;
  const int span = kReduceThreads * reduce_pieces(a->top_k);
  long long blocks = (static_cast<long long>(a->tokens) * (a->d >> 3) + span - 1) / span;
  if (blocks > 0x7fffffffLL) return -2;
  if (blocks < 1) blocks = 1;    // a call without tokens still consumes its completion count
  using Kernel = void (*)(CcfReduceArgs);
  static const Kernel plain[kMaxK + 1] = {combine_reduce_kernel<0, false>, combine_reduce_kernel<1, false>, combine_reduce_kernel<2, false>,
                                          combine_reduce_kernel<3, false>, combine_reduce_kernel<4, false>, combine_reduce_kernel<5, false>,
                                          combine_reduce_kernel<6, false>, combine_reduce_kernel<7, false>, combine_reduce_kernel<8, false>};
  static const Kernel router[kMaxK + 1] = {nullptr, combine_reduce_kernel<1, true>, combine_reduce_kernel<2, true>,
                                           combine_reduce_kernel<3, true>, combine_reduce_kernel<4, true>, combine_reduce_kernel<5, true>,
                                           combine_reduce_kernel<6, true>, combine_reduce_kernel<7, true>, combine_reduce_kernel<8, true>};
  const Kernel kern = a->wg != nullptr ? router[a->top_k] : plain[a->top_k > kMaxK ? 0 : a->top_k];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(kReduceThreads);
  cfg.stream = reinterpret_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1] = {early_attribute()};
  cfg.attrs = attr;
  cfg.numAttrs = a->early;
  cudaError_t err = cudaLaunchKernelEx(&cfg, kern, *a);
  return err == cudaSuccess ? 0 : -static_cast<int>(err);
}

int ccf_router_dw(const int* raw_order, const int* count_raw, const float* g, const void* x, void* dwg, void* db, int slots, int d,
                  int e, int top_k, int fp16, void* stream) {
  using namespace ccf;
  if (d < 8 || d % 8 != 0 || e < 1 || e > CCF_MAX_GROUPS || top_k < 1 || (reinterpret_cast<uintptr_t>(x) & 15)) return -2;
  const int splits = group_splits((d + 127) / 128 * e, slots / e);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((d + 127) / 128, e, splits);
  cfg.blockDim = dim3(256);
  cfg.stream = reinterpret_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1] = {cluster_attribute(1, 1, splits)};
  cfg.attrs = attr;
  cfg.numAttrs = splits > 1 ? 1 : 0;
  cudaError_t err = cudaLaunchKernelEx(&cfg, router_dw_kernel, raw_order, count_raw, g, x, dwg, db, d, top_k, fp16);
  return err == cudaSuccess ? 0 : -static_cast<int>(err);
}

}  // extern "C"
