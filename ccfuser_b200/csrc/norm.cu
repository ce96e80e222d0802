// LayerNorm forward and backward for 2-byte activations, fp32 statistics: one warp per row forward, up to eight backward.
//
// The transformer blocks around the MoE layers (the reference's example models are stock GPT-2 / BERT / Transformer-XL,
// mix_moe/mix_moe/examples/models/moe_gpt.py, moe_bert.py, transformer-xl/mem_transformer_mix_moe.py) normalise a
// [tokens, d_model] matrix twice per block. Both passes are bound by reading and writing that matrix once; the
// backward also reduces the weight and bias gradients over all rows: per-thread partial sums over the rows a thread visits,
// one partial row per block, added in block order by a second small kernel.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "dispatch.cuh"   // pack2 / unpack2
#include "norm.h"
#include "sm100.cuh"

namespace ccf {

constexpr int kLnThreads = 256;
constexpr int kLnWarps = kLnThreads / 32;

// Blocks of the forward kernel per SM: as many as the registers of its packed rows allow.
template <int kV>
constexpr int kLnBlocks = kV >= 8 ? 2 : kV >= 4 ? 3 : 4;

// kV = 16-byte pieces of a row per lane (row length <= 256 * kV elements). Bound by reading x and writing y once. The grid is one
// wave, each warp walks rows `warps` apart and requests its next row before it works on the current one: with a block per eight
// rows the launch ran its waves one after the other, each of them a load, two reductions and a store. gamma and beta stay in
// shared memory. Cold, in a graph, before and now, us: 16384 x 2048 38.4 and 29.0 (4.6 TB/s), 8192 x 2048 20.5 and 17.7,
// 2048 x 2048 9.2 and 7.3, 8192 x 768 9.9 and 8.4, 16 x 2048 5.9 and 3.7, 4100 x 264 (one wave either way) 3.7 and 3.9.
template <int kV>
__global__ void __launch_bounds__(kLnThreads, kLnBlocks<kV>)
layernorm_fwd_kernel(const void* __restrict__ x, const void* __restrict__ gamma, const void* __restrict__ beta, void* __restrict__ y,
                     float* __restrict__ mean_out, float* __restrict__ rstd_out, int rows, int d, float eps, int fp16) {
  __shared__ uint4 gs[32 * kV], bs[32 * kV];
  const int lane = threadIdx.x & 31, vecs = d >> 3;
  const uint32_t warps = gridDim.x * kLnWarps, n_rows = static_cast<uint32_t>(rows);
  uint32_t row = blockIdx.x * kLnWarps + (threadIdx.x >> 5);
  // the row stays packed (8 registers per 16-byte piece instead of 16 floats)
  uint4 xn[kV];
  auto fetch = [&](uint32_t r) {
#pragma unroll
    for (int i = 0; i < kV; ++i) {
      const int v = lane + 32 * i;
      xn[i] = make_uint4(0, 0, 0, 0);
      if (r < n_rows && v < vecs) xn[i] = __ldg(reinterpret_cast<const uint4*>(x) + static_cast<size_t>(r) * vecs + v);
    }
  };
  fetch(row);
  for (int v = threadIdx.x; v < vecs; v += kLnThreads) {
    gs[v] = __ldg(reinterpret_cast<const uint4*>(gamma) + v);
    bs[v] = beta != nullptr ? __ldg(reinterpret_cast<const uint4*>(beta) + v) : make_uint4(0, 0, 0, 0);
  }
  __syncthreads();
  for (; row < n_rows; row += warps) {
    uint4 xv[kV];
#pragma unroll
    for (int i = 0; i < kV; ++i) xv[i] = xn[i];
    fetch(row + warps);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < kV; ++i) {
      const uint32_t q[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 t = unpack2(q[j], fp16);
        sum += t.x + t.y;
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const float mean = sum / d;
    float var = 0.f;
#pragma unroll
    for (int i = 0; i < kV; ++i) {
      if (lane + 32 * i < vecs) {
        const uint32_t q[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 t = unpack2(q[j], fp16);
          const float c0 = t.x - mean, c1 = t.y - mean;
          var = fmaf(c0, c0, fmaf(c1, c1, var));
        }
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) var += __shfl_xor_sync(0xffffffffu, var, off);
    const float rstd = rsqrtf(var / d + eps);
    if (lane == 0) {
      mean_out[row] = mean;
      rstd_out[row] = rstd;
    }
    uint4* yr = reinterpret_cast<uint4*>(y) + static_cast<size_t>(row) * vecs;
#pragma unroll
    for (int i = 0; i < kV; ++i) {
      const int v = lane + 32 * i;
      if (v >= vecs) continue;
      const uint4 g = gs[v], b = bs[v];
      const uint32_t xq[4] = {xv[i].x, xv[i].y, xv[i].z, xv[i].w}, gq[4] = {g.x, g.y, g.z, g.w}, bq[4] = {b.x, b.y, b.z, b.w};
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 xf = unpack2(xq[j], fp16), gf = unpack2(gq[j], fp16), bf = unpack2(bq[j], fp16);
        o[j] = pack2((xf.x - mean) * rstd * gf.x + bf.x, (xf.y - mean) * rstd * gf.y + bf.y, fp16);
      }
      yr[v] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// Backward. With xh = (x - mean) * rstd and g = dy * gamma:
//   dx = rstd * (g - mean_row(g) - xh * mean_row(g * xh)),   dgamma = sum_rows dy * xh,   dbeta = sum_rows dy.
// Bound by reading x and dy and writing dx once. kW warps share a row, eight columns per thread, so that a thread meets
// the same columns in every row it visits and its dgamma / dbeta sums are 16 registers (a warp per row needed a whole row's:
// one block per SM, and a second pass over x and dy instead). The rows of a block arrive by bulk copies, up to kLnStages
// pairs of row groups ahead: with loads to registers 16 warps per SM held 32 KB in flight, a third of what the memory
// rate takes. The row sums meet in shared memory with one barrier per stage, which also frees the stage, and each block
// leaves its partial dgamma / dbeta in `part` ([blocks, 2, d] fp32), which layernorm_bwd_finish_kernel adds in block order:
// no atomics, no zeroed buffers, no conversion passes. A copy that does not arrive within the limit ends the block: time-out
// in the status word, no further requests, NaN in the rows it leaves undone and in its partial sums. 8192 x 2048 bf16:
// 39 + 7 us, where a dx kernel, a parameter kernel, two fills and two conversions took 37 + 16 + 6 us and four launches more.
constexpr int kLnRows = 2;       // rows per group and stage
constexpr int kLnStages = 6;
template <int kW>
__global__ void __launch_bounds__(256, 2) layernorm_bwd_kernel(const void* __restrict__ x, const void* __restrict__ dy,
                                                               const void* __restrict__ gamma, const float* __restrict__ mean_in,
                                                               const float* __restrict__ rstd_in, void* __restrict__ dx,
                                                               float* __restrict__ part, int rows, int d, int fp16,
                                                               int* status, unsigned long long wait_limit_ns) {
  constexpr int kG = kLnWarps / kW;             // rows that a block works on side by side
  constexpr int kStageRows = kG * kLnRows;      // consecutive rows: at most 8 KB each of x and dy
  extern __shared__ __align__(16) uint8_t ln_ring[];   // [kLnStages][x rows, dy rows]
  __shared__ float2 red[2][kG][kLnRows][kW];
  __shared__ float psum[kG > 1 ? kG - 1 : 1][2][kW * 256];
  __shared__ __align__(8) uint64_t full[kLnStages];
  __shared__ int abort_word, lost_at;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grp = warp / kW, wr = warp % kW;
  const int v = wr * 32 + lane, vecs = d >> 3;  // this thread's 16-byte piece of a row
  const bool col_on = v < vecs;
  const uint32_t row_bytes = static_cast<uint32_t>(d) * 2u, half = kStageRows * row_bytes;
  const uint32_t ring = smem_u32(ln_ring);
  float pg[8] = {0, 0, 0, 0, 0, 0, 0, 0}, pb[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  uint4 g4 = make_uint4(0, 0, 0, 0);
  if (col_on) g4 = __ldg(reinterpret_cast<const uint4*>(gamma) + v);
  const uint32_t gq[4] = {g4.x, g4.y, g4.z, g4.w};
  const int step = static_cast<int>(gridDim.x) * kStageRows;
  if (threadIdx.x == 0) {
    abort_word = 0;
    lost_at = 0x7fffffff;
    for (int k = 0; k < kLnStages; ++k) mbar_init(smem_u32(&full[k]), 1);
    fence_barrier_init();
  }
  __syncthreads();
  auto request = [&](int base, int slot) {      // thread 0
    if (base >= rows) return;
    const uint32_t bytes = static_cast<uint32_t>(min(kStageRows, rows - base)) * row_bytes, bar = smem_u32(&full[slot]);
    const size_t off = static_cast<size_t>(base) * row_bytes;
    mbar_arrive_expect_tx(bar, 2 * bytes);
    bulk_load(ring + slot * 2 * half, reinterpret_cast<const uint8_t*>(x) + off, bytes, bar);
    bulk_load(ring + slot * 2 * half + half, reinterpret_cast<const uint8_t*>(dy) + off, bytes, bar);
  };
  float mn[kLnRows], rn[kLnRows];
  auto stats = [&](int base) {                  // one stage ahead of their use
#pragma unroll
    for (int u = 0; u < kLnRows; ++u) {
      const int row = base + u * kG + grp;
      mn[u] = row < rows ? __ldg(mean_in + row) : 0.f;
      rn[u] = row < rows && col_on ? __ldg(rstd_in + row) : 0.f;   // 0: pieces outside contribute nothing below
    }
  };
  int buf = 0, slot = 0, parity = 0;
  bool lost = false;
  int base = static_cast<int>(blockIdx.x) * kStageRows;
  if (threadIdx.x == 0)
    for (int k = 0; k < kLnStages; ++k) request(base + k * step, k);
  stats(base);
  for (; base < rows; base += step, buf ^= 1) {   // the same trips for every thread of the block
    uint4 xv[kLnRows], dv[kLnRows];
    float mu[kLnRows], rs[kLnRows];
    // the full limit whatever is on record: these copies depend on no peer, so a lost one is no reason to give them up sooner
    const bool here = mbar_wait(smem_u32(&full[slot]), parity, &abort_word, wait_limit_ns);
#pragma unroll
    for (int u = 0; u < kLnRows; ++u) {
      const int r = u * kG + grp;
      xv[u] = make_uint4(0, 0, 0, 0);
      dv[u] = make_uint4(0, 0, 0, 0);
      if (base + r < rows && col_on) {
        const uint8_t* at = ln_ring + slot * 2 * half + r * row_bytes + v * 16;
        xv[u] = *reinterpret_cast<const uint4*>(at);
        dv[u] = *reinterpret_cast<const uint4*>(at + half);
      }
      mu[u] = mn[u];
      rs[u] = rn[u];
    }
    stats(base + step);
    float s1[kLnRows], s2[kLnRows];
#pragma unroll
    for (int u = 0; u < kLnRows; ++u) {
      const uint32_t xq[4] = {xv[u].x, xv[u].y, xv[u].z, xv[u].w}, dq[4] = {dv[u].x, dv[u].y, dv[u].z, dv[u].w};
      s1[u] = s2[u] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 xf = unpack2(xq[j], fp16), df = unpack2(dq[j], fp16), gf = unpack2(gq[j], fp16);
        const float h0 = (xf.x - mu[u]) * rs[u], h1 = (xf.y - mu[u]) * rs[u];
        const float g0 = df.x * gf.x, g1 = df.y * gf.y;
        s1[u] += g0 + g1;
        s2[u] = fmaf(g0, h0, fmaf(g1, h1, s2[u]));
        pg[2 * j] = fmaf(df.x, h0, pg[2 * j]);
        pg[2 * j + 1] = fmaf(df.y, h1, pg[2 * j + 1]);
        pb[2 * j] += df.x;
        pb[2 * j + 1] += df.y;
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
      for (int u = 0; u < kLnRows; ++u) {
        s1[u] += __shfl_xor_sync(0xffffffffu, s1[u], off);
        s2[u] += __shfl_xor_sync(0xffffffffu, s2[u], off);
      }
    }
    if constexpr (kW > 1) {
      if (lane == 0) {
#pragma unroll
        for (int u = 0; u < kLnRows; ++u) red[buf][grp][u][wr] = make_float2(s1[u], s2[u]);
      }
    }
    if (!here) lost_at = base;
    __syncthreads();   // row sums are there and the stage has been read; `red`'s other half is written after the next one
    // a thread that gave up its wait takes the whole block out of the loop: every thread sees the same pass number here, even if
    // one that is already in the next pass has written that pass's (a barrier with a reduction in it took 0.5 us of 28 more)
    lost = *const_cast<volatile int*>(&lost_at) <= base;
    if (lost) break;
    if (threadIdx.x == 0) request(base + kLnStages * step, slot);
    if (++slot == kLnStages) { slot = 0; parity ^= 1; }
    if constexpr (kW > 1) {
#pragma unroll
      for (int u = 0; u < kLnRows; ++u) {
        s1[u] = s2[u] = 0.f;
#pragma unroll
        for (int k = 0; k < kW; ++k) {
          const float2 r = red[buf][grp][u][k];
          s1[u] += r.x;
          s2[u] += r.y;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < kLnRows; ++u) {
      const int row = base + u * kG + grp;
      if (row >= rows || !col_on) continue;
      const float m1 = s1[u] / d, m2 = s2[u] / d;
      const uint32_t xq[4] = {xv[u].x, xv[u].y, xv[u].z, xv[u].w}, dq[4] = {dv[u].x, dv[u].y, dv[u].z, dv[u].w};
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 xf = unpack2(xq[j], fp16), df = unpack2(dq[j], fp16), gf = unpack2(gq[j], fp16);
        const float h0 = (xf.x - mu[u]) * rs[u], h1 = (xf.y - mu[u]) * rs[u];
        o[j] = pack2(rs[u] * (df.x * gf.x - m1 - h0 * m2), rs[u] * (df.y * gf.y - m1 - h1 * m2), fp16);
      }
      reinterpret_cast<uint4*>(dx)[static_cast<size_t>(row) * vecs + v] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
  if (lost) {
    if (threadIdx.x == 0) report_status(status, CCF_ERR_MBAR_TIMEOUT, 0x50);
    for (; base < rows; base += step) {
      for (int u = 0; u < kLnRows; ++u) {
        const int row = base + u * kG + grp;
        if (row < rows && col_on)   // 0x7fff: NaN in both element types
          reinterpret_cast<uint4*>(dx)[static_cast<size_t>(row) * vecs + v] = make_uint4(0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu);
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) pg[i] = pb[i] = __int_as_float(0x7fc00000);
    // give copies still in flight time to land before the shared memory goes away
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 50000ull) __nanosleep(1000);
  }
  // the block's row groups add up, then one partial row of dgamma and of dbeta per block
  if constexpr (kG > 1) {
    if (grp > 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        psum[grp - 1][0][i * (kW * 32) + v] = pg[i];
        psum[grp - 1][1][i * (kW * 32) + v] = pb[i];
      }
    }
    __syncthreads();
    if (grp == 0) {
      for (int k = 0; k < kG - 1; ++k) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          pg[i] += psum[k][0][i * (kW * 32) + v];
          pb[i] += psum[k][1][i * (kW * 32) + v];
        }
      }
    }
  }
  if (grp == 0 && col_on) {
    float4* og = reinterpret_cast<float4*>(part + static_cast<size_t>(blockIdx.x) * 2 * d) + 2 * v;
    og[0] = make_float4(pg[0], pg[1], pg[2], pg[3]);
    og[1] = make_float4(pg[4], pg[5], pg[6], pg[7]);
    float4* ob = og + (d >> 2);
    ob[0] = make_float4(pb[0], pb[1], pb[2], pb[3]);
    ob[1] = make_float4(pb[4], pb[5], pb[6], pb[7]);
  }
}

// Block: 32 columns of dgamma (blockIdx.y = 0) or dbeta (1), 8 lanes over the partial rows.
__global__ void __launch_bounds__(256) layernorm_bwd_finish_kernel(const float* __restrict__ part, int blocks, int d, void* dgamma,
                                                                   void* dbeta, int fp16) {
  __shared__ float red[8][32];
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), ly = threadIdx.x >> 5;
  float s = 0.f;
  if (c < d) {
#pragma unroll 8
    for (int b = ly; b < blocks; b += 8) s += __ldg(part + (static_cast<size_t>(b) * 2 + blockIdx.y) * d + c);
  }
  red[ly][threadIdx.x & 31] = s;
  __syncthreads();
  if (ly == 0 && c < d) {
#pragma unroll
    for (int k = 1; k < 8; ++k) s += red[k][threadIdx.x];
    void* out = blockIdx.y == 0 ? dgamma : dbeta;
    if (fp16) reinterpret_cast<__half*>(out)[c] = __float2half(s);
    else reinterpret_cast<__nv_bfloat16*>(out)[c] = __float2bfloat16(s);
  }
}

// blocks of the backward kernel = rows of its partial-sum buffer: two per SM, fewer for few rows
static int ln_bwd_blocks(int rows, int d) {
  const int w = (d + 255) / 256, kw = w <= 1 ? 1 : w <= 2 ? 2 : w <= 4 ? 4 : 8;
  const int per = kLnWarps / kw * kLnRows, blocks = (rows + per - 1) / per;
  return blocks < 2 * 148 ? blocks : 2 * 148;
}

// The kernels move 16 bytes at a time.
template <typename... T>
static bool aligned16(const T*... p) {
  return ((reinterpret_cast<uintptr_t>(p) | ...) & 15) == 0;
}

template <int kV>
static int launch_ln_fwd(const void* x, const void* gamma, const void* beta, void* out, float* mean, float* rstd, int rows, int d,
                         float eps, int fp16, cudaStream_t st) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int need = (rows + kLnWarps - 1) / kLnWarps, wave = kLnBlocks<kV> * (sms > 0 ? sms : 1), blocks = need < wave ? need : wave;
  layernorm_fwd_kernel<kV><<<blocks, kLnThreads, 0, st>>>(x, gamma, beta, out, mean, rstd, rows, d, eps, fp16);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -static_cast<int>(e);
}

}  // namespace ccf

extern "C" {

// Largest row length the kernels take (8 pieces of 16 bytes per lane).
int ccf_layernorm_max_d() { return 2048; }

// y = (x - mean) * rstd * gamma + beta over the last dimension of x [rows, d] (2-byte elements, gamma / beta of the same
// type, beta may be null); mean and rstd [rows] fp32 are written for the backward pass. d % 8 == 0, d <= 2048, x, y, gamma and
// beta on 16-byte boundaries.
int ccf_layernorm_fwd(const void* x, const void* gamma, const void* beta, void* y, float* mean, float* rstd, int rows,
                      int d, float eps, int fp16, void* stream) {
  using namespace ccf;
  if (rows < 1 || d < 8 || d % 8 != 0 || d > 2048 || !aligned16(x, gamma, beta, y)) return -2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (d <= 512) return launch_ln_fwd<2>(x, gamma, beta, y, mean, rstd, rows, d, eps, fp16, st);
  if (d <= 1024) return launch_ln_fwd<4>(x, gamma, beta, y, mean, rstd, rows, d, eps, fp16, st);
  return launch_ln_fwd<8>(x, gamma, beta, y, mean, rstd, rows, d, eps, fp16, st);
}

// Rows of the partial-sum buffer that ccf_layernorm_bwd needs for this size.
int ccf_layernorm_bwd_parts(int rows, int d) { return rows < 1 || d < 8 ? 0 : ccf::ln_bwd_blocks(rows, d); }

// dx [rows, d], dgamma [d] and dbeta [d] (element type; dbeta may be null) are written. `part`: scratch of
// ccf_layernorm_bwd_parts(rows, d) x 2 x d floats; it, x, dy, gamma and dx on 16-byte boundaries. A wait that exceeds the
// limit goes to `status`.
int ccf_layernorm_bwd(const void* x, const void* dy, const void* gamma, const float* mean, const float* rstd, void* dx,
                      float* part, void* dgamma, void* dbeta, int rows, int d, int fp16, int* status,
                      unsigned long long wait_limit_ns, void* stream) {
  using namespace ccf;
  if (rows < 1 || d < 8 || d % 8 != 0 || d > 2048 || !aligned16(x, dy, gamma, dx, part)) return -2;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int blocks = ln_bwd_blocks(rows, d);
  const int w = (d + 255) / 256, kw = w <= 1 ? 1 : w <= 2 ? 2 : w <= 4 ? 4 : 8;
  const int smem = kLnStages * 2 * (kLnWarps / kw * kLnRows) * d * 2;   // at most 96 KB
  auto kern = d <= 256 ? layernorm_bwd_kernel<1> : d <= 512 ? layernorm_bwd_kernel<2> : d <= 1024 ? layernorm_bwd_kernel<4>
                                                                                    : layernorm_bwd_kernel<8>;
  static bool configured[64][4] = {};   // per device and instantiation: the attribute belongs to the (function, device) pair
  int dev = 0;
  cudaGetDevice(&dev);
  bool& set = configured[dev & 63][kw == 1 ? 0 : kw == 2 ? 1 : kw == 4 ? 2 : 3];
  if (!set) {
    const cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kLnStages * 16384);
    if (err != cudaSuccess) return -static_cast<int>(err);
    set = true;
  }
  kern<<<blocks, 256, smem, st>>>(x, dy, gamma, mean, rstd, dx, part, rows, d, fp16, status, wait_limit_ns);
  layernorm_bwd_finish_kernel<<<dim3((d + 31) / 32, dbeta != nullptr ? 2 : 1), 256, 0, st>>>(part, blocks, d, dgamma, dbeta, fp16);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -static_cast<int>(e);
}

}  // extern "C"
