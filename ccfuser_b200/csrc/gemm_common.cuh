// Pieces shared by the one-CTA (gemm.cu) and two-CTA (gemm2.cu) grouped GEMM kernels: tile geometry, epilogue
// arithmetic, staged row I/O, the per-tile epilogue and the optional trace.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "dispatch.cuh"
#include "gemm_args.h"
#include "sm100.cuh"

namespace ccf {

constexpr int BM = 128, BN = 256, BK = 64, UK = 16;
constexpr int kEpiWarps = 8;            // two per TMEM lane quarter, each takes half of the columns
// Two more warps per CTA exist only for the dispatch role: with them the row push runs next to the MMA and epilogue warps
// (which start on the tiles made of this rank's own rows) instead of in front of the epilogue.
constexpr int kCommWarps = 2;
constexpr int kThreads = 64 + 32 * kEpiWarps + 32 * kCommWarps;
constexpr int kTmemCols = 512;
constexpr int MAJ_K = 0, MAJ_MN = 1;
constexpr int kEpiStageBytes = 2048;  // per epilogue warp: 32 rows x 64 bytes, XOR-swizzled

// Host: tensor map of a 2-D row-major view [rows, cols] of 2-byte elements, rows ld elements apart (0: cols), with box {box_cols,
// box_rows} (defined in gemm.cu). A box is as wide as its swizzle: 64 columns for the operands of an MMA (128 bytes), 32 for the staging
// areas of the epilogues (64 bytes, stage_off); no other width is taken. Returns 0 or a negative error code.
int make_tmap(CUtensorMap* m, const void* base, long long rows, long long cols, int box_cols, int box_rows, int fp16, long long ld = 0);

// Descriptor of an operand in a pipeline stage as the MMA reads it: its base, the step of one 16-deep MMA, and any other place in
// shared memory (only the 14 address bits differ, in units of 16 bytes; shared memory ends below 2^18).
__device__ __forceinline__ uint64_t operand_desc(uint32_t smem_addr, int major) {
  return major == MAJ_K ? make_smem_desc(smem_addr, 16, 1024) : make_smem_desc(smem_addr, 8192, 1024);
}
__device__ __forceinline__ constexpr uint32_t desc_step(int major) { return major == MAJ_K ? 32 : 2048; }
__device__ __forceinline__ uint64_t desc_at(uint64_t base, uint32_t bytes) { return base + (bytes >> 4); }

struct Tile {
  int g;           // group (expert)
  int row0;        // row-grouped: first A/C row; k-grouped: first output row inside the group (m0)
  int n0;          // first output column (for SWIGLU: first *output* column, 128 per tile)
  int rows_valid;  // valid rows of the tile
  int kblocks;     // 64-deep reduction steps
  int krow0;       // k-grouped: first reduction row
};

// ---------------------------------------------------------------------------------------------------
// epilogue math
// ---------------------------------------------------------------------------------------------------
// The normal distribution function, 1/2 + x Q(x^2), saturated to [0, 1]: Q is a degree-8 polynomial in x^2 (erf(z) ~= z P(z^2) on
// |z| <= 3, fitted minimax-style, with z = x / sqrt 2 folded into the coefficients; |error| <= 1.3e-5 in fp32 Horner form), x^2 held at
// its end of the range, 18. Beyond it x Q(18) passes 1/2 and the saturation gives 0 and 1 themselves. No MUFU operation and no branch:
// libm's erff and the exp/rcp-based forms kept the SFU pipe busy for ~4 k cycles per 128x256 tile.
// Two elements at a time (packed fp32 multiply-adds): the epilogue warps are bound by the instructions they issue, and the
// polynomial is most of an activation epilogue's. Squares held from above and a sum that saturates take 14 instructions per pair and
// activation where a clamped argument took 17, and 19 where 27 for the derivative.
__device__ __forceinline__ float fma_sat(float a, float b, float c) {
  float y;
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}
__device__ __forceinline__ f32x2 normal_cdf2(float x0, float x1, f32x2 square) {
  float u0, u1;
  upk2(square, u0, u1);
  const f32x2 u = pk2(fminf(u0, 18.f), fminf(u1, 18.f));
  f32x2 p = bc2(5.626733150e-11f);
  p = fma2(p, u, bc2(-5.371842857e-09f));
  p = fma2(p, u, bc2(2.268288109e-07f));
  p = fma2(p, u, bc2(-5.646201720e-06f));
  p = fma2(p, u, bc2(9.359050174e-05f));
  p = fma2(p, u, bc2(-1.109399655e-03f));
  p = fma2(p, u, bc2(9.818117358e-03f));
  p = fma2(p, u, bc2(-6.634692151e-02f));
  p = fma2(p, u, bc2(3.989031268e-01f));
  upk2(p, u0, u1);
  return pk2(fma_sat(x0, u0, 0.5f), fma_sat(x1, u1, 0.5f));
}
__device__ __forceinline__ float fast_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));  // branch-free, 1 ulp: keeps the element loops interleavable
  return y;
}
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void gelu2(float& x0, float& x1) {
  const f32x2 x = pk2(x0, x1);
  upk2(mul2(x, normal_cdf2(x0, x1, mul2(x, x))), x0, x1);
}
// f *= gelu'(x) = cdf(x) + x pdf(x)
__device__ __forceinline__ void gelu_grad2(float& f0, float& f1, float x0, float x1) {
  const f32x2 x = pk2(x0, x1), square = mul2(x, x);
  const f32x2 cdf = normal_cdf2(x0, x1, square);
  float e0, e1;
  upk2(mul2(square, bc2(-0.72134752044448170f)), e0, e1);   // -x^2 / 2 as a power of two
  const f32x2 density = pk2(fast_exp2(e0), fast_exp2(e1));
  upk2(mul2(pk2(f0, f1), fma2(mul2(x, bc2(0.3989422804014327f)), density, cdf)), f0, f1);
}
// The activation switch sits outside the element loop: with a branch per element the compiler cannot
// interleave the 32 independent dependency chains and the epilogue ran ~200 clocks per element.
__device__ __forceinline__ void act32(float (&f)[32], int act) {
  if (act == CCF_ACT_GELU) {
#pragma unroll
    for (int i = 0; i < 32; i += 2) gelu2(f[i], f[i + 1]);
  } else if (act == CCF_ACT_RELU) {
#pragma unroll
    for (int i = 0; i < 32; ++i) f[i] = fmaxf(f[i], 0.f);
  }
}
// f[i] *= act'(pz[i])
__device__ __forceinline__ void act_grad32(float (&f)[32], const float (&pz)[32], int act) {
  if (act == CCF_ACT_GELU) {
#pragma unroll
    for (int i = 0; i < 32; i += 2) gelu_grad2(f[i], f[i + 1], pz[i], pz[i + 1]);
  } else if (act == CCF_ACT_RELU) {
#pragma unroll
    for (int i = 0; i < 32; ++i) f[i] = pz[i] > 0.f ? f[i] : 0.f;
  }
}

// SwiGLU backward for two elements: a = gradient of silu(g) * u; g and u come packed in wg / wu and leave as their gradients
__device__ __forceinline__ void dswiglu2(float a0, float a1, uint32_t& wg, uint32_t& wu, int fp16) {
  const float2 gp = unpack2(wg, fp16), up = unpack2(wu, fp16);
  const f32x2 a = pk2(a0, a1), g = pk2(gp.x, gp.y), u = pk2(up.x, up.y);
  const float s0 = fast_rcp(1.f + __expf(-gp.x)), s1 = fast_rcp(1.f + __expf(-gp.y));
  const f32x2 sg = pk2(s0, s1);
  const f32x2 dg = mul2(mul2(a, u), mul2(sg, fma2(g, pk2(1.f - s0, 1.f - s1), bc2(1.f))));
  const f32x2 du = mul2(mul2(a, g), sg);
  float d0, d1;
  upk2(dg, d0, d1);
  wg = pack2(d0, d1, fp16);
  upk2(du, d0, d1);
  wu = pack2(d0, d1, fp16);
}

__device__ __forceinline__ float load_elem(const void* p, size_t i, int fp16) {
  if (fp16) return __half2float(reinterpret_cast<const __half*>(p)[i]);
  return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]);
}

// 32 consecutive 2-byte elements -> floats (64 bytes, 16-byte aligned)
__device__ __forceinline__ void load32(const void* p, float (&f)[32], int fp16) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint4 v = __ldg(q + i);
    uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 t = unpack2(w[j], fp16);
      f[i * 8 + j * 2] = t.x;
      f[i * 8 + j * 2 + 1] = t.y;
    }
  }
}

__device__ __forceinline__ void store32(void* p, const float (&f)[32], int fp16) {
  uint4* q = reinterpret_cast<uint4*>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint4 v;
    v.x = pack2(f[i * 8 + 0], f[i * 8 + 1], fp16);
    v.y = pack2(f[i * 8 + 2], f[i * 8 + 3], fp16);
    v.z = pack2(f[i * 8 + 4], f[i * 8 + 5], fp16);
    v.w = pack2(f[i * 8 + 6], f[i * 8 + 7], fp16);
    q[i] = v;
  }
}

__device__ __forceinline__ void store32_f32(float* p, const float (&f)[32]) {
  float4* q = reinterpret_cast<float4*>(p);
#pragma unroll
  for (int i = 0; i < 8; ++i) q[i] = make_float4(f[i * 4], f[i * 4 + 1], f[i * 4 + 2], f[i * 4 + 3]);
}

// 32 bias values as raw 16-byte words (same address for every lane: a broadcast load), applied later so that the
// load latency of chunk c+1 hides behind the math of chunk c
__device__ __forceinline__ void load_bias_raw(const void* bias, size_t elem_off, uint4 (&raw)[4]) {
  const uint4* q = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(bias) + elem_off);
#pragma unroll
  for (int i = 0; i < 4; ++i) raw[i] = __ldg(q + i);
}
__device__ __forceinline__ void add_bias_raw(float (&f)[32], const uint4 (&raw)[4], int fp16) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 t = unpack2(w[j], fp16);
      float &f0 = f[i * 8 + j * 2], &f1 = f[i * 8 + j * 2 + 1];
      upk2(add2(pk2(f0, f1), pk2(t.x, t.y)), f0, f1);
    }
  }
}

__device__ __forceinline__ void acc_to_float(const uint32_t (&r)[32], float (&f)[32]) {
#pragma unroll
  for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(r[i]);
}


// ---------------------------------------------------------------------------------------------------
// Epilogue row I/O through a per-warp shared-memory staging buffer (32 rows x 64 bytes, XOR-swizzled).
// In the TMEM register layout every lane owns one row, so a direct vector store writes 16 bytes to 32
// different rows per instruction: 4096 partial-sector requests per 128x256 tile and output, which capped
// the tensor pipe at ~46 % for two-output epilogues. Staged, each instruction moves 8 rows x 64 contiguous
// bytes (full 32-byte sectors). Lane l owns row l; `row_ptr` is the global address of this lane's
// 64-byte segment (0 = skip the row).
// ---------------------------------------------------------------------------------------------------
__host__ __device__ __forceinline__ constexpr uint32_t stage_off(int row, int piece) {
  return static_cast<uint32_t>(row * 64 + ((piece ^ ((row >> 1) & 3)) << 4));
}
// It has to be the 64-byte swizzle of a bulk tensor copy (address bits 4 and 5 exclusive-or bits 7 and 8): staged_store_tma hands the area
// over as a box of 32 columns.
constexpr bool stage_is_swizzled_64() {
  for (int row = 0; row < 32; ++row)
    for (int piece = 0; piece < 4; ++piece) {
      const uint32_t at = static_cast<uint32_t>(row * 64 + piece * 16);
      if (stage_off(row, piece) != (at ^ ((at >> 3) & 0x30u))) return false;
    }
  return true;
}
static_assert(stage_is_swizzled_64(), "layout of the staging area");

__device__ __forceinline__ void staged_store64(uint32_t stage, int lane, const uint32_t (&w)[16],
                                               unsigned long long row_ptr) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + stage_off(lane, j)), "r"(w[4 * j]),
                 "r"(w[4 * j + 1]), "r"(w[4 * j + 2]), "r"(w[4 * j + 3])
                 : "memory");
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = 8 * i + (lane >> 2), piece = lane & 3;
    const unsigned long long p = __shfl_sync(0xffffffffu, row_ptr, row);
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(stage + stage_off(row, piece))
                 : "memory");
    if (p != 0ull) *reinterpret_cast<uint4*>(p + piece * 16) = v;
  }
  __syncwarp();
}

// Bulk tensor stores. The staging area is laid out as the 64-byte swizzle has it, so that a staged chunk can leave as one box of 32
// columns x 32 rows: the CTA-pair kernel stores its activations, their gradients and weight gradients so. Read back and stored by the
// warp itself a chunk took eight more shared- and global-memory instructions and two turns through the staging area in the warp's own
// chain. Saved pre-activations come straight into their row's lane: the second quarter of a sector is an L1 hit. 4 groups of 4096 rows,
// 1024 x 4096, clocks per launch, with the shorter normal_cdf2 and the accumulator read when it is due (32 registers fewer):
// GELU 193 k -> 167 k, GELU' 228 k -> 176 k (of 120 k that the MMAs take).
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, uint32_t smem_src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(reinterpret_cast<uint64_t>(m)),
               "r"(smem_src), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(kPending) : "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void staged_store_tma(uint32_t stage, int lane, const uint32_t (&w)[16], const CUtensorMap* m, int col, int row) {
  if (elect_one()) bulk_wait_read<0>();   // the store before this one has read the staging area
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + stage_off(lane, j)), "r"(w[4 * j]), "r"(w[4 * j + 1]),
                 "r"(w[4 * j + 2]), "r"(w[4 * j + 3])
                 : "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (elect_one()) {
    tma_store_2d(m, stage, col, row);
    bulk_commit();
  }
  __syncwarp();
}
// one lane's 64 bytes of a row that the launch only reads
__device__ __forceinline__ void fetch_row64(unsigned long long p, bool ok, uint32_t (&w)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (ok) v = __ldg(reinterpret_cast<const uint4*>(p) + i);
    w[4 * i] = v.x;
    w[4 * i + 1] = v.y;
    w[4 * i + 2] = v.z;
    w[4 * i + 3] = v.w;
  }
}

__device__ __forceinline__ void pack32(const float (&f)[32], uint32_t (&w)[16], int fp16) {
#pragma unroll
  for (int i = 0; i < 16; ++i) w[i] = pack2(f[2 * i], f[2 * i + 1], fp16);
}
__device__ __forceinline__ void unpack32(const uint32_t (&w)[16], float (&f)[32], int fp16) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float2 t = unpack2(w[i], fp16);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
// byte address of element (row, col) of a 2-byte matrix with leading dimension ld
__device__ __forceinline__ unsigned long long addr2(const void* base, long long row, long long ld, int col) {
  return reinterpret_cast<unsigned long long>(base) + static_cast<unsigned long long>((row * ld + col) * 2);
}

// Optional per-tile trace: slot `ev` of tile number `seq` of this CTA gets the SM clock (clock64).
__device__ __forceinline__ void trace_ev(const CcfGemmArgs& a, int seq, int ev) {
  if (a.trace != nullptr && seq < a.trace_tiles)
    a.trace[(static_cast<size_t>(blockIdx.x) * a.trace_tiles + seq) * 8 + ev] = clock64();
}


// ---------------------------------------------------------------------------------------------------
// Epilogue of one accumulator tile for one epilogue warp: lane l owns tile row q*32 + l, the warp covers
// n_chunks chunks of 32 columns starting at chunk `half * n_chunks`. Shared by the one-CTA and the two-CTA kernels.
//   row_base     first output row of this CTA's 128 accumulator rows (group offset included for k-grouped mode)
//   rows_valid   rows of this CTA's part that hold data
//   rows_store   rows of this CTA's part that may be written at all (rows in [rows_valid, rows_store) get zeros)
//   out_map      kTma: tensor maps of the outputs (boxes of 32 x 32), which leave by bulk tensor stores
//   acquire      waits for the accumulator (false: given up); what the first chunk needs from global memory is requested before
//   release      hands the accumulator back to the MMA warp; called once the warp's last part of it is in registers, with that part's
//                arithmetic and stores still to come
// Returns where the row went (COMBINE) so that the caller can report completion; `here` false if the accumulator never came.
// ---------------------------------------------------------------------------------------------------
struct CombineDest {
  int rank;
  int units;   // 32-column pieces of the row that this warp stored
  bool ok;
  bool here;
};

// In-place SGD epilogue (STORE with sgd_lr != 0): the weights under the tile are read before they are rewritten. One
// 32-column chunk of a warp's 32 rows is 2 KB, so a warp that asked for it only when it needed it kept 16 KB per SM in
// flight and the kernel ran at the latency of a DRAM read per chunk. sgd_prefetch_l2 asks L2 for this lane's row of the
// tile part as soon as the tile is known (before its accumulator is complete); sgd_fetch_lin reads one chunk in the layout
// of the staged accesses (row 8 i + lane / 4, piece lane % 4) into registers one chunk ahead of its use. Measured on the
// 64-expert GPT-MoE step: asking for the NEXT tile's weights instead, or reading two chunks ahead, was slower than this.
__device__ __forceinline__ void sgd_prefetch_l2(const CcfGemmArgs& args, long long row_base, int n0, int rows_valid, int q,
                                                int half, int lane) {
  const int r_in_tile = q * 32 + lane;
  if (r_in_tile >= rows_valid) return;
  const int n_chunks = args.bn == 128 ? 2 : 4;
  const int n = n0 + half * n_chunks * 32;
  if (n >= args.n) return;
  const char* p = reinterpret_cast<const char*>(args.out0) + (static_cast<size_t>(row_base + r_in_tile) * args.ld_out + n) * 2;
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
  if (n_chunks == 4 && n + 64 < args.n) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + 128));
}
// Staged accesses for rows that lie one after the other in memory (every epilogue but COMBINE: row r of the warp's 32
// rows is at base + r * stride, the first rows_ok of them exist). The addresses are computed, not shuffled from the lane
// that owns the row: eight shuffles fewer per staged access, 15 % of the time of a launch that is bound by its epilogue.
__device__ __forceinline__ void sgd_fetch_lin(unsigned long long base, unsigned long long stride, int rows_ok, int lane,
                                              uint4 (&v)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = 8 * i + (lane >> 2), piece = lane & 3;
    v[i] = make_uint4(0u, 0u, 0u, 0u);
    if (row < rows_ok) v[i] = *reinterpret_cast<const uint4*>(base + row * stride + piece * 16);
  }
}
// the same for matrices that the launch only reads
__device__ __forceinline__ void fetch_lin(unsigned long long base, unsigned long long stride, int rows_ok, int lane, uint4 (&v)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = 8 * i + (lane >> 2), piece = lane & 3;
    v[i] = make_uint4(0u, 0u, 0u, 0u);
    if (row < rows_ok) v[i] = __ldg(reinterpret_cast<const uint4*>(base + row * stride + piece * 16));
  }
}
__device__ __forceinline__ void staged_store64_lin(uint32_t stage, int lane, const uint32_t (&w)[16], unsigned long long base,
                                                   unsigned long long stride, int rows_ok) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + stage_off(lane, j)), "r"(w[4 * j]),
                 "r"(w[4 * j + 1]), "r"(w[4 * j + 2]), "r"(w[4 * j + 3])
                 : "memory");
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = 8 * i + (lane >> 2), piece = lane & 3;
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(stage + stage_off(row, piece))
                 : "memory");
    if (row < rows_ok) *reinterpret_cast<uint4*>(base + row * stride + piece * 16) = v;
  }
  __syncwarp();
}
// a chunk fetched by sgd_fetch_lin or fetch_lin, transposed through the warp's staging area into one row per lane
__device__ __forceinline__ void unstage(uint32_t stage, int lane, const uint4 (&v)[4], uint32_t (&w)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = 8 * i + (lane >> 2), piece = lane & 3;
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + stage_off(row, piece)), "r"(v[i].x), "r"(v[i].y),
                 "r"(v[i].z), "r"(v[i].w)
                 : "memory");
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(w[4 * j]), "=r"(w[4 * j + 1]), "=r"(w[4 * j + 2]), "=r"(w[4 * j + 3])
                 : "r"(stage + stage_off(lane, j))
                 : "memory");
  }
  __syncwarp();
}

// kFp16 is a template argument: as a run-time value every conversion of an element pair computed both types' results and
// selected one, about a third of an epilogue's instructions.
template <int kEpi, int kFp16, bool kTma, typename Acquire, typename Release>
__device__ __forceinline__ CombineDest epilogue_tile(const CcfGemmArgs& args, const Tile& ti, long long row_base,
                                                     int rows_valid, int rows_store, bool have_acc, uint32_t t_row,
                                                     uint32_t stage, int q, int half, int lane, const CUtensorMap* const (&out_map)[3],
                                                     Acquire acquire, Release release) {
  constexpr int fp16 = kFp16;
  CombineDest cd;
  cd.rank = 0;
  cd.units = 0;
  cd.ok = false;
  cd.here = false;
  const int r_in_tile = q * 32 + lane;
  const bool valid = r_in_tile < rows_valid;
  const long long orow = row_base + r_in_tile;

  // COMBINE: where this row goes
  int c_rank = 0, c_slot = 0;
  float c_gate = 1.f;
  bool c_ok = false;
  if constexpr (kEpi == CCF_EPI_COMBINE) {
    if (valid) {
      const int packed = args.row_src[orow];
      c_rank = (packed >> 24) & 0xff;
      c_slot = packed & 0xffffff;
      c_gate = args.row_gate ? args.row_gate[orow] : 1.f;
      c_ok = c_rank < args.world && c_slot < args.max_slots;
      if (!c_ok) report_status(args.status, CCF_ERR_BOUNDS, static_cast<int>(orow) & 0xffffff);
    }
  }

  // chunks of 32 accumulator columns; this warp takes n_chunks of them starting at chunk0
  // 32-column chunks per warp: half of a 256-column tile (or of the 128 output columns of a SwiGLU tile, or of a
  // 128-column narrow tile)
  const int n_chunks = (kEpi == CCF_EPI_SWIGLU || args.bn == 128) ? 2 : 4;
  const int chunk0 = half * n_chunks;
  // A warp whose 32 rows all lie beyond the data has nothing to compute: with few rows per expert (decoding, the last tile
  // of every group) most warps are of that kind and only held the others' issue slots. Outputs that a weight-gradient
  // reduction may read get their zeros.
  if (q * 32 >= rows_valid) {
    if (!acquire()) return cd;
    cd.here = true;
    release();
    if constexpr (kEpi != CCF_EPI_STORE && kEpi != CCF_EPI_COMBINE) {
      const uint32_t zero[16] = {};
      const int ok = min(32, max(0, rows_store - q * 32));
      for (int c = 0; c < n_chunks; ++c) {
        const int n = ti.n0 + (chunk0 + c) * 32;
        if (n >= args.n || ok == 0) break;
        auto put = [&](void* p, int i) {
          if (p == nullptr) return;
          if constexpr (kTma) staged_store_tma(stage, lane, zero, out_map[i], n, static_cast<int>(row_base) + q * 32);
          else
            staged_store64_lin(stage, lane, zero, addr2(p, row_base + q * 32, args.ld_out, n),
                               static_cast<unsigned long long>(args.ld_out) * 2ull, ok);
        };
        put(args.out0, 0);
        if constexpr (kEpi != CCF_EPI_DACT) put(args.out1, 1);
        if constexpr (kEpi == CCF_EPI_SWIGLU) put(args.out2, 2);
      }
    }
    return cd;
  }
  constexpr bool kBias0Prefetch = (kEpi == CCF_EPI_STORE || kEpi == CCF_EPI_BIAS_ACT || kEpi == CCF_EPI_COMBINE);
  uint4 bcur[4], bnext[4];
  const bool has_b0 = kBias0Prefetch && args.bias0 != nullptr;
  if (has_b0 && ti.n0 + chunk0 * 32 < args.n)
    load_bias_raw(args.bias0, static_cast<size_t>(ti.g) * args.n + ti.n0 + chunk0 * 32, bnext);
  // in-place SGD never carries a bias (the host refuses the combination): the bias registers hold the weights' chunks
  const bool sgd = kEpi == CCF_EPI_STORE && args.sgd_lr != 0.f && !args.out_fp32;
  // every epilogue but COMBINE: the warp's 32 rows follow each other in the output and auxiliary matrices; the first
  // lin_rows of them hold data, the first lin_rows_store may be written (zeros beyond the data)
  const unsigned long long lin_stride = static_cast<unsigned long long>(args.ld_out) * 2ull;
  const int lin_rows = min(32, max(0, rows_valid - q * 32));
  const int lin_rows_store = min(32, max(0, rows_store - q * 32));
  auto lin_of = [&](const void* p) { return addr2(p, row_base + q * 32, args.ld_out, 0); };
  const unsigned long long lin_base = lin_of(args.out0);
  // a chunk of the warp's 32 rows into output i
  auto put = [&](const uint32_t (&w)[16], int i, void* p, int n) {
    if constexpr (kTma) {
      if (lin_rows_store > 0) staged_store_tma(stage, lane, w, out_map[i], n, static_cast<int>(row_base) + q * 32);
    } else {
      staged_store64_lin(stage, lane, w, lin_of(p) + n * 2ull, lin_stride, lin_rows_store);
    }
  };
  if (sgd) sgd_fetch_lin(lin_base + (ti.n0 + chunk0 * 32) * 2ull, lin_stride, ti.n0 + chunk0 * 32 < args.n ? lin_rows : 0, lane, bnext);
  // DACT, DSWIGLU: the saved pre-activations, one chunk ahead like the bias: loaded where they are used, each chunk of a tile
  // waited for one more trip to memory (4 experts x 4096 rows, 1024 -> 4096, GELU': 151 us a launch, 144 so)
  uint4 unext[4];
  uint32_t arow[16], urow[16];   // kTma: this lane's row, no staging
  auto fetch_aux = [&](int c) {
    const int n = ti.n0 + c * 32, ok = n < args.n ? lin_rows : 0;
    if constexpr (kTma) {
      if constexpr (kEpi == CCF_EPI_DACT || kEpi == CCF_EPI_DSWIGLU) fetch_row64(lin_of(args.aux0) + n * 2ull + lane * lin_stride, lane < ok, arow);
      if constexpr (kEpi == CCF_EPI_DSWIGLU) fetch_row64(lin_of(args.aux1) + n * 2ull + lane * lin_stride, lane < ok, urow);
    } else {
      if constexpr (kEpi == CCF_EPI_DACT || kEpi == CCF_EPI_DSWIGLU) fetch_lin(lin_of(args.aux0) + n * 2ull, lin_stride, ok, lane, bnext);
      if constexpr (kEpi == CCF_EPI_DSWIGLU) fetch_lin(lin_of(args.aux1) + n * 2ull, lin_stride, ok, lane, unext);
    }
  };
  fetch_aux(chunk0);
  if (!acquire()) return cd;
  cd.here = true;
  // An accumulator chunk is requested where it is due, in every epilogue: a second chunk in registers, requested ahead, was never faster.
  // Due / ahead, us: pair kernel, 4 experts of 4096 rows, 1024 x 4096: GELU 122.7 / 124.2, GELU' 128-138 / 141-147, rows combined 105 / 108,
  // input gradient 116-126 / 109-121 (noise), stored weight gradients 108-116 / 112-116; in place, 16 x 1024 rows, 2048 x 8192: 463 / 465.
  // One-CTA kernel, 3001 rows, 16 experts of 768 x 3072: ReLU 33.7 / 33.9, ReLU' 32.0 / 32.8, weight gradients 29.2 / 30.3, combined 44.9 / 45.0,
  // input gradient 34.5 / 36.5; 64 x 256 rows, 1024 x 4096, weight gradients 183-205 / 185-208
  // not unrolled: the body is large and every launch pays for fetching the kernel's code once per SM
#pragma unroll 1
  for (int c = 0; c < n_chunks; ++c) {
    const int cg = chunk0 + c;
    const int n = ti.n0 + cg * 32;
    float f[32];
    uint32_t w[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) bcur[i] = bnext[i];
    if (has_b0 && c + 1 < n_chunks && n + 32 < args.n)
      load_bias_raw(args.bias0, static_cast<size_t>(ti.g) * args.n + n + 32, bnext);
    if (sgd && c + 1 < n_chunks)
      sgd_fetch_lin(lin_base + (n + 32) * 2ull, lin_stride, n + 32 < args.n ? lin_rows : 0, lane, bnext);
    if (have_acc) {
      uint32_t racc[32];
      tmem_ld32(t_row + cg * 32, racc);
      tmem_ld_wait();
      acc_to_float(racc, f);
      if constexpr (kEpi != CCF_EPI_SWIGLU) {
        if (c + 1 == n_chunks) release();
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) f[i] = 0.f;
    }
    if constexpr (kEpi == CCF_EPI_SWIGLU) {
      // f = gate pre-activation (accumulator columns cg*32..), u = up pre-activation (+128)
      float u[32];
      if (have_acc) {
        uint32_t racc[32];
        tmem_ld32(t_row + 128 + cg * 32, racc);
        tmem_ld_wait();
        acc_to_float(racc, u);
        if (c + 1 == n_chunks) release();
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) u[i] = 0.f;
      }
      if (n < args.n) {
        if (args.bias1) {
          float b[32];
          load32(reinterpret_cast<const uint16_t*>(args.bias1) + static_cast<size_t>(ti.g) * args.n + n, b, fp16);
#pragma unroll
          for (int i = 0; i < 32; ++i) f[i] += b[i];
        }
        if (args.bias0) {
          float b[32];
          load32(reinterpret_cast<const uint16_t*>(args.bias0) + static_cast<size_t>(ti.g) * args.n + n, b, fp16);
#pragma unroll
          for (int i = 0; i < 32; ++i) u[i] += b[i];
        }
        if (!valid) {
#pragma unroll
          for (int i = 0; i < 32; ++i) { f[i] = 0.f; u[i] = 0.f; }
        }
        if (args.out1) {
          pack32(f, w, fp16);
          put(w, 1, args.out1, n);
        }
        if (args.out2) {
          pack32(u, w, fp16);
          put(w, 2, args.out2, n);
        }
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const f32x2 sg = pk2(fast_rcp(1.f + __expf(-f[i])), fast_rcp(1.f + __expf(-f[i + 1])));
          upk2(mul2(mul2(pk2(f[i], f[i + 1]), sg), pk2(u[i], u[i + 1])), f[i], f[i + 1]);
        }
        pack32(f, w, fp16);
        put(w, 0, args.out0, n);
      }
    } else if (n < args.n) {  // column edge: chunks beyond the matrix are skipped
      if constexpr (kEpi == CCF_EPI_STORE) {
        if (has_b0) add_bias_raw(f, bcur, fp16);
        if (args.out_fp32) {
          if (valid) store32_f32(reinterpret_cast<float*>(args.out0) + orow * args.ld_out + n, f);
        } else if (sgd) {
          // the accumulator is a weight gradient and out0 the weights themselves: plain SGD applied here saves writing
          // the gradient, and the optimizer's pass that would read it and the weights again
          unstage(stage, lane, bcur, w);
          const float lr = args.sgd_lr, wd = args.sgd_wd;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float2 p = unpack2(w[j], fp16);
            const f32x2 p2 = pk2(p.x, p.y);
            float n0, n1;
            upk2(fma2(bc2(-lr), fma2(bc2(wd), p2, pk2(f[2 * j], f[2 * j + 1])), p2), n0, n1);
            w[j] = pack2(n0, n1, fp16);
          }
          staged_store64_lin(stage, lane, w, lin_base + n * 2ull, lin_stride, lin_rows);
        } else {
          pack32(f, w, fp16);
          if constexpr (kTma) staged_store_tma(stage, lane, w, out_map[0], n, static_cast<int>(row_base) + q * 32);
          else staged_store64_lin(stage, lane, w, lin_base + n * 2ull, lin_stride, lin_rows);
        }
      } else if constexpr (kEpi == CCF_EPI_BIAS_ACT) {
        if (has_b0) add_bias_raw(f, bcur, fp16);
        if (lin_rows < 32 && !valid) {
#pragma unroll
          for (int i = 0; i < 32; ++i) f[i] = 0.f;
        }
        if (args.out1) {
          pack32(f, w, fp16);
          put(w, 1, args.out1, n);
        }
        act32(f, args.act);  // rows beyond the group hold zeros: act(0) = 0 for every supported activation
        pack32(f, w, fp16);
        put(w, 0, args.out0, n);
      } else if constexpr (kEpi == CCF_EPI_COMBINE) {
        if (has_b0) add_bias_raw(f, bcur, fp16);
#pragma unroll
        for (int i = 0; i < 32; i += 2) upk2(mul2(pk2(f[i], f[i + 1]), bc2(c_gate)), f[i], f[i + 1]);
        pack32(f, w, fp16);
        // peer stores over NVLink (or local when c_rank is this rank), 64 contiguous bytes per row
        staged_store64(stage, lane, w, c_ok ? addr2(args.peer_comb[c_rank], c_slot, args.ld_out, n) : 0ull);
      } else if constexpr (kEpi == CCF_EPI_DACT) {
        {
          float pz[32];
          if constexpr (kTma) {
            unpack32(arow, pz, fp16);
          } else {
            unstage(stage, lane, bcur, w);
            unpack32(w, pz, fp16);
          }
          if (c + 1 < n_chunks) fetch_aux(cg + 1);
          act_grad32(f, pz, args.act);
          if (lin_rows < 32 && !valid) {
#pragma unroll
            for (int i = 0; i < 32; ++i) f[i] = 0.f;
          }
        }
        pack32(f, w, fp16);
        put(w, 0, args.out0, n);
      } else if constexpr (kEpi == CCF_EPI_DSWIGLU) {
        uint32_t wu[16];
        if constexpr (kTma) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            w[j] = arow[j];
            wu[j] = urow[j];
          }
        } else {
          unstage(stage, lane, bcur, w);
          unstage(stage, lane, unext, wu);
        }
        if (c + 1 < n_chunks) fetch_aux(cg + 1);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          dswiglu2(valid ? f[2 * j] : 0.f, valid ? f[2 * j + 1] : 0.f, w[j], wu[j], fp16);
        }
        put(w, 0, args.out0, n);
        put(wu, 1, args.out1, n);
      }
    }
  }
  cd.rank = c_rank;
  cd.units = min(n_chunks, max(0, (args.n - ti.n0) / 32 - chunk0));
  cd.ok = c_ok;
  return cd;
}

// COMBINE: tell every source rank how many pieces of its rows are now in its buffer. A piece is 32 columns of a row in every kernel and
// for every tile width: the rank that stores and the rank that waits each choose their kernel from their own number of tokens,
// and the count that the one sends is the one that the other expects all the same (n / 32 per row). The fence waits for the
// tile's stores to be performed, which held up the next tile's epilogue and, at the end, the kernel: a single rank does without
// (128 tokens, 8 experts, 4096 x 14336, second projection: 195 us with it, 186 without; 16 tokens, 16 experts, 1024 x 4096: 42.8 and 35.9).
__device__ __forceinline__ void combine_signal(const CcfGemmArgs& args, const CombineDest& cd, int lane) {
  if (!args.count_rows) return;
  __threadfence_system();
  __syncwarp();
  for (int s = 0; s < args.world; ++s) {
    const unsigned m = __ballot_sync(0xffffffffu, cd.ok && cd.rank == s);
    if (m != 0u && cd.units > 0 && lane == 0) red_release_sys_add(args.peer_done[s], cd.units * __popc(m));
  }
}

// Rows of a chunk: a chunk is pushed by one warp from start to end. With only a few thousand rows in all (the latency-bound serving
// shapes) chunks of two rows spread them over more warps, and the first tile's rows are complete after microseconds instead of tens.
__host__ __device__ constexpr int dispatch_chunk(int kept) { return kept <= 4096 ? 2 : 8; }

// Whether epilogue warps help the dedicated ones of the first n_comm_ctas of `ctas` CTAs to push `kept` rows (dispatch_role). Not where it
// costs: of one chunk per dedicated warp or less (more warps only contend for the counter), and of more than 4096 rows in the kernel for
// few rows, where the first wave needs few of them and more rows under way at once make those late. Whole training passes replayed from
// a graph, us without and with help, rows = slots of the call, all CTAs pushing (one chunk per warp: 592 rows):
//   kernel for few rows   768 x 3072, 16 experts: 592 rows 189 / 187, 1024 203 / 198, 2048 226 / 217, 4096 297 / 266;
//                         1024 x 4096, 16 experts: 256 rows 250 / 256, 592 248 / 250, 1024 263 / 261, 4096 361 / 339;
//                         64 experts: 256 rows 702 / 711, 1024 711 / 710, 4096 764 / 750, 6144 807 / 807, 8192 840 / 843, 12288 911 / 904,
//                         16384 1072 / 1094
//   pair kernel           1024 x 4096, 4 experts: 4096 rows 316 / 287, 6144 407 / 396, 8192 472 /
//                         456, 12288 650 / 618, 16384 821 / 783; 512 x 2048, 8 experts: 6144 238 / 230, 16384 401 / 360
// With several ranks the claims are the same and nobody waits for a helper; it has not been measured there.
__host__ __device__ constexpr bool dispatch_help(int kept, int n_comm_ctas, int ctas, bool pair_kernel) {
  const int chunks = (kept + dispatch_chunk(kept) - 1) / dispatch_chunk(kept);
  return kept <= 4096 ? chunks > kCommWarps * (n_comm_ctas < ctas ? n_comm_ctas : ctas) : pair_kernel;
}

// The dispatch role as the epilogue warps of a GEMM kernel run it before their first accumulator is due. Only the
// kernels whose A operand is the receive buffer carry it: the forward ones (bias + activation, SwiGLU) push x rows, the
// backward ones (activation derivative) push g * dy rows; every other epilogue compiles to nothing here.
// `comm_warp`: the caller is one of the CTA's dedicated dispatch warps (else an epilogue warp); args.comm_warps says
// which of the two kinds carries the role in this launch. Where the dedicated ones do, epilogue warps that pass `first_acc`, the
// barrier of their first accumulator, help until it is complete: until then they have nothing else to do, and the first tiles wait
// for rows that two warps per SM push at the pace of their memory latencies. Passes, before and with help: GELU' of 16384 rows,
// 4 experts of 1024 x 4096 (pair kernel: the first wave of tiles needs a quarter of all rows) 186 -> 149 us; ReLU and ReLU' of 3001 rows,
// 16 experts of 768 x 3072 (kernel for few rows, chunks of two) 45.5 -> 37.4 and 57 -> 45 us. dispatch_help says where they do.
template <int kEpi, bool kPairKernel = false>
__device__ __forceinline__ void dispatch_role(const CcfGemmArgs& args, bool comm_warp, uint32_t first_acc = 0) {
  const bool carries = comm_warp == (args.comm_warps != 0);
  if (!carries && first_acc == 0) return;
  if (static_cast<int>(blockIdx.x) >= args.n_comm_ctas) return;
  const uint32_t stop = carries ? 0u : first_acc;
  const int kept = args.disp.order_off[args.disp.e_total];
  if (!carries && !dispatch_help(kept, args.n_comm_ctas, static_cast<int>(gridDim.x), kPairKernel)) return;
  if constexpr (kEpi == CCF_EPI_BIAS_ACT || kEpi == CCF_EPI_SWIGLU) {
    if (dispatch_chunk(kept) == 2) dispatch_rows<2, false>(args.disp, args.status, stop);
    else dispatch_rows<8, false>(args.disp, args.status, stop);
  } else if constexpr (kEpi == CCF_EPI_DACT || kEpi == CCF_EPI_DSWIGLU) {
    if (dispatch_chunk(kept) == 2) dispatch_rows<2, true>(args.disp, args.status, stop);
    else dispatch_rows<8, true>(args.disp, args.status, stop);
  }
}

// two-CTA kernels (gemm2.cu), selected by the same key as the one-CTA ones
int launch_pair_by_key(int key, const CUtensorMap* tm, const CcfGemmArgs& a, int grid, int early, cudaStream_t stream);
// few rows per group: weights on the M side (gemm_swap.cu)
int launch_swap_by_key(int b_major, int epi, const CUtensorMap* tm, const CcfGemmArgs& a, int grid, int early, cudaStream_t stream);
int swap_box_rows(bool big);
// weight gradients of few rows per group (gemm_wgrad.cu)
int launch_wgrad(const CUtensorMap* tm, const CcfGemmArgs& a, int grid, int early, cudaStream_t stream);

}  // namespace ccf
