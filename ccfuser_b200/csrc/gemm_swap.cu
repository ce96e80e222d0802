// Row-grouped GEMM for few rows per group (tcgen05 cta_group::2, weights on the M side): a CTA pair computes 256 output features
// of ALL rows of a group, D^T[features, rows] = W[features, k] * X[rows, k]^T. Used for the forward and input-gradient GEMMs of
// calls that expect at most a few hundred rows per expert (decoding, serving batches, many experts).
//
// Why the operands change sides: with the rows on the M side (gemm.cu, gemm2.cu) a tile is 128 or 256 rows high whatever the
// group holds. 16 tokens on 16 experts multiply 126 rows of padding per expert, and an expert of 270 rows needs a third 128-row
// tile. On the N side the tile is as wide as the group's rows rounded up to 16, every weight is read once, and a stage of the
// pipeline holds 16 KB of weights beside only the rows there are: with few rows nearly all of shared memory is weights in flight.
//
//   tile        256 features (128 per CTA) x up to 320 rows of one group (128 for SwiGLU, whose accumulator is two wide)
//   parts       a tile of more columns than an accumulator holds is two parts that share every stage of weights
//   accumulators  ring of 2 x 256 or, when some group has more than 256 rows, 3 x 160 TMEM columns: with two parts per tile the
//               next tile's first part has a free accumulator while the last tile's parts are stored
//   tiles       pair p takes tiles p, p + pairs, ...; where the last round would leave half of the pairs or more without one, its tiles
//               come in pieces of their rows (swap_last_round). One round of few tiles gained most: second projection of 300 rows, 4
//               experts of 1024 x 4096 (16 tiles) 42 -> 33 us, 8 experts of 768 x 3072 36 -> 29; 64 experts of 256 rows, 1024 x 4096
//               (3.5 rounds) 154 -> 148. Every sum runs over k in order on one pair, as in gemm2.cu, so that a row's result
//               does not depend on what is routed beside it. A version in which the pairs shared the k-blocks of the last tiles through
//               an fp32 workspace gave that up, and cost more than the even split saved: of 1032 launches measured (512 x 2048 to
//               4096 x 14336, 4 to 64 experts, 8 to 320 rows each) it was slower in 308 and more than 4 % faster in 33; 8 experts of
//               256 rows, 4096 x 14336: 255 us without against 300 with it for the second projection, 470 against 628 for its
//               input gradient; 4 experts of 8 rows, 4096 x 1024, SwiGLU, input gradient: 73 against 48.
//
// The epilogue reads the accumulator in fragments of 8 features x 8 rows and transposes them by stmatrix into the warp's staging
// area, from where rows leave as 64-byte segments like those of the other kernels. Arrival gating, dispatch role, combine with
// completion counters: as in gemm2.cu. No TMA load uses cluster multicast.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <string.h>

#include "gemm_common.cuh"
#include "pair.cuh"
#include "swap_shape.h"

namespace ccf {

constexpr int kSwMaxStages = 12;
constexpr int kSwPipeBytes = 206 * 1024;
constexpr int kSwWBytes = BM * BK * 2;       // this CTA's 128 features of one k-block
// rows of the two boxes that tokens come in, one TMA instruction each: with boxes of 16 alone the eight instructions of a 256-row
// k-block took 400 clocks longer than its loads
constexpr int kSwBox = 16, kSwBig = 64;
constexpr int kSwMaxBufs = 3;

// What an epilogue warp has in hand, kept in shared memory: as registers it pushed the epilogue's own values out to local memory.
struct SwapWork {
  int t;                                             // next tile
  int g, row0, tokens, zero_rows, n0, parts, np;     // SwapTile
};

struct __align__(16) CtrlS {
  uint64_t full[kSwMaxStages];     // used on the leader: both CTAs' loads complete on it
  uint64_t empty[kSwMaxStages];    // one per CTA: the leader's MMA thread commits to both
  uint64_t acc_full[kSwMaxBufs];
  uint64_t acc_empty[kSwMaxBufs];  // used on the leader: 2 * kEpiWarps arrivals
  uint32_t tmem_base;
  int abort_word;
  SwapShape shape;
  SwapRound round;
  int mt_prefix[CCF_MAX_GROUPS + 1];   // row tiles, prefix over groups
  int base[CCF_MAX_GROUPS];
  int rows[CCF_MAX_GROUPS];
  SwapWork work[kEpiWarps];
};

constexpr int kSwSmemBytes = 1024 + kSwPipeBytes + kEpiWarps * kEpiStageBytes + static_cast<int>(sizeof(CtrlS));
static_assert(kSwSmemBytes <= 232448, "shared memory of one CTA");

// ---- fragments --------------------------------------------------------------------------------------
// 16 TMEM lanes x 32 columns: register 4 j + 2 s + b of lane l = (lane 8 s + l / 4, column 8 j + 2 (l % 4) + b)
__device__ __forceinline__ void tmem_ld_16x256b_x4(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// this warp's 32 features x 32 rows: element 16 h + 4 j + 2 s + b = (feature 16 h + 8 s + l / 4, row 8 j + 2 (l % 4) + b)
__device__ __forceinline__ void tmem_ld_frag(uint32_t taddr, uint32_t (&r)[32]) {
  tmem_ld_16x256b_x4(taddr, r);
  tmem_ld_16x256b_x4(taddr + (16u << 16), r + 16);
}
// word m = 8 h + 2 j + s holds rows (8 j + 2 (l % 4), + 1) of feature 8 p + l / 4, p = 2 h + s
__device__ __forceinline__ constexpr int frag_piece(int m) { return 2 * (m >> 3) + (m & 1); }

// fragments -> staging area (32 rows x 32 features, 64 bytes a row, swizzled like every staged access)
__device__ __forceinline__ void frag_to_stage(uint32_t stage, int lane, const uint32_t (&w)[16]) {
#pragma unroll
  for (int j = 0; j < 4; ++j)
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};"
                 ::"r"(stage + stage_off(8 * j + (lane & 7), lane >> 3)), "r"(w[2 * j]), "r"(w[2 * j + 1]), "r"(w[8 + 2 * j]), "r"(w[9 + 2 * j])
                 : "memory");
  __syncwarp();
}
__device__ __forceinline__ void stage_to_frag(uint32_t stage, int lane, uint32_t (&w)[16]) {
#pragma unroll
  for (int j = 0; j < 4; ++j)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(w[2 * j]), "=r"(w[2 * j + 1]), "=r"(w[8 + 2 * j]), "=r"(w[9 + 2 * j])
                 : "r"(stage + stage_off(8 * j + (lane & 7), lane >> 3))
                 : "memory");
  __syncwarp();
}
// Rows 8 i + l / 4 of the chunk, piece l % 4; `to` is this lane's place in the first eight rows, `step` the distance of eight rows.
// Rows below `valid` as they are, zeros up to `end`.
__device__ __forceinline__ void frag_store(uint32_t stage, int lane, const uint32_t (&w)[16], char* to, unsigned long long step, int valid,
                                           int end) {
  frag_to_stage(stage, lane, w);
  uint4 v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v[i].x), "=r"(v[i].y), "=r"(v[i].z), "=r"(v[i].w)
                 : "r"(stage + stage_off(8 * i + (lane >> 2), lane & 3))
                 : "memory");
  if (valid >= 32) {
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(to + i * step) = v[i];
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = 8 * i + (lane >> 2);
      if (row < end) *reinterpret_cast<uint4*>(to + i * step) = row < valid ? v[i] : make_uint4(0u, 0u, 0u, 0u);
    }
  }
  __syncwarp();
}
__device__ __forceinline__ void frag_fetch(const char* from, unsigned long long step, int valid, int lane, uint4 (&v)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i] = make_uint4(0u, 0u, 0u, 0u);
    if (8 * i + (lane >> 2) < valid) v[i] = __ldg(reinterpret_cast<const uint4*>(from + i * step));
  }
}
// a chunk fetched by frag_fetch, as fragments
__device__ __forceinline__ void fetched_to_frag(uint32_t stage, int lane, const uint4 (&v)[4], uint32_t (&w)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + stage_off(8 * i + (lane >> 2), lane & 3)), "r"(v[i].x),
                 "r"(v[i].y), "r"(v[i].z), "r"(v[i].w)
                 : "memory");
  __syncwarp();
  stage_to_frag(stage, lane, w);
}

// ---- tiles --------------------------------------------------------------------------------------------
// The next tile of an epilogue warp; out of line, the registers it needs are not the epilogue's.
__device__ __noinline__ bool swap_next(const CtrlS* ctrl, SwapWork* w, int n_pairs, int num_groups) {
  int t = w->t;
  __syncwarp();
  SwapTile ti;
  do {
    if (t >= ctrl->round.items) return false;
    ti = decode_swap_item(t, ctrl, num_groups);
    t += n_pairs;
  } while (ti.tokens <= 0);
  if ((threadIdx.x & 31) == 0) *w = SwapWork{t, ti.g, ti.row0, ti.tokens, ti.zero_rows, ti.n0, ti.parts, ti.np};
  __syncwarp();
  return true;
}

// Tile tables of one launch, filled by one warp of every CTA at start-up
template <int kEpi>
__device__ __forceinline__ void swap_tables_warp(const CcfGemmArgs& args, CtrlS* ctrl, int lane) {
  constexpr bool kWide = kEpi == CCF_EPI_SWIGLU;
  int max_rows = 0, total_rows = 0;
  for (int g0 = 0; g0 < args.num_groups; g0 += 32) {
    const int g = g0 + lane;
    if (g < args.num_groups) {
      const int gr = args.group_rows[g];
      ctrl->rows[g] = gr;
      ctrl->base[g] = args.group_base[g];
      max_rows = max(max_rows, gr);
      total_rows += gr;
    }
  }
  max_rows = __reduce_max_sync(0xffffffffu, max_rows);
  total_rows = __reduce_add_sync(0xffffffffu, total_rows);
  __syncwarp();
  int acc = 0, max_half = 0;   // max_half: rows of tokens a CTA holds per stage
  const int width = swap_width(max_rows, kWide), cap = swap_cap(max_rows, kWide);
  for (int g0 = 0; g0 < args.num_groups; g0 += 32) {
    const int g = g0 + lane;
    int mt = 0;
    if (g < args.num_groups) {
      const int gr = ctrl->rows[g];
      mt = (gr + cap - 1) / cap;
      if (mt > 0) max_half = max(max_half, swap_half_rows(swap_round16((gr + mt - 1) / mt), width));
    }
    int sm = mt;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sm, off);
      if (lane >= off) sm += v;
    }
    if (g < args.num_groups) ctrl->mt_prefix[g] = acc + sm - mt;
    acc += __shfl_sync(0xffffffffu, sm, 31);
  }
  max_half = __reduce_max_sync(0xffffffffu, max_half);
  if (lane == 0) {
    ctrl->mt_prefix[args.num_groups] = acc;
    ctrl->shape = swap_shape(args, acc, total_rows, max_half, width, kWide, kSwPipeBytes, kSwMaxStages);
    ctrl->round = swap_last_round(ctrl->shape.total_tiles, static_cast<int>(gridDim.x) >> 1, min(max_rows, cap));
  }
}

// ---- epilogue -----------------------------------------------------------------------------------------
// One part of a tile for one warp: 32 features (fbase ...), the 32-row chunks first, first + 2, ... of the part.
struct SwapPart {
  int g;
  int row0;    // first row of the part
  int valid;   // rows that hold data
  int end;     // rows to be written (zeros beyond `valid`)
  int np;      // accumulator columns
  int first;   // this warp's first chunk
};

// `acquire` waits for the accumulator (false: given up); bias and saved inputs are requested before.
// `release` hands it back; called once this warp's last chunk of it is in registers.
template <int kEpi, int kFp16, typename Acquire, typename Release>
__device__ __forceinline__ void swap_epilogue(const CcfGemmArgs& args, const SwapPart& pt, uint32_t t_col, uint32_t up_col,
                                              uint32_t stage, int fbase, int lane, Acquire acquire, Release release) {
  constexpr int fp16 = kFp16;
  constexpr bool kWide = kEpi == CCF_EPI_SWIGLU;
  const int n_acc = (pt.np + 31) >> 5;   // chunks with an accumulator
  const unsigned long long step = static_cast<unsigned long long>(args.ld_out) * 16ull;   // bytes of eight rows
  // this lane's place in row l / 4 of the part, bytes
  const long long at0 = ((pt.row0 + (lane >> 2)) * args.ld_out + fbase + (lane & 3) * 8) * 2;
  auto at = [&](const void* p, int c) {
    return const_cast<char*>(reinterpret_cast<const char*>(p)) + (at0 + 4ll * c * static_cast<long long>(step));
  };
  float b0[4] = {0, 0, 0, 0}, b1[4] = {0, 0, 0, 0};
  {
    const size_t off = static_cast<size_t>(pt.g) * args.n + fbase + (lane >> 2);
    if (kEpi != CCF_EPI_DACT && kEpi != CCF_EPI_DSWIGLU && args.bias0 != nullptr) {
#pragma unroll
      for (int p = 0; p < 4; ++p) b0[p] = load_elem(args.bias0, off + 8 * p, fp16);
    }
    if (kWide && args.bias1 != nullptr) {
#pragma unroll
      for (int p = 0; p < 4; ++p) b1[p] = load_elem(args.bias1, off + 8 * p, fp16);
    }
  }
  uint4 an0[4], an1[4];   // auxiliary inputs of the next chunk
  auto fetch = [&](int c) {
    if constexpr (kEpi == CCF_EPI_DACT || kEpi == CCF_EPI_DSWIGLU) frag_fetch(at(args.aux0, c), step, pt.valid - 32 * c, lane, an0);
    if constexpr (kEpi == CCF_EPI_DSWIGLU) frag_fetch(at(args.aux1, c), step, pt.valid - 32 * c, lane, an1);
  };
  // COMBINE: where row `lane` of the next chunk goes, a chunk ahead like the auxiliary inputs: read where they were used, the two stood
  // a trip to memory in front of every chunk's shuffles
  int dest_next = -1;
  float gate_next = 1.f;
  auto fetch_dest = [&](int c) {
    if constexpr (kEpi == CCF_EPI_COMBINE) {
      dest_next = -1;
      if (lane < pt.valid - 32 * c) {
        const int row = pt.row0 + 32 * c + lane;
        dest_next = args.row_src[row];
        if (args.row_gate != nullptr) gate_next = args.row_gate[row];
      }
    }
  };
  fetch(pt.first);
  fetch_dest(pt.first);
  if (!acquire()) return;
  if (pt.first >= n_acc || pt.first * 32 >= pt.end) release();   // no chunk of it is this warp's
  int sent = 0;   // COMBINE: lane s counts the rows stored for rank s
#pragma unroll 1
  for (int c = pt.first; c * 32 < pt.end; c += 2) {
    const int valid = pt.valid - 32 * c, end = pt.end - 32 * c;
    float f[32];
    uint32_t w[16];
    auto load = [&](float (&v)[32], uint32_t col) {
      if (c < n_acc) {
        uint32_t r[32];
        tmem_ld_frag(col + 32 * c, r);
        tmem_ld_wait();
        acc_to_float(r, v);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = 0.f;
      }
    };
    auto add_bias = [&](float (&v)[32], const float (&b)[4]) {
#pragma unroll
      for (int m = 0; m < 16; ++m) upk2(add2(pk2(v[2 * m], v[2 * m + 1]), bc2(b[frag_piece(m)])), v[2 * m], v[2 * m + 1]);
    };
    auto pack = [&](const float (&v)[32]) {
#pragma unroll
      for (int m = 0; m < 16; ++m) w[m] = pack2(v[2 * m], v[2 * m + 1], fp16);
    };
    load(f, t_col);
    const bool last = c < n_acc && (c + 2 >= n_acc || (c + 2) * 32 >= pt.end);   // of those this warp looks at
    if (!kWide && last) release();
    if constexpr (kEpi == CCF_EPI_SWIGLU) {
      add_bias(f, b1);   // the first accumulator is the gate projection
      float u[32];
      load(u, up_col);
      if (last) release();
      add_bias(u, b0);
      if (args.out1) {
        pack(f);
        frag_store(stage, lane, w, at(args.out1, c), step, valid, end);
      }
      if (args.out2) {
        pack(u);
        frag_store(stage, lane, w, at(args.out2, c), step, valid, end);
      }
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        const f32x2 sg = pk2(fast_rcp(1.f + __expf(-f[i])), fast_rcp(1.f + __expf(-f[i + 1])));
        upk2(mul2(mul2(pk2(f[i], f[i + 1]), sg), pk2(u[i], u[i + 1])), f[i], f[i + 1]);
      }
      pack(f);
      frag_store(stage, lane, w, at(args.out0, c), step, valid, end);
    } else if constexpr (kEpi == CCF_EPI_BIAS_ACT) {
      add_bias(f, b0);
      if (args.out1) {
        pack(f);
        frag_store(stage, lane, w, at(args.out1, c), step, valid, end);
      }
      act32(f, args.act);
      pack(f);
      frag_store(stage, lane, w, at(args.out0, c), step, valid, end);
    } else if constexpr (kEpi == CCF_EPI_COMBINE) {
      add_bias(f, b0);
      // lane l: where row l of the chunk goes
      int packed = dest_next;
      const float gate = gate_next;
      if (lane < valid && (packed < 0 || ((packed >> 24) & 0xff) >= args.world || (packed & 0xffffff) >= args.max_slots)) {
        report_status(args.status, CCF_ERR_BOUNDS, (pt.row0 + 32 * c + lane) & 0xffffff);
        packed = -1;
      }
      if ((c + 2) * 32 < pt.end) fetch_dest(c + 2);
      if (args.row_gate != nullptr) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float g0 = __shfl_sync(0xffffffffu, gate, 8 * j + 2 * (lane & 3));
          const float g1 = __shfl_sync(0xffffffffu, gate, 8 * j + 2 * (lane & 3) + 1);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int m = 8 * (k >> 1) + 2 * j + (k & 1);
            upk2(mul2(pk2(f[2 * m], f[2 * m + 1]), pk2(g0, g1)), f[2 * m], f[2 * m + 1]);
          }
        }
      }
      pack(f);
      frag_to_stage(stage, lane, w);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = 8 * i + (lane >> 2), piece = lane & 3;
        const int to = __shfl_sync(0xffffffffu, packed, row);
        uint4 v;
        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "r"(stage + stage_off(row, piece))
                     : "memory");
        // peer stores over NVLink (or local when the row came from this rank)
        if (to >= 0)
          *reinterpret_cast<uint4*>(addr2(args.peer_comb[(to >> 24) & 0xff], to & 0xffffff, args.ld_out, fbase) + piece * 16) = v;
      }
      __syncwarp();
      if (args.count_rows)
        for (int s = 0; s < args.world; ++s) {
          const unsigned m = __ballot_sync(0xffffffffu, packed >= 0 && ((packed >> 24) & 0xff) == s);
          if (lane == s) sent += __popc(m);
        }
    } else if constexpr (kEpi == CCF_EPI_DACT) {
      fetched_to_frag(stage, lane, an0, w);
      if ((c + 2) * 32 < pt.end) fetch(c + 2);
      float pz[32];
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const float2 t = unpack2(w[m], fp16);
        pz[2 * m] = t.x;
        pz[2 * m + 1] = t.y;
      }
      act_grad32(f, pz, args.act);
      pack(f);
      frag_store(stage, lane, w, at(args.out0, c), step, valid, end);
    } else if constexpr (kEpi == CCF_EPI_DSWIGLU) {
      uint32_t wu[16];
      fetched_to_frag(stage, lane, an0, w);
      fetched_to_frag(stage, lane, an1, wu);
      if ((c + 2) * 32 < pt.end) fetch(c + 2);
#pragma unroll
      for (int j = 0; j < 16; ++j) dswiglu2(f[2 * j], f[2 * j + 1], w[j], wu[j], fp16);
      frag_store(stage, lane, w, at(args.out0, c), step, valid, end);
      frag_store(stage, lane, wu, at(args.out1, c), step, valid, end);
    }
  }
  if (kEpi == CCF_EPI_COMBINE && args.count_rows) {
    // tell every source rank how many of its rows (for these 32 features) are now in its buffer
    __threadfence_system();
    __syncwarp();
    if (sent > 0) red_release_sys_add(args.peer_done[lane], sent);
  }
}

// ---- the kernel -----------------------------------------------------------------------------------------
template <int kWMajor, int kEpi, int kFp16>
__global__ void __launch_bounds__(kThreads, 1)
grouped_gemm_swap_kernel(const __grid_constant__ CUtensorMap tmX0, const __grid_constant__ CUtensorMap tmX1,
                         const __grid_constant__ CUtensorMap tmW0, const __grid_constant__ CUtensorMap tmW1,
                         const __grid_constant__ CUtensorMap tmXb0, const __grid_constant__ CUtensorMap tmXb1,
                         const __grid_constant__ CcfGemmArgs args) {
  constexpr bool kWide = kEpi == CCF_EPI_SWIGLU;   // two accumulators: gate and up projection
  constexpr uint32_t kW = (kWide ? 2 : 1) * kSwWBytes;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  CtrlS* ctrl = reinterpret_cast<CtrlS*>(smem + kSwPipeBytes + kEpiWarps * kEpiStageBytes);
  const uint32_t smem_base = smem_u32(smem);
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();   // 0 = leader (issues the MMAs), 1 = peer
  const int pair = static_cast<int>(blockIdx.x) >> 1;
  const int n_pairs = static_cast<int>(gridDim.x) >> 1;
  volatile int* abort_word = &ctrl->abort_word;

  // ---- set-up ------------------------------------------------------------------------------------
  if (threadIdx.x == 0) {
    for (int s = 0; s < kSwMaxStages; ++s) {
      mbar_init(smem_u32(&ctrl->full[s]), 1);
      mbar_init(smem_u32(&ctrl->empty[s]), 1);
    }
    for (int s = 0; s < kSwMaxBufs; ++s) {
      mbar_init(smem_u32(&ctrl->acc_full[s]), 1);
      mbar_init(smem_u32(&ctrl->acc_empty[s]), 2 * kEpiWarps);
    }
    ctrl->abort_word = 0;
    fence_barrier_init();
    fence_proxy_async();
    prefetch_tensormap(&tmX0);
    prefetch_tensormap(&tmW0);
    prefetch_tensormap(&tmXb0);
    if (args.kseg > 1 || kWide) {
      prefetch_tensormap(&tmX1);
      prefetch_tensormap(&tmXb1);
      prefetch_tensormap(&tmW1);
    }
  }
  wait_for_previous();
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(&ctrl->tmem_base), kTmemCols);
    tmem_relinquish_pair();
  }
  const uint64_t limit = fail_fast_limit(args.status, args.wait_limit_ns);
  if (warp == 2) swap_tables_warp<kEpi>(args, ctrl, lane);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  let_next_in();
  const uint32_t tmem_base = ctrl->tmem_base;
  const SwapShape& sh = ctrl->shape;
  const int stages = sh.stages;
  const uint32_t stage_bytes = sh.stage_bytes;
  const int kb_per_seg = (args.k + BK - 1) / BK, kblocks = sh.kblocks, items = ctrl->round.items;

  if (threadIdx.x == 0 && args.trace != nullptr) trace_ev(args, args.trace_tiles - 1, 0);

  if (warp == 0) {
    // ======================= TMA producer (both CTAs) =======================
    int stage = 0, phase = 0, seq = 0;
    bool ok = true, all_in = false;
    const int nh = static_cast<int>(cta) * BM;
    const uint32_t bar_own0 = smem_u32(&ctrl->full[0]), full_leader0 = map_to_cta(bar_own0, 0), empty0 = smem_u32(&ctrl->empty[0]);
    auto load_weights = [&](const CUtensorMap* mw, int w_row, int n_col, int kk, uint32_t sw, uint32_t bar) {
      if constexpr (kWMajor == MAJ_K) {
        if constexpr (kWide) {
          tma_load_2d_pair(sw, &tmW1, bar, kk, w_row);                // gate projection
          tma_load_2d_pair(sw + kSwWBytes, &tmW0, bar, kk, w_row);    // up projection
        } else {
          tma_load_2d_pair(sw, mw, bar, kk, w_row);
        }
      } else {
        tma_load_2d_pair(sw, mw, bar, n_col, w_row + kk);
        tma_load_2d_pair(sw + 8192, mw, bar, n_col + 64, w_row + kk);
      }
    };
    for (int t = pair; t < items && ok; t += n_pairs) {
      const SwapTile ti = decode_swap_item(t, ctrl, args.num_groups);
      if (ti.tokens <= 0) continue;
      if (lane == 0) trace_ev(args, seq, 0);
      const int half = ti.np >> 1, boxes = (half + kSwBox - 1) / kSwBox;
      const uint32_t bytes = 2 * (kW + static_cast<uint32_t>(ti.parts * boxes * (kSwBox * 128)));   // of both CTAs
      const int n_col = ti.n0 + nh, w_row = ti.g * args.b_group_rows + (kWMajor == MAJ_K ? n_col : 0);
      const int x_row = ti.row0 + static_cast<int>(cta) * half;
      // The first stages' weights are requested before the rows are waited for: they depend on nothing.
      int pre = 0;
      if (seq == 0) {
        pre = min(stages, kblocks);
        if (elect_one()) {
          for (int i = 0; i < pre; ++i) {
            const int seg = i >= kb_per_seg ? 1 : 0;   // at most two segments
            if (cta == 0) mbar_arrive_expect_tx(smem_u32(&ctrl->full[i]), bytes);
            load_weights(seg ? &tmW1 : &tmW0, w_row, n_col, (i - seg * kb_per_seg) * BK, smem_base + i * stage_bytes,
                         map_to_cta(smem_u32(&ctrl->full[i]), 0));
          }
        }
        __syncwarp();
      }
      if (args.tile_flags != nullptr && !all_in) {
        int state = 1;
        // the count of all arrived rows is read alongside: once it is complete, later tiles skip the flags and their latency
        const int total = lane == 31 && args.total_index >= 0 ? ld_acquire_sys(args.tile_flags + args.total_index) : 0;
        const int first = ti.row0 >> 7, last = (ti.row0 + ti.tokens - 1) >> 7, end = ctrl->base[ti.g] + ctrl->rows[ti.g];
        if (first + lane <= last) {   // at most four 128-row tiles
          const int r = first + lane;
          if (!wait_flag_ge(args.tile_flags + r, min(128, end - (r << 7)), limit)) state = 0;
        }
        state = __all_sync(0xffffffffu, state);
        if (state == 0) {
          report_status(args.status, CCF_ERR_FLAG_TIMEOUT, first);
          *abort_word = 1;
          break;
        }
        all_in = __shfl_sync(0xffffffffu, args.total_index >= 0 && total >= sh.total_rows, 31);
        fence_proxy_async();   // generic-proxy peer stores -> async-proxy (TMA) reads
      }
      if (lane == 0) trace_ev(args, seq, 1);
      const CUtensorMap *mw = &tmW0, *mx = &tmX0, *mxb = &tmXb0;
      int kk = 0;
      for (int kb = 0; kb < kblocks; ++kb, kk += BK) {
        if (kb == kb_per_seg) {
          mw = &tmW1;
          mx = &tmX1;
          mxb = &tmXb1;
          kk = 0;
        }
        const bool armed = pre > 0;
        if (armed) --pre;
        else if (!mbar_wait_cluster(empty0 + 8 * stage, phase ^ 1, abort_word, limit)) {
          report_status(args.status, CCF_ERR_MBAR_TIMEOUT, 0x32);
          ok = false;
          break;
        }
        if (elect_one()) {
          const uint32_t bar = full_leader0 + 8 * stage, sw = smem_base + stage * stage_bytes;
          if (!armed) {
            if (cta == 0) mbar_arrive_expect_tx(bar_own0 + 8 * stage, bytes);
            load_weights(mw, w_row, n_col, kk, sw, bar);
          }
          uint32_t sx = sw + kW;
          for (int p = 0; p < ti.parts; ++p) {
            int r = x_row + p * ti.np, left = boxes;
            for (; left >= kSwBig / kSwBox; left -= kSwBig / kSwBox, r += kSwBig, sx += kSwBig * 128) tma_load_2d_pair(sx, mxb, bar, kk, r);
            for (; left > 0; --left, r += kSwBox, sx += kSwBox * 128) tma_load_2d_pair(sx, mx, bar, kk, r);
          }
        }
        __syncwarp();
        if (++stage == stages) { stage = 0; phase ^= 1; }
      }
      if (lane == 0) trace_ev(args, seq, 2);
      ++seq;
    }
  } else if (warp == 1) {
    // ======================= MMA issuer (leader CTA only) =======================
    if (cta == 0) {
      const uint64_t desc_w = operand_desc(smem_base, kWMajor), desc_x = operand_desc(smem_base + kW, MAJ_K);
      const uint32_t full0 = smem_u32(&ctrl->full[0]), empty0 = smem_u32(&ctrl->empty[0]);
      int stage = 0, phase = 0, buf = 0, bphase = 0, seq = 0;
      bool ok = true;
      for (int t = pair; t < items && ok; t += n_pairs) {
        const SwapTile ti = decode_swap_item(t, ctrl, args.num_groups);
        if (ti.tokens <= 0) continue;
        const uint32_t idesc = make_idesc(PM, ti.np, args.fp16, kWMajor, MAJ_K);
        const uint32_t part_bytes = static_cast<uint32_t>((((ti.np >> 1) + kSwBox - 1) / kSwBox) * kSwBox) * 128;
        if (lane == 0) trace_ev(args, seq, 3);
        const int b1 = buf + 1 < sh.bufs ? buf + 1 : 0;
        const uint32_t d0 = tmem_base + buf * sh.buf_cols, d1 = tmem_base + b1 * sh.buf_cols;
        for (int p = 0; p < ti.parts && ok; ++p) {
          const int b = p == 0 ? buf : b1;
          if (!mbar_wait_cluster(smem_u32(&ctrl->acc_empty[b]), (p == 0 || b1 != 0 ? bphase : bphase ^ 1) ^ 1, abort_word, limit)) {
            report_status(args.status, CCF_ERR_MBAR_TIMEOUT, 0x34);
            ok = false;
          }
        }
        const bool two = !kWide && ti.parts > 1;
        for (int kb = 0; kb < kblocks && ok; ++kb) {
          if (!mbar_wait_cluster(full0 + 8 * stage, phase, abort_word, limit)) {
            report_status(args.status, CCF_ERR_MBAR_TIMEOUT, 0x35);
            ok = false;
            break;
          }
          tc_fence_after();
          if (elect_one()) {
            if (kb == 0) trace_ev(args, seq, 4);
            const uint32_t at = static_cast<uint32_t>(stage) * stage_bytes;
            const uint32_t acc = kb > 0 ? 1u : 0u;
#pragma unroll
            for (int a = 0; a < (kWide ? 2 : 1); ++a) {
#pragma unroll
              for (int k = 0; k < BK / UK; ++k)
                umma_f16_pair(d0 + a * 128, desc_at(desc_w, at + a * kSwWBytes + k * desc_step(kWMajor)),
                              desc_at(desc_x, at + k * desc_step(MAJ_K)), idesc, k > 0 ? 1u : acc);
            }
            if (two) {
#pragma unroll
              for (int k = 0; k < BK / UK; ++k)
                umma_f16_pair(d1, desc_at(desc_w, at + k * desc_step(kWMajor)),
                              desc_at(desc_x, at + part_bytes + k * desc_step(MAJ_K)), idesc, k > 0 ? 1u : acc);
            }
            umma_commit_pair(empty0 + 8 * stage);   // hand the stage back to both producers
          }
          __syncwarp();
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
        if (ok && elect_one()) {
          umma_commit_pair(smem_u32(&ctrl->acc_full[buf]));
          if (two) umma_commit_pair(smem_u32(&ctrl->acc_full[b1]));
          trace_ev(args, seq, 5);
        }
        __syncwarp();
        buf += ti.parts;
        if (buf >= sh.bufs) { buf -= sh.bufs; bphase ^= 1; }
        ++seq;
      }
    }
  } else if (warp >= 2 + kEpiWarps) {
    // ======================= dispatch warps =======================
    dispatch_role<kEpi>(args, true);
    if (warp == 2 + kEpiWarps && lane == 0 && args.trace != nullptr && args.comm_warps) trace_ev(args, args.trace_tiles - 1, 1);
  } else {
    // ======================= epilogue (warps 2..9, both CTAs) =======================
    const int q = warp & 3;
    const int hw = (warp - 2) >> 2;
    dispatch_role<kEpi>(args, false, smem_u32(&ctrl->acc_full[0]));
    if (warp == 2 && lane == 0 && args.trace != nullptr && !args.comm_warps) trace_ev(args, args.trace_tiles - 1, 1);
    int buf = 0, bphase = 0, seq = 0;
    bool ok = true;
    const uint32_t stage = smem_base + kSwPipeBytes + (warp - 2) * kEpiStageBytes;
    // outputs that a reduction over rows reads get zeros up to the next multiple of its 64-row step
    const bool zeros = kEpi == CCF_EPI_DACT || kEpi == CCF_EPI_DSWIGLU || ((kEpi == CCF_EPI_BIAS_ACT || kWide) && args.out1 != nullptr);
    SwapWork* const w = &ctrl->work[warp - 2];
    if (lane == 0) w->t = pair;
    __syncwarp();
    while (ok && swap_next(ctrl, w, n_pairs, args.num_groups)) {
      for (int p = 0; p < w->parts; ++p) {
        const int fbase = w->n0 + static_cast<int>(cta) * BM + q * 32, np = w->np;
        // two warps share a part's chunks; with an odd number they take turns in having one more
        const int chunks = (np + 31) >> 5, c0 = hw ^ (p & chunks & 1);
        const uint32_t col = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + buf * sh.buf_cols;
        auto release = [&] {   // all TMEM reads of this accumulator are complete: hand it back to the MMA warp
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster_relaxed(map_to_cta(smem_u32(&ctrl->acc_empty[buf]), 0));
        };
        auto acquire = [&] {
          if (!mbar_wait_cluster(smem_u32(&ctrl->acc_full[buf]), bphase, abort_word, limit)) {
            report_status(args.status, CCF_ERR_MBAR_TIMEOUT, 0x37);
            ok = false;
            return false;
          }
          tc_fence_after();
          if (p == 0 && warp == 2 && lane == 0) trace_ev(args, seq, 6);
          return true;
        };
        if (fbase < args.n) {
          SwapPart pt;
          pt.g = w->g;
          pt.np = np;
          pt.first = c0;
          pt.row0 = w->row0 + p * np;
          pt.valid = min(np, w->tokens - p * np);
          pt.end = pt.valid + (zeros && p == w->parts - 1 ? w->zero_rows : 0);
          swap_epilogue<kEpi, kFp16>(args, pt, col, col + (sh.buf_cols >> 1), stage, fbase, lane, acquire, release);
        } else if (acquire()) {
          release();
        }
        if (!ok) break;
        if (++buf == sh.bufs) { buf = 0; bphase ^= 1; }
      }
      if (warp == 2 && lane == 0) trace_ev(args, seq, 7);
      ++seq;
    }
  }

  // ---- tear-down -----------------------------------------------------------------------------------
  tc_fence_before();
  __syncthreads();
  if (ctrl->abort_word) {
    // give copies still in flight time to land before shared memory and TMEM go away
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 50000ull) __nanosleep(1000);
    __syncthreads();
  }
  cluster_sync_all();   // neither CTA frees TMEM or leaves while the other may still use the pair's resources
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
  if (threadIdx.x == 0) {
    __threadfence();
    const int done = atomicAdd(args.sched + 1, 1);
    if (done == static_cast<int>(gridDim.x) - 1) {
      if constexpr (kEpi == CCF_EPI_COMBINE) {
        if (args.send_finish) {
          __threadfence_system();
          for (int s = 0; s < args.world; ++s) red_release_sys_add(args.peer_done[s], 1);
        }
      }
      args.sched[0] = 0;
      args.sched[1] = 0;
      args.sched[2] = 0;
      __threadfence();
    }
  }
}

template <int W, int E, int FP16>
static int launch_swap_variant_of(const CUtensorMap* tm, const CcfGemmArgs& args, int grid, int early, cudaStream_t stream) {
  auto kern = grouped_gemm_swap_kernel<W, E, FP16>;
  // the attribute belongs to the (function, device) pair: set it once per device this process launches on
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSwSmemBytes);
    if (e != cudaSuccess) return -static_cast<int>(e);
    configured[dev & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid & ~1);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSwSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2] = {cluster_attribute(2, 1, 1), early_attribute()};
  cfg.attrs = attr;
  cfg.numAttrs = early ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tm[0], tm[1], tm[2], tm[3], tm[4], tm[5], args);
  return e == cudaSuccess ? 0 : -static_cast<int>(e);
}

template <int W, int E>
static int launch_swap_variant(const CUtensorMap* tm, const CcfGemmArgs& args, int grid, int early, cudaStream_t stream) {
  return args.fp16 ? launch_swap_variant_of<W, E, 1>(tm, args, grid, early, stream) : launch_swap_variant_of<W, E, 0>(tm, args, grid, early, stream);
}

int swap_box_rows(bool big) { return big ? kSwBig : kSwBox; }

// Called by ccf_gemm_launch (gemm.cu) for row-grouped launches with `few_rows` set; returns -6 for a combination that does not exist.
// tm[0], tm[1]: rows in boxes of 16; tm[4], tm[5]: the same in boxes of 64; tm[2], tm[3]: weights.
int launch_swap_by_key(int b_major, int epi, const CUtensorMap* tm, const CcfGemmArgs& a, int grid, int early, cudaStream_t stream) {
  switch ((b_major << 4) | epi) {
    case (MAJ_K << 4) | CCF_EPI_BIAS_ACT: return launch_swap_variant<MAJ_K, CCF_EPI_BIAS_ACT>(tm, a, grid, early, stream);
    case (MAJ_K << 4) | CCF_EPI_SWIGLU: return launch_swap_variant<MAJ_K, CCF_EPI_SWIGLU>(tm, a, grid, early, stream);
    case (MAJ_K << 4) | CCF_EPI_COMBINE: return launch_swap_variant<MAJ_K, CCF_EPI_COMBINE>(tm, a, grid, early, stream);
    case (MAJ_MN << 4) | CCF_EPI_DACT: return launch_swap_variant<MAJ_MN, CCF_EPI_DACT>(tm, a, grid, early, stream);
    case (MAJ_MN << 4) | CCF_EPI_DSWIGLU: return launch_swap_variant<MAJ_MN, CCF_EPI_DSWIGLU>(tm, a, grid, early, stream);
    case (MAJ_MN << 4) | CCF_EPI_COMBINE: return launch_swap_variant<MAJ_MN, CCF_EPI_COMBINE>(tm, a, grid, early, stream);
    default: return -6;
  }
}

}  // namespace ccf

namespace ccf {

// The tables of a launch, on the host
struct SwapTables {
  SwapShape shape;
  SwapRound round;
  int half;
  int mt_prefix[CCF_MAX_GROUPS + 1], base[CCF_MAX_GROUPS], rows[CCF_MAX_GROUPS];
};
static int swap_tables_host(const int* group_rows, int num_groups, int n, int k, int kseg, int wide, int n_pairs, SwapTables* c) {
  if (num_groups < 1 || num_groups > CCF_MAX_GROUPS) return -2;
  CcfGemmArgs a;
  memset(&a, 0, sizeof(a));
  a.n = n;
  a.k = k;
  a.kseg = kseg;
  int max_rows = 0, total = 0, tiles = 0, half = 0, base = 0;
  for (int g = 0; g < num_groups; ++g) {
    max_rows = group_rows[g] > max_rows ? group_rows[g] : max_rows;
    total += group_rows[g];
  }
  const int width = swap_width(max_rows, wide != 0), rows_cap = swap_cap(max_rows, wide != 0);
  for (int g = 0; g < num_groups; ++g) {
    c->rows[g] = group_rows[g];
    c->base[g] = base;
    c->mt_prefix[g] = tiles;
    base += (group_rows[g] + 127) / 128 * 128;
    const int mt = (group_rows[g] + rows_cap - 1) / rows_cap;
    if (mt == 0) continue;
    const int h = swap_half_rows(swap_round16((group_rows[g] + mt - 1) / mt), width);
    half = h > half ? h : half;
    tiles += mt;
  }
  c->mt_prefix[num_groups] = tiles;
  c->half = half;
  c->shape = swap_shape(a, tiles, total, half, width, wide != 0, kSwPipeBytes, kSwMaxStages);
  c->round = swap_last_round(c->shape.total_tiles, n_pairs, swap_min(max_rows, rows_cap));
  return 0;
}

}  // namespace ccf

// The whole tiles of a launch of the swapped kernel, before those of its last round are cut (ccf_debug_swap_items), computed on the
// host with the kernel's own functions: out[9 i ...] = {pair, tile, first k-block, one past the last, first pair that works on the tile,
// number of such pairs, rows per stage of the launch, stages, number of tiles}. Host arrays in, nothing touches a device. Returns the
// number of records (only the first `cap` are written).
extern "C" int ccf_debug_swap_segments(const int* group_rows, int num_groups, int n, int k, int kseg, int wide, int n_pairs, int* out,
                                       int cap) {
  using namespace ccf;
  SwapTables c;
  if (int rc = swap_tables_host(group_rows, num_groups, n, k, kseg, wide, n_pairs, &c)) return rc;
  const SwapShape& s = c.shape;
  int i = 0;
  for (int p = 0; p < n_pairs; ++p)
    for (int t = p; t < s.total_tiles; t += n_pairs, ++i) {
      const int rec[9] = {p, t, 0, s.kblocks, p, 1, c.half, s.stages, s.total_tiles};
      if (i < cap) memcpy(out + 9 * i, rec, sizeof(rec));
    }
  return i;
}

// What every CTA pair of such a launch works on, in order: out[12 i ...] = {pair, item, first item of the last round if it is cut (else
// the number of items), group, first row in the group, rows, rows behind them that get zeros, first feature, parts, columns of a part,
// rows per stage that it takes, rows per stage that there are}. Groups lie as they do in a launch, on multiples of 128 rows.
extern "C" int ccf_debug_swap_items(const int* group_rows, int num_groups, int n, int k, int kseg, int wide, int n_pairs, int* out, int cap) {
  using namespace ccf;
  SwapTables c;
  if (int rc = swap_tables_host(group_rows, num_groups, n, k, kseg, wide, n_pairs, &c)) return rc;
  int i = 0;
  for (int p = 0; p < n_pairs; ++p)
    for (int w = p; w < c.round.items; w += n_pairs) {
      const SwapTile t = decode_swap_item(w, &c, num_groups);
      if (t.tokens <= 0) continue;
      const int rec[12] = {p, w, c.round.whole, t.g, t.row0 - c.base[t.g], t.tokens, t.zero_rows, t.n0, t.parts, t.np,
                           t.parts * ((((t.np >> 1) + kSwBox - 1) / kSwBox) * kSwBox), c.half};
      if (i < cap) memcpy(out + 12 * i, rec, sizeof(rec));
      ++i;
    }
  return i;
}
