// Weight-gradient GEMM for few rows per group (k-grouped, tcgen05 cta_group::2): C_g[M, N] = sum over the group's rows A[r, M]^T B[r, N],
// stored, or applied to the weights in place (w -= lr * (C_g + wd * w)).
//
// With a few hundred rows per group a 256 x 256 tile is a handful of k-blocks: 2048 clocks of tensor pipe per 256 rows, against
// 64 KB per CTA of result to write and, in place, as much to read. The launch is bound by moving the weights, and in the general
// kernels (gemm.cu, gemm2.cu) by the epilogue that moves them: 24 shared- and global-memory instructions per warp and 32 columns, with
// one 2 KB chunk per warp in flight. Here the weights travel by TMA:
//
//   ring of 16 KB chunks (128 rows x 64 columns, 128-byte swizzle). In place: a producer warp loads chunks ahead of the accumulators,
//   the epilogue warps update them where they lie (one row per lane; 16-byte accesses of eight lanes fall into different banks), a
//   store warp writes them back, and a chunk whose store has been read is loaded again. Without weights the chunks are output buffers.
//
// Measured, pair kernel / this one, operands of several layers in turn, us (plain and in place): 16 x 256 rows, 768 x 3072: 31 / 25 and 51 / 37; 64 x 256,
// 1024 x 4096: 186 / 147 and 346 / 219; 64 x 256, 2048 x 8192: 842 / 611 and 1343 / 770 (4.3 GB read and written: 5.6 TB/s);
// 16 x 512, 2048 x 8192: 255 / 240 and 375 / 283. With more rows the main loop decides, and the pair kernel's deeper ring wins:
// 16 x 1024 rows 411 / 447 and 478 / 496 (wgrad_few in runtime.cu).
//
// Everything else is as in gemm2.cu: CTA pairs, MN-major operands, two accumulators. All waits are bounded; no TMA load uses cluster
// multicast.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "gemm_common.cuh"
#include "pair.cuh"

namespace ccf {

// Four k-blocks of operands beside five chunks. With three and seven a stage's round trip from L2 did not fit behind the other two, and
// a k-block took 800 clocks instead of 600 (64 x 256 rows, 1024 x 4096, plain: 172 -> 156 us). With four chunks updates in place wait for
// their weights (64 x 256 rows, 2048 x 8192: 812 -> 866 us); five stages and four chunks are no faster than this.
constexpr int kWgStages = 4;                         // k-blocks of operands
constexpr int kWgStageBytes = 2 * BM * BK * 2;       // this CTA's 128 rows of A^T and its half of B
constexpr int kWgChunks = 5;
static_assert(kWgChunks >= 4, "ChunkPos moves by up to a tile's four chunks and wraps once");
constexpr int kWgChunkBytes = BM * 64 * 2;
constexpr int kWgThreads = 384;                      // warps 0 operands, 1 MMA, 2 weights, 3 stores, 4..11 epilogue

struct __align__(16) CtrlW {
  uint64_t full[kWgStages];      // used on the leader
  uint64_t empty[kWgStages];     // one per CTA
  uint64_t acc_full[2];
  uint64_t acc_empty[2];         // used on the leader: 2 * 8 arrivals
  uint64_t loaded[kWgChunks];    // weights of the chunk have landed
  uint64_t done[kWgChunks];      // four epilogue warps have written it
  uint64_t free_[kWgChunks];     // its store has read it
  uint32_t tmem_base;
  int abort_word;
  int base[CCF_MAX_GROUPS];
  int rows[CCF_MAX_GROUPS];
};
constexpr int kWgSmemBytes = 1024 + kWgStages * kWgStageBytes + kWgChunks * kWgChunkBytes + static_cast<int>(sizeof(CtrlW));
static_assert(kWgSmemBytes <= 232448, "shared memory of one CTA");

__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* m, int c0, int c1) {
  asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(m)), "r"(c0), "r"(c1) : "memory");
}

struct WgTile {
  int g, m0, n0, kblocks, krow0, chunks;   // chunks: 64-column chunks inside the matrix
};
// Stored: along the shorter side of the result first, so that the pairs of a wave share the fewest panels (64 x 384 rows, 2048 x 8192:
// 885 -> 785 us). In place: columns first, so that a wave reads and writes whole rows of the weights (64 x 512 rows: 1127 against 1276).
template <bool kSgd>
__device__ __forceinline__ WgTile decode_wg_tile(int t, const CcfGemmArgs& a, const CtrlW* c, int mt, int nt) {
  WgTile ti;
  ti.g = t / (mt * nt);
  const int local = t - ti.g * (mt * nt);
  int i, j;
  if (!kSgd && mt < nt) {
    j = local / mt;
    i = local - j * mt;
  } else {
    i = local / nt;
    j = local - i * nt;
  }
  ti.m0 = i * PM;
  ti.n0 = j * BN;
  ti.kblocks = (c->rows[ti.g] + BK - 1) / BK;
  ti.krow0 = c->base[ti.g];
  ti.chunks = min(4, (a.n - ti.n0 + 63) >> 6);
  return ti;
}

// position in the ring of chunks
struct ChunkPos {
  int slot = 0, phase = 0;
  __device__ __forceinline__ void advance(int n) {
    slot += n;
    if (slot >= kWgChunks) { slot -= kWgChunks; phase ^= 1; }
  }
};

template <int kFp16, bool kSgd>
__global__ void __launch_bounds__(kWgThreads, 1)
grouped_wgrad_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CcfGemmArgs args) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  CtrlW* ctrl = reinterpret_cast<CtrlW*>(smem + kWgStages * kWgStageBytes + kWgChunks * kWgChunkBytes);
  const uint32_t smem_base = smem_u32(smem), ring = smem_base + kWgStages * kWgStageBytes;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();
  const int pair = static_cast<int>(blockIdx.x) >> 1, n_pairs = static_cast<int>(gridDim.x) >> 1;
  volatile int* abort_word = &ctrl->abort_word;
  const int mt = args.m_per_group / PM, nt = (args.n + BN - 1) / BN, total = args.num_groups * mt * nt;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kWgStages; ++s) {
      mbar_init(smem_u32(&ctrl->full[s]), 1);
      mbar_init(smem_u32(&ctrl->empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&ctrl->acc_full[s]), 1);
      mbar_init(smem_u32(&ctrl->acc_empty[s]), 2 * kEpiWarps);
    }
    for (int s = 0; s < kWgChunks; ++s) {
      mbar_init(smem_u32(&ctrl->loaded[s]), 1);
      mbar_init(smem_u32(&ctrl->done[s]), 4);
      mbar_init(smem_u32(&ctrl->free_[s]), 1);
    }
    ctrl->abort_word = 0;
    fence_barrier_init();
    fence_proxy_async();
    prefetch_tensormap(&tmA);
    prefetch_tensormap(&tmB);
    prefetch_tensormap(&tmC);
  }
  wait_for_previous();
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(&ctrl->tmem_base), kTmemCols);
    tmem_relinquish_pair();
  }
  const uint64_t limit = fail_fast_limit(args.status, args.wait_limit_ns);
  for (int g = static_cast<int>(threadIdx.x) - 64; g >= 0 && g < args.num_groups; g += kWgThreads - 64) {
    ctrl->rows[g] = args.group_rows[g];
    ctrl->base[g] = args.group_base[g];
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  let_next_in();
  const uint32_t tmem_base = ctrl->tmem_base;
  if (threadIdx.x == 0 && args.trace != nullptr) trace_ev(args, args.trace_tiles - 1, 0);

  if (warp == 0) {
    // ======================= operands (both CTAs) =======================
    int stage = 0, phase = 0, seq = 0;
    bool ok = true;
    const uint32_t full0 = smem_u32(&ctrl->full[0]), leader0 = map_to_cta(full0, 0), empty0 = smem_u32(&ctrl->empty[0]);
    for (int t = pair; t < total && ok; t += n_pairs, ++seq) {
      const WgTile ti = decode_wg_tile<kSgd>(t, args, ctrl, mt, nt);
      const int m = ti.m0 + static_cast<int>(cta) * BM, n = ti.n0 + static_cast<int>(cta) * (BN / 2);
      if (lane == 0) trace_ev(args, seq, 0);
      // The operands of this pair's next tile are asked of L2 a tile ahead: four stages do not cover a trip to DRAM, and all pairs of a
      // wave meet a group's rows for the first time together (64 x 256 rows, 1024 x 4096: 156 -> 145 us). The pairs that share a panel
      // take its k-blocks in turns. In place the weights decide, and it gives nothing.
      if constexpr (!kSgd) {
        if (t + n_pairs < total) {
          const WgTile nx = decode_wg_tile<kSgd>(t + n_pairs, args, ctrl, mt, nt);
          const int pm = nx.m0 + static_cast<int>(cta) * BM, pn = nx.n0 + static_cast<int>(cta) * (BN / 2);
          if (elect_one()) {
            for (int kb = nx.n0 / BN; kb < nx.kblocks; kb += nt) {
              tma_prefetch_2d(&tmA, pm, nx.krow0 + kb * BK);
              tma_prefetch_2d(&tmA, pm + 64, nx.krow0 + kb * BK);
            }
            for (int kb = nx.m0 / PM; kb < nx.kblocks; kb += mt) {
              tma_prefetch_2d(&tmB, pn, nx.krow0 + kb * BK);
              tma_prefetch_2d(&tmB, pn + 64, nx.krow0 + kb * BK);
            }
          }
          __syncwarp();
        }
      }
      for (int kb = 0; kb < ti.kblocks; ++kb) {
        if (!mbar_wait_cluster(empty0 + 8 * stage, phase ^ 1, abort_word, limit)) {
          report_status(args.status, CCF_ERR_MBAR_TIMEOUT, 0x60);
          ok = false;
          break;
        }
        if (elect_one()) {
          const uint32_t sa = smem_base + stage * kWgStageBytes, sb = sa + BM * BK * 2, bar = leader0 + 8 * stage;
          const int r = ti.krow0 + kb * BK;
          if (cta == 0) mbar_arrive_expect_tx(full0 + 8 * stage, 2 * kWgStageBytes);
          tma_load_2d_pair(sa, &tmA, bar, m, r);
          tma_load_2d_pair(sa + 8192, &tmA, bar, m + 64, r);
          tma_load_2d_pair(sb, &tmB, bar, n, r);
          tma_load_2d_pair(sb + 8192, &tmB, bar, n + 64, r);
        }
        __syncwarp();
        if (++stage == kWgStages) { stage = 0; phase ^= 1; }
      }
      if (lane == 0) trace_ev(args, seq, 2);
    }
  } else if (warp == 1) {
    // ======================= MMA issuer (leader CTA only) =======================
    if (cta == 0) {
      const uint32_t idesc = make_idesc(PM, BN, args.fp16, MAJ_MN, MAJ_MN);
      const uint64_t desc_a = operand_desc(smem_base, MAJ_MN), desc_b = operand_desc(smem_base + BM * BK * 2, MAJ_MN);
      int stage = 0, phase = 0, as = 0, aphase = 0, seq = 0;
      bool ok = true;
      for (int t = pair; t < total && ok; t += n_pairs, ++seq) {
        const WgTile ti = decode_wg_tile<kSgd>(t, args, ctrl, mt, nt);
        if (ti.kblocks == 0) continue;   // empty group: the epilogue takes zeros
        if (!mbar_wait_cluster(smem_u32(&ctrl->acc_empty[as]), aphase ^ 1, abort_word, limit)) {
          report_status(args.status, CCF_ERR_MBAR_TIMEOUT, 0x61);
          break;
        }
        tc_fence_after();
        if (lane == 0) trace_ev(args, seq, 3);
        const uint32_t d_tmem = tmem_base + as * BN;
        for (int kb = 0; kb < ti.kblocks; ++kb) {
          if (!mbar_wait_cluster(smem_u32(&ctrl->full[stage]), phase, abort_word, limit)) {
            report_status(args.status, CCF_ERR_MBAR_TIMEOUT, 0x62);
            ok = false;
            break;
          }
          tc_fence_after();
          if (elect_one()) {
            if (kb == 0) trace_ev(args, seq, 4);
            const uint32_t at = static_cast<uint32_t>(stage) * kWgStageBytes;
#pragma unroll
            for (int k = 0; k < BK / UK; ++k)
              umma_f16_pair(d_tmem, desc_at(desc_a, at + k * desc_step(MAJ_MN)), desc_at(desc_b, at + k * desc_step(MAJ_MN)), idesc,
                            (kb > 0 || k > 0) ? 1u : 0u);
            umma_commit_pair(smem_u32(&ctrl->empty[stage]));
            if (kb == ti.kblocks - 1) {
              umma_commit_pair(smem_u32(&ctrl->acc_full[as]));
              trace_ev(args, seq, 5);
            }
          }
          __syncwarp();
          if (++stage == kWgStages) { stage = 0; phase ^= 1; }
        }
        if (++as == 2) { as = 0; aphase ^= 1; }
      }
    }
  } else if (warp == 2) {
    // ======================= weights =======================
    if constexpr (kSgd) {
      ChunkPos pos;
      bool ok = true;
      for (int t = pair; t < total && ok; t += n_pairs) {
        const WgTile ti = decode_wg_tile<kSgd>(t, args, ctrl, mt, nt);
        const int row = ti.g * args.m_per_group + ti.m0 + static_cast<int>(cta) * BM;
        for (int c = 0; c < ti.chunks; ++c, pos.advance(1)) {
          if (!mbar_wait(smem_u32(&ctrl->free_[pos.slot]), pos.phase ^ 1, abort_word, limit)) {
            report_status(args.status, CCF_ERR_MBAR_TIMEOUT, 0x63);
            ok = false;
            break;
          }
          if (elect_one()) {
            mbar_arrive_expect_tx(smem_u32(&ctrl->loaded[pos.slot]), kWgChunkBytes);
            tma_load_2d(ring + pos.slot * kWgChunkBytes, &tmC, smem_u32(&ctrl->loaded[pos.slot]), ti.n0 + 64 * c, row);
          }
          __syncwarp();
        }
      }
    }
  } else if (warp == 3) {
    // ======================= stores: one thread, since bulk groups belong to the thread that issued them =======================
    if (elect_one()) {
      ChunkPos pos, freed;
      bool ok = true;
      [[maybe_unused]] int pending = 0;   // stores that may still be reading their chunk
      for (int t = pair; t < total && ok; t += n_pairs) {
        const WgTile ti = decode_wg_tile<kSgd>(t, args, ctrl, mt, nt);
        const int row = ti.g * args.m_per_group + ti.m0 + static_cast<int>(cta) * BM;
        for (int c = 0; c < ti.chunks; ++c, pos.advance(1)) {
          if (!mbar_wait(smem_u32(&ctrl->done[pos.slot]), pos.phase, abort_word, limit)) {
            report_status(args.status, CCF_ERR_MBAR_TIMEOUT, 0x64);
            ok = false;
            break;
          }
          tma_store_2d(&tmC, ring + pos.slot * kWgChunkBytes, ti.n0 + 64 * c, row);
          bulk_commit();
          // In place a chunk is handed back as soon as it has been read: the next weights wait for it (64 x 256 rows, 2048 x 8192: 810 ->
          // 768 us). Without weights to load the older of two is, and the stores follow each other closer (1024 x 4096: 153 against 165).
          if constexpr (kSgd) {
            bulk_wait_read<0>();
            mbar_arrive(smem_u32(&ctrl->free_[freed.slot]));
            freed.advance(1);
          } else if (++pending == 2) {   // the older one has been read by now, or nearly
            bulk_wait_read<1>();
            mbar_arrive(smem_u32(&ctrl->free_[freed.slot]));
            freed.advance(1);
            pending = 1;
          }
        }
      }
      bulk_wait_all();
    }
    __syncwarp();
  } else {
    // ======================= epilogue (warps 4..11, both CTAs) =======================
    const int q = warp & 3, half = (warp - 4) >> 2;   // TMEM lane quarter; chunks half, half + 2 of every tile
    const float lr = args.sgd_lr, wd = args.sgd_wd;
    int as = 0, aphase = 0, seq = 0;
    ChunkPos pos;
    bool ok = true;
    // this lane's row of a chunk: 16-byte piece p lies at p ^ (row mod 8)
    const uint32_t row_at = static_cast<uint32_t>((q * 32 + lane) * 128), swz = static_cast<uint32_t>(lane & 7) << 4;
    for (int t = pair; t < total && ok; t += n_pairs, ++seq) {
      const WgTile ti = decode_wg_tile<kSgd>(t, args, ctrl, mt, nt);
      const bool have_acc = ti.kblocks > 0;
      if (have_acc) {
        if (!mbar_wait_cluster(smem_u32(&ctrl->acc_full[as]), aphase, abort_word, limit)) {
          report_status(args.status, CCF_ERR_MBAR_TIMEOUT, 0x65);
          break;
        }
        tc_fence_after();
      }
      if (warp == 4 && lane == 0) trace_ev(args, seq, 6);
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + as * BN;
      auto release = [&] {
        if (!have_acc) return;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster_relaxed(map_to_cta(smem_u32(&ctrl->acc_empty[as]), 0));
      };
      ChunkPos cp = pos;
      cp.advance(half);
      if (half >= ti.chunks) release();
      for (int c = half; c < ti.chunks; c += 2, cp.advance(2)) {
        // in place: the weights are there; else: the chunk's last store has read it
        const uint32_t bar = kSgd ? smem_u32(&ctrl->loaded[cp.slot]) : smem_u32(&ctrl->free_[cp.slot]);
        if (!mbar_wait(bar, kSgd ? cp.phase : cp.phase ^ 1, abort_word, limit)) {
          report_status(args.status, CCF_ERR_MBAR_TIMEOUT, 0x66);
          ok = false;
          break;
        }
        const uint32_t at = ring + cp.slot * kWgChunkBytes + row_at;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float f[32];
          if (have_acc) {
            uint32_t r[32];
            tmem_ld32(t_row + c * 64 + h * 32, r);
            tmem_ld_wait();
            acc_to_float(r, f);
            if (h == 1 && c + 2 >= ti.chunks) release();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) f[i] = 0.f;
          }
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const uint32_t a = at + ((static_cast<uint32_t>(h * 4 + p) << 4) ^ swz);
            uint32_t w[4];
            if constexpr (kSgd) {
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(a) : "memory");
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float2 v = unpack2(w[j], kFp16);
                const f32x2 w2 = pk2(v.x, v.y);
                float n0, n1;
                upk2(fma2(bc2(-lr), fma2(bc2(wd), w2, pk2(f[8 * p + 2 * j], f[8 * p + 2 * j + 1])), w2), n0, n1);
                w[j] = pack2(n0, n1, kFp16);
              }
            } else {
#pragma unroll
              for (int j = 0; j < 4; ++j) w[j] = pack2(f[8 * p + 2 * j], f[8 * p + 2 * j + 1], kFp16);
            }
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // these writes before the store's reads
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctrl->done[cp.slot]));
      }
      if (warp == 4 && lane == 0) trace_ev(args, seq, 7);
      pos.advance(ti.chunks);
      if (have_acc && ++as == 2) { as = 0; aphase ^= 1; }
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
}

template <int FP16, bool SGD>
static int launch_wgrad_variant(const CUtensorMap* tm, const CcfGemmArgs& args, int grid, int early, cudaStream_t stream) {
  auto kern = grouped_wgrad_kernel<FP16, SGD>;
  // the attribute belongs to the (function, device) pair: set it once per device this process launches on
  static bool configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgSmemBytes);
    if (e != cudaSuccess) return -static_cast<int>(e);
    configured[dev & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid & ~1);
  cfg.blockDim = dim3(kWgThreads);
  cfg.dynamicSmemBytes = kWgSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2] = {cluster_attribute(2, 1, 1), early_attribute()};
  cfg.attrs = attr;
  cfg.numAttrs = early ? 2 : 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tm[0], tm[2], tm[4], args);
  return e == cudaSuccess ? 0 : -static_cast<int>(e);
}

// tm[0]: A, tm[2]: B, tm[4]: the result (boxes of 64 columns x 128 rows)
int launch_wgrad(const CUtensorMap* tm, const CcfGemmArgs& a, int grid, int early, cudaStream_t stream) {
  const bool sgd = a.sgd_lr != 0.f;
  if (a.fp16) return sgd ? launch_wgrad_variant<1, true>(tm, a, grid, early, stream) : launch_wgrad_variant<1, false>(tm, a, grid, early, stream);
  return sgd ? launch_wgrad_variant<0, true>(tm, a, grid, early, stream) : launch_wgrad_variant<0, false>(tm, a, grid, early, stream);
}

}  // namespace ccf
