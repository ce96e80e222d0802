// Raw PTX wrappers for the Blackwell (sm_100a) data path: mbarrier, TMA tiled loads, tcgen05 MMA with
// TMEM accumulators, shared-memory matrix descriptors. No CUTLASS / CuTe dependency.
//
// Every wait is bounded: it gives up after `limit_ns` of wall time (globaltimer) or when the CTA-wide
// abort word is set, and returns false so that the caller can record a status and leave the kernel
// through its normal exit (TMEM freed, no trap).
#pragma once
#include <cuda_runtime.h>
#include <cuda.h>
#include <stdint.h>

namespace ccf {

// ----------------------------------------------------------------------------------------------
// small helpers
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

// True in one lane of a converged warp, the same one every time. TMA and tcgen05 instructions take their operands from uniform
// registers; behind this predicate the compiler knows that one lane runs and issues them back to back. Behind `lane == 0` it
// does not, and a tcgen05.mma took 138 clocks to issue whatever its size, where a 128 x 256 x 16 one takes 128 to run (an isolated
// loop of either, one CTA per SM; with this predicate the loop runs at 128).
__device__ __forceinline__ bool elect_one() {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok));
  return ok != 0;
}

// host: launch attribute of a cluster
inline cudaLaunchAttribute cluster_attribute(unsigned x, unsigned y, unsigned z) {
  cudaLaunchAttribute a;
  a.id = cudaLaunchAttributeClusterDimension;
  a.val.clusterDim.x = x;
  a.val.clusterDim.y = y;
  a.val.clusterDim.z = z;
  return a;
}

// Launches of one pass can follow each other without the gap of a stream's order: a kernel with this attribute may be set up while the
// kernel in front of it still runs, and waits for its end, and its memory, in wait_for_previous().
// Only for calls of few slots: 16 tokens, 16 experts of 1024 x 4096 92 -> 84 us a pass, 777 tokens, 64 experts of 2048 x 8192 717 -> 714;
// at 16384 slots, where the gaps are a percent of a pass, passes of 4 experts of 1024 x 4096 and of 64 of 2048 x 8192 were 1 to 3 % slower
// with it (942 -> 952 and 4949 -> 5112 us). In between nothing is slower outside the noise, and small layers gain: the line could lie higher. us
// without / with at 4096, 6144, 8192, 12288 and 16384 slots:
//   512 x 2048, 16 experts     inference 86 / 76, 100 / 88, 117 / 107, 130 / 121, 143 / 132; training 246 / 240, 272 / 259, 318 / 300, 364 / 346, 407 / 386
//   1024 x 4096, 16 experts    inference 131 / 123, 165 / 157, 200 / 191, 255 / 244, 284 / 277; training 375 / 361, 468 / 455, 577 / 560, 736 / 721, 862 / 850
//   2048 x 8192, 64 experts    inference 724 / 719, 757 / 751, 791 / 786, 902 / 896, 1078 / 1079; training 2445 / 2419, 2547 / 2550, 2750 / 2725,
//                              3303 and 2913 / 3302 and 3318 (two runs each), 3965 / 4021
// Not under capture: the edges of a graph leave 0.4 us, and with the attribute 128 tokens, 4096 x 14336, took 511 us instead of 508.
constexpr long long kEarlySlots = 4096;
inline int early_launches(long long slots, cudaStream_t stream) {
  if (slots > kEarlySlots) return 0;
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &st) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return st == cudaStreamCaptureStatusNone;
}
inline cudaLaunchAttribute early_attribute() {
  cudaLaunchAttribute a;
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}
// Every thread calls wait_for_previous() before its first access to memory that another kernel may write or read. Only then is the next
// kernel let in: what runs before its own wait overlaps this kernel alone, never one further back. A kernel with tensor memory takes it
// in between: columns held during the wait could be the ones that the kernel in front still needs, and since one thread of a CTA is enough
// to let the next kernel in, its CTAs could otherwise hold the columns that this CTA has yet to get, and wait for it.
// It costs nothing: 16 tokens, 16 experts of 1024 x 4096 83.3 us a pass, with the columns taken in front of the wait 84.5.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_in() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void after_previous() {
  wait_for_previous();
  let_next_in();
}
// A pointer for reads behind wait_for_previous(): reads through the read-only path are otherwise free to move in front of it.
template <typename T>
__device__ __forceinline__ T* behind(T* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}

// ----------------------------------------------------------------------------------------------
// packed fp32 pairs: one instruction for two fused multiply-adds, each rounded as the scalar one
// ----------------------------------------------------------------------------------------------
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void upk2(f32x2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 bc2(float v) { return pk2(v, v); }

// ----------------------------------------------------------------------------------------------
// mbarrier
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait. `abort_word` lives in shared memory; whoever times out sets it, everyone else sees it.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_word,
                                          uint64_t limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 63u) == 0u) {
      if (*abort_word) return false;
      if (globaltimer_ns() - t0 > limit_ns) {
        *abort_word = 1;
        return false;
      }
    }
  }
  return true;
}

// ----------------------------------------------------------------------------------------------
// thread-block clusters
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of the same shared-memory location in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t cluster_addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr) : "memory");
  return v;
}

// ----------------------------------------------------------------------------------------------
// TMA (tiled 2-D loads, this GPU's memory only, never multicast)
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}

// c0 = coordinate along the contiguous dimension (elements), c1 = row
__device__ __forceinline__ void tma_load_2d(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar, int c0,
                                            int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_dst), "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}

// untiled copy global -> shared (16-byte aligned addresses, size a multiple of 16 bytes)
__device__ __forceinline__ void bulk_load(uint32_t smem_dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_dst),
               "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
               : "memory");
}

// ----------------------------------------------------------------------------------------------
// tcgen05: TMEM allocation, MMA, commit, loads, fences
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// D[tmem] (+)= A[smem desc] * B[smem desc]; one thread issues.
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// The mbarrier gets one arrival when every MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns -> 32 registers per thread (thread i = lane i of the warp's quarter)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ----------------------------------------------------------------------------------------------
// descriptors
// ----------------------------------------------------------------------------------------------
// Shared-memory matrix descriptor, 128-byte swizzle, Blackwell version field = 1.
//   K-major  tile (rows x 64 elements of 2 bytes, one 128-byte row per matrix row as TMA writes it):
//            SBO = 1024 B (eight rows), LBO unused; advance 32 B per UMMA_K = 16.
//   MN-major tile (boxes of 64 MN-elements x BK k-rows, 128 B per k-row):
//            SBO = 1024 B (eight k-rows), LBO = byte distance of two 64-element MN groups
//            (= BK * 128 B when every group is one TMA box); advance 2048 B per UMMA_K = 16.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= static_cast<uint64_t>(1) << 46;  // descriptor version (Blackwell)
  d |= static_cast<uint64_t>(2) << 61;  // SWIZZLE_128B
  return d;
}

// Instruction descriptor for kind::f16 with fp32 accumulation.
//   fp16_inputs: 0 = bf16 operands, 1 = fp16 operands; a_mn / b_mn: 1 = MN-major operand.
__host__ __device__ __forceinline__ uint32_t make_idesc(int m, int n, int fp16_inputs, int a_mn, int b_mn) {
  uint32_t fmt = fp16_inputs ? 0u : 1u;
  uint32_t d = 0;
  d |= 1u << 4;              // accumulator format F32
  d |= fmt << 7;             // A format
  d |= fmt << 10;            // B format
  d |= uint32_t(a_mn) << 15;
  d |= uint32_t(b_mn) << 16;
  d |= uint32_t(n >> 3) << 17;
  d |= uint32_t(m >> 4) << 24;
  return d;
}

// ----------------------------------------------------------------------------------------------
// system-scope flags (peer memory over NVLink)
// ----------------------------------------------------------------------------------------------
__device__ __forceinline__ void red_release_sys_add(int* addr, int v) {
  asm volatile("red.release.sys.global.add.s32 [%0], %1;" ::"l"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void red_release_gpu_add(int* addr, int v) {
  asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_release_sys(int* addr, int v) {
  asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_acquire_sys(const int* addr) {
  int v;
  asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(addr) : "memory");
  return v;
}
__device__ __forceinline__ int ld_relaxed_sys(const int* addr) {
  int v;
  asm volatile("ld.relaxed.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(addr) : "memory");
  return v;
}

// Spin until *addr has reached target (bounded); the completion counters wrap around, so it is their distance that counts.
// Returns false on timeout.
__device__ __forceinline__ bool flag_reached(const int* addr, int target) {
  return static_cast<int>(static_cast<unsigned>(ld_acquire_sys(addr)) - static_cast<unsigned>(target)) >= 0;
}
__device__ __forceinline__ bool wait_flag_ge(const int* addr, int target, uint64_t limit_ns) {
  if (flag_reached(addr, target)) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (!flag_reached(addr, target)) {
    if ((++spins & 31u) == 0u) {
      if (globaltimer_ns() - t0 > limit_ns) return false;
      __nanosleep(64);
    }
  }
  return true;
}

}  // namespace ccf
