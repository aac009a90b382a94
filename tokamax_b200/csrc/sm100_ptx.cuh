// Thin inline-PTX layer for sm_100a: mbarrier, TMA tile loads, tcgen05 (UMMA) MMA with
// TMEM accumulators, TMEM load/store, and the shared-memory / instruction descriptors the
// MMA consumes.  Everything here is single-CTA (cta_group::1) and uses plain TMA loads only.
//
// Every wait on an mbarrier is bounded: after kWaitLimitCycles the waiter raises a
// CTA-wide abort flag plus a global error word and falls through, so a protocol bug ends
// the kernel with a status code instead of hanging the GPU.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cstdint>

namespace sb {

// ----------------------------------------------------------------------------------------
// error reporting
// ----------------------------------------------------------------------------------------
// Layout of the device error record (4 x uint32): [0] code (0 = ok), [1] blockIdx.x |
// blockIdx.y<<16, [2] tag of the barrier that timed out, [3] threadIdx.x.
enum : uint32_t { kErrNone = 0, kErrWaitTimeout = 1 };

constexpr long long kWaitLimitCycles = 1500000000ll;  // ~0.8 s at 1.9 GHz

struct AbortCtx {
  volatile uint32_t* cta_flag;   // shared memory word, non-zero once any wait gave up
  uint32_t* global_err;          // device error record (may not be null)
  long long limit_cycles = kWaitLimitCycles;  // a compile-time constant wherever it is not set
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// One lane of a converged warp.  The threads that issue TMA copies and MMAs are chosen with this and
// not with `lane == 0`: from elect.sync the compiler knows that a single thread runs what follows, and
// the MMA's operands (descriptors, TMEM addresses, all of them uniform registers) then cost it a few
// instructions.  Behind a lane test it needs 90 .. 110 cycles for an MMA that runs 64, so that the
// issuing thread was what the kernels waited for.  Measured, `lane == 0` -> elect (us):
//   forward causal 8192, 4 x 32 / 8 heads   2153 -> 1983     forward / backward, one launch each, causal 8192,
//   fused dkv, the same                     5718 -> 5706     16 / 8 heads, head dim 256:  787 -> 676 (forward),
//   dq, causal 4096, 2 x 16 / 1 heads, d 64  163 -> 146      864 -> 772 (dq), 1130 -> 994 (dk), 739 -> 618 (dv)
//   dkv, the same                            870 -> 745
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(pred));
  return pred != 0;
}

// ----------------------------------------------------------------------------------------
// mbarrier
// ----------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: gives up after ab.limit_cycles (by default under a second), or as soon as another thread
// of the CTA has given up.  Returns false if the wait was abandoned.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const AbortCtx& ab,
                                          uint32_t tag) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long start = clock64();
  for (uint32_t spin = 0;; ++spin) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((spin & 15u) == 15u) {
      if (*ab.cta_flag) return false;
      if (clock64() - start > ab.limit_cycles) break;
    }
  }
  *ab.cta_flag = 1u;
  if (atomicCAS(ab.global_err, 0u, (uint32_t)kErrWaitTimeout) == 0u) {
    ab.global_err[1] = blockIdx.x | (blockIdx.y << 16);
    ab.global_err[2] = tag;
    ab.global_err[3] = threadIdx.x;
  }
  return false;
}

// Before a CTA leaves whose waits have run out: its copies, MMAs and answers from cluster launch control may still be in
// flight towards shared memory and TMEM that are another CTA's next.  They land within microseconds.
constexpr long long kDrainCycles = 1000000ll;  // ~0.5 ms
__device__ __forceinline__ void drain_after_give_up(const volatile uint32_t* cta_flag) {
  if (*cta_flag == 0u) return;
  const long long start = clock64();
  while (clock64() - start < kDrainCycles) {
  }
}

// ----------------------------------------------------------------------------------------
// thread-block clusters: barrier over all threads of the cluster, loads from a peer CTA's shared memory
// ----------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();  // .aligned: the warp's threads together
  asm volatile(
      "barrier.cluster.arrive.release.aligned;\n\t"
      "barrier.cluster.wait.acquire.aligned;\n" ::
          : "memory");
}
// address, in the cluster's shared window, of what `p` is in this CTA, in CTA `rank`
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ float4 cluster_ld_v4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ uint32_t cluster_ld_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

// ----------------------------------------------------------------------------------------
// cluster launch control: a running CTA takes over the next one that has not been launched yet
// ----------------------------------------------------------------------------------------
// Asks for it; the answer (16 bytes, 16-byte aligned shared memory) completes 16 bytes on `bar`.  No further
// request may follow one that was refused.
__device__ __forceinline__ void clc_request(void* answer, uint64_t* bar) {
  asm volatile(
      "clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
          smem_u32(answer)),
      "r"(smem_u32(bar))
      : "memory");
}
// blockIdx.x of the CTA whose work this one takes over, or -1: none is left.
__device__ __forceinline__ int clc_block(const void* answer) {
  int block;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 r;\n\t"
      "ld.shared.b128 r, [%1];\n\t"
      "mov.s32 %0, -1;\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %0, r;\n\t}\n"
      : "=r"(block)
      : "r"(smem_u32(answer))
      : "memory");
  return block;
}

// 16 bytes of shared memory, whether or not they have been read before
__device__ __forceinline__ int4 ld_again(const int4* p) {
  int4 v;
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(smem_u32(p))
               : "memory");
  return v;
}

// ----------------------------------------------------------------------------------------
// TMA (tiled, no multicast)
// ----------------------------------------------------------------------------------------
__device__ __forceinline__ void tma_prefetch_desc(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
}

__device__ __forceinline__ void tma_load_4d(void* smem_dst, const void* tmap, uint64_t* bar,
                                            int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5}], [%6];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(c2),
        "r"(c3), "r"(smem_u32(bar))
      : "memory");
}

// Untiled bulk copy global -> shared (both addresses 16-byte aligned, size a multiple of 16).
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gmem_src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(gmem_src)), "r"(bytes),
        "r"(smem_u32(bar))
      : "memory");
}

// Bulk reduction shared -> global: adds `bytes` of fp32 to what is there (both addresses 16-byte aligned, size a multiple of
// 16).  A bulk group of its own; the shared memory may be written again behind bulk_wait_read().
__device__ __forceinline__ void bulk_reduce_add(float* gmem_dst, const void* smem_src, uint32_t bytes) {
  asm volatile(
      "cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;\n\t"
      "cp.async.bulk.commit_group;"
      :
      : "l"(gmem_dst), "r"(smem_u32(smem_src)), "r"(bytes)
      : "memory");
}
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void tma_store_4d(const void* tmap, const void* smem_src, int c0,
                                             int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
      :
      : "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(smem_src)), "r"(c0), "r"(c1), "r"(c2),
        "r"(c3)
      : "memory");
}
__device__ __forceinline__ void tma_store_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void tma_store_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ----------------------------------------------------------------------------------------
// tcgen05: TMEM allocation, fences, commit
// ----------------------------------------------------------------------------------------
// Warp-collective.  Writes the TMEM base address to *smem_dst.
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Fence the MMA-issuing thread executes between an mbarrier wait and the MMAs that consume what
// the wait published (TMEM written by other warps' tcgen05.st, or TMEM columns other warps have
// finished reading): the consumer half of the before_thread_sync / after_thread_sync pair the
// tcgen05 ordering rules ask for.
__device__ __forceinline__ void mma_issue_fence() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// One thread: the mbarrier receives one arrival once every tcgen05 async op this thread
// issued before the commit has completed.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

// ----------------------------------------------------------------------------------------
// descriptors
// ----------------------------------------------------------------------------------------
// Shared-memory matrix descriptor, 128-byte swizzle, descriptor version 1 (sm_100).
//   bits [0,14)  start address >> 4        bits [16,30) leading byte offset >> 4
//   bits [32,46) stride byte offset >> 4   bits [46,48) version = 1
//   bits [61,64) layout type (2 = SWIZZLE_128B)
// Kept as two 32-bit words: every field that changes from one K-slice to the next lives in the
// low word (the start address), so stepping through a tile is one 32-bit add per operand — the
// thread that issues the MMAs shares its scheduler with busy compute warps, and the fewer
// instructions it needs per MMA the closer the issue rate gets to what the tensor pipe can take.
struct SmemDesc {
  uint32_t lo, hi;
};
__device__ __forceinline__ SmemDesc make_smem_desc_sw128(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  SmemDesc d;
  d.lo = ((saddr & 0x3FFFFu) >> 4) | (((lbo_bytes >> 4) & 0x3FFFu) << 16);
  d.hi = ((sbo_bytes >> 4) & 0x3FFFu) | (1u << 14) | (2u << 29);
  return d;
}
// The same descriptor `bytes` further into the tile (bytes a multiple of 16; shared memory is
// smaller than 2^18 bytes, so the 14-bit address field cannot carry into its neighbour).
__device__ __forceinline__ SmemDesc desc_at(SmemDesc d, uint32_t bytes) {
  d.lo += bytes >> 4;
  return d;
}

// Instruction descriptor for kind::f16 with bf16 A/B and fp32 accumulation.
//   [4,6) D format (1 = f32)  [7,10) A format (1 = bf16)  [10,13) B format (1 = bf16)
//   [15] A major (0 = K)      [16] B major (0 = K, 1 = MN)
//   [17,23) N >> 3            [24,29) M >> 4
__host__ __device__ constexpr uint32_t make_idesc_bf16(int m, int n, bool a_mn_major,
                                                       bool b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn_major ? 1u : 0u) << 15) |
         ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// Instruction descriptor for kind::f8f6f4 with e4m3 A/B (format code 0) and fp32 accumulation;
// the other fields are those of make_idesc_bf16.
__host__ __device__ constexpr uint32_t make_idesc_e4m3(int m, int n, bool a_mn_major,
                                                       bool b_mn_major) {
  return (1u << 4) | ((a_mn_major ? 1u : 0u) << 15) | ((b_mn_major ? 1u : 0u) << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, SmemDesc a, SmemDesc b, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}\n"
      :
      : "r"(d_tmem), "r"(a.lo), "r"(a.hi), "r"(b.lo), "r"(b.hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]   (A: one row per lane, two 16-bit values per column)
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, SmemDesc b, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}\n"
      :
      : "r"(d_tmem), "r"(a_tmem), "r"(b.lo), "r"(b.hi), "r"(idesc), "r"(accumulate)
      : "memory");
}

// The same two forms for 8-bit operands (K = 32 per instruction; A in TMEM holds four values per
// column).
__device__ __forceinline__ void umma_ss_f8(uint32_t d_tmem, SmemDesc a, SmemDesc b, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], da, db, %5, p;\n\t}\n"
      :
      : "r"(d_tmem), "r"(a.lo), "r"(a.hi), "r"(b.lo), "r"(b.hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_ts_f8(uint32_t d_tmem, uint32_t a_tmem, SmemDesc b, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
      "mov.b64 db, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], [%1], db, %4, p;\n\t}\n"
      :
      : "r"(d_tmem), "r"(a_tmem), "r"(b.lo), "r"(b.hi), "r"(idesc), "r"(accumulate)
      : "memory");
}

// ----------------------------------------------------------------------------------------
// TMEM <-> registers.  32x32b: thread t of the warp owns TMEM lane (32*(warp%4) + t) and
// reads/writes N consecutive 32-bit columns starting at the column in taddr.
// ----------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
        "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
        "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
        "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
        "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
        "r"(r[14]), "r"(r[15])
      : "memory");
}
// 16x256b / 16x128b: 16 lanes of TMEM (the lane in taddr and the 15 behind it), in the fragments of the matrix instructions:
// thread t holds rows t / 4 and t / 4 + 8.  A load brings 32-bit columns 8 k + 2 (t % 4) and the one behind it as
// r[4 k + 2 h], r[4 k + 2 h + 1] (h: which of the two rows); a store takes column 4 k + t % 4 from r[2 k + h], so that the
// 16-bit pairs of a load's columns go back as they lie.
constexpr uint32_t kLanes16 = 16u << 16;  // 16 lanes on in a TMEM address
__device__ __forceinline__ void tmem_ld_frag(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_frag(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
      : "memory");
}
// Four 8 x 8 matrices of 16-bit values from such fragments to shared memory: thread t gives the address of row t % 8 of
// matrix t / 8.
__device__ __forceinline__ void stmatrix_x4(uint32_t saddr, uint32_t m0, uint32_t m1, uint32_t m2, uint32_t m3) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(m0), "r"(m1), "r"(m2),
               "r"(m3)
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// ----------------------------------------------------------------------------------------
// small math helpers
// ----------------------------------------------------------------------------------------
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Three-input maximum (one instruction on sm_100).
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// tanh of two values of at most 1/2 each: y p(y^2) with p of degree 4 through tanh(y) / y at the Chebyshev nodes of 0 .. 1/4,
// two-wide in fp32 (error 4.1e-8 absolute, 1.1e-7 relative; 1 - 2 / (e + 1) on the same range 1.7e-7 absolute).  The scores of a soft
// cap lie far inside it, and it spares two of the three special-function operations a score, which take 3072 of a
// 128 x 128 tile's cycles: 3 x 1664, 12 / 4 heads, d 80, window 768: forward 63.8 -> 54.2 us, fused dkv 95.7 -> 82.0; 4 x 4096,
// 16 / 8, d 128: a pass 754 -> 641.
__device__ __forceinline__ float2 tanh_small(float2 y) {
  auto two = [](float c) { return make_float2(c, c); };
  const float2 z = __fmul2_rn(y, y);
  float2 p = __ffma2_rn(two(0.017131345346570015f), z, two(-0.05298423767089844f));
  p = __ffma2_rn(p, z, two(0.133247509598732f));
  p = __ffma2_rn(p, z, two(-0.3333306908607483f));
  p = __ffma2_rn(p, z, two(1.0f));
  return __fmul2_rn(p, y);
}
// Whether tanh_small() serves for a x, all N values x of all lanes of a warp (a > 0).
template <int N>
__device__ __forceinline__ bool tanh_is_small(const float (&x)[N], float a) {
  float top0 = 0.f, top1 = 0.f;
#pragma unroll
  for (int j = 0; j < N; j += 4) {
    top0 = max3(top0, fabsf(x[j]), fabsf(x[j + 1]));
    top1 = max3(top1, fabsf(x[j + 2]), fabsf(x[j + 3]));
  }
  return !__any_sync(0xffffffffu, fmaxf(top0, top1) * a > 0.5f);
}
// tanh of two values, in the form that each by itself calls for: tanh_small() up to 1/2, 1 - 2 / (e + 1) above, e = 2^(2 log2(e) y)
// (e = inf gives 1, e = 0 gives -1; tanh.approx.f32, relative error 2^-11, is too coarse for logits that must hold 1e-3 after
// being multiplied by a cap of tens).
__device__ __forceinline__ float2 tanh_each(float2 y) {
  auto two = [](float c) { return make_float2(c, c); };
  const float2 t = tanh_small(y), w = __fmul2_rn(y, two(2.8853900817779268f));
  const float2 d = __fadd2_rn(make_float2(ex2(w.x), ex2(w.y)), two(1.0f));
  const float2 u = __ffma2_rn(make_float2(rcp(d.x), rcp(d.y)), two(-2.0f), two(1.0f));
  return make_float2(fabsf(y.x) <= 0.5f ? t.x : u.x, fabsf(y.y) <= 0.5f ? t.y : u.y);
}
// x <- tanh(a x), N values a lane, by a whole warp; `small`: tanh_is_small() of them, which spares the second form.  Which of the
// two a value takes must not hang on the vote: a score's last bits would depend on all else that its warp holds, masked keys
// and other documents among it.  (Warps of both kinds pay for both forms: scores of 16 times the spread, 444 tiles: forward
// 8 heads, window 768, 135 -> 148 us, dkv 166 -> 175; causal, d 64, 1371 -> 1475, 1728 -> 1840.)
template <int N>
__device__ __forceinline__ void tanh_all(float (&x)[N], float a, bool small) {
  if (!small) {
#pragma unroll
    for (int j = 0; j < N; j += 2) {
      const float2 t = tanh_each(__fmul2_rn(make_float2(x[j], x[j + 1]), make_float2(a, a)));
      x[j] = t.x;
      x[j + 1] = t.y;
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < N; j += 2) {
    const float2 t = tanh_small(__fmul2_rn(make_float2(x[j], x[j + 1]), make_float2(a, a)));
    x[j] = t.x;
    x[j + 1] = t.y;
  }
}
template <int N>
__device__ __forceinline__ void tanh_all(float (&x)[N], float a) {
  tanh_all(x, a, tanh_is_small(x, a));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// Bit i: byte i of w is not 0.  (The product brings the four bits, 8 apart, side by side.)
__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t w) {
  const uint32_t top = (((w & 0x7f7f7f7fu) + 0x7f7f7f7fu) | w) & 0x80808080u;
  return (top >> 7) * 0x01020408u >> 24;
}

// Register reallocation between warpgroups (all four warps of a warpgroup must execute it).
template <int N>
__device__ __forceinline__ void setmaxnreg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void setmaxnreg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

// Named barrier among a subset of warps (ids 1..15; id 0 is __syncthreads).
__device__ __forceinline__ void named_barrier_sync(uint32_t id, uint32_t nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

}  // namespace sb
