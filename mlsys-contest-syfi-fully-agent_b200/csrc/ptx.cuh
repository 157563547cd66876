// Thin inline-PTX wrappers for the sm_100a features the kernels use:
// mbarrier (with bounded waits), TMA tiled loads (no multicast), tcgen05
// (TMEM allocation, UMMA issue/commit, TMEM loads) and their fences.
//
// Every wait in this file is bounded: after MOE_WAIT_LIMIT_NS without progress
// it raises a CTA-wide abort flag and returns false, so a kernel can never spin
// forever; the caller records an error bit and falls through to its teardown.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#ifndef MOE_WAIT_LIMIT_NS
#define MOE_WAIT_LIMIT_NS 400000000ull   // 0.4 s: four orders of magnitude above any legitimate wait here
#endif

namespace moe {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// One lane of a converged warp, always the same one.  Around tcgen05 and TMA instructions this and not `lane == 0`: four
// UMMAs and a commit measured 200 clocks of issue under it and 430 under `lane == 0`, whatever the UMMAs' size.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xFFFFFFFF;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(p));
  return p != 0;
}
// The warp's index as a value the compiler knows to be the same in all lanes.
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xFFFFFFFFu, static_cast<int>(threadIdx.x >> 5), 0); }

// ----------------------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(bar),
               "r"(bytes)
               : "memory");
}

// One poll by all 32 lanes of a converged warp: true in every lane if the phase is complete for all of them.
__device__ __forceinline__ bool mbar_try_wait_all(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "vote.sync.all.pred q, p, 0xFFFFFFFF;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

// Bounded wait of a whole converged warp.  Every lane gets the same answer: what follows a wait in the kernels (elect.sync,
// ballots, shuffles, tcgen05.ld) needs all 32 lanes, and lanes that left on a timeout while others saw the phase
// complete would be waited for without a limit.  `abort_flag` lives in shared memory and is shared by every role of the
// CTA: the first warp that times out sets it, the others see it on a later poll and leave too.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  uint64_t t0 = 0;
  uint32_t spins = 0;
  while (!mbar_try_wait_all(bar, parity)) {
    if ((++spins & 0x3Fu) == 0) {
      const uint64_t t = globaltimer_ns();
      if (t0 == 0) t0 = t;
      const bool late = t - t0 > MOE_WAIT_LIMIT_NS;
      if (late) *abort_flag = 1;
      if (__any_sync(0xFFFFFFFFu, late || *abort_flag != 0)) return false;
    }
  }
  return true;
}

// The same with one poll in front of the loop, for the kernels that run the same waits over and over: the large-batch
// GEMMs take 1.2 to 2 % less with it (T = 14107: 0.6 % less than with a wait that does not vote, instead of 1.5 % more).
// A decode call, which runs every wait a few times, takes up to 0.5 us more with it.
__device__ __forceinline__ bool mbar_wait_hot(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  return mbar_try_wait_all(bar, parity) || mbar_wait(bar, parity, abort_flag);
}

// ----------------------------------------------------------------------------- cp.async (4 bytes per thread)
// Asynchronous copy global -> shared memory; `cp_async_arrive` makes the mbarrier phase wait for all of the calling
// thread's earlier copies (one ordinary arrival, counted in the barrier's init count, when they have landed).
__device__ __forceinline__ void cp_async4(uint32_t dst_smem, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst_smem), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// Teardown of a CTA that has given up a wait, before it frees its TMEM and returns: its own copies and UMMAs may still be
// in flight, and they write shared memory and TMEM that belong to somebody else once it has left.  The barriers they
// report to can be half armed (a role that left early has not arrived), so this waits for time and not for them:
// MOE_ABORT_SETTLE_NS, hundreds of times what a load or a stage of UMMAs takes.
// The warp that frees the TMEM does it; it keeps the CTA's shared memory as well.
#ifndef MOE_ABORT_SETTLE_NS
#define MOE_ABORT_SETTLE_NS 1000000ull
#endif
__device__ __forceinline__ void settle_after_abort() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  const uint64_t t0 = globaltimer_ns();
  while (globaltimer_ns() - t0 < MOE_ABORT_SETTLE_NS) __nanosleep(1000);
}

// ----------------------------------------------------------------------------- TMA (tiled, no multicast)
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}

// 3-D / 4-D tiled loads global -> this CTA's shared memory, completion on an mbarrier.
// x is the innermost (byte) coordinate and must be a multiple of 16 for u8 data.
__device__ __forceinline__ void tma_load_3d(uint32_t dst_smem, const CUtensorMap* m, int x, int y, int z, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst_smem, const CUtensorMap* m, int x, int y, int z, int w,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
      ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
      : "memory");
}

// Request a tile of a 3-D tensor map into L2 only (no shared-memory destination, no completion to wait for).
__device__ __forceinline__ void tma_prefetch_l2_3d(const CUtensorMap* m, int x, int y, int z) {
  asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(z)
               : "memory");
}

// ----------------------------------------------------------------------------- tcgen05 / TMEM
// Allocate `ncols` (power of two >= 32) TMEM columns; the base address is written to *smem_dst.
// Must be executed by one full warp.
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

__device__ __forceinline__ void tc_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Shared-memory matrix descriptor for a K-major operand tile stored as rows of
// 128 bytes with the 128-byte swizzle (what a TMA SWIZZLE_128B box of 128 bytes
// inner extent produces): 8-row groups are 1024 bytes apart (SBO), the leading
// offset is unused for swizzled K-major layouts, descriptor version 1 (sm_100),
// layout type 2 (SWIZZLE_128B).
__host__ __device__ constexpr uint64_t umma_desc_k_sw128(uint32_t smem_addr) {
  return static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4)        // start address, bits [0,14)
         | (static_cast<uint64_t>(1) << 16)                         // leading byte offset (ignored), bits [16,30)
         | (static_cast<uint64_t>(1024 >> 4) << 32)                 // stride byte offset, bits [32,46)
         | (static_cast<uint64_t>(1) << 46)                         // version = 1, bits [46,48)
         | (static_cast<uint64_t>(2) << 61);                        // SWIZZLE_128B, bits [61,64)
}

// Instruction descriptor for kind::f8f6f4, A and B both e4m3 and K-major, fp32 accumulate.
__host__ __device__ constexpr uint32_t umma_idesc_e4m3(int M, int N) {
  return (1u << 4)                                   // D format: f32
         | (0u << 7) | (0u << 10)                    // A, B format: e4m3
         | (0u << 15) | (0u << 16)                   // A, B K-major
         | (static_cast<uint32_t>(N >> 3) << 17)     // N / 8
         | (static_cast<uint32_t>(M >> 4) << 24);    // M / 16
}

// D[tmem] (+)= A[smem] * B[smem]^T, one 128 x N x 32 fp8 UMMA.  Issued by ONE thread.
__device__ __forceinline__ void umma_f8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// mbarrier arrive once all UMMAs previously issued by this thread have completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// TMEM -> registers: this warp's 32 lanes x 8 consecutive fp32 columns.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr)
      : "memory");
}

// TMEM -> registers: this warp's 32 lanes x 16 consecutive fp32 columns.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// TMEM -> registers: this warp's 32 lanes x 32 consecutive fp32 columns.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

// 32-byte store (a full DRAM sector) of eight consecutive floats; the address must be 32-byte aligned.
__device__ __forceinline__ void st_global_v8(float* p, const float* v) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

// acc[0..N) += v[0..N) * f with the packed two-element fp32 FMA of sm_100 (each element is one IEEE fma, the
// same result as fmaf): half the instructions of the scalar form.
template <int N>
__device__ __forceinline__ void fma_scaled(float* acc, const float* v, float f) {
  const float2 ff = make_float2(f, f);
#pragma unroll
  for (int x = 0; x < N / 2; ++x) {
    const float2 r = __ffma2_rn(make_float2(v[2 * x], v[2 * x + 1]), ff, make_float2(acc[2 * x], acc[2 * x + 1]));
    acc[2 * x] = r.x;
    acc[2 * x + 1] = r.y;
  }
}

// Register reallocation between warpgroups (each executed by all four warps of a warpgroup).
template <int N>
__device__ __forceinline__ void setmaxnreg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void setmaxnreg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }

// Named barrier for a subset of the CTA's warps.
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

}  // namespace moe
