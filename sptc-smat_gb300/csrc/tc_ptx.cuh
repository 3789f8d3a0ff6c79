// tc_ptx.cuh — inline-PTX building blocks for sm_103a: mbarriers with bounded
// waits, bulk copies, tcgen05 (TMEM alloc, MMA, commit, loads) and the
// shared-memory matrix descriptors the MMA reads its operands through.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>
#include <cstdint>

namespace smat {
namespace dev {

// A bounded wait gives up after this long (ns, unless the launch passes a
// limit of its own) and reports SMAT_ERR_TIMEOUT.
constexpr uint64_t kWaitTimeoutNs = 4000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// One lane of a converged warp. Code under this predicate is known to run on a
// single lane, so the compiler keeps descriptors and barrier addresses in
// uniform registers; under `lane == 0` it does not (measured: one thread
// issues a 128 x 16 x 16 tcgen05.mma every 64-75 cycles here, every 108-137
// there, and a 4 KB bulk copy every 55 instead of 110).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(p));
  return p != 0;
}

// Polls a phase up to a few hundred times (tens of microseconds) in a loop
// whose branch takes the barrier's predicate itself: about 75 cycles a turn
// when the phase is already complete, against 150-230 for a C++ loop over
// mbar_try_wait. Waits that outlast it go on in mbar_wait, which keeps time.
__device__ __forceinline__ bool mbar_poll(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n .reg .u32 it;\n mov.u32 it, 0;\n"
      "POLL:\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n @p bra DONE;\n"
      " add.u32 it, it, 1;\n setp.lt.u32 p, it, 400;\n @p bra POLL;\n setp.ne.u32 p, it, it;\n"
      "DONE:\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Wait for the phase with the given parity to complete. Gives up when the
// CTA's abort flag is raised or after `lim` ns; in the latter case it raises
// the abort flag and records `where` in the global error word.
static __device__ __noinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort, int* err,
                                       int where, uint64_t lim) {
  const uint64_t t0 = globaltimer();
  for (;;) {
    if (mbar_poll(bar, parity)) return true;
    if (*abort) return false;
    if (globaltimer() - t0 > lim) {
      *abort = 1;
      atomicCAS(err, 0, where);
      return false;
    }
  }
}

// mbar_wait for waits expected to be long (a whole panel): after a few
// polls the thread sleeps between them so that it leaves the issue slots of
// its SM sub-partition to the warps on the critical path.
static __device__ __noinline__ bool mbar_wait_sleepy(uint32_t bar, uint32_t parity, volatile int* abort, int* err,
                                              int where, uint64_t lim) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer();
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if (it > 4) __nanosleep(256);
    if ((it & 7u) == 0) {
      if (*abort) return false;
      if (globaltimer() - t0 > lim) {
        *abort = 1;
        atomicCAS(err, 0, where);
        return false;
      }
    }
  }
}

// 1-D bulk copy global -> this CTA's shared memory, completing on `bar`.
// Both addresses 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar)
      : "memory");
}
__device__ __forceinline__ uint64_t make_l2_policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t make_l2_policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
// Generic-proxy writes to shared memory made visible to the async proxy
// (the tensor core's operand reads) before a barrier hands them over.
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Two e4m3 values (low byte -> low half) to two FP16 values, exactly.
__device__ __forceinline__ __half2 e4m3x2_to_half2(uint16_t v) {
  uint32_t r;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(r) : "h"(v));
  return *reinterpret_cast<__half2*>(&r);
}

// The 128-byte line of `p` into L2.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Programmatic dependent launch: wait until the kernels this one was launched
// behind are complete and their writes visible (nothing to wait for in an
// ordinary launch); let the kernel launched behind this one begin its set-up.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------- tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem),
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

// D[tmem] (+)= A[smem] * B[smem], kind::f16 (FP16 or BF16 in, FP32 accumulate).
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                         uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrive once on `bar` when every tcgen05 operation this thread issued so far
// has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   bar)
               : "memory");
}

// Each thread of the warp reads 16 consecutive 32-bit TMEM columns of its lane.
__device__ __forceinline__ void tmem_ld_x16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// Each thread of the warp writes zeros to 16 consecutive 32-bit TMEM
// columns of its lane, and waits until the stores are done.
__device__ __forceinline__ void tmem_st_x16_zero(uint32_t taddr) {
  const uint32_t z = 0;
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
      "r"(z)
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Each thread of the warp reads 32 consecutive 32-bit TMEM columns of its
// lane (one load and one wait for what two x16 loads would bring).
__device__ __forceinline__ void tmem_ld_x32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}

// Shared-memory matrix descriptor of a K-major operand stored with the
// 32-byte swizzle: rows of 32 bytes (16 x 16-bit elements = one MMA K step),
// 8-row groups 256 bytes apart. The tile must start on a 256-byte boundary.
__device__ __forceinline__ uint64_t desc_kmajor_sw32(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);  // start address, 16-byte units
  d |= static_cast<uint64_t>(1) << 16;                  // leading-dim offset (unused here)
  d |= static_cast<uint64_t>(256 >> 4) << 32;           // stride-dim offset: 256 B
  d |= static_cast<uint64_t>(1) << 46;                  // descriptor version for tcgen05
  d |= static_cast<uint64_t>(6) << 61;                  // layout: 32-byte swizzle
  return d;
}

// Shared-memory matrix descriptor of the M operand stored MN-major with the
// 128-byte swizzle: K rows of 64 16-bit values (128 bytes), 8-row groups 1,024
// bytes apart (stride), the next 64 values of M `lead` bytes on (leading
// dimension). The tile must start on a 1,024-byte boundary.
__device__ __forceinline__ uint64_t desc_mnmajor_sw128(uint32_t saddr, uint32_t lead) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(lead >> 4) << 16;
  d |= static_cast<uint64_t>(1024 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;  // descriptor version for tcgen05
  d |= static_cast<uint64_t>(2) << 61;  // layout: 128-byte swizzle
  return d;
}

// 16 bytes global -> shared through the load path, zeros when bytes == 0.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// One arrival on `bar` (counted against its expected arrivals) when this
// thread's earlier cp.async have landed.
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// Predicated forms for whole-warp code: a branch around a few lanes' copies
// splits the warp, and putting it together again costs more than they do (one
// polling lane in place of 32 took the R-MAT step from 115 to 149 us).
__device__ __forceinline__ void mbar_expect_tx_if(uint32_t bar, uint32_t bytes, bool pred) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;\n}" ::"r"(
          bar),
      "r"(bytes), "r"((uint32_t)pred)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx_if(uint32_t bar, uint32_t bytes, bool pred) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %2, 0;\n @p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n}" ::"r"(
          bar),
      "r"(bytes), "r"((uint32_t)pred)
      : "memory");
}
__device__ __forceinline__ void bulk_load_hint_if(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar,
                                                  uint64_t policy, bool pred) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %5, 0;\n"
      " @p cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], "
      "%4;\n}" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(bar), "l"(policy), "r"((uint32_t)pred)
      : "memory");
}

}  // namespace dev
}  // namespace smat
