// Device helpers shared by the tcgen05 kernels (k_tc.cu, k_fp4.cu): bounded mbarrier waits, TMA
// loads, cluster addressing and TMEM reads.
#pragma once
#include <cuda_runtime.h>
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cstdint>

namespace sg {
namespace tc {

// cuTensorMapEncodeTiled of the driver (nullptr when it has none), and the device address of the error
// flag every tcgen05 kernel reports expired waits to (nullptr on failure)
PFN_cuTensorMapEncodeTiled_v12000 tc_encode_fn();
int* tc_error_flag();

// Dynamic shared memory of a kernel about to be launched.  An earlier launch's error comes back first: setting the
// attribute clears it unread (CUDA 13.0), and that launch's output would be taken for written.
inline cudaError_t set_dynamic_smem(const void* kernel, size_t bytes) {
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? e : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

constexpr unsigned long long kWaitBudgetNs = 4000000000ull;  // 4 s per wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: returns false (and records ``code`` at ``err``) when the budget runs out
// or another thread of this kernel already gave up.  The global timer is read only after 64 failed
// tries: a read takes longer than most waits of a pipeline in flow.
__device__ __forceinline__ bool mbar_wait_budget(uint64_t* bar, uint32_t parity, int code,
                                                 volatile int* abort_flag, unsigned long long budget_ns,
                                                 int* err) {
  unsigned long long t0 = 0;
  for (uint32_t it = 1;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 63u) == 0u) {
      if (*abort_flag) return false;
      const unsigned long long t = gtimer();
      if (t0 == 0) t0 = t;
      if (t - t0 > budget_ns) {
        *abort_flag = 1;
        atomicCAS(err, 0, code);
        return false;
      }
    }
  }
}

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int code,
                                          volatile int* abort_flag, int* err) {
  return mbar_wait_budget(bar, parity, code, abort_flag, kWaitBudgetNs, err);
}

// Bounded wait with a sleeping back-off between polls, for waits that last a whole chunk of MMAs:
// the drain warps share the SM's schedulers with the single-lane TMA and MMA loops.
__device__ __forceinline__ bool mbar_wait_sleep(uint64_t* bar, uint32_t parity, int code,
                                                volatile int* abort_flag, int* err) {
  if (mbar_try_wait(bar, parity)) return true;
  unsigned long long t0 = 0;
  unsigned ns = 32;
  for (uint32_t it = 1;; ++it) {
    __nanosleep(ns);
    if (mbar_try_wait(bar, parity)) return true;
    if (ns < 256) ns <<= 1;
    if ((it & 15u) != 0u) continue;
    if (*abort_flag) return false;
    const unsigned long long t = gtimer();
    if (t0 == 0) t0 = t;
    if (t - t0 > kWaitBudgetNs) {
      *abort_flag = 1;
      atomicCAS(err, 0, code);
      return false;
    }
  }
}

// Bounded wait at teardown: the MMAs a CTA issued complete within microseconds once issued (their
// operands are already in shared memory), so this wait ignores the abort flag and gives up after
// 1 s without recording anything.
__device__ __forceinline__ void mbar_wait_teardown(uint64_t* bar, uint32_t parity) {
  const unsigned long long t0 = gtimer();
  while (!mbar_try_wait(bar, parity))
    if (gtimer() - t0 > 1000000000ull) return;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar,
                                            int32_t x, int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

// One lane of a converged warp, by elect.sync.  Behind a test of the lane number the same MMA loop took 45 clocks an
// instruction, behind this 17 (128 x 32 x 16 BF16, its operands' own rate).
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.b32 %0, 1, 0, q;\n\t}" : "=r"(e));
  return e != 0;
}

// ``bytes`` contiguous bytes (a multiple of 16, both addresses on 16-byte boundaries)
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Address of the same shared-memory location in CTA ``rank`` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}

// Arrive once on an mbarrier given by its cluster address (this CTA's or the peer's), with the default release
// at CTA scope: what these arrivals publish is in TMEM, ordered by the tcgen05 waits and fences before
// them.  (A release at cluster scope took 1,000-1,300 clocks of the arriving warp.)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster) : "memory");
}

// CTA-pair load: the box lands in this CTA's shared memory and completes its transaction bytes on
// the mbarrier at cluster address ``bar_cluster``, which may sit in the pair's other CTA.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint32_t bar_cluster,
                                                 int32_t x, int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster), "r"(x), "r"(y)
      : "memory");
}

template <bool kPair>
__device__ __forceinline__ void umma_commit(uint32_t bar_cluster) {
  if constexpr (kPair)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(bar_cluster) : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(bar_cluster) : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace tc
}  // namespace sg
