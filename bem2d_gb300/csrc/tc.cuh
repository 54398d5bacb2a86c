// tcgen05 / mbarrier helpers shared by the tensor-core kernels.
#pragma once

#include <cuda_runtime.h>

namespace bem2d_gpu {
namespace tc {

constexpr unsigned long long kWaitNs = 2000000000ull;  // 2 s

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mma_commit(unsigned long long* m) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(m)));
}
__device__ __forceinline__ void mbar_init(unsigned long long* m, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* m, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(m)),
               "r"(bytes));
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* m) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(m)) : "memory");
}
__device__ __forceinline__ bool mbar_test(unsigned long long* m, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(m)), "r"(parity)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait for phase `parity` of the mbarrier (try_wait suspends the
// thread for a short while between polls): false after kWaitNs of device
// time, or, if `abort` is given, as soon as another role has given up.
__device__ __forceinline__ bool mbar_wait(unsigned long long* m, unsigned parity,
                                          const volatile int* abort) {
  if (mbar_test(m, parity)) return true;
  const unsigned long long t0 = global_ns();
  for (unsigned it = 1;; ++it) {
    if (mbar_test(m, parity)) return true;
    if ((it & 15u) == 0u) {
      if (abort && *abort) return false;
      if (global_ns() - t0 > kWaitNs) return false;
    }
  }
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, unsigned bytes,
                                          unsigned long long* m) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(m))
      : "memory");
}

// ---- cluster exchange through asynchronous remote stores ----------------------
// Address of shared-memory variable p in the CTA of rank `rank`.
__device__ __forceinline__ unsigned map_rank(const void* p, unsigned rank) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
// 16 bytes to a mapped address; they count 16 on the mbarrier (same CTA).
__device__ __forceinline__ void store_async(unsigned dst, uint4 v, unsigned mbar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, "
      "[%5];" ::"r"(dst),
      "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(mbar)
      : "memory");
}
// 8 bytes, counted the same way.
__device__ __forceinline__ void store_async8(unsigned dst, float2 v, unsigned mbar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::
          "r"(dst),
      "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(mbar)
      : "memory");
}
// Bulk copy from this CTA's shared memory to a mapped address (multiples of 16
// bytes); the bytes count on the mbarrier (same CTA as the destination).
__device__ __forceinline__ void copy_to_rank(unsigned dst, const void* src, unsigned bytes,
                                             unsigned mbar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, "
      "[%3];" ::"r"(dst),
      "r"(smem_u32(src)), "r"(bytes), "r"(mbar)
      : "memory");
}
__device__ __forceinline__ bool mbar_test_cluster(unsigned long long* m, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n .reg .pred p;\n"
      " mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(smem_u32(m)), "r"(parity)
      : "memory");
  return done != 0;
}
// As mbar_wait, for data that other CTAs of the cluster have stored; a thread
// that gives up sets *abort, and nobody waits again after that.
__device__ __forceinline__ bool mbar_wait_cluster(unsigned long long* m, unsigned parity,
                                                  volatile int* abort) {
  if (mbar_test_cluster(m, parity)) return *abort == 0;
  const unsigned long long t0 = global_ns();
  for (unsigned it = 1;; ++it) {
    if (mbar_test_cluster(m, parity)) return *abort == 0;
    if ((it & 15u) == 0u) {
      if (*abort) return false;
      if (global_ns() - t0 > kWaitNs) {
        *abort = 1;
        return false;
      }
    }
  }
}

}  // namespace tc
}  // namespace bem2d_gpu
