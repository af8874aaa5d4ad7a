// Asynchronous copies into shared memory and the barriers they complete on (sm_100a).
#pragma once

#include <cstdint>
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

// cuTensorMapEncodeTiled of the loaded driver (NULL: not available)
PFN_cuTensorMapEncodeTiled_v12000 hm_tensor_map_encoder();

namespace hm {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long* b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// a bounded wait: false if the copy has not landed after ~2^20 polls
__device__ __forceinline__ bool mbar_wait(unsigned long long* b, uint32_t parity) {
  for (int i = 0; i < (1 << 20); ++i)
    if (mbar_try_wait(b, parity)) return true;
  return false;
}

// an arrival that also announces the bytes of the copies that complete on b
__device__ __forceinline__ void mbar_expect(unsigned long long* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes)
               : "memory");
}

// single elements where `on` (a predicate, not a branch around the copy), in groups that are
// waited for in order
template <typename T>
__device__ __forceinline__ void copy_async(void* dst, const T* src, bool on) {
  asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %3, 0;\n @p cp.async.ca.shared.global [%0], [%1], %2;\n}" ::"r"(
                   smem_u32(dst)),
               "l"(src), "n"(sizeof(T)), "r"((uint32_t)on)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all but the newest N groups of this thread have landed
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

}  // namespace hm
