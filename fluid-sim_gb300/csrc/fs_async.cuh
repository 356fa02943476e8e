// fs_async.cuh -- asynchronous global -> shared copies (cp.async).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fs {

// 4-byte asynchronous global -> shared copies (no register round trip, all of
// a thread's copies in flight at once); wait_all before the barrier that
// publishes them.
__device__ __forceinline__ void cp_async4(float* sdst, const float* gsrc) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(sdst)),
               "l"((size_t)__cvta_generic_to_global(gsrc))
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

}  // namespace fs
