// Asynchronous copies from global to shared memory (cp.async; dst: a shared
// address): no registers are held while the data is in flight.  With ok = false nothing is read and
// the destination is filled with zeros (src must still be a valid address).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fgb {

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src),
               "r"(ok ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src),
               "r"(ok ? 8 : 0)
               : "memory");
}
// Waits for every copy this thread has issued.
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

}  // namespace fgb
