// Asynchronous copies of 16 bytes from global to shared memory, in groups (cp.async).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

// Four floats; both addresses on 16 bytes.  Not inside: the destination is filled with zeros and nothing is read.
__device__ __forceinline__ void cp16(float* dst, const float* src, bool inside) {
    const int n = inside ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(n)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// All but the newest N groups of this thread's copies have landed.
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

static inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }
