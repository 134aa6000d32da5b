// Asynchronous global -> shared copies.
#pragma once

#include <cstdint>

namespace spme {
namespace {

// Asynchronous global -> shared copies (cp.async, completion tracked per thread).
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src)
                 : "memory");
}
template <int B>
__device__ __forceinline__ void cp_async_small(void *dst, const void *src) {
    static_assert(B == 4 || B == 8, "4 or 8 bytes");
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(dst)), "l"(src),
                 "n"(B)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// A mesh index past the periodic boundary (a halo can be wider than the mesh).
__device__ __forceinline__ int wrap_index(int i, int K) {
    while (i >= K) i -= K;
    return i;
}

}  // namespace
}  // namespace spme
