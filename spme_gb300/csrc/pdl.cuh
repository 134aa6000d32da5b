// Dependent launches: a kernel launched with pdl_launch may be set up while the stream's
// kernel before it drains, and waits for that kernel's end (and, through its own wait, for
// all earlier ones) in pdl_wait, the first statement of every such kernel.
// Kernels launched the ordinary way may stand anywhere between them.
// Time per call, ordinary launches -> these: drop-in N = 2000 285 -> 252 us, N = 20011,
// R = 8 343 -> 321 us, N = 300 in a graph 106 -> 101 us, N = 2e5, R = 16 3.28 -> 3.24 ms.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace spme {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t pdl_launch(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...a) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &attr;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kern, std::forward<A>(a)...);
}

}  // namespace spme
