// Helpers shared by the column-gather spreads (spread_cols.cu, spread_march.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "cp_async.cuh"

namespace spme {

// fn(std::integral_constant<int, i>) for i = 0 .. N-1, unrolled at compile time.
template <typename Fn, int... Is>
__device__ __forceinline__ void static_for_impl(Fn &&fn, std::integer_sequence<int, Is...>) {
    (fn(std::integral_constant<int, Is>{}), ...);
}
template <int N, typename Fn>
__device__ __forceinline__ void static_for(Fn &&fn) {
    static_for_impl(fn, std::make_integer_sequence<int, N>{});
}

// Components per lane for C components (chunks of 16 CPL components per block).
__host__ __device__ constexpr int cols_cpl(int C) { return C <= 16 ? 1 : (C <= 32 ? 2 : 3); }
// Padded components per lane in the gathered force rows.
__host__ __device__ constexpr int cols_pcpl(int cpl) { return cpl == 3 ? 4 : cpl; }

// n values from a 16-byte aligned address, global or shared (vector loads where
// they fit).
template <int NV>
__device__ __forceinline__ void load_vec(const float *__restrict__ src, float (&w)[NV]) {
    constexpr int NQ = NV / 4;
#pragma unroll
    for (int v = 0; v < NQ; v++) {
        const float4 q = reinterpret_cast<const float4 *>(src)[v];
        w[4 * v] = q.x;
        w[4 * v + 1] = q.y;
        w[4 * v + 2] = q.z;
        w[4 * v + 3] = q.w;
    }
#pragma unroll
    for (int j = NQ * 4; j < NV; j++) w[j] = src[j];
}
template <int NV>
__device__ __forceinline__ void load_vec(const double *__restrict__ src, double (&w)[NV]) {
    constexpr int NQ = NV / 2;
#pragma unroll
    for (int v = 0; v < NQ; v++) {
        const double2 q = reinterpret_cast<const double2 *>(src)[v];
        w[2 * v] = q.x;
        w[2 * v + 1] = q.y;
    }
#pragma unroll
    for (int j = NQ * 2; j < NV; j++) w[j] = src[j];
}

}  // namespace spme
