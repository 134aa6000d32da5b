// Fused z transform + k-space influence + inverse z transform in FP64, K = R1 R2 (2^a
// 3^b 5^c up to 256): the operation of zfft.cu on the half spectrum G[c][z][y][K/2+1].
//
// A block transforms W columns of the flattened (y, kx) plane for the three components
// of one right-hand side: R1-point transforms straight from global loads, an exchange
// through shared memory, R2-point transforms in place (frequency k1 + R1 k2 at k1 R2 +
// k2), the influence, and the same steps backwards.  The influence is m g - c k (k g)
// (20 operations for three components instead of 27 with the tensor's entries), except
// on the kx = 0 and K/2 planes, where couplings of the averaged tensor vanish.
// Bound: the FP64 pipe (a warp instruction each 16 cycles): the kernel spends shared
// memory and loads freely and keeps FP64 instructions few and lanes full.
// Stage (with the z transforms of both directions, which cuFFT's 3D transforms did): K =
// 256, R = 1 2.69 ms, 93 % of the FP64 pipe for its 58 instructions per point and component;
// K = 128 .338; K = 90, R = 4 .539.
#pragma once

#include "fft_dft.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace spme {
namespace {

// Columns per block: 8 (the blocks' last warps are fuller), or 4 where 8 leave SMs without
// a block (K <= 48, a plane has at most 150 chunks of 8: N = 300, K = 32 18.4 us with 8, 16.4
// with 4) or leave fewer than three blocks per SM (K > 128).
__host__ __device__ constexpr int z64_cols(int K) { return K <= 48 || K > 128 ? 4 : 8; }
__host__ __device__ constexpr int z64_threads(int R1, int R2) {
    return (3 * z64_cols(R1 * R2) * (R1 > R2 ? R1 : R2) + 31) / 32 * 32;
}
__host__ __device__ constexpr int z64_minb(int R1, int R2) {
    const int R = R1 > R2 ? R1 : R2, m = 65536 / ((4 * R + 64) * z64_threads(R1, R2));
    return m < 1 ? 1 : m > 8 ? 8 : m;
}

template <int R1, int R2>
__global__ void __launch_bounds__(z64_threads(R1, R2), z64_minb(R1, R2))
k_z64(double2 *__restrict__ G, const double2 *__restrict__ tab2, const double2 *__restrict__ tw,
      double twopi_L, const double *__restrict__ twopi_Ls, int R) {
    pdl_wait();
    constexpr int K = R1 * R2, Kh = K / 2 + 1, W = z64_cols(K), NT = z64_threads(R1, R2);
    constexpr int plane = K * Kh;
    extern __shared__ __align__(16) unsigned char zsm[];
    double2 *sm = reinterpret_cast<double2 *>(zsm);  // [3][K][W]
    const int tid = threadIdx.x, w = tid % W, id = tid / W;
    const int fl = blockIdx.x * W + w;
    const bool valid = fl < plane;
    if (twopi_Ls) {  // batch: blockIdx.y = system and right-hand side
        const int sys = blockIdx.y / R;
        twopi_L = twopi_Ls[sys];
        tab2 += (size_t)sys * K * plane;
    }
    {
        const int d = id / R2, n2 = id - d * R2;
        if (d < 3 && valid) {
            const double2 *g = G + ((size_t)(3 * blockIdx.y + d) * K + n2) * plane + fl;
            double2 v[R1];
#pragma unroll
            for (int n1 = 0; n1 < R1; n1++) v[n1] = g[(size_t)n1 * R2 * plane];
            z_dft<R1, false>(v);
            double2 *x = sm + (d * K + n2) * W + w;
            x[0] = v[0];
#pragma unroll
            for (int k1 = 1; k1 < R1; k1++) {
                const int ks = z_signed<double>(k1, R1);
                const double2 t = __ldg(tw + n2 * (ks < 0 ? -ks : ks));
                x[k1 * R2 * W] = z_tw(v[k1], t.x, ks < 0 ? -t.y : t.y);
            }
        }
    }
    __syncthreads();
    const int d2 = id / R1, k1 = id - d2 * R1;
    double2 *x2 = sm + (d2 * K + k1 * R2) * W + w;
    if (d2 < 3 && valid) {
        double2 v[R2];
#pragma unroll
        for (int n2 = 0; n2 < R2; n2++) v[n2] = x2[n2 * W];
        z_dft<R2, false>(v);
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) x2[k2 * W] = v[k2];
    }
    __syncthreads();
    if (valid) {
        const int ky = fl / Kh, kx = fl - ky * Kh;
        const double kxv = (double)kx * twopi_L;
        const double kyv = (double)(ky <= K / 2 ? ky : ky - K) * twopi_L;
        const bool xplane = kx == 0 || 2 * kx == K, sy = ky == 0 || 2 * ky == K;
        for (int i = id; i < K; i += NT / W) {
            const int r = i / R2, kz = r + R1 * z_k2(z_signed<double>(r, R1) < 0, i % R2, R2);
            const double kzv = (double)(kz <= K / 2 ? kz : kz - K) * twopi_L;
            const double2 mc = __ldg(tab2 + (size_t)kz * plane + fl);
            double2 *q = sm + i * W + w;
            const double2 g0 = q[0], g1 = q[K * W], g2 = q[2 * K * W];
            if (xplane) {
                // the ij coupling survives where both axes or neither hold a zero or
                // Nyquist index (x does)
                const bool sz = kz == 0 || 2 * kz == K;
                const double cx = mc.y * kxv, cy = mc.y * kyv, cz = mc.y * kzv;
                const double b1 = sy ? -cx * kyv : 0.0, b2 = sz ? -cx * kzv : 0.0;
                const double b4 = sy == sz ? -cy * kzv : 0.0;
                const double b0 = mc.x - cx * kxv, b3 = mc.x - cy * kyv, b5 = mc.x - cz * kzv;
                q[0] = z_fma(b2, g2, z_fma(b1, g1, z_scale(b0, g0)));
                q[K * W] = z_fma(b4, g2, z_fma(b3, g1, z_scale(b1, g0)));
                q[2 * K * W] = z_fma(b5, g2, z_fma(b4, g1, z_scale(b2, g0)));
            } else {
                const double2 s = z_scale(-mc.y, z_fma(kzv, g2, z_fma(kyv, g1, z_scale(kxv, g0))));
                q[0] = z_fma(kxv, s, z_scale(mc.x, g0));
                q[K * W] = z_fma(kyv, s, z_scale(mc.x, g1));
                q[2 * K * W] = z_fma(kzv, s, z_scale(mc.x, g2));
            }
        }
    }
    __syncthreads();
    if (d2 < 3 && valid) {
        double2 v[R2];
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++) v[k2] = x2[k2 * W];
        z_dft<R2, true>(v);
        x2[0] = v[0];
        const bool neg = z_signed<double>(k1, R1) < 0;
        const int ks = neg ? R1 - k1 : k1;  // |signed k1|
#pragma unroll
        for (int n2 = 1; n2 < R2; n2++) {
            const double2 t = __ldg(tw + n2 * ks);
            x2[n2 * W] = z_tw(v[n2], t.x, neg ? t.y : -t.y);
        }
    }
    __syncthreads();
    {
        const int d = id / R2, n2 = id - d * R2;
        if (d < 3 && valid) {
            const double2 *x = sm + (d * K + n2) * W + w;
            double2 v[R1];
#pragma unroll
            for (int q = 0; q < R1; q++) v[q] = x[q * R2 * W];
            z_dft<R1, true>(v);
            double2 *g = G + ((size_t)(3 * blockIdx.y + d) * K + n2) * plane + fl;
#pragma unroll
            for (int n1 = 0; n1 < R1; n1++) g[(size_t)n1 * R2 * plane] = v[n1];
        }
    }
}

template <int R1, int R2>
cudaError_t launch_z64_k(double *G, const double *tab2, const double *tw, double L,
                         const double *twopi_Ls, int nsys, int R, cudaStream_t s) {
    constexpr int K = R1 * R2, W = z64_cols(K), smem = 3 * K * W * (int)sizeof(double2);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k_z64<R1, R2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return e;
    }
    const unsigned nb = (K * (K / 2 + 1) + W - 1) / W;
    pdl_launch(k_z64<R1, R2>, dim3(nb, R * nsys), z64_threads(R1, R2), smem, s, 
        reinterpret_cast<double2 *>(G), reinterpret_cast<const double2 *>(tab2),
        reinterpret_cast<const double2 *>(tw), 2.0 * M_PI / L, twopi_Ls, R);
    return cudaGetLastError();
}

}  // namespace
}  // namespace spme
