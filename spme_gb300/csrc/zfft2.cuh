// Fused z-transform + k-space influence + inverse z-transform for K = R1 R2 (FP32):
// the operation of zfft.cu with compile-time radices and the influence inside the
// second pass.
//
// Forward, per column and component: R1-point transforms over n1 (z = n2 + R2 n1),
// twiddles w_K^{n2 k1}, then R2-point transforms over n2 give the frequencies
// kz = k1 + R1 k2; the inverse runs the same steps backwards.  A thread of the
// second pass holds the R2 frequencies of its k1 for all three components, so
// the influence is applied in registers and the inverse R2-point transforms
// follow at once: three passes over shared memory per right-hand side (forward
// R1, second pass, inverse R1) with two barriers between them, instead of a pass
// per radix pair and direction plus one for the influence (five at K = 256), and no
// digit reversal.  The R1 passes give each component its own threads (3 R2 of them per
// column), so with R1 near 3 R2 both kinds of pass keep the block's threads busy.
// Complex sums are two-lane additions.
// Data movement as in zfft.cu: chunks of W columns of the flattened z-plane
// (TMA boxes, loads and stores), two buffers per block, a dedicated TMA warp.
// Right-hand sides are split over blockIdx.y where the chunks alone would leave
// SMs idle.
// Bound: HBM (one read and one write of the half spectrum, 0.98 ms at K = 256, R =
// 16), then shared-memory traffic and latency at one or two blocks per SM.
// Influence stage, radix passes of zfft.cu -> here: K = 256, R = 16 1.80 -> 1.20 ms;
// K = 160, R = 16 .780 -> .350; K = 128, R = 1 .037 -> .021; K = 75, R = 8 .154 -> .025.
// Sixteen- by ten-point factors (K = 160: one thread per column and index for all three
// components) need 168 registers a thread; 20 x 8 needs 126.
#pragma once

#include "fft_dft.cuh"
#include "kernels.h"
#include "tma.cuh"
#include "pdl.cuh"

namespace spme {
namespace {

// Shared-memory layout (bytes from the 128-aligned base): two buffers of three
// K x W component blocks, the twiddles e^{-2 pi i e / K}, barriers full[b] (TMA
// load of buffer b landed) and done[b] (the compute warps finished buffer b).
struct ZSmem2 {
    size_t comp, buf_bytes, tw_off, bar_off, total;
    __host__ __device__ constexpr ZSmem2(int K, int W)
        : comp(((size_t)K * W * sizeof(float2) + 127) & ~(size_t)127),  // TMA: 128-aligned
          buf_bytes(3 * comp),
          tw_off(2 * buf_bytes),
          bar_off(tw_off + (((size_t)K * sizeof(float2) + 15) & ~(size_t)15)),
          total(bar_off + 4 * sizeof(uint64_t)) {}
};

__host__ __device__ constexpr int z2_threads(int W, int R1, int R2) {
    return (W * (R1 > 3 * R2 ? R1 : 3 * R2) + 31) / 32 * 32;
}
// Blocks per SM: what shared memory allows at the registers the passes want.
__host__ __device__ constexpr int z2_minb(int W, int R1, int R2) {
    const int regs = 8 * R2 + 32 > 2 * R1 + 32 ? 8 * R2 + 32 : 2 * R1 + 32;
    const int bs = (int)(224 * 1024 / (ZSmem2(R1 * R2, W).total + 1152));
    const int br = 65536 / (regs * ((z2_threads(W, R1, R2) + 32 + 127) / 128 * 128));
    const int m = bs < br ? bs : br;
    return m < 1 ? 1 : m > 8 ? 8 : m;
}

// Whether the influence table is read for every right-hand side instead of held: where the
// radices leave no registers for it.  At K = 256 a block's shared memory leaves too little L1
// for the spills.  Stage in ms, held / read again, R = 16: K = 256 1.66 / 1.20, K = 250 (25 x 10)
// 1.87 / 1.37, K = 240 1.14 / 1.06, K = 150 .341 / .313; K = 216 (24 x 9) .793 / .834, K = 160
// .342 / .366, K = 75 .041 / .043.
__host__ __device__ constexpr bool z2_reload(int W, int R1, int R2) {
    const int regs = 65536 / (z2_minb(W, R1, R2) * ((z2_threads(W, R1, R2) + 32 + 127) / 128 * 128));
    return R1 >= 24 && (R2 >= 10 || regs <= 104);
}

template <int N>
__device__ __forceinline__ void z2_sync() {
    asm volatile("bar.sync 1, %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ bool z2_sync_and(bool p) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred q, o;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "bar.red.and.pred o, 1, %2, q;\n\t"
        "selp.u32 %0, 1, 0, o;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)p), "n"(N)
        : "memory");
    return r != 0;
}

// One block per chunk of W consecutive columns, range of right-hand sides
// [blockIdx.y rs, +rs) and system blockIdx.z (batches: R right-hand sides and one table
// each, box sizes through twopi_Ls).  Threads 0 .. CT-1 transform (thread = column + W index),
// the warp after them moves data.
template <int W, int R1, int R2>
__global__ void __launch_bounds__(z2_threads(W, R1, R2) + 32, z2_minb(W, R1, R2))
k_zfft2(const __grid_constant__ CUtensorMap gmap, const float2 *__restrict__ tab2,
        const float2 *__restrict__ tw_g, float twopi_L, const double *__restrict__ twopi_Ls, int R,
        int rs, int *__restrict__ err) {
    pdl_wait();
    constexpr int K = R1 * R2, Kh = K / 2 + 1, CT = z2_threads(W, R1, R2);
    const int plane = K * Kh;
    const int f0 = blockIdx.x * W, tid = threadIdx.x;
    const int rb = blockIdx.y * rs, nr = min(rs, R - rb);
    const int c0 = 3 * (blockIdx.z * R + rb);  // first component
    if (twopi_Ls) twopi_L = (float)twopi_Ls[blockIdx.z];
    tab2 += (size_t)blockIdx.z * K * plane;
    extern __shared__ __align__(128) unsigned char zsm_raw[];
    unsigned char *zsm = zsm_raw + ((128u - (smem_addr(zsm_raw) & 127u)) & 127u);
    constexpr ZSmem2 lay(K, W);
    constexpr int GS = (int)(lay.comp / sizeof(float2));  // component stride (complex values)
    float2 *const buf0 = reinterpret_cast<float2 *>(zsm);
    float2 *const buf1 = reinterpret_cast<float2 *>(zsm + lay.buf_bytes);
    float2 *tw = reinterpret_cast<float2 *>(zsm + lay.tw_off);
    uint64_t *full = reinterpret_cast<uint64_t *>(zsm + lay.bar_off);
    uint64_t *done = full + 2;

    if (tid == 0) {
        mbar_init(&full[0], 1);
        mbar_init(&full[1], 1);
        mbar_init(&done[0], CT);
        mbar_init(&done[1], CT);
        mbar_fence_init();
    }
    for (int e = tid; e < K; e += CT + 32) tw[e] = tw_g[e];
    __syncthreads();

    if (tid >= CT) {
        // ---- TMA warp (one lane) ----
        if (tid != CT) return;
        const uint32_t bytes = (uint32_t)(3 * K * W * sizeof(float2));
        auto issue_load = [&](int r, int b) {
            mbar_expect_tx(&full[b], bytes);
            float2 *dst = b ? buf1 : buf0;
            for (int d = 0; d < 3; d++)
                tma_load_3d(dst + d * GS, &gmap, 2 * f0, 0, c0 + 3 * r + d, &full[b]);
        };
        issue_load(0, 0);
        int issued = 1;
        if (nr > 1) issue_load(1, 1), issued = 2;
        int r = 0;
        for (; r < nr; r++) {
            const int b = r & 1;
            if (!mbar_wait(&done[b], (uint32_t)((r >> 1) & 1))) break;
            const float2 *src = b ? buf1 : buf0;
            for (int d = 0; d < 3; d++)
                tma_store_3d(&gmap, 2 * f0, 0, c0 + 3 * r + d, src + d * GS);
            bulk_commit_group();
            if (r + 2 < nr) {
                bulk_wait_read_all();  // buffer b is free again
                issue_load(r + 2, b);
                issued++;
            }
        }
        if (r < nr) {
            atomicExch(err, 1);
            // loads of right-hand sides r .. issued-1 may still be in flight
            for (int q = r; q < issued; q++) mbar_wait(&full[q & 1], (uint32_t)((q >> 1) & 1));
        }
        bulk_wait_all();
        return;
    }

    // ---- compute warps ----
    // column; in the R1 passes component d1 and n2, in the second k1 = id
    const int w = tid % W, id = tid / W, d1 = id / R2, n2 = id - d1 * R2;
    const int fl = f0 + w;
    const bool valid = fl < plane;
    const int ky = valid ? fl / Kh : 0, kx = valid ? fl - ky * Kh : 0;
    const float kxv = (float)kx * twopi_L;  // kx <= K/2: non-negative wavenumber
    const float kyv = (float)(ky <= K / 2 ? ky : ky - K) * twopi_L;
    // kx = 0 and (even K) K/2 planes hold k and -k: there the tensor is averaged with
    // its mirror (the Hermitian part of the result): with s_i = +1 for a zero or
    // Nyquist index and -1 otherwise, the ij coupling survives when s_i s_j = +1
    // (s_x = +1 on these planes)
    const bool xplane = valid && (kx == 0 || (K % 2 == 0 && kx == K / 2));
    const bool sy = ky == 0 || (K % 2 == 0 && ky == K / 2);
    // the influence table of this thread's frequencies: read once for all its right-hand
    // sides, or (RELOAD) for each between the passes
    constexpr bool RELOAD = z2_reload(W, R1, R2);
    float2 mc[R2];
    auto load_mc = [&]() {
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++)
            mc[k2] = id < R1 && valid ? __ldg(tab2 + (size_t)(id + R1 * k2) * plane + fl)
                                      : make_float2(0.f, 0.f);
    };
    if constexpr (!RELOAD) load_mc();

    for (int r = 0; r < nr; r++) {
        const int b = r & 1;
        const bool ok = mbar_wait(&full[b], (uint32_t)((r >> 1) & 1));
        if (!z2_sync_and<CT>(ok)) {
            if (tid == 0) atomicExch(err, 1);
            break;
        }
        float2 *B = (b ? buf1 : buf0) + w;
        float2 *x1 = B + d1 * GS + n2 * W;
        // forward R1-point transforms over n1, in place (k1 where n1 was)
        if (id < 3 * R2) {
            float2 v[R1];
#pragma unroll
            for (int n1 = 0; n1 < R1; n1++) v[n1] = x1[n1 * R2 * W];
            z_dft<R1, false>(v);
            x1[0] = v[0];
#pragma unroll
            for (int k1 = 1; k1 < R1; k1++) {
                const float2 t = tw[n2 * k1];
                x1[k1 * R2 * W] = z_tw(v[k1], t.x, t.y);
            }
        }
        if constexpr (RELOAD) load_mc();
        z2_sync<CT>();
        // second pass: R2-point transforms, influence, inverse R2-point transforms
        if (id < R1) {
            float2 *x = B + id * R2 * W;
            float2 v[3][R2];
#pragma unroll
            for (int d = 0; d < 3; d++) {
#pragma unroll
                for (int q = 0; q < R2; q++) v[d][q] = x[d * GS + q * W];
                z_dft<R2, false>(v[d]);
            }
#pragma unroll
            for (int k2 = 0; k2 < R2; k2++) {
                const int kz = id + R1 * k2;
                const float kzv = (float)(kz <= K / 2 ? kz : kz - K) * twopi_L;
                const float m2 = mc[k2].x, c = mc[k2].y;
                const float cx = c * kxv, cy = c * kyv, cz = c * kzv;
                float b1 = -cx * kyv, b2 = -cx * kzv, b4 = -cy * kzv;
                if (xplane) {
                    const bool sz = kz == 0 || (K % 2 == 0 && kz == K / 2);
                    if (!sy) b1 = 0.f;
                    if (!sz) b2 = 0.f;
                    if (sy != sz) b4 = 0.f;
                }
                const float b0 = m2 - cx * kxv, b3 = m2 - cy * kyv, b5 = m2 - cz * kzv;
                const float2 g0 = v[0][k2], g1 = v[1][k2], g2 = v[2][k2];
                const float2 B1 = make_float2(b1, b1), B2 = make_float2(b2, b2), B4 = make_float2(b4, b4);
                v[0][k2] = __ffma2_rn(B2, g2, __ffma2_rn(B1, g1, __fmul2_rn(make_float2(b0, b0), g0)));
                v[1][k2] = __ffma2_rn(B4, g2, __ffma2_rn(make_float2(b3, b3), g1, __fmul2_rn(B1, g0)));
                v[2][k2] = __ffma2_rn(make_float2(b5, b5), g2, __ffma2_rn(B4, g1, __fmul2_rn(B2, g0)));
            }
#pragma unroll
            for (int d = 0; d < 3; d++) {
                z_dft<R2, true>(v[d]);
                x[d * GS] = v[d][0];
#pragma unroll
                for (int q = 1; q < R2; q++) {
                    const float2 t = tw[id * q];
                    x[d * GS + q * W] = z_tw(v[d][q], t.x, -t.y);
                }
            }
        }
        z2_sync<CT>();
        // inverse R1-point transforms over k1
        if (id < 3 * R2) {
            float2 v[R1];
#pragma unroll
            for (int k1 = 0; k1 < R1; k1++) v[k1] = x1[k1 * R2 * W];
            z_dft<R1, true>(v);
#pragma unroll
            for (int n1 = 0; n1 < R1; n1++) x1[n1 * R2 * W] = v[n1];
        }
        // hand the buffer to the TMA warp (its store reads what this thread wrote)
        fence_proxy_async();
        mbar_arrive(&done[b]);
    }
}

template <int W, int R1, int R2>
cudaError_t launch_z2(const CUtensorMap &map, const float *tab2, const float *tw, double L,
                      const double *twopi_Ls, int nsys, int R, int *err, cudaStream_t s) {
    constexpr int K = R1 * R2;
    constexpr size_t smem = ZSmem2(K, W).total + 128;
    auto kern = k_zfft2<W, R1, R2>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int nchunk = (K * (K / 2 + 1) + W - 1) / W;
    const long blocks = (long)nchunk * nsys;
    // right-hand sides per block: all of them, or fewer (at least two, for the second
    // buffer) until the resident blocks are filled about four times
    int rs = R;
    while (rs > 2 && blocks * ((R + rs - 1) / rs) < 608L * z2_minb(W, R1, R2)) rs = (rs + 1) / 2;
    pdl_launch(kern, dim3(nchunk, (R + rs - 1) / rs, nsys), z2_threads(W, R1, R2) + 32, smem, s, 
        map, reinterpret_cast<const float2 *>(tab2), reinterpret_cast<const float2 *>(tw),
        (float)(2.0 * M_PI / L), twopi_Ls, R, rs, err);
    return cudaGetLastError();
}

}  // namespace
}  // namespace spme
