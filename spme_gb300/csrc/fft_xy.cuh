// Two-factor x and y transforms of the mesh's z-planes, K = R1 R2 (K = 2^a 3^b 5^c
// up to 256): real planes [planes][K][K] <-> half spectra [planes][K][K/2+1], cuFFT's
// layouts and unnormalised conventions.
//
// Each transform is R1-point transforms over n1 (n = n2 + R2 n1), twiddles
// w_K^{n2 k1} (k1 signed in FP64, fft_dft.cuh), one exchange through shared memory and R2-point
// transforms over n2 (frequency k1 + R1 k2); the inverse of x runs the same steps backwards.  Global
// loads go straight to the first pass's registers and results leave from the last
// pass's, so a thread has R1 independent loads in flight.
// x: two consecutive real rows a, b of one component are one complex row a + i b; the
// spectra are Z[k] + conj Z[K-k] and -i (Z[k] - conj Z[K-k]) up to a factor 1/2, which the
// first pass's twiddles carry.  Rows of two components never share one: they may belong to
// right-hand sides or systems of other magnitude, whose rounding (or NaN) would pass over.
// With odd K the last row of a component (it has K^2) is paired with zeros.
// y: in place, W columns of the flattened (plane, kx) list per block, so no lane is
// idle at the end of a plane.
// Bound: FP64 by the FP64 pipe (a warp instruction each 16 cycles; about 14 instructions
// per real point along x, 24 per complex point along y at K = 256: 2.24 of the 2.48 ms);
// FP32 by HBM (four passes, 1.94 of the 2.08 ms at K = 256, 48 components).
// Forward x and y against cuFFT (FP64: its whole 3D transform): K = 256, R = 1 FP64
// 5.12 -> 2.48 ms for x and y (the z transform is in the fused kernel), K = 90, R = 4
// 1.05 -> .48; FP32 against its 2D transforms, R = 16: K = 256 2.44 -> 2.08, K = 160 .80 ->
// .59, K = 75 .173 -> .081.  Inverse alike.
#pragma once

#include "fft_dft.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace spme {
namespace {

// Row pairs per block of the x transforms.
constexpr int kXPairs = 16;
// Columns per block of the y transform: 16, or 8 in FP32 where the passes' thread counts
// (R1 and R2 per column) are so unlike that smaller blocks overlap better: K = 75 (15 x 5),
// R = 16, x and y forward .081 ms with 8 and .089 with 16; K = 160 (16 x 10) .609 and .593;
// 32 columns lose everywhere (K = 160 .699).
template <typename T>
__host__ __device__ constexpr int xy_cols(int R1, int R2) { return sizeof(T) == 4 && R1 > 2 * R2 ? 8 : 16; }
// Row stride (complex values) of the [k1][n2] exchange of the x transforms: odd, so that
// reads along k1 fall on different banks.
__host__ __device__ constexpr int x_stride(int R2) { return R2 | 1; }

// Row pairs of a component; the first row of pair q of all components' pairs (rows and
// above: past the last), and whether the pair has a second one.
__host__ __device__ constexpr int x_pairs(int K) { return (K * K + 1) / 2; }
template <int K>
__device__ __forceinline__ long x_row(long q) {
    return K % 2 == 0 ? 2 * q : 2 * q - q / x_pairs(K);
}
template <int K>
__device__ __forceinline__ bool x_two(long ra, long rows) {
    return K % 2 == 0 ? ra + 1 < rows : (ra + 1) % (K * K) != 0;
}

template <typename T>
__host__ __device__ constexpr int xy_minb(int threads, int R) {
    // registers: the transform's values and as many temporaries
    const int regs = (sizeof(T) == 8 ? 4 : 2) * R + (sizeof(T) == 8 ? 64 : 40);
    const int m = 65536 / (regs * ((threads + 31) / 32 * 32));
    return m < 1 ? 1 : m * ((threads + 31) / 32 * 32) > 2048 ? 2048 / ((threads + 31) / 32 * 32) : m;
}

__host__ __device__ constexpr int zmax(int a, int b) { return a > b ? a : b; }

template <typename T, int R1, int R2>
__global__ void __launch_bounds__(kXPairs * zmax(R1, R2), xy_minb<T>(kXPairs * zmax(R1, R2), zmax(R1, R2)))
k_fft_x_fwd(const T *__restrict__ mesh, typename ZVec<T>::type *__restrict__ G,
            const typename ZVec<T>::type *__restrict__ tw, long rows) {
    pdl_wait();
    using V = typename ZVec<T>::type;
    constexpr int K = R1 * R2, Kh = K / 2 + 1, P = kXPairs, RS = x_stride(R2);
    extern __shared__ __align__(16) unsigned char xsm[];
    V *sm = reinterpret_cast<V *>(xsm);
    const int tid = threadIdx.x;
    const long q0 = (long)blockIdx.x * P;
    {
        const int p = tid / R2, n2 = tid - p * R2;
        const long ra = x_row<K>(q0 + p);
        if (p < P && ra < rows) {
            const T *a = mesh + ra * K + n2;
            const bool two = x_two<K>(ra, rows);
            V v[R1];
#pragma unroll
            for (int n1 = 0; n1 < R1; n1++) v[n1] = z_make(a[n1 * R2], two ? a[K + n1 * R2] : T(0));
            z_dft<R1, false>(v);
            V *x = sm + p * (R1 * RS) + n2;
            x[0] = z_scale(T(0.5), v[0]);
#pragma unroll
            for (int k1 = 1; k1 < R1; k1++) {
                const int ks = z_signed<T>(k1, R1);
                const V t = tw[n2 * (ks < 0 ? -ks : ks)];
                x[k1 * RS] = z_tw(z_scale(T(0.5), v[k1]), t.x, ks < 0 ? -t.y : t.y);
            }
        }
    }
    __syncthreads();
    {
        // thread (p, k1) holds frequencies k = k1 + R1 k2; for k <= K/2 it needs Z[K-k]
        // of thread R1 - k1
        static_assert(R1 >= R2, "R1 threads per pair");
        // register k2 holds k = k1 + R1 z_k2(k2); those of k2 < H may be k <= K/2
        constexpr int H = (Kh + R1 - 1) / R1 + 1 < R2 ? (Kh + R1 - 1) / R1 + 1 : R2;
        const int p = tid / R1, k1 = tid - p * R1;
        const bool neg = z_signed<T>(k1, R1) < 0;
        const long ra = x_row<K>(q0 + p);
        V *x = sm + p * (R1 * RS);
        const V *xc = x + (k1 == 0 ? R2 : (R1 - k1) * RS + R2 - 1);  // frequency K - k1
        V v[R2];
        if (p < P) {
            x += k1 * RS;
#pragma unroll
            for (int n2 = 0; n2 < R2; n2++) v[n2] = x[n2];
            z_dft<R2, false>(v);
#pragma unroll
            for (int k2 = 0; k2 < R2; k2++) {
                const int q = z_k2(neg, k2, R2);
                if (2 * (k1 + R1 * q) > K) x[q] = v[k2];
            }
        }
        __syncthreads();
        if (p < P && ra < rows) {
            V *g = G + ra * Kh + k1;
            const bool two = x_two<K>(ra, rows);
#pragma unroll
            for (int k2 = 0; k2 < H; k2++) {
                const int q = z_k2(neg, k2, R2), k = k1 + R1 * q;
                if (k >= Kh) continue;
                const V z = v[k2], w = k == 0 || 2 * k == K ? z : xc[-q];
                g[R1 * q] = z_make(z.x + w.x, z.y - w.y);
                if (two) g[R1 * q + Kh] = z_make(z.y + w.y, w.x - z.x);
            }
        }
    }
}

template <typename T, int R1, int R2>
__global__ void __launch_bounds__(kXPairs * zmax(R1, R2), xy_minb<T>(kXPairs * zmax(R1, R2), zmax(R1, R2)))
k_fft_x_inv(const typename ZVec<T>::type *__restrict__ G, T *__restrict__ mesh,
            const typename ZVec<T>::type *__restrict__ tw, long rows) {
    pdl_wait();
    using V = typename ZVec<T>::type;
    constexpr int K = R1 * R2, Kh = K / 2 + 1, P = kXPairs, RS = x_stride(R2);
    extern __shared__ __align__(16) unsigned char xsm[];
    V *sm = reinterpret_cast<V *>(xsm);
    const int tid = threadIdx.x;
    const long q0 = (long)blockIdx.x * P;
    {
        // Z[k] = A[k] + i B[k], Z[K-k] = conj A[k] + i conj B[k]; the imaginary parts of the
        // zero and Nyquist frequencies are those of a real row, zero.  Thread (p, k1) loads
        // k = k1 + R1 k2 <= K/2, which its R2 transform needs itself, and leaves the
        // mirrored value for thread R1 - k1.
        static_assert(R1 >= R2, "R1 threads per pair");
        // register k2 holds k = k1 + R1 z_k2(k2); those of k2 < H may be k <= K/2
        constexpr int H = (Kh + R1 - 1) / R1 + 1 < R2 ? (Kh + R1 - 1) / R1 + 1 : R2;
        const int p = tid / R1, k1 = tid - p * R1;
        const bool neg = z_signed<T>(k1, R1) < 0;
        const long ra = x_row<K>(q0 + p);
        V *x = sm + p * (R1 * RS);
        V *xc = x + (k1 == 0 ? R2 : (R1 - k1) * RS + R2 - 1);  // frequency K - k1
        V v[R2];
        if (p < P && ra < rows) {
            const V *g = G + ra * Kh + k1;
            const bool two = x_two<K>(ra, rows);
            V a[H], c[H];
#pragma unroll
            for (int k2 = 0; k2 < H; k2++) {
                const int q = z_k2(neg, k2, R2);
                const bool in = k1 + R1 * q < Kh;
                a[k2] = in ? g[R1 * q] : z_make(T(0), T(0));
                c[k2] = in && two ? g[R1 * q + Kh] : z_make(T(0), T(0));
            }
#pragma unroll
            for (int k2 = 0; k2 < H; k2++) {
                const int q = z_k2(neg, k2, R2), k = k1 + R1 * q;
                if (k == 0 || 2 * k == K) a[k2].y = c[k2].y = T(0);
                v[k2] = z_make(a[k2].x - c[k2].y, a[k2].y + c[k2].x);
                if (k > 0 && k < Kh && 2 * k != K)
                    xc[-q] = z_make(a[k2].x + c[k2].y, c[k2].x - a[k2].y);
            }
        }
        __syncthreads();
        if (p < P) {
            x += k1 * RS;
#pragma unroll
            for (int k2 = 0; k2 < R2; k2++) {
                const int q = z_k2(neg, k2, R2);
                if (k2 >= H || k1 + R1 * q >= Kh) v[k2] = x[q];
            }
            z_dft<R2, true>(v);
            x[0] = v[0];
            const int ks = neg ? R1 - k1 : k1;  // |signed k1|
#pragma unroll
            for (int n2 = 1; n2 < R2; n2++) {
                const V t = tw[n2 * ks];
                x[n2] = z_tw(v[n2], t.x, neg ? t.y : -t.y);
            }
        }
    }
    __syncthreads();
    {
        const int p = tid / R2, n2 = tid - p * R2;
        const long ra = x_row<K>(q0 + p);
        if (p < P && ra < rows) {
            const V *x = sm + p * (R1 * RS) + n2;
            V v[R1];
#pragma unroll
            for (int k1 = 0; k1 < R1; k1++) v[k1] = x[k1 * RS];
            z_dft<R1, true>(v);
            T *a = mesh + ra * K + n2;
#pragma unroll
            for (int n1 = 0; n1 < R1; n1++) a[n1 * R2] = v[n1].x;
            if (x_two<K>(ra, rows)) {
#pragma unroll
                for (int n1 = 0; n1 < R1; n1++) a[K + n1 * R2] = v[n1].y;
            }
        }
    }
}

// Both directions: the inverse transform is the forward one of the values with real and
// imaginary parts exchanged, exchanged back.
template <typename T, int R1, int R2>
__global__ void __launch_bounds__(xy_cols<T>(R1, R2) * zmax(R1, R2), xy_minb<T>(xy_cols<T>(R1, R2) * zmax(R1, R2), zmax(R1, R2)))
k_fft_y(typename ZVec<T>::type *__restrict__ G, const typename ZVec<T>::type *__restrict__ tw, long cols,
        int inv) {
    pdl_wait();
    using V = typename ZVec<T>::type;
    constexpr int K = R1 * R2, Kh = K / 2 + 1, W = xy_cols<T>(R1, R2);
    extern __shared__ __align__(16) unsigned char xsm[];
    const int w = threadIdx.x % W, id = threadIdx.x / W;
    const long q = (long)blockIdx.x * W + w;
    const bool live = q < cols;
    const long pl = live ? q / Kh : 0;
    V *g = G + pl * ((long)K * Kh) + (live ? q - pl * Kh : 0);
    V *sm = reinterpret_cast<V *>(xsm) + w;
    if (id < R2 && live) {
        V v[R1];
#pragma unroll
        for (int n1 = 0; n1 < R1; n1++) v[n1] = g[(long)(id + n1 * R2) * Kh];
        if (inv) {
#pragma unroll
            for (int n1 = 0; n1 < R1; n1++) v[n1] = z_make(v[n1].y, v[n1].x);
        }
        z_dft<R1, false>(v);
        sm[id * W] = v[0];
#pragma unroll
        for (int k1 = 1; k1 < R1; k1++) {
            const int ks = z_signed<T>(k1, R1);
            const V t = tw[id * (ks < 0 ? -ks : ks)];
            sm[(k1 * R2 + id) * W] = z_tw(v[k1], t.x, ks < 0 ? -t.y : t.y);
        }
    }
    __syncthreads();
    if (id < R1 && live) {
        V v[R2];
#pragma unroll
        for (int n2 = 0; n2 < R2; n2++) v[n2] = sm[(id * R2 + n2) * W];
        z_dft<R2, false>(v);
        if (inv) {
#pragma unroll
            for (int k2 = 0; k2 < R2; k2++) v[k2] = z_make(v[k2].y, v[k2].x);
        }
#pragma unroll
        for (int k2 = 0; k2 < R2; k2++)
            g[(long)(id + R1 * z_k2(z_signed<T>(id, R1) < 0, k2, R2)) * Kh] = v[k2];
    }
}

template <typename T, int R1, int R2>
cudaError_t launch_xy(bool inv, T *mesh, T *G, long comps, const T *tw, cudaStream_t s) {
    using V = typename ZVec<T>::type;
    constexpr int K = R1 * R2, Kh = K / 2 + 1, P = kXPairs, W = xy_cols<T>(R1, R2), M = zmax(R1, R2);
    constexpr int xsmem = P * R1 * x_stride(R2) * (int)sizeof(V), ysmem = K * W * (int)sizeof(V);
    const long rows = comps * K * K, cols = comps * K * Kh;
    const unsigned xb = (unsigned)((comps * x_pairs(K) + P - 1) / P), yb = (unsigned)((cols + W - 1) / W);
    V *g = reinterpret_cast<V *>(G);
    const V *t = reinterpret_cast<const V *>(tw);
    auto kx = inv ? reinterpret_cast<const void *>(k_fft_x_inv<T, R1, R2>)
                  : reinterpret_cast<const void *>(k_fft_x_fwd<T, R1, R2>);
    cudaError_t e = cudaSuccess;
    if (xsmem > 48 * 1024) e = cudaFuncSetAttribute(kx, cudaFuncAttributeMaxDynamicSharedMemorySize, xsmem);
    if (e == cudaSuccess && ysmem > 48 * 1024)
        e = cudaFuncSetAttribute(k_fft_y<T, R1, R2>, cudaFuncAttributeMaxDynamicSharedMemorySize, ysmem);
    if (e != cudaSuccess) return e;
    if (inv) {
        pdl_launch(k_fft_y<T, R1, R2>, yb, W * M, ysmem, s, g, t, cols, 1);
        pdl_launch(k_fft_x_inv<T, R1, R2>, xb, P * M, xsmem, s, g, mesh, t, rows);
    } else {
        pdl_launch(k_fft_x_fwd<T, R1, R2>, xb, P * M, xsmem, s, mesh, g, t, rows);
        pdl_launch(k_fft_y<T, R1, R2>, yb, W * M, ysmem, s, g, t, cols, 0);
    }
    return cudaGetLastError();
}

}  // namespace
}  // namespace spme
