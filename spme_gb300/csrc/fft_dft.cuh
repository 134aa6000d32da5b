// Small complex DFTs in registers with compile-time twiddles, shared by the
// two-factor transforms (zfft2.cuh, fft_xy.cuh, zfft64.cu).  V is float2 (complex
// sums as two-lane operations) or double2.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace spme {
namespace {

template <typename T>
struct ZVec;
template <>
struct ZVec<float> {
    using type = float2;
};
template <>
struct ZVec<double> {
    using type = double2;
};

__device__ __forceinline__ float2 z_make(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ double2 z_make(double x, double y) { return make_double2(x, y); }
__device__ __forceinline__ float2 z_add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ double2 z_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 z_sub(float2 a, float2 b) {
    return __ffma2_rn(make_float2(-1.f, -1.f), b, a);
}
__device__ __forceinline__ double2 z_sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// a + c b and c b for a real c
__device__ __forceinline__ float2 z_fma(float c, float2 b, float2 a) {
    return __ffma2_rn(make_float2(c, c), b, a);
}
__device__ __forceinline__ double2 z_fma(double c, double2 b, double2 a) {
    return make_double2(fma(c, b.x, a.x), fma(c, b.y, a.y));
}
__device__ __forceinline__ float2 z_scale(float c, float2 b) { return __fmul2_rn(make_float2(c, c), b); }
__device__ __forceinline__ double2 z_scale(double c, double2 b) { return make_double2(c * b.x, c * b.y); }
// a times a twiddle of the table: cos and sin in FP32; cos - 1 and sin in FP64, where a
// twiddle near 1 keeps its full precision (same four operations), and the low
// frequencies, which carry the result, meet only such twiddles.  Error of the reciprocal
// part, cos - 1 against cos: FP64 K = 32 5.6e-16, 6.1e-16, K = 128 3.7e-16, 4.1e-16; FP32 K =
// 256 3.0e-7, 2.4e-7 (the second rounding of full size costs more than the twiddles' error).
__device__ __forceinline__ float2 z_tw(float2 a, float c, float s) {
    return make_float2(a.x * c - a.y * s, a.x * s + a.y * c);
}
__device__ __forceinline__ double2 z_tw(double2 a, double c, double s) {
    return make_double2(fma(a.x, c, fma(-a.y, s, a.x)), fma(a.y, c, fma(a.x, s, a.y)));
}

// Twiddles of the composite radices, correctly rounded:
// Taylor series in double-double arithmetic (Dekker's products) after reduction to
// [-pi/4, pi/4].  Evaluated at compile time only.
struct DD {
    double h, l;
};
__host__ __device__ constexpr DD dd_sum(double a, double b) {
    const double s = a + b, t = s - a;
    return {s, (a - (s - t)) + (b - t)};
}
__host__ __device__ constexpr DD dd_add(DD a, DD b) {
    const DD s = dd_sum(a.h, b.h);
    return dd_sum(s.h, s.l + (a.l + b.l));
}
__host__ __device__ constexpr DD dd_mul(DD a, DD b) {
    const double f = 134217729.0;  // 2^27 + 1
    const double ah = f * a.h - (f * a.h - a.h), al = a.h - ah;
    const double bh = f * b.h - (f * b.h - b.h), bl = b.h - bh;
    const double p = a.h * b.h, e = ((ah * bh - p) + ah * bl + al * bh) + al * bl;
    return dd_sum(p, e + (a.h * b.l + a.l * b.h));
}
__host__ __device__ constexpr DD dd_div(DD a, double b) {
    const double q = a.h / b;
    const DD r = dd_add(a, dd_mul({-q, 0.0}, {b, 0.0}));
    return dd_sum(q, (r.h + r.l) / b);
}
// sin x (o = 1) or cos x - 1 (o = 0): sum of (-1)^k x^(2k+o) / (2k+o)!
__host__ __device__ constexpr double dd_series(DD x, int o) {
    const DD x2 = dd_mul(x, x);
    DD t = o ? x : DD{1.0, 0.0}, s = o ? x : DD{0.0, 0.0};
    for (int k = 1; k < 16; k++) {
        t = dd_div(dd_mul(t, x2), -(double)((2 * k + o) * (2 * k + o - 1)));
        s = dd_add(s, t);
    }
    return s.h;
}
// Quarter turns nearest to m/n of a turn, and the rest as cos - 1 and sin of x = 2 pi (m/n -
// q/4), |x| <= pi/4.
__host__ __device__ constexpr int root_turns(int m, int n) { return (4 * m + n / 2) / n; }
__host__ __device__ constexpr DD root_angle(int m, int n) {
    return dd_div(dd_mul({3.141592653589793116, 1.2246467991473532e-16},
                         {(double)(4 * m - root_turns(m, n) * n), 0.0}),
                  2.0 * n);
}
__host__ __device__ constexpr double root_cos1(int m, int n) { return dd_series(root_angle(m, n), 0); }
__host__ __device__ constexpr double root_sin(int m, int n) { return dd_series(root_angle(m, n), 1); }

// The first factor of a composite radix.
__host__ __device__ constexpr int z_split(int R) {
    return R % 4 == 0 ? 4 : R % 2 == 0 ? 2 : R % 3 == 0 ? 3 : 5;
}

// y[qb][pa] *= w_R^{qb pa} (conjugated: INV), I = qb A + pa
template <typename V, int R, bool INV, int A, int B, int I>
__device__ __forceinline__ void z_twiddle(V (&y)[B][A]) {
    constexpr int m = (I / A) * (I % A);
    V &a = y[I / A][I % A];
    using T = decltype(a.x);
    if constexpr (m != 0) {
        // e^{-2 pi i m / R} = (-i)^q e^{-i x}
        constexpr int q = root_turns(m, R) % 4;
        if constexpr (q == 1) a = INV ? z_make(-a.y, a.x) : z_make(a.y, -a.x);
        if constexpr (q == 2) a = z_make(-a.x, -a.y);
        if constexpr (q == 3) a = INV ? z_make(a.y, -a.x) : z_make(-a.y, a.x);
        if constexpr (4 * m != root_turns(m, R) * R) {
            using S = std::remove_reference_t<T>;
            constexpr S c = S(root_cos1(m, R) + (sizeof(S) == 4 ? 1.0 : 0.0)), sn = S(root_sin(m, R));
            a = z_tw(a, c, INV ? sn : -sn);
        }
    }
}
template <typename V, int R, bool INV, int A, int B, int... I>
__device__ __forceinline__ void z_twiddles(V (&y)[B][A], std::integer_sequence<int, I...>) {
    (z_twiddle<V, R, INV, A, B, I>(y), ...);
}

// K = R1 R2 transforms: the residue k1 of the frequencies as a signed number in FP64 (twiddles
// w^{n2 k1} with n2 |k1| <= K / 2), so that frequencies near zero of either sign meet
// twiddles near 1.  The R2-point transform of a k1 < 0 gives k1 + R1 k2 at k2, which is
// (R1 + k1) + R1 (k2 - 1).
template <typename T>
__host__ __device__ constexpr int z_signed(int k1, int R1) {
    return sizeof(T) == 8 && 2 * k1 > R1 ? k1 - R1 : k1;
}
// k2 counted from the residue k1 >= 0
__device__ __forceinline__ int z_k2(bool neg, int k2, int R2) {
    return k2 == 0 ? (neg ? R2 - 1 : 0) : k2 - (int)neg;
}

// In-place DFT of v (natural order in and out): out[p] = sum_q v[q] w^{pq}, w =
// e^{-2 pi i / R}, or its conjugate (INV).
template <int R, bool INV, typename V>
__device__ __forceinline__ void z_dft(V (&v)[R]) {
    using T = std::remove_reference_t<decltype(v[0].x)>;
    if constexpr (R == 1) {
    } else if constexpr (R == 2) {
        const V a = v[0];
        v[0] = z_add(a, v[1]);
        v[1] = z_sub(a, v[1]);
    } else if constexpr (R == 3) {
        constexpr T h = T(0.86602540378443864676);
        const V t = z_add(v[1], v[2]), u = z_sub(v[1], v[2]);
        const V m = z_fma(T(-0.5), t, v[0]);
        v[0] = z_add(v[0], t);
        // forward: v1 = m - i h u, v2 = m + i h u; inverse the other way round
        const V a = z_make(fma(h, u.y, m.x), fma(-h, u.x, m.y));
        const V b = z_make(fma(-h, u.y, m.x), fma(h, u.x, m.y));
        v[1] = INV ? b : a;
        v[2] = INV ? a : b;
    } else if constexpr (R == 4) {
        const V s02 = z_add(v[0], v[2]), d02 = z_sub(v[0], v[2]), s13 = z_add(v[1], v[3]);
        // -i (v1 - v3) forward, +i (v1 - v3) inverse
        const V jd = INV ? z_make(v[3].y - v[1].y, v[1].x - v[3].x)
                         : z_make(v[1].y - v[3].y, v[3].x - v[1].x);
        v[0] = z_add(s02, s13);
        v[1] = z_add(d02, jd);
        v[2] = z_sub(s02, s13);
        v[3] = z_sub(d02, jd);
    } else if constexpr (R == 5) {
        constexpr T c1 = T(0.30901699437494742410), c2 = T(-0.80901699437494742410),
                    s1 = T(0.95105651629515357212), s2 = T(0.58778525229247312917);
        const V t1 = z_add(v[1], v[4]), t2 = z_add(v[2], v[3]);
        const V u1 = z_sub(v[1], v[4]), u2 = z_sub(v[2], v[3]);
        const V m1 = z_fma(c2, t2, z_fma(c1, t1, v[0]));
        const V m2 = z_fma(c1, t2, z_fma(c2, t1, v[0]));
        const V n1 = z_fma(s2, u2, z_scale(s1, u1));
        const V n2 = z_fma(-s1, u2, z_scale(s2, u1));
        v[0] = z_add(v[0], z_add(t1, t2));
        // forward: v1 = m1 - i n1, v4 = m1 + i n1; inverse the other way round
        const V a1 = z_make(m1.x + n1.y, m1.y - n1.x), b1 = z_make(m1.x - n1.y, m1.y + n1.x);
        const V a2 = z_make(m2.x + n2.y, m2.y - n2.x), b2 = z_make(m2.x - n2.y, m2.y + n2.x);
        v[1] = INV ? b1 : a1;
        v[4] = INV ? a1 : b1;
        v[2] = INV ? b2 : a2;
        v[3] = INV ? a2 : b2;
    } else {
        // R = A B: q = qb + B qa, p = pa + A pb
        constexpr int A = z_split(R), B = R / A;
        V y[B][A];
#pragma unroll
        for (int qb = 0; qb < B; qb++) {
#pragma unroll
            for (int qa = 0; qa < A; qa++) y[qb][qa] = v[qb + B * qa];
            z_dft<A, INV>(y[qb]);
        }
        z_twiddles<V, R, INV, A, B>(y, std::make_integer_sequence<int, A * B>{});
#pragma unroll
        for (int pa = 0; pa < A; pa++) {
            V t[B];
#pragma unroll
            for (int qb = 0; qb < B; qb++) t[qb] = y[qb][pa];
            z_dft<B, INV>(t);
#pragma unroll
            for (int pb = 0; pb < B; pb++) v[pa + A * pb] = t[pb];
        }
    }
}

}  // namespace
}  // namespace spme
