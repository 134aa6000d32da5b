// FP64 real-space Ewald RPY pair sum over a cell list within rc, plus the self
// term (the operator of realspace.cu, for FP64 engines).
//
// What bounds it: a warp's FP64 instruction holds the SM's FP64 pipe for 16
// cycles (1/64 of the FP32 rate on this GPU), so everything but FP64
// instructions is nearly free and the sum costs (FP64 warp instructions per
// pair) x (idle lanes).  Hence:
//   * candidates are tested in FP32 only (a superset of the pairs within rc; the
//     exact FP64 distance is needed for the pair anyway), and the hits of up to 16
//     particles are listed together, so that the pair loop has no idle lanes but
//     those of its last round;
//   * the pair functions come from a table in s = r^2 (PairTable): no square root
//     and no division, the unit vector is folded in as G/r^2: 29 FP64 instructions
//     per pair and right-hand side (geometry 6, segment offset 1, two Horner chains
//     of degree six 12, application 10);
//   * the listed pairs are split evenly over the lanes (realspace_pairs.cuh), which
//     accumulate in registers: no 5-step FP64 butterfly per particle.
// N = 1e6, L = 480, rc = 10 (38 pairs per particle), one right-hand side:
// 15.19 -> 3.28 ms; N = 1e5, L = 220: 1.645 -> 0.357 ms (FP64 pipe floor 2.0 ms: 36
// FP64 warp instructions per particle at 16 cycles each).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "realspace_pairs.cuh"
#include "pdl.cuh"

namespace spme {

namespace {

// M_real(r) = F I + G rhat rhat: Beenakker's real-space form divided by a, and
// for r < 2a plus (overlap RPY - far-field RPY), written in the cancellation-free
// form of realspace.cu: x = xi r, S(x) = erf(x)/x and psi(x) = (erf(x) -
// 2x e^{-x^2}/sqrt(pi)) / x^3, for x < 0.5 from their Maclaurin series in x^2
// (thirteen terms: below 1e-19 relative; the factor 2/sqrt(pi) outside).  `near`
// selects the form; both are analytic on either side of r = 2a.
__host__ __device__ inline void real_FG(double r, double xi, double a, bool near, double &F,
                                        double &G) {
    const double rsp = 0.56418958354775628695;  // 1/sqrt(pi)
    const double x = xi * r, x2 = x * x, e = exp(-x2);
    if (near) {
        double S = 0.0, P = 0.0;
        if (x < 0.5) {
            const double ks[13] = {1.0, -1.0 / 3, 1.0 / 10, -1.0 / 42, 1.0 / 216,
                                   -1.0 / 1320, 1.0 / 9360, -1.0 / 75600, 1.0 / 685440,
                                   -1.0 / 6894720, 1.0 / 76204800, -1.0 / 918086400,
                                   1.0 / 11975040000};
            const double kp[13] = {2.0 / 3, -2.0 / 5, 1.0 / 7, -1.0 / 27, 1.0 / 132,
                                   -1.0 / 780, 1.0 / 5400, -1.0 / 42840, 1.0 / 383040,
                                   -1.0 / 3810240, 1.0 / 41731200, -1.0 / 498960000,
                                   1.0 / 6466521600};
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
            for (int k = 12; k >= 0; k--) {
                S = S * x2 + ks[k];
                P = P * x2 + kp[k];
            }
            S *= 2.0 * rsp;
            P *= 2.0 * rsp;
        } else {
            const double ef = erf(x);
            S = ef / x;
            P = (ef - 2.0 * rsp * x * e) / (x2 * x);
        }
        const double x4 = x2 * x2, xi3a2 = xi * xi * xi * a * a;
        F = xi * (-0.75 * S + rsp * e * (3.0 * x2 - 4.5)) +
            xi3a2 * (-0.5 * P + rsp * e * (4.0 * x4 - 20.0 * x2 + 14.0)) +
            (1.0 - 9.0 * r / (32.0 * a)) / a;
        G = xi * (-0.75 * S + rsp * e * (1.5 - 3.0 * x2)) +
            xi3a2 * (1.5 * P + rsp * e * (-4.0 * x4 + 16.0 * x2 - 2.0)) + 3.0 * r / (32.0 * a * a);
        return;
    }
    const double ec = erfc(x);
    const double r2 = r * r, a3 = a * a * a, ir = 1.0 / r, ir3 = ir * ir * ir, ir2 = ir * ir;
    const double xi2 = xi * xi, xi3 = xi2 * xi, xi5 = xi3 * xi2, xi7 = xi5 * xi2;
    const double f = ec * (0.75 * a * ir + 0.5 * a3 * ir3) +
                     e * rsp * (4.0 * xi7 * a3 * r2 * r2 + 3.0 * xi3 * a * r2 -
                                20.0 * xi5 * a3 * r2 - 4.5 * xi * a + 14.0 * xi3 * a3 +
                                xi * a3 * ir2);
    const double g = ec * (0.75 * a * ir - 1.5 * a3 * ir3) +
                     e * rsp * (-4.0 * xi7 * a3 * r2 * r2 - 3.0 * xi3 * a * r2 +
                                16.0 * xi5 * a3 * r2 + 1.5 * xi * a - 2.0 * xi3 * a3 -
                                3.0 * xi * a3 * ir2);
    F = f / a;
    G = g / a;
}

// A = F and B = G / r^2 at s = r^2 (B = 0 at s = 0, where the pair has no
// direction): from the table, or directly where s lies outside it.
__device__ __forceinline__ void pair_AB(const PairTable &tb, double s, double xi, double a,
                                        double &Av, double &Bv) {
    const long long bits = __double_as_longlong(s);
    if (tb.coef && bits >= tb.lo_bits && bits <= tb.hi_bits) {
        const int hw = (int)(bits >> 32);
        const int seg = (hw >> tb.shift) - tb.base + (bits >= tb.mid_bits ? 1 : 0);
        // offset from the segment's centre: same exponent, so the difference is exact
        const double ctr = __hiloint2double((hw & ~((1 << tb.shift) - 1)) | (1 << (tb.shift - 1)), 0);
        const double v = s - ctr;
        const double2 *c =
            reinterpret_cast<const double2 *>(tb.coef) + (size_t)seg * (kPairDeg + 1);
        double2 q = __ldg(c + kPairDeg);
        Av = q.x;
        Bv = q.y;
#pragma unroll
        for (int k = kPairDeg - 1; k >= 0; k--) {
            q = __ldg(c + k);
            Av = fma(Av, v, q.x);
            Bv = fma(Bv, v, q.y);
        }
        return;
    }
    const double r = sqrt(s);
    double F, G;
    real_FG(r, xi, a, r < 2.0 * a, F, G);
    Av = F;
    Bv = s > 0.0 ? G / s : 0.0;
}

template <int RB>
__device__ __forceinline__ void realspace64_body(const RealArgs<double> &A, int cell) {
    const long long rc2_bits = __double_as_longlong(A.rc2);
    realspace_few_body<double, RB>(A, cell, A.L, A.h, A.rc2, A.self_c,
                                   [&](double s, double &Av, double &Bv) {
                                       if (__double_as_longlong(s) >= rc2_bits) return false;
                                       pair_AB(A.tab, s, A.xi, A.a, Av, Bv);
                                       return true;
                                   });
}

template <int RB>
__global__ void __launch_bounds__(kRsThreads, RB == 1 ? 7 : 4) k_realspace64(RealArgs<double> A) {
    pdl_wait();
    realspace64_body<RB>(A, blockIdx.x);
}

// Many systems in one persistent launch over their cells.
template <int RB>
__global__ void __launch_bounds__(kRsThreads, RB == 1 ? 7 : 4)
k_realspace64_batch(const RealArgs<double> *__restrict__ sys, const int *__restrict__ prefix,
                    int nsys, int total) {
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int k = batch_find(prefix, nsys, w);
        realspace64_body<RB>(sys[k], w - prefix[k]);
        __syncthreads();
    }
}

// Right-hand sides per sweep: the fewest sweeps of at most 4 (12 FP64
// accumulators per lane), evenly filled.
int sweep_width(int R) {
    const int n = (R + 3) / 4;
    return (R + n - 1) / n;
}

template <int RB>
cudaError_t launch_batch64(const RealArgs<double> *sys, const int *prefix, int nsys, int total,
                           cudaStream_t s) {
    auto kern = k_realspace64_batch<RB>;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kRsThreads, 0);
    const int grid = std::max(1, std::min(total, sms * std::max(per_sm, 1)));
    kern<<<grid, kRsThreads, 0, s>>>(sys, prefix, nsys, total);
    return cudaGetLastError();
}

}  // namespace

template <>
cudaError_t launch_realspace<double>(int nc, const int *cell_off, const int *cell_perm,
                                     const void *cpos, const double *F, const double *, int R,
                                     double L, double rc, double xi, double a, int with_self,
                                     const PairTable &tab, double *W, cudaStream_t s) {
    if (R <= 0) return cudaSuccess;
    const RealArgs<double> A = real_args<double>(nc, cell_off, cell_perm, cpos, F, nullptr, R, L, rc,
                                                 xi, a, with_self, tab, W);
    const int ncell = nc * nc * nc;
    switch (sweep_width(R)) {
        case 1: pdl_launch(k_realspace64<1>, ncell, kRsThreads, 0, s, A); break;
        case 2: pdl_launch(k_realspace64<2>, ncell, kRsThreads, 0, s, A); break;
        case 3: pdl_launch(k_realspace64<3>, ncell, kRsThreads, 0, s, A); break;
        default: pdl_launch(k_realspace64<4>, ncell, kRsThreads, 0, s, A); break;
    }
    return cudaGetLastError();
}

template <>
cudaError_t launch_realspace_batch<double>(const RealArgs<double> *sys, const int *prefix,
                                           int nsys, int total, int R, cudaStream_t s) {
    if (total <= 0 || R <= 0) return cudaSuccess;
    switch (sweep_width(R)) {
        case 1: return launch_batch64<1>(sys, prefix, nsys, total, s);
        case 2: return launch_batch64<2>(sys, prefix, nsys, total, s);
        case 3: return launch_batch64<3>(sys, prefix, nsys, total, s);
        default: return launch_batch64<4>(sys, prefix, nsys, total, s);
    }
}

namespace {

long long bits_of(double v) {
    long long b;
    std::memcpy(&b, &v, sizeof(b));
    return b;
}

// Polynomials (degree kPairDeg, in the offset from the segment's centre) of A = F
// and B = G / s on [s0, s0 + h], interleaved, through the values at the Chebyshev
// nodes.
void fit_segment(double s0, double h, double xi, double a, bool near, double *out) {
    constexpr int n = kPairDeg + 1;
    static double node[n], cs[n][n], cheb[n][n];  // cheb[k][i]: the power i in T_k
    static const bool once = [] {
        for (int j = 0; j < n; j++) {
            node[j] = std::cos(M_PI * (j + 0.5) / n);
            for (int k = 0; k < n; k++) cs[k][j] = std::cos(M_PI * k * (j + 0.5) / n);
        }
        cheb[0][0] = cheb[1][1] = 1.0;
        for (int k = 2; k < n; k++)
            for (int i = 0; i < n; i++) cheb[k][i] = (i ? 2.0 * cheb[k - 1][i - 1] : 0.0) - cheb[k - 2][i];
        return true;
    }();
    (void)once;
    double f[2][n];
    for (int j = 0; j < n; j++) {
        const double s = s0 + 0.5 * h * (node[j] + 1.0);
        real_FG(std::sqrt(s), xi, a, near, f[0][j], f[1][j]);
        f[1][j] /= s;
    }
    for (int w = 0; w < 2; w++) {
        // Chebyshev coefficients, then powers of t, then of the offset v = t h / 2
        double o[n] = {};
        for (int k = 0; k < n; k++) {
            double q = 0.0;
            for (int j = 0; j < n; j++) q += f[w][j] * cs[k][j];
            const double c = (k ? 2.0 : 1.0) * q / n;
            for (int i = k & 1; i <= k; i += 2) o[i] += c * cheb[k][i];
        }
        double sc = 1.0;
        for (int i = 0; i < n; i++) {
            out[2 * i + w] = o[i] * sc;
            sc /= 0.5 * h;
        }
    }
}

}  // namespace

bool build_pair_table(double xi, double a, double rc, std::vector<double> *coef, PairTable *t) {
    // s in [lo, mid): overlap form (r < 2a); [mid, rc^2]: far form.  Below lo =
    // (a/2)^2 the closed form is evaluated directly (rare pairs).
    const double lo = 0.25 * a * a, mid = 4.0 * a * a, hi = rc * rc;
    if (hi <= lo) return false;
    // (2^m segments per octave of s: twice those that pass, so that the fit, 2^-7 of the
    // bound then, stays below the rounding of the values it goes through.  Every fourth
    // segment, and the ends of either form, is tried: the error varies slowly along s, and
    // all of them took an engine's creation from 1.26 to 1.70 ms at N = 300)
    bool passed = false;
    for (int m = 6; m <= (passed ? 11 : 10); m++) {
        const int shift = 20 - m;
        auto seg_of = [&](double s) { return (int)((bits_of(s) >> 32) >> shift); };
        auto start_of = [&](int g) {
            const long long b = ((long long)g << shift) << 32;
            double s;
            std::memcpy(&s, &b, sizeof(s));
            return s;
        };
        const int base = seg_of(lo), last = seg_of(hi);
        // the segment holding mid has both forms: the near one at its own index, the
        // far one at the next, and all later segments shift by one
        const int gm = mid > hi ? last + 1 : seg_of(mid);
        const int n = last - base + 1 + (gm <= last ? 1 : 0);
        coef->assign((size_t)n * (kPairDeg + 1) * 2, 0.0);
        bool ok = true;
        for (int q = 0; q < n && ok; q++) {
            const bool near = q <= gm - base;
            if (!passed && q % 4 && q != n - 1 && q != gm - base && q != gm - base + 1) continue;
            const int g = base + q - (near ? 0 : 1);
            const double s0 = start_of(g), h = start_of(g + 1) - s0;
            double *c = coef->data() + (size_t)q * (kPairDeg + 1) * 2;
            fit_segment(s0, h, xi, a, near, c);
            // the fit between the nodes, relative to the function scale there
            for (int p = 0; p <= 8 && ok && !passed; p++) {
                const double s = s0 + h * p / 8.0, v = s - (s0 + 0.5 * h);
                if (s < lo || s > hi || (near != (s < mid))) continue;
                double F, G;
                real_FG(std::sqrt(s), xi, a, near, F, G);
                double A = c[2 * kPairDeg], B = c[2 * kPairDeg + 1];
                for (int k = kPairDeg - 1; k >= 0; k--) {
                    A = A * v + c[2 * k];
                    B = B * v + c[2 * k + 1];
                }
                const double scale = std::fabs(F) + std::fabs(G) + 1e-300;
                ok = std::fabs(A - F) <= 2e-13 * scale && std::fabs(B * s - G) <= 2e-13 * scale;
            }
        }
        if (!ok) continue;
        if (!passed) {
            passed = true;
            continue;
        }
        t->coef = nullptr;  // the caller points it at the device copy
        t->lo_bits = bits_of(lo);
        t->mid_bits = bits_of(mid);
        t->hi_bits = bits_of(hi);
        t->base = base;
        t->shift = shift;
        return true;
    }
    return false;
}

}  // namespace spme
