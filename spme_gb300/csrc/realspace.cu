// FP32 real-space Ewald RPY pair sum over a cell list within rc, plus the self
// term (FP64: realspace_fp64.cu).  The reference has no real-space part (it
// computes only M_recip, old-version/spme.c:560-726); this restates Beenakker, J.
// Chem. Phys. 85, 1581 (1986), in the reference's units (mobility x 6 pi eta,
// matching scalar_recip at old-version/spme.c:43-60), with the RPY overlap form
// for pairs closer than 2a.
//
// What bounds it: issued instructions (the sum was 71 % issue-active at 1814 warp
// instructions per particle for 16 right-hand sides), so pairs are listed first
// and everything after runs with full warps:
//   * one CTA per cell of edge >= rc stages the candidates of the 27 neighbour cells
//     once; each warp lists the pairs within rc of up to 16 of its particles
//     (ballot-compacted, realspace_pairs.cuh);
//   * the pair functions are evaluated 32 listed pairs at a time;
//   * up to kRealFew right-hand sides: the listed pairs are split evenly over the
//     lanes, which accumulate in registers (realspace_few_body); a partner's row is
//     padded to 16-byte vectors, as every lane reads another row;
//   * more: lanes as (pair slot, two right-hand sides) apply the evaluated pairs with
//     two-lane FMAs (fma.rn.f32x2); the partner's force rows come component by
//     component (F2[j][d][r]), so a right-hand side pair is one 8-byte load and a
//     row's load touches one line instead of the whole interleaved row.
// More right-hand sides: sums of a window's pairs (64, split over the slots) are plain FP32;
// longer runs, the sum over the slots and the self term carry TwoSum; fewer: ShareSum
// (realspace_pairs.cuh).  Plain sums were 5 % (R = 16) to 11 % (R = 1) faster and 1 to 2 % less exact.
// Measured (ms): N = 1e6, R = 16 1.65 -> 1.62, R = 4 1.35 -> 1.32, R = 1 1.32 -> 0.92; N = 2e5, R = 16
// 0.442 -> 0.428; N = 1e5, R = 1 0.161 -> 0.112; 64 uneven systems, R = 4 1.53 -> 1.50.  The
// partners' rows come mostly from L2 (12 % L1 hits), whose latency bounds it now; more warps
// per SM at fewer registers spill (1.57 ms at 12 blocks where 10 took 1.52), a table of the pair functions in
// shared-memory-free FP32 cost more in scattered loads than it saved (1.64 ms).
#include <algorithm>
#include <cmath>
#include <vector>

#include "realspace_pairs.cuh"
#include "pdl.cuh"

namespace spme {

namespace {

// M_real(r) = F I + G rhat rhat: Beenakker's real-space form divided by a, and
// for r < 2a plus (overlap RPY - far-field RPY).  For r < 2a the 1/r and 1/r^3
// terms of the two cancel; written with x = xi r, S(x) = erf(x)/x and psi(x)
// they cancel analytically (no loss of precision as r -> 0, finite at r = 0):
//   F = xi [-3/4 S + e (3x^2 - 9/2)/sqrt(pi)] + xi^3 a^2 [-psi/2 + e (4x^4 - 20x^2 + 14)/sqrt(pi)]
//       + (1 - 9r/(32a)) / a
//   G = xi [-3/4 S + e (3/2 - 3x^2)/sqrt(pi)] + xi^3 a^2 [3psi/2 + e (-4x^4 + 16x^2 - 2)/sqrt(pi)]
//       + 3r/(32 a^2)
// with e = exp(-x^2); S and psi from their series for x < 0.5.
// FP32 engines: F, G and ir = 1/r (0 at r = 0) from r^2, with the launch's
// coefficients (RealCoef): one reciprocal square root gives r, 1/r and the
// unit vector; the far field (r >= 2a) is real_FG's far form divided through
// by a, the near field real_FG's cancellation-free form with FP32 constants.
__device__ __forceinline__ void real_FG_f32(float r2, const RealCoef &c, float &F, float &G,
                                            float &ir) {
    constexpr float rsp = 0.56418958354775628695f;  // 1/sqrt(pi)
    // (below r = 1e-18 as at r = 0: the caller's 1/r^2 would overflow, and G vanishes there)
    ir = r2 >= 1e-36f ? rsqrtf(r2) : 0.f;
    const float r = r2 * ir;
    if (r2 < c.a2x4) {
        const float x = c.xi * r, x2 = x * x, e = expf(-x2);
        float S, P;
        if (x < 0.5f) {
            constexpr float ks[10] = {1.0f, -1.0f / 3, 1.0f / 10, -1.0f / 42, 1.0f / 216,
                                      -1.0f / 1320, 1.0f / 9360, -1.0f / 75600,
                                      1.0f / 685440, -1.0f / 6894720};
            constexpr float kp[10] = {2.0f / 3, -2.0f / 5, 1.0f / 7, -1.0f / 27, 1.0f / 132,
                                      -1.0f / 780, 1.0f / 5400, -1.0f / 42840,
                                      1.0f / 383040, -1.0f / 3810240};
            S = 0.f;
            P = 0.f;
#pragma unroll
            for (int k = 9; k >= 0; k--) {
                S = fmaf(S, x2, ks[k]);
                P = fmaf(P, x2, kp[k]);
            }
            S *= 2.f * rsp;
            P *= 2.f * rsp;
        } else {
            const float ef = erff(x), ix = 1.f / x;
            S = ef * ix;
            P = (ef - 2.f * rsp * x * e) * (ix * ix * ix);
        }
        const float x4 = x2 * x2, re = rsp * e;
        F = c.xi * (-0.75f * S + re * (3.f * x2 - 4.5f)) +
            c.xi3a2 * (-0.5f * P + re * (4.f * x4 - 20.f * x2 + 14.f)) + (c.ia - c.n1 * r);
        G = c.xi * (-0.75f * S + re * (1.5f - 3.f * x2)) +
            c.xi3a2 * (1.5f * P + re * (-4.f * x4 + 16.f * x2 - 2.f)) + c.n2 * r;
        return;
    }
    const float ec = erfcf(c.xi * r), e = expf(-c.xi2 * r2);
    const float ir2 = ir * ir, ir3 = ir2 * ir, r4 = r2 * r2;
    const float pF = fmaf(c.A4, r4, fmaf(c.A2, r2, fmaf(c.Am2, ir2, c.A0)));
    const float pG = fmaf(-c.A4, r4, fmaf(c.B2, r2, fmaf(c.Bm2, ir2, c.B0)));
    F = ec * fmaf(c.c1, ir3, 0.75f * ir) + e * pF;
    G = ec * fmaf(c.c3, ir3, 0.75f * ir) + e * pG;
}

template <int RB>
__device__ __forceinline__ void real_few(const RealArgs<float> &A, int cell) {
    realspace_few_body<float, RB>(A, cell, A.cf.L, A.cf.h, A.cf.rc2, A.cf.self_c,
                                  [&](float s, float &Av, float &Bv) {
                                      float ir;
                                      real_FG_f32(s, A.cf, Av, Bv, ir);
                                      Bv *= ir * ir;
                                      return true;
                                  });
}

constexpr int kWin = 64;      // pairs evaluated together
constexpr int kListM = 512;   // listed pairs per warp

struct ManyShared {
    float4 r0[kWin];  // displacement, A
    float2 r1[kWin];  // B, partner (bits)
    float4 pf[kGroup];
    uint32_t list[kListM];
    int beg[kGroup + 2];
};

// One cell, more than kRealFew right-hand sides: RL lanes of two right-hand sides
// each, 32 / RL pair slots; blocks of 2 RL right-hand sides in sequence.
template <int RL>
__device__ __forceinline__ void real_many(const RealArgs<float> &A, int cell) {
    constexpr int PS = 32 / RL;
    constexpr int kFold = kWin / PS;  // pairs per slot summed in plain FP32, at most
    __shared__ CellShared<float> csh;
    __shared__ ManyShared wsh[kRsWarps];
    const int ib0 = __ldg(A.cell_off + cell), ie = __ldg(A.cell_off + cell + 1);
    if (ib0 == ie) return;  // uniform over the block
    const Cell<float> cl(csh, cell, A.nc, A.cell_off, A.cell_perm, A.cpos, A.cf.L, A.cf.h,
                         A.cf.rc2);
    const int R = A.R, R2 = rows_even(R), C = 3 * R;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int slot = lane / RL, rl = lane % RL;
    ManyShared &ws = wsh[warp];

    // this warp's share of the cell's particles, kGroup at a time
    const int half = (ie - ib0 + kRsWarps - 1) / kRsWarps;
    const int wb = ib0 + warp * half, we = min(ie, wb + half);
    for (int g0 = wb; g0 < we; g0 += kGroup) {
        const int np = min(kGroup, we - g0);
        if (lane < np) {
            const float4 p = cl.cpos[g0 + lane];
            ws.pf[lane] = make_float4(p.x, p.y, p.z, __int_as_float(A.cell_perm[g0 + lane]));
        }
        __syncwarp();
        for (int rb = 0; rb < R; rb += 2 * RL) {
            const int r = rb + 2 * rl;  // this lane's right-hand sides r, r + 1
            const bool live = r < R;
            const float *__restrict__ Fr = A.F2 + r;
            ListState ls;
            // sums of the current particle: two-lane partial sums, moved to compensated
            // ones before a slot has more than kFold pairs
            float2 s0 = make_float2(0.f, 0.f), s1 = s0, s2 = s0;
            PairSum<float> sum[6];
            int nfold = 0, cnt = 0;
            auto fold = [&]() {
                const float v[6] = {s0.x, s1.x, s2.x, s0.y, s1.y, s2.y};
#pragma unroll
                for (int q = 0; q < 6; q++) sum[q].add(v[q]);
                s0 = s1 = s2 = make_float2(0.f, 0.f);
                nfold++;
                cnt = 0;
            };
            while (ls.il < np) {
                const int ilo = ls.il;
                const int nh = list_pairs<true, kListM>(cl, ws.pf, np, ws.list, ws.beg, ls, PS);
                const int last = ls.q0 == 0 ? ls.il - 1 : ls.il;
                int wend = 0;  // entries [wend - kWin, wend) are evaluated
                for (int ip = ilo; ip <= last; ip++) {
                    int k = ws.beg[ip];
                    const int e = ws.beg[ip + 1];
                    while (k < e) {
                        if (k >= wend) {
                            __syncwarp();
#pragma unroll
                            for (int v = 0; v < kWin / 32; v++) {
                                const int t = wend + 32 * v + lane;
                                if (t < nh) {
                                    const uint32_t ent = ws.list[t];
                                    const float4 me = ws.pf[ent >> 28];
                                    float d0 = 0.f, d1 = 0.f, d2 = 0.f, Av = 0.f, Bv = 0.f;
                                    int j = -1;  // padding: the row of zeros
                                    if ((ent & kNoCand) != kNoCand) {
                                        float x, y, z;
                                        cl.candidate((int)(ent & kNoCand), x, y, z, j);
                                        d0 = me.x - x;
                                        d1 = me.y - y;
                                        d2 = me.z - z;
                                        cl.min_image(d0, d1, d2);
                                        float ir;
                                        real_FG_f32(fmaf(d2, d2, fmaf(d1, d1, d0 * d0)), A.cf, Av,
                                                    Bv, ir);
                                        Bv *= ir * ir;
                                    }
                                    const int q = 32 * v + lane;
                                    ws.r0[q] = make_float4(d0, d1, d2, Av);
                                    ws.r1[q] = make_float2(Bv, __int_as_float(j));
                                }
                            }
                            wend += kWin;
                            __syncwarp();
                        }
                        const int ke = min(e, wend);
                        const int o = wend - kWin - slot;
                        // (whole pairs per slot: the list is padded)
                        if (cnt + (ke - k) / PS > kFold) fold();
                        cnt += (ke - k) / PS;
                        if (live) {
#pragma unroll 2
                            for (int q = k - o; q < ke - o; q += PS) {
                                const float4 a = ws.r0[q];
                                const float2 b = ws.r1[q];
                                const float *fj =
                                    Fr + (ptrdiff_t)__float_as_int(b.y) * (3 * R2);
                                const float2 f0 = __ldg(reinterpret_cast<const float2 *>(fj));
                                const float2 f1 = __ldg(reinterpret_cast<const float2 *>(fj + R2));
                                const float2 f2 =
                                    __ldg(reinterpret_cast<const float2 *>(fj + 2 * R2));
                                const float2 d0 = make_float2(a.x, a.x), d1 = make_float2(a.y, a.y),
                                             d2 = make_float2(a.z, a.z), Av = make_float2(a.w, a.w);
                                const float2 g = __fmul2_rn(
                                    make_float2(b.x, b.x),
                                    __ffma2_rn(d2, f2, __ffma2_rn(d1, f1, __fmul2_rn(d0, f0))));
                                // (one rounding of a pair's term into the sum)
                                s0 = __fadd2_rn(s0, __ffma2_rn(g, d0, __fmul2_rn(Av, f0)));
                                s1 = __fadd2_rn(s1, __ffma2_rn(g, d1, __fmul2_rn(Av, f1)));
                                s2 = __fadd2_rn(s2, __ffma2_rn(g, d2, __fmul2_rn(Av, f2)));
                            }
                        }
                        k = ke;
                    }
                    if (ip == ls.il) break;  // cut: goes on in the next list
                    // the slots' sums and the self term, compensated, to the particle's row:
                    // half of the slots take the first right-hand side, half the second
                    const int ii = __float_as_int(ws.pf[ip].w);
                    const bool second = (lane & RL) != 0;
                    PairSum<float> t[3];
                    if (nfold) {
                        fold();
#pragma unroll
                        for (int d = 0; d < 3; d++) {
                            t[d] = second ? sum[3 + d] : sum[d];
                            t[d].join(shfl_xor(second ? sum[d] : sum[3 + d], RL));
                            sum[d] = sum[3 + d] = PairSum<float>();
                        }
                    } else {
                        const float v[6] = {s0.x, s1.x, s2.x, s0.y, s1.y, s2.y};
#pragma unroll
                        for (int d = 0; d < 3; d++) {
                            t[d].s = second ? v[3 + d] : v[d];
                            t[d].add(__shfl_xor_sync(0xffffffffu, second ? v[d] : v[3 + d], RL));
                        }
                    }
                    s0 = s1 = s2 = make_float2(0.f, 0.f);
                    nfold = cnt = 0;
#pragma unroll
                    for (int w = 2 * RL; w < 32; w <<= 1) {
#pragma unroll
                        for (int d = 0; d < 3; d++) t[d].join(shfl_xor(t[d], w));
                    }
                    const int rs = r + (int)second;
                    if (slot < 2 && rs < R) {
                        const float *fi = A.F2 + (size_t)ii * (size_t)(3 * R2) + rs;
                        float *o = A.W + (size_t)ii * C + 3 * rs;
#pragma unroll
                        for (int d = 0; d < 3; d++) {
                            if (A.with_self) t[d].add(A.cf.self_c * __ldg(fi + d * R2));
                            o[d] = t[d].value();
                        }
                    }
                }
                __syncwarp();
            }
        }
    }
}

// W: lanes per right-hand side pair group of the many-right-hand-sides form (0: the
// few-right-hand-sides form with RB right-hand sides per sweep).
template <int W, int RB>
__device__ __forceinline__ void real_body(const RealArgs<float> &A, int cell) {
    if constexpr (W > 0) real_many<W>(A, cell);
    else real_few<RB>(A, cell);
}

template <int W, int RB>
__global__ void __launch_bounds__(kRsThreads, 10) k_realspace(RealArgs<float> A) {
    pdl_wait();
    real_body<W, RB>(A, blockIdx.x);
}

// Many systems in one persistent launch over their cells.
template <int W, int RB>
__global__ void __launch_bounds__(kRsThreads, 10)
k_realspace_batch(const RealArgs<float> *__restrict__ sys, const int *__restrict__ prefix,
                  int nsys, int total) {
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int k = batch_find(prefix, nsys, w);
        // (a copy: fields read through the list would be loaded again after every store)
        const RealArgs<float> A = sys[k];
        real_body<W, RB>(A, w - prefix[k]);
        __syncthreads();
    }
}

struct Launch {
    const RealArgs<float> *sys;  // batched: work list, prefix, systems, cells
    const int *prefix;
    int nsys, total;
    cudaStream_t s;
};

template <int W, int RB>
cudaError_t launch_form(const RealArgs<float> *one, const Launch &l) {
    if (one) {
        pdl_launch(k_realspace<W, RB>, l.total, kRsThreads, 0, l.s, *one);
        return cudaGetLastError();
    }
    auto kern = k_realspace_batch<W, RB>;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kRsThreads, 0);
    const int grid = std::max(1, std::min(l.total, sms * std::max(per_sm, 1)));
    kern<<<grid, kRsThreads, 0, l.s>>>(l.sys, l.prefix, l.nsys, l.total);
    return cudaGetLastError();
}

cudaError_t launch_any(const RealArgs<float> *one, int R, const Launch &l) {
    if (l.total <= 0 || R <= 0) return cudaSuccess;
    switch (R) {
        case 1: return launch_form<0, 1>(one, l);
        case 2: return launch_form<0, 2>(one, l);
        default:
            if (R <= 4) return launch_form<2, 0>(one, l);
            if (R <= 8) return launch_form<4, 0>(one, l);
            if (R <= 16) return launch_form<8, 0>(one, l);
            return launch_form<16, 0>(one, l);
    }
}

}  // namespace

double real_self_coeff(double xi, double a) {
    const double rsp = 0.56418958354775628695;
    return (1.0 - 6.0 * xi * a * rsp + 40.0 / 3.0 * xi * xi * xi * a * a * a * rsp) / a;
}

template <typename T>
RealArgs<T> real_args(int nc, const int *cell_off, const int *cell_perm, const void *cpos,
                      const T *F, const T *F2, int R, double L, double rc, double xi, double a, int with_self,
                      const PairTable &tab, T *W) {
    RealArgs<T> A;
    A.nc = nc;
    A.cell_off = cell_off;
    A.cell_perm = cell_perm;
    A.cpos = cpos;
    A.F = F;
    A.F2 = F2;
    A.W = W;
    A.R = R;
    A.with_self = with_self;
    A.L = L;
    A.h = L / nc;
    A.rc2 = rc * rc;
    A.xi = xi;
    A.a = a;
    A.self_c = real_self_coeff(xi, a);
    A.tab = tab;
    const double rsp = 0.56418958354775628695, a2 = a * a, xi2 = xi * xi, xi3 = xi2 * xi,
                 xi5 = xi3 * xi2, xi7 = xi5 * xi2;
    RealCoef &c = A.cf;
    c.xi = (float)xi;
    c.xi2 = (float)xi2;
    c.a2x4 = (float)(4.0 * a2);
    c.xi3a2 = (float)(xi3 * a2);
    c.ia = (float)(1.0 / a);
    c.n1 = (float)(9.0 / (32.0 * a2));
    c.n2 = (float)(3.0 / (32.0 * a2));
    c.A4 = (float)(4.0 * rsp * xi7 * a2);
    c.A2 = (float)(rsp * (3.0 * xi3 - 20.0 * xi5 * a2));
    c.A0 = (float)(rsp * (-4.5 * xi + 14.0 * xi3 * a2));
    c.Am2 = (float)(rsp * xi * a2);
    c.B2 = (float)(rsp * (-3.0 * xi3 + 16.0 * xi5 * a2));
    c.B0 = (float)(rsp * (1.5 * xi - 2.0 * xi3 * a2));
    c.Bm2 = (float)(-3.0 * rsp * xi * a2);
    c.c1 = (float)(0.5 * a2);
    c.c3 = (float)(-1.5 * a2);
    c.L = (float)L;
    c.h = (float)A.h;
    c.rc2 = (float)A.rc2;
    c.self_c = (float)A.self_c;
    return A;
}

template <>
cudaError_t launch_realspace<float>(int nc, const int *cell_off, const int *cell_perm,
                                    const void *cpos, const float *F, const float *F2, int R,
                                    double L, double rc, double xi, double a, int with_self,
                                    const PairTable &tab, float *W, cudaStream_t s) {
    if (!F2) return cudaErrorInvalidValue;
    const RealArgs<float> A = real_args<float>(nc, cell_off, cell_perm, cpos, F, F2, R, L, rc, xi,
                                               a, with_self, tab, W);
    return launch_any(&A, R, Launch{nullptr, nullptr, 0, nc * nc * nc, s});
}

template <>
cudaError_t launch_realspace_batch<float>(const RealArgs<float> *sys, const int *prefix, int nsys,
                                          int total, int R, cudaStream_t s) {
    return launch_any(nullptr, R, Launch{sys, prefix, nsys, total, s});
}

template RealArgs<float> real_args<float>(int, const int *, const int *, const void *,
                                          const float *, const float *, int, double, double,
                                          double, double, int, const PairTable &, float *);
template RealArgs<double> real_args<double>(int, const int *, const int *, const void *,
                                            const double *, const double *, int, double, double,
                                            double, double, int, const PairTable &, double *);

}  // namespace spme
