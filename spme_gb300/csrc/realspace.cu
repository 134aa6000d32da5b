// FP32 real-space Ewald RPY pair sum over a cell list within rc, plus the self
// term (FP64: realspace_fp64.cu).  The reference has no real-space part (it computes only M_recip,
// old-version/spme.c:560-726); this restates Beenakker, J. Chem. Phys. 85,
// 1581 (1986), in the reference's units (mobility x 6 pi eta, matching
// scalar_recip at old-version/spme.c:43-60), with the RPY overlap form for
// pairs closer than 2a.
//
// One CTA per cell of edge >= rc; a warp per particle of the cell against the
// candidates of the 27 neighbour cells (details at the kernel below).
#include <algorithm>
#include <cmath>

#include "kernels.h"

namespace spme {

namespace {

constexpr int kThreads = 64;  // two warps per cell: ~4-5 particles each at typical densities

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
    ir = r2 > 0.f ? rsqrtf(r2) : 0.f;
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

// Accumulator across pair batches: FP32 with Knuth's TwoSum error term carried
// alongside (the FP64 pipe is a small fraction of the FP32 rate on this GPU, and
// a handful of double adds per particle had become the kernel's limiter).
struct PairSum {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float t = s + x, bp = t - s;
        c += (s - (t - bp)) + (x - bp);
        s = t;
    }
    __device__ __forceinline__ void add(const PairSum &o) {
        add(o.s);
        c += o.c;
    }
    __device__ __forceinline__ float value() const { return s + c; }
};

__device__ __forceinline__ PairSum shfl_xor(const PairSum &a, int o) {
    PairSum b;
    b.s = __shfl_xor_sync(0xffffffffu, a.s, o);
    b.c = __shfl_xor_sync(0xffffffffu, a.c, o);
    return b;
}

constexpr int kWarps = kThreads / 32;
constexpr int kCap = 512;  // candidates staged in shared memory per cell

// Positions are stored relative to the corner of their cell (edge h = L/nc), so
// the displacement to a candidate in neighbour cell c_i + dc is (o_i - o_j) -
// dc*h, accurate in FP32 for any box size.
//
// One CTA per cell.  The candidates of the 27 neighbour cells are staged once
// in shared memory (positions in the frame of the CTA's cell), then each warp
// takes one of the cell's particles at a time:
//   1. lanes test 32 candidates at a time for r < rc and compact the hits
//      into a per-warp buffer (ballot + popc);
//   2. every 32 hits, lanes evaluate the 32 pair functions F, G and unit
//      vectors (all lanes busy);
//   3. lanes as (pair, right-hand side) apply the batch to the forces:
//      u_i[r] += F f_j[r] + G rhat (rhat . f_j[r]).
// Sums over one batch run in FP32, across batches in compensated FP32 (TwoSum,
// PairSum).  No block barrier after the staging.  More than kCap candidates (very dense cells)
// take a second path that reads candidates straight from global memory.
// 64 registers, 16 blocks (32 warps) per SM (measured faster than the
// unconstrained 80 registers).
__device__ __forceinline__ void realspace_body(const RealArgs<float> &A, int cell) {
    const int nc = A.nc;
    const int *__restrict__ cell_off = A.cell_off;
    const int *__restrict__ cell_perm = A.cell_perm;
    const float4 *__restrict__ cpos = reinterpret_cast<const float4 *>(A.cpos);
    const float *__restrict__ F = A.F;
    float *__restrict__ W = A.W;
    const int R = A.R, with_self = A.with_self;
    const float L = A.cf.L, h = A.cf.h, rc2 = A.cf.rc2, self_c = A.cf.self_c;
    __shared__ int nb_beg[27], nb_pre[28], nnb;
    __shared__ float nb_shift[27][3];
    // a staged candidate: position in the CTA cell's frame and particle id in
    // one 16-byte record
    struct __align__(16) Cand {
        float x, y, z;
        int j;
    };
    __shared__ Cand cand[kCap];
    constexpr int kU = 2;  // candidates tested per lane per iteration
    __shared__ int hits[kWarps][32 + 32 * kU];  // up to 31 carried + 32 kU new
    // one record per buffered pair: unit vector and F in one 16-byte vector,
    // then G and the start of the partner's force row (aligned as that vector)
    struct PairRec {
        float4 rf;  // (rhat_x, rhat_y, rhat_z, F)
        const float *frow;
        float gfac;
    };
    __shared__ PairRec prec[kWarps][32];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int C = 3 * R;
    // neighbour table: lane k of warp 0 takes neighbour cell k (27 of them, or
    // the cell alone when nc < 3), candidate offsets by a warp scan
    if (warp == 0) {
        const int ccx = cell % nc, ccy = (cell / nc) % nc, ccz = cell / (nc * nc);
        const int nk = nc >= 3 ? 27 : 1;
        int cnt = 0;
        if (lane < nk) {
            const int dx = nk == 1 ? 0 : lane % 3 - 1, dy = nk == 1 ? 0 : (lane / 3) % 3 - 1,
                      dz = nk == 1 ? 0 : lane / 9 - 1;
            auto wrap = [nc](int v) { return v < 0 ? v + nc : (v >= nc ? v - nc : v); };
            const int c2 = (wrap(ccz + dz) * nc + wrap(ccy + dy)) * nc + wrap(ccx + dx);
            const int b = __ldg(cell_off + c2);
            cnt = __ldg(cell_off + c2 + 1) - b;
            nb_beg[lane] = b;
            nb_shift[lane][0] = dx * h;
            nb_shift[lane][1] = dy * h;
            nb_shift[lane][2] = dz * h;
        }
        int inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane < nk) nb_pre[lane] = inc - cnt;
        if (lane == nk - 1) {
            nb_pre[nk] = inc;
            nnb = nk;
        }
    }
    __syncthreads();
    const int ncand = nb_pre[nnb];
    const bool staged = ncand <= kCap;
    // neighbour k holding candidate q: nb_pre[k] <= q < nb_pre[k + 1]
    auto find_nb = [&](int q) {
        int lo = 0, hi = nnb;
        while (hi - lo > 1) {
            const int m = (lo + hi) >> 1;
            if (nb_pre[m] <= q) lo = m; else hi = m;
        }
        return lo;
    };
    if (staged) {
        for (int q = tid; q < ncand; q += kThreads) {
            const int k = find_nb(q);
            const int js = nb_beg[k] + (q - nb_pre[k]);
            const auto p = cpos[js];
            Cand c;
            c.x = p.x + nb_shift[k][0];
            c.y = p.y + nb_shift[k][1];
            c.z = p.z + nb_shift[k][2];
            c.j = cell_perm[js];
            cand[q] = c;
        }
    }
    __syncthreads();
    const bool single = nc < 3;
    const float invL = 1.f / L;
    const int ib0 = cell_off[cell], ie = cell_off[cell + 1];

    // candidate q -> position in this cell's frame and particle id
    auto candidate = [&](int q, float &x, float &y, float &z, int &j) {
        if (staged) {
            const Cand c = cand[q];
            x = c.x;
            y = c.y;
            z = c.z;
            j = c.j;
        } else {
            const int k = find_nb(q);
            const int js = nb_beg[k] + (q - nb_pre[k]);
            const auto p = cpos[js];
            x = p.x + nb_shift[k][0];
            y = p.y + nb_shift[k][1];
            z = p.z + nb_shift[k][2];
            j = cell_perm[js];
        }
    };

    const int RL = R >= 32 ? 32 : (R > 16 ? 32 : (R > 8 ? 16 : (R > 4 ? 8 : (R > 2 ? 4 : (R > 1 ? 2 : 1)))));
    const int PR = 32 / RL;             // pairs applied in parallel
    const int pp = lane / RL, rl = lane % RL;

    for (int i = ib0 + warp; i < ie; i += kWarps) {
        const auto pi = cpos[i];
        const int ii = cell_perm[i];
        for (int rb = 0; rb < R; rb += RL) {
            const int r = rb + rl;
            const bool rok = r < R;
            PairSum a0, a1, a2;
            int nh = 0;  // buffered hits (warp-uniform)
            // evaluate and apply `m` buffered hits; returns this lane's partial sums
            auto flush = [&](int m, float &s0, float &s1, float &s2) {
                if (lane < m) {
                    float x, y, z;
                    int j;
                    candidate(hits[warp][lane], x, y, z, j);
                    float d0 = pi.x - x, d1 = pi.y - y, d2 = pi.z - z;
                    if (single) {
                        d0 -= L * rintf(d0 * invL);
                        d1 -= L * rintf(d1 * invL);
                        d2 -= L * rintf(d2 * invL);
                    }
                    float Fv, Gv;
                    float ir;  // coincident particles (r = 0): no direction, the G term vanishes
                    real_FG_f32(d0 * d0 + d1 * d1 + d2 * d2, A.cf, Fv, Gv, ir);
                    PairRec &pq = prec[warp][lane];
                    pq.rf.x = d0 * ir;
                    pq.rf.y = d1 * ir;
                    pq.rf.z = d2 * ir;
                    pq.rf.w = Fv;
                    pq.gfac = Gv;
                    pq.frow = F + (size_t)j * C;
                }
                __syncwarp();
                s0 = s1 = s2 = 0.f;
                if (rok) {
#pragma unroll 4
                    for (int k = pp; k < m; k += PR) {
                        const PairRec &pq = prec[warp][k];
                        const auto rf = pq.rf;
                        const float *fj = pq.frow + 3 * r;
                        const float f0 = __ldg(fj), f1 = __ldg(fj + 1), f2 = __ldg(fj + 2);
                        const float rx = rf.x, ry = rf.y, rz = rf.z;
                        const float Fk = rf.w, Gd = pq.gfac * (rx * f0 + ry * f1 + rz * f2);
                        s0 += Fk * f0 + Gd * rx;
                        s1 += Fk * f1 + Gd * ry;
                        s2 += Fk * f2 + Gd * rz;
                    }
                }
                __syncwarp();
            };
            // candidate q within rc of particle i (and not i itself)
            auto test = [&](int q) {
                bool hit = false;
                if (q < ncand) {
                    float x, y, z;
                    int j;
                    candidate(q, x, y, z, j);
                    if (j != ii) {
                        float d0 = pi.x - x, d1 = pi.y - y, d2 = pi.z - z;
                        if (single) {
                            d0 -= L * rintf(d0 * invL);
                            d1 -= L * rintf(d1 * invL);
                            d2 -= L * rintf(d2 * invL);
                        }
                        hit = d0 * d0 + d1 * d1 + d2 * d2 < rc2;
                    }
                }
                return hit;
            };
            // kU candidates per lane per iteration: hits are appended in candidate
            // order and evaluated 32 at a time
            const unsigned below = (1u << lane) - 1u;
            for (int q0 = 0; q0 < ncand; q0 += 32 * kU) {
                bool hu[kU];
#pragma unroll
                for (int v = 0; v < kU; v++) hu[v] = test(q0 + 32 * v + lane);
#pragma unroll
                for (int v = 0; v < kU; v++) {
                    const unsigned mv = __ballot_sync(0xffffffffu, hu[v]);
                    if (hu[v]) hits[warp][nh + __popc(mv & below)] = q0 + 32 * v + lane;
                    nh += __popc(mv);
                }
                __syncwarp();
                while (nh >= 32) {
                    float s0, s1, s2;
                    flush(32, s0, s1, s2);
                    a0.add(s0);
                    a1.add(s1);
                    a2.add(s2);
                    // the rest (at most 32 kU - 1 entries) moves down by 32
                    const int rest = nh - 32;
                    int e[kU];
#pragma unroll
                    for (int v = 0; v < kU; v++)
                        e[v] = lane + 32 * v < rest ? hits[warp][32 + 32 * v + lane] : 0;
                    __syncwarp();
#pragma unroll
                    for (int v = 0; v < kU; v++)
                        if (lane + 32 * v < rest) hits[warp][32 * v + lane] = e[v];
                    nh = rest;
                    __syncwarp();
                }
            }
            if (nh > 0) {
                float s0, s1, s2;
                flush(nh, s0, s1, s2);
                a0.add(s0);
                a1.add(s1);
                a2.add(s2);
            }
            // sum the PR pair slots of each right-hand side
            for (int o = RL; o < 32; o <<= 1) {
                a0.add(shfl_xor(a0, o));
                a1.add(shfl_xor(a1, o));
                a2.add(shfl_xor(a2, o));
            }
            if (pp == 0 && rok) {
                const float *fi = F + (size_t)ii * C + 3 * r;
                if (with_self) {
                    a0.add(self_c * fi[0]);
                    a1.add(self_c * fi[1]);
                    a2.add(self_c * fi[2]);
                }
                float *o = W + (size_t)ii * C + 3 * r;
                o[0] = a0.value();
                o[1] = a1.value();
                o[2] = a2.value();
            }
        }
    }
}

__global__ void __launch_bounds__(kThreads, 16) k_realspace(RealArgs<float> A) {
    realspace_body(A, blockIdx.x);
}

// Many systems in one persistent launch over their cells.
__global__ void __launch_bounds__(kThreads, 16)
k_realspace_batch(const RealArgs<float> *__restrict__ sys, const int *__restrict__ prefix,
                  int nsys, int total) {
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int k = batch_find(prefix, nsys, w);
        realspace_body(sys[k], w - prefix[k]);
        __syncthreads();
    }
}

}  // namespace

double real_self_coeff(double xi, double a) {
    const double rsp = 0.56418958354775628695;
    return (1.0 - 6.0 * xi * a * rsp + 40.0 / 3.0 * xi * xi * xi * a * a * a * rsp) / a;
}

template <typename T>
RealArgs<T> real_args(int nc, const int *cell_off, const int *cell_perm, const void *cpos,
                      const T *F, int R, double L, double rc, double xi, double a, int with_self,
                      const PairTable &tab, T *W) {
    RealArgs<T> A;
    A.nc = nc;
    A.cell_off = cell_off;
    A.cell_perm = cell_perm;
    A.cpos = cpos;
    A.F = F;
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
                                    const void *cpos, const float *F, int R, double L, double rc,
                                    double xi, double a, int with_self, const PairTable &tab,
                                    float *W, cudaStream_t s) {
    const int ncell = nc * nc * nc;
    const RealArgs<float> A = real_args<float>(nc, cell_off, cell_perm, cpos, F, R, L, rc, xi, a,
                                               with_self, tab, W);
    k_realspace<<<ncell, kThreads, 0, s>>>(A);
    return cudaGetLastError();
}

template <>
cudaError_t launch_realspace_batch<float>(const RealArgs<float> *sys, const int *prefix, int nsys,
                                          int total, int, cudaStream_t s) {
    if (total <= 0) return cudaSuccess;
    auto kern = k_realspace_batch;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, 0);
    const int grid = std::max(1, std::min(total, sms * std::max(per_sm, 1)));
    kern<<<grid, kThreads, 0, s>>>(sys, prefix, nsys, total);
    return cudaGetLastError();
}

template RealArgs<float> real_args<float>(int, const int *, const int *, const void *,
                                          const float *, int, double, double, double, double, int,
                                          const PairTable &, float *);
template RealArgs<double> real_args<double>(int, const int *, const int *, const void *,
                                            const double *, int, double, double, double, double,
                                            int, const PairTable &, double *);

}  // namespace spme
