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
//     per pair and right-hand side (geometry 6, segment offset 1, two cubic-sextic
//     Horner chains 12, application 10);
//   * the listed pairs are split evenly over the lanes (contiguous shares), which
//     accumulate in registers; a particle's partial sums, one per share it
//     touches, are added in list order: a fixed order on every run, and a few
//     additions instead of a 5-step butterfly per particle.
// N = 1e6, L = 480, rc = 10 (38 pairs per particle), one right-hand side:
// 15.19 -> 3.30 ms; N = 1e5, L = 220: 1.645 -> 0.358 ms (FP64 pipe floor 2.0 ms: 36
// FP64 warp instructions per particle at 16 cycles each).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "kernels.h"

namespace spme {

namespace {

constexpr int kThreads = 64;  // two warps per cell: ~4-5 particles each at typical densities
constexpr int kWarps = kThreads / 32;
constexpr int kCap = 512;    // candidates staged in shared memory per cell
constexpr int kList = 512;   // listed pairs per warp
constexpr int kGroup = 16;   // particles listed together (4 bits of a list entry)
constexpr int kU = 2;        // candidates tested per lane per iteration

// M_real(r) = F I + G rhat rhat: Beenakker's real-space form divided by a, and
// for r < 2a plus (overlap RPY - far-field RPY), written in the cancellation-free
// form of realspace.cu: x = xi r, S(x) = erf(x)/x and psi(x) = (erf(x) -
// 2x e^{-x^2}/sqrt(pi)) / x^3, for x < 0.5 from their Maclaurin series in x^2
// (ten terms: below 1e-17 relative; the factor 2/sqrt(pi) outside).  `near`
// selects the form; both are analytic on either side of r = 2a.
__host__ __device__ inline void real_FG(double r, double xi, double a, bool near, double &F,
                                        double &G) {
    const double rsp = 0.56418958354775628695;  // 1/sqrt(pi)
    const double x = xi * r, x2 = x * x, e = exp(-x2);
    if (near) {
        double S = 0.0, P = 0.0;
        if (x < 0.5) {
            const double ks[10] = {1.0, -1.0 / 3, 1.0 / 10, -1.0 / 42, 1.0 / 216,
                                   -1.0 / 1320, 1.0 / 9360, -1.0 / 75600,
                                   1.0 / 685440, -1.0 / 6894720};
            const double kp[10] = {2.0 / 3, -2.0 / 5, 1.0 / 7, -1.0 / 27, 1.0 / 132,
                                   -1.0 / 780, 1.0 / 5400, -1.0 / 42840,
                                   1.0 / 383040, -1.0 / 3810240};
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
            for (int k = 9; k >= 0; k--) {
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
        const double2 *c = reinterpret_cast<const double2 *>(tb.coef) + (size_t)seg * (kPairDeg + 1);
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
struct WarpSh {
    static constexpr int S = 3 * RB;
    double first[32][S], last[32][S];  // a lane's first and last partial sum
    double mid[kGroup][S];             // a particle wholly inside one lane's share
    double res[kGroup][S];
    double px[kGroup], py[kGroup], pz[kGroup];
    float4 pf[kGroup];                 // FP32 position, particle id (bits)
    uint32_t list[kList];              // particle (4 bits) | candidate
    int beg[kGroup + 1];               // first entry of each particle
};

// One cell: a warp lists the pairs of up to kGroup of its particles and sums
// them (RB right-hand sides per sweep).
template <int RB>
__device__ __forceinline__ void realspace64_body(const RealArgs<double> &A, int cell) {
    constexpr int S = 3 * RB;
    __shared__ int nb_beg[27], nb_pre[28], nnb;
    __shared__ double nb_shift[27][3];
    __shared__ float4 cf[kCap];  // staged candidates: FP32 position, particle id (bits)
    __shared__ double cx[kCap], cy[kCap], cz[kCap];
    __shared__ WarpSh<RB> wsh[kWarps];

    const int nc = A.nc, C = 3 * A.R;
    const double L = A.L, h = A.h;
    const double4_32a *__restrict__ cpos = reinterpret_cast<const double4_32a *>(A.cpos);
    const int *__restrict__ cell_perm = A.cell_perm;
    const double *__restrict__ F = A.F;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ib0 = __ldg(A.cell_off + cell), ie = __ldg(A.cell_off + cell + 1);
    if (ib0 == ie) return;  // uniform over the block
    // neighbour table: lane k of warp 0 takes neighbour cell k (27 of them, or the
    // cell alone when nc < 3), candidate offsets by a warp scan
    if (warp == 0) {
        const int ccx = cell % nc, ccy = (cell / nc) % nc, ccz = cell / (nc * nc);
        const int nk = nc >= 3 ? 27 : 1;
        int cnt = 0;
        if (lane < nk) {
            const int dx = nk == 1 ? 0 : lane % 3 - 1, dy = nk == 1 ? 0 : (lane / 3) % 3 - 1,
                      dz = nk == 1 ? 0 : lane / 9 - 1;
            auto wrap = [nc](int v) { return v < 0 ? v + nc : (v >= nc ? v - nc : v); };
            const int c2 = (wrap(ccz + dz) * nc + wrap(ccy + dy)) * nc + wrap(ccx + dx);
            const int b = __ldg(A.cell_off + c2);
            cnt = __ldg(A.cell_off + c2 + 1) - b;
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
            const double4_32a p = cpos[js];
            const double x = p.x + nb_shift[k][0], y = p.y + nb_shift[k][1],
                         z = p.z + nb_shift[k][2];
            cx[q] = x;
            cy[q] = y;
            cz[q] = z;
            cf[q] = make_float4((float)x, (float)y, (float)z, __int_as_float(cell_perm[js]));
        }
    }
    __syncthreads();
    // candidate q in the frame of this cell
    auto candidate = [&](int q, double &x, double &y, double &z, int &j) {
        if (staged) {
            x = cx[q];
            y = cy[q];
            z = cz[q];
            j = __float_as_int(cf[q].w);
        } else {
            const int k = find_nb(q);
            const int js = nb_beg[k] + (q - nb_pre[k]);
            const double4_32a p = cpos[js];
            x = p.x + nb_shift[k][0];
            y = p.y + nb_shift[k][1];
            z = p.z + nb_shift[k][2];
            j = cell_perm[js];
        }
    };
    // The FP32 test accepts a superset of the pairs within rc: coordinates lie
    // within 3 cells (one cell of edge L: within L, minimum image), so FP32
    // rounding moves d^2 by far less than the margin.
    const bool single = nc < 3;
    const float pre_r2 = (float)(A.rc2 * 1.0001 + 9e-5 * h * h);
    const float Lf = (float)L, iLf = 1.f / Lf;
    const double invL = 1.0 / L;
    const long long rc2_bits = __double_as_longlong(A.rc2);
    const unsigned below = (1u << lane) - 1u;
    WarpSh<RB> &ws = wsh[warp];

    // this warp's share of the cell's particles, kGroup at a time
    const int half = (ie - ib0 + kWarps - 1) / kWarps;
    const int wb = ib0 + warp * half, we = min(ie, wb + half);
    for (int g0 = wb; g0 < we; g0 += kGroup) {
        const int np = min(kGroup, we - g0);
        if (lane < np) {
            const double4_32a p = cpos[g0 + lane];
            ws.px[lane] = p.x;
            ws.py[lane] = p.y;
            ws.pz[lane] = p.z;
            ws.pf[lane] = make_float4((float)p.x, (float)p.y, (float)p.z,
                                      __int_as_float(cell_perm[g0 + lane]));
        }
        for (int r0 = 0; r0 < A.R; r0 += RB) {
            for (int t = lane; t < np * S; t += 32) ws.res[t / S][t % S] = 0.0;
            if (lane == 0) ws.beg[0] = 0;
            __syncwarp();
            float4 me = ws.pf[0];
            int il = 0, q0 = 0, nh = 0, ilo = 0;
            while (true) {
                // list pairs (particle, candidate) while a test's hits are sure to fit
                while (il < np && nh <= kList - 32 * kU) {
                    bool hit[kU];
#pragma unroll
                    for (int v = 0; v < kU; v++) {
                        const int q = q0 + 32 * v + lane;
                        hit[v] = false;
                        if (q < ncand) {
                            float4 c;
                            if (staged) {
                                c = cf[q];
                            } else {
                                double x, y, z;
                                int j;
                                candidate(q, x, y, z, j);
                                c = make_float4((float)x, (float)y, (float)z, __int_as_float(j));
                            }
                            float e0 = me.x - c.x, e1 = me.y - c.y, e2 = me.z - c.z;
                            if (single) {
                                e0 -= Lf * rintf(e0 * iLf);
                                e1 -= Lf * rintf(e1 * iLf);
                                e2 -= Lf * rintf(e2 * iLf);
                            }
                            hit[v] = e0 * e0 + e1 * e1 + e2 * e2 < pre_r2 &&
                                     __float_as_int(c.w) != __float_as_int(me.w);
                        }
                    }
#pragma unroll
                    for (int v = 0; v < kU; v++) {
                        const unsigned m = __ballot_sync(0xffffffffu, hit[v]);
                        if (hit[v])
                            ws.list[nh + __popc(m & below)] =
                                (uint32_t)(q0 + 32 * v + lane) | ((uint32_t)il << 28);
                        nh += __popc(m);
                    }
                    q0 += 32 * kU;
                    if (q0 >= ncand) {
                        q0 = 0;
                        il++;
                        if (il < np) me = ws.pf[il];
                        if (lane == 0) ws.beg[il] = nh;
                    }
                }
                if (il < np && lane == 0) ws.beg[il + 1] = nh;  // cut: this list's part ends here
                __syncwarp();
                // sum the listed pairs: lane's share [lane c, lane c + c)
                const int c = (nh + 31) >> 5;
                double acc[S];
#pragma unroll
                for (int k = 0; k < S; k++) acc[k] = 0.0;
                int cur = -1, nseg = 0;
                const int e1 = min(nh, lane * c + c);
                for (int t = lane * c; t < e1; t++) {
                    const uint32_t ent = ws.list[t];
                    const int ip = (int)(ent >> 28);
                    if (ip != cur) {
                        if (cur >= 0) {
                            double *dst = nseg == 0 ? ws.first[lane] : ws.mid[cur];
#pragma unroll
                            for (int k = 0; k < S; k++) dst[k] = acc[k];
                            nseg++;
#pragma unroll
                            for (int k = 0; k < S; k++) acc[k] = 0.0;
                        }
                        cur = ip;
                    }
                    double x, y, z;
                    int j;
                    candidate((int)(ent & 0x0fffffffu), x, y, z, j);
                    double d0 = ws.px[ip] - x, d1 = ws.py[ip] - y, d2 = ws.pz[ip] - z;
                    if (single) {
                        d0 -= L * rint(d0 * invL);
                        d1 -= L * rint(d1 * invL);
                        d2 -= L * rint(d2 * invL);
                    }
                    const double s = fma(d2, d2, fma(d1, d1, d0 * d0));
                    if (__double_as_longlong(s) < rc2_bits) {
                        double Av, Bv;
                        pair_AB(A.tab, s, A.xi, A.a, Av, Bv);
                        const double *fj = F + (size_t)j * C + 3 * r0;
#pragma unroll
                        for (int r = 0; r < RB; r++) {
                            if (RB == 1 || r0 + r < A.R) {
                                const double f0 = __ldg(fj + 3 * r), f1 = __ldg(fj + 3 * r + 1),
                                             f2 = __ldg(fj + 3 * r + 2);
                                const double g = Bv * fma(d2, f2, fma(d1, f1, d0 * f0));
                                acc[3 * r] = fma(g, d0, fma(Av, f0, acc[3 * r]));
                                acc[3 * r + 1] = fma(g, d1, fma(Av, f1, acc[3 * r + 1]));
                                acc[3 * r + 2] = fma(g, d2, fma(Av, f2, acc[3 * r + 2]));
                            }
                        }
                    }
                }
                if (cur >= 0) {
                    double *dst = nseg == 0 ? ws.first[lane] : ws.last[lane];
#pragma unroll
                    for (int k = 0; k < S; k++) dst[k] = acc[k];
                }
                __syncwarp();
                // a particle's partial sums in share order: a share's first partial sum
                // when the particle's entries reach its start, its last when they reach
                // its end, else the one in between
                const int npl = min(il, np - 1) - ilo + 1;
                for (int t = lane; t < npl * S; t += 32) {
                    const int ip = ilo + t / S, k = t % S;
                    const int b = ws.beg[ip], e = ws.beg[ip + 1];
                    if (e <= b) continue;
                    double sum = ws.res[ip][k];
                    for (int l = b / c; l * c < e; l++) {
                        const double v = b <= l * c ? ws.first[l][k]
                                                    : (e >= min(nh, l * c + c) ? ws.last[l][k]
                                                                               : ws.mid[ip][k]);
                        sum += v;
                    }
                    ws.res[ip][k] = sum;
                }
                __syncwarp();
                if (il >= np) break;
                nh = 0;
                ilo = il;
                if (lane == 0) ws.beg[il] = 0;
            }
            for (int t = lane; t < np * S; t += 32) {
                const int ip = t / S, k = t % S;
                if (r0 + k / 3 < A.R) {
                    const size_t at = (size_t)__float_as_int(ws.pf[ip].w) * C + 3 * r0 + k;
                    const double v = ws.res[ip][k];
                    A.W[at] = A.with_self ? fma(A.self_c, F[at], v) : v;
                }
            }
            __syncwarp();
        }
    }
}

template <int RB>
__global__ void __launch_bounds__(kThreads, RB == 1 ? 7 : 4) k_realspace64(RealArgs<double> A) {
    realspace64_body<RB>(A, blockIdx.x);
}

// Many systems in one persistent launch over their cells.
template <int RB>
__global__ void __launch_bounds__(kThreads, RB == 1 ? 7 : 4)
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
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, 0);
    const int grid = std::max(1, std::min(total, sms * std::max(per_sm, 1)));
    kern<<<grid, kThreads, 0, s>>>(sys, prefix, nsys, total);
    return cudaGetLastError();
}

}  // namespace

template <>
cudaError_t launch_realspace<double>(int nc, const int *cell_off, const int *cell_perm,
                                     const void *cpos, const double *F, int R, double L,
                                     double rc, double xi, double a, int with_self,
                                     const PairTable &tab, double *W, cudaStream_t s) {
    if (R <= 0) return cudaSuccess;
    const RealArgs<double> A = real_args<double>(nc, cell_off, cell_perm, cpos, F, R, L, rc, xi,
                                                 a, with_self, tab, W);
    const int ncell = nc * nc * nc;
    switch (sweep_width(R)) {
        case 1: k_realspace64<1><<<ncell, kThreads, 0, s>>>(A); break;
        case 2: k_realspace64<2><<<ncell, kThreads, 0, s>>>(A); break;
        case 3: k_realspace64<3><<<ncell, kThreads, 0, s>>>(A); break;
        default: k_realspace64<4><<<ncell, kThreads, 0, s>>>(A); break;
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

// Polynomials (degree kPairDeg, in the offset from the segment's centre) of
// A = F and B = G / s on [s0, s0 + h], interleaved, through the values at the
// Chebyshev nodes.
void fit_segment(double s0, double h, double xi, double a, bool near, double *out) {
    constexpr int n = kPairDeg + 1;
    double f[2][n], c[2][n];
    for (int j = 0; j < n; j++) {
        const double s = s0 + 0.5 * h * (std::cos(M_PI * (j + 0.5) / n) + 1.0);
        real_FG(std::sqrt(s), xi, a, near, f[0][j], f[1][j]);
        f[1][j] /= s;
    }
    for (int w = 0; w < 2; w++) {
        for (int k = 0; k < n; k++) {
            double q = 0.0;
            for (int j = 0; j < n; j++) q += f[w][j] * std::cos(M_PI * k * (j + 0.5) / n);
            c[w][k] = (k ? 2.0 : 1.0) * q / n;
        }
        // Chebyshev to powers of t, then of the offset v = t h / 2
        double t0[n] = {1.0}, t1[n] = {0.0, 1.0}, o[n];
        for (int i = 0; i < n; i++) o[i] = c[w][0] * t0[i] + c[w][1] * t1[i];
        for (int k = 2; k < n; k++) {
            double t2[n];
            for (int i = 0; i < n; i++) t2[i] = (i ? 2.0 * t1[i - 1] : 0.0) - t0[i];
            for (int i = 0; i < n; i++) {
                o[i] += c[w][k] * t2[i];
                t0[i] = t1[i];
                t1[i] = t2[i];
            }
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
    for (int m = 6; m <= 10; m++) {  // 2^m segments per octave of s
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
            const int g = base + q - (near ? 0 : 1);
            const double s0 = start_of(g), h = start_of(g + 1) - s0;
            double *c = coef->data() + (size_t)q * (kPairDeg + 1) * 2;
            fit_segment(s0, h, xi, a, near, c);
            // the fit between the nodes, relative to the function scale there
            for (int p = 0; p <= 16 && ok; p++) {
                const double s = s0 + h * p / 16.0, v = s - (s0 + 0.5 * h);
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
