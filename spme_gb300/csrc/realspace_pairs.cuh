// Cell candidates, pair listing and the few-right-hand-sides pair sum shared by the
// FP64 (realspace_fp64.cu) and FP32 (realspace.cu) real-space kernels.
#pragma once

#include "kernels.h"

namespace spme {
namespace {

constexpr int kRsThreads = 64;  // two warps per cell: ~4-5 particles each at typical densities
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kCap = 512;    // candidates staged in shared memory per cell
constexpr int kGroup = 16;   // particles listed together (4 bits of a list entry)
constexpr int kU = 2;        // candidates tested per lane per iteration

template <typename G> struct Geo4;
template <> struct Geo4<float> { using type = float4; };
template <> struct Geo4<double> { using type = double4_32a; };

__device__ __forceinline__ float d_rint(float x) { return rintf(x); }
__device__ __forceinline__ double d_rint(double x) { return rint(x); }

// The candidates of one cell (the particles of its 27 neighbour cells, or of the
// single cell when nc < 3), in the frame of that cell: FP32 position and particle
// id, and for FP64 engines the FP64 position too.
template <typename G>
struct CellShared {
    static constexpr bool kDbl = sizeof(G) == 8;
    float4 cf[kCap];
    G cx[kDbl ? kCap : 1], cy[kDbl ? kCap : 1], cz[kDbl ? kCap : 1];
    G nb_shift[27][3];
    int nb_beg[27], nb_pre[28], nnb;
};

template <typename G>
struct Cell {
    using V4 = typename Geo4<G>::type;
    CellShared<G> &sh;
    const V4 *__restrict__ cpos;
    const int *__restrict__ perm;
    int ncand;
    bool staged, single;
    G L, invL;
    float Lf, iLf, pre_r2;

    // neighbour k holding candidate q: nb_pre[k] <= q < nb_pre[k + 1]
    __device__ __forceinline__ int find_nb(int q) const {
        int lo = 0, hi = sh.nnb;
        while (hi - lo > 1) {
            const int m = (lo + hi) >> 1;
            if (sh.nb_pre[m] <= q) lo = m; else hi = m;
        }
        return lo;
    }
    // candidate q from global memory (cells with more than kCap candidates)
    __device__ __forceinline__ void fetch(int q, G &x, G &y, G &z, int &j) const {
        const int k = find_nb(q);
        const int js = sh.nb_beg[k] + (q - sh.nb_pre[k]);
        const V4 p = cpos[js];
        x = p.x + sh.nb_shift[k][0];
        y = p.y + sh.nb_shift[k][1];
        z = p.z + sh.nb_shift[k][2];
        j = perm[js];
    }
    __device__ __forceinline__ void candidate(int q, G &x, G &y, G &z, int &j) const {
        if (!staged) {
            fetch(q, x, y, z, j);
            return;
        }
        const float4 c = sh.cf[q];
        j = __float_as_int(c.w);
        if constexpr (sizeof(G) == 8) {
            x = sh.cx[q];
            y = sh.cy[q];
            z = sh.cz[q];
        } else {
            x = c.x;
            y = c.y;
            z = c.z;
        }
    }

    // every thread of the block; ends with a barrier
    __device__ __forceinline__ Cell(CellShared<G> &s, int cell, int nc, const int *cell_off,
                                    const int *cell_perm, const void *pos, G L_, G h, G rc2)
        : sh(s), cpos(reinterpret_cast<const V4 *>(pos)), perm(cell_perm), L(L_) {
        const int tid = threadIdx.x, lane = tid & 31;
        // neighbour table: lane k of warp 0 takes neighbour cell k, candidate offsets by
        // a warp scan
        if (tid < 32) {
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
                sh.nb_beg[lane] = b;
                sh.nb_shift[lane][0] = dx * h;
                sh.nb_shift[lane][1] = dy * h;
                sh.nb_shift[lane][2] = dz * h;
            }
            int inc = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += t;
            }
            if (lane < nk) sh.nb_pre[lane] = inc - cnt;
            if (lane == nk - 1) {
                sh.nb_pre[nk] = inc;
                sh.nnb = nk;
            }
        }
        __syncthreads();
        ncand = sh.nb_pre[sh.nnb];
        staged = ncand <= kCap;
        if (staged) {
            for (int q = tid; q < ncand; q += kRsThreads) {
                G x, y, z;
                int j;
                fetch(q, x, y, z, j);
                if constexpr (sizeof(G) == 8) {
                    sh.cx[q] = x;
                    sh.cy[q] = y;
                    sh.cz[q] = z;
                }
                sh.cf[q] = make_float4((float)x, (float)y, (float)z, __int_as_float(j));
            }
        }
        __syncthreads();
        single = nc < 3;
        invL = G(1) / L;
        Lf = (float)L;
        iLf = 1.f / Lf;
        // FP64: the FP32 test accepts a superset of the pairs within rc (coordinates lie
        // within 3 cells, or within L of the single cell, so FP32 rounding moves d^2 by
        // far less than the margin); FP32: the test itself
        pre_r2 = sizeof(G) == 8 ? (float)(rc2 * G(1.0001) + G(9e-5) * h * h) : (float)rc2;
    }

    __device__ __forceinline__ void min_image(G &d0, G &d1, G &d2) const {
        if (single) {
            d0 -= L * d_rint(d0 * invL);
            d1 -= L * d_rint(d1 * invL);
            d2 -= L * d_rint(d2 * invL);
        }
    }
};

// Lists pairs (particle il << 28 | candidate) of a warp's particles pf[0 .. np)
// (FP32 position, id) into list, resumable: stops when the hits of one more test
// might not fit, or when all are listed.  beg[i]: first entry of particle i in
// this list, beg[i + 1] its end.  PAD: each particle's entries are filled up to a
// multiple of pad with entries that name no candidate (q = kNoCand).
constexpr uint32_t kNoCand = 0x0fffffffu;
struct ListState {
    int il = 0, q0 = 0;  // next particle and candidate to test
};
template <bool PAD, int LIST, bool FAST, typename G>
__device__ __forceinline__ int list_pairs_t(const Cell<G> &cell, const float4 *pf, int np,
                                            uint32_t *list, int *beg, ListState &s, int pad) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int ncand = cell.ncand, room = LIST - 32 * kU - (PAD ? pad : 0);
    int nh = 0;
    if (lane == 0) beg[s.il] = 0;
    float4 me = pf[s.il];
    while (s.il < np && nh <= room) {
        bool hit[kU];
#pragma unroll
        for (int v = 0; v < kU; v++) {
            const int q = s.q0 + 32 * v + lane;
            hit[v] = false;
            if (q < ncand) {
                float4 c;
                if (FAST || cell.staged) {
                    c = cell.sh.cf[q];
                } else {
                    G x, y, z;
                    int j;
                    cell.fetch(q, x, y, z, j);
                    c = make_float4((float)x, (float)y, (float)z, __int_as_float(j));
                }
                float e0 = me.x - c.x, e1 = me.y - c.y, e2 = me.z - c.z;
                if (!FAST && cell.single) {
                    e0 -= cell.Lf * rintf(e0 * cell.iLf);
                    e1 -= cell.Lf * rintf(e1 * cell.iLf);
                    e2 -= cell.Lf * rintf(e2 * cell.iLf);
                }
                hit[v] = e0 * e0 + e1 * e1 + e2 * e2 < cell.pre_r2 &&
                         __float_as_int(c.w) != __float_as_int(me.w);
            }
        }
#pragma unroll
        for (int v = 0; v < kU; v++) {
            const unsigned m = __ballot_sync(0xffffffffu, hit[v]);
            if (hit[v])
                list[nh + __popc(m & below)] =
                    (uint32_t)(s.q0 + 32 * v + lane) | ((uint32_t)s.il << 28);
            nh += __popc(m);
        }
        s.q0 += 32 * kU;
        if (s.q0 >= ncand || nh > room) {
            if (PAD) {
                const int full = (nh + pad - 1) / pad * pad;
                if (lane < full - nh) list[nh + lane] = kNoCand | ((uint32_t)s.il << 28);
                nh = full;
            }
            if (lane == 0) beg[s.il + 1] = nh;
            if (s.q0 >= ncand) {
                s.q0 = 0;
                s.il++;
                if (s.il < np) me = pf[s.il];
            }
        }
    }
    __syncwarp();
    return nh;
}

// (the usual cell, staged and without minimum images, in a loop of its own)
template <bool PAD, int LIST, typename G>
__device__ __forceinline__ int list_pairs(const Cell<G> &cell, const float4 *pf, int np,
                                          uint32_t *list, int *beg, ListState &s, int pad) {
    if (cell.staged && !cell.single)
        return list_pairs_t<PAD, LIST, true>(cell, pf, np, list, beg, s, pad);
    return list_pairs_t<PAD, LIST, false>(cell, pf, np, list, beg, s, pad);
}

// Sum of partial sums: FP64 plain; FP32 with Knuth's TwoSum error term carried
// alongside.
template <typename T>
struct PairSum {
    T s = T(0);
    __device__ __forceinline__ void add(T x) { s += x; }
    __device__ __forceinline__ void join(PairSum o) { s += o.s; }
    __device__ __forceinline__ T value() const { return s; }
};
template <>
struct PairSum<float> {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float t = s + x, bp = t - s;
        c += (s - (t - bp)) + (x - bp);
        s = t;
    }
    __device__ __forceinline__ void join(PairSum o) {
        add(o.s);
        c += o.c;
    }
    __device__ __forceinline__ float value() const { return s + c; }
};
__device__ __forceinline__ PairSum<float> shfl_xor(PairSum<float> a, int w) {
    a.s = __shfl_xor_sync(0xffffffffu, a.s, w);
    a.c = __shfl_xor_sync(0xffffffffu, a.c, w);
    return a;
}

// The sum over a lane's pairs of one particle, RB right-hand sides: component k = 3 r + d.
// FP64: plain.  FP32: component pairs as two-lane operations, moved to compensated
// sums every kRun pairs (RB = 1: each pair).
template <typename T, int RB>
struct ShareSum {
    T acc[3 * RB] = {};
    // row: the partner's force row, from right-hand side r0 on, of which nr are left
    __device__ __forceinline__ void pair(T A, T B, const T (&d)[3], const T *__restrict__ row, int nr) {
#pragma unroll
        for (int r = 0; r < RB; r++) {
            if (RB == 1 || r < nr) {
                const T f0 = __ldg(row + 3 * r), f1 = __ldg(row + 3 * r + 1), f2 = __ldg(row + 3 * r + 2);
                const T g = B * fma(d[2], f2, fma(d[1], f1, d[0] * f0));
                acc[3 * r] = fma(g, d[0], fma(A, f0, acc[3 * r]));
                acc[3 * r + 1] = fma(g, d[1], fma(A, f1, acc[3 * r + 1]));
                acc[3 * r + 2] = fma(g, d[2], fma(A, f2, acc[3 * r + 2]));
            }
        }
    }
    __device__ __forceinline__ void step(int) {}
    __device__ __forceinline__ void finish() {}
    __device__ __forceinline__ PairSum<T> get(int k) const { return PairSum<T>{acc[k]}; }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < 3 * RB; k++) acc[k] = T(0);
    }
};
template <int RB>
struct ShareSum<float, RB> {
    static constexpr int H = (3 * RB + 1) / 2, kRun = RB;
    float2 run[H] = {}, s[H] = {}, c[H] = {};
    static __device__ __forceinline__ float2 sub(float2 a, float2 b) {
        return __ffma2_rn(make_float2(-1.f, -1.f), b, a);
    }
    __device__ __forceinline__ void pair(float A, float B, const float (&d)[3], const float *row) {
        float g[RB];
#pragma unroll
        for (int r = 0; r < RB; r++)
            g[r] = B * fmaf(d[2], row[3 * r + 2], fmaf(d[1], row[3 * r + 1], d[0] * row[3 * r]));
#pragma unroll
        for (int m = 0; m < H; m++) {
            constexpr int last = 3 * RB - 1;  // (odd 3 RB: the second lane again, unused)
            const int k = 2 * m, l = 2 * m + 1 <= last ? 2 * m + 1 : last;
            const float2 t = __ffma2_rn(make_float2(g[k / 3], g[l / 3]),
                                        make_float2(d[k % 3], d[l % 3]),
                                        __fmul2_rn(make_float2(A, A), make_float2(row[k], row[l])));
            run[m] = kRun == 1 ? t : __fadd2_rn(run[m], t);
        }
        if (kRun == 1) fold();
    }
    // TwoSum of run into (s, c)
    __device__ __forceinline__ void fold() {
#pragma unroll
        for (int m = 0; m < H; m++) {
            const float2 t = __fadd2_rn(s[m], run[m]), bp = sub(t, s[m]);
            c[m] = __fadd2_rn(c[m], __fadd2_rn(sub(s[m], sub(t, bp)), sub(run[m], bp)));
            s[m] = t;
            run[m] = make_float2(0.f, 0.f);
        }
    }
    // after the lane's pair i
    __device__ __forceinline__ void step(int i) {
        if (kRun > 1 && i % kRun == kRun - 1) fold();
    }
    __device__ __forceinline__ void finish() {
        if (kRun > 1) fold();
    }
    __device__ __forceinline__ PairSum<float> get(int k) const {
        PairSum<float> v;
        v.s = k & 1 ? s[k / 2].y : s[k / 2].x;
        v.c = k & 1 ? c[k / 2].y : c[k / 2].x;
        return v;
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int m = 0; m < H; m++) s[m] = c[m] = make_float2(0.f, 0.f);
    }
};

constexpr int kList = 512;  // listed pairs per warp (few right-hand sides)

template <typename T, int RB>
struct FewShared {
    static constexpr int S = 3 * RB;
    PairSum<T> first[32][S], last[32][S];  // a lane's first and last partial sum
    PairSum<T> res[kGroup][S];
    T px[kGroup], py[kGroup], pz[kGroup];
    float4 pf[kGroup];            // FP32 position, particle id (bits)
    uint32_t list[kList];
    int beg[kGroup + 2];
};

// One cell, RB right-hand sides per sweep: a warp lists the pairs of up to kGroup
// of its particles; the list is split evenly over the lanes (contiguous shares),
// which evaluate (pair_AB: A = F, B = G / r^2 at s = r^2) and accumulate in
// registers; a particle's partial sums, one per share it touches, are added in
// list order: the same order on every run, a few additions instead of a butterfly
// per particle.  FP32 sums are compensated all the way (ShareSum).
template <typename T, int RB, typename AB>
__device__ __forceinline__ void realspace_few_body(const RealArgs<T> &A, int cell, T L, T h, T rc2,
                                                   T self_c, AB pair_AB) {
    constexpr int S = 3 * RB;
    __shared__ CellShared<T> csh;
    __shared__ FewShared<T, RB> wsh[kRsWarps];
    const int ib0 = __ldg(A.cell_off + cell), ie = __ldg(A.cell_off + cell + 1);
    if (ib0 == ie) return;  // uniform over the block
    const Cell<T> cl(csh, cell, A.nc, A.cell_off, A.cell_perm, A.cpos, L, h, rc2);
    const int C = 3 * A.R;
    const T *__restrict__ F = A.F;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    FewShared<T, RB> &ws = wsh[warp];

    // this warp's share of the cell's particles, kGroup at a time
    const int half = (ie - ib0 + kRsWarps - 1) / kRsWarps;
    const int wb = ib0 + warp * half, we = min(ie, wb + half);
    for (int g0 = wb; g0 < we; g0 += kGroup) {
        const int np = min(kGroup, we - g0);
        if (lane < np) {
            const auto p = cl.cpos[g0 + lane];
            ws.px[lane] = p.x;
            ws.py[lane] = p.y;
            ws.pz[lane] = p.z;
            ws.pf[lane] = make_float4((float)p.x, (float)p.y, (float)p.z,
                                      __int_as_float(A.cell_perm[g0 + lane]));
        }
        for (int r0 = 0; r0 < A.R; r0 += RB) {
            for (int t = lane; t < np * S; t += 32) ws.res[t / S][t % S] = PairSum<T>();
            __syncwarp();
            ListState ls;
            while (ls.il < np) {
                const int ilo = ls.il;
                const int nh = list_pairs<false, kList>(cl, ws.pf, np, ws.list, ws.beg, ls, 0);
                // sum the listed pairs: lane's share [lane c, lane c + c)
                const int c = (nh + 31) >> 5;
                ShareSum<T, RB> acc;
                // the sum of particle cur, whose entries in the share end here: the lane's
                // first or last partial sum, or all of the particle's in this list
                int cur = -1, nseg = 0;
                auto put = [&](bool at_end) {
                    acc.finish();
                    if (nseg == 0 || at_end) {
                        PairSum<T> *dst = nseg == 0 ? ws.first[lane] : ws.last[lane];
#pragma unroll
                        for (int k = 0; k < S; k++) dst[k] = acc.get(k);
                    } else {
#pragma unroll
                        for (int k = 0; k < S; k++) ws.res[cur][k].join(acc.get(k));
                    }
                    acc.clear();
                    nseg++;
                };
                const int e1 = min(nh, lane * c + c);
                for (int t = lane * c; t < e1; t++) {
                    const uint32_t ent = ws.list[t];
                    const int ip = (int)(ent >> 28);
                    if (ip != cur) {
                        if (cur >= 0) put(false);
                        cur = ip;
                    }
                    T x, y, z;
                    int j;
                    cl.candidate((int)(ent & 0x0fffffffu), x, y, z, j);
                    T d[3] = {ws.px[ip] - x, ws.py[ip] - y, ws.pz[ip] - z};
                    cl.min_image(d[0], d[1], d[2]);
                    const T s = fma(d[2], d[2], fma(d[1], d[1], d[0] * d[0]));
                    T Av, Bv;
                    if constexpr (sizeof(T) == 4) {
                        // (one sweep of all RB = R) the padded row as 16-byte vectors
                        constexpr int SV = (S + 3) / 4 * 4;
                        T row[SV];
                        const float4 *f4 =
                            reinterpret_cast<const float4 *>(A.F2) + (size_t)j * (SV / 4);
#pragma unroll
                        for (int q = 0; q < SV / 4; q++) {
                            const float4 v = __ldg(f4 + q);
                            row[4 * q] = v.x;
                            row[4 * q + 1] = v.y;
                            row[4 * q + 2] = v.z;
                            row[4 * q + 3] = v.w;
                        }
                        pair_AB(s, Av, Bv);
                        acc.pair(Av, Bv, d, row);
                    } else if (pair_AB(s, Av, Bv)) {
                        acc.pair(Av, Bv, d, F + (size_t)j * C + 3 * r0, A.R - r0);
                    }
                    acc.step(t - lane * c);
                }
                if (cur >= 0) put(true);
                __syncwarp();
                // a particle's partial sums in share order: a share's first partial sum
                // when the particle's entries reach its start, its last when they reach
                // its end (entries that reach neither are in res)
                const int npl = min(ls.il, np - 1) - ilo + 1;
                for (int t = lane; t < npl * S; t += 32) {
                    const int ip = ilo + t / S, k = t % S;
                    // (the particle after the last finished one is listed only when the
                    // list was cut inside it)
                    if (ip == ls.il && ls.q0 == 0) continue;
                    const int b = ws.beg[ip], e = ws.beg[ip + 1];
                    if (e <= b) continue;
                    if (b % c && e < min(nh, b / c * c + c)) continue;
                    PairSum<T> sum = ws.res[ip][k];
                    for (int l = b / c; l * c < e; l++)
                        sum.join(b <= l * c ? ws.first[l][k] : ws.last[l][k]);
                    ws.res[ip][k] = sum;
                }
                __syncwarp();
            }
            for (int t = lane; t < np * S; t += 32) {
                const int ip = t / S, k = t % S;
                if (r0 + k / 3 < A.R) {
                    const size_t at = (size_t)__float_as_int(ws.pf[ip].w) * C + 3 * r0 + k;
                    PairSum<T> v = ws.res[ip][k];
                    if (A.with_self) v.add(self_c * F[at]);
                    A.W[at] = v.value();
                }
            }
            __syncwarp();
        }
    }
}

}  // namespace
}  // namespace spme
