// FP32 spread of 3R force components onto the K^3 mesh, marching up z (restates
// old-version/spme_kernel.c:231-312: grid[c][ind] += P * f_c).
//
// The column gather of spread_cols.cu, with the staging shared by a block instead
// of done by every warp, and no z tiles.  Its warps each looked up, weighted and
// ranked the visits of their own two columns (35 of 57 warp instructions per
// visit) and visited a particle again in the next z tile.  Here:
//   * a block owns 8 x YB columns and marches up z over a segment of planes.  A
//     half-warp holds XW neighbouring columns of one y row, its 16 lanes up to 16 CPL
//     force components (c = c0 + lane + 16 k), and in registers a window of planes
//     (as pairs, for the two-lane FMA fma.rn.f32x2): the 8 planes of the current
//     group and the p - 1 above them;
//   * the particles whose stencil starts in a group and reaches the block are looked
//     up once per block (from the start-cell offsets of the (y, x, z) order, one
//     visit per thread, four groups at a time), and their force rows, records and
//     weights staged once, asynchronously, for all 8 warps;
//   * a warp takes the staged visits that cover one of its columns (a ballot per
//     start pair: the accumulators' indices are compile-time), each with straight-line
//     code for its planes;
//   * a finished group is transposed through shared memory and written as rows of 8
//     columns (whole 32-byte sectors), once: no zeroing, no atomics, and the order of
//     every sum is fixed (visits in slot order).
// Bounds: issue and the FMA pipe in the visit loop (31 warp instructions per visit,
// 12 of them two-lane FMAs), then the barriers between batches.  Measured against
// the column gather, p = 6: N = 1e6, K = 256: R = 16 2.78 -> 2.09 ms, R = 4 1.90 ->
// 0.97 ms; N = 2e5, K = 160, R = 16 (p = 8): 0.635 -> 0.534 ms (1.13 -> 0.72 ms); 64
// uneven systems, R = 4: 1.90 -> 1.03 ms.  Tried and dropped: groups of 4 planes (four
// blocks per SM, 32 % more instructions: 0.58 ms at K = 160), the next visit's
// operands loaded ahead (0.56), z tiles of 16 planes with the same shared staging
// (0.58).
#include <algorithm>
#include <utility>

#include "kernels.h"
#include "spread_cols.cuh"
#include "pdl.cuh"

namespace spme {

namespace {

// A visit whose stencil starts in plane pair B of the group: P/2 + 1 pairs of
// planes (the staged weights put an odd start's planes one slot later; an even
// start's last pair is zero).  f: the lane's forces times the column's w_x w_y.
template <int P, int CPL, int XW, int B, int NA, int NW>
__device__ __forceinline__ void add_visit(float2 (&acc)[XW][NA][CPL], const float (&w)[NW],
                                          const float (&f)[XW][CPL]) {
    static_assert(NW >= P + 2 && B + P / 2 + 1 <= NA, "weights and window");
#pragma unroll
    for (int x = 0; x < XW; x++) {
        float2 fd[CPL];
#pragma unroll
        for (int k = 0; k < CPL; k++) fd[k] = make_float2(f[x][k], f[x][k]);
#pragma unroll
        for (int i = 0; i < P / 2 + 1; i++) {
            const float2 wp = make_float2(w[2 * i], w[2 * i + 1]);
#pragma unroll
            for (int k = 0; k < CPL; k++) acc[x][B + i][k] = __ffma2_rn(wp, fd[k], acc[x][B + i][k]);
        }
    }
}

// Shape of a block for CPL components per lane: 8 x YB columns, marching up z.  A
// half-warp's lanes hold XW neighbouring columns, so the 8 warps cover 8 / (2 XW)
// column groups of YB rows.
constexpr int kXB = 8, kWarps = 8, kThreads = 32 * kWarps;
__host__ __device__ constexpr int march_xw(int cpl) { return cpl <= 2 ? 2 : 1; }
__host__ __device__ constexpr int march_yb(int cpl) { return 2 * march_xw(cpl) * kWarps / kXB; }

constexpr int kVisits = kThreads;  // visits looked up together (one per thread)
constexpr int kChunk = 4;          // groups looked up together
constexpr int kG = 8;              // planes accumulated and retired together (a group)
constexpr int kBatch = 64;         // visits staged together

// A block's shared memory: start-column runs, looked-up visits ordered by group,
// one batch's weights, two batches' force rows and records, and the transpose
// buffer of a retired group.
template <int P, int CPL>
struct MarchShared {
    static constexpr int XW = march_xw(CPL), YB = march_yb(CPL);
    static constexpr int NQ = (kXB + P - 1) * (YB + P - 1);
    static constexpr int WR = (P + 2 + 3) / 4 * 4;  // staged z weights (whole 16 bytes)
    static constexpr int LR = 16 * cols_pcpl(CPL);  // a staged force row (values)
    static constexpr int RP = (3 * P + 3) / 4;  // 16-byte pieces of a record
    static constexpr int RS = RP * 4;
    // the window of a group in registers: plane pairs of its kG planes and of the
    // P - 1 after them
    static constexpr int NB = kG / 2;  // start pairs in a group
    static constexpr int NA = NB + P / 2;
    // component stride of the transpose buffer: the two half-warps' stores of one
    // plane fall on different banks
    static constexpr int ROW = kG * YB * kXB + 2;
    __align__(16) float rows[2][kBatch][LR];
    __align__(16) float rec[kBatch][RS];
    __align__(16) float wz[kBatch][WR];         // z weights (odd starts one slot later)
    __align__(16) float wxy[kBatch][YB * kXB];  // w_x w_y of the block's columns (0: not covered)
    __align__(16) float out[16 * CPL][ROW];
    int slot[kVisits];
    uint32_t info[kVisits];  // plane in the group, x and y offsets of the block (+ 8)
    int begA[NQ], nA[NQ], begB[NQ], pre[NQ + 1];
    int wsum[kWarps];
    int gcnt[kChunk][kWarps], gbase[kChunk + 1];
};

// One block's work: columns [8 bx, +8) x [YB by, +YB), planes [zs, ze) of z segment
// and component chunk bz (A.nzt segments of A.zseg planes per chunk).  Runs as the
// body of the single-system kernel and of the batched one.
template <int P, int CPL>
__device__ __forceinline__ void spread_march_body(const SpreadColsArgs<float> &A, int bx, int by,
                                                  int bz) {
    using Sh = MarchShared<P, CPL>;
    constexpr int XW = Sh::XW, YB = Sh::YB, WR = Sh::WR, LR = Sh::LR, ROW = Sh::ROW;
    constexpr int NA = Sh::NA, NB = Sh::NB;
    constexpr int PC = cols_pcpl(CPL);  // padded components per lane in a force row
    constexpr int CC = 16 * CPL;        // components per block
    extern __shared__ __align__(16) unsigned char sp_raw[];
    Sh &st = *reinterpret_cast<Sh *>(sp_raw);
    const int C = A.C, RW = A.RW, K = A.K, WS = A.ws;
    const int *__restrict__ soff = A.soff;
    const float *__restrict__ rec_w = A.rec_w;
    const float *__restrict__ Fs = A.Fs;

    const int x0 = bx * kXB, y0 = by * YB;
    const int nx = min(kXB, K - x0), ny = min(YB, K - y0);
    const int chunk = bz / A.nzt;
    const int zs = bz % A.nzt * A.zseg, ze = min(zs + A.zseg, K);
    const int cb = chunk * CC;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int half = lane >> 4, l16 = lane & 15;
    // the warp's columns: [wc, wc + 2 XW) of row wy
    constexpr int WPR = kXB / (2 * XW);
    const int wc = 2 * XW * (warp % WPR), wy = warp / WPR;

    float2 acc[XW][NA][CPL];
#pragma unroll
    for (int x = 0; x < XW; x++)
#pragma unroll
        for (int i = 0; i < NA; i++)
#pragma unroll
            for (int k = 0; k < CPL; k++) acc[x][i][k] = make_float2(0.f, 0.f);

    // the retired group at planes [pz, pz + kG), waiting in st.out to be written
    int pz = -1;
    const size_t K3 = (size_t)K * K * K;
    const int nc = min(CC, C - cb);
    // every thread, after a barrier: rows of 8 columns (whole 32-byte sectors in
    // FP32); a thread keeps one column (pair) slot and walks the components
    auto write_out = [&]() {
        float *base = A.mesh + (size_t)cb * K3 + ((size_t)pz * K + y0) * K + x0;
        const float *tsm = &st.out[0][0];
        const int zn = min(kG, ze - pz);
        pz = -1;
        if ((K & 1) == 0) {
            // even K: pairs of columns (8-byte loads and stores; ROW is even)
            constexpr int SL = kG * YB * kXB / 2, CS = kThreads >= SL ? kThreads / SL : 1;
            static_assert(kThreads % SL == 0 || SL % kThreads == 0, "row split");
            for (int q = tid % SL; q < SL; q += kThreads) {
                const int x = 2 * (q % (kXB / 2)), zy = q / (kXB / 2), y = zy % YB, z = zy / YB;
                if (z >= zn || y >= ny || x >= nx) continue;  // K, x0 + x even: x + 1 < nx
                float2 *dst = reinterpret_cast<float2 *>(base + ((size_t)z * K + y) * K + x);
                const float2 *src = reinterpret_cast<const float2 *>(tsm) + q;
#pragma unroll 4
                for (int c = tid / SL; c < nc; c += CS)
                    dst[(size_t)c * (K3 / 2)] = src[(size_t)c * (ROW / 2)];
            }
            return;
        }
        constexpr int SL = kG * YB * kXB, CS = kThreads >= SL ? kThreads / SL : 1;
        static_assert(kThreads % SL == 0 || SL % kThreads == 0, "row split");
        for (int q = tid % SL; q < SL; q += kThreads) {
            const int x = q % kXB, zy = q / kXB, y = zy % YB, z = zy / YB;
            if (z >= zn || y >= ny || x >= nx) continue;
            float *dst = base + ((size_t)z * K + y) * K + x;
            const float *src = tsm + q;
            for (int c = tid / SL; c < nc; c += CS) dst[(size_t)c * K3] = src[(size_t)c * ROW];
        }
    };
    // the group at zg is complete: its planes go to st.out (unless they lie below the
    // segment), the window moves up by kG planes
    auto retire = [&](int zg) {
        if (zg >= zs) {
            if (pz >= 0) {
                __syncthreads();
                write_out();
                __syncthreads();
            }
            float *tsm = &st.out[0][0];
#pragma unroll
            for (int z = 0; z < kG; z++)
#pragma unroll
                for (int k = 0; k < CPL; k++)
#pragma unroll
                    for (int x = 0; x < XW; x++) {
                        const float2 a = acc[x][z >> 1][k];
                        tsm[(l16 + 16 * k) * ROW + (z * YB + wy) * kXB + wc + XW * half + x] =
                            (z & 1) ? a.y : a.x;
                    }
            pz = zg;
        }
#pragma unroll
        for (int x = 0; x < XW; x++)
#pragma unroll
            for (int k = 0; k < CPL; k++) {
#pragma unroll
                for (int i = 0; i < NA; i++)
                    acc[x][i][k] = i + NB < NA ? acc[x][i + NB < NA ? i + NB : 0][k]
                                               : make_float2(0.f, 0.f);
            }
    };

    const int nsx = nx + P - 1, nq = nsx * (ny + P - 1);
    static_assert(Sh::NQ <= kThreads, "one start column per thread");
    // start planes from zs - (P - 1), in chunks of kChunk groups (fewer where a chunk
    // has more visits than are looked up together)
    constexpr int kBelow = (P - 1 + kG - 1) / kG * kG;
    for (int zc = zs - kBelow, np; zc < ze; zc += np) {
        // start columns that reach the block, one per thread: z runs of start cells,
        // part A [max(lo, 0), hi) and part B [lo + K, K) when lo < 0
        int M;
        for (np = kG * kChunk;; np /= 2) {
            const int lo = max(zc, zs - (P - 1)), hi = max(0, min(zc + np, ze));
            const int hiB = min(0, zc + np);
            int cnt = 0;
            if (tid < nq) {
                const int ty = tid / nsx, tx = tid - ty * nsx;
                const int sy = pmod(y0 - (P - 1) + ty, K), sx = pmod(x0 - (P - 1) + tx, K);
                const size_t base = ((size_t)sy * K + sx) * K;
                const int bA = __ldg(soff + base + max(lo, 0));
                const int eA = __ldg(soff + base + hi);
                int bB = 0, eB = 0;
                if (lo < 0) {
                    bB = __ldg(soff + base + lo + K);
                    eB = __ldg(soff + base + hiB + K);
                }
                st.begA[tid] = bA;
                st.nA[tid] = eA - bA;
                st.begB[tid] = bB;
                cnt = (eA - bA) + (eB - bB);
            }
            int inc = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += t;
            }
            if (lane == 31) st.wsum[warp] = inc;
            __syncthreads();
            int before = 0;
            M = 0;
#pragma unroll
            for (int w = 0; w < kWarps; w++) {
                const int v = st.wsum[w];
                before += w < warp ? v : 0;
                M += v;
            }
            if (tid < nq) st.pre[tid] = before + inc - cnt;
            if (tid == 0) st.pre[nq] = M;
            __syncthreads();
            if (M <= kVisits || np == kG) break;
        }
        const int ng = np / kG;  // groups of this chunk

        for (int vb = 0; vb == 0 || vb < M; vb += kVisits) {
            const int nv = min(kVisits, M - vb);
            // look up one visit per thread: its start column by binary search, its
            // slot, its group and its offsets from the block
            int s = 0, grp = -1;
            uint32_t info = 0;
            if (tid < nv) {
                const int v = vb + tid;
                int a = 0, b = nq;  // pre[a] <= v < pre[b]
                while (b - a > 1) {
                    const int m = (a + b) >> 1;
                    if (st.pre[m] <= v) a = m; else b = m;
                }
                const int r = v - st.pre[a];
                const bool partB = r >= st.nA[a];
                s = partB ? st.begB[a] + (r - st.nA[a]) : st.begA[a] + r;
                int sx, sy, sz;
                unpack_start(__ldg(A.rec_start + s), sx, sy, sz);
                int rx = x0 - sx, ry = y0 - sy;  // in [-(XB-1), P-1] after wrapping
                rx += rx > P - 1 ? -K : (rx < -(kXB - 1) ? K : 0);
                ry += ry > P - 1 ? -K : (ry < -(YB - 1) ? K : 0);
                const int dz = sz - (partB ? K : 0) - zc;
                grp = dz / kG;
                info = (uint32_t)(dz % kG) | (uint32_t)(rx + 8) << 8 | (uint32_t)(ry + 8) << 16;
            }
            // order by group, stable in the visit order (the same on every run)
            int rank = 0;
#pragma unroll
            for (int g = 0; g < kChunk; g++) {
                const unsigned m = __ballot_sync(0xffffffffu, grp == g);
                if (grp == g) rank = __popc(m & ((1u << lane) - 1u));
                if (lane == 0) st.gcnt[g][warp] = __popc(m);
            }
            __syncthreads();
            if (warp == 0) {
                int c = (&st.gcnt[0][0])[lane];  // kChunk x kWarps = 32 entries
                static_assert(kChunk * kWarps == 32, "one entry per lane");
                int inc = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += t;
                }
                (&st.gcnt[0][0])[lane] = inc - c;
                if (lane % kWarps == 0) st.gbase[lane / kWarps] = inc - c;
                if (lane == 31) st.gbase[kChunk] = inc;
            }
            __syncthreads();
            if (grp >= 0) {
                const int pos = st.gcnt[grp][warp] + rank;
                st.slot[pos] = s;
                st.info[pos] = info;
            }
            __syncthreads();
            // visits [b, b + n) asynchronously: force rows into buffer buf, records
            auto fetch = [&](int b, int n, int buf) {
                const int *slot = st.slot + b;
                if constexpr (CPL > 1) {
                    constexpr int VW = 4, NCH = LR / VW;
                    for (int t = tid; t < n * NCH; t += kThreads) {
                        const int v = t / NCH, q = t - v * NCH;
                        cp_async16(&st.rows[buf][v][q * VW],
                                   Fs + (size_t)slot[v] * RW + (size_t)chunk * LR + q * VW);
                    }
                } else {
                    constexpr int VW = 4;
                    if (C % VW == 0) {  // rows of whole 16-byte pieces
                        constexpr int NCH = 16 / VW;
                        for (int t = tid; t < n * NCH; t += kThreads) {
                            const int v = t / NCH, q = t - v * NCH;
                            if (q * VW < C)
                                cp_async16(&st.rows[buf][v][q * VW],
                                           Fs + (size_t)slot[v] * RW + q * VW);
                        }
                    } else {
                        for (int t = tid; t < n * 16; t += kThreads) {
                            const int v = t >> 4, c = t & 15;
                            if (c < C)
                                cp_async_small<4>(&st.rows[buf][v][c],
                                                  Fs + (size_t)slot[v] * RW + c);
                        }
                    }
                }
                for (int t = tid; t < n * Sh::RP; t += kThreads) {
                    const int v = t / Sh::RP, q = t - v * Sh::RP;
                    cp_async16(&st.rec[v][q * 4], rec_w + (size_t)slot[v] * WS + q * 4);
                }
            };
            // batches never cross a group
            auto batch_len = [&](int b) {
                int g = 0;
                while (g + 1 < ng && st.gbase[g + 1] <= b) g++;
                return min(kBatch, st.gbase[g + 1] - b);
            };
            const bool last = vb + kVisits >= M;
            int b = 0, n = nv > 0 ? batch_len(0) : 0, buf = 0;
            if (n > 0) fetch(0, n, 0);
            for (int g = 0; g < ng; g++) {
                const int gend = st.gbase[g + 1];
                while (b < gend) {
                    cp_async_wait_all();
                    // the batch landed for every thread; every warp is done with the last
                    __syncthreads();
                    if (pz >= 0) write_out();
                    const int nn = b + n < nv ? batch_len(b + n) : 0;
                    {
                        // weights of the batch: TV threads per visit
                        constexpr int TV = kThreads / kBatch;
                        const int j = tid / TV, i = tid % TV;
                        if (j < n) {
                            const uint32_t in = st.info[b + j];
                            const int dz = (int)(in & 255u), rx = (int)(in >> 8 & 255u) - 8,
                                      ry = (int)(in >> 16 & 255u) - 8;
                            const float *rec = st.rec[j];
                            const int shift = dz & 1;
#pragma unroll
                            for (int q = i; q < WR; q += TV) {
                                const int w = q - shift;
                                st.wz[j][q] = w >= 0 && w < P ? rec[2 * P + w] : 0.f;
                            }
                            float wyv[YB];
#pragma unroll
                            for (int y = 0; y < YB; y++) {
                                const int oy = ry + y;
                                wyv[y] = oy >= 0 && oy < P ? rec[P + oy] : 0.f;
                            }
#pragma unroll
                            for (int c = i; c < kXB; c += TV) {
                                const int ox = rx + c;
                                const float wx = ox >= 0 && ox < P ? rec[ox] : 0.f;
#pragma unroll
                                for (int y = 0; y < YB; y++) st.wxy[j][y * kXB + c] = wx * wyv[y];
                            }
                        }
                    }
                    __syncthreads();
                    if (nn > 0) fetch(b + n, nn, buf ^ 1);  // (the records are consumed)
                    // a lane looks at visits lane, lane + 32, ...: the warp takes those that
                    // cover one of its columns, one start position in the group after the
                    // other
                    constexpr int NV = kBatch / 32;
                    int bk[NV];
#pragma unroll
                    for (int v = 0; v < NV; v++) {
                        bk[v] = -1;
                        if (lane + 32 * v < n) {
                            const uint32_t in = st.info[b + lane + 32 * v];
                            const int ox = (int)(in >> 8 & 255u) - 8 + wc,
                                      oy = (int)(in >> 16 & 255u) - 8 + wy;
                            if (ox + 2 * XW - 1 >= 0 && ox < P && oy >= 0 && oy < P)
                                bk[v] = (int)(in & 255u) >> 1;
                        }
                    }
                    const float *rows = &st.rows[buf][0][0];
                    const float *wxy = &st.wxy[0][0] + wy * kXB + wc + XW * half;
                    static_for<NB>([&](auto bc) {
                        constexpr int B = decltype(bc)::value;
#pragma unroll
                        for (int v = 0; v < NV; v++) {
                            unsigned m = __ballot_sync(0xffffffffu, bk[v] == B);
                            while (m) {
                                const int j = 32 * v + __ffs(m) - 1;
                                m &= m - 1;
                                float f[XW][CPL], w[WR];
                                if constexpr (CPL > 1) {
                                    float fv[PC];
                                    load_vec<PC>(rows + j * LR + l16 * PC, fv);
#pragma unroll
                                    for (int x = 0; x < XW; x++) {
                                        const float c = wxy[j * (YB * kXB) + x];
#pragma unroll
                                        for (int k = 0; k < CPL; k++) f[x][k] = fv[k] * c;
                                    }
                                } else {
                                    // (lanes without a component read stale values they never
                                    // write out)
                                    const float fv = rows[j * LR + l16];
#pragma unroll
                                    for (int x = 0; x < XW; x++)
                                        f[x][0] = fv * wxy[j * (YB * kXB) + x];
                                }
                                load_vec<WR>(&st.wz[j][0], w);
                                add_visit<P, CPL, XW, B, NA, WR>(acc, w, f);
                            }
                        }
                    });
                    b += n;
                    n = nn;
                    buf ^= 1;
                }
                if (last) retire(zc + g * kG);
            }
            __syncthreads();  // the looked-up visits are replaced
            if (pz >= 0) {
                write_out();
                __syncthreads();
            }
        }
    }
}

// Blocks per SM: one component per lane 4 (64 registers), two 2 (128: two columns
// of two components per lane), three 3 (80; shared memory too).
__host__ __device__ constexpr int march_minb(int cpl) { return cpl == 1 ? 4 : cpl == 2 ? 2 : 3; }

template <int P, int CPL>
__global__ void __launch_bounds__(kThreads, march_minb(CPL))
k_spread_march(SpreadColsArgs<float> A) {
    pdl_wait();
    spread_march_body<P, CPL>(A, blockIdx.x, blockIdx.y, blockIdx.z);
}

// Many systems in one persistent launch: work item w (a block of one system)
// -> system k with prefix[k] <= w < prefix[k + 1]; the order p of each system
// selects the body.
template <int CPL>
__global__ void __launch_bounds__(kThreads, march_minb(CPL))
k_spread_march_batch(const SpreadColsSys<float> *__restrict__ sys, const int *__restrict__ prefix,
                     int nsys, int total) {
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int k = batch_find(prefix, nsys, w);
        const SpreadColsSys<float> S = sys[k];
        const int local = w - prefix[k];
        const int bx = local % S.gx, rest = local / S.gx;
        const int by = rest % S.gy, bz = rest / S.gy;
        switch (S.p) {
            case 4: spread_march_body<4, CPL>(S.args, bx, by, bz); break;
            case 6: spread_march_body<6, CPL>(S.args, bx, by, bz); break;
            default: spread_march_body<8, CPL>(S.args, bx, by, bz); break;
        }
        __syncthreads();  // shared memory is reused by the next work item
    }
}

// Blocks of a system's spread without z segments.
long march_columns(int K, int C) {
    const int cpl = cols_cpl(C), YB = march_yb(cpl), CC = 16 * cpl;
    return (long)((K + kXB - 1) / kXB) * ((K + YB - 1) / YB) * ((C + CC - 1) / CC);
}

// Planes per z segment: the columns are cut where those of the whole launch
// (`columns`) do not fill the GPU about twice over, into segments of at least 16
// planes (a segment visits again the particles of the p - 1 planes below it:
// with 2400 columns asked for, R = 16 at K = 128 took 0.310 instead of 0.285 ms).
int march_zseg(int K, long columns) {
    int nseg = 1;
    while (columns * nseg < 800 && K / (2 * nseg) >= 16) nseg *= 2;
    return ((K + nseg - 1) / nseg + kG - 1) / kG * kG;
}

template <int P, int CPL>
cudaError_t launch_t(const SpreadColsArgs<float> &A, const SpreadColsGrid &g, cudaStream_t s) {
    constexpr size_t smem = sizeof(MarchShared<P, CPL>);
    auto kern = k_spread_march<P, CPL>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    pdl_launch(kern, dim3(g.x, g.y, g.blocks / (g.x * g.y)), kThreads, smem, s, A);
    return cudaGetLastError();
}

template <int P>
cudaError_t launch_p(const SpreadColsArgs<float> &A, const SpreadColsGrid &g, cudaStream_t s) {
    switch (cols_cpl(A.C)) {
        case 1: return launch_t<P, 1>(A, g, s);
        case 2: return launch_t<P, 2>(A, g, s);
        default: return launch_t<P, 3>(A, g, s);
    }
}

template <int CPL>
cudaError_t launch_batch(const SpreadColsSys<float> *sys, const int *prefix, int nsys, int total,
                         cudaStream_t s) {
    constexpr size_t smem = std::max(
        {sizeof(MarchShared<4, CPL>), sizeof(MarchShared<6, CPL>), sizeof(MarchShared<8, CPL>)});
    auto kern = k_spread_march_batch<CPL>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem);
    const int grid = std::max(1, std::min(total, sms * std::max(per_sm, 1)));
    kern<<<grid, kThreads, smem, s>>>(sys, prefix, nsys, total);
    return cudaGetLastError();
}

}  // namespace

SpreadColsGrid spread_march_grid(int K, int C, long columns) {
    const int cpl = cols_cpl(C), YB = march_yb(cpl), CC = 16 * cpl;
    SpreadColsGrid g;
    g.x = (K + kXB - 1) / kXB;
    g.y = (K + YB - 1) / YB;
    g.columns = march_columns(K, C);
    g.zseg = march_zseg(K, columns > 0 ? columns : g.columns);
    g.nzt = (K + g.zseg - 1) / g.zseg;
    g.blocks = g.x * g.y * g.nzt * ((C + CC - 1) / CC);
    return g;
}

cudaError_t launch_spread_march(SpreadColsArgs<float> A, int p, cudaStream_t s) {
    const SpreadColsGrid g = spread_march_grid(A.K, A.C, 0);
    A.nzt = g.nzt;
    A.zseg = g.zseg;
    switch (p) {
        case 4: return launch_p<4>(A, g, s);
        case 6: return launch_p<6>(A, g, s);
        case 8: return launch_p<8>(A, g, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_spread_march_batch(const SpreadColsSys<float> *sys, const int *prefix, int nsys,
                                      int total, int C, cudaStream_t s) {
    if (total <= 0) return cudaSuccess;
    switch (cols_cpl(C)) {
        case 1: return launch_batch<1>(sys, prefix, nsys, total, s);
        case 2: return launch_batch<2>(sys, prefix, nsys, total, s);
        default: return launch_batch<3>(sys, prefix, nsys, total, s);
    }
}

}  // namespace spme
