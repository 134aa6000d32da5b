// FP32 interpolation of the 3R mesh components back to the particles (restates
// old-version/spme_kernel.c:8-70: v_i = sum_j P_ij grid[c][ind_ij]; FP64 in
// interp_fp64.cu).
//
// One CTA per mesh tile.  For 4 components at a time it stages the tile
// plus its (p-1) upper halo in shared memory as a dense box
// [4][HZB][HYB][HX] (HX = 24 wide: every lane's x offset fits; at 16x8x4
// tiles the component-plane stride is 24 (mod 32) words, so the gather below
// is bank-conflict free):
//   * one TMA (cp.async.bulk.tensor) load per chunk, completing on an mbarrier
//     (bounded wait, error flag on timeout); for tiles whose halo wraps the
//     periodic boundary the part past K arrives as zeros and is patched with
//     16-byte asynchronous copies (all rows with such copies when TMA is unavailable).
// Each warp then interpolates the tile's own particles from shared memory:
// at p = 4, 6 two particles per warp with lanes = (x column pair,
// component) and two-lane FMAs (interp_pairs); otherwise one particle per warp
// with lanes = (x offset 0..7, component 0..3).  The x offsets are summed with
// shuffles.  Every particle is handled by exactly one CTA; a tile's halo is
// staged again by its neighbours (from L2 where it is still cached).
#include <algorithm>

#include "cp_async.cuh"
#include "kernels.h"
#include "tma.cuh"
#include "pdl.cuh"

namespace spme {

namespace {

constexpr int kThreads = 256;
// Staged row width (elements) HX: 24, or 16 for boxes copied without TMA at tiles of at most
// 8 columns (tx + 7 columns are read): the copies are what those cost.  Interpolation at
// K = 75, C = 24, p = 4, 8x8x8 tiles 0.111 -> 0.080 ms.  A TMA box stays 24 wide: dense
// 16-wide components would all start on the same banks.
constexpr int kHX = kInterpMaxRow;
__host__ __device__ constexpr bool narrow_row(bool use_tma, int tx) { return !use_tma && tx <= 8; }

constexpr int kCG = 4;  // components of a box

// A half-warp's copy of one particle record for interp_pairs: lane j of the
// half holds weights j and 16 + j (the record's 3p weights: x, y, z), plus
// the stencil start; read by shuffles within the half.
struct HalfRec {
    float wa, wb;
    uint32_t st;
};

template <int P>
__device__ __forceinline__ HalfRec load_pair_rec(const InterpArgs<float> &A, int s) {
    const int j = threadIdx.x & 15;
    const float *rw = A.rec_w + (size_t)s * A.ws;
    HalfRec r;
    r.wa = j < 3 * P ? __ldg(rw + j) : 0.f;
    r.wb = j < 3 * P - 16 ? __ldg(rw + 16 + j) : 0.f;
    r.st = __ldg(A.rec_start + s);
    return r;
}

// p = 4 or 6: two particles per warp, one per
// half-warp, lanes of a half = (x pair 0..3, component 0..3).  A lane's x pair
// starts at an even box column (the particle's first column, or the one before
// it when that is odd), is read with one 8-byte load and meets its two x
// weights (times the y weight) in one two-lane FMA (fma.rn.f32x2): each load
// and FMA instruction covers two mesh points.  Columns outside the stencil
// carry zero weights (the box is 24 columns wide: a pair ends at most at
// column tx + 6).  The next pair's records are loaded while this pair is
// interpolated; rec0 is the warp's first pair, loaded once per tile.
template <int P, int HX>
__device__ __forceinline__ void interp_pairs(const float *box, int PS, int HYB,
                                             const InterpArgs<float> &A, int c0, int nc,
                                             int pbeg, int pend, int ox, int oy, int oz,
                                             HalfRec rec0) {
    constexpr int kWarps = kThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int h = lane >> 4, xp = (lane >> 2) & 3, cl = lane & 3;
    const int C = A.C;
    HalfRec nxt = rec0;
    for (int s0 = pbeg + 2 * warp; s0 < pend; s0 += 2 * kWarps) {
        const HalfRec r = nxt;
        if (s0 + 2 * kWarps < pend) nxt = load_pair_rec<P>(A, min(s0 + 2 * kWarps + h, pend - 1));
        // weight i of this half's particle
        auto w = [&](int i) {
            return i < 16 ? __shfl_sync(0xffffffffu, r.wa, i, 16)
                          : __shfl_sync(0xffffffffu, r.wb, i - 16, 16);
        };
        const int s = s0 + h;
        int sx, sy, sz;
        unpack_start(r.st, sx, sy, sz);
        const int lx = sx - ox, ly = sy - oy, lz = sz - oz;  // own tile: no wrap
        const int odd = lx & 1;
        const int i0 = 2 * xp - odd;  // stencil column of the pair's first point
        const float x0 = __shfl_sync(0xffffffffu, r.wa, i0 & 15, 16);
        const float x1 = __shfl_sync(0xffffffffu, r.wa, i0 + 1, 16);
        const float wx0 = i0 >= 0 && i0 < P ? x0 : 0.f;
        const float wx1 = i0 + 1 < P ? x1 : 0.f;
        float2 wxy[P];
        float wz[P];
#pragma unroll
        for (int y = 0; y < P; y++) {
            const float wy = w(P + y);
            wxy[y] = make_float2(wx0 * wy, wx1 * wy);
        }
#pragma unroll
        for (int z = 0; z < P; z++) wz[z] = w(2 * P + z);
        const float *base = box + (size_t)cl * PS + (lz * HYB + ly) * HX + (lx - odd) + 2 * xp;
        float2 acc = make_float2(0.f, 0.f);
        // sum over y with w_x w_y first, then one w_z per plane
#pragma unroll
        for (int z = 0; z < P; z++) {
            const float *pz = base + z * HYB * HX;
            float2 t = make_float2(0.f, 0.f);
#pragma unroll
            for (int y = 0; y < P; y++)
                t = __ffma2_rn(wxy[y], *reinterpret_cast<const float2 *>(pz + y * HX), t);
            acc = __ffma2_rn(make_float2(wz[z], wz[z]), t, acc);
        }
        float a = acc.x + acc.y;
        a += __shfl_xor_sync(0xffffffffu, a, 4);
        a += __shfl_xor_sync(0xffffffffu, a, 8);
        if (s < pend && xp == 0 && cl < nc) {
            float *out = A.W + (size_t)__ldg(A.rec_idx + s) * C + c0 + cl;
            *out = A.accumulate ? *out + a : a;
        }
    }
}

// One tile's work (the body of the single-system kernel and of the batched
// one); tmap is read only when use_tma is set.
template <int P, int HX>
__device__ __forceinline__ void interp_body(const CUtensorMap *tmap, const InterpArgs<float> &A,
                                            int tile) {
    constexpr int VW = 4;        // values per 16-byte vector
    constexpr int NV = HX / VW;  // vectors per staged row
    const int use_tma = A.use_tma;
    const int *__restrict__ tile_off = A.tile_off;
    const int *__restrict__ rec_idx = A.rec_idx;
    const uint32_t *__restrict__ rec_start = A.rec_start;
    const float *__restrict__ rec_w = A.rec_w;
    const float *__restrict__ mesh = A.mesh;
    float *__restrict__ W = A.W;
    int *__restrict__ err = A.err;
    const MeshGeom &g = A.g;
    const int C = A.C, cb = A.cb, ce = A.ce, accumulate = A.accumulate, WS = A.ws;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    // TMA destinations must be 128-byte aligned (128 spare bytes are allocated)
    float *box = reinterpret_cast<float *>(smem_raw + ((128 - (smem_addr(smem_raw) & 127)) & 127));

    const int pbeg = tile_off[tile], pend = tile_off[tile + 1];
    if (pbeg == pend) return;
    const int K = g.K;
    const int HYB = g.ty + P - 1, HZB = g.tz + P - 1;
    // component-plane stride: 8 or 24 (mod 32) words
    const int PS = HZB * HYB * HX + (HX == 16 ? 8 : 0);
    const int tix = tile % g.ntx, tiy = (tile / g.ntx) % g.nty, tiz = tile / (g.ntx * g.nty);
    const int ox = tix * g.tx, oy = tiy * g.ty, oz = tiz * g.tz;
    const int hx = min(g.tx, K - ox) + P - 1;
    const int hy = min(g.ty, K - oy) + P - 1;
    const int hz = min(g.tz, K - oz) + P - 1;
    // TMA: the box's innermost start coordinate times the element size must be a
    // multiple of 16 bytes.  A halo that wraps the periodic boundary is loaded by
    // TMA too (the part past K arrives as zeros) and the wrapped part patched
    // with asynchronous copies.
    const bool wraps = ox + hx > K || oy + hy > K || oz + hz > K;
    const bool tma = use_tma && ((size_t)ox * sizeof(float)) % 16 == 0;
    const size_t K2 = (size_t)K * K, K3 = K2 * K;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int xs = lane >> 2, cl = lane & 3;

    if (tma && threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    __syncthreads();

    // rows [c][z][y][0..HX) of the halo region with asynchronous copies of 16, 8 or 4
    // bytes.  Through registers a thread waited for each vector: K = 75, C = 24 0.121 ms, here
    // 0.111; 64 systems of K = 24 to 100, C = 12 1.47, 1.27 ms.
    auto stage_rows = [&](int c0, int nc) {
        const bool vec = (K % VW) == 0 && (ox % VW) == 0, two = ((K | ox) & 1) == 0;
        DivMod dnv, dhy, dhz;
        dnv.init(NV);
        dhy.init(hy);
        dhz.init(hz);
        const int nrow = nc * hz * hy;
        for (int q = threadIdx.x; q < nrow * NV; q += kThreads) {
            int v, y, z;
            const int row = dnv.div(q, v);
            const int cz = dhy.div(row, y);
            const int c = dhz.div(cz, z);
            int gy = oy + y, gz = oz + z;
            gy -= gy >= K ? K : 0;
            gz -= gz >= K ? K : 0;
            const int x0 = ox + v * VW;
            const float *src = mesh + (size_t)(c0 + c) * K3 + (size_t)gz * K2 + (size_t)gy * K;
            float *dst = box + (size_t)c * PS + (z * HYB + y) * HX + v * VW;
            if (vec) {
                cp_async16(dst, src + wrap_index(x0, K));
            } else if (two) {
#pragma unroll
                for (int e = 0; e < VW; e += 2) cp_async_small<8>(dst + e, src + wrap_index(x0 + e, K));
            } else {
#pragma unroll
                for (int e = 0; e < VW; e++) cp_async_small<4>(dst + e, src + wrap_index(x0 + e, K));
            }
        }
        cp_async_wait_all();
        __syncthreads();
    };

    // p = 4, 6: two particles per warp, x columns in pairs (interp_pairs)
    constexpr bool kPairs = P == 4 || P == 6;
    // after a TMA box of a tile whose halo wraps: the elements past the periodic
    // boundary (zeros in the box) by 16-byte copies, one thread per box row: a
    // row past K in y or z is copied whole, other rows only from column K - ox on
    const int xw0 = ox + hx > K ? (K - ox) / VW : NV;  // first vector holding a wrapped column
    const int xw1 = (hx - 1) / VW;                     // last vector of the halo
    auto patch_wrapped = [&](int c0, int nc) {
        DivMod dhy, dhz;
        dhy.init(hy);
        dhz.init(hz);
        const int nrow = nc * hz * hy;
        for (int row = threadIdx.x; row < nrow; row += kThreads) {
            int y, z;
            const int cz = dhy.div(row, y);
            const int c = dhz.div(cz, z);
            int gy = oy + y, gz = oz + z;
            const bool row_wraps = gy >= K || gz >= K;
            if (!row_wraps && xw0 == NV) continue;
            gy -= gy >= K ? K : 0;
            gz -= gz >= K ? K : 0;
            const float *src = mesh + (size_t)(c0 + c) * K3 + (size_t)gz * K2 + (size_t)gy * K;
            float *dst = box + (size_t)c * PS + (z * HYB + y) * HX;
            const int v1 = row_wraps ? NV - 1 : xw1;
            for (int v = row_wraps ? 0 : xw0; v <= v1; v++) {
                const int x0 = ox + v * VW;
                cp_async16(dst + v * VW, src + wrap_index(x0, K));  // (a TMA box: K, ox % 4 == 0)
            }
        }
        cp_async_wait_all();
        __syncthreads();
    };

    // the warp's first particle's record, the same for every component chunk:
    // loaded once, before the first box is waited for
    constexpr int kWarps = kThreads / 32;
    float wreg_0 = 0.f;
    uint32_t st_0 = 0;
    int idx_0 = 0;
    HalfRec hrec_0{0.f, 0.f, 0u};
    if constexpr (kPairs) {
        if (pbeg + 2 * warp < pend)
            hrec_0 = load_pair_rec<P>(A, min(pbeg + 2 * warp + (lane >> 4), pend - 1));
    } else if (pbeg + warp < pend) {
        const int s = pbeg + warp;
        wreg_0 = lane < 3 * P ? __ldg(rec_w + (size_t)s * WS + lane) : 0.f;
        st_0 = __ldg(rec_start + s);
        idx_0 = __ldg(rec_idx + s);
    }

    int chunk = 0;
    for (int c0 = cb; c0 < ce; c0 += kCG, chunk++) {
        const int nc = min(kCG, ce - c0);
        if (tma) {
            if (threadIdx.x == 0) {
                fence_proxy_async();  // order earlier generic reads of the box before the TMA write
                mbar_expect_tx(&bar, (uint32_t)((size_t)kCG * PS * sizeof(float)));
                tma_load_4d(box, tmap, ox, oy, oz, c0, &bar);
            }
            const bool ok = mbar_wait(&bar, (uint32_t)(chunk & 1));
            if (!__syncthreads_and(ok)) {  // uniform decision: all threads give up together
                if (threadIdx.x == 0) atomicExch(err, 1);
                return;
            }
            if (wraps) patch_wrapped(c0, nc);
        } else {
            stage_rows(c0, nc);
        }
        if constexpr (kPairs) {
            interp_pairs<P, HX>(box, PS, HYB, A, c0, nc, pbeg, pend, ox, oy, oz, hrec_0);
            __syncthreads();  // the box is rewritten by the next chunk
            continue;
        }
        // the next particle's record is loaded while this one is interpolated
        float wreg_n = wreg_0;
        uint32_t st_n = st_0;
        int idx_n = idx_0;
        for (int s = pbeg + warp; s < pend; s += kWarps) {
            const float wreg = wreg_n;
            const uint32_t st = st_n;
            const int idx = idx_n;
            if (s + kWarps < pend) {
                const int sn = s + kWarps;
                wreg_n = lane < 3 * P ? __ldg(rec_w + (size_t)sn * WS + lane) : 0.f;
                st_n = __ldg(rec_start + sn);
                idx_n = __ldg(rec_idx + sn);
            }
            int sx, sy, sz;
            unpack_start(st, sx, sy, sz);
            const int lx = sx - ox, ly = sy - oy, lz = sz - oz;  // own tile: no wrap
            const float wxv = __shfl_sync(0xffffffffu, wreg, xs < P ? xs : P - 1);
            const float wx = xs < P ? wxv : 0.f;
            float wxy[P], wz[P];
#pragma unroll
            for (int y = 0; y < P; y++) wxy[y] = wx * __shfl_sync(0xffffffffu, wreg, P + y);
#pragma unroll
            for (int z = 0; z < P; z++) wz[z] = __shfl_sync(0xffffffffu, wreg, 2 * P + z);
            float acc = 0.f;
            const float *base = box + (size_t)cl * PS + (lz * HYB + ly) * HX + lx + xs;
            // sum over y with w_x w_y first, then one w_z per plane
#pragma unroll
            for (int z = 0; z < P; z++) {
                const float *pz = base + z * HYB * HX;
                float t = 0.f;
#pragma unroll
                for (int y = 0; y < P; y++) t += wxy[y] * pz[y * HX];
                acc += wz[z] * t;
            }
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (xs == 0 && cl < nc) {
                float *out = W + (size_t)idx * C + c0 + cl;
                *out = accumulate ? *out + acc : acc;
            }
        }
        __syncthreads();  // the box is rewritten by the next chunk
    }
}

template <int P, int HX>
// blocks per SM that the 4-component box's shared memory allows (16x8x4 tiles)
__global__ void __launch_bounds__(kThreads, 5)
k_interp(const __grid_constant__ CUtensorMap tmap, InterpArgs<float> A) {
    pdl_wait();
    // tiles z fastest: blocks launched together are z neighbours, whose boxes
    // share p - 1 of their tz + p - 1 planes (read from L2 by the later ones)
    const int b = blockIdx.x, ntx = A.g.ntx, nty = A.g.nty, ntz = A.g.ntz;
    const int tiz = b % ntz, rest = b / ntz;
    interp_body<P, HX>(&tmap, A, (tiz * nty + rest / ntx) * ntx + rest % ntx);
}

// Many systems in one persistent launch over their tiles: each system's boxes
// by TMA through its own descriptor in the work list where its mesh rows allow
// it, by asynchronous copies otherwise; the order p of each system selects the body
// (the batch launches one such kernel per order).
__global__ void __launch_bounds__(kThreads)
k_interp_batch(const InterpSys<float> *__restrict__ sys, const int *__restrict__ prefix, int nsys,
               int total) {
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int k = batch_find(prefix, nsys, w);
        const InterpArgs<float> A = sys[k].args;
        // the system's TMA box stays in the global work list (a descriptor in
        // global memory; never a local copy)
        const CUtensorMap *tmap = A.use_tma ? &sys[k].tmap : nullptr;
        const int tile = w - prefix[k];
        if (narrow_row(A.use_tma, A.g.tx)) {
            switch (A.g.p) {
                case 4: interp_body<4, 16>(tmap, A, tile); break;
                case 6: interp_body<6, 16>(tmap, A, tile); break;
                default: interp_body<8, 16>(tmap, A, tile); break;
            }
        } else {
            switch (A.g.p) {
                case 4: interp_body<4, kHX>(tmap, A, tile); break;
                case 6: interp_body<6, kHX>(tmap, A, tile); break;
                default: interp_body<8, kHX>(tmap, A, tile); break;
            }
        }
        __syncthreads();
    }
}

template <int P>
cudaError_t launch_p(const InterpMaps &maps, InterpArgs<float> A, cudaStream_t s) {
    const MeshGeom &g = A.g;
    const size_t smem = interp_smem_bytes(g, sizeof(float));
    auto kern = narrow_row(maps.ok4, g.tx) ? k_interp<P, 16> : k_interp<P, kHX>;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    A.ws = RecordWidth<float, P>::value;
    pdl_launch(kern, g.ntx * g.nty * g.ntz, kThreads, smem, s, maps.cg4, A);
    return cudaGetLastError();
}

bool encode_box(CUtensorMap *m, const void *mesh, int K, int C, const MeshGeom &g, size_t elem,
                int CG) {
    EncodeTiledFn fn = encode_fn();
    if (!fn || (K * elem) % 16 != 0 || ((uintptr_t)mesh % 16) != 0) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)K, (cuuint64_t)K, (cuuint64_t)K, (cuuint64_t)C};
    const cuuint64_t strides[3] = {(cuuint64_t)K * elem, (cuuint64_t)K * K * elem,
                                   (cuuint64_t)K * K * K * elem};
    const int row = elem == 8 ? interp64_row(g.tx + g.p - 1) : kHX;
    const cuuint32_t box[4] = {(cuuint32_t)row, (cuuint32_t)(g.ty + g.p - 1),
                               (cuuint32_t)(g.tz + g.p - 1), (cuuint32_t)CG};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    if (box[1] > 256 || box[2] > 256) return false;
    CUresult r = fn(m, elem == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
                    4, const_cast<void *>(mesh), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

}  // namespace

size_t interp_smem_bytes(const MeshGeom &g, size_t elem) {
    const size_t rows = (size_t)(g.tz + g.p - 1) * (g.ty + g.p - 1);
    // FP64: the box and one row sum per thread
    if (elem == 8)
        return (rows * interp64_row(g.tx + g.p - 1) + kInterp64Threads) * elem + 128;
    return 4 * rows * kHX * elem + 128;
}

bool interp_tile_ok(const MeshGeom &g, size_t elem) {
    return (size_t)4 * (g.tz + g.p - 1) * (g.ty + g.p - 1) * kHX * elem + 128 <= 220 * 1024;
}

bool make_interp_box(CUtensorMap *map, const void *mesh, int C, const MeshGeom &g, size_t elem) {
    return encode_box(map, mesh, g.K, C, g, elem, elem == 8 ? 1 : 4);
}

bool make_interp_maps(InterpMaps *maps, const void *mesh, int C, const MeshGeom &g, size_t elem) {
    maps->ok4 = encode_box(&maps->cg4, mesh, g.K, C, g, elem, elem == 8 ? 1 : 4);
    return maps->ok4;
}

template <>
cudaError_t launch_interp<float>(const InterpMaps &maps, const int *tile_off, int n, const int *rec_idx,
                                 const uint32_t *rec_start, const float *rec_w, const float *mesh,
                                 int C, int cb, int ce, const MeshGeom &g, float *W, int accumulate,
                                 int *err, cudaStream_t s) {
    if (n <= 0 || cb >= ce) return cudaSuccess;
    if (cb < 0 || ce > C) return cudaErrorInvalidValue;
    if (g.tx + 7 > kHX || g.tx + g.p - 1 > kHX) return cudaErrorInvalidValue;
    const InterpArgs<float> A{tile_off, rec_idx, rec_start, rec_w, mesh, W, err, g, C, cb, ce,
                              accumulate, maps.ok4 ? 1 : 0, 0};
    switch (g.p) {
        case 4: return launch_p<4>(maps, A, s);
        case 6: return launch_p<6>(maps, A, s);
        case 8: return launch_p<8>(maps, A, s);
        default: return cudaErrorInvalidValue;
    }
}

template <>
cudaError_t launch_interp_batch<float>(const InterpSys<float> *sys, const int *prefix, int nsys,
                                       int total, size_t smem, cudaStream_t s) {
    if (total <= 0) return cudaSuccess;
    auto kern = k_interp_batch;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem);
    const int grid = std::max(1, std::min(total, sms * std::max(per_sm, 1)));
    kern<<<grid, kThreads, smem, s>>>(sys, prefix, nsys, total);
    return cudaGetLastError();
}

}  // namespace spme
