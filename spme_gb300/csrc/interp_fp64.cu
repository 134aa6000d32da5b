// FP64 interpolation of the 3R mesh components back to the particles (restates
// old-version/spme_kernel.c:8-70; FP32 in interp.cu).
//
// What bounds it: the FP64 pipe (16 cycles of the SM's pipe per warp
// instruction), so idle lanes and reductions are what costs.  One CTA per mesh
// tile and component stages the tile plus its (p - 1) upper halo with a TMA box,
// and a lane takes one (particle, y row of its stencil): p planes of p points,
// the x sum kept in a register, one multiply by w_z per plane, and the p rows of
// a particle are added from shared memory: 43 FP64 instructions per lane and
// 8.3 warp instructions per particle at p = 6 (6.75 is the minimum), no
// shuffles.  Box rows are 2 (mod 4) doubles long, so the p rows of a particle
// start on different banks.  One component per CTA (19 KB boxes, eleven CTAs
// per SM at 8x8x8 tiles) hides the box loads: with the three components of a
// right-hand side per CTA and the right-hand sides in sequence, N = 3e4, K = 90,
// p = 8, R = 5 took 1.19 ms.
// N = 1e6, K = 256, p = 6, one right-hand side, 8x8x8 tiles: 3.54 -> 1.50 ms;
// N = 1e5, K = 128: 0.395 -> 0.168 ms; K = 90, p = 8, R = 5: 0.897 -> 0.561 ms.
#include <algorithm>

#include "cp_async.cuh"
#include "kernels.h"
#include "tma.cuh"
#include "pdl.cuh"

namespace spme {

namespace {

constexpr int kThreads = kInterp64Threads;
constexpr int kWarps = kThreads / 32;

// One tile's work (the body of the single-system kernel and of the batched
// one); tmap is read only when use_tma is set.
template <int P>
__device__ __forceinline__ void interp64_body(const CUtensorMap *tmap,
                                              const InterpArgs<double> &A, int tile, int comp) {
    constexpr int kUnits = kThreads / P * P;  // (particle, row) pairs per round
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bar;
    // TMA destinations must be 128-byte aligned (128 spare bytes are allocated)
    double *box =
        reinterpret_cast<double *>(smem_raw + ((128 - (smem_addr(smem_raw) & 127)) & 127));
    const MeshGeom &g = A.g;
    const int pbeg = A.tile_off[tile], pend = A.tile_off[tile + 1];
    if (pbeg == pend) return;
    const int K = g.K;
    const int HX = interp64_row(g.tx + P - 1), HY = g.ty + P - 1, HZ = g.tz + P - 1;
    const int PS = HZ * HY * HX;  // box size
    double *part = box + PS;  // [kThreads] row sums
    const int ox = tile % g.ntx * g.tx, oy = tile / g.ntx % g.nty * g.ty,
              oz = tile / (g.ntx * g.nty) * g.tz;
    const int hx = min(g.tx, K - ox) + P - 1, hy = min(g.ty, K - oy) + P - 1,
              hz = min(g.tz, K - oz) + P - 1;
    // TMA: the box's innermost start coordinate must be 16-byte aligned (an even
    // ox).  A halo that wraps the periodic boundary arrives as zeros and is patched.
    const bool wraps = ox + hx > K || oy + hy > K || oz + hz > K;
    const bool tma = A.use_tma && (ox & 1) == 0;
    const size_t K2 = (size_t)K * K;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tma && tid == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    __syncthreads();

    // rows of the halo region with asynchronous copies, a warp per row: all of it, or only
    // what lies past the periodic boundary.  Loads through registers waited for each row:
    // the N = 300, K = 32 step took 111 us with them, 108 without.
    const double *mesh = A.mesh + (size_t)comp * K2 * K;
    auto stage_rows = [&](bool only_wrapped) {
        for (int row = warp; row < hz * hy; row += kWarps) {
            const int y = row % hy, z = row / hy;
            const int gy = oy + y, gz = oz + z;
            if (lane < hx && (!only_wrapped || gy >= K || gz >= K || ox + lane >= K))
                cp_async_small<8>(box + (z * HY + y) * HX + lane,
                                  mesh + (size_t)wrap_index(gz, K) * K2 +
                                      (size_t)wrap_index(gy, K) * K + wrap_index(ox + lane, K));
        }
        cp_async_wait_all();
        __syncthreads();
    };

    if (tma) {
        if (tid == 0) {
            fence_proxy_async();  // order earlier generic reads of the box before the TMA write
            mbar_expect_tx(&bar, (uint32_t)((size_t)PS * sizeof(double)));
            tma_load_4d(box, tmap, ox, oy, oz, comp, &bar);
        }
        const bool ok = mbar_wait(&bar, 0);
        if (!__syncthreads_and(ok)) {  // uniform decision: all threads give up together
            if (tid == 0) atomicExch(A.err, 1);
            return;
        }
        if (wraps) stage_rows(true);
    } else {
        stage_rows(false);
    }
    for (int p0 = pbeg; p0 < pend; p0 += kUnits / P) {
        const int np = min(kUnits / P, pend - p0);
        if (tid < np * P) {
            const int s = p0 + tid / P, y = tid % P;
            const double *rw = A.rec_w + (size_t)s * A.ws;
            int sx, sy, sz;
            unpack_start(__ldg(A.rec_start + s), sx, sy, sz);
            double wx[P], wz[P];
#pragma unroll
            for (int j = 0; j < P; j++) {
                wx[j] = __ldg(rw + j);
                wz[j] = __ldg(rw + 2 * P + j);
            }
            const double *base = box + ((sz - oz) * HY + (sy - oy) + y) * HX + (sx - ox);
            double acc = 0.0;
#pragma unroll
            for (int z = 0; z < P; z++) {
                const double *m = base + z * HY * HX;
                double t = wx[0] * m[0];
#pragma unroll
                for (int x = 1; x < P; x++) t = fma(wx[x], m[x], t);
                acc = fma(wz[z], t, acc);
            }
            part[tid] = __ldg(rw + P + y) * acc;
        }
        __syncthreads();
        if (tid < np) {
            double v = part[tid * P];
#pragma unroll
            for (int y = 1; y < P; y++) v += part[tid * P + y];
            double *out = A.W + (size_t)__ldg(A.rec_idx + p0 + tid) * A.C + comp;
            *out = A.accumulate ? *out + v : v;
        }
        __syncthreads();  // part is rewritten
    }
}

template <int P>
__global__ void __launch_bounds__(kThreads)
k_interp64(const __grid_constant__ CUtensorMap tmap, InterpArgs<double> A) {
    pdl_wait();
    // tiles z fastest, as in the FP32 kernel: z neighbours share halo planes
    const int b = blockIdx.x, ntx = A.g.ntx, nty = A.g.nty, ntz = A.g.ntz;
    const int tiz = b % ntz, rest = b / ntz;
    interp64_body<P>(&tmap, A, (tiz * nty + rest / ntx) * ntx + rest % ntx,
                      A.cb + blockIdx.y);
}

// Many systems in one persistent launch over their tiles.
__global__ void __launch_bounds__(kThreads)
k_interp64_batch(const InterpSys<double> *__restrict__ sys, const int *__restrict__ prefix,
                 int nsys, int total) {
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        const int k = batch_find(prefix, nsys, w);
        const InterpArgs<double> A = sys[k].args;
        const CUtensorMap *tmap = A.use_tma ? &sys[k].tmap : nullptr;
        const int tile = w - prefix[k];
        for (int c = A.cb; c < A.ce; c++) {
            switch (A.g.p) {
                case 4: interp64_body<4>(tmap, A, tile, c); break;
                case 6: interp64_body<6>(tmap, A, tile, c); break;
                default: interp64_body<8>(tmap, A, tile, c); break;
            }
            __syncthreads();
        }
    }
}

template <int P>
cudaError_t launch_p(const CUtensorMap &map, const InterpArgs<double> &A, cudaStream_t s) {
    const size_t smem = interp_smem_bytes(A.g, sizeof(double));
    auto kern = k_interp64<P>;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    pdl_launch(kern, dim3(A.g.ntx * A.g.nty * A.g.ntz, A.ce - A.cb), kThreads, smem, s, map, A);
    return cudaGetLastError();
}

}  // namespace

template <>
cudaError_t launch_interp<double>(const InterpMaps &maps, const int *tile_off, int n,
                                  const int *rec_idx, const uint32_t *rec_start,
                                  const double *rec_w, const double *mesh, int C, int cb, int ce,
                                  const MeshGeom &g, double *W, int accumulate, int *err,
                                  cudaStream_t s) {
    if (n <= 0 || cb >= ce) return cudaSuccess;
    if (cb < 0 || ce > C) return cudaErrorInvalidValue;
    if (g.tx + 7 > kInterpMaxRow) return cudaErrorInvalidValue;
    InterpArgs<double> A{tile_off, rec_idx, rec_start, rec_w, mesh, W, err, g, C, cb, ce,
                         accumulate, maps.ok4 ? 1 : 0, 0};
    switch (g.p) {
        case 4: A.ws = RecordWidth<double, 4>::value; return launch_p<4>(maps.cg4, A, s);
        case 6: A.ws = RecordWidth<double, 6>::value; return launch_p<6>(maps.cg4, A, s);
        case 8: A.ws = RecordWidth<double, 8>::value; return launch_p<8>(maps.cg4, A, s);
        default: return cudaErrorInvalidValue;
    }
}

template <>
cudaError_t launch_interp_batch<double>(const InterpSys<double> *sys, const int *prefix, int nsys,
                                        int total, size_t smem, cudaStream_t s) {
    if (total <= 0) return cudaSuccess;
    auto kern = k_interp64_batch;
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
