// Spread of few force components onto the K^3 mesh through per-tile boxes
// (restates old-version/spme_kernel.c:231-312: grid[c][ind] += P * f_c).
//
// With few components (C = 3 for one right-hand side) there is too little to put
// across the lanes of a warp per mesh column, and in FP64 an idle lane costs as
// much as a busy one (16 cycles of the SM's FP64 pipe per warp instruction).
// Here the lanes hold the p^3 stencil points of one particle instead:
//   * a warp owns one mesh tile and one component: the tile and its upper p - 1
//     halo are a box in shared memory (no other warp writes it, the points of one
//     particle are distinct: no atomics, a fixed order), and the warp adds its
//     tile's particles one after the other, 32 stencil points per instruction;
//   * the p^2 products w_y w_z and the p products w_x f are formed once per
//     particle (two warp multiplies at p = 6) and read back from shared memory, so
//     a point costs one FMA: 9 FP64 warp instructions per particle and component
//     at p = 6 (6.75 is the minimum);
//   * boxes are written to a scratch array, and a second kernel adds the up to
//     (1 + (p - 1) / t)^3 boxes that cover a mesh point, in tile order: every mesh
//     point is written once (no clearing), the result is the same on every run.
// Bounds: FP64 the FP64 pipe (0.55 ms per component at N = 1e6, p = 6), then the
// boxes' traffic and additions ((13/8)^3 = 4.3 meshes with 8x8x8 tiles, 0.26 ms
// per component); FP32 shared-memory wavefronts.  C = 3, p = 6, 8x8x8 tiles: FP64
// N = 1e6, K = 256: 8.97 (column gather) -> 2.43 ms; N = 1e5, K = 128: 0.938 ->
// 0.285 ms; FP32 N = 1e5: 0.145 (tile kernel) -> 0.119 ms.
#include <algorithm>
#include <vector>

#include "kernels.h"
#include "pdl.cuh"

namespace spme {

namespace {

// Box edges of a tile (the last tiles of an axis use a part of theirs).
struct BoxDim {
    int x, y, z, vol;
};
__host__ __device__ inline BoxDim box_dim(const MeshGeom &g) {
    BoxDim b;
    b.x = g.tx + g.p - 1;
    b.y = g.ty + g.p - 1;
    b.z = g.tz + g.p - 1;
    b.vol = b.x * b.y * b.z;
    return b;
}

// One warp per (tile, component c0 + blockIdx.y); box of component slot
// blockIdx.y of tile t at boxes[(blockIdx.y ntiles + t) vol].
template <typename T, int P>
__global__ void __launch_bounds__(32)
k_spread_box(const int *__restrict__ tile_off, const int *__restrict__ rec_idx,
             const uint32_t *__restrict__ rec_start, const T *__restrict__ rec_w,
             const T *__restrict__ F, int C, int c0, MeshGeom g, T *__restrict__ boxes) {
    pdl_wait();
    constexpr int WS = RecordWidth<T, P>::value;
    constexpr int NP3 = P * P * P, NJ = (NP3 + 31) / 32;
    constexpr int NPR = P * P + P;  // products: w_y w_z (p^2), then w_x f (p)
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ T prod[2][NPR];
    T *box = reinterpret_cast<T *>(smem_raw);
    const int tile = blockIdx.x, lane = threadIdx.x;
    const int pbeg = __ldg(tile_off + tile), pend = __ldg(tile_off + tile + 1);
    const BoxDim b = box_dim(g);
    const int ox = tile % g.ntx * g.tx, oy = tile / g.ntx % g.nty * g.ty,
              oz = tile / (g.ntx * g.nty) * g.tz;
    // this lane's stencil points k = lane + 32 j: offset in the box, index of
    // w_y w_z; the x index repeats with period PX in j (32 j mod p)
    constexpr int PX = P == 6 ? 3 : 1;
    int off[NJ], pyz[NJ], px[PX];
#pragma unroll
    for (int j = 0; j < NJ; j++) {
        const int k = lane + 32 * j, yz = k / P;
        off[j] = (yz / P * b.y + yz % P) * b.x + k % P;
        pyz[j] = min(yz, P * P - 1);
        if (j < PX) px[j] = P * P + k % P;
    }
    // ... and its products: lane m forms a w_z with a = w_y (m < p^2), or w_x f
    constexpr int NM = (NPR + 31) / 32;
    int ma[NM], mb[NM];
#pragma unroll
    for (int q = 0; q < NM; q++) {
        const int m = lane + 32 * q;
        ma[q] = m < P * P ? P + m % P : min(m - P * P, P - 1);
        mb[q] = m < P * P ? 2 * P + m / P : -1;
    }
    for (int i = lane; i < b.vol; i += 32) box[i] = T(0);

    // the next particle's record and force are loaded while this one is added
    // (records staged 16 at a time in shared memory: no faster in FP32, 0.60 vs
    // 0.55 ms in FP64 at N = 1e6, where they cost two warps per SM)
    const T *__restrict__ Fc = F + c0 + blockIdx.y;
    T w_n = T(0), f_n = T(0);
    uint32_t st_n = 0;
    int id_n = 0;
    if (pbeg < pend) {
        w_n = lane < 3 * P ? __ldg(rec_w + (size_t)pbeg * WS + lane) : T(0);
        st_n = __ldg(rec_start + pbeg);
        f_n = __ldg(Fc + (size_t)__ldg(rec_idx + pbeg) * C);
        if (pbeg + 1 < pend) id_n = __ldg(rec_idx + pbeg + 1);
    }
    for (int s = pbeg; s < pend; s++) {
        const T w = w_n, f = f_n;
        const uint32_t st = st_n;
        if (s + 1 < pend) {
            w_n = lane < 3 * P ? __ldg(rec_w + (size_t)(s + 1) * WS + lane) : T(0);
            st_n = __ldg(rec_start + s + 1);
            f_n = __ldg(Fc + (size_t)id_n * C);
            if (s + 2 < pend) id_n = __ldg(rec_idx + s + 2);
        }
        T *pr = prod[s & 1];
#pragma unroll
        for (int q = 0; q < NM; q++) {
            const T a = __shfl_sync(0xffffffffu, w, ma[q]);
            const T wz = __shfl_sync(0xffffffffu, w, mb[q] < 0 ? 0 : mb[q]);
            if (lane + 32 * q < NPR) pr[lane + 32 * q] = a * (mb[q] < 0 ? f : wz);
        }
        __syncwarp();  // products visible; the previous particle's points are written
        int sx, sy, sz;
        unpack_start(st, sx, sy, sz);
        T *bp = box + ((sz - oz) * b.y + (sy - oy)) * b.x + (sx - ox);
        T v[NJ], gx[PX];
#pragma unroll
        for (int j = 0; j < PX; j++) gx[j] = pr[px[j]];
#pragma unroll
        for (int j = 0; j < NJ; j++)
            if (NP3 % 32 == 0 || lane + 32 * j < NP3) v[j] = bp[off[j]];
#pragma unroll
        for (int j = 0; j < NJ; j++)
            if (NP3 % 32 == 0 || lane + 32 * j < NP3)
                bp[off[j]] = v[j] + gx[j % PX] * pr[pyz[j]];
    }
    __syncwarp();
    T *out = boxes + ((size_t)blockIdx.y * gridDim.x + tile) * b.vol;
    for (int i = lane; i < b.vol; i += 32) out[i] = box[i];
}

// mesh[c0 + c][z][y][x] = the sum of the boxes covering (z, y, x).  tab: for each
// axis (x, y, z) and coordinate the up to four tiles covering it, as offsets
// into a component's boxes that add up over the axes (-1: none).  MX, MY, MZ:
// the most tiles covering a coordinate, 2 (tiles that divide K and are at least
// p - 1 wide) or 4; the loads of a z pair are all in flight together.  A row's
// missing y and z tiles are skipped (an FP64 addition of zero costs as much as
// any other) but in FP32 with at most 2 tiles, where the branches cost more.
template <typename T, int MX, int MY, int MZ>
__global__ void __launch_bounds__(256)
k_box_sum(const T *__restrict__ boxes, const int4 *__restrict__ tab, int K, size_t slot, int c0,
          T *__restrict__ mesh) {
    pdl_wait();
    const int row = blockIdx.x * blockDim.y + threadIdx.y;
    if (row >= K * K) return;
    const int y = row % K, z = row / K;
    const int4 y4 = __ldg(tab + K + y), z4 = __ldg(tab + 2 * K + z);
    const int ey[4] = {y4.x, y4.y, y4.z, y4.w}, ez[4] = {z4.x, z4.y, z4.z, z4.w};
    const T *__restrict__ src = boxes + blockIdx.y * slot;
    T *out = mesh + ((size_t)(c0 + blockIdx.y) * K * K + row) * K;
    for (int x = threadIdx.x; x < K; x += blockDim.x) {
        const int4 x4 = __ldg(tab + x);
        const int ex[4] = {x4.x, x4.y, x4.z, x4.w};
        T sum = T(0);
        auto add_pair = [&](int k0) {  // the tiles k0 and k0 + 1 along z
            T v[2][MY][MX];
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
                for (int j = 0; j < MY; j++)
#pragma unroll
                    for (int i = 0; i < MX; i++)
                        v[k][j][i] = (ex[i] | ey[j] | ez[k0 + k]) < 0
                                         ? T(0)
                                         : __ldg(src + ex[i] + ey[j] + ez[k0 + k]);
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
                for (int j = 0; j < MY; j++)
                    if ((sizeof(T) == 4 && MZ == 2) || (ey[j] | ez[k0 + k]) >= 0) {
#pragma unroll
                        for (int i = 0; i < MX; i++) sum += v[k][j][i];
                    }
        };
        add_pair(0);
        if (MZ > 2 && ez[2] >= 0) add_pair(2);
        out[x] = sum;
    }
}

template <typename T>
void launch_sum(const T *boxes, const BoxTable &bt, const MeshGeom &g, size_t slot, int c0, int nc,
                T *mesh, cudaStream_t s) {
    const int bx = g.K < 128 ? (g.K + 31) / 32 * 32 : 128, by = 256 / bx;
    const int m = (bt.most[0] > 2) | (bt.most[1] > 2) << 1 | (bt.most[2] > 2) << 2;
    auto kern = m == 0   ? k_box_sum<T, 2, 2, 2>
                : m == 1 ? k_box_sum<T, 4, 2, 2>
                : m == 2 ? k_box_sum<T, 2, 4, 2>
                : m == 4 ? k_box_sum<T, 2, 2, 4>
                         : k_box_sum<T, 4, 4, 4>;
    pdl_launch(kern, dim3((g.K * g.K + by - 1) / by, nc), dim3(bx, by), 0, s, boxes, bt.tab, g.K, slot, c0,
                                                                      mesh);
}

template <typename T, int P>
cudaError_t launch_box_t(const int *tile_off, const int *rec_idx, const uint32_t *rec_start,
                         const T *rec_w, const T *F, int C, const MeshGeom &g, T *boxes, int nslot,
                         const BoxTable &bt, T *mesh, cudaStream_t s) {
    const BoxDim b = box_dim(g);
    const size_t smem = (size_t)b.vol * sizeof(T);
    const int ntiles = g.ntx * g.nty * g.ntz;
    auto kern = k_spread_box<T, P>;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return e;
    const size_t slot = (size_t)ntiles * b.vol;
    for (int c0 = 0; c0 < C; c0 += nslot) {
        const int nc = C - c0 < nslot ? C - c0 : nslot;
        pdl_launch(kern, dim3(ntiles, nc), 32, smem, s, tile_off, rec_idx, rec_start, rec_w, F, C, c0, g,
                                                boxes);
        launch_sum<T>(boxes, bt, g, slot, c0, nc, mesh, s);
    }
    return cudaGetLastError();
}

}  // namespace

bool spread_box_ok(const MeshGeom &g, size_t elem) {
    // (offsets into one component's boxes fit 31 bits)
    return (size_t)box_dim(g).vol * elem <= 200 * 1024 &&
           (long long)g.ntx * g.nty * g.ntz * box_dim(g).vol < (1LL << 31);
}

size_t spread_box_bytes(const MeshGeom &g, size_t elem) {
    return (size_t)g.ntx * g.nty * g.ntz * box_dim(g).vol * elem;
}

// A coordinate of an axis with nt tiles of edge t is covered by its own tile
// and the lower ones within p - 1, wrap-aware (a box wider than the mesh covers
// it twice); at most four for edges >= 4 and p <= 8.
bool make_box_table(const MeshGeom &g, std::vector<int> *tab, int (*most)[3]) {
    const BoxDim b = box_dim(g);
    const int K = g.K, t[3] = {g.tx, g.ty, g.tz}, nt[3] = {g.ntx, g.nty, g.ntz};
    const int tile_step[3] = {b.vol, g.ntx * b.vol, g.nty * g.ntx * b.vol};
    const int step[3] = {1, b.x, b.y * b.x};
    tab->assign((size_t)3 * K * 4, -1);
    (*most)[0] = (*most)[1] = (*most)[2] = 0;
    for (int a = 0; a < 3; a++)
        for (int q = nt[a] - 1; q >= 0; q--)
            for (int l = 0; l < std::min(t[a], K - q * t[a]) + g.p - 1; l++) {
                int *e = tab->data() + ((size_t)a * K + (q * t[a] + l) % K) * 4, n = 0;
                while (n < 4 && e[n] >= 0) n++;
                if (n == 4) return false;
                e[n] = q * tile_step[a] + l * step[a];
                (*most)[a] = std::max((*most)[a], n + 1);
            }
    return true;
}

template <typename T>
cudaError_t launch_spread_box(const int *tile_off, const int *rec_idx, const uint32_t *rec_start,
                              const T *rec_w, const T *F, int C, const MeshGeom &g, T *boxes,
                              int nslot, const BoxTable &bt, T *mesh, cudaStream_t s) {
    if (nslot < 1 || !bt.tab || !spread_box_ok(g, sizeof(T))) return cudaErrorInvalidValue;
    switch (g.p) {
        case 4: return launch_box_t<T, 4>(tile_off, rec_idx, rec_start, rec_w, F, C, g, boxes, nslot, bt, mesh, s);
        case 6: return launch_box_t<T, 6>(tile_off, rec_idx, rec_start, rec_w, F, C, g, boxes, nslot, bt, mesh, s);
        case 8:
            if constexpr (sizeof(T) == 4) return cudaErrorInvalidValue;  // (never chosen)
            else return launch_box_t<T, 8>(tile_off, rec_idx, rec_start, rec_w, F, C, g, boxes, nslot, bt, mesh, s);
        default: return cudaErrorInvalidValue;
    }
}

template cudaError_t launch_spread_box<float>(const int *, const int *, const uint32_t *,
                                              const float *, const float *, int, const MeshGeom &,
                                              float *, int, const BoxTable &, float *,
                                              cudaStream_t);
template cudaError_t launch_spread_box<double>(const int *, const int *, const uint32_t *,
                                               const double *, const double *, int,
                                               const MeshGeom &, double *, int, const BoxTable &,
                                               double *, cudaStream_t);

}  // namespace spme
