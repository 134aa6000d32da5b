// Host-side launchers for the GB300 SPME-RPY kernels (sm_103a).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <vector>

#include "common.cuh"

namespace spme {

// Lets a kernel take smem bytes of dynamic shared memory.  The limit belongs to the kernel,
// not to a launch: a smaller one set for another engine's tile would hold for launches of
// other threads and for graphs captured before, so kernels whose need varies always get
// the same one (above every tile the engines accept).
constexpr size_t kSmemLimit = 220 * 1024;
template <typename F>
cudaError_t allow_smem(F kern, size_t smem) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(smem > kSmemLimit ? smem : kSmemLimit));
}

// ---- P-build and counting sorts (pbuild.cu) -------------------------------
// Sort keys with a slot within each key (atomic counts): the mesh tile of the
// stencil start (key1), the stencil-start cell ((sy K + sx) K + sz, K^3 keys;
// key2), the real-space cell (nc^3 cells of edge L/nc; key3), in one pass over
// the positions.  A null count skips that key.  With a mesh key, pstart (n)
// and pfrac (3n values of the engine's type: float when fp32) receive each
// particle's packed stencil start and fractional mesh coordinates; with the
// cell key, prel (n float4 / double4_32a) its position relative to its cell.
void launch_all_keys(const double *pos, int n, const MeshGeom &g, int nc, int *key1, int *count1,
                     int *slot1, int *key2, int *count2, int *slot2, int *key3, int *count3,
                     int *slot3, uint32_t *pstart, void *pfrac, void *prel, bool fp32,
                     cudaStream_t s);
// Real-space cell key (nc^3 cells of edge L/nc) and slot within its cell.
void launch_cell_keys(const double *pos, int n, double L, int nc, int *key, int *count,
                      int *slot, cudaStream_t s);
// Up to kMaxSorts counting sorts of the same n particles together (one launch for
// all of them per stage).  Sort j's counts are count[first .. first + nkeys) (first
// = the keys of the sorts before it); key[i] is particle i's key.  On entry perm[i]
// is particle i's slot within its key (from the atomic counts, in no fixed order);
// on return off[0 .. nkeys] holds the keys' offsets and perm[off[k] .. off[k + 1])
// lists key k's particles in increasing index.  scan_tmp: scan_tmp_elems(all keys)
// ints; tmp: n ints per sort.  Returns the kernels launched.
constexpr int kMaxSorts = 3;
struct Sort {
    const int *key;
    int *perm, *off;
    long first;
    int nkeys;
};
struct Sorts {
    Sort s[kMaxSorts];
    int count;
};
size_t scan_tmp_elems(long nkeys);
int launch_sorts(const Sorts &S, const int *count, int n, int *scan_tmp, int *tmp, cudaStream_t s);
// One set of B-spline records in sorted order (perm): idx[s] = perm[s], the packed
// stencil start, and p weights per axis (record width RecordWidth<T,P>).
template <typename T>
struct RecordSet {
    const int *perm;
    int *idx;
    uint32_t *start;
    T *w;
};
// Up to two record sets from launch_all_keys' per-particle starts and fractional
// coordinates and, if cpos is not null, the cell-relative positions in cell order,
// cpos[s] = prel[cperm[s]] (float4 or double4_32a), in one launch.
template <typename T>
void launch_records(const uint32_t *pstart, const T *pfrac, int n, int p, int nset,
                    const RecordSet<T> *sets, const void *prel, const int *cperm, void *cpos,
                    cudaStream_t s);
// Cell-sorted positions relative to their cell's lower corner (float4 or double4_32a).
void launch_cell_positions(const double *pos, const int *perm, int n, double L, int nc,
                           bool fp32, void *cpos, cudaStream_t s);

// ---- spread / interpolate (spread.cu, interp.cu) --------------------------
template <typename T>
cudaError_t launch_spread(const int *tile_off, const int *rec_idx, const uint32_t *rec_start,
                          const T *rec_w, const T *F, int C, const MeshGeom &g, T *mesh,
                          cudaStream_t s);
// Column-gather spread (spread_cols.cu): records sorted by stencil-start cell,
// start_off[(sy K + sx) K + sz] the offsets of that order (K^3 + 1 entries),
// Fs the force rows in the same order.  Usable when spread_cols_ok(K, C, elem, p).
bool spread_cols_ok(int K, int C, size_t elem, int p);
// Row width (elements) of the force rows the column-gather spread reads: each
// lane's components contiguous and padded (C <= 16: C, unpadded).
int spread_cols_row_width(int C);
// Fs[s] = the row of F[idx[s]] (C components) in that padded layout.
template <typename T>
void launch_gather_cols_rows(const T *F, const int *idx, int n, int C, T *Fs, cudaStream_t s);
// Arguments of one system's column-gather spread: start-cell offsets of this
// system (indexed by its own (sy K + sx) K + sz), records and force rows
// indexed by sorted slot, ws the record stride (elements).
template <typename T>
struct SpreadColsArgs {
    const int *soff;
    const uint32_t *rec_start;
    const T *rec_w;
    const T *Fs;
    T *mesh;
    int C, RW, K, nzt, zseg, ws;  // nzt z tiles or segments of zseg planes
};
// A system of a batched launch: its arguments, order and blocks along x and y.
template <typename T>
struct SpreadColsSys {
    SpreadColsArgs<T> args;
    int p, gx, gy;
};
// Blocks of one system's column-gather spread: along x and y, z tiles or segments
// (and their planes), in all (with component chunks), and without z segments;
// columns: the last summed over the systems of a launch (0: this system alone).
struct SpreadColsGrid {
    int x, y, nzt, zseg, blocks;
    long columns;
};
SpreadColsGrid spread_cols_grid(int K, int C, size_t elem, long columns);
// The z-marching form of the FP32 column gather (spread_march.cu; chosen by
// launch_spread_cols and its batched form): same records, rows and offsets.
// launch_spread_march sets A.nzt and A.zseg.  FP32 batches always take it.
SpreadColsGrid spread_march_grid(int K, int C, long columns);
cudaError_t launch_spread_march(SpreadColsArgs<float> A, int p, cudaStream_t s);
cudaError_t launch_spread_march_batch(const SpreadColsSys<float> *sys, const int *prefix, int nsys,
                                      int total, int C, cudaStream_t s);
// All systems (same C) in one persistent launch; prefix[k] = the first block
// of system k (nsys + 1 entries, prefix[nsys] = total), both on the device.
template <typename T>
cudaError_t launch_spread_cols_batch(const SpreadColsSys<T> *sys, const int *prefix, int nsys,
                                     int total, int C, cudaStream_t s);
template <>
cudaError_t launch_spread_cols_batch<float>(const SpreadColsSys<float> *, const int *, int, int,
                                            int, cudaStream_t);
template <>
cudaError_t launch_spread_cols_batch<double>(const SpreadColsSys<double> *, const int *, int, int,
                                             int, cudaStream_t);
template <typename T>
cudaError_t launch_spread_cols(const int *start_off, const uint32_t *rec_start, const T *rec_w,
                               const T *Fs, int C, const MeshGeom &g, T *mesh, cudaStream_t s);
// Spread through per-tile boxes (spread_box.cu), for few components: records in
// tile order, any K; boxes: scratch of nslot * spread_box_bytes (nslot
// components per launch).  Usable when spread_box_ok(g, elem).
// bt: make_box_table's offsets on the device (3 K entries of four) and the most
// tiles that cover a coordinate of each axis; false if one has over four.
struct BoxTable {
    const int4 *tab = nullptr;
    int most[3] = {0, 0, 0};
};
bool spread_box_ok(const MeshGeom &g, size_t elem);
size_t spread_box_bytes(const MeshGeom &g, size_t elem);
bool make_box_table(const MeshGeom &g, std::vector<int> *tab, int (*most)[3]);
template <typename T>
cudaError_t launch_spread_box(const int *tile_off, const int *rec_idx, const uint32_t *rec_start,
                              const T *rec_w, const T *F, int C, const MeshGeom &g, T *boxes,
                              int nslot, const BoxTable &bt, T *mesh, cudaStream_t s);
// TMA descriptor of the real mesh [C][K][K][K] for the interpolation halo
// boxes: FP32 (interp.cu) 4 components of rows of kInterpMaxRow points (more
// blocks per SM than 8 components, measured faster), FP64 (interp_fp64.cu) one
// component of rows of interp64_row(tx + p - 1) points.
constexpr int kInterpMaxRow = 24;
constexpr int kInterp64Threads = 128;
// Row length of an FP64 box: the least r >= n that is 2 (mod 4) (bank spread of
// neighbouring rows; whole 16-byte vectors).
__host__ __device__ constexpr int interp64_row(int n) { return n + (6 - n % 4) % 4; }
struct InterpMaps {
    CUtensorMap cg4;
    bool ok4 = false;
};
bool make_interp_maps(InterpMaps *maps, const void *mesh, int C, const MeshGeom &g, size_t elem);
// Dynamic shared memory of the interpolation kernel.
size_t interp_smem_bytes(const MeshGeom &g, size_t elem);
// Tile shapes the engines accept: four components of the tile and its halo, rows
// of kInterpMaxRow points, within 220 KB.
bool interp_tile_ok(const MeshGeom &g, size_t elem);
// Arguments of one system's interpolation (records indexed by sorted slot,
// stride ws; tile_off indexed by this system's tiles; W rows by particle).
template <typename T>
struct InterpArgs {
    const int *tile_off;
    const int *rec_idx;
    const uint32_t *rec_start;
    const T *rec_w;
    const T *mesh;
    T *W;
    int *err;
    MeshGeom g;
    int C, cb, ce, accumulate, use_tma, ws;
};
// One system of a batched interpolation: its arguments and, when args.use_tma
// is set, its TMA box over its own mesh (make_interp_box; read by the kernel
// from this global work list, 64-byte aligned).
template <typename T>
struct InterpSys {
    CUtensorMap tmap;
    InterpArgs<T> args;
};
// The TMA box of one mesh (false where TMA does not apply: K * elem
// not a multiple of 16 bytes, an unaligned mesh, or no driver entry point).
bool make_interp_box(CUtensorMap *map, const void *mesh, int C, const MeshGeom &g, size_t elem);
// All systems in one persistent launch over their tiles (prefix as for the
// spread; smem = the largest interp_smem_bytes of the systems).
template <typename T>
cudaError_t launch_interp_batch(const InterpSys<T> *sys, const int *prefix, int nsys, int total,
                                size_t smem, cudaStream_t s);
// Components [cb, ce) of the C-component mesh (cb a multiple of 12, or 0) into
// W[n][C]; err: device flag set to 1 if a TMA wait timed out.
template <typename T>
cudaError_t launch_interp(const InterpMaps &maps, const int *tile_off, int n, const int *rec_idx,
                          const uint32_t *rec_start, const T *rec_w, const T *mesh, int C,
                          int cb, int ce, const MeshGeom &g, T *W, int accumulate, int *err,
                          cudaStream_t s);
template <>
cudaError_t launch_interp<float>(const InterpMaps &, const int *, int, const int *,
                                 const uint32_t *, const float *, const float *, int, int, int,
                                 const MeshGeom &, float *, int, int *, cudaStream_t);
template <>
cudaError_t launch_interp_batch<float>(const InterpSys<float> *, const int *, int, int, size_t,
                                       cudaStream_t);
template <>
cudaError_t launch_interp<double>(const InterpMaps &, const int *, int, const int *,
                                  const uint32_t *, const double *, const double *, int, int, int,
                                  const MeshGeom &, double *, int, int *, cudaStream_t);
template <>
cudaError_t launch_interp_batch<double>(const InterpSys<double> *, const int *, int, int, size_t,
                                        cudaStream_t);

// ---- host tables (engine.cu) ----------------------------------------------
// |b(m)|^2 = 1 / |sum_{j<p-1} M_p(j+1) e^{i j 2 pi m'/K}|^2 (old-version/spme.c:109-126).
void host_moduli2(int K, int p, std::vector<double> &out);

// ---- k-space influence (influence.cu) -------------------------------------
// tab[(z*K + y)*Kh + kx] = (S(k)|b|^2 / V, S(k)|b|^2 / (V k^2)), zero at k = 0.
template <typename T>
void launch_influence_table(T *tab2, const double *bmod2, int K, double L, double xi,
                            double a, cudaStream_t s);
// In-place influence on the component-major half spectrum G[c][(z*K+y)*Kh+kx].
template <typename T>
void launch_influence(T *G, const T *tab2, int K, double L, int R, cudaStream_t s);

// ---- fused z-FFT + influence + inverse z-FFT (zfft.cu) --------------------
struct ZPlan {
    int K;
    int nst;              // radix stages
    int rad[12];          // radices, first stage of the inverse (DIT) first
    int len_before_last;  // product of the first nst-1 radices
    int npass;            // passes of one or two stages
    int pcode[12];        // 10 * R1 + R2 (R2 = 1: single stage)
    int pspan[12];        // span of the pass's first (R1) stage in DIT order
};
// Radix plan, twiddles e^{-2 pi i e/K} (re, im pairs; re - 1 for the sizes of the
// FP64 two-factor kernels) and the digit-reversal
// permutation (position p holds frequency perm[p]) for length-K transforms.
bool make_zplan(int K, size_t elem, ZPlan *zp, std::vector<double> *tw, std::vector<int> *perm);
// Columns per block for K (0 if K does not fit the fused kernel).
int zfft_width(int K, size_t elem);
// Two-factor form of the same operation (zfft2.cu; FP32, K <= 256): columns per
// block (0: not this K), and its launch.  Batches: nsys systems of R right-hand sides each,
// spectra and tables consecutive, 2 pi / L of every system at twopi_Ls (L unused);
// else 1 and null.
int zfft2_width(int K);
cudaError_t launch_zfft2(int K, const CUtensorMap &map, const float *tab2, const float *tw, double L,
                         const double *twopi_Ls, int nsys, int R, int *err, cudaStream_t s);
// Its FP64 form (zfft64.cu; K of fft_xy_ok, elem 8), on G in place.
cudaError_t launch_zfft64(int K, double *G, const double *tab2, const double *tw, double L,
                          const double *twopi_Ls, int nsys, int R, cudaStream_t s);
// Two-factor x and y transforms of the z-planes of comps consecutive meshes (fft_xy.cuh; K =
// 2^a 3^b 5^c, 16 to 256, fft_xy_ok): mesh -> G, or G -> mesh (inv; G is overwritten), every
// mesh on its own.  tw as for the z transform.
bool fft_xy_ok(int K, size_t elem);
template <typename T>
cudaError_t launch_fft_xy(int K, bool inv, T *mesh, T *G, long comps, const T *tw, cudaStream_t s);
template <>
cudaError_t launch_fft_xy<float>(int, bool, float *, float *, long, const float *, cudaStream_t);
template <>
cudaError_t launch_fft_xy<double>(int, bool, double *, double *, long, const double *, cudaStream_t);
// One-pass 2D (y, x) transforms of the mesh's z-planes (FP32; K = 128, 160,
// 256): real planes [planes][K][K] <-> half spectra [planes][K][K/2+1], cuFFT's
// layouts and unnormalised conventions.  tables: make_fft2d_tables' bytes on
// the device.
bool fft2d_ok(int K, size_t elem);
size_t fft2d_table_bytes(int K);
bool make_fft2d_tables(int K, std::vector<unsigned char> *out);
cudaError_t launch_fft2d_r2c(int K, const float *mesh, float *G, long planes, const void *tables,
                             cudaStream_t s);
cudaError_t launch_fft2d_c2r(int K, const float *G, float *mesh, long planes, const void *tables,
                             cudaStream_t s);
// TMA descriptor over the half spectrum G[C][K][K][K/2+1] (complex of elem-byte
// reals), z-planes viewed as flat rows.
bool make_zfft_map(CUtensorMap *map, void *G, int K, int C, size_t elem);
// On the half spectrum after 2D (y, x) R2C transforms: FFT along z,
// influence (table as launch_influence), inverse FFT along z, Hermitian part of
// the kx = 0 and K/2 planes.  tw: K complex twiddles of type T; perm: K ints.
template <typename T>
cudaError_t launch_zfft_influence(const CUtensorMap &map, T *G, const T *tab2, const T *tw,
                                  const int *perm, const ZPlan &zp, double L, int R, int *err,
                                  cudaStream_t s);

// ---- real-space pair sum + self term (realspace.cu) -----------------------
// Table of the real-space pair functions for FP64 engines (xi and a fixed per
// engine), in s = r^2: A = F and B = G / s as polynomials of degree kPairDeg in
// the offset from the segment's centre, interleaved.  Segments split each
// octave of s evenly (2^(20 - shift) of them), so the segment is the top bits
// of s: segment g = high word >> shift has index g - base below mid = (2a)^2
// and one more from mid on (the segment holding mid carries both forms).  Used
// for lo <= s <= hi (compared as bits); a null coef means no table.
constexpr int kPairDeg = 6;
struct PairTable {
    const double *coef = nullptr;
    long long lo_bits = 0, mid_bits = 0, hi_bits = 0;
    int base = 0, shift = 14;
};
// Fits the table on the host (the segments that meet 2e-13 relative between nodes, halved:
// the error left is that of the closed form's values); false if no fit meets that within
// 1024 segments per octave.
bool build_pair_table(double xi, double a, double rc, std::vector<double> *coef, PairTable *t);
// cpos: float4 for T = float, double4_32a for T = double (cell-relative); FP32 in
// realspace.cu (tab unused), FP64 in realspace_fp64.cu.  F2 (FP32; unused in FP64):
// the force rows as that kernel reads them, real_row(R) values each: for up to
// kRealFew right-hand sides in F's order padded to 16 bytes, for more by component
// ([d][rows_even(R)]); the padding is zero, and so are the real_lead(R) values before F2
// (row -1, which padding entries of the pair lists take: a particle's own row there
// would turn an infinite force into 0 inf).
// The line between the forms: with 3 and 4 right-hand sides the compensated sums of the
// first (per lane) need more registers and shared memory: N = 1e6, R = 3 1.37 against 1.31 ms,
// R = 4 1.53 against 1.31, at volume fraction 0.12 2.72 against 2.07; at R = 2 1.07 ms.
constexpr int kRealFew = 2;
__host__ __device__ constexpr int rows_even(int R) { return (R + 1) & ~1; }
__host__ __device__ constexpr int real_row(int R) {
    return R <= kRealFew ? (3 * R + 3) / 4 * 4 : 3 * rows_even(R);
}
// Zeros before the rows of up to R right-hand sides (256-byte steps).
__host__ __device__ constexpr int real_lead(int R) { return (3 * rows_even(R) + 63) / 64 * 64; }
// The place of right-hand side r, component d in such a row.
__host__ __device__ constexpr int real_at(int R, int r, int d) {
    return R <= kRealFew ? 3 * r + d : d * rows_even(R) + r;
}
template <typename T>
cudaError_t launch_realspace(int nc, const int *cell_off, const int *cell_perm, const void *cpos,
                             const T *F, const T *F2, int R, double L, double rc, double xi, double a,
                             int with_self, const PairTable &tab, T *W, cudaStream_t s);
// FP32 pair-function coefficients of one (xi, a) and the FP32 copies of the
// geometry (real_args fills them): far field (r >= 2a), with ir = 1/r,
//   F = erfc(xi r) (0.75 ir + c1 ir^3) + e^{-xi^2 r^2} (A4 r^4 + A2 r^2 + A0 + Am2 ir^2)
//   G = erfc(xi r) (0.75 ir + c3 ir^3) + e^{-xi^2 r^2} (-A4 r^4 + B2 r^2 + B0 + Bm2 ir^2)
// near field: xi, xi3a2 = xi^3 a^2, ia = 1/a, n1 = 9/(32 a^2), n2 = 3/(32 a^2).
struct RealCoef {
    float xi, xi2, a2x4, xi3a2, ia, n1, n2;
    float A4, A2, A0, Am2, B2, B0, Bm2, c1, c3;
    float L, h, rc2, self_c;
};
// Arguments of one system's real-space sum (cell_off indexed by this system's
// cells; slots, positions and rows global).
template <typename T>
struct RealArgs {
    const int *cell_off;
    const int *cell_perm;
    const void *cpos;
    const T *F;
    const T *F2;
    T *W;
    int nc, R, with_self;
    double L, h, rc2, xi, a, self_c;
    PairTable tab;
    RealCoef cf;
};
double real_self_coeff(double xi, double a);
template <typename T>
RealArgs<T> real_args(int nc, const int *cell_off, const int *cell_perm, const void *cpos,
                      const T *F, const T *F2, int R, double L, double rc, double xi, double a, int with_self,
                      const PairTable &tab, T *W);
// All systems (R right-hand sides each) in one persistent launch over their cells
// (prefix as for the spread).
template <typename T>
cudaError_t launch_realspace_batch(const RealArgs<T> *sys, const int *prefix, int nsys,
                                   int total, int R, cudaStream_t s);

template <>
cudaError_t launch_realspace<float>(int, const int *, const int *, const void *, const float *,
                                    const float *, int, double, double, double, double, int, const PairTable &,
                                    float *, cudaStream_t);
template <>
cudaError_t launch_realspace<double>(int, const int *, const int *, const void *, const double *,
                                     const double *, int, double, double, double, double, int, const PairTable &,
                                     double *, cudaStream_t);
template <>
cudaError_t launch_realspace_batch<float>(const RealArgs<float> *, const int *, int, int, int,
                                          cudaStream_t);
template <>
cudaError_t launch_realspace_batch<double>(const RealArgs<double> *, const int *, int, int, int,
                                           cudaStream_t);

// ---- layout conversions (pack.cu) -----------------------------------------
// W = self_c * F (the self term alone, when no real-space sum is requested)
template <typename T>
void launch_self(const T *F, int n, int R, double self_c, T *W, cudaStream_t s);
template <typename T>
void launch_pack(const T *f, long ld, int n, int R, T *F, cudaStream_t s);
// u[r*ld + 3i + d] = beta*u + alpha*W[i][3r+d]   (u not read when beta == 0)
// Tiled (shared-memory) forms of launch_pack / launch_unpack(_sum): coalesced on
// both sides; W2 may be null (plain unpack).  Up to 48 KB of shared memory.
// Right-hand sides [r0, r1) of f into their columns of F[n][3R] and, if F2 is not
// null, their places in F2[n][real_row(R)] (with the last ones, zeros in its padding).
template <typename T>
void launch_pack_tiled(const T *f, long ld, int n, int R, int r0, int r1, T *F, T *F2,
                       cudaStream_t s);
// (launch_unpack_tiled: right-hand sides [r0, r1) of the R in W / W2.)
template <typename T>
void launch_unpack_tiled(const T *W, const T *W2, int n, int R, int r0, int r1, double alpha,
                         double beta, T *u, long ld, cudaStream_t s);
template <typename T>
void launch_unpack(const T *W, int n, int R, double alpha, double beta, T *u, long ld,
                   cudaStream_t s);

}  // namespace spme
