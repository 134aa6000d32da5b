// Launch of the two-factor fused z transform (zfft2.cuh) for every supported K.
#include <cmath>

#include "zfft2.cuh"

namespace spme {

namespace {

// K = R1 R2 for the even-sized planes (K (K/2 + 1) even: 16-byte plane strides) of
// K = 2^a 3^b 5^c, 16 <= K <= 256 (one TMA box per component): the pair with the
// smallest max(3 R2, R1), the threads per column (R1 passes: one per component and
// n2; second pass: one per k1).
#define SPME_Z2_LIST(X)                                                                    \
    X(8, 2) X(6, 3) X(10, 2) X(8, 3) X(9, 3) X(10, 3) X(8, 4) X(9, 4) X(10, 4) X(12, 4)     \
    X(10, 5) X(9, 6) X(12, 5) X(16, 4) X(12, 6) X(15, 5) X(16, 5) X(15, 6) X(16, 6)        \
    X(20, 5) X(18, 6) X(20, 6) X(16, 8) X(15, 9) X(18, 8) X(25, 6) X(20, 8) X(18, 9)       \
    X(20, 9) X(24, 8) X(25, 8) X(24, 9) X(24, 10) X(27, 9) X(25, 10) X(32, 8)


// Columns per block: 16 (128-byte rows), or 8 where 16 leave one or two blocks per SM
// and 8 at least twice as many that the registers still allow.  Influence stage in ms,
// 16 / 8 columns: K = 75, R = 8 .025 / .025; K = 96, R = 16 .076 / .080; K = 100 .092 /
// .088; K = 160 .356 / .350 (R = 1 .041 / .035); K = 192 .526 / .552 (R = 1 .061 / .051);
// K = 200 .685 / .654; K = 240 1.07 / 1.38; K = 256 1.19 / 1.54.
constexpr int z2_width(int K) { return K >= 100 && K <= 200 ? 8 : 16; }

}  // namespace

int zfft2_width(int K) {
#define SPME_Z2_CASE(A, B) \
    if (K == A * B) return z2_width(A * B);
    SPME_Z2_LIST(SPME_Z2_CASE)
#undef SPME_Z2_CASE
    return 0;
}

cudaError_t launch_zfft2(int K, const CUtensorMap &map, const float *tab2, const float *tw, double L,
                         const double *twopi_Ls, int nsys, int R, int *err, cudaStream_t s) {
#define SPME_Z2_CASE(A, B) \
    if (K == A * B) return launch_z2<z2_width(A * B), A, B>(map, tab2, tw, L, twopi_Ls, nsys, R, err, s);
    SPME_Z2_LIST(SPME_Z2_CASE)
#undef SPME_Z2_CASE
    return cudaErrorInvalidValue;
}

}  // namespace spme
