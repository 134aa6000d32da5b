// Launch of the two-factor x and y transforms (fft_xy.cuh), FP32.
#include "fft_list.h"
#include "fft_xy.cuh"

namespace spme {

bool fft_xy_ok(int K, size_t elem) {
    // FP32 27 x 9: few threads in the first pass, 3.2 ms against 2.6 of cuFFT's 2D transforms
    // (R = 16); the others win or tie from K = 16 on
    if (elem == 4 && K == 27 * 9) return false;
#define SPME_CASE(A, B) \
    if (K == A * B) return true;
    SPME_FFT_LIST(SPME_CASE)
#undef SPME_CASE
    return false;
}

template <>
cudaError_t launch_fft_xy<float>(int K, bool inv, float *mesh, float *G, long comps, const float *tw,
                                 cudaStream_t s) {
#define SPME_CASE(A, B) \
    if (K == A * B) return launch_xy<float, A, B>(inv, mesh, G, comps, tw, s);
    SPME_FFT_LIST(SPME_CASE)
#undef SPME_CASE
    return cudaErrorInvalidValue;
}

}  // namespace spme
