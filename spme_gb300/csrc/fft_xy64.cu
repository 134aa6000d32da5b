// Launch of the two-factor x and y transforms (fft_xy.cuh), FP64.
#include "fft_list.h"
#include "fft_xy.cuh"

namespace spme {

template <>
cudaError_t launch_fft_xy<double>(int K, bool inv, double *mesh, double *G, long comps, const double *tw,
                                 cudaStream_t s) {
#define SPME_CASE(A, B) \
    if (K == A * B) return launch_xy<double, A, B>(inv, mesh, G, comps, tw, s);
    SPME_FFT_LIST(SPME_CASE)
#undef SPME_CASE
    return cudaErrorInvalidValue;
}

}  // namespace spme
