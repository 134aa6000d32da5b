// Launch of the FP64 fused z transform (zfft64.cuh).
#include <cmath>

#include "fft_list.h"
#include "zfft64.cuh"

namespace spme {

cudaError_t launch_zfft64(int K, double *G, const double *tab2, const double *tw, double L,
                          const double *twopi_Ls, int nsys, int R, cudaStream_t s) {
#define SPME_CASE(A, B) \
    if (K == A * B) return launch_z64_k<A, B>(G, tab2, tw, L, twopi_Ls, nsys, R, s);
    SPME_FFT_LIST(SPME_CASE)
#undef SPME_CASE
    return cudaErrorInvalidValue;
}

}  // namespace spme
