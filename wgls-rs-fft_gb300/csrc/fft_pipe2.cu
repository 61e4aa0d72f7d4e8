// Warp-column pass pairs (fft_pipe.cuh): both passes of N = 2^15 .. 2^20.
#include "fft_pipe.cuh"

namespace gbfft {

bool pipe2_kernel_info(int logr1, int logr2, PipeDesc &d, int loge) {
#define GBFFT_P2(A, B, E) \
    if (logr1 == A && logr2 == B && loge == E) { pipe_describe<A, B, A + B, 0, E>(d); return true; }
    GBFFT_P2(7, 8, 4)
    GBFFT_P2(8, 8, 4)
    GBFFT_P2(9, 8, 5)
    GBFFT_P2(9, 9, 5)
    GBFFT_P2(10, 9, 5)
    GBFFT_P2(10, 10, 5)
#undef GBFFT_P2
    return false;
}

}  // namespace gbfft
