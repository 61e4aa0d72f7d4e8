// Warp-column pass pairs (fft_pipe.cuh): the last two passes of a three-pass
// transform with radices (2^(L-16), 256, 256), N = 2^21 .. 2^26.
#include "fft_pipe.cuh"

namespace gbfft {

bool pipe3_kernel_info(int logn, PipeDesc &d) {
#define GBFFT_P3(L) \
    if (logn == L) { pipe_describe<8, 8, L, L - 16, 4>(d); return true; }
    GBFFT_P3(21)
    GBFFT_P3(22)
    GBFFT_P3(23)
    GBFFT_P3(24)
    GBFFT_P3(25)
    GBFFT_P3(26)
#undef GBFFT_P3
    return false;
}

}  // namespace gbfft
