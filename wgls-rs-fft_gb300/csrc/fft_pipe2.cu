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

bool pipe_wide_info(int logn, FusedDesc &d) {
    switch (logn) {
        case 21: pipe_describe<11, 10, 21, 0, 6>(d.pipe); break;
        case 22: pipe_describe<11, 11, 22, 0, 6>(d.pipe); break;
        default: return false;
    }
    d.logra = 11;
    d.logrb = logn - 11;
    d.logn = logn;
    d.groups_per_transform = 1;
    d.group_samples = 1ull << logn;
    return true;
}

}  // namespace gbfft
