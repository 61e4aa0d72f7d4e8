// Single-pass split form, one operand kind (fft_rows_tc.cuh).
#include "fft_rows_tc.cuh"

namespace gbfft {

template bool rows_tc_info_kind<kTcBF16>(int logn, RowsKernelInfo &k);

}  // namespace gbfft
