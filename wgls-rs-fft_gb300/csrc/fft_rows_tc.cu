// Host side of the split form's single-pass kernels (fft_rows_tc.cuh); each
// operand kind is compiled in a file of its own.
#include <algorithm>

#include "gbfft_internal.h"
#include "gbfft_plan.h"
#include "fft_tc.cuh"

namespace gbfft {

template <int KIND>
bool rows_tc_info_kind(int logn, RowsKernelInfo &k);

bool rows_tc_kernel_info(int logn, int precision, RowsKernelInfo &k) {
    switch (tc_kind_of_precision(precision)) {
        case kTcBF16: return rows_tc_info_kind<kTcBF16>(logn, k);
        case kTcBF16X6: return rows_tc_info_kind<kTcBF16X6>(logn, k);
        case kTcTF32: return rows_tc_info_kind<kTcTF32>(logn, k);
        default: return rows_tc_info_kind<kTcF16>(logn, k);
    }
}

cudaError_t rows_tc_prepare(RowsKernelInfo &k) {
    cudaError_t e = cudaSuccess;
    for (const void *fn : {k.fn, k.fn_inv})
        if (e == cudaSuccess && k.smem > 48 * 1024)
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem);
    for (const void *fn : {k.fn_persistent, k.fn_persistent_inv})
        if (e == cudaSuccess && fn && k.persist_smem > 48 * 1024)
            e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.persist_smem);
    return e;
}

cudaError_t rows_tc_launch(const RowsKernelInfo &k, const float2 *in, float2 *out, uint64_t batch,
                           const float2 *tw, int direction, int logn, const void *gtab, uint32_t *err, int sms,
                           cudaStream_t stream, LoadOps ops) {
    if (batch == 0) return cudaSuccess;
    const bool inv = direction == GBFFT_INVERSE;
    const float scale = inv ? ldexpf(1.0f, -logn) : 1.0f;
    float in_im = inv ? -1.0f : 1.0f;
    float out_re = scale, out_im = inv ? -scale : 1.0f;
    const uint4 *g = (const uint4 *)gtab;
    void *args[] = {(void *)&in,     (void *)&out,    (void *)&batch, (void *)&tw, (void *)&in_im,
                    (void *)&out_re, (void *)&out_im, (void *)&ops,   (void *)&g,  (void *)&err};
    // The tile loop from three tiles a resident CTA (7.5 M samples) on: below, its
    // last wave and its smaller CTAs cost what the shared set-up saves (2^8 x 4096
    // FP16: 8.2 us one-shot, 10.3 looped; 2^8 x 16384: 18.5, 18.8).
    const uint64_t resident = (uint64_t)k.persist_ctas_per_sm * (uint64_t)std::max(1, sms);
    const uint64_t tiles = (batch + k.persist_transforms - 1) / k.persist_transforms;
    if (k.fn_persistent && tiles >= 3 * resident)
        return launch_overlapped(inv ? k.fn_persistent_inv : k.fn_persistent, dim3((unsigned)resident),
                                dim3(k.persist_threads), args, k.persist_smem, stream);
    const uint64_t ctas = (batch + k.transforms_per_cta - 1) / k.transforms_per_cta;
    return launch_overlapped(inv ? k.fn_inv : k.fn, dim3((unsigned)ctas), dim3(k.threads), args, k.smem, stream);
}

}  // namespace gbfft
