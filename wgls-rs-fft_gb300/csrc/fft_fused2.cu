// Fused pass pairs (fft_fused.cuh): the two-pass instantiations
// (N = 2^15 .. 2^20, both passes in one launch) and the host side shared with
// the three-pass pairs (fft_fused3.cu).
#include <algorithm>
#include <cstring>

#include "gbfft_internal.h"
#include "gbfft_plan.h"
#include "fft_pipe.cuh"
#include "tensor_map.h"

namespace gbfft {

bool fused2_kernel_info(int logr1, int logr2, FusedDesc &d, int loge) {
    pipe2_kernel_info(logr1, logr2, d.pipe, loge);
    if (loge == 5) {
#define GBFFT_F2E(A, B, T) \
    if (logr1 == A && logr2 == B) { fused_describe<A, B, T, A + B, 0, 5>(d); return true; }
        GBFFT_F2E(7, 8, 128)
        GBFFT_F2E(8, 8, 128)
        GBFFT_F2E(9, 8, 256)
        GBFFT_F2E(9, 9, 256)
        GBFFT_F2E(10, 9, 512)
        GBFFT_F2E(10, 10, 512)
#undef GBFFT_F2E
        return false;
    }
    if (loge != 4) return false;
#define GBFFT_F2(A, B, T) \
    if (logr1 == A && logr2 == B) { fused_describe<A, B, T, A + B, 0>(d); return true; }
    GBFFT_F2(7, 6, 128)
    GBFFT_F2(7, 7, 128)
    GBFFT_F2(7, 8, 256)
    GBFFT_F2(8, 8, 256)
    GBFFT_F2(9, 8, 512)
    GBFFT_F2(9, 9, 512)
    GBFFT_F2(10, 9, 1024)
    GBFFT_F2(10, 10, 1024)
#undef GBFFT_F2
    return false;
}

int pass_sub_segments(int logr, int loge, TwiddleSegment *out, uint64_t base, int &entries) {
    switch (loge * 16 + logr) {
#define GBFFT_SEG(E, R) \
    case E * 16 + R: entries = SubCfg<R, E>::tw_entries(); return subcfg_segments<R, E>(out, base);
        GBFFT_SEG(5, 7) GBFFT_SEG(5, 8) GBFFT_SEG(5, 9) GBFFT_SEG(5, 10)
        GBFFT_SEG(4, 11) GBFFT_SEG(4, 5) GBFFT_SEG(4, 6) GBFFT_SEG(4, 7) GBFFT_SEG(4, 8) GBFFT_SEG(4, 9) GBFFT_SEG(4, 10)
#undef GBFFT_SEG
        default: entries = 0; return -1;
    }
}

// Disjoint: the launch writes outputs while it still reads inputs, which the first of
// three passes has copied out of the way of an output that overlaps them.
bool wide_usable(const float2 *in, const float2 *out, uint64_t samples, const LoadOps &ops) {
    const uintptr_t a = (uintptr_t)in, b = (uintptr_t)out;
    return (a > b ? a - b : b - a) >= samples * sizeof(float2) && ((a | b) & 15u) == 0 && !ops.win &&
           ops.noise_sigma == 0.f && tensor_map_encoder() != nullptr;
}

cudaError_t fused_prepare(FusedDesc &d) {
    cudaError_t e = cudaSuccess;
    if (d.smem > 48 * 1024) {
        e = cudaFuncSetAttribute(d.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)d.smem);
        if (e != cudaSuccess) return e;
    }
    if (d.pipe.fn) {
        e = cudaFuncSetAttribute(d.pipe.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)d.pipe.smem);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.pipe.ctas_per_sm, d.pipe.fn, d.pipe.threads,
                                                              d.pipe.smem);
        if (e != cudaSuccess) return e;
    }
    if (!d.fn) return e;  // the wide two-pass launch has no barrier form
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.ctas_per_sm, d.fn, d.threads, d.smem);
    if (e != cudaSuccess || d.tmem_cols <= 0) return e;
    // Split forms: the occupancy query answers 1 for kernels that allocate
    // tensor memory, although the SM runs as many such CTAs as registers and
    // shared memory allow (tcgen05.alloc only waits while the SM's 512 TMEM
    // columns are taken, and each CTA allocates before it claims any work, so
    // such a wait never holds up a dependency).  Count them from the kernel's
    // resources, bounded by the columns each CTA holds for its whole run.
    cudaFuncAttributes fa;
    int dev = 0, smem_sm = 0, regs_sm = 0, threads_sm = 0;
    if ((e = cudaFuncGetAttributes(&fa, d.fn)) != cudaSuccess) return e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&threads_sm, cudaDevAttrMaxThreadsPerMultiProcessor, dev)) != cudaSuccess) return e;
    const int warps = (d.threads + 31) / 32;
    const int regs_cta = ((fa.numRegs + 7) / 8) * 8 * 32 * warps;  // allocated per warp in units of 8 per thread
    const size_t smem_cta = d.smem + fa.sharedSizeBytes + 1024;      // 1 KB reserved per CTA
    int fit = std::min(regs_sm / std::max(1, regs_cta), threads_sm / std::max(1, d.threads));
    fit = std::min<int>(fit, (int)(smem_sm / smem_cta));
    d.ctas_per_sm = std::max(1, std::min(std::max(d.ctas_per_sm, fit), 512 / d.tmem_cols));
    return cudaSuccess;
}

uint32_t fused_lag(uint64_t inflight, uint32_t tiles_per_group, uint64_t group_samples, uint64_t ngroups) {
    const uint64_t per = 2ull * tiles_per_group;
    // enough queue between producer and consumer that consumers rarely wait
    uint64_t lag = (2 * inflight + per - 1) / per;
    // ... but a window of intermediates that stays well inside L2
    const uint64_t cap = std::max<uint64_t>(1, kFusedWindowBytes / (8ull * group_samples));
    lag = std::min(std::max<uint64_t>(lag, 1), cap);
    return (uint32_t)std::min<uint64_t>(lag, ngroups);
}

// 3-D tensor map of float pairs: `cols` complex a row, `rows` rows of stride
// `cols`, `mats` matrices back to back; boxes of box_cols columns x <= 256 rows.
static bool pipe_map(CUtensorMap *map, const void *base, uint64_t cols, uint64_t rows, uint64_t mats, int box_cols) {
    PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t dims[3] = {2 * cols, rows, mats};
    const cuuint64_t strides[2] = {cols * sizeof(float2), rows * cols * sizeof(float2)};
    const cuuint32_t box[3] = {2u * (cuuint32_t)box_cols, (cuuint32_t)std::min<uint64_t>(rows, 256), 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void *)base, dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE,
                  box_cols == 16  ? CU_TENSOR_MAP_SWIZZLE_128B
                  : box_cols == 8 ? CU_TENSOR_MAP_SWIZZLE_64B
                                  : CU_TENSOR_MAP_SWIZZLE_32B,
                  // 32-byte rows: fetch 64 bytes, the neighbouring tile's share (2^22 x 16: 346
                  // us; 32, 128 and 256 bytes 359, 359, 363)
                  box_cols >= 8 ? CU_TENSOR_MAP_L2_PROMOTION_L2_128B : CU_TENSOR_MAP_L2_PROMOTION_L2_64B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The first pass alone of a transform of 2^logn samples, through the ring of tiles of a
// shorter pair whose pass A has its radix: the queue is cut off before the first B
// item.  A group is as many columns as that pair's transform has: group g's tiles are
// columns g N' / R .. of the long transform (the maps' third dimension), and its
// output the next N' samples.  One transform a launch: two dimensions of the map are
// its rows and the groups.  For N = 2^26, whose radix-2^10 first pass ran one CTA an SM
// in lock-step (194 us where radix 2^9 takes 164): 2^26 x 1 470.6 -> 460 us.  Needs what
// the wide pairs need (wide_usable); the pass kernel otherwise.
cudaError_t pipe_first_launch(const FusedDesc &d, const float2 *in, float2 *out, int logn, const float2 *tw_a,
                              float in_im, uint32_t *ctr, uint32_t *err, int sms, cudaStream_t stream) {
    PipeParams Q;
    memset(&Q, 0, sizeof Q);
    const uint64_t cols = 1ull << (d.logn - d.logra);
    PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    const cuuint64_t dims[3] = {2 * cols, 1ull << d.logra, 1ull << (logn - d.logn)};
    const cuuint64_t strides[2] = {sizeof(float2) << (logn - d.logra), cols * sizeof(float2)};
    const cuuint32_t box[3] = {(cuuint32_t)(2 * d.pipe.box_cols_a), 256, 1}, estr[3] = {1, 1, 1};
    if (!encode || encode(&Q.map_in, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void *)in, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    FusedParams &P = Q.f;
    P.in = in;
    P.out = out;
    P.batch = P.ngroups = P.lag = 1u << (logn - d.logn);
    P.nitems = d.pipe.tiles_per_group * P.ngroups;
    P.tw_a = P.tw_b = tw_a;
    P.in_im = in_im;
    P.out_re = P.out_im = 1.0f;
    P.ctr = ctr;
    P.err = err;
    P.spin_limit = 1u << 22;
    void *args[] = {(void *)&Q};
    const uint64_t ctas = (uint64_t)d.pipe.ctas_per_sm * (uint64_t)std::max(1, sms);
    return launch_overlapped(d.pipe.fn, dim3((unsigned)std::min<uint64_t>(P.nitems, ctas)), dim3(d.pipe.threads), args,
                             d.pipe.smem, stream);
}

cudaError_t fused_launch(const FusedDesc &d, const float2 *in, float2 *out, uint64_t batch, const float2 *tw_a,
                         const float2 *tw_b, const float2 *tw_lo, const float2 *tw_hi, float in_im, float out_re,
                         float out_im, LoadOps ops, uint32_t *ctr, uint32_t *err, int sms, cudaStream_t stream,
                         const void *gtab, const uint64_t *tab_in, const uint64_t *tab_out) {
    FusedParams P;
    P.tab_in = tab_in;
    P.tab_out = tab_out;
    P.in = in;
    P.out = out;
    P.batch = (uint32_t)batch;
    P.ngroups = (uint32_t)(batch * d.groups_per_transform);
    P.tw_a = tw_a;
    P.tw_b = tw_b;
    P.tw_lo = tw_lo;
    P.tw_hi = tw_hi;
    P.in_im = in_im;
    P.out_re = out_re;
    P.out_im = out_im;
    P.ops = ops;
    P.ctr = ctr;
    P.err = err;
    P.spin_limit = 1u << 22;  // ~0.5 s of 128 ns polls; a healthy wait is a few microseconds
    P.gtab = (const uint4 *)gtab;
    // The warp-column form (fft_pipe.cuh) needs tensor maps: buffers on 16-byte
    // boundaries, and no tables of row addresses.  It is the faster one wherever
    // its ring of tiles fills (2^16 x 1024: 297 -> 230 us, 2^16 x 32: 21.0 -> 17.0),
    // but takes longer to start: a launch of no more tiles than resident CTAs, or of
    // a single group (no second pass can start before the whole first one is done),
    // is left to the barrier form (2^16 x 4: 9.4 us here against 8.1, 2^17 x 4 12.7
    // against 11.7, 2^20 x 1 18.5 against 18.2).  Except where every tile has a CTA of
    // its own and the barrier form's are radix-2^10 tiles, whose 16 warps go through
    // them in lock-step: 2^19 x 1 13.7 us here against 17.5.  Load options stay with
    // the barrier form, whose lanes run along the columns: here they run along the
    // rows, and each window factor would be a sector of its own (2^16 x 1024: 342
    // against 315 us).
    const uint64_t pipe_ctas = (uint64_t)d.pipe.ctas_per_sm * (uint64_t)std::max(1, sms);
    const uint64_t tiles = 2ull * d.pipe.tiles_per_group * P.ngroups;
    const bool filled = tiles > pipe_ctas ? P.ngroups > 1 : d.logra == 10;
    if (d.pipe.fn && !tab_in && !tab_out && (((uintptr_t)in | (uintptr_t)out) & 15u) == 0 && (filled || !d.fn) &&
        !(d.pipe.first && (ops.win || ops.noise_sigma != 0.f))) {
        PipeParams Q;
        const uint64_t n = 1ull << d.logn, ra = 1ull << d.logra, rb = 1ull << d.logrb, p = 1ull << d.logpa;
        if (pipe_map(&Q.map_in, in, n / ra, ra, batch, d.pipe.box_cols_a) &&
            pipe_map(&Q.map_mid, out, d.logpa ? p : n / ra, ra, d.logpa ? batch * (n / ra / p) : batch,
                     d.pipe.box_cols_a) &&
            pipe_map(&Q.map_io, out, n / rb, rb, batch, d.pipe.box_cols_b)) {
            P.nitems = 2u * d.pipe.tiles_per_group * P.ngroups;
            P.lag = fused_lag(pipe_ctas * d.pipe.slots, d.pipe.tiles_per_group, d.group_samples, P.ngroups);
            Q.fact_a = d.pipe.fact_a;
            Q.fact_b = d.pipe.fact_b;
            Q.f = P;
            void *args[] = {(void *)&Q};
            return launch_overlapped(d.pipe.fn, dim3((unsigned)std::min<uint64_t>(P.nitems, pipe_ctas)),
                                    dim3(d.pipe.threads), args, d.pipe.smem, stream);
        }
    }
    if (!d.fn) return cudaErrorInvalidValue;
    const uint64_t ctas = (uint64_t)std::max(1, d.ctas_per_sm) * (uint64_t)std::max(1, sms);
    P.nitems = 2u * d.tiles_per_group * P.ngroups;
    P.lag = fused_lag(ctas, d.tiles_per_group, d.group_samples, P.ngroups);
    const uint64_t grid = std::min<uint64_t>((uint64_t)P.nitems, ctas);
    void *args[] = {(void *)&P};
    return launch_overlapped(d.fn, dim3((unsigned)grid), dim3(d.threads), args, d.smem, stream);
}

}  // namespace gbfft
