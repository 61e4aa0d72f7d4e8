// Split-precision tensor-core form of the single-pass transform (N = 2^4 .. 2^14),
// replacing, like fft_rows.cu, the reference's per-stage global passes
// (larsjoost/wgls-rs-fft src/shaders.rs:8-106, dispatched by src/lib.rs:582-628).
//
// The same tile as fft_rows.cu -- G whole transforms a CTA, 16 samples a
// thread, radix-16 sub-passes with shared-memory exchanges, one HBM read and
// one write per sample -- with every radix-16 butterfly set run on the tcgen05
// tensor cores (fft_tc.cuh; the radix 2/4/8 remainder stays on the FP32
// pipes).  Two forms:
//   * one-shot, one CTA per tile of 4096 samples, which sets up TMEM, the
//     mbarrier and the G parts for its one tile: launches of a few waves;
//   * a persistent loop over tiles of 2048 samples, which sets them up once for
//     its whole run and brings the next tile toward L2 while one is computed:
//     everything larger.  512 MB each way, one-shot -> loop: N = 2^8 FP16 218 ->
//     191 us, TF32 349 -> 257, BF16 x 6 298 -> 242; 2^11 253 -> 229, 404 -> 293,
//     334 -> 281; 2^12 TF32 467 -> 427, BF16 x 6 411 -> 384; 2^13 730 -> 597, 500 ->
//     472; 2^14 FP16 513 -> 468.
// Every completion wait is bounded.
// TF32 needs 256 B of operands per thread, so it stops at N = 2^13.
#pragma once
#include "gbfft_internal.h"
#include "gbfft_plan.h"
#include "fft_tc.cuh"
#include "fft_tiles.cuh"

namespace gbfft {

__host__ __device__ constexpr uint32_t rtc_tmem_cols(int nmma) {
    return nmma * 32 <= 32 ? 32 : (nmma * 32 <= 64 ? 64 : (nmma * 32 <= 128 ? 128 : 256));
}

template <int LOGN, int KIND, bool LOOP>
struct RowsTcCfg {
    using S = SubCfg<LOGN>;
    using Gm = TcGeom<KIND>;
    static_assert(LOGN >= 4, "a radix-16 sub-pass needs 16 samples a thread");
    // Samples a CTA (one transform above that).  One-shot: 4096, as the FP32 tile.
    // Tile loop: 2048 -- 128 threads, one M = 128 product a sub-pass, eight CTAs an
    // SM whose barriers and MMA round trips interleave.
    static constexpr int TILE = LOOP ? 2048 : 4096;
    static constexpr int G = S::N >= TILE ? 1 : TILE / S::N;
    static constexpr int THREADS = G * S::T;
    static_assert(THREADS % 128 == 0, "one M = 128 MMA per 128 threads");
    static constexpr int NMMA = THREADS / 128;
    static constexpr uint32_t TMEM_COLS = rtc_tmem_cols(NMMA);
    static constexpr size_t TILE_BYTES = (size_t)G * rows_buf_stride<LOGN>() * sizeof(float2);
    static constexpr size_t A_BYTES = (size_t)THREADS * Gm::ROW_BYTES;
    static constexpr size_t A_ALL = Gm::PARTS * A_BYTES;
    // the A operand parts alias the exchange tile (tc_dft16 waits for its readers)
    static constexpr size_t REGION = ((A_ALL > TILE_BYTES ? A_ALL : TILE_BYTES) + 1023) & ~(size_t)1023;
    static constexpr size_t OFF_G = REGION;
    static constexpr size_t OFF_MISC = OFF_G + Gm::PARTS * (size_t)Gm::G_BYTES;
    static constexpr size_t SMEM = OFF_MISC + 64;
    // CTAs an SM: by registers (64 a thread) and shared memory (1 KB reserved a CTA)
    static constexpr int FIT = (int)((228u * 1024u) / (SMEM + 1024u));
    static constexpr int MINB = !LOOP ? (THREADS >= 1024 ? 1 : (THREADS >= 512 ? 2 : 4))
                                      : (1024 / THREADS < FIT ? 1024 / THREADS : FIT);
    static_assert(MINB >= 1 && MINB * TMEM_COLS <= 512, "tensor memory of an SM");
    // Where the loop is built: not for the 16-bit kinds at 2^12 and 2^13, whose one-shot
    // tiles are as large and as many an SM (2^13 FP16, 2048 transforms: 102.4 us one-shot,
    // 108.8 looped in 6.7 rounds; 8192: 393, 383), nor for BF16 x 6 at 2^14 (2896 transforms:
    // 467.6, 480.4; 588: 95.6, 100.2)
    static constexpr bool HAS_LOOP = LOGN < 12 || Gm::ELEM == 4 || (Gm::PARTS == 3 ? LOGN < 14 : LOGN == 14);
};

template <int LOGN, int DIRC, int KIND, bool LOOP>
__global__ void __launch_bounds__(RowsTcCfg<LOGN, KIND, LOOP>::THREADS, RowsTcCfg<LOGN, KIND, LOOP>::MINB)
fft_rows_tc_kernel(const float2 *in, float2 *out, uint64_t batch, const float2 *__restrict__ tw,
                   float in_im_sign, float out_re_scale, float out_im_scale, LoadOps ops,
                   const uint4 *__restrict__ gtab, uint32_t *err) {
    stream_order();
    using C = RowsTcCfg<LOGN, KIND, LOOP>;
    using Gm = TcGeom<KIND>;
    extern __shared__ __align__(1024) uint8_t smem_rtc[];
    uint64_t *bar = (uint64_t *)(smem_rtc + C::OFF_MISC);
    uint32_t *s_taddr = (uint32_t *)(smem_rtc + C::OFF_MISC + 8);
    int *s_abort = (int *)(smem_rtc + C::OFF_MISC + 12);
    const int tid = threadIdx.x;
    const uint4 *gsrc = gtab + Gm::GTAB_OFF / 16;
    uint4 *gdst = (uint4 *)(smem_rtc + C::OFF_G);
    for (int i = tid; i < Gm::PARTS * Gm::G_BYTES / 16; i += C::THREADS) gdst[i] = gsrc[i];
    if (tid < 32) tmem_alloc(s_taddr, C::TMEM_COLS);
    if (tid == 0) {
        mbar_init(bar, 1);
        *s_abort = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    TcState st;
    tc_state_parts<KIND>(st, smem_rtc, C::A_BYTES, smem_rtc + C::OFF_G);
    st.bar = bar;
    st.abort = s_abort;
    st.err = err;
    st.taddr = *s_taddr;
    st.parity = 0;
    st.nmma = C::NMMA;
    st.spin_limit = kTcSpinLimit;

    for (uint64_t tile = blockIdx.x;;) {
        if constexpr (LOOP) {
            // the next tile's samples toward L2: one 128-byte line a thread
            const uint64_t next = tile + gridDim.x;
            if (next * C::G + (uint32_t)tid / C::S::T < batch)
                prefetch_l2(in + next * (C::G * C::S::N) + (uint32_t)tid * 16u);
        }
        auto ref = [&](int g) {
            const uint64_t row = tile * C::G + g;
            return RowRef{in + row * C::S::N, out + row * C::S::N, row < batch, in_im_sign, out_re_scale,
                          out_im_scale, (uint32_t)row};
        };
        rows_tile<LOGN, C::G, DIRC, 4>(ref, tw, (float2 *)smem_rtc, ops, DftTc<KIND>{&st});
        if constexpr (!LOOP) break;
        __syncthreads();  // shared memory is reused by the next tile
        tile += gridDim.x;
        if (tile * C::G >= batch || *s_abort) break;
    }

    tc_fence_before();
    __syncthreads();
    if (tid == 0 && *s_abort) {
        // a wait gave up: let the MMAs that were issued finish before freeing TMEM
        for (uint32_t polls = 0; polls < kTcSpinLimit && !mbar_try_wait(bar, st.parity ^ 1u); ++polls) {
        }
    }
    __syncthreads();
    tc_fence_after();
    if (tid < 32) tmem_dealloc(st.taddr, C::TMEM_COLS);
}

template <int LOGN, int KIND>
void rows_tc_describe(RowsKernelInfo &k) {
    using C = RowsTcCfg<LOGN, KIND, false>;
    using L = RowsTcCfg<LOGN, KIND, true>;
    k.fn = (const void *)fft_rows_tc_kernel<LOGN, -1, KIND, false>;
    k.fn_inv = (const void *)fft_rows_tc_kernel<LOGN, 1, KIND, false>;
    k.threads = C::THREADS;
    k.transforms_per_cta = C::G;
    k.smem = C::SMEM;
    k.fn_persistent = nullptr;
    k.fn_persistent_inv = nullptr;
    if constexpr (L::HAS_LOOP) {
        k.fn_persistent = (const void *)fft_rows_tc_kernel<LOGN, -1, KIND, true>;
        k.fn_persistent_inv = (const void *)fft_rows_tc_kernel<LOGN, 1, KIND, true>;
    }
    k.persist_ctas_per_sm = L::MINB;
    k.persist_threads = L::THREADS;
    k.persist_transforms = L::G;
    k.persist_smem = L::SMEM;
    k.nseg = subcfg_segments<LOGN>(k.segs, 0);
    k.tw_entries = SubCfg<LOGN>::tw_entries();
}

template <int KIND>
bool rows_tc_info_kind(int logn, RowsKernelInfo &k) {
    switch (logn) {
#define GBFFT_RTC(L) \
    case L: rows_tc_describe<L, KIND>(k); return true;
        GBFFT_RTC(4) GBFFT_RTC(5) GBFFT_RTC(6) GBFFT_RTC(7) GBFFT_RTC(8) GBFFT_RTC(9) GBFFT_RTC(10)
        GBFFT_RTC(11) GBFFT_RTC(12) GBFFT_RTC(13)
#undef GBFFT_RTC
        case 14:
            if constexpr (KIND == kTcTF32) return false;  // 256 KB of TF32 operands
            else {
                rows_tc_describe<14, KIND>(k);
                return true;
            }
        default: return false;
    }
}

}  // namespace gbfft
