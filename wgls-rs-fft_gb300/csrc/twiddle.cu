// Device-side twiddle-table generation.  Every table entry is computed in
// FP64 with sincospi on an exactly representable argument (2 e / M, M a power
// of two) and rounded once to FP32.  This is the one step of the transform
// kept in FP64.  The reference builds its table on the host from an f32 angle
// (larsjoost/wgls-rs-fft src/lib.rs:761-769), whose rounding reaches ~ulp(2 pi).
#include "gbfft_internal.h"
#include "gbfft_plan.h"
#include "fft_tiles.cuh"

namespace gbfft {

constexpr int kMaxSegments = 32;

struct SegmentList {
    TwiddleSegment s[kMaxSegments];
    int n;
};

__global__ void twiddle_fill_kernel(float2 *table, SegmentList list, uint64_t total) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    // locate the segment (segments are few; linear scan over prefix counts)
    uint64_t base = 0;
    int s = 0;
    for (; s < list.n; ++s) {
        if (i < base + list.s[s].count) break;
        base += list.s[s].count;
    }
    if (s >= list.n) return;
    const TwiddleSegment seg = list.s[s];
    const uint64_t li = i - base;
    uint64_t e;
    if (seg.kind == 0) {
        const uint64_t p = 1ull << seg.logp;
        e = (li / p + 1) * (li % p);
    } else {
        e = li << seg.logstride;
    }
    const uint64_t m = 1ull << seg.logm;
    e &= (m - 1);
    // angle = -2 pi e / M  ->  sincospi(-2 e / M); 2e/M is exact in FP64.
    const double x = -2.0 * (double)e / (double)m;
    double sn, cs;
    sincospi(x, &sn, &cs);
    table[seg.offset + li] = make_float2((float)cs, (float)sn);
}

cudaError_t twiddle_fill(float2 *table, const TwiddleSegment *segs, int nseg, cudaStream_t stream) {
    if (nseg <= 0) return cudaSuccess;
    if (nseg > kMaxSegments) return cudaErrorInvalidValue;
    SegmentList list;
    uint64_t total = 0;
    for (int i = 0; i < nseg; ++i) {
        list.s[i] = segs[i];
        total += segs[i].count;
    }
    list.n = nseg;
    if (total == 0) return cudaSuccess;
    const unsigned threads = 256;
    const uint64_t blocks = (total + threads - 1) / threads;
    twiddle_fill_kernel<<<(unsigned)blocks, threads, 0, stream>>>(table, list, total);
    return cudaGetLastError();
}

// Inter-pass factors of a warp-column pass (gbfft_plan.h), one float4 a thread:
// products of the two-level table's entries, as every other form of the pass
// computes them, so that all forms give the same bits.
__global__ void factors_fill_kernel(float4 *out, const float2 *__restrict__ lo, const float2 *__restrict__ hi,
                                    int split, int logn, int logr, int logp, int loge, int logtile, int soa,
                                    uint64_t total) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int logt = logr - loge, E = 1 << loge, T = 1 << logt;
    const uint32_t pairs = 1u << (logtile - logr - 1);  // column pairs of a tile
    const uint32_t per = pairs * (uint32_t)(E + T);
    const uint64_t tile = i / per;
    uint32_t r = (uint32_t)(i % per);
    const bool f = r < pairs * (uint32_t)E;
    if (!f) r -= pairs * (uint32_t)E;
    const uint32_t k = 2 * ((uint32_t)tile * pairs + (f ? r >> loge : r >> logt));
    // W_{R p}^{k T e} or W_{R p}^{k t} as a power of W_N
    const uint32_t m = f ? r & (uint32_t)(E - 1) : r & (uint32_t)(T - 1);
    const int sh = logn - logp - (f ? loge : logr);
    const float2 a = twiddle_2level(lo, hi, (k * m) << sh, split);
    const float2 b = twiddle_2level(lo, hi, ((k + 1) * m) << sh, split);
    out[i] = soa ? make_float4(a.x, b.x, a.y, b.y) : make_float4(a.x, a.y, b.x, b.y);
}

uint64_t factors_count(int logr, int logp, int loge) {
    return ((uint64_t)((1 << loge) + (1 << (logr - loge))) << logp) / 2;
}

cudaError_t factors_fill(float4 *out, const float2 *lo, const float2 *hi, int split, int logn, int logr, int logp,
                         int loge, int logtile, bool soa, cudaStream_t stream) {
    const uint64_t total = factors_count(logr, logp, loge);
    factors_fill_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(out, lo, hi, split, logn, logr, logp,
                                                                            loge, logtile, soa ? 1 : 0, total);
    return cudaGetLastError();
}

// Hann window w_i = 0.5 (1 - cos(2 pi i / (n - 1))) in FP64, rounded once to
// f32 (the formula of the reference's host-side window, tests/test_utils.rs:
// 39-48); n == 1 gives w_0 = 1.
__global__ void hann_fill_kernel(float *w, uint64_t n) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    w[i] = n == 1 ? 1.0f : (float)(0.5 * (1.0 - cospi(2.0 * (double)i / (double)(n - 1))));
}

cudaError_t hann_fill(float *w, uint64_t n, cudaStream_t stream) {
    const unsigned threads = 256;
    hann_fill_kernel<<<(unsigned)((n + threads - 1) / threads), threads, 0, stream>>>(w, n);
    return cudaGetLastError();
}

// A launch that follows another in its stream starts 2 to 4 us after it ends.  As a
// programmatic launch the device brings the next grid up during the one before, and
// stream_wait() holds it until that is complete: a pair of 2^10 x 9 transforms called
// from C 8.2 -> 4.1 us (then the calls themselves), 2^16 x 32 21.0 -> 17.1, 2^18 x 1
// 14.3 -> 11.3, 2^24 x 1 132 -> 120, 2^9 x 100003 119.5 -> 117.3, 2^16 x 1024 231.5 ->
// 229.8.  Into a capture goes an ordinary launch: the graph has edges of its own (and
// starts its nodes 2 us apart), and the node fits whatever body it is put into.
cudaError_t launch_overlapped(const void *fn, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t stream) {
    if (stream_capturing(stream)) return cudaLaunchKernel(fn, grid, block, args, smem, stream);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
}

}  // namespace gbfft
