// Queue, descriptor and parameter structures of the ragged kernels (fft_ragged.cu,
// fft_ragged_pipe.cu).
#pragma once
#include "gbfft_internal.h"
#include "gbfft_plan.h"
#include "gbfft_ragged.h"
#include "fft_tiles.cuh"

namespace gbfft {

constexpr int kRagThreads = 512;
constexpr int kRagMaxLogN = 18;
constexpr int kRagRowsMaxLogN = 13;

struct RagXform {
    uint64_t offset;     // complex samples from the start of in/out
    uint64_t ws_offset;  // two-pass transforms: start of their workspace slice
    int32_t logn;
    int32_t dir;         // GBFFT_FORWARD / GBFFT_INVERSE
    uint32_t tiles1;     // two-pass transforms: number of first-pass items
    uint32_t pad;
};

struct RagItem {
    uint32_t kind;
    uint32_t a;  // kind 0: first index into order[]; kind 1/2: transform id
    uint32_t b;  // kind 0: transforms in the item;   kind 1/2: tile index
    uint32_t logn;
};

struct RagParams {
    const float2 *in;
    float2 *out;
    float2 *ws;
    int p1_to_out;  // out of place: first-pass output goes to `out` (ws unused)
    const RagItem *items;
    uint32_t nitems;
    uint32_t spin_limit;
    const RagXform *xf;
    const uint32_t *order;
    uint32_t *item_counter;
    uint32_t *done1;
    uint32_t *error;
    uint32_t *exits;        // CTAs that have left
    uint32_t *host_error;   // pinned host word: set by the last CTA of a launch that gave up; the host clears it
    uint32_t counters;      // words from item_counter on: zero before and after a launch
    const float2 *sub[16];   // sub-pass tables of a length-2^L in-SMEM FFT
    const float2 *lo[kRagMaxLogN + 1];
    const float2 *hi[kRagMaxLogN + 1];
    int split[kRagMaxLogN + 1];
};

__host__ __device__ constexpr int rag_logr1(int L) { return L / 2 + (L & 1); }
__host__ __device__ constexpr int rag_logr2(int L) { return L / 2; }
__host__ __device__ constexpr int rag_groups(int logr) { return kRagThreads / (kCols << (logr - 4)); }

__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// End of every CTA.  The last one reports the error flag to the host and zeroes the
// counters for the next launch, so that a launch is one kernel.  A memset before it and
// a copy of the flag after it were two more nodes of the graph: 300 transforms of
// 2^0..2^8 11.6 -> 9.3 us, 1000 of 2^8..2^12 15.7 -> 12.9, 200 of 2^8..2^18 73 -> 68
// (10,000, without the pause between launches, 2090 -> 2109).
template <int THREADS>
__device__ __forceinline__ void rag_finish(const RagParams &P, int *flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        *flag = atomicAdd(P.exits, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!*flag) return;
    __threadfence();
    // (set only: a good launch after it must not take an unread report back)
    if (threadIdx.x == 0 && *(volatile uint32_t *)P.error != 0u) *(volatile uint32_t *)P.host_error = 1u;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < P.counters; i += THREADS) P.item_counter[i] = 0u;
}

// ---- the warp-column form (fft_ragged_pipe.cu) ------------------------------
// A queue item in the ring, with all that its tile needs of its transform.
struct alignas(16) RagPipeItem {
    uint64_t offset;  // two-pass items: the transform's first sample
    uint32_t id;      // transform; kind 0: first index into order[]
    uint32_t tile;    // tile of the pass; kind 0: transforms in the item
    uint32_t kind;    // 0, 1, 2 as RagItem; kRagEnd
    uint32_t logn;
    int32_t dir;
    uint32_t tiles1;  // first-pass items of the transform
};
constexpr uint32_t kRagEnd = 3;

// Radices of the two passes there: 2^15 takes 2^7 first, so that the factors of a
// second-pass tile of every size but 2^14 fit the ring.
__host__ __device__ constexpr int rag_pipe_logr1(int L) { return L == 15 ? 7 : rag_logr1(L); }
__host__ __device__ constexpr int rag_pipe_logr2(int L) { return L - rag_pipe_logr1(L); }

struct RagPipeTables {
    const float2 *sub9, *sub13;                 // 32-sample sub-pass tables of 2^9 and 2^13 points
    const float4 *fact[kRagMaxLogN + 1 - 14];   // inter-pass factors of 2^14 .. 2^18
};

cudaError_t ragged_pipe_prepare();
cudaError_t ragged_pipe_launch(const RagParams &P, const RagPipeTables &t, uint64_t extent, int sms, cudaStream_t stream);

}  // namespace gbfft
