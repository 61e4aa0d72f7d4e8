// Ragged batches out of place, FP32, as the warp-column pass pairs run them
// (fft_pipe.cuh): the ring of tiles, loader, storer and compute roles, fed by the
// ragged queue (fft_ragged.cu: the same items, a longer lag).
//
// The barrier form spent its time as the fused pairs did: each 512-thread CTA in
// lock-step from its loads to its stores (1250 transforms of 2^8 .. 2^18: 370 us,
// 2.7 TB/s of the input and output).  Here, 310 us (3.2 TB/s), an item is a 64 KB tile that the loader thread brings in while
// two groups of 8 warps work on the ones before it:
//   * two-pass transforms (N = 2^14 .. 2^18): [R rows][8192 / R columns] boxes.  A
//     transform may start at any even sample, so one tensor map a size describes
//     the whole buffer as rows of N / R samples in which a row may be read from any
//     column on into the next row (extent 2 N / R at a pitch of N / R): sample
//     offset o is column o mod N / R of row o div N / R.
//   * groups of single-pass transforms (N <= 2^13): the compute group reads and
//     writes them itself, with the slot as its exchange buffer.
// What is left is the pass pairs' own bound (data written, read back and rewritten
// through L2) and the two tile radices a size mix alternates between.  96 registers a
// thread; the bodies of 2^9 .. 2^13 single-pass groups spill, which a mix with few of
// them does not see.  Waiting, publication and bounded waits as in fft_pipe.cuh.
#include <algorithm>
#include <cstring>

#include "fft_ragged.cuh"
#include "fft_pipe.cuh"
#include "tensor_map.h"

namespace gbfft {

namespace {

struct RagPipe {
    static constexpr int LOGTILE = 13, GROUPS = 2, SLOTS = 3, WPG = 8, COMPUTE = GROUPS * WPG;
    static constexpr int THREADS = (COMPUTE + 2) * 32;
    static constexpr uint32_t TILE_BYTES = 8u << LOGTILE;
    using K7 = PairTile<7, LOGTILE>;
    using K8 = PairTile<8, LOGTILE>;
    using K9 = ColTile<9, LOGTILE>;
    static_assert(K7::WARPS == WPG && K8::WARPS == WPG && K9::WARPS == WPG, "a group of warps takes a tile");
    // shared memory: tiles | factors a slot (2^14's, 12 KB a tile, stay in global
    // memory) | sub-pass tables | items, mbarriers, flags
    static constexpr int TW_BYTES = K8::TW_BYTES > K9::TW_BYTES ? K8::TW_BYTES : K9::TW_BYTES;
    static constexpr int OFF_TW = SLOTS * (int)TILE_BYTES;
    static constexpr int OFF_SUB7 = OFF_TW + SLOTS * TW_BYTES;
    static constexpr int OFF_SUB8 = OFF_SUB7 + K7::SUB_BYTES;
    static constexpr int OFF_SUB9 = OFF_SUB8 + K8::SUB_BYTES;
    static constexpr int OFF_ITEMS = OFF_SUB9 + K9::SUB_BYTES;
    static constexpr int OFF_BARS = OFF_ITEMS + 2 * SLOTS * (int)sizeof(RagPipeItem);
    static constexpr size_t SMEM = (size_t)OFF_BARS + (SLOTS + 6 * SLOTS) * 8 + 16;
    static_assert(SMEM <= 227 * 1024, "shared memory of a CTA");
};

struct RagPipeParams {
    CUtensorMap in[5], out[5];  // by log2 N - 14: first-pass input, second-pass input and output
    RagPipeTables t;
    RagParams r;
};

struct RagBars {
    uint64_t *free, *full, *done, *retired;
    RagPipeItem *item;
    volatile int *abort;
};

// Boxes of a tile of radix 2^logr: 8192 / R columns in boxes of 16, at most 256 rows each.
template <class F>
__device__ __forceinline__ void rag_boxes(uint32_t slot, int logr, F f) {
    const int R = 1 << logr, rows = R < 256 ? R : 256, cols = 8192 >> logr;
    for (int cb = 0; cb < cols; cb += 16)
        for (int r = 0; r < R; r += rows) f(slot + (uint32_t)(cb / 16 * R + r) * 128u, cb, r);
}

// Coordinates of column `col` of the pass's tile space, row r, of the transform at `offset`.
__device__ __forceinline__ void rag_xy(const RagPipeItem &it, int logr, uint32_t col, int r, int &x, int &y) {
    const int lc = (int)it.logn - logr;  // log2 of the columns
    x = 2 * (int)((uint32_t)(it.offset & ((1ull << lc) - 1)) + col);
    y = (int)(it.offset >> lc) + r;
}

__device__ __forceinline__ void rag_loader(const RagPipeParams &P, uint8_t *smem, const RagBars &B) {
    constexpr uint32_t S = RagPipe::SLOTS, D = 2 * S;
    const RagParams &R = P.r;
    const uint64_t first = l2_evict_first(), normal = l2_evict_normal();
    const bool once = R.nitems <= gridDim.x;
    auto claim = [&]() { return once ? kPipeEnd : atomicAdd(R.item_counter, 1u); };
    auto fetch = [&](uint32_t idx) {
        RagPipeItem it;
        it.kind = kRagEnd;
        if (idx < R.nitems) {
            const RagItem q = R.items[idx];
            it = RagPipeItem{0, q.a, q.b, q.kind, q.logn, 0, 0};
            if (q.kind != 0) {
                const RagXform x = R.xf[q.a];
                it.offset = x.offset;
                it.dir = x.dir;
                it.tiles1 = x.tiles1;
            }
        }
        return it;
    };
    // claims two ahead and items one ahead: no round trip delays a load
    RagPipeItem next = fetch(atomicAdd(R.item_counter, 1u));
    uint32_t claimed = claim();
    uint32_t i = 0;
    bool ok = true;
    for (; next.kind != kRagEnd; ++i) {
        const RagPipeItem it = next;
        const uint32_t s = i % S;
        next = fetch(claimed);
        claimed = claim();
        if (it.kind == 2) {
            uint32_t polls = 0;
            while (ld_acquire_gpu(R.done1 + it.id) < it.tiles1) {
                // no more items either once some CTA has given up
                if (++polls > R.spin_limit || *B.abort || *(volatile uint32_t *)R.error != 0u) {
                    ok = false;
                    break;
                }
                __nanosleep(64);
            }
            if (!ok) break;
            fence_proxy_async_global();  // the acquired data before the TMA's reads
        }
        if (i >= D && !(ok = pipe_wait(B.retired + i % D, (i / D - 1) & 1u, B.abort))) break;
        if (i >= S && !(ok = pipe_wait(B.free + s, (i / S - 1) & 1u, B.abort))) break;
        B.item[i % D] = it;
        uint64_t *bar = B.full + i % D;
        if (it.kind == 0) {
            mbar_arrive(bar);
            continue;
        }
        const int m = (int)it.logn - 14;
        const bool a = it.kind == 1;
        const int logr = a ? rag_pipe_logr1(it.logn) : rag_pipe_logr2(it.logn);
        const bool factors = !a && it.logn > 14;
        const uint32_t tw = !factors ? 0u : (uint32_t)(logr == 8 ? RagPipe::K8::TW_BYTES : RagPipe::K9::TW_BYTES);
        mbar_expect(bar, RagPipe::TILE_BYTES + tw);
        const uint32_t col0 = it.tile * (8192u >> logr);
        rag_boxes(smem_u32(smem) + s * RagPipe::TILE_BYTES, logr, [&](uint32_t dst, int cb, int r) {
            int x, y;
            rag_xy(it, logr, col0 + cb, r, x, y);
            tma_load_box(dst, a ? &P.in[m] : &P.out[m], x, y, 0, smem_u32(bar), a ? first : normal);
        });
        if (factors)
            bulk_load(smem_u32(smem) + RagPipe::OFF_TW + s * RagPipe::TW_BYTES,
                      P.t.fact[m] + (size_t)it.tile * (tw / 16), tw, smem_u32(bar));
    }
    for (uint32_t e = 0; ok && e < (uint32_t)RagPipe::GROUPS; ++e) {
        const uint32_t n = i + e;
        if (n >= D && !(ok = pipe_wait(B.retired + n % D, (n / D - 1) & 1u, B.abort))) break;
        if (n >= S && !(ok = pipe_wait(B.free + n % S, (n / S - 1) & 1u, B.abort))) break;
        B.item[n % D].kind = kRagEnd;
        mbar_arrive(B.full + n % D);
    }
    if (!ok) {
        // a wait gave up: tell the other roles and the host, then let this CTA's loads
        // land before its shared memory goes away
        *B.abort = 1;
        atomicExch(R.error, 1u);
        for (uint32_t n = i > S ? i - S : 0; n < i; ++n)
            for (uint32_t polls = 0; polls < (1u << 20) && !mbar_try_wait(B.full + n % D, (n / D) & 1u); ++polls) {
            }
    }
}

__device__ __forceinline__ void rag_storer(const RagPipeParams &P, uint8_t *smem, const RagBars &B) {
    constexpr uint32_t S = RagPipe::SLOTS, D = 2 * S;
    const uint64_t first = l2_evict_first();
    for (uint32_t i = 0;; ++i) {
        const uint32_t s = i % S;
        if (!pipe_wait(B.done + i % D, (i / D) & 1u, B.abort)) {
            *B.abort = 1;
            atomicExch(P.r.error, 1u);
            break;
        }
        const RagPipeItem it = B.item[i % D];
        mbar_arrive(B.retired + i % D);  // the ring entry is read
        if (it.kind == kRagEnd) break;
        if (it.kind == 1) {
            red_release(P.r.done1 + it.id);
        } else if (it.kind == 2) {
            const int logr = rag_pipe_logr2(it.logn);
            const uint32_t col0 = it.tile * (8192u >> logr);
            rag_boxes(smem_u32(smem) + s * RagPipe::TILE_BYTES, logr, [&](uint32_t src, int cb, int r) {
                int x, y;
                rag_xy(it, logr, col0 + cb, r, x, y);
                tma_store_box(&P.out[it.logn - 14], x, y, 0, src, first);
            });
            bulk_commit();
            bulk_wait_read();
            mbar_arrive(B.free + s, RagPipe::WPG);
        }
    }
    bulk_wait_all();
}

// A two-pass item of radix 2^LOGR on a landed tile.  The item is read from the ring
// each time it is needed: held in registers across the butterflies it costs spills.
template <class K, int LOGR>
__device__ __forceinline__ void rag_tile(const RagPipeParams &P, const volatile RagPipeItem &it, uint8_t *slot,
                                         const uint8_t *sub, const float4 *tab, int group, int warp, int lane,
                                         uint64_t *free) {
    typename K::Values v;
    int t, c;
    K::place(warp, lane, t, c);
    K::run(
        slot, t, c, sub, v, group,
        [&](typename K::Values &x) {
            if (it.kind == 1) K::conj(x, it.dir == GBFFT_INVERSE ? -1.0f : 1.0f);
            else K::twiddle(tab, t, c, x);
        },
        [&] {
            if (it.kind == 1) {  // the slot is read: the loader may have it
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(free);
            }
        });
    if (it.kind == 1) {
        const uint32_t col = it.tile * (8192u >> LOGR) + (uint32_t)c;
        K::store_columns(P.r.out + it.offset + ((uint64_t)col << LOGR), t, v, l2_evict_last());
    } else {
        const bool inv = it.dir == GBFFT_INVERSE;
        const float sc = inv ? __uint_as_float((127u - it.logn) << 23) : 1.0f;
        K::scale(v, sc, inv ? -sc : sc);
        K::stage(slot, t, c, v, group);
    }
}

// Butterflies of a group of 256 threads with a barrier of its own.
struct RagGroup : DftRegs {
    static constexpr int group_threads = 256;
    int barrier;
};

template <int L, int LE>
__device__ __forceinline__ void rag_group_rows(const RagParams &P, const float2 *tw, const volatile RagPipeItem &item,
                                               float2 *buf, RagGroup eng) {
    constexpr int G = 256 / SubCfg<L, LE>::T;  // transforms a round
    const struct { uint32_t id, tile; } it{item.id, item.tile};
    for (uint32_t g0 = 0; g0 < it.tile; g0 += G) {
        auto ref = [&](int g) {
            const bool act = g0 + (uint32_t)g < it.tile;
            const RagXform x = P.xf[P.order[it.id + (act ? g0 + g : 0)]];
            const bool inv = x.dir == GBFFT_INVERSE;
            const float sc = inv ? ldexpf(1.0f, -L) : 1.0f;
            return RowRef{P.in + x.offset, P.out + x.offset, act, inv ? -1.0f : 1.0f, sc, inv ? -sc : 1.0f, 0u};
        };
        rows_tile<L, G, 0, LE>(ref, tw, buf, LoadOps{nullptr, 0u, 0.f, 0u}, eng);
        tile_sync(eng);  // the buffer is reused
    }
}

__global__ void __launch_bounds__(RagPipe::THREADS, 1) fft_ragged_pipe_kernel(const __grid_constant__ RagPipeParams P) {
    using C = RagPipe;
    extern __shared__ __align__(1024) uint8_t smem_rp[];
    constexpr int S = C::SLOTS, D = 2 * S;
    uint64_t *bars = (uint64_t *)(smem_rp + C::OFF_BARS);
    int *s_abort = (int *)(bars + S + 3 * D);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const RagBars B{bars, bars + S, bars + S + D, bars + S + 2 * D, (RagPipeItem *)(smem_rp + C::OFF_ITEMS), s_abort};
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) mbar_init(B.free + s, C::WPG);
        for (int s = 0; s < D; ++s) {
            mbar_init(B.full + s, 1);
            mbar_init(B.done + s, C::WPG);
            mbar_init(B.retired + s, 1);
        }
        *s_abort = 0;
    }
    if (P.r.sub[7]) C::K7::fill_sub(smem_rp + C::OFF_SUB7, P.r.sub[7], threadIdx.x, C::THREADS);
    if (P.r.sub[8]) C::K8::fill_sub(smem_rp + C::OFF_SUB8, P.r.sub[8], threadIdx.x, C::THREADS);
    if (P.t.sub9) C::K9::fill_sub(smem_rp + C::OFF_SUB9, P.t.sub9, threadIdx.x, C::THREADS);
    stream_wait();  // (the tables above are complete before a plan's first launch)
    __syncthreads();
    if (warp == C::COMPUTE) {
        if (lane == 0) rag_loader(P, smem_rp, B);
    } else if (warp == C::COMPUTE + 1) {
        if (lane == 0) rag_storer(P, smem_rp, B);
    } else {
        const int cg = warp / C::WPG, wg = warp % C::WPG;
        RagGroup eng;
        eng.barrier = 1 + cg;
        for (uint32_t i = (uint32_t)cg;; i += C::GROUPS) {
            const uint32_t s = i % S;
            // the group's warps share a barrier: they go on or leave together
            const bool ok = __all_sync(0xffffffffu, pipe_wait(B.full + i % D, (i / D) & 1u, B.abort));
            if (!group_all(3 + cg, C::WPG * 32, ok)) {
                if (lane == 0) {
                    *B.abort = 1;
                    atomicExch(P.r.error, 1u);
                }
                break;
            }
            const volatile RagPipeItem &it = B.item[i % D];
            const uint32_t kind = it.kind;
            uint8_t *slot = smem_rp + s * C::TILE_BYTES;
            if (kind == 0) {
                switch (it.logn) {
#define GBFFT_RP_ROWS(L) \
        case L: rag_group_rows<L, 4>(P.r, P.r.sub[L], it, (float2 *)slot, eng); break;
                    GBFFT_RP_ROWS(0) GBFFT_RP_ROWS(1) GBFFT_RP_ROWS(2) GBFFT_RP_ROWS(3) GBFFT_RP_ROWS(4)
                    GBFFT_RP_ROWS(5) GBFFT_RP_ROWS(6) GBFFT_RP_ROWS(7) GBFFT_RP_ROWS(8) GBFFT_RP_ROWS(9)
                    GBFFT_RP_ROWS(10) GBFFT_RP_ROWS(11) GBFFT_RP_ROWS(12)
#undef GBFFT_RP_ROWS
                    case 13: rag_group_rows<13, 5>(P.r, P.t.sub13, it, (float2 *)slot, eng); break;
                    default: break;
                }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(B.free + s);
            } else if (kind != kRagEnd) {
                const int logr = kind == 1 ? rag_pipe_logr1(it.logn) : rag_pipe_logr2(it.logn);
                const float4 *tab = (const float4 *)(smem_rp + C::OFF_TW + s * C::TW_BYTES);
                if (logr == 7) {
                    // (second passes of radix 2^7 are 2^14's: factors from global memory)
                    rag_tile<C::K7, 7>(P, it, slot, smem_rp + C::OFF_SUB7,
                                       P.t.fact[0] + (size_t)it.tile * (C::K7::TW_BYTES / 16), cg, wg, lane, B.free + s);
                } else if (logr == 8) {
                    rag_tile<C::K8, 8>(P, it, slot, smem_rp + C::OFF_SUB8, tab, cg, wg, lane, B.free + s);
                } else {
                    rag_tile<C::K9, 9>(P, it, slot, smem_rp + C::OFF_SUB9, tab, cg, wg, lane, B.free + s);
                }
                fence_proxy_async_smem();  // this lane's accesses of the slot before the TMA's
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(B.done + i % D);
            if (kind == kRagEnd) break;
        }
    }
    // the loader's and the storer's other lanes are here already: the barrier below is a
    // whole warp's
    __syncwarp();
    __syncthreads();  // (s_abort is no longer read)
    rag_finish<C::THREADS>(P.r, s_abort);
}

}  // namespace

cudaError_t ragged_pipe_prepare() {
    return cudaFuncSetAttribute((const void *)fft_ragged_pipe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)RagPipe::SMEM);
}

cudaError_t ragged_pipe_launch(const RagParams &P, const RagPipeTables &t, uint64_t extent, int sms, cudaStream_t stream) {
    PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    if (!encode) return cudaErrorNotSupported;
    RagPipeParams Q;
    memset(&Q, 0, sizeof Q);
    Q.t = t;
    Q.r = P;
    for (int L = 14; L <= kRagMaxLogN; ++L) {
        if (!t.fact[L - 14]) continue;
        for (int pass = 0; pass < 2; ++pass) {
            const int logr = pass ? rag_pipe_logr2(L) : rag_pipe_logr1(L);
            const uint64_t cols = 1ull << (L - logr), rows = std::max<uint64_t>(1, extent >> (L - logr));
            const cuuint64_t dims[3] = {4 * cols, rows, 1}, strides[2] = {cols * sizeof(float2), rows * cols * sizeof(float2)};
            const cuuint32_t box[3] = {32, (cuuint32_t)std::min(256, 1 << logr), 1}, estr[3] = {1, 1, 1};
            if (encode(pass ? &Q.out[L - 14] : &Q.in[L - 14], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                       pass ? (void *)P.out : (void *)P.in, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return cudaErrorInvalidValue;
        }
    }
    void *args[] = {(void *)&Q};
    return launch_overlapped((const void *)fft_ragged_pipe_kernel, dim3(std::min<unsigned>(P.nitems, (unsigned)std::max(1, sms))),
                         dim3(RagPipe::THREADS), args, RagPipe::SMEM, stream);
}

}  // namespace gbfft
