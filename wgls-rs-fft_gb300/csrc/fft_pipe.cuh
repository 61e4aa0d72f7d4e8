// Two consecutive global passes in one persistent launch, as in fft_fused.cuh
// (same groups, same queue, same L2-resident intermediate), with the tiles
// moved by the tensor memory accelerator and no CTA barrier in the loop.
//
// What held the barrier form back (N = 2^16 x 1024: 297 us, DRAM at 42 %,
// issue at 39 %): every tile ran load -> barrier -> exchange -> barrier ->
// ... in lock-step over 8 warps, so each warp waited for the slowest load of
// the tile and for three to four barriers (6.4 of 20 cycles an instruction),
// and nothing of the next tile was in flight meanwhile.  Here a CTA is a ring
// of SLOTS shared-memory tiles and three roles:
//   * the loader thread claims queue items in order, waits for a B item's group
//     (ctr[2 + group]) and brings the tile in with one to four TMA boxes, and its
//     inter-pass twiddle factors with a bulk copy;
//   * GROUPS groups of compute warps take the slots in turn; a column stays in
//     one warp (fft_warp.cuh), so warps meet only at the slots' mbarriers:
//     `full` (tile and factors are there) and `done` (the group is through);
//   * the storer thread retires slots in order: it stores a staged tile with TMA
//     boxes, hands the slot back (`free`) and publishes pass-A tiles.
// A first pass stores its columns straight from registers (a column's outputs
// are contiguous) and hands the slot back itself, right after its last read;
// every other pass writes its results back into the slot.
//
// Every wait ends: the queue claims are made in order, a tile that has been
// loaded depends on nothing, and the storer publishes a CTA's finished tiles
// whatever its loader is waiting for, so the oldest unfinished item always
// proceeds.  Each wait is bounded all the same; on expiry the launch's error
// flag is raised, every role leaves, and the loader waits (bounded) for its
// copies in flight.
// Pass-A data crosses proxies: the compute warps' stores (generic) or the TMA
// store (async, complete) -> done / bulk-group wait -> release, counter; and
// counter (acquire) -> proxy fence -> TMA load.
#pragma once
#include <cuda.h>

#include "gbfft_plan.h"
#include "fft_fused.cuh"
#include "fft_tc.cuh"
#include "fft_warp.cuh"

namespace gbfft {

template <int LOGR, int LOGTILE, int LE> struct PipeTileOf;
template <int LOGR, int LOGTILE> struct PipeTileOf<LOGR, LOGTILE, 4> { using type = PairTile<LOGR, LOGTILE>; };
template <int LOGR, int LOGTILE> struct PipeTileOf<LOGR, LOGTILE, 5> { using type = ColTile<LOGR, LOGTILE>; };

template <int LOGR, int LOGTILE> struct PipeTileOf<LOGR, LOGTILE, 6> { using type = WideTile<LOGR, LOGTILE>; };

template <int LOGRA, int LOGRB, int LOGN, int LOGPA, int LE>
struct PipeCfg {
    // LE 4 (pair tiles): 32 KB tiles, two groups of 4 warps on three slots, two
    // CTAs an SM.  LE 5 (one column a thread): 64 KB tiles (a radix-2^10 tile of 8
    // columns), two groups of 8 warps on three slots, one CTA an SM; LE 6 (wide
    // tiles, radix 2^10 and 2^11): the same.
    static constexpr int LOGTILE = LE == 4 ? 12 : 13;
    static constexpr int GROUPS = 2, SLOTS = 3;
    static constexpr int WPG = LE == 4 ? 4 : 8;  // warps a group
    static constexpr int MINB = LE == 4 ? 2 : 1;
    static constexpr int COMPUTE = GROUPS * WPG;
    static constexpr int THREADS = (COMPUTE + 2) * 32;
    static constexpr uint32_t TILE_BYTES = 8u << LOGTILE;
    using KA = typename PipeTileOf<LOGRA, LOGTILE, LE>::type;
    using KB = typename PipeTileOf<LOGRB, LOGTILE, LE>::type;
    static_assert(KA::WARPS == WPG && KB::WARPS == WPG, "a group of warps takes a tile");
    static_assert(LOGPA == 0 ? LOGN == LOGRA + LOGRB : (LOGRA == LOGRB && KA::COLS == 16 && LOGPA >= 4),
                  "two-pass transform, or the last two passes (R1, R, R) of three");
    static constexpr bool FIRST_A = LOGPA == 0;
    static constexpr int LOGPB = LOGPA + LOGRA;
    static constexpr uint32_t GPT = FIRST_A ? 1u : (1u << LOGPA) / kCols;
    static constexpr uint32_t T = FIRST_A ? 1u << (LOGN - LOGTILE) : (1u << LOGRB);
    static constexpr uint64_t GROUP_SAMPLES = (uint64_t)T << LOGTILE;
    // shared memory: tiles | per-slot inter-pass factors | sub-pass tables
    static constexpr int TW_BYTES = (!FIRST_A && KA::TW_BYTES > KB::TW_BYTES) ? KA::TW_BYTES : KB::TW_BYTES;
    static constexpr int OFF_TW = SLOTS * (int)TILE_BYTES;
    static constexpr int OFF_SUBA = OFF_TW + SLOTS * TW_BYTES;
    static constexpr int OFF_SUBB = LOGRA == LOGRB ? OFF_SUBA : OFF_SUBA + KA::SUB_BYTES;
    static constexpr int OFF_BARS = OFF_SUBB + KB::SUB_BYTES;  // mbarriers, queue positions, flags
    static constexpr size_t SMEM = (size_t)OFF_BARS + (SLOTS + 6 * SLOTS) * 8 + 2 * SLOTS * 4 + 8;
};

struct PipeParams {
    CUtensorMap map_in;   // pass A's input, [batch][R_A rows][N / R_A columns]
    CUtensorMap map_mid;  // pass A's output (three passes only)
    CUtensorMap map_io;   // the output buffer as pass B reads and writes it
    const float4 *fact_a, *fact_b;  // inter-pass factors, a block of TW_BYTES a tile
    FusedParams f;
};

constexpr uint32_t kPipeEnd = 0xffffffffu;
constexpr uint32_t kPipeBarSpin = 1u << 24;  // mbarrier polls (a few tenths of a second at the least)

// L2 priorities.  Pass A's input and the final values pass through once
// (evict_first); the intermediate is stored with evict_last and read back with
// normal priority, so that its lines are not written to HBM before pass B
// overwrites them (2^16 x 1024: 244.7 -> 239.4 us, 2^22 x 16: 422.8 -> 410.7 us
// against a normal store and an evict_first read).
__device__ __forceinline__ uint64_t l2_evict_first() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_evict_normal() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_evict_last() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void tma_load_box(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar,
                                             uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint "
        "[%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(dst),
        "l"((uint64_t)map), "r"(x), "r"(y), "r"(z), "r"(bar), "l"(policy)
        : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
        "l"((uint64_t)src), "r"(bytes), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_store_box(const CUtensorMap *map, int x, int y, int z, uint32_t src,
                                              uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group.L2::cache_hint [%0, {%1, %2, %3}], [%4], %5;" ::"l"(
            (uint64_t)map),
        "r"(x), "r"(y), "r"(z), "r"(src), "l"(policy)
        : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async_global() {
    asm volatile("fence.proxy.async.global;" ::: "memory");
}
// release at GPU scope of everything this thread has observed, then count
__device__ __forceinline__ void red_release(uint32_t *p) {
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar, uint32_t count = 1) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// Bounded wait of one thread; false once any role of the CTA has given up.
__device__ __forceinline__ bool pipe_wait(uint64_t *bar, uint32_t parity, volatile int *abort) {
    for (uint32_t polls = 0; !mbar_try_wait(bar, parity);)
        if (*abort || ++polls > kPipeBarSpin) return false;
    return true;
}

// Whether `ok` holds for all `threads` threads that meet at named barrier `id`.
__device__ __forceinline__ bool group_all(int id, int threads, bool ok) {
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %3, 0;\n\t"
        "bar.red.and.pred p, %1, %2, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(all)
        : "r"(id), "r"(threads), "r"((uint32_t)ok)
        : "memory");
    return all != 0;
}

// Boxes of a tile: at most 256 rows of BOXC columns each.
template <class K, class F>
__device__ __forceinline__ void pipe_boxes(uint32_t slot, uint32_t col0, F f) {
    constexpr int RB = K::R > 256 ? 256 : K::R;
#pragma unroll
    for (int cb = 0; cb < K::COLS / K::BOXC; ++cb)
#pragma unroll
        for (int r = 0; r < K::R; r += RB)
            f(slot + (uint32_t)(cb * K::R + r) * K::ROWB, 2 * (int)(col0 + cb * K::BOXC), r);
}

// Column 0 of a queue item's tile.
template <class C>
__device__ __forceinline__ uint32_t pipe_col0(bool is_a, uint32_t g, uint32_t tile) {
    if (C::FIRST_A) return tile * (uint32_t)(is_a ? C::KA::COLS : C::KB::COLS);
    return (tile * C::GPT + g) * (uint32_t)kCols;
}

// free: one a slot.  The others and the items' queue positions are rings of twice
// the slots: a first-pass slot is free (and reloaded) before the storer has
// published its tile; and with two groups on three slots a group meets every
// other use of a slot, so a `full` barrier a slot could complete a phase that the
// waiting group never looks at, and the parity of its own phase would be
// ambiguous.  Entry i mod 2 S is always the same group's.
struct PipeBars {
    uint64_t *full, *free, *done, *retired;
    volatile uint32_t *item;
    volatile int *abort;
};

// One thread.
template <class C, int LOGPA>
__device__ __forceinline__ void pipe_loader(const PipeParams &P, uint8_t *smem, const PipeBars &B) {
    const FusedParams &F = P.f;
    constexpr uint32_t T = C::T, GPT = C::GPT, S = C::SLOTS, D = 2 * S;
    const uint64_t first = l2_evict_first(), normal = l2_evict_normal();
    const bool once = F.nitems <= gridDim.x;  // an item a CTA: claiming ahead would leave other CTAs idle
    const uint32_t sbase = smem_u32(smem);
    // two claims ahead: a claim's round trip never delays a load
    uint32_t claim0 = fused_claim(F), claim1 = once ? kPipeEnd : atomicAdd(F.ctr, 1u), i = 0;
    bool ok = true;
    for (; claim0 < F.nitems; ++i) {
        const uint32_t idx = claim0, s = i % S;
        claim0 = claim1;
        claim1 = once ? kPipeEnd : atomicAdd(F.ctr, 1u);
        bool is_a;
        uint32_t grp, tile;
        fused_item<T>(F, idx, is_a, grp, tile);
        const uint32_t b = grp / GPT, g = grp % GPT;
        const uint32_t col0 = pipe_col0<C>(is_a, g, tile);
        if (!is_a) {
            uint32_t polls = 0;
            while (fused_ld_acquire(F.ctr + 2 + grp) < T) {
                // no more items either once some CTA has given up
                if (++polls > F.spin_limit || *B.abort || *(volatile uint32_t *)F.err != 0u) {
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
        B.item[i % D] = idx;
        const uint32_t slot = sbase + s * C::TILE_BYTES, bar = smem_u32(B.full + i % D);
        const bool factors = !is_a || !C::FIRST_A;
        mbar_expect(B.full + i % D, C::TILE_BYTES + (factors ? (is_a ? C::KA::TW_BYTES : C::KB::TW_BYTES) : 0));
        if (is_a)
            pipe_boxes<typename C::KA>(slot, col0, [&](uint32_t a, int x, int y) {
                tma_load_box(a, &P.map_in, x, y, (int)b, bar, first);
            });
        else
            pipe_boxes<typename C::KB>(slot, col0, [&](uint32_t a, int x, int y) {
                tma_load_box(a, &P.map_io, x, y, (int)b, bar, normal);
            });
        if (factors) {
            // block k0 / COLS of the pass's factor table
            using KA = typename C::KA;
            using KB = typename C::KB;
            const uint32_t k0 = col0 & ((1u << (is_a ? LOGPA : C::LOGPB)) - 1);
            const float4 *src = is_a ? P.fact_a + (size_t)(k0 / KA::COLS) * (KA::TW_BYTES / 16)
                                     : P.fact_b + (size_t)(k0 / KB::COLS) * (KB::TW_BYTES / 16);
            bulk_load(sbase + C::OFF_TW + s * C::TW_BYTES, src, is_a ? KA::TW_BYTES : KB::TW_BYTES, bar);
        }
    }
    // end of the queue: one end marker for each compute group
    for (uint32_t e = 0; ok && e < (uint32_t)C::GROUPS; ++e) {
        const uint32_t n = i + e, s = n % S;
        if (n >= D && !(ok = pipe_wait(B.retired + n % D, (n / D - 1) & 1u, B.abort))) break;
        if (n >= S && !(ok = pipe_wait(B.free + s, (n / S - 1) & 1u, B.abort))) break;
        B.item[n % D] = kPipeEnd;
        mbar_arrive(B.full + n % D);
    }
    if (!ok) {
        // a wait gave up: tell the other roles and the host, then let this
        // CTA's loads land before its shared memory goes away
        *B.abort = 1;
        atomicExch(F.err, 1u);
        for (uint32_t n = i > S ? i - S : 0; n < i; ++n)
            for (uint32_t polls = 0; polls < (1u << 20) && !mbar_try_wait(B.full + n % D, (n / D) & 1u); ++polls) {
            }
    }
}

template <class C, int LOGN, int LOGPA>
__device__ __forceinline__ void pipe_storer(const PipeParams &P, uint8_t *smem, const PipeBars &B) {
    const FusedParams &F = P.f;
    constexpr uint32_t T = C::T, GPT = C::GPT, S = C::SLOTS, D = 2 * S;
    const uint64_t first = l2_evict_first(), last = l2_evict_last();
    for (uint32_t i = 0;; ++i) {
        const uint32_t s = i % S;
        if (!pipe_wait(B.done + i % D, (i / D) & 1u, B.abort)) {
            *B.abort = 1;
            atomicExch(F.err, 1u);
            break;
        }
        const uint32_t idx = B.item[i % D];
        mbar_arrive(B.retired + i % D);  // the ring entry is read
        if (idx == kPipeEnd) break;
        bool is_a;
        uint32_t grp, tile;
        fused_item<T>(F, idx, is_a, grp, tile);
        const uint32_t b = grp / GPT, g = grp % GPT;
        const uint32_t col0 = pipe_col0<C>(is_a, g, tile);
        const uint32_t slot = smem_u32(smem) + s * C::TILE_BYTES;
        if (!is_a) {
            pipe_boxes<typename C::KB>(slot, col0, [&](uint32_t a, int x, int y) {
                tma_store_box(&P.map_io, x, y, (int)b, a, first);
            });
            bulk_commit();
            bulk_wait_read();
            mbar_arrive(B.free + s, C::WPG);
        } else {
            if (!C::FIRST_A) {
                // output of column j: row pos at (j / p) R p + (j mod p) + pos p
                const uint32_t jhi = col0 >> LOGPA, jlo = col0 & ((1u << LOGPA) - 1);
                constexpr int LOGJ = LOGN - 8 - LOGPA;  // log2 of the j / p values a transform
                pipe_boxes<typename C::KA>(slot, jlo, [&](uint32_t a, int x, int y) {
                    tma_store_box(&P.map_mid, x, y, (int)((b << LOGJ) + jhi), a, last);
                });
                bulk_commit();
                bulk_wait_read();
                mbar_arrive(B.free + s, C::WPG);
                bulk_wait_all();  // complete, not only read
            }
            red_release(F.ctr + 2 + grp);
        }
    }
    bulk_wait_all();
}

// Pass-A or pass-B work of one warp on a landed tile.
template <class C, int LOGN, int LOGPA, bool IS_A>
__device__ __forceinline__ void pipe_compute(const FusedParams &F, uint8_t *smem, uint32_t s, uint32_t grp,
                                             uint32_t tile, int group, int warp, int lane, uint64_t *free) {
    using K = std::conditional_t<IS_A, typename C::KA, typename C::KB>;
    constexpr bool FIRST = IS_A && C::FIRST_A;
    const uint32_t b = grp / C::GPT, g = grp % C::GPT;
    const uint32_t col0 = pipe_col0<C>(IS_A, g, tile);
    uint8_t *slot = smem + s * C::TILE_BYTES;
    const uint8_t *sub = smem + (IS_A ? C::OFF_SUBA : C::OFF_SUBB);
    typename K::Values v;
    int t, c;
    K::place(warp, lane, t, c);
    auto pre = [&](typename K::Values &x) {
        if constexpr (FIRST) {
            K::conj(x, F.in_im);  // (unconditional: a branch here costs 76 bytes of spills)
        } else {
            K::twiddle((const float4 *)(smem + C::OFF_TW + s * C::TW_BYTES), t, c, x);
        }
    };
    K::run(slot, t, c, sub, v, group, pre, [&] {
        if constexpr (FIRST) {
            fence_proxy_async_smem();  // this lane's accesses of the slot before the TMA's
            __syncwarp();
            if (lane == 0) mbar_arrive(free);
        }
    });
    if constexpr (FIRST) {
        // a first pass alone (pipe_first_launch) writes more than L2 holds: its output
        // passes through (2^26: 463.5 us with evict_last, 460.1 with evict_first)
        const uint64_t policy = F.nitems == F.ngroups * C::T ? l2_evict_first() : l2_evict_last();
        K::store_columns(F.out + ((uint64_t)b << LOGN) + ((uint64_t)(col0 + c) << (K::S::LOGT + K::LE)), t, v, policy);
    } else {
        if (!IS_A && (F.out_re != 1.0f || F.out_im != 1.0f)) K::scale(v, F.out_re, F.out_im);
        K::stage(slot, t, c, v, group);
    }
}

template <int LOGRA, int LOGRB, int LOGN, int LOGPA, int LE>
__global__ void __launch_bounds__(PipeCfg<LOGRA, LOGRB, LOGN, LOGPA, LE>::THREADS,
                                  (PipeCfg<LOGRA, LOGRB, LOGN, LOGPA, LE>::MINB))
fft_pipe_kernel(const __grid_constant__ PipeParams P) {
    using C = PipeCfg<LOGRA, LOGRB, LOGN, LOGPA, LE>;
    extern __shared__ __align__(1024) uint8_t smem_pipe[];  // (no static shared memory: it would cost 1 KB)
    constexpr int S = C::SLOTS, D = 2 * S;
    uint64_t *bars = (uint64_t *)(smem_pipe + C::OFF_BARS);
    uint32_t *s_item = (uint32_t *)(bars + S + 3 * D);
    int *s_abort = (int *)(s_item + D);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const PipeBars B{bars + S, bars, bars + S + D, bars + S + 2 * D, s_item, s_abort};
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) mbar_init(B.free + s, C::WPG);
        for (int s = 0; s < D; ++s) {
            mbar_init(B.full + s, 1);
            mbar_init(B.done + s, C::WPG);
            mbar_init(B.retired + s, 1);
        }
        *s_abort = 0;
    }
    C::KA::fill_sub(smem_pipe + C::OFF_SUBA, P.f.tw_a, threadIdx.x, C::THREADS);
    if (C::OFF_SUBB != C::OFF_SUBA) C::KB::fill_sub(smem_pipe + C::OFF_SUBB, P.f.tw_b, threadIdx.x, C::THREADS);
    stream_wait();  // (the tables above are complete before a plan's first launch)
    __syncthreads();
    if (warp == C::COMPUTE) {
        if (lane == 0) pipe_loader<C, LOGPA>(P, smem_pipe, B);
    } else if (warp == C::COMPUTE + 1) {
        if (lane == 0) pipe_storer<C, LOGN, LOGPA>(P, smem_pipe, B);
    } else {
        const int wg = warp % C::WPG, cg = warp / C::WPG;
        for (uint32_t i = (uint32_t)cg;; i += C::GROUPS) {
            const uint32_t s = i % S;
            bool ok = __all_sync(0xffffffffu, pipe_wait(B.full + i % D, (i / D) & 1u, B.abort));
            // warps that share named barriers go on or leave together (names 9, 10; 1 .. 8
            // are the column pairs')
            if constexpr (LE == 6) ok = group_all(9 + cg, C::WPG * 32, ok);
            if (!ok) {
                if (lane == 0) {
                    *B.abort = 1;
                    atomicExch(P.f.err, 1u);
                }
                break;
            }
            const uint32_t idx = B.item[i % D];
            if (idx != kPipeEnd) {
                bool is_a;
                uint32_t grp, tile;
                fused_item<C::T>(P.f, idx, is_a, grp, tile);
                if (is_a) pipe_compute<C, LOGN, LOGPA, true>(P.f, smem_pipe, s, grp, tile, cg, wg, lane, B.free + s);
                else pipe_compute<C, LOGN, LOGPA, false>(P.f, smem_pipe, s, grp, tile, cg, wg, lane, B.free + s);
                fence_proxy_async_smem();  // this lane's accesses of the slot before the TMA's
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(B.done + i % D);
            if (idx == kPipeEnd) break;
        }
    }
    __syncwarp();
    fused_finish<C::THREADS>(P.f, s_abort + 1);
}

template <int LOGRA, int LOGRB, int LOGN, int LOGPA, int LE>
inline void pipe_describe(PipeDesc &d) {
    using C = PipeCfg<LOGRA, LOGRB, LOGN, LOGPA, LE>;
    static_assert((C::SMEM + 1024) * C::MINB <= 228 * 1024, "shared memory of an SM (1 KB a CTA is reserved)");
    d.fn = (const void *)fft_pipe_kernel<LOGRA, LOGRB, LOGN, LOGPA, LE>;
    d.threads = C::THREADS;
    d.smem = C::SMEM;
    d.slots = C::SLOTS;
    d.ctas_per_sm = C::MINB;
    d.tiles_per_group = C::T;
    d.first = C::FIRST_A;
    d.loge = C::KA::LE;
    d.logtile = C::LOGTILE;
    d.soa = C::KA::SOA;
    d.box_cols_a = C::KA::BOXC;
    d.box_cols_b = C::KB::BOXC;
}

}  // namespace gbfft
