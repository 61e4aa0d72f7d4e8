// Column transforms that stay inside one warp, over tiles staged in shared
// memory by the tensor memory accelerator (TMA).
//
// A tile is [R rows][C columns] of complex<f32> (R = 2^LOGR, C columns of one
// global Stockham pass).  Every column is transformed by T = R / E threads of
// ONE warp (E samples a column and thread, T = 8, 16 or 32), so the exchange
// between the two register sub-passes needs a __syncwarp and no CTA barrier,
// and it runs in the column's own storage: the tile is the only buffer.
//
// Lanes of a column run along its rows (stride = one tile row), which on a
// plain row-major tile would put them all on one bank.  The TMA lays the tile
// out with its swizzle (the 16-byte chunk index XOR the row), so 8 consecutive
// rows of one 16-byte chunk -- two adjacent columns -- cover all 32 banks.
//
//   PairTile: E = 16, a thread takes both columns of a chunk as (re, re'),
//     (im, im') pairs (fft_pair.cuh): 16-byte accesses, conflict-free, half
//     the instructions and half the twiddle loads a sample.
//   ColTile: E = 32, one column a thread, for R = 512 and 1024 (two columns of
//     32 samples would not fit the registers); a half-warp holds 8 consecutive
//     t of two adjacent columns (T <= 16), conflict-free; for T = 32 a warp has
//     one column and its accesses take twice the minimum of wavefronts.
//
// Twiddles: the sub-pass table sits in shared memory, and the inter-pass
// factors W_{R p}^{(t + T e) k} = w[k][t] * f[k][e] of a tile come with the
// tile, as one bulk copy from the plan's table (factors_fill), so the compute
// warps never wait for a global load.
#pragma once
#include "fft_pair.cuh"
#include "fft_tiles.cuh"

namespace gbfft {

// Store with an L2 eviction priority.
__device__ __forceinline__ void st_policy(float2 *p, float2 v, uint64_t policy) {
    asm volatile("st.global.L2::cache_hint.v2.f32 [%0], {%1, %2}, %3;" ::"l"(p), "f"(v.x), "f"(v.y), "l"(policy)
                 : "memory");
}

// Byte offset, in the tile, of (row, 16-byte chunk) as the TMA's swizzle lays
// it out: boxes of BOXC columns (128-, 64- or 32-byte rows) follow one another.
template <int LOGR, int BOXC>
GBFFT_HD uint32_t warp_tile_off(uint32_t row, uint32_t chunk) {
    if constexpr (BOXC == 16)
        return ((chunk >> 3) << (LOGR + 7)) + (row << 7) + (((chunk & 7) ^ (row & 7)) << 4);
    else if constexpr (BOXC == 8)
        return (row << 6) + ((chunk ^ ((row >> 1) & 3)) << 4);
    else
        return (row << 5) + ((chunk ^ ((row >> 2) & 1)) << 4);
}
// Change of warp_tile_off when the row's low three bits are XORed with i.
template <int BOXC>
GBFFT_HD constexpr uint32_t warp_xor(uint32_t i) {
    return BOXC == 16 ? ((i << 7) | (i << 4)) : (BOXC == 8 ? ((i << 6) | ((i >> 1) << 4)) : ((i << 5) | ((i >> 2) << 4)));
}
// Row that holds element `pos` of a column between the sub-passes: its low
// three bits XOR those of pos >> LE, so that the stride-E writes of 8
// consecutive t fall on 8 different rows mod 8 (and so do the reads t + T e).
template <int LE>
GBFFT_HD uint32_t warp_xrow(uint32_t pos) { return pos ^ ((pos >> LE) & 7u); }

// What both tile forms share.
template <int LOGR, int LOGTILE, int LE>
struct WarpTile {
    using S = SubCfg<LOGR, LE>;
    static_assert(S::NSUB == 2, "two register sub-passes");
    static_assert(S::LOGT >= 3 && S::LOGT <= 5 && S::LOGT <= LE, "a column is 8 .. 32 lanes of one warp");
    static constexpr int R = 1 << LOGR, E = S::E, T = S::T;
    static constexpr int COLS = 1 << (LOGTILE - LOGR);  // columns of the tile
    static constexpr int BOXC = COLS >= 16 ? 16 : 8;    // columns of one TMA box
    static_assert(COLS >= 8, "TMA boxes of at least 64-byte rows");
    static constexpr int ROWB = BOXC * 8;               // bytes of a tile row
    // inter-pass factors of a tile: f[chunk][e], then w[chunk][t], a float4
    // (two columns) each
    static constexpr int TW_BYTES = COLS * (E + T) * (int)sizeof(float2);
};

// A last sub-pass of radix R1 < 16: 16 / R1 butterflies, butterfly b's twiddles
// wt[m] * W_16^{m b}.
template <int R1>
__device__ __forceinline__ void pair_factored(const Pair (&wt)[R1], Pair (&x)[16]) {
    constexpr int NB = 16 / R1;
    auto body = [&](auto bc) {
        constexpr int b = decltype(bc)::value;
        Pair y[R1];
        y[0] = x[b];
        auto apply = [&](auto mc) {
            constexpr int M = decltype(mc)::value + 1;
            y[M] = pair_mul(pair_mul_w16c<(M * b) & 15>(x[b + M * NB]), wt[M]);
        };
        [&]<int... Ms>(std::integer_sequence<int, Ms...>) {
            (apply(std::integral_constant<int, Ms>{}), ...);
        }(std::make_integer_sequence<int, R1 - 1>{});
        PairDft<R1>::run(y);
#pragma unroll
        for (int q = 0; q < R1; ++q) x[b + q * NB] = y[q];
    };
    [&]<int... Bs>(std::integer_sequence<int, Bs...>) {
        (body(std::integral_constant<int, Bs>{}), ...);
    }(std::make_integer_sequence<int, NB>{});
}

// Two columns a thread, 16 samples of each.
template <int LOGR, int LOGTILE>
struct PairTile : WarpTile<LOGR, LOGTILE, 4> {
    using B = WarpTile<LOGR, LOGTILE, 4>;
    using S = typename B::S;
    static constexpr int LE = 4, E = 16, T = S::T;
    static constexpr bool SOA = true;
    static constexpr int WARPS = B::COLS / 2 * T / 32;
    // sub-pass table, each entry doubled: (re, re, im, im)
    static constexpr int SUB_BYTES = S::tw_entries() * 16;
    using Values = Pair[E];

    __device__ __forceinline__ static void fill_sub(uint8_t *tab, const float2 *__restrict__ tw, int tid, int nt) {
        for (int i = tid; i < S::tw_entries(); i += nt) {
            const float2 w = ld_tw(tw + i);
            ((float4 *)tab)[i] = make_float4(w.x, w.x, w.y, w.y);
        }
    }
    // thread's t, first column c and chunk
    GBFFT_HD static void place(int warp, int lane, int &t, int &c) {
        t = lane & (T - 1);
        c = 2 * (warp * (32 / T) + (lane >> S::LOGT));
    }
    // One pass over the thread's columns of a landed tile; x[b + q * (E >> LR)]
    // = output q of butterfly t + T b.  `pre` conjugates or applies twiddles;
    // `read` is called after the last read of the tile.
    template <class Pre, class Read>
    __device__ __forceinline__ static void run(uint8_t *tile, int t, int c, const uint8_t *sub, Pair (&x)[E],
                                               int, Pre pre, Read read) {
        const uint32_t off0 = warp_tile_off<LOGR, B::BOXC>((uint32_t)t, (uint32_t)c >> 1);
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const float4 q = *(const float4 *)(tile + off0 + e * (T * B::ROWB));
            x[e] = Pair{make_float2(q.x, q.z), make_float2(q.y, q.w)};
        }
        pre(x);
        PairDft<E>::run(x);
        __syncwarp();  // every lane has read its samples: the columns' storage is free
        const uint32_t offw = warp_tile_off<LOGR, B::BOXC>(((uint32_t)t << LE) | ((uint32_t)t & 7u), (uint32_t)c >> 1);
#pragma unroll
        for (int q = 0; q < E; ++q)
            *(float4 *)(tile + (offw ^ warp_xor<B::BOXC>(q & 7)) + (q & ~7) * B::ROWB) =
                make_float4(x[q].re.x, x[q].re.y, x[q].im.x, x[q].im.y);
        __syncwarp();
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const float4 q = *(const float4 *)(tile + (off0 ^ warp_xor<B::BOXC>((e >> (LE - S::LOGT)) & 7)) +
                                               e * (T * B::ROWB));
            x[e] = Pair{make_float2(q.x, q.y), make_float2(q.z, q.w)};
        }
        read();
        const float4 *tw = (const float4 *)sub + t;
        constexpr int R1 = 1 << S::logr(1), P = 1 << S::tw_logp(1);
        Pair wt[R1];
#pragma unroll
        for (int m = 1; m < R1; ++m) {
            const float4 w = tw[(m - 1) * P];
            wt[m] = Pair{make_float2(w.x, w.y), make_float2(w.z, w.w)};
            if constexpr (R1 == 16) x[m] = pair_mul(x[m], wt[m]);
        }
        if constexpr (R1 == 16) PairDft<16>::run(x);
        else pair_factored<R1>(wt, x);
    }
    // inter-pass factors from the tile's table
    __device__ __forceinline__ static void twiddle(const float4 *tab, int t, int c, Pair (&x)[E]) {
        const float4 *f = tab + (c >> 1) * E;
        const float4 wq = tab[B::COLS / 2 * E + ((c >> 1) << S::LOGT) + t];
        const Pair w{make_float2(wq.x, wq.y), make_float2(wq.z, wq.w)};
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const float4 q = f[e];
            x[e] = pair_mul(x[e], pair_mul(w, Pair{make_float2(q.x, q.y), make_float2(q.z, q.w)}));
        }
    }
    __device__ __forceinline__ static void conj(Pair (&x)[E], float s) {
#pragma unroll
        for (int e = 0; e < E; ++e) x[e].im = pmul(x[e].im, pset(s));
    }
    __device__ __forceinline__ static void scale(Pair (&x)[E], float re, float im) {
#pragma unroll
        for (int e = 0; e < E; ++e) x[e] = Pair{pmul(x[e].re, pset(re)), pmul(x[e].im, pset(im))};
    }
    // first pass: column c's outputs are contiguous at dst (dst already at column c)
    __device__ __forceinline__ static void store_columns(float2 *dst, int t, const Pair (&x)[E], uint64_t policy) {
        constexpr int LR = S::logr(1), LP = S::logp(1), NB = E >> LR;
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int q = 0; q < (1 << LR); ++q) {
                const Pair &v = x[b + q * NB];
                float2 *d = dst + t + T * b + (q << LP);
                st_policy(d, make_float2(v.re.x, v.im.x), policy);
                st_policy(d + B::R, make_float2(v.re.y, v.im.y), policy);
            }
    }
    // back into the tile in natural row order, for a TMA store
    __device__ __forceinline__ static void stage(uint8_t *tile, int t, int c, const Pair (&x)[E], int) {
        constexpr int LR = S::logr(1), LP = S::logp(1), NB = E >> LR;
        const uint32_t off0 = warp_tile_off<LOGR, B::BOXC>((uint32_t)t, (uint32_t)c >> 1);
        __syncwarp();  // every lane has read its exchanged samples
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int q = 0; q < (1 << LR); ++q) {  // T b and q << LP are multiples of 8
                const Pair &v = x[b + q * NB];
                *(float4 *)(tile + off0 + (T * b + (q << LP)) * B::ROWB) =
                    make_float4(v.re.x, v.im.x, v.re.y, v.im.y);
            }
    }
};

// Two columns a thread, 16 samples of each, columns of 2^10 or 2^11 points over
// T = 64 or 128 threads (two or four warps): three sub-passes (16 x 16 x 4 or 8),
// whose exchanges meet at a named barrier of the column pair's warps.  2^11 rows
// of 4 columns (32 bytes a row) make N = 2^21 and 2^22 two-pass transforms.
template <int LOGR, int LOGTILE>
struct WideTile {
    using S = SubCfg<LOGR, 4>;
    static_assert(S::NSUB == 3 && S::LOGT >= 6 && S::LOGT <= 7, "64 or 128 threads a column pair");
    static constexpr int LE = 4, E = 16, R = 1 << LOGR, T = S::T, W = T / 32;
    static constexpr bool SOA = true;
    static constexpr int COLS = 1 << (LOGTILE - LOGR), BOXC = COLS, ROWB = BOXC * 8;
    static_assert(COLS == 4 || COLS == 8, "one box a row");
    static constexpr int WARPS = COLS / 2 * W;
    static constexpr int TW_BYTES = COLS * (E + T) * (int)sizeof(float2);
    // doubled table of sub-pass 1, plain one of sub-pass 2
    static constexpr int R2 = 1 << S::logr(2), SUB1 = S::tw_count(1);
    static constexpr int SUB_BYTES = SUB1 * 16 + S::tw_count(2) * 8;
    using Values = Pair[E];

    __device__ __forceinline__ static void fill_sub(uint8_t *tab, const float2 *__restrict__ tw, int tid, int nt) {
        for (int i = tid; i < SUB1; i += nt) {
            const float2 w = ld_tw(tw + i);
            ((float4 *)tab)[i] = make_float4(w.x, w.x, w.y, w.y);
        }
        for (int i = tid; i < S::tw_count(2); i += nt) ((float2 *)(tab + SUB1 * 16))[i] = ld_tw(tw + SUB1 + i);
    }
    GBFFT_HD static void place(int warp, int lane, int &t, int &c) {
        t = (warp % W) * 32 + lane;
        c = 2 * (warp / W);
    }
    // Barrier of the column pair's T threads: names 1 .. 4 for group 0, 5 .. 8 for
    // group 1 whatever the radix, so that the groups' tiles, which may differ in
    // radix, never meet at one name with different thread counts.
    __device__ __forceinline__ static void pair_sync(int c, int group) {
        static_assert(COLS / 2 <= 4, "four barrier names a group");
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group * 4 + (c >> 1)), "n"(T) : "memory");
    }
    // rows of the exchange after sub-pass 0, as warp_xrow<4>: change of the read
    // offset of row t + T e
    GBFFT_HD static uint32_t read_xor(int t, int e) {
        return warp_xor<BOXC>((uint32_t)((t >> 4) + (T / 16) * e) & 7u);
    }
    template <class Pre, class Read>
    __device__ __forceinline__ static void run(uint8_t *tile, int t, int c, const uint8_t *sub, Pair (&x)[E], int group,
                                               Pre pre, Read read) {
        auto sync = [&] { pair_sync(c, group); };
        const uint32_t off0 = warp_tile_off<LOGR, BOXC>((uint32_t)t, (uint32_t)c >> 1);
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const float4 q = *(const float4 *)(tile + off0 + e * (T * ROWB));
            x[e] = Pair{make_float2(q.x, q.z), make_float2(q.y, q.w)};
        }
        pre(x);
        PairDft<E>::run(x);
        sync();  // the pair's threads have read their samples: its storage is free
        const uint32_t offw = warp_tile_off<LOGR, BOXC>(((uint32_t)t << 4) | ((uint32_t)t & 7u), (uint32_t)c >> 1);
#pragma unroll
        for (int q = 0; q < E; ++q)
            *(float4 *)(tile + (offw ^ warp_xor<BOXC>(q & 7)) + (q & ~7) * ROWB) =
                make_float4(x[q].re.x, x[q].re.y, x[q].im.x, x[q].im.y);
        sync();
        const uint32_t offr = off0 ^ read_xor(t, 0);
        const float4 *tw1 = (const float4 *)sub + (t & 15);
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const float4 q = *(const float4 *)(tile + (offr ^ read_xor(0, e)) + e * (T * ROWB));
            x[e] = Pair{make_float2(q.x, q.y), make_float2(q.z, q.w)};
            if (e > 0) {
                const float4 w = tw1[(e - 1) * 16];
                x[e] = pair_mul(x[e], Pair{make_float2(w.x, w.y), make_float2(w.z, w.w)});
            }
        }
        PairDft<E>::run(x);
        sync();
        const uint32_t off1 = warp_tile_off<LOGR, BOXC>((uint32_t)(((t >> 4) << 8) + (t & 15)), (uint32_t)c >> 1);
#pragma unroll
        for (int q = 0; q < E; ++q)
            *(float4 *)(tile + off1 + q * (16 * ROWB)) = make_float4(x[q].re.x, x[q].re.y, x[q].im.x, x[q].im.y);
        sync();
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const float4 q = *(const float4 *)(tile + off0 + e * (T * ROWB));
            x[e] = Pair{make_float2(q.x, q.y), make_float2(q.z, q.w)};
        }
        read();
        Pair wt[R2];
        const float2 *tw2 = (const float2 *)(sub + SUB1 * 16) + t;
#pragma unroll
        for (int m = 1; m < R2; ++m) {
            const float2 w = tw2[(m - 1) * T];
            wt[m] = Pair{pset(w.x), pset(w.y)};
        }
        pair_factored<R2>(wt, x);
    }
    __device__ __forceinline__ static void twiddle(const float4 *tab, int t, int c, Pair (&x)[E]) {
        const float4 *f = tab + (c >> 1) * E;
        const float4 wq = tab[COLS / 2 * E + ((c >> 1) << S::LOGT) + t];
        const Pair w{make_float2(wq.x, wq.y), make_float2(wq.z, wq.w)};
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const float4 q = f[e];
            x[e] = pair_mul(x[e], pair_mul(w, Pair{make_float2(q.x, q.y), make_float2(q.z, q.w)}));
        }
    }
    __device__ __forceinline__ static void conj(Pair (&x)[E], float s) {
#pragma unroll
        for (int e = 0; e < E; ++e) x[e].im = pmul(x[e].im, pset(s));
    }
    __device__ __forceinline__ static void scale(Pair (&x)[E], float re, float im) {
#pragma unroll
        for (int e = 0; e < E; ++e) x[e] = Pair{pmul(x[e].re, pset(re)), pmul(x[e].im, pset(im))};
    }
    __device__ __forceinline__ static void store_columns(float2 *dst, int t, const Pair (&x)[E], uint64_t policy) {
#pragma unroll
        for (int b = 0; b < E / R2; ++b)
#pragma unroll
            for (int q = 0; q < R2; ++q) {
                const Pair &v = x[b + q * (E / R2)];
                float2 *d = dst + t + T * b + (q << 8);
                st_policy(d, make_float2(v.re.x, v.im.x), policy);
                st_policy(d + R, make_float2(v.re.y, v.im.y), policy);
            }
    }
    // The pair's storage is read by other warps until all have passed sub-pass 2's
    // reads: one more barrier before the results go back into it.
    __device__ __forceinline__ static void stage(uint8_t *tile, int t, int c, const Pair (&x)[E], int group) {
        pair_sync(c, group);
        const uint32_t off0 = warp_tile_off<LOGR, BOXC>((uint32_t)t, (uint32_t)c >> 1);
#pragma unroll
        for (int b = 0; b < E / R2; ++b)
#pragma unroll
            for (int q = 0; q < R2; ++q) {
                const Pair &v = x[b + q * (E / R2)];
                *(float4 *)(tile + off0 + (T * b + (q << 8)) * ROWB) = make_float4(v.re.x, v.im.x, v.re.y, v.im.y);
            }
    }
};

// One column a thread, 32 samples.  Packed butterflies for every radix (scalar
// ones, as the barrier form runs pairs with a radix-2^10 pass: 2^19 288 against
// 274 us, 2^20 351 against 324; same bits).
template <int LOGR, int LOGTILE>
struct ColTile : WarpTile<LOGR, LOGTILE, 5> {
    using B = WarpTile<LOGR, LOGTILE, 5>;
    using S = typename B::S;
    static constexpr int LE = 5, E = 32, T = S::T;
    static constexpr bool SOA = false;
    static constexpr int WARPS = B::COLS * T / 32;
    static constexpr int SUB_BYTES = (S::tw_entries() * 8 + 15) & ~15;
    using Values = float2[E];

    __device__ __forceinline__ static void fill_sub(uint8_t *tab, const float2 *__restrict__ tw, int tid, int nt) {
        for (int i = tid; i < S::tw_entries(); i += nt) ((float2 *)tab)[i] = ld_tw(tw + i);
    }
    GBFFT_HD static void place(int warp, int lane, int &t, int &c) {
        int cw;
        if constexpr (S::LOGT == 3) {
            t = lane & 7;
            cw = lane >> 3;
        } else if constexpr (S::LOGT == 4) {
            t = (lane & 7) | ((lane >> 4) << 3);
            cw = (lane >> 3) & 1;
        } else {
            t = lane;
            cw = 0;
        }
        c = warp * (32 / T) + cw;
    }
    __device__ __forceinline__ static uint32_t off(uint32_t row, uint32_t c) {
        return warp_tile_off<LOGR, B::BOXC>(row, c >> 1) + ((c & 1) << 3);
    }
    template <class Pre, class Read>
    __device__ __forceinline__ static void run(uint8_t *tile, int t, int c, const uint8_t *sub, float2 (&v)[E],
                                               int, Pre pre, Read read) {
        DftRegs eng;
        const uint32_t off0 = off((uint32_t)t, (uint32_t)c);
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = *(const float2 *)(tile + off0 + e * (T * B::ROWB));
        pre(v);
        subpass_run<LOGR, 0, LE, DftRegs, true>(v, t, (const float2 *)sub, eng);
        __syncwarp();
        const uint32_t offw = off(((uint32_t)t << LE) | ((uint32_t)t & 7u), (uint32_t)c);
#pragma unroll
        for (int q = 0; q < E; ++q)
            *(float2 *)(tile + (offw ^ warp_xor<B::BOXC>(q & 7)) + (q & ~7) * B::ROWB) = v[q];
        __syncwarp();
#pragma unroll
        for (int e = 0; e < E; ++e)
            v[e] = *(const float2 *)(tile + (off0 ^ warp_xor<B::BOXC>((e >> (LE - S::LOGT)) & 7)) +
                                     e * (T * B::ROWB));
        read();
        subpass_run<LOGR, 1, LE, DftRegs, true>(v, t, (const float2 *)sub, eng);
    }
    __device__ __forceinline__ static void twiddle(const float4 *tab, int t, int c, float2 (&v)[E]) {
        // entries of column c: half c & 1 of its chunk's float4s
        const float2 *f = (const float2 *)(tab + (c >> 1) * E) + (c & 1);
        const float2 w = ((const float2 *)(tab + B::COLS / 2 * E + ((c >> 1) << S::LOGT) + t))[c & 1];
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = cmul(v[e], cmul(w, f[2 * e]));
    }
    __device__ __forceinline__ static void conj(float2 (&v)[E], float s) {
#pragma unroll
        for (int e = 0; e < E; ++e) v[e].y *= s;
    }
    __device__ __forceinline__ static void scale(float2 (&v)[E], float re, float im) {
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = make_float2(v[e].x * re, v[e].y * im);
    }
    __device__ __forceinline__ static void store_columns(float2 *dst, int t, const float2 (&v)[E], uint64_t policy) {
        constexpr int LR = S::logr(1), LP = S::logp(1), NB = E >> LR;
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int q = 0; q < (1 << LR); ++q) st_policy(dst + t + T * b + (q << LP), v[b + q * NB], policy);
    }
    __device__ __forceinline__ static void stage(uint8_t *tile, int t, int c, const float2 (&v)[E], int) {
        constexpr int LR = S::logr(1), LP = S::logp(1), NB = E >> LR;
        const uint32_t off0 = off((uint32_t)t, (uint32_t)c);
        __syncwarp();
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int q = 0; q < (1 << LR); ++q)
                *(float2 *)(tile + off0 + (T * b + (q << LP)) * B::ROWB) = v[b + q * NB];
    }
};

}  // namespace gbfft
