// Host-side check of the warp-column tiles (fft_warp.cuh, fft_pair.cuh),
// compiled for the host by nvcc and run by tests/test_warp_tiles.py.
// Per tile (kind 4: two columns a thread, 5: one, 6: two, over several warps):
//   * the offsets a thread reads its samples from are the ones at which a tensor
//     map with 128-, 64- or 32-byte swizzle puts (row, column) -- modelled here from
//     the linear address alone -- and cover the tile once;
//   * the in-warp exchange writes every slot of the columns once and reads each
//     element back where it was written, by lanes of the same warp only;
//   * worst bank conflicts of one access, in passes over what the banks allow
//     (8-byte lanes by half-warps, 16-byte lanes by quarter-warps).
// Prints: tile KIND LOGR LOGTILE ok conflicts
//         dft R ok     (PairDft<R> gives Dft<R>'s bits in both lanes)
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <random>
#include <set>
#include <vector>

#include "fft_warp.cuh"
using namespace gbfft;

// Byte at which the tensor-map copy puts byte `lin` of a box of ROWB-byte rows.
static uint32_t tma_swizzle(uint32_t lin, int rowb) {
    return lin ^ (((lin >> 7) & (rowb == 128 ? 7u : rowb == 64 ? 3u : 1u)) << 4);
}

// passes of one warp access beyond one per group of lanes that fills the banks
static int conflicts(const std::vector<uint32_t> &addr, int bytes) {
    const int group = 128 / bytes;  // lanes that fill the 32 banks once
    int worst = 1;
    for (size_t g = 0; g < addr.size(); g += group) {
        std::map<uint32_t, std::set<uint32_t>> banks;
        for (int l = 0; l < group; ++l)
            for (int w = 0; w < bytes / 4; ++w) {
                const uint32_t word = addr[g + l] / 4 + w;
                banks[word % 32].insert(word);
            }
        for (auto &b : banks) worst = std::max(worst, (int)b.second.size());
    }
    return worst;
}

template <class K, int KIND, int LOGR, int LOGTILE>
static void check() {
    using S = typename K::S;
    constexpr int R = 1 << LOGR, T = S::T, E = K::E, COLS = K::COLS, STEP = KIND == 4 ? 2 : 1, BYTES = 8 * STEP;
    bool ok = true;
    int worst = 1;
    auto off = [](uint32_t row, uint32_t c) {
        return warp_tile_off<LOGR, K::BOXC>(row, c >> 1) + (KIND == 5 ? (c & 1) << 3 : 0);
    };
    std::vector<int> landed(COLS * R, 0), slot(COLS * R, -1), owner_warp(COLS * R, -1);
    for (int pass = 0; pass < 3; ++pass)  // 0: landing reads, 1: exchange writes, 2: exchange reads
        for (int w = 0; w < K::WARPS; ++w)
            for (int i = 0; i < E; ++i) {
                std::vector<uint32_t> addr;
                for (int lane = 0; lane < 32; ++lane) {
                    int t, c;
                    K::place(w, lane, t, c);
                    uint32_t a, pos;
                    if (pass == 0) {
                        pos = t + T * i;
                        a = off(t, c) + i * T * K::ROWB;
                    } else if (pass == 1) {
                        pos = (t << K::LE) + i;
                        a = (off(((uint32_t)t << K::LE) | ((uint32_t)t & 7u), c) ^ warp_xor<K::BOXC>(i & 7)) +
                            (i & ~7) * K::ROWB;
                    } else {
                        pos = t + T * i;
                        a = (off(t, c) ^ warp_xor<K::BOXC>((i >> (K::LE - S::LOGT)) & 7)) + i * T * K::ROWB;
                    }
                    addr.push_back(a);
                    if (a + BYTES > (uint32_t)(COLS * R * 8)) {
                        ok = false;
                        continue;
                    }
                    for (int k = 0; k < STEP; ++k) {
                        const int s = a / 8 + k, id = (c + k) * R + (int)pos;
                        if (pass == 0) {
                            const uint32_t box = (c + k) / K::BOXC, lin = pos * K::ROWB + ((c + k) % K::BOXC) * 8;
                            if (box * R * K::ROWB + tma_swizzle(lin, K::ROWB) != (uint32_t)s * 8) ok = false;
                            landed[s]++;
                            owner_warp[s] = w;
                        } else if (pass == 1) {
                            if (slot[s] != -1 || owner_warp[s] != w) ok = false;
                            slot[s] = id;
                        } else if (slot[s] != id) {
                            ok = false;
                        }
                    }
                }
                worst = std::max(worst, conflicts(addr, BYTES));
            }
    for (int v : landed) ok = ok && v == 1;
    printf("tile %d %d %d %d %d\n", KIND, LOGR, LOGTILE, ok ? 1 : 0, worst);
}

// Wide tiles (kind 6): a column pair's threads span W warps; two exchanges.
template <int LOGR, int LOGTILE>
static void check_wide() {
    using K = WideTile<LOGR, LOGTILE>;
    constexpr int R = K::R, T = K::T, E = K::E, COLS = K::COLS;
    bool ok = true;
    int worst = 1;
    std::vector<int> landed(COLS * R, 0);
    std::vector<int> slot;
    for (int pass = 0; pass < 6; ++pass) {  // landing | exchange 0 write, read | exchange 1 write, read | staging
        if (pass == 1 || pass == 3 || pass == 5) slot.assign(COLS * R, -1);
        for (int w = 0; w < K::WARPS; ++w)
            for (int i = 0; i < E; ++i) {
                std::vector<uint32_t> addr;
                for (int lane = 0; lane < 32; ++lane) {
                    int t, c;
                    K::place(w, lane, t, c);
                    auto off = [&](uint32_t row) { return warp_tile_off<LOGR, K::BOXC>(row, (uint32_t)c >> 1); };
                    uint32_t a, pos;
                    if (pass == 0 || pass == 4) {
                        pos = t + T * i;
                        a = off(t) + i * T * K::ROWB;
                    } else if (pass == 1) {
                        pos = 16 * t + i;
                        a = (off(((uint32_t)t << 4) | ((uint32_t)t & 7u)) ^ warp_xor<K::BOXC>(i & 7)) + (i & ~7) * K::ROWB;
                    } else if (pass == 2) {
                        pos = t + T * i;
                        a = (off(t) ^ K::read_xor(t, 0) ^ K::read_xor(0, i)) + i * T * K::ROWB;
                    } else if (pass == 3) {
                        pos = ((t >> 4) << 8) + (t & 15) + 16 * i;
                        a = off(((t >> 4) << 8) + (t & 15)) + i * 16 * K::ROWB;
                    } else {  // slot i holds output q = i / (E / R2) of butterfly t + T b, b = i % (E / R2)
                        const int b = i % (E / K::R2), q = i / (E / K::R2);
                        pos = t + T * b + 256 * q;
                        a = off(t) + (T * b + 256 * q) * K::ROWB;
                    }
                    addr.push_back(a);
                    if (a + 16 > (uint32_t)(COLS * R * 8) || a % 16) {
                        ok = false;
                        continue;
                    }
                    for (int k = 0; k < 2; ++k) {
                        const int s = a / 8 + k, id = (c + k) * R + (int)pos;
                        const uint32_t lin = pos * K::ROWB + (c + k) * 8;
                        if ((pass == 0 || pass == 5) && tma_swizzle(lin, K::ROWB) != (uint32_t)s * 8) ok = false;
                        if (pass == 0) landed[s]++;
                        else if (pass == 2 || pass == 4) ok = ok && slot[s] == id;
                        else {
                            ok = ok && slot[s] == -1;
                            slot[s] = id;
                        }
                    }
                }
                worst = std::max(worst, conflicts(addr, 16));
            }
    }
    for (int v : landed) ok = ok && v == 1;
    printf("tile 6 %d %d %d %d\n", LOGR, LOGTILE, ok ? 1 : 0, worst);
}

template <int R>
static void dft() {
    std::mt19937 g(R);
    std::normal_distribution<float> nd;
    bool ok = true;
    for (int rep = 0; rep < 200; ++rep) {
        float2 a[R], b[R];
        Pair x[R];
        for (int i = 0; i < R; ++i) {
            a[i] = make_float2(nd(g), nd(g));
            b[i] = make_float2(nd(g), nd(g));
            x[i] = Pair{make_float2(a[i].x, b[i].x), make_float2(a[i].y, b[i].y)};
        }
        Dft<R>::template run<false>(a);
        Dft<R>::template run<false>(b);
        PairDft<R>::run(x);
        for (int i = 0; i < R; ++i) {
            const float want[4] = {a[i].x, b[i].x, a[i].y, b[i].y};
            const float got[4] = {x[i].re.x, x[i].re.y, x[i].im.x, x[i].im.y};
            ok = ok && memcmp(want, got, sizeof want) == 0;
        }
    }
    printf("dft %d %d\n", R, ok ? 1 : 0);
}

int main() {
    check<PairTile<7, 12>, 4, 7, 12>();
    check<PairTile<8, 12>, 4, 8, 12>();
    check<ColTile<8, 13>, 5, 8, 13>();
    check<ColTile<9, 13>, 5, 9, 13>();
    check<ColTile<10, 13>, 5, 10, 13>();
    check_wide<10, 13>();
    check_wide<11, 13>();
    dft<2>();
    dft<4>();
    dft<8>();
    dft<16>();
    return 0;
}
