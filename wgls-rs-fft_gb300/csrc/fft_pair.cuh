// Two columns a thread: complex values held as (re, re'), (im, im') pairs so
// that every butterfly and every twiddle multiply is made of two-lane FP32
// instructions with no swaps between the lanes.
//
// The single-column form packs (re, im): adds are two-lane by nature, but a
// multiply by -i or by a twiddle mixes the lanes and costs moves.  With two
// columns side by side a complex multiply is four two-lane instructions for
// two samples, and -i is a renaming of registers.  Same operations in the same
// order as Dft<R> and cmul, each lane rounded like the scalar instruction.
#pragma once
#include "fft_smem.cuh"

namespace gbfft {

struct Pair {
    float2 re, im;  // .x: first column, .y: second
};

GBFFT_HD float2 padd(float2 a, float2 b) {
#ifdef GBFFT_PACKED_F32
    return __fadd2_rn(a, b);
#else
    return make_float2(a.x + b.x, a.y + b.y);
#endif
}
GBFFT_HD float2 psub(float2 a, float2 b) {
#ifdef GBFFT_PACKED_F32
    return __fadd2_rn(a, make_float2(-b.x, -b.y));
#else
    return make_float2(a.x - b.x, a.y - b.y);
#endif
}
GBFFT_HD float2 pmul(float2 a, float2 b) {
#ifdef GBFFT_PACKED_F32
    return __fmul2_rn(a, b);
#else
    return make_float2(a.x * b.x, a.y * b.y);
#endif
}
GBFFT_HD float2 pfma(float2 a, float2 b, float2 c) {
#ifdef GBFFT_PACKED_F32
    return __ffma2_rn(a, b, c);
#else
    return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
#endif
}
GBFFT_HD float2 pneg(float2 a) { return make_float2(-a.x, -a.y); }
GBFFT_HD float2 pset(float f) { return make_float2(f, f); }

GBFFT_HD Pair operator+(Pair a, Pair b) { return Pair{padd(a.re, b.re), padd(a.im, b.im)}; }
GBFFT_HD Pair operator-(Pair a, Pair b) { return Pair{psub(a.re, b.re), psub(a.im, b.im)}; }
// a - i b, a + i b
GBFFT_HD Pair sub_i(Pair a, Pair b) { return Pair{padd(a.re, b.im), psub(a.im, b.re)}; }
GBFFT_HD Pair add_i(Pair a, Pair b) { return Pair{psub(a.re, b.im), padd(a.im, b.re)}; }
// s + f y, f a real factor
GBFFT_HD Pair pair_fma(float f, Pair y, Pair s) {
    return Pair{pfma(pset(f), y.re, s.re), pfma(pset(f), y.im, s.im)};
}
// s - i f y
GBFFT_HD Pair pair_fma_mi(float f, Pair y, Pair s) {
    return Pair{pfma(pset(f), y.im, s.re), pfma(pset(-f), y.re, s.im)};
}
// a * w, w = (re, re'), (im, im')
GBFFT_HD Pair pair_mul(Pair a, Pair w) {
    return Pair{pfma(a.re, w.re, pneg(pmul(a.im, w.im))), pfma(a.re, w.im, pmul(a.im, w.re))};
}

template <int R> struct PairDft;

template <> struct PairDft<2> {
    GBFFT_HD static void run(Pair *x) {
        const Pair a = x[0], b = x[1];
        x[0] = a + b;
        x[1] = a - b;
    }
};
template <> struct PairDft<4> {
    GBFFT_HD static void run(Pair *x) {
        const Pair s02 = x[0] + x[2], d02 = x[0] - x[2], s13 = x[1] + x[3], d13 = x[1] - x[3];
        x[0] = s02 + s13;
        x[2] = s02 - s13;
        x[1] = sub_i(d02, d13);
        x[3] = add_i(d02, d13);
    }
};
template <> struct PairDft<8> {  // as Dft<8>
    GBFFT_HD static void run(Pair *x) {
        Pair a[4], b[4];
        GBFFT_UNROLL
        for (int k = 0; k < 4; ++k) {
            a[k] = x[k] + x[k + 4];
            b[k] = x[k] - x[k + 4];
        }
        PairDft<4>::run(a);
        const Pair q1 = sub_i(b[1], b[1]);                                        // b1 (1 - i)
        const Pair q3 = Pair{psub(b[3].im, b[3].re), padd(b[3].re, b[3].im)};     // re, -im of b3 (-1 - i)
        const Pair s02 = sub_i(b[0], b[2]), d02 = add_i(b[0], b[2]);
        const Pair S = Pair{padd(q1.re, q3.re), psub(q1.im, q3.im)};
        const Pair D = Pair{psub(q1.re, q3.re), padd(q1.im, q3.im)};
        x[0] = a[0];
        x[2] = a[1];
        x[4] = a[2];
        x[6] = a[3];
        x[1] = pair_fma(kSqrtHalf, S, s02);
        x[3] = pair_fma_mi(kSqrtHalf, D, d02);
        x[5] = pair_fma(-kSqrtHalf, S, s02);
        x[7] = pair_fma_mi(-kSqrtHalf, D, d02);
    }
};
template <> struct PairDft<16> {  // as Dft<16>
    GBFFT_HD static void run(Pair *x) {
        Pair z[4][4];
        GBFFT_UNROLL
        for (int n1 = 0; n1 < 4; ++n1) {
            Pair t[4] = {x[n1], x[n1 + 4], x[n1 + 8], x[n1 + 12]};
            PairDft<4>::run(t);
            GBFFT_UNROLL
            for (int k2 = 0; k2 < 4; ++k2) z[n1][k2] = t[k2];
        }
        {
            Pair t[4] = {z[0][0], z[1][0], z[2][0], z[3][0]};
            PairDft<4>::run(t);
            x[0] = t[0];
            x[4] = t[1];
            x[8] = t[2];
            x[12] = t[3];
        }
        const float2 tn = pset(kTan1_16), ntn = pset(-kTan1_16);
        {  // k2 = 1
            const Pair a = z[1][1], b = z[3][1], q = z[2][1];
            const Pair p1 = Pair{pfma(a.im, tn, a.re), pfma(a.re, ntn, a.im)};       // a (1 - i t)
            // b (t - i): (t re + im, t im - re)
            const Pair p3 = Pair{pfma(b.re, tn, b.im), pfma(b.im, tn, pneg(b.re))};
            const Pair q2 = sub_i(q, q);  // q (1 - i)
            const Pair s02 = pair_fma(kSqrtHalf, q2, z[0][1]), d02 = pair_fma(-kSqrtHalf, q2, z[0][1]);
            const Pair P = p1 + p3, Q = p1 - p3;
            x[1] = pair_fma(kCos1_16, P, s02);
            x[5] = pair_fma_mi(kCos1_16, Q, d02);
            x[9] = pair_fma(-kCos1_16, P, s02);
            x[13] = pair_fma_mi(-kCos1_16, Q, d02);
        }
        {  // k2 = 2
            const Pair a = z[1][2], b = z[3][2];
            const Pair q1 = sub_i(a, a);
            const Pair q3 = Pair{psub(b.im, b.re), padd(b.re, b.im)};  // re, -im of b (-1 - i)
            const Pair s02 = sub_i(z[0][2], z[2][2]), d02 = add_i(z[0][2], z[2][2]);
            const Pair S = Pair{padd(q1.re, q3.re), psub(q1.im, q3.im)};
            const Pair D = Pair{psub(q1.re, q3.re), padd(q1.im, q3.im)};
            x[2] = pair_fma(kSqrtHalf, S, s02);
            x[6] = pair_fma_mi(kSqrtHalf, D, d02);
            x[10] = pair_fma(-kSqrtHalf, S, s02);
            x[14] = pair_fma_mi(-kSqrtHalf, D, d02);
        }
        {  // k2 = 3
            const Pair a = z[1][3], b = z[3][3], q = z[2][3];
            const Pair p1 = Pair{pfma(a.re, tn, a.im), pfma(a.im, tn, pneg(a.re))};  // a (t - i)
            const Pair p3 = Pair{pfma(b.im, tn, b.re), pfma(b.re, ntn, b.im)};       // b (1 - i t)
            const Pair q2 = Pair{psub(q.im, q.re), padd(q.re, q.im)};                // re, -im of q (-1 - i)
            const Pair s02 = Pair{pfma(pset(kSqrtHalf), q2.re, z[0][3].re), pfma(pset(-kSqrtHalf), q2.im, z[0][3].im)};
            const Pair d02 = Pair{pfma(pset(-kSqrtHalf), q2.re, z[0][3].re), pfma(pset(kSqrtHalf), q2.im, z[0][3].im)};
            const Pair P = p1 - p3, Q = p1 + p3;
            x[3] = pair_fma(kCos1_16, P, s02);
            x[7] = pair_fma_mi(kCos1_16, Q, d02);
            x[11] = pair_fma(-kCos1_16, P, s02);
            x[15] = pair_fma_mi(-kCos1_16, Q, d02);
        }
    }
};

// a * W_16^I for a compile-time I.
template <int I>
GBFFT_HD Pair pair_mul_w16c(Pair a) {
    constexpr int i = I & 15;
    if constexpr (i == 0) return a;
    else if constexpr (i >= 8) {
        const Pair b = pair_mul_w16c<i - 8>(a);
        return Pair{pneg(b.re), pneg(b.im)};
    } else if constexpr (i >= 4) {
        const Pair b = pair_mul_w16c<i - 4>(a);
        return Pair{b.im, pneg(b.re)};
    } else if constexpr (i == 2) {
        return Pair{pmul(padd(a.re, a.im), pset(kSqrtHalf)), pmul(psub(a.im, a.re), pset(kSqrtHalf))};
    } else {  // 1, 3: a (c - i s)
        constexpr float c = i == 1 ? kCos1_16 : kSin1_16, s = i == 1 ? kSin1_16 : kCos1_16;
        return Pair{pfma(a.re, pset(c), pmul(a.im, pset(s))), pfma(a.im, pset(c), pmul(a.re, pset(-s)))};
    }
}

}  // namespace gbfft
