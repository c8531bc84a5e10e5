// Sum of squared float32 differences as accurate as float64 arithmetic gives
// it, without float64 in the loop (a GB300 SM does two float64 FMAs per clock
// against 128 in float32): the difference, its square and the additions are
// carried with their rounding errors (error-free transformations: Knuth's
// two-sum and two-difference, the product's error by FMA) in three float32
// words.  Differences whose squares float32 cannot hold so, and values that
// are not numbers, take a float64 branch.
//
// Two words are not enough, although a sum of random roundings would average
// out: an odd square is 1 mod 8, so where its last bit is rounded off alone
// the tie always falls to the even side below, and the sum lost 1 to 3e-15 of
// itself at differences of 0.1 to 0.3.  Relative error of the sums of 32
// elements that a thread adds before float64 takes over, differences of 0.03 /
// 0.3 / a constant: 3e-17 / 5e-17 / 5e-17 (float64: 4e-17 / 1.1e-16 / 4.6e-16).
//
// What bounds it: issue, about 90 instructions for four elements (60 where
// the vote below finds the differences exact).  k_sqerr at 2048 x 2048 x 8 and
// x 24: 52 and 148 us (two words 47 and 136, float64 254 and 742).
#pragma once

#include "sci_common.cuh"

namespace sci {

// Sum of terms with its rounding errors: hi + lo.
struct Comp {
    float hi, lo;
    __device__ __forceinline__ void add(float v) {
        const float t = hi + v, z = t - hi;
        lo += (hi - (t - z)) + (v - z);
        hi = t;
    }
    // An infinite total has no rounding error (inf - inf is not one).
    __device__ __forceinline__ double take() {
        const double r = isfinite(hi) ? (double)hi + (double)lo : (double)hi;
        hi = lo = 0.f;
        return r;
    }
};

// a + b rounded; err the rest, exactly.
__device__ __forceinline__ f2 two_sum(f2 a, f2 b, f2 &err) {
    const f2 t = add2(a, b), z = sub2(t, a);
    err = add2(sub2(a, sub2(t, z)), sub2(b, z));
    return t;
}

// a b rounded; err the rest, exactly.  The product is formed by halves: ptxas
// contracts a packed product and a packed sum into an FMA, explicit rounding or
// not, and the rest needs the rounded product.
__device__ __forceinline__ f2 two_mul(f2 a, f2 b, f2 &err) {
    const f2 t = mk2(__fmul_rn(lo(a), lo(b)), __fmul_rn(hi(a), hi(b)));
    err = fma2(a, b, sub2(mk2(0.f, 0.f), t));
    return t;
}

struct SquareSum {
    // Calls of add4 between two of take() at most: a word then holds 128 squares
    // of at most 1e36.  take() is a dozen float64 operations, 16 clocks of the
    // SM's float64 pipe each and warp: with one for 8 calls k_sqerr took 160 us
    // at 2048 x 2048 x 24 instead of 148.
    static constexpr int kMost = 64;
    f2 s0, s1, s2;  // sum of the even and the odd elements, in three words
    double wide;
    __device__ __forceinline__ void clear() {
        s0.v = s1.v = s2.v = 0ull;
        wide = 0.0;
    }
    // Adds (x_k - y_k)^2, given d_k = x_k - y_k rounded, k < 4.  Called by
    // the active lanes of a warp together.
    __device__ __forceinline__ void add4(const float (&x)[4], const float (&y)[4],
                                         const float (&d)[4]) {
        // The largest difference is 0 or 1e-12 to 1e18: its square holds the
        // words of all four (what the others' lose below 1e-45 is 2^-69 of it).
        constexpr unsigned least = 0x2b8cbcccu, span = 0x5d5e0b6bu - least;  // 1e-12f, 1e18f
        unsigned most = 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) most = max(most, __float_as_uint(d[k]) & 0x7fffffffu);
        const bool out = most != 0u && most - least > span;
        // x - y = d + dl exactly, (d + dl)^2 = d^2 + 2 d dl + dl^2: words t (of
        // d^2), m (about 2^-24 of it) and l (2^-48)
        f2 D[2], dl[2], t[2], m[2], l[2];
        unsigned rest = 0u;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const f2 X = mk2(x[2 * h], x[2 * h + 1]), Y = mk2(y[2 * h], y[2 * h + 1]);
            D[h] = mk2(d[2 * h], d[2 * h + 1]);
            const f2 z = sub2(D[h], X);
            dl[h] = sub2(sub2(X, sub2(D[h], z)), add2(Y, z));
            t[h] = two_mul(D[h], D[h], m[h]);
            l[h].v = 0ull;
            rest |= __float_as_uint(lo(dl[h])) | __float_as_uint(hi(dl[h]));
        }
        // Values within a factor of two of each other differ exactly: a vote
        // mostly leaves the rest out where the frames agree, and the float64
        // form, which would otherwise be issued under a predicate by every warp.
        const unsigned lanes = __activemask();
        if (__any_sync(lanes, out || (rest << 1) != 0u)) {
            if (__any_sync(lanes, out)) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const double e = (double)x[k] - (double)y[k];
                    wide += e * e;
                }
                return;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                f2 pe, me;
                const f2 p = two_mul(add2(D[h], D[h]), dl[h], pe);
                m[h] = two_sum(m[h], p, me);
                l[h] = add2(fma2(dl[h], dl[h], pe), me);
            }
        }
        // the two pairs to one, then into the total
        f2 e0, e1, e2, e3, e4;
        const f2 tt = two_sum(t[0], t[1], e0);
        const f2 mm = two_sum(e0, two_sum(m[0], m[1], e1), e2);
        s0 = two_sum(s0, tt, e0);
        s1 = two_sum(s1, two_sum(e0, mm, e3), e4);
        s2 = add2(s2, add2(add2(add2(e1, e2), add2(e3, e4)), add2(l[0], l[1])));
    }
    __device__ __forceinline__ void add4(float4 a, float4 b) {
        const float x[4] = {a.x, a.y, a.z, a.w}, y[4] = {b.x, b.y, b.z, b.w};
        const float d[4] = {a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w};
        add4(x, y, d);
    }
    __device__ __forceinline__ double take() {
        const double r = (((double)lo(s0) + (double)hi(s0)) +
                          (((double)lo(s1) + (double)hi(s1)) + (double)(lo(s2) + hi(s2)))) +
                         wide;
        clear();
        return r;
    }
};

}  // namespace sci
