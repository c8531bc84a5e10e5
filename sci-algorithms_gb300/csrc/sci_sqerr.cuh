// Sum of squared float32 differences to float64 accuracy without float64
// arithmetic in the loop (a GB300 SM does two float64 FMAs per clock against
// 128 in float32): each square is an exact float32 product pair of an exact
// difference pair, and the pairs are added with compensated float32
// additions (relative error about 2^-45).  Differences whose squares float32
// cannot hold so, and values that are not numbers, take a float64 branch.
#pragma once

#include "sci_common.cuh"

namespace sci {

// Sum of terms with its rounding errors: hi + lo.
struct Comp {
    float hi, lo;
    __device__ __forceinline__ void add(float v, float v_lo) {
        const float t = hi + v, z = t - hi;
        lo += ((hi - (t - z)) + (v - z)) + v_lo;
        hi = t;
    }
    // An infinite total has no rounding error (inf - inf is not one).
    __device__ __forceinline__ double take() {
        const double r = isfinite(hi) ? (double)hi + (double)lo : (double)hi;
        hi = lo = 0.f;
        return r;
    }
};

struct SquareSum {
    Comp c;
    double wide;
    __device__ __forceinline__ void clear() {
        c = {0.f, 0.f};
        wide = 0.0;
    }
    // Adds (x_k - y_k)^2, given d_k = x_k - y_k rounded, k < 4.  Called by
    // the active lanes of a warp together.
    __device__ __forceinline__ void add4(const float (&x)[4], const float (&y)[4],
                                         const float (&d)[4]) {
        // differences of 0 or of 1e-12 to 1e18: their bits less one, as
        // unsigned, put 0 last; a vote, so that the float64 form is not
        // issued under a predicate by every warp
        unsigned most = 0u, least = ~0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const unsigned m = __float_as_uint(d[k]) & 0x7fffffffu;
            most = max(most, m);
            least = min(least, m - 1u);
        }
        const bool out = most > __float_as_uint(1e18f) || least < __float_as_uint(1e-12f);
        if (__any_sync(__activemask(), out)) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const double e = (double)x[k] - (double)y[k];
                wide += e * e;
            }
            return;
        }
        // x - y = d + dl exactly; d^2 = t + its rounding error.  The
        // products are scalar: ptxas contracts a packed product and a packed
        // sum into an FMA, explicit rounding or not, and the error terms
        // need the rounded product.
        f2 t[2], e[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float d0 = d[2 * h], d1 = d[2 * h + 1];
            const f2 X = mk2(x[2 * h], x[2 * h + 1]), Y = mk2(y[2 * h], y[2 * h + 1]);
            const f2 D = mk2(d0, d1), z = sub2(D, X);
            const f2 dl = sub2(sub2(X, sub2(D, z)), add2(Y, z));
            t[h] = mk2(__fmul_rn(d0, d0), __fmul_rn(d1, d1));
            e[h] = fma2(add2(D, D), dl, fma2(D, D, sub2(mk2(0.f, 0.f), t[h])));
        }
        // t[0] + t[1], exactly as a sum and its error, then into the total
        const f2 u = add2(t[0], t[1]), z = sub2(u, t[0]);
        const f2 ue = add2(add2(sub2(t[0], sub2(u, z)), sub2(t[1], z)), add2(e[0], e[1]));
        c.add(lo(u), lo(ue));
        c.add(hi(u), hi(ue));
    }
    __device__ __forceinline__ void add4(float4 a, float4 b) {
        const float x[4] = {a.x, a.y, a.z, a.w}, y[4] = {b.x, b.y, b.z, b.w};
        const float d[4] = {a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w};
        add4(x, y, d);
    }
    __device__ __forceinline__ double take() {
        const double r = c.take() + wide;
        wide = 0.0;
        return r;
    }
};

}  // namespace sci
