// Per-frame PSNR and SSIM of a reconstructed stack against the ground truth
// in one pass: the diagnostics the drivers report per coded-frame block
// (compare_psnr / compare_ssim with data_range = 1, PnP_SCI/python/
// pnp_sci_algo.py:702-705, joint_pnp_sci_algo.py, scikit-image 0.16).
//
// SSIM (Wang et al. 2004, scikit-image's defaults): 7 x 7 uniform windows,
// sample covariance (N / (N - 1)), K1 = 0.01, K2 = 0.03, averaged over the
// frame cropped by 3 pixels.  Every window of the cropped region lies inside
// the frame, so the border extension of the uniform filter never enters the
// mean.
//
// What bounds it.  Two frames are read once (8 bytes per pixel), 0.04 ms at
// 2048 x 2048 x 8; the arithmetic of the windows is what costs.  With the
// SSIM of a window in float64 (about 45 operations a pixel on a part that
// does two float64 FMAs per clock and SM) and every window summed from
// shared memory anew (196 loads a pixel) the pass took 3.5 ms.  Here:
//
//  * A warp owns a band of 128 columns (4 per lane) of one frame and marches
//    down a chunk of rows with the last 7 rows in registers, so that a row
//    is loaded once per band and window sums are separable: the moments of
//    each 7-row column segment first, then of 7 neighbouring columns (6 of
//    them shuffled in per lane of 4).
//  * Moments are merged, not subtracted: sum (p - m)^2 of a column about its
//    own mean, then sum over columns of those plus the spread of the column
//    means.  No cancellation.
//  * The two moments needed are those of s = x + y and d = x - y, carried as
//    one packed pair: with B1 = Mx^2 + My^2 + C1 and B2 = Vx + Vy + C2,
//      SSIM = (1 - Md^2 / B1) (1 - Vd / B2),
//      Mx^2 + My^2 = (Ms^2 + Md^2) / 2,  Vx + Vy = (Vs + Vd) / 2,
//    so 1 - SSIM = e1 + e2 - e1 e2 is a sum of float32 quotients that are
//    small where the images agree; its rounding is relative to 1 - SSIM.
//  * Sums: squared errors (sci_sqerr.cuh) over 64 rows and 1 - SSIM, with
//    compensated float32 additions, over 8 rows, then in float64.
//
// Measured at 2048 x 2048 x 8: 0.202 ms for the kernel (3.4 ms in float64),
// 0.184 of it without the squared error's third word and the windows' range
// check; the packed float32 arithmetic of the windows bounds it (no spills at
// 3 blocks per SM; 4 blocks spill).  Against float64 (rms over frames, this
// kernel / float64 quotients of float32 moments): mean SSIM at noise 0.003 2e-12
// to 2e-11 / 4e-10 to 2e-9, at 0.03 4e-11 to 3e-10 / 3e-10 to 2e-9 (64 x 64 to
// 2048 x 2048).  The rounding of x + y is shared by the 49 windows of a pixel,
// so between frames that differ more it averages out less than roundings of
// each window's own: at 0.1 2e-10 to 1.4e-9 / 1e-11 to 1e-9, at 0.3 7e-11 to
// 2e-9 / 1e-12 to 5e-10.  PSNR: as float64 gives it.
#include <algorithm>

#include "sci_sqerr.cuh"

namespace sci {
namespace {

constexpr int R = 3, WIN = 2 * R + 1;
constexpr int WPB = 4;           // warps per block
constexpr int BAND = 128;        // columns of a warp's window, 4 per lane
constexpr int HALO = 4;          // its first and last columns, owned by the neighbours
constexpr int OWN = BAND - 2 * HALO;
constexpr int MIN_ROWS = 8;      // rows per chunk at least (6 more are read)
constexpr int RESIDENT = 3;      // blocks per SM the registers are sized for

struct Metrics {
    const float *a, *b;
    double *sqerr, *ssim_sum;
    int H, W, rows, nbands, nchunks;
    int64_t items;
    float scale;         // power of two near 1 / data_range, for the windows
    // 49^2 C1 and 7 48 C2 of the scaled frames, as pairs
    float c1, c1_lo, c2, c2_lo;
    double C1, C2;       // of the frames as they are
};

// 1 - SSIM of the window around (i, j), its moments about the means as float32
// sums over the window and the quotient in float64, of the frames as they are:
// for windows whose squared sums the packed form cannot hold (frames far
// outside the data range) and those with a value that is not a number.
__device__ __forceinline__ double wide_window(const float *a, const float *b, int W, int i, int j,
                                              double C1, double C2) {
    float sx = 0.f, sy = 0.f, vx = 0.f, vy = 0.f, vxy = 0.f, mx = 0.f, my = 0.f;
#pragma unroll 1
    for (int t = 0; t < 2 * WIN; ++t) {
        const int64_t p = (int64_t)(i - R + (t < WIN ? t : t - WIN)) * W + (j - R);
        if (t == WIN) {
            mx = sx * (1.f / (WIN * WIN));
            my = sy * (1.f / (WIN * WIN));
        }
#pragma unroll 1
        for (int v = 0; v < WIN; ++v) {
            const float x = a[p + v], y = b[p + v], dx = x - mx, dy = y - my;
            if (t < WIN) {
                sx += x;
                sy += y;
            } else {
                vx = fmaf(dx, dx, vx);
                vy = fmaf(dy, dy, vy);
                vxy = fmaf(dx, dy, vxy);
            }
        }
    }
    const double n = 1.0 / (WIN * WIN - 1), Mx = mx, My = my;
    return 1.0 - ((2.0 * Mx * My + C1) * (2.0 * (n * vxy) + C2)) /
                     ((Mx * Mx + My * My + C1) * (n * vx + n * vy + C2));
}

// v / (h + c + c_lo).  The rounding of h + c goes into the reciprocal's
// Newton step: left out, it has one sign for whole binades of h (c's last
// bits are the same everywhere), a bias of the mean by up to 2^-25.
__device__ __forceinline__ float quotient(float v, float h, float c, float c_lo) {
    const float b = h + c, err = (c - (b - h)) + c_lo;
    const float q = rcp_approx(b);
    return v * fmaf(q, fmaf(-err, q, fmaf(-b, q, 1.f)), q);
}

template <bool VEC>
__device__ __forceinline__ float4 load4(const float *p, int col, int W) {
    if (VEC) return col < W ? ldg4(p + col) : make_float4(0.f, 0.f, 0.f, 0.f);
    return make_float4(col < W ? __ldg(p + col) : 0.f, col + 1 < W ? __ldg(p + col + 1) : 0.f,
                       col + 2 < W ? __ldg(p + col + 2) : 0.f,
                       col + 3 < W ? __ldg(p + col + 3) : 0.f);
}

__device__ __forceinline__ f2 shfl_up2(f2 v) {
    f2 r;
    r.v = __shfl_up_sync(0xffffffffu, v.v, 1);
    return r;
}
__device__ __forceinline__ f2 shfl_down2(f2 v) {
    f2 r;
    r.v = __shfl_down_sync(0xffffffffu, v.v, 1);
    return r;
}

// VEC: rows are aligned for 16-byte loads (W % 4 == 0).
template <bool VEC>
__global__ void __launch_bounds__(WPB * 32, RESIDENT) k_frame_metrics(Metrics P) {
    const int64_t item = (int64_t)blockIdx.x * WPB + (threadIdx.x >> 5);
    if (item >= P.items) return;
    const int lane = threadIdx.x & 31, H = P.H, W = P.W;
    const int band = (int)(item % P.nbands);
    const int64_t q = item / P.nbands;
    const int chunk = (int)(q % P.nchunks);
    const int64_t frame = q / P.nchunks;
    const int c0 = band * OWN, col = c0 + 4 * lane;
    const int own_lo = band == 0 ? 0 : c0 + HALO;
    const int own_hi = band == P.nbands - 1 ? W : c0 + BAND - HALO;
    const int r0 = chunk * P.rows, r1 = min(r0 + P.rows, H);
    const int q0 = max(0, r0 - R), q1 = min(H, r1 + R);   // input rows
    const int i0 = max(r0, R), i1 = min(r1, H - R);       // window centres
    const float *pa = P.a + frame * H * W, *pb = P.b + frame * H * W;
    // owned columns are whole lanes (own_lo, own_hi are multiples of 4, and
    // columns past the frame read as 0 in both frames); the windows' are not
    const bool own = col >= own_lo && col < own_hi;
    float win[4];
    int wins = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const bool w = own && col + k >= R && col + k < W - R;
        win[k] = w ? 1.f : 0.f;
        wins += w;
    }

    const f2 seventh = mk2(1.f / 7.f, 1.f / 7.f), seven = mk2(7.f, 7.f);
    f2 p[WIN + 1][4];  // (s, d) of rows row - 6 .. row + 1
#pragma unroll
    for (int r = 0; r <= WIN; ++r)
#pragma unroll
        for (int k = 0; k < 4; ++k) p[r][k].v = 0ull;
    SquareSum se;
    se.clear();
    Comp ds = {0.f, 0.f};
    double sse = 0.0, dssim = 0.0;

    // A new row: its (s, d), scaled, into slot q, its squared error into the
    // sums (as it is: SquareSum holds any range, and a scaled value could
    // leave float32's).
    auto take_row = [&](float4 va, float4 vb, f2 (&q)[4], bool count) {
        const float x[4] = {va.x, va.y, va.z, va.w}, y[4] = {vb.x, vb.y, vb.z, vb.w};
        float d[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            d[k] = x[k] - y[k];
            q[k] = mk2((x[k] + y[k]) * P.scale, d[k] * P.scale);
        }
        if (count) se.add4(x, y, d);
    };
    // The windows of one row of centres, from the sums of the common six
    // rows and the seventh row `o`; held rows are p[1 .. 6] and o.  Returns
    // the windows left to wide_window, a bit each.
    auto windows = [&](const f2 (&common)[4], const f2 (&o)[4]) {
        unsigned wide = 0u;
        f2 T[10], M[10];  // columns col - 3 .. col + 6: sum and centred sum of squares
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const f2 sum = add2(common[k], o[k]), mean = mul2(sum, seventh);
            f2 c = sub2(o[k], mean), v = mul2(c, c);
#pragma unroll
            for (int r = 1; r < WIN; ++r) {
                c = sub2(p[r][k], mean);
                v = fma2(c, c, v);
            }
            T[k + 3] = sum;
            M[k + 3] = v;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            T[k] = shfl_up2(T[k + 4]);
            M[k] = shfl_up2(M[k + 4]);
            T[k + 7] = shfl_down2(T[k + 3]);
            M[k + 7] = shfl_down2(M[k + 3]);
        }
        // windows: columns k .. k + 6 of the ten, 3 .. 6 in all of them
        const f2 Tc = add2(add2(T[3], T[4]), add2(T[5], T[6]));
        const f2 Mc = add2(add2(M[3], M[4]), add2(M[5], M[6]));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            f2 S = Tc, V = Mc;
#pragma unroll
            for (int c = k; c < k + WIN; ++c)
                if (c < 3 || c > 6) {
                    S = add2(S, T[c]);
                    V = add2(V, M[c]);
                }
            const f2 mean = mul2(S, seventh);  // of the column sums
            f2 d = sub2(T[k], mean), w = mul2(d, d);
#pragma unroll
            for (int c = k + 1; c < k + WIN; ++c) {
                d = sub2(T[c], mean);
                w = fma2(d, d, w);
            }
            // e1 = Md^2 / B1 times 49^2 over 49^2, e2 = Vd / B2 times 7 48
            // over 7 48, so that no factor is rounded
            V = fma2(V, seven, w);
            const f2 S2 = mul2(S, S);
            const float h1 = 0.5f * (lo(S2) + hi(S2)), h2 = 0.5f * (lo(V) + hi(V));
            const float e1 = quotient(hi(S2), h1, P.c1, P.c1_lo);
            const float e2 = quotient(hi(V), h2, P.c2, P.c2_lo);
            const bool held = h1 + h2 < 1e30f;
            ds.add(held ? fmaf(-e1, e2, e1 + e2) * win[k] : 0.f);
            if (!held && win[k] != 0.f) wide |= 1u << k;
        }
        return wide;
    };

    float4 n0a = load4<VEC>(pa + (int64_t)q0 * W, col, W);
    float4 n0b = load4<VEC>(pb + (int64_t)q0 * W, col, W);
    float4 n1a = load4<VEC>(pa + (int64_t)(q0 + 1) * W, col, W);
    float4 n1b = load4<VEC>(pb + (int64_t)(q0 + 1) * W, col, W);
    // two rows at a time: the ring moves by register copies once per pair
    // (48 of them; unrolling it away takes 7 copies of this body, more than
    // the instruction cache holds)
#pragma unroll 1
    for (int row = q0; row < q1; row += 2) {
        take_row(n0a, n0b, p[6], row >= r0 && row < r1);
        take_row(n1a, n1b, p[7], row + 1 >= r0 && row + 1 < r1);
        const int64_t next = (int64_t)min(row + 2, q1 - 1) * W, next1 = (int64_t)min(row + 3, q1 - 1) * W;
        n0a = load4<VEC>(pa + next, col, W);
        n0b = load4<VEC>(pb + next, col, W);
        n1a = load4<VEC>(pa + next1, col, W);
        n1b = load4<VEC>(pb + next1, col, W);
        f2 common[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            common[k] = add2(add2(add2(p[1][k], p[2][k]), add2(p[3][k], p[4][k])),
                             add2(p[5][k], p[6][k]));
        const int i = row - R;  // centre of rows row - 6 .. row
        unsigned wide = 0u;
        if (i >= i0 && i < i1) wide = windows(common, p[0]);
        if (i + 1 >= i0 && i + 1 < i1) wide |= windows(common, p[7]) << 4;
        if ((row & 6) == 6) dssim += ds.take();
        if ((row & (SquareSum::kMost - 2)) == SquareSum::kMost - 2) {  // a call a row
            const double a = se.take();
            sse += own ? a : 0.0;
        }
#pragma unroll
        for (int r = 0; r < WIN - 1; ++r)
#pragma unroll
            for (int k = 0; k < 4; ++k) p[r][k] = p[r + 2][k];
        for (; wide; wide &= wide - 1) {
            const int t = __ffs(wide) - 1;
            dssim += wide_window(pa, pb, W, i + (t >> 2), col + (t & 3), P.C1, P.C2);
        }
        __syncwarp();
    }
    const double a = se.take();
    sse += own ? a : 0.0;
    dssim += ds.take();
    double ss = wins ? (double)wins * max(0, i1 - i0) - dssim : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sse += __shfl_xor_sync(0xffffffffu, sse, o);
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
    }
    if (lane == 0) {
        atomicAdd(P.sqerr + frame, sse);
        atomicAdd(P.ssim_sum + frame, ss);
    }
}

}  // namespace
}  // namespace sci

using namespace sci;

extern "C" int sci_frame_metrics(const float *orig, const float *x, int64_t nframes, int64_t H,
                                 int64_t W, double data_range, double *sqerr, double *ssim_sum,
                                 void *stream) {
    SCI_CHECK_ARG(orig && x && sqerr && ssim_sum, "sci_frame_metrics: null pointer");
    SCI_CHECK_ARG(nframes >= 1 && nframes <= 65535 && H >= WIN && W >= WIN && H <= (1 << 24) &&
                      W <= (1 << 24),
                  "sci_frame_metrics: frames must be at least 7 x 7 (nframes <= 65535)");
    SCI_CHECK_ARG(data_range > 0.0, "sci_frame_metrics: data_range must be > 0");
    const cudaStream_t s = as_stream(stream);
    SCI_CUDA(cudaMemsetAsync(sqerr, 0, sizeof(double) * (size_t)nframes, s));
    SCI_CUDA(cudaMemsetAsync(ssim_sum, 0, sizeof(double) * (size_t)nframes, s));
    Metrics P{};
    P.a = orig;
    P.b = x;
    P.sqerr = sqerr;
    P.ssim_sum = ssim_sum;
    P.H = (int)H;
    P.W = (int)W;
    // frames scaled by a power of two to a data range in [1, 2)
    const int e = std::max(-120, std::min(120, ilogb(data_range)));
    P.scale = (float)ldexp(1.0, -e);
    P.C1 = (0.01 * data_range) * (0.01 * data_range);
    P.C2 = (0.03 * data_range) * (0.03 * data_range);
    const double unscale2 = ldexp(1.0, 2 * e);
    const double c1 = 2401.0 * P.C1 / unscale2, c2 = 336.0 * P.C2 / unscale2;
    P.c1 = (float)c1;
    P.c1_lo = (float)(c1 - P.c1);
    P.c2 = (float)c2;
    P.c2_lo = (float)(c2 - P.c2);
    // the bands' owned columns cover the frame: the last one's reach W
    P.nbands = 1 + (int)std::max<int64_t>(0, (W - BAND + OWN - 1) / OWN);
    // one wave of resident warps: a chunk of r rows reads r + 6, so taller
    // chunks cost less as long as every warp slot has one
    const int64_t cols = nframes * P.nbands, slots = (int64_t)kSMs * RESIDENT * WPB;
    const int64_t most = (H + MIN_ROWS - 1) / MIN_ROWS;
    P.nchunks = (int)std::max<int64_t>(1, std::min(most, slots / cols));
    P.rows = (int)((H + P.nchunks - 1) / P.nchunks);
    P.nchunks = (int)((H + P.rows - 1) / P.rows);
    P.items = cols * P.nchunks;
    const unsigned g = (unsigned)((P.items + WPB - 1) / WPB);
    if (W % 4 == 0 && aligned16(orig) && aligned16(x))
        k_frame_metrics<true><<<g, WPB * 32, 0, s>>>(P);
    else
        k_frame_metrics<false><<<g, WPB * 32, 0, s>>>(P);
    SCI_LAUNCHED("k_frame_metrics");
    return SCI_OK;
}
