// Adjoint of the Chambolle TV (fixed number of updates) on register tiles.
//
// Per dual update k (last to first): with g_k = grad u_k, n_k = |g_k|,
// r_k = 1 / (1 + tw n_k) and p_{k+1} = r_k (p_k - tau g_k):
//   gbar_k = -tau r_k pbar_{k+1} - (tw r_k / n_k) <pbar_{k+1}, p_{k+1}> g_k
//            (0 for the second term where g_k = 0)
//   ubar_k = -div gbar_k;  fbar += ubar_k;  pbar_k = r_k pbar_{k+1} + grad ubar_k
// from pbar_U = grad xbar, fbar = xbar (u_U = f - div p_U with ubar_U = xbar).
//
// All updates of a window in one block, laid out as the forward's tiles
// (sci_tv_tile.cuh): pairs of rows packed, pbar and fbar in registers
// throughout, u_k and p_{k+1} of the window loaded once per update (the tape;
// 11 planes in all), two barriers per update for the rows of gbar and ubar
// that cross warps, HALO rings of halo.  One launch per outer iteration
// instead of one per update: xbar in, fbar out and the tape are all that
// moves (13 planes; pbar and fbar made it 33).
#pragma once

#include "sci_tv_tile.cuh"

namespace sci {
namespace tv {
namespace tile {

struct Adj {
    // u_0 = f + lam (q phi) as load_f's PROJ 2 forms it
    const float *f;       // [nf][H][W]
    const float *cmap, *phi, *lam_dev;
    int frame0, B;
    const float *tape_u;  // u_1 .. u_{U-1}: [U-1][nf][H][W]
    const float *tape_p;  // 4 p_1 .. 4 p_U: [U][nf][2][H][W]
    const float *xbar;
    float *fbar;
    int nf, H, W, U, nbands, nchunks, vec;
    float tw;
    int early;  // more blocks than fit at once
};

template <int C, int N, int NW, int MODE>
__device__ __forceinline__ void adjoint(const Adj &P, int frame, int tr, int tc,
                                        Smem<C, NW> &sm) {
    using G = Geo<C, N, NW>;
    constexpr bool EDGE = MODE != INSIDE;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int H = P.H, W = P.W;
    int c0, own_c0, own_c1, t0, own_r0, own_r1;
    window(W, G::COLS, tc, P.nbands, c0, own_c0, own_c1);
    window(H, G::ROWS, tr, P.nchunks, t0, own_r0, own_r1);
    const int col = c0 + C * lane, row = t0 + 2 * N * w;
    const int64_t hw = (int64_t)H * W;

    if (EDGE && row >= H) {  // a warp below the frame only keeps the barriers
        const float zero[C] = {};
        sm.u.put(w, lane, zero);
        for (int k = P.U - 1; k >= 0; --k) {
            __syncthreads();
            if (k > 0) __syncthreads();
        }
        return;
    }
    const Cells<C, N, MODE> X(t0, row, col, H, W);
    // the row below a thread's rows (past an inner window's last: any row, it
    // is halo)
    const auto below_off = X.at(min(row + 2 * N, H - 1), col, max(t0 - 1, 0), H, W);
    const bool below_in = row + 2 * N < H;
    // forward differences of pair (j, c), 0 across the frame's last row / column
    auto grad = [&](const f2 (&v)[N][C], const float (&below)[C], const f2 right_lane, int j, int c,
                    f2 &gr, f2 &gc) {
        const f2 right = c + 1 < C ? v[j][c + 1 < C ? c + 1 : 0] : right_lane;
        const f2 dn = j + 1 < N ? v[j + 1 < N ? j + 1 : 0][c] : mk2(hi(v[0][c]), below[c]);
        gr = sub2(dn, v[j][c]);
        gc = sub2(right, v[j][c]);
        if (EDGE) {
            if (col + c >= W - 1) gc.v = 0ull;
            gr = mk2(row + j >= H - 1 ? 0.f : lo(gr), row + N + j >= H - 1 ? 0.f : hi(gr));
        }
    };

    f2 fb[N][C], br[N][C], bc[N][C];
    {
        const float *xb = P.xbar + (int64_t)frame * hw;
        float below[C];
        X.load(xb, fb);
        X.load(xb, below_off, below_in, below);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const f2 right = shfl_dn(fb[j][0]);
#pragma unroll
            for (int c = 0; c < C; ++c) grad(fb, below, right, j, c, br[j][c], bc[j][c]);
        }
    }
    const f2 one2 = mk2(1.f, 1.f), tw2 = mk2(P.tw, P.tw), ntau2 = mk2(-0.25f, -0.25f);
    const f2 ntw4 = mk2(-0.25f * P.tw, -0.25f * P.tw);  // the tape holds 4 p
    for (int k = P.U - 1; k >= 0; --k) {
        const float *uk = (k == 0 ? P.f : P.tape_u + (int64_t)(k - 1) * P.nf * hw) +
                          (int64_t)frame * hw;
        const float *pk = P.tape_p + ((int64_t)k * P.nf + frame) * 2 * hw;
        f2 u[N][C], gr[N][C], gc[N][C], ri[N][C];
        float below[C];
        if (k == 0) {
#pragma unroll
            for (int j = 0; j < N; ++j) {
                float a[2][C];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    load_f<2>(P, X, uk, frame, X.off[h][j], X.inside(h, j), a[h]);
#pragma unroll
                for (int c = 0; c < C; ++c) u[j][c] = mk2(a[0][c], a[1][c]);
            }
            load_f<2>(P, X, uk, frame, below_off, below_in, below);
        } else {
            X.load(uk, u);
            X.load(uk, below_off, below_in, below);
        }
        X.load(pk, gr);  // p until gbar takes its place
        X.load(pk + hw, gc);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const f2 right = shfl_dn(u[j][0]);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                f2 g1, g2;
                grad(u, below, right, j, c, g1, g2);
                const f2 s = fma2(g1, g1, mul2(g2, g2));
                // n is 0 or at least 1.08e-19 (the root of the least normal
                // number). Below that |g| gives n = 0 and the bound stands for
                // it: the second term is then 0 where g is, and else at most
                // tw |pbar| |p|, as for any g
                const float n0 = sqrt_approx(lo(s)), n1 = sqrt_approx(hi(s));
                const f2 den = fma2(tw2, mk2(n0, n1), one2);
                ri[j][c] = mk2(rcp_approx(lo(den)), rcp_approx(hi(den)));
                const f2 in = mk2(rcp_approx(fmaxf(n0, 1e-19f)), rcp_approx(fmaxf(n1, 1e-19f)));
                const f2 dot = fma2(bc[j][c], gc[j][c], mul2(br[j][c], gr[j][c]));
                const f2 coef = mul2(mul2(mul2(ntw4, ri[j][c]), dot), in);
                const f2 tr = mul2(ntau2, ri[j][c]);
                gr[j][c] = fma2(tr, br[j][c], mul2(coef, g1));
                gc[j][c] = fma2(tr, bc[j][c], mul2(coef, g2));
                if (EDGE) {
                    if (col + c >= W - 1) gc[j][c].v = 0ull;
                    gr[j][c] = mk2(row + j >= H - 1 ? 0.f : lo(gr[j][c]),
                                   row + N + j >= H - 1 ? 0.f : hi(gr[j][c]));
                }
            }
        }
        // ubar = -div gbar, into u
        float edge[C], above[C];
#pragma unroll
        for (int c = 0; c < C; ++c) edge[c] = hi(gr[N - 1][c]), above[c] = 0.f;
        sm.p.put(w, lane, edge);
        __syncthreads();
        if (w > 0) sm.p.get(w - 1, lane, above);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            f2 left_lane = shfl_up(gc[j][C - 1]);
            if (lane == 0) left_lane.v = 0ull;  // column -1, or halo
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const f2 up = j > 0 ? gr[j > 0 ? j - 1 : 0][c] : mk2(above[c], lo(gr[N - 1][c]));
                const f2 left = c > 0 ? gc[j][c > 0 ? c - 1 : 0] : left_lane;
                u[j][c] = sub2(left, sub2(add2(gr[j][c], gc[j][c]), up));
                fb[j][c] = add2(fb[j][c], u[j][c]);
            }
        }
        if (k == 0) break;
        // pbar_k = r_k pbar_{k+1} + grad ubar
#pragma unroll
        for (int c = 0; c < C; ++c) edge[c] = lo(u[0][c]), below[c] = hi(u[N - 1][c]);
        sm.u.put(w, lane, edge);
        __syncthreads();
        if (w + 1 < NW) sm.u.get(w + 1, lane, below);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const f2 right = shfl_dn(u[j][0]);
#pragma unroll
            for (int c = 0; c < C; ++c) {
                f2 g1, g2;
                grad(u, below, right, j, c, g1, g2);
                br[j][c] = fma2(ri[j][c], br[j][c], g1);
                bc[j][c] = fma2(ri[j][c], bc[j][c], g2);
            }
        }
    }
    const bool cols = col >= own_c0 && col < own_c1;
    X.store(P.fbar + (int64_t)frame * hw, fb, cols && row >= own_r0 && row < own_r1,
            cols && row + N >= own_r0 && row + N < own_r1);
}

template <int C, int N, int NW, int MINB>
__global__ void __launch_bounds__(NW * 32, MINB) k_tv_adjoint(Adj P) {
    __shared__ Smem<C, NW> sm;
    grid_dep_wait();
    if (P.early) grid_dep_launch();
    const unsigned t = blockIdx.x / (unsigned)P.nbands;  // windows of a frame adjacent
    const int tc = (int)(blockIdx.x - t * (unsigned)P.nbands);
    const int frame = (int)(t / (unsigned)P.nchunks);
    const int tr = (int)(t - (unsigned)frame * (unsigned)P.nchunks);
    const bool edge = tr == P.nchunks - 1 || tc == P.nbands - 1;
    if (P.vec < 0) adjoint<C, N, NW, EDGE_WIDE>(P, frame, tr, tc, sm);
    else if (!P.vec) adjoint<C, N, NW, EDGE_SCALAR>(P, frame, tr, tc, sm);
    else if (edge) adjoint<C, N, NW, EDGE_VEC>(P, frame, tr, tc, sm);
    else adjoint<C, N, NW, INSIDE>(P, frame, tr, tc, sm);
}

}  // namespace tile
}  // namespace tv
}  // namespace sci
