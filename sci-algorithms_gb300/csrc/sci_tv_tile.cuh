// Chambolle TV pass on register tiles: all dual updates of a window of one
// frame by one block, every pixel of the window owned by one thread.
//
// The same arithmetic, operation for operation, as the lean row pipeline
// (sci_tv_slim.cuh) with the dual field held as 4 p, so the frames are
// bit-identical; what differs is the schedule.  The row pipeline marches a
// warp down a chunk of rows through a chain of S dependent stages per row:
// on a small frame that chain, not the work, is the time.  Here a block
// holds a window of 32 C columns x 2 N NW rows -- 64 x 48, or 64 x 32 where
// there are few -- thread = C columns x 2 N rows, f, u and p held by the thread
// for all updates (the larger window, at 80 registers, spills 180 to 300 bytes
// of them; more registers and fewer warps were slower), two block barriers per
// update and no chain longer than one update.
//
//  * Pairs.  A packed f32x2 value holds rows j and j + N of a thread's
//    2 N rows (same column), so the neighbour below is the next pair, the
//    neighbour to the right the next column's pair: every addition of the
//    update is packed and no halves are re-paired, except once per update
//    at the seam between the two halves.
//  * Neighbours.  Columns of other lanes by shuffle; the row below a warp's
//    last and the row of p above its first through one shared-memory row per
//    warp, written before and read after the update's two barriers.
//  * Halo.  Windows overlap by HALO = 4 = S rows and columns on each side
//    (flush with the frame's edges, where none is needed): each update
//    invalidates one more ring of an interior window's border.
//  * What bounds it: issue.  About 80 instructions a pixel and pass (4
//    updates: 30 packed FP32, 8 MUFU, 5 shuffles, 14 register moves that
//    pair scalar results), 53-60 % of the issue slots at 24 warps per SM, and
//    1.38 times the pixels in halo.  In a solve, against the row pipeline: 64 x
//    32 windows (32 warps per SM) at 256 x 256 x 8 9 us against 19; 64 x 48 (24
//    warps) at 256 x 256 x 28 17 against 24 and 512 x 512 x 10 21 against 30; 8
//    x 2048 x 2048 takes 180 us against 123, so large frames keep the row
//    pipeline (sci_tv_rule.cuh).
//  * Stop test as in the row pipeline: per-frame float64 energies, the last
//    block decides (k_tv_tile), a second launch of the same body with the
//    shorter update count rewrites the frames that stop (k_tv_tile_fix).
#pragma once

#include <type_traits>

#include "sci_tv.cuh"

namespace sci {
namespace tv {
namespace tile {

constexpr int HALO = SMAX;

template <int C, int N, int NW>
struct Geo {
    static_assert(C == 2, "loads, stores and exchanges are of two columns");
    static constexpr int COLS = 32 * C, ROWS = 2 * N * NW;
};

// Window `i` of an axis of n cells starts at i * (width - 2 HALO) and owns
// what lies HALO or more cells inside it (all of it at the frame's edges).
// The last one may reach past the frame: cells outside read as 0 and stay 0
// (no gradient crosses the last row or column), so they add nothing.
__host__ __device__ inline int window_count(int n, int width) {
    const int own = width - 2 * HALO;
    return n <= width ? 1 : 1 + (n - width + own - 1) / own;
}
__device__ __forceinline__ void window(int n, int width, int i, int count, int &start, int &lo,
                                       int &hi) {
    start = i * (width - 2 * HALO);
    lo = i == 0 ? 0 : start + HALO;
    hi = i == count - 1 ? n : start + width - HALO;
}

// How a window's rows are read and written: aligned vectors of a window
// inside the frame; aligned vectors with bounds; scalars with bounds; the same
// where a window's rows span 4 GB or more.
enum { INSIDE = 0, EDGE_VEC = 1, EDGE_SCALAR = 2, EDGE_WIDE = 3 };

// Where a thread's rows lie in every plane of a frame: a base per window (the
// same for the block) and a byte offset per row, formed once, so that a load
// or store costs one addition.  Offsets are 32 bits but for EDGE_WIDE.  Rows
// and columns outside the frame are clamped into it and their
// values replaced by 0.
template <int C, int N, int MODE>
struct Cells {
    static constexpr bool SCALAR = MODE >= EDGE_SCALAR;
    using Off = typename std::conditional<MODE == EDGE_WIDE, int64_t, unsigned>::type;
    int64_t base;    // element offset of the window's row max(t0 - 1, 0)
    Off off[2][N];   // rows row + j + h N
    int rows, cols;  // of the thread's cells, how many lie inside the frame
    unsigned step;   // scalars: bytes to the second column (0 outside)

    __device__ __forceinline__ Off at(int r, int col, int tb, int H, int W) const {
        const int c = SCALAR ? min(col, W - 1) : (MODE == INSIDE ? col : min(col, W - C));
        return ((Off)((MODE == INSIDE ? r : min(r, H - 1)) - tb) * (Off)W + (Off)c) * 4;
    }
    __device__ __forceinline__ Cells(int t0, int row, int col, int H, int W) {
        const int tb = max(t0 - 1, 0);
        base = (int64_t)tb * W;
        rows = H - row;
        cols = W - col;
        step = cols > 1 ? 4u : 0u;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < N; ++j)
                off[h][j] = MODE == INSIDE ? at(row, col, tb, H, W) + (Off)(j + h * N) * (Off)W * 4
                                           : at(row + j + h * N, col, tb, H, W);
    }
    // Plain loads, not the read-only path: with programmatic launches the
    // rows may be written by the kernel before while this one's blocks
    // already wait.
    __device__ __forceinline__ void load(const float *plane, Off o, bool row_in,
                                         float (&v)[C]) const {
        const char *p = reinterpret_cast<const char *>(plane + base), *q = p + o;
        if (SCALAR) {
            // in this order: the two loads touch the same sectors, and a row's
            // lines leave L1 before a second sweep over the rows
            float a, b;
            asm volatile("ld.global.f32 %0, [%1];" : "=f"(a) : "l"(q));
            asm volatile("ld.global.f32 %0, [%1];" : "=f"(b) : "l"(p + (Off)(o + step)));
            v[0] = row_in && cols > 0 ? a : 0.f;
            v[C - 1] = row_in && cols > 1 ? b : 0.f;
            return;
        }
        const float2 t = *reinterpret_cast<const float2 *>(q);
        v[0] = t.x, v[1] = t.y;
        if (MODE != INSIDE) {
#pragma unroll
            for (int c = 0; c < C; ++c) v[c] = row_in && cols > 0 ? v[c] : 0.f;
        }
    }
    __device__ __forceinline__ bool inside(int h, int j) const {
        return MODE == INSIDE || j + h * N < rows;
    }
    __device__ __forceinline__ void load(const float *plane, int h, int j, float (&v)[C]) const {
        load(plane, off[h][j], inside(h, j), v);
    }
    // the thread's rows of a plane as pairs
    __device__ __forceinline__ void load(const float *plane, f2 (&v)[N][C]) const {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            float a[2][C];
            load(plane, 0, j, a[0]);
            load(plane, 1, j, a[1]);
#pragma unroll
            for (int c = 0; c < C; ++c) v[j][c] = mk2(a[0][c], a[1][c]);
        }
    }
    // its upper and lower N rows of a plane, where `top`, `bottom` say that
    // the window owns them
    __device__ __forceinline__ void store(float *plane, const f2 (&v)[N][C], bool top,
                                          bool bottom) const {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (!(h ? bottom : top)) continue;
#pragma unroll
            for (int j = 0; j < N; ++j) {
                if (!inside(h, j)) break;
                float *q = reinterpret_cast<float *>(reinterpret_cast<char *>(plane + base) +
                                                     off[h][j]);
                float a[C];
#pragma unroll
                for (int c = 0; c < C; ++c) a[c] = h ? hi(v[j][c]) : lo(v[j][c]);
                if (SCALAR) {
#pragma unroll
                    for (int c = 0; c < C; ++c)
                        if (c < cols) q[c] = a[c];
                } else {
                    *reinterpret_cast<float2 *>(q) = make_float2(a[0], a[1]);
                }
            }
        }
    }
};

// One row of the input f of a frame (its stack at fb): the stored values, or
// with the projection applied as it is loaded -- PROJ 1, 3: a packed binary
// mask (proj_px); PROJ 4: a float mask; PROJ 5: the spectral projection; PROJ 2: the unrolled solver's v = x + lam (q phi_b), with a
// float mask per frame of a scene, the map q per scene and lam in device
// memory.
template <int PROJ, int C, int N, int MODE, typename Args>
__device__ __forceinline__ void load_f(const Args &P, const Cells<C, N, MODE> &X,
                                       const float *fb, int frame,
                                       typename Cells<C, N, MODE>::Off o, bool in,
                                       float (&v)[C], int row = 0, int col = 0) {
    X.load(fb, o, in, v);
    if constexpr (PROJ == 1 || PROJ == 3) {
        float cm[C], wb[C];
        X.load(P.cmap, o, in, cm);
        X.load(reinterpret_cast<const float *>(P.bits), o, in, wb);
#pragma unroll
        for (int c = 0; c < C; ++c)
            v[c] = proj_px(P.lam, cm[c], v[c], __float_as_uint(wb[c]), 1u << frame);
    } else if constexpr (PROJ == 5) {
        // one aperture for all bands, the map on the detector: band b's columns
        // lie B b to the right in rows of frame0 columns (scalars: any step)
        const float *q = P.cmap + (int64_t)(MODE == INSIDE ? row : min(row, P.H - 1)) * P.frame0 +
                         P.B * frame;
        float m[C];
        X.load(P.phi, o, in, m);
#pragma unroll
        for (int c = 0; c < C; ++c)
            v[c] = fmaf(P.lam, q[MODE == INSIDE ? col + c : min(col + c, P.W - 1)] * m[c], v[c]);
    } else if constexpr (PROJ == 4) {
        float q[C], m[C];
        X.load(P.cmap, o, in, q);
        X.load(P.phi + (int64_t)frame * P.H * P.W, o, in, m);
#pragma unroll
        for (int c = 0; c < C; ++c) v[c] = fmaf(P.lam, q[c] * m[c], v[c]);
    } else if constexpr (PROJ == 2) {
        const int64_t hw = (int64_t)P.H * P.W;
        const int g = P.frame0 + frame, n = g / P.B;
        float q[C], m[C];
        X.load(P.cmap + n * hw, o, in, q);
        X.load(P.phi + (g - n * P.B) * hw, o, in, m);
        const float lam = *P.lam_dev;
#pragma unroll
        for (int c = 0; c < C; ++c) v[c] = fmaf(lam, q[c] * m[c], v[c]);
    }
}

__device__ __forceinline__ f2 shfl_dn(f2 v) {
    f2 r;
    r.v = __shfl_down_sync(FULL, v.v, 1);
    return r;
}
__device__ __forceinline__ f2 shfl_up(f2 v) {
    f2 r;
    r.v = __shfl_up_sync(FULL, v.v, 1);
    return r;
}

// One row of C columns per lane and warp, for the rows that cross warps.
template <int C, int NW>
struct Exchange {
    float v[NW][32 * C];
    __device__ __forceinline__ void put(int w, int lane, const float (&x)[C]) {
        float *p = &v[w][lane * C];
        *reinterpret_cast<float2 *>(p) = make_float2(x[0], x[1]);
    }
    __device__ __forceinline__ void get(int w, int lane, float (&x)[C]) const {
        const float *p = &v[w][lane * C];
        const float2 t = *reinterpret_cast<const float2 *>(p);
        x[0] = t.x, x[1] = t.y;
    }
};

template <int C, int NW>
struct Smem {
    Exchange<C, NW> u, p;       // first row of u, last row of p of each warp
    float energy[SMAX][NW];
};

// The window of one block: nup dual updates (nup <= SMAX) of tile (tr, tc)
// of `frame`.  PIN: start from p_a (P.p_in).  OUT_U: write u (and resid,
// with PROJ 3 t = u + (u - f)), else p (P.p_out).  ENERGY: add the pass's
// energy sums.  TAPE: also write every p_k (as 4 p) and, for k < nup, u_k
// (P.tape_p, P.tape_u).  EDGE: the window reaches
// the frame's last row or column.
template <int C, int N, int NW, bool PIN, bool OUT_U, bool ENERGY, int PROJ, bool TAPE, int MODE>
__device__ __forceinline__ void run(const Pass &P, int frame, int tr, int tc, int nup,
                                    Smem<C, NW> &sm) {
    using G = Geo<C, N, NW>;
    constexpr bool EDGE = MODE != INSIDE;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int H = P.H, W = P.W;
    int c0, own_c0, own_c1, t0, own_r0, own_r1;
    window(W, G::COLS, tc, P.nbands, c0, own_c0, own_c1);
    window(H, G::ROWS, tr, P.nchunks, t0, own_r0, own_r1);
    const int col = c0 + C * lane, row = t0 + 2 * N * w;  // this thread's first
    const int64_t hw = (int64_t)H * W;
    const float *fb = P.f + (int64_t)frame * P.fs;
    // halves of a thread's rows are owned or not, up to the frame's last row
    static_assert(HALO % N == 0 && HALO % C == 0, "window edges split no half and no lane");
    const bool cols = col >= own_c0 && col < own_c1;
    const bool top = cols && row >= own_r0 && row < own_r1;
    const bool bottom = cols && row + N >= own_r0 && row + N < own_r1;
    const Cells<C, N, MODE> X(t0, row, col, H, W);
    auto store = [&](float *plane, const f2 (&v)[N][C]) { X.store(plane, v, top, bottom); };

    // A warp below the frame only keeps the barriers; the warp above reads
    // zeros from it.
    if (EDGE && row >= H) {
        const float zero[C] = {};
        sm.u.put(w, lane, zero);
        for (int k = 1; k <= nup; ++k) {
            __syncthreads();
            if (OUT_U || k < nup) __syncthreads();
        }
        if (ENERGY) {
            if (lane < SMAX) sm.energy[lane][w] = 0.f;
            __syncthreads();
        }
        return;
    }

    f2 f[N][C], u[N][C], pr[N][C], pc[N][C];
    // ---- input rows
#pragma unroll
    for (int j = 0; j < N; ++j) {
        float v[2][C];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            load_f<PROJ>(P, X, fb, frame, X.off[h][j], X.inside(h, j), v[h], row + j + h * N, col);
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
            f[j][c] = mk2(v[0][c], v[1][c]);
            u[j][c] = f[j][c];
            pr[j][c].v = pc[j][c].v = 0ull;
        }
    }

    const f2 one2 = mk2(1.f, 1.f), tw2 = mk2(P.tw, P.tw), q2 = mk2(-0.25f, -0.25f);
    const f2 w2 = mk2(16.f * P.weight, 16.f * P.weight);  // the sums are 16-fold (4 p)
    f2 ek[SMAX];
#pragma unroll
    for (int k = 0; k < SMAX; ++k) ek[k].v = 0ull;

    // u = f - div p / 4 from p, its row above the warp's first in `above` and
    // the column left of lane 0's in `left0` (PIN's first; else the window's
    // halo or the frame's edge, 0); adds the sum of (div p)^2 to e.
    auto divergence = [&](const float (&above)[C], const f2 (&left0)[N], bool sum, f2 &e) {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            f2 left = shfl_up(pc[j][C - 1]);
            if (lane == 0) left = left0[j];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const f2 up = j > 0 ? pr[j > 0 ? j - 1 : 0][c] : mk2(above[c], lo(pr[N - 1][c]));
                const f2 l = c > 0 ? pc[j][c > 0 ? c - 1 : 0] : left;
                const f2 d = sub2(sub2(add2(pr[j][c], pc[j][c]), up), l);
                u[j][c] = fma2(q2, d, f[j][c]);
                if (ENERGY && sum) e = fma2(d, d, e);
            }
        }
    };

    f2 zero_left[N];
#pragma unroll
    for (int j = 0; j < N; ++j) zero_left[j].v = 0ull;
    if (PIN) {  // p_a and u_a = f - div p_a / 4
        const float *pb = P.p_in + (int64_t)frame * 2 * hw;
        float above[C];
        f2 left0[N];
        X.load(pb, X.at(max(row - 1, 0), col, max(t0 - 1, 0), H, W), true, above);
#pragma unroll
        for (int c = 0; c < C; ++c) above[c] = row > 0 ? above[c] : 0.f;
        const unsigned lo0 = (unsigned)max(c0 - 1, 0);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            float a[2][C], b[2][C], l[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                X.load(pb, h, j, a[h]);
                X.load(pb + hw, h, j, b[h]);
                const int r = row + j + h * N;
                const float t = pb[hw + ((unsigned)min(r, H - 1) * (unsigned)W + lo0)];
                l[h] = c0 > 0 && r < H ? t : 0.f;
            }
#pragma unroll
            for (int c = 0; c < C; ++c) {
                pr[j][c] = mk2(a[0][c], a[1][c]);
                pc[j][c] = mk2(b[0][c], b[1][c]);
            }
            left0[j] = mk2(l[0], l[1]);
        }
        divergence(above, left0, true, ek[0]);
    }

#pragma unroll
    for (int k = 1; k <= SMAX; ++k) {
        if (k > nup) break;
        // ---- p_k from u_{k-1}
        float first[C], below[C];
#pragma unroll
        for (int c = 0; c < C; ++c) first[c] = lo(u[0][c]);
        sm.u.put(w, lane, first);
        __syncthreads();
        // below the window: no gradient (halo, or rows past the frame, whose 0
        // has to stay 0)
#pragma unroll
        for (int c = 0; c < C; ++c) below[c] = hi(u[N - 1][c]);
        if (w + 1 < NW) sm.u.get(w + 1, lane, below);
#pragma unroll
        for (int j = 0; j < N; ++j) {
            f2 uR = shfl_dn(u[j][0]);
            if (EDGE && lane == 31) uR = u[j][C - 1];  // as below the window
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const f2 uc = u[j][c];
                f2 right = c + 1 < C ? u[j][c + 1 < C ? c + 1 : 0] : uR;
                f2 dn = j + 1 < N ? u[j + 1 < N ? j + 1 : 0][c] : mk2(hi(u[0][c]), below[c]);
                if (EDGE) {  // no gradient across the last column / row
                    if (col + c == W - 1) right = uc;
                    dn = mk2(row + j == H - 1 ? lo(uc) : lo(dn),
                             row + N + j == H - 1 ? hi(uc) : hi(dn));
                }
                const f2 gc = sub2(right, uc), gr = sub2(dn, uc);
                const f2 s = fma2(gr, gr, mul2(gc, gc));
                const f2 n = mk2(sqrt_approx(lo(s)), sqrt_approx(hi(s)));
                const f2 den = fma2(tw2, n, one2);
                const f2 ri = mk2(rcp_approx(lo(den)), rcp_approx(hi(den)));
                pr[j][c] = mul2(sub2(pr[j][c], gr), ri);
                pc[j][c] = mul2(sub2(pc[j][c], gc), ri);
                if (ENERGY) ek[k - 1] = fma2(w2, n, ek[k - 1]);
            }
        }
        if (TAPE) {
            float *tp = P.tape_p + ((int64_t)(k - 1) * P.nf + frame) * 2 * hw;
            store(tp, pr);
            store(tp + hw, pc);
        }
        if (!OUT_U && k == nup) break;  // p alone goes on
        // ---- u_k = f - div p_k / 4
        float last[C], above[C];
#pragma unroll
        for (int c = 0; c < C; ++c) last[c] = hi(pr[N - 1][c]);
        sm.p.put(w, lane, last);
        __syncthreads();
#pragma unroll
        for (int c = 0; c < C; ++c) above[c] = 0.f;
        if (w > 0) sm.p.get(w - 1, lane, above);
        divergence(above, zero_left, k < SMAX && k < nup, ek[k < SMAX ? k : 0]);
        if (TAPE && k < nup) store(P.tape_u + ((int64_t)(k - 1) * P.nf + frame) * hw, u);
    }

    // ---- owned rows out
    if (OUT_U) {
        float *ub = P.u + (int64_t)frame * P.fs;
        store(ub, u);
        if (PROJ == 3 || (PROJ == 0 && !TAPE && P.resid)) {
            f2 t[N][C];  // u - f, or t = u + (u - f)
#pragma unroll
            for (int j = 0; j < N; ++j)
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    t[j][c] = sub2(u[j][c], f[j][c]);
                    if (PROJ == 3) t[j][c] = add2(u[j][c], t[j][c]);
                }
            store((PROJ == 3 ? P.tout : P.resid) + (int64_t)frame * P.fs, t);
        }
    } else if (!TAPE) {
        float *pb = P.p_out + (int64_t)frame * 2 * hw;
        store(pb, pr);
        store(pb + hw, pc);
    }

    if (ENERGY) {
        // a lane's at most 4 N C values and the warp's 32 lanes in float32,
        // warps and blocks in float64
#pragma unroll
        for (int k = 0; k < SMAX; ++k) {
            float v = (top ? lo(ek[k]) : 0.f) + (bottom ? hi(ek[k]) : 0.f);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
            if (lane == 0) sm.energy[k][w] = v;
        }
        __syncthreads();
        if (threadIdx.x < P.S) {
            const int k = threadIdx.x;
            double v = 0.0;
            for (int i = 0; i < NW; ++i) v += (double)sm.energy[k][i];
            atomicAdd(P.energy + ((int64_t)frame * P.K + P.a + k) * 2, 0.0625 * v);
            if (P.ticket) __threadfence();
        }
    }
}

template <int C, int N, int NW, bool PIN, bool OUT_U, bool ENERGY, int PROJ, bool TAPE = false>
__device__ __forceinline__ void run_mode(const Pass &P, int frame, int tr, int tc, int nup,
                                         Smem<C, NW> &sm) {
    // the first windows of an axis need no bounds: they start at 0
    const bool edge = tr == P.nchunks - 1 || tc == P.nbands - 1;
    if (TAPE && P.vec < 0) run<C, N, NW, PIN, OUT_U, ENERGY, PROJ, TAPE, TAPE ? EDGE_WIDE : EDGE_SCALAR>(P, frame, tr, tc, nup, sm);
    else if (!P.vec) run<C, N, NW, PIN, OUT_U, ENERGY, PROJ, TAPE, EDGE_SCALAR>(P, frame, tr, tc, nup, sm);
    else if (edge) run<C, N, NW, PIN, OUT_U, ENERGY, PROJ, TAPE, EDGE_VEC>(P, frame, tr, tc, nup, sm);
    else run<C, N, NW, PIN, OUT_U, ENERGY, PROJ, TAPE, INSIDE>(P, frame, tr, tc, nup, sm);
}

// Block -> (frame, window); the frames of a window are adjacent blocks (they
// share its rows of the residual map and the mask words in L2).
__device__ __forceinline__ void decode(const Pass &P, int &frame, int &tr, int &tc) {
    const unsigned t = blockIdx.x / (unsigned)P.nf;
    frame = (int)(blockIdx.x - t * (unsigned)P.nf);
    tr = (int)(t / (unsigned)P.nbands);
    tc = (int)(t - (unsigned)tr * (unsigned)P.nbands);
}

template <int C, int N, int NW, int MINB, bool PIN, bool OUT_U, int PROJ>
__global__ void __launch_bounds__(NW * 32, MINB) k_tv_tile(Pass P) {
    __shared__ Smem<C, NW> sm;
    grid_dep_wait();
    if (P.early) grid_dep_launch();
    int frame, tr, tc;
    decode(P, frame, tr, tc);
    if (!(PIN && P.done[frame] >= 0))  // not stopped in an earlier pass
        run_mode<C, N, NW, PIN, OUT_U, true, PROJ>(P, frame, tr, tc, P.S, sm);
    if (P.ticket && threadIdx.x < 32) {
        __syncwarp();
        decide_stops(P, threadIdx.x);
    }
}

// A run of P.S updates of v = x + lam (q phi) that writes its tape, and u with
// OUT_U; no stop test.
template <int C, int N, int NW, int MINB, bool OUT_U>
__global__ void __launch_bounds__(NW * 32, MINB) k_tv_tile_tape(Pass P) {
    __shared__ Smem<C, NW> sm;
    grid_dep_wait();
    if (P.early) grid_dep_launch();
    int frame, tr, tc;
    decode(P, frame, tr, tc);
    run_mode<C, N, NW, false, OUT_U, false, 2, true>(P, frame, tr, tc, P.S, sm);
}

// Frames whose rule fired at step j in this pass's window, with j - a updates.
template <int C, int N, int NW, int MINB, bool PIN, int PROJ>
__global__ void __launch_bounds__(NW * 32, MINB) k_tv_tile_fix(Pass P) {
    __shared__ Smem<C, NW> sm;
    grid_dep_wait();
    if (P.early) grid_dep_launch();
    int frame, tr, tc;
    decode(P, frame, tr, tc);
    const int j = P.stopj[frame];
    if (j == -2) return;  // stopped in an earlier window
    const bool lead = tr == 0 && tc == 0 && threadIdx.x == 0;
    if (j < 0) {
        if (lead && P.steps && P.a + P.S == P.K - 1) P.steps[frame] = P.K;
        return;
    }
    if (lead) {
        P.done[frame] = j;
        if (P.steps) P.steps[frame] = j + 1;
    }
    run_mode<C, N, NW, PIN, true, false, PROJ>(P, frame, tr, tc, j - P.a, sm);
}

}  // namespace tile
}  // namespace tv
}  // namespace sci
