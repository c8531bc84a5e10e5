// Differentiable unrolled GAP-TV: forward with outer-iterate checkpoints and
// a hand-written reverse pass.
//
// Model (a batch of N scenes sharing one learnable mask):
//   Phi = sigmoid(logits) (B x H x W), Phi_sum = sum_b Phi_b,
//   y_n = A(x_true_n), x^0 = At(y / Phi_sum),
//   for k < K (GAP with acceleration, pnp_sci_algo.py:641-643):
//     yb = A(x^k); y1 += y - yb; q = (y1 - yb) / Phi_sum;
//     v^k = x^k + lambda_k At(q);   x^{k+1} = TV(v^k)   (fixed T Chambolle
//     steps, no stop test: the stop rule is not differentiable)
//   loss = mean (x^K - x_true)^2.
// The forward keeps x^k and q^k and the reverse pass recomputes each TV
// call's tape (u_k, p_{k+1}) from them, some frames at a time; with
// SCI_UNROLLED_TAPE=1 the forward's TV writes the tapes as it runs and keeps
// them, when they fit (up to 48 GiB), and the reverse pass reads them.  The
// reverse pass runs the adjoint of every TV step:
//   p_{k+1} = (p_k - tau g_k) r_k,  r_k = 1 / (1 + (tau/w) n_k),  n_k = |g_k|,
//   gbar_k = -tau r_k pbar_{k+1} - (tau/w) r_k (g_k / n_k) <pbar_{k+1}, p_{k+1}>
//            (0 for the second term where g_k = 0: the safe-norm convention),
//   ubar_k = -div gbar_k,  fbar += ubar_k,  pbar_k = r_k pbar_{k+1} + grad ubar_k.
// then the adjoint of the projection (including d/dPhi through A, At and
// Phi_sum, and d/dlambda_k), and finally of the measurement and x^0.
#include <algorithm>
#include <cstdlib>
#include <string>

#include "sci_common.cuh"
#include "sci_graph.cuh"
#include "sci_sqerr.cuh"

namespace sci {

int tv_launch_flags(const float *f, float *u, float *resid, int64_t nf, int64_t H, int64_t W,
                    int64_t fs, float weight, float eps, int K, int *steps, double *energy_out,
                    void *workspace, size_t ws_bytes, cudaStream_t s, int force_R, int flags);
int tv_tape(const float *x, const float *q, const float *phi, const float *lam, int64_t frame0,
            int64_t nf, int64_t B, int64_t H, int64_t W, float weight, int U, float *u,
            float *tape_p, float *tape_u, cudaStream_t s);
int tv_adjoint(const float *x, const float *q, const float *phi, const float *lam, int64_t frame0,
               int64_t nf, int64_t B, int64_t H, int64_t W, float weight, int U,
               const float *tape_p, const float *tape_u, const float *xbar, float *fbar,
               cudaStream_t s);
size_t tv_workspace_bytes(int64_t nf, int64_t H, int64_t W, int K);

namespace unr {

constexpr int kNoStop = 1;  // tv_launch_flags: run all steps, no stop test

inline dim3 grid1(int64_t n, int t) {
    int64_t b = (n + t - 1) / t;
    if (b > (int64_t)kSMs * 16) b = (int64_t)kSMs * 16;
    return dim3((unsigned)(b < 1 ? 1 : b));
}

#define GRID_LOOP(i, n)                                                          \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n);    \
         i += (int64_t)gridDim.x * blockDim.x)

// ------------------------------------------------------------- forward
__global__ void k_mask(const float *__restrict__ logits, float *__restrict__ phi,
                       float *__restrict__ ps, int B, int64_t hw) {
    GRID_LOOP(p, hw) {
        float s = 0.f;
        for (int b = 0; b < B; ++b) {
            const float m = 1.f / (1.f + expf(-logits[b * hw + p]));
            phi[b * hw + p] = m;
            s += m;
        }
        ps[p] = s;
    }
}

// y_n = A(x_true_n); x^0_n = At(y_n / Phi_sum)
__global__ void k_meas_x0(const float *__restrict__ xt, const float *__restrict__ phi,
                          const float *__restrict__ ps, float *__restrict__ y,
                          float *__restrict__ x0, int N, int B, int64_t hw) {
    GRID_LOOP(i, (int64_t)N * hw) {
        const int n = (int)(i / hw);
        const int64_t p = i - (int64_t)n * hw;
        const float *xn = xt + (int64_t)n * B * hw;
        float s = 0.f;
        for (int b = 0; b < B; ++b) s = fmaf(xn[b * hw + p], phi[b * hw + p], s);
        y[i] = s;
        const float s0 = s / ps[p];
        float *x0n = x0 + (int64_t)n * B * hw;
        for (int b = 0; b < B; ++b) x0n[b * hw + p] = phi[b * hw + p] * s0;
    }
}

// V pixels of a map, V = 4 with 16-byte loads (hw % 4 == 0, aligned) or 1.
template <int V>
__device__ __forceinline__ void ldv(const float *p, float (&v)[V]) {
    if constexpr (V == 4) {
        const float4 t = *reinterpret_cast<const float4 *>(p);
        v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
    } else {
        v[0] = *p;
    }
}
template <int V>
__device__ __forceinline__ void stv(float *p, const float (&v)[V]) {
    if constexpr (V == 4) *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else *p = v[0];
}

// yb = A(x); y1 += y - yb (from 0 at the first iteration); q = (y1 - yb) /
// Phi_sum; v = x + lambda (phi q) when v is given
template <int V>
__global__ void __launch_bounds__(256) k_proj_fwd(
    const float *__restrict__ x, const float *__restrict__ phi, const float *__restrict__ ps,
    const float *__restrict__ y, float *__restrict__ y1, float *__restrict__ q,
    float *__restrict__ v, const float *__restrict__ lambdas, int k, int N, int B, int64_t hw) {
    const float lam = lambdas[k];
    GRID_LOOP(g, (int64_t)N * hw / V) {
        const int64_t i = g * V;
        const int n = (int)(i / hw);
        const int64_t p = i - (int64_t)n * hw;
        const float *xn = x + (int64_t)n * B * hw + p;
        float yb[V], t[V], a[V], m[V], r[V];
#pragma unroll
        for (int e = 0; e < V; ++e) yb[e] = t[e] = 0.f;
#pragma unroll 8
        for (int b = 0; b < B; ++b) {
            ldv<V>(xn + b * hw, a);
            ldv<V>(phi + b * hw + p, m);
#pragma unroll
            for (int e = 0; e < V; ++e) yb[e] = fmaf(a[e], m[e], yb[e]);
        }
        if (k) ldv<V>(y1 + i, t);
        ldv<V>(y + i, a);
        ldv<V>(ps + p, m);
#pragma unroll
        for (int e = 0; e < V; ++e) {
            t[e] = t[e] + (a[e] - yb[e]);
            r[e] = (t[e] - yb[e]) / m[e];
        }
        stv<V>(y1 + i, t);
        stv<V>(q + i, r);
        if (!v) continue;
        float *vn = v + (int64_t)n * B * hw + p;
#pragma unroll 8
        for (int b = 0; b < B; ++b) {
            ldv<V>(xn + b * hw, a);
            ldv<V>(phi + b * hw + p, m);
#pragma unroll
            for (int e = 0; e < V; ++e) a[e] = fmaf(lam, r[e] * m[e], a[e]);
            stv<V>(vn + b * hw, a);
        }
    }
}

// *out += sum (a - b)^2, or grad = gscale (a - b).  n4: groups of four with
// 16-byte loads (0 where a pointer is not on such a boundary).  The squares in
// float64 and scalar loads took 40 us at 16 x 256 x 256 x 8 (67 MB read).
template <bool GRAD>
__global__ void __launch_bounds__(256) k_mse(const float *__restrict__ a,
                                             const float *__restrict__ b,
                                             float *__restrict__ grad, float gscale, int64_t n,
                                             int64_t n4, double *out) {
    double acc = 0.0;
    SquareSum se;
    se.clear();
    int held = 0;
    GRID_LOOP(q, n4) {
        const float4 x = ldg4(a + 4 * q), y = ldg4(b + 4 * q);
        if (GRAD) {
            st4(grad + 4 * q, make_float4(gscale * (x.x - y.x), gscale * (x.y - y.y),
                                          gscale * (x.z - y.z), gscale * (x.w - y.w)));
        } else {
            se.add4(x, y);
            if (++held == SquareSum::kMost) {
                acc += se.take();
                held = 0;
            }
        }
    }
    GRID_LOOP(r, n - 4 * n4) {
        const int64_t i = 4 * n4 + r;
        const float d = a[i] - b[i];
        if (GRAD) grad[i] = gscale * d;
        else acc += (double)d * d;
    }
    if (!GRAD) rn_flush(acc + se.take(), out);
}

// --------------------------------------------------- projection adjoint
// Accumulates dPhi, dPhi_sum and d lambda_k, carries dy1 and dy, and writes
// xbar^k, from vbar^k and the projection's q = (y1 - A x) / Phi_sum.  A block
// is 32 groups of V pixels by IL item lanes; lane l takes items l, l + IL, ...
// (TI of them at a time, their per-item scalars in registers).  Sums over
// items are reduced over the lanes in shared memory in a fixed order, FB
// frames per barrier, so the result does not depend on scheduling.  Bound by
// the stacks it moves (vbar and x read, xbar written); with q recomputed (x
// read twice), one pixel per thread and no loads in flight beside the current
// frame's it took 84 us at 16 x 256 x 256 x 8 against 29.
constexpr int IL = 8, FB = 8;

template <int V, int TI>
__global__ void __launch_bounds__(32 * IL) k_proj_bwd(
    const float *__restrict__ vb, const float *__restrict__ x, const float *__restrict__ phi,
    const float *__restrict__ ps, const float *__restrict__ q, const float *__restrict__ lambdas,
    int k, float *__restrict__ y1c, float *__restrict__ ybar, float *__restrict__ phib,
    float *__restrict__ psb, double *__restrict__ lamb, float *__restrict__ xb, int N, int B,
    int64_t hw) {
    __shared__ __align__(16) float red[FB][IL][32 * V];
    __shared__ double lred[IL];
    const int64_t p = ((int64_t)blockIdx.x * 32 + threadIdx.x) * V;
    const bool in = p < hw;
    const float lam = lambdas[k];
    float s[V], psacc[V];
#pragma unroll
    for (int e = 0; e < V; ++e) s[e] = 1.f, psacc[e] = 0.f;
    if (in) ldv<V>(ps + p, s);
    double lacc = 0.0;
    for (int n0 = 0; n0 < N; n0 += TI * IL) {
        float ql[TI][V], yl[TI][V];  // q * lambda and dL/dyb per item of this lane
#pragma unroll
        for (int t = 0; t < TI; ++t) {
            const int n = n0 + threadIdx.y + t * IL;
#pragma unroll
            for (int e = 0; e < V; ++e) ql[t][e] = yl[t][e] = 0.f;
            if (!in || n >= N) continue;
            const float *vn = vb + (int64_t)n * B * hw + p;
            float pv[V], a[V], m[V], y1t[V], yb[V];
#pragma unroll
            for (int e = 0; e < V; ++e) pv[e] = 0.f;
#pragma unroll 8
            for (int b = 0; b < B; ++b) {
                ldv<V>(vn + b * hw, a);
                ldv<V>(phi + b * hw + p, m);
#pragma unroll
                for (int e = 0; e < V; ++e) pv[e] = fmaf(a[e], m[e], pv[e]);
            }
            const int64_t i = (int64_t)n * hw + p;
            ldv<V>(q + i, a);
            ldv<V>(y1c + i, y1t);
            ldv<V>(ybar + i, yb);
#pragma unroll
            for (int e = 0; e < V; ++e) {
                lacc += (double)pv[e] * a[e];
                const float qb = lam * pv[e];
                y1t[e] += qb / s[e];
                psacc[e] -= qb * a[e] / s[e];
                yl[t][e] = -qb / s[e] - y1t[e];
                ql[t][e] = a[e] * lam;
                yb[e] += y1t[e];
            }
            stv<V>(ybar + i, yb);
            stv<V>(y1c + i, y1t);
        }
        // per frame: x bar of every item, and this lane's part of dPhi_b
        for (int b0 = 0; b0 < B; b0 += FB) {
            const int nb = min(FB, B - b0);
#pragma unroll 4
            for (int f = 0; f < nb; ++f) {
                const int b = b0 + f;
                float part[V], m[V];
#pragma unroll
                for (int e = 0; e < V; ++e) part[e] = 0.f, m[e] = 0.f;
                if (in) ldv<V>(phi + b * hw + p, m);
#pragma unroll
                for (int t = 0; t < TI; ++t) {
                    const int n = n0 + threadIdx.y + t * IL;
                    if (!in || n >= N) continue;
                    const int64_t o = ((int64_t)n * B + b) * hw + p;
                    float v[V], xv[V], r[V];
                    ldv<V>(vb + o, v);
                    ldv<V>(x + o, xv);
#pragma unroll
                    for (int e = 0; e < V; ++e) {
                        r[e] = fmaf(m[e], yl[t][e], v[e]);
                        part[e] += fmaf(ql[t][e], v[e], xv[e] * yl[t][e]);
                    }
                    stv<V>(xb + o, r);
                }
                stv<V>(&red[f][threadIdx.y][threadIdx.x * V], part);
            }
            __syncthreads();
            if (in && threadIdx.y < nb) {
                const int b = b0 + threadIdx.y;
                float tot[V], a[V];
#pragma unroll
                for (int e = 0; e < V; ++e) tot[e] = 0.f;
#pragma unroll
                for (int l = 0; l < IL; ++l) {
                    ldv<V>(&red[threadIdx.y][l][threadIdx.x * V], a);
#pragma unroll
                    for (int e = 0; e < V; ++e) tot[e] += a[e];
                }
                ldv<V>(phib + b * hw + p, a);
#pragma unroll
                for (int e = 0; e < V; ++e) a[e] += tot[e];
                stv<V>(phib + b * hw + p, a);
            }
            __syncthreads();
        }
    }
    stv<V>(&red[0][threadIdx.y][threadIdx.x * V], psacc);
    for (int o = 16; o > 0; o >>= 1) lacc += __shfl_xor_sync(0xffffffffu, lacc, o);
    if (threadIdx.x == 0) lred[threadIdx.y] = lacc;
    __syncthreads();
    if (in && threadIdx.y == 0) {
        float tot[V], a[V];
        ldv<V>(psb + p, tot);
#pragma unroll
        for (int e = 0; e < V; ++e) psacc[e] = 0.f;
#pragma unroll
        for (int l = 0; l < IL; ++l) {
            ldv<V>(&red[0][l][threadIdx.x * V], a);
#pragma unroll
            for (int e = 0; e < V; ++e) psacc[e] += a[e];
        }
#pragma unroll
        for (int e = 0; e < V; ++e) tot[e] += psacc[e];
        stv<V>(psb + p, tot);
    }
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        double tot = 0.0;
        for (int l = 0; l < IL; ++l) tot += lred[l];
        atomicAdd(lamb + k, tot);
    }
}

template <int V, typename... A>
void launch_proj_bwd(int64_t hw, int N, cudaStream_t s, A... a) {
    const dim3 g((unsigned)((hw / V + 31) / 32)), b(32, IL);
    if (N <= IL) k_proj_bwd<V, 1><<<g, b, 0, s>>>(a...);
    else if (N <= 2 * IL) k_proj_bwd<V, 2><<<g, b, 0, s>>>(a...);
    else k_proj_bwd<V, 4><<<g, b, 0, s>>>(a...);
}

// Adjoint of x^0 = At(y / Phi_sum), y = A(x_true), Phi_sum = sum Phi_b and
// Phi = sigmoid(logits), in two passes: by item the adjoint of y (in place of
// ybar) and of Phi_sum (t), by frame dPhi and with it dlogits.  As one pass
// with a thread per pixel over items and frames, dPhi added up in memory, it
// took 81 us at 16 x 256 x 256 x 8.
template <int V>
__global__ void __launch_bounds__(256) k_init_bwd_y(
    const float *__restrict__ x0b, const float *__restrict__ phi, const float *__restrict__ ps,
    const float *__restrict__ y, float *__restrict__ ybar, float *__restrict__ t, int N, int B,
    int64_t hw) {
    GRID_LOOP(g, (int64_t)N * hw / V) {
        const int64_t i = g * V;
        const int n = (int)(i / hw);
        const int64_t p = i - (int64_t)n * hw;
        const float *xn = x0b + (int64_t)n * B * hw + p;
        float s0b[V], a[V], m[V], s[V], yb[V];
#pragma unroll
        for (int e = 0; e < V; ++e) s0b[e] = 0.f;
#pragma unroll 8
        for (int b = 0; b < B; ++b) {
            ldv<V>(xn + b * hw, a);
            ldv<V>(phi + b * hw + p, m);
#pragma unroll
            for (int e = 0; e < V; ++e) s0b[e] = fmaf(m[e], a[e], s0b[e]);
        }
        ldv<V>(ps + p, s);
        ldv<V>(y + i, a);
        ldv<V>(ybar + i, yb);
#pragma unroll
        for (int e = 0; e < V; ++e) {
            const float s0 = a[e] / s[e];
            yb[e] = yb[e] + s0b[e] / s[e];
            m[e] = s0b[e] * s0 / s[e];
        }
        stv<V>(ybar + i, yb);
        stv<V>(t + i, m);
    }
}

template <int V>
__global__ void __launch_bounds__(256) k_init_bwd_phi(
    const float *__restrict__ x0b, const float *__restrict__ xt, const float *__restrict__ phi,
    const float *__restrict__ ps, const float *__restrict__ y, const float *__restrict__ ybar,
    const float *__restrict__ t, const float *__restrict__ phib, const float *__restrict__ psb,
    float *__restrict__ glog, int N, int B, int64_t hw) {
    GRID_LOOP(g, (int64_t)B * hw / V) {
        const int64_t i = g * V;
        const int b = (int)(i / hw);
        const int64_t p = i - (int64_t)b * hw;
        float s[V], acc[V], sum[V];
        ldv<V>(ps + p, s);
        ldv<V>(psb + p, sum);
        ldv<V>(phib + i, acc);
#pragma unroll 4
        for (int n = 0; n < N; ++n) {
            float yn[V], yt[V], tn[V], xb[V], x[V];
            ldv<V>(y + n * hw + p, yn);
            ldv<V>(ybar + n * hw + p, yt);
            ldv<V>(t + n * hw + p, tn);
            ldv<V>(x0b + ((int64_t)n * B + b) * hw + p, xb);
            ldv<V>(xt + ((int64_t)n * B + b) * hw + p, x);
#pragma unroll
            for (int e = 0; e < V; ++e) {
                sum[e] -= tn[e];
                acc[e] += fmaf(yn[e] / s[e], xb[e], x[e] * yt[e]);
            }
        }
        float m[V];
        ldv<V>(phi + i, m);
#pragma unroll
        for (int e = 0; e < V; ++e) m[e] = (acc[e] + sum[e]) * m[e] * (1.f - m[e]);
        stv<V>(glog + i, m);
    }
}

struct Ws {
    float *phi, *ps, *y, *X, *Q, *y1, *V;      // forward; Q: q^k of every iteration
    // tape of `frames` frames of one iteration: u_1..u_{U-1}, 4 p_1..4 p_U;
    // stored (when they fit): of every frame and iteration, kept by the forward
    bool stored;
    int64_t frames;
    float *tu, *tp;                            // [frames (U-1) hw], [frames 2 U hw] (x K stored)
    float *fb, *xb, *y1c, *ybar, *phib, *psb;  // reverse
    double *loss;
    void *tv;
    size_t tv_bytes;
};

// Whether the forward keeps the TV tape of every outer iteration (3 (T-1) - 1
// planes per iteration) for the reverse pass.  By default it keeps
// only the outer iterates and the reverse pass recomputes each inner TV
// loop (the checkpoint-only form); SCI_UNROLLED_TAPE=1 stores the tapes
// instead when they fit in 48 GiB.
bool stored_tape(int64_t N, int64_t B, int64_t H, int64_t W, int K, int T) {
    const char *e = getenv("SCI_UNROLLED_TAPE");
    if (!(e && e[0] == '1')) return false;
    const double bytes = 4.0 * (double)(N * B * H * W) * 3.0 * (T - 1) * K;
    return bytes <= 48.0 * (1ull << 30);
}

// Frames whose tape the reverse pass recomputes and consumes at a time: the
// tape stays in L2 (it is overwritten there by the next frames' and never
// needed in HBM) as long as it is small against the 129 MB, and a launch
// should fill the GPU.  Measured at one shape, 16 x 256 x 256 x 8 (2.9 MB of
// tape a frame), forward and reverse pass: 16 frames at a time, fewest of those
// tried, 6.91 ms, 24 6.95, 32 7.01, 48 7.14, 64 7.17, all 128 7.45.
int64_t tape_frames(int64_t nf, int64_t hw, int U) {
    const int64_t frame = 4 * hw * (3 * U - 1);
    const int64_t l2 = (40 << 20) / frame, fill = (1 << 20) / hw;
    return std::max<int64_t>(1, std::min(nf, std::max(l2, fill)));
}

size_t layout(int64_t N, int64_t B, int64_t H, int64_t W, int K, int T, Ws *w, char *base) {
    const size_t hw = (size_t)(H * W), nbhw = (size_t)(N * B) * hw, nhw = (size_t)N * hw;
    const int U = T - 1;
    const bool st = stored_tape(N, B, H, W, K, T);
    const size_t frames = st ? (size_t)(N * B) : (size_t)tape_frames(N * B, H * W, U);
    const size_t kept = st ? (size_t)K : 1;
    size_t off = 0;
    auto take = [&](size_t floats) {
        size_t o = off;
        off += (floats * 4 + 255) & ~size_t(255);
        return o;
    };
    const size_t o_phi = take(B * hw), o_ps = take(hw), o_y = take(nhw);
    const size_t o_X = take((K + 1) * nbhw), o_Q = take((size_t)K * nhw), o_y1 = take(nhw);
    const size_t o_V = take(st ? 1 : nbhw);
    const size_t o_tu = take(kept * (U > 1 ? U - 1 : 1) * frames * hw);
    const size_t o_tp = take(kept * U * 2 * frames * hw);
    const size_t o_fb = take(nbhw), o_xb = take(nbhw), o_y1c = take(nhw), o_ybar = take(nhw);
    const size_t o_phib = take(B * hw), o_psb = take(hw), o_loss = take(4);
    const size_t tvb = tv_workspace_bytes(N * B, H, W, T);
    const size_t o_tv = off;
    off += (tvb + 255) & ~size_t(255);
    if (w) {
        auto F = [&](size_t o) { return reinterpret_cast<float *>(base + o); };
        w->phi = F(o_phi); w->ps = F(o_ps); w->y = F(o_y); w->X = F(o_X); w->Q = F(o_Q);
        w->y1 = F(o_y1); w->V = F(o_V); w->tu = F(o_tu); w->tp = F(o_tp);
        w->fb = F(o_fb); w->xb = F(o_xb); w->y1c = F(o_y1c);
        w->ybar = F(o_ybar); w->phib = F(o_phib); w->psb = F(o_psb);
        w->loss = reinterpret_cast<double *>(base + o_loss);
        w->stored = st;
        w->frames = (int64_t)frames;
        w->tv = base + o_tv;
        w->tv_bytes = tvb;
    }
    return off;
}

int check(int64_t N, int64_t B, int64_t H, int64_t W, int K, int T, float weight) {
    SCI_CHECK_ARG(N >= 1 && B >= 1 && H >= 1 && W >= 1 && K >= 1, "unrolled: invalid sizes");
    SCI_CHECK_ARG(N * B <= 65535 && H <= (1 << 19), "unrolled: N * B <= 65535 frames");
    SCI_CHECK_ARG(T >= 2 && T <= 5, "unrolled: tv_iters must be in [2, 5] (got %d)", T);
    SCI_CHECK_ARG(weight > 0.f, "unrolled: tv_weight must be > 0");
    return SCI_OK;
}

// forward: fills the checkpoints; loss (device double) = mean sq. error
int forward(const float *logits, const float *lambdas, const float *xt, int64_t N, int64_t B,
            int64_t H, int64_t W, int K, int T, float weight, Ws &w, cudaStream_t s) {
    const int64_t hw = H * W, nbhw = N * B * hw;
    const dim3 g = grid1(N * hw, 256);
    k_mask<<<grid1(hw, 256), 256, 0, s>>>(logits, w.phi, w.ps, (int)B, hw);
    k_meas_x0<<<g, 256, 0, s>>>(xt, w.phi, w.ps, w.y, w.X, (int)N, (int)B, hw);
    SCI_LAUNCHED("k_meas_x0");
    const int U = T - 1;
    const bool v4 = hw % 4 == 0 && aligned16(w.phi);
    for (int k = 0; k < K; ++k) {
        const float *Xk = w.X + k * nbhw;
        float *Xn = w.X + (k + 1) * nbhw, *q = w.Q + k * N * hw;
        if (v4)
            k_proj_fwd<4><<<grid1(N * hw / 4, 256), 256, 0, s>>>(
                Xk, w.phi, w.ps, w.y, w.y1, q, w.stored ? nullptr : w.V, lambdas, k, (int)N,
                (int)B, hw);
        else
            k_proj_fwd<1><<<g, 256, 0, s>>>(Xk, w.phi, w.ps, w.y, w.y1, q,
                                            w.stored ? nullptr : w.V, lambdas, k, (int)N, (int)B,
                                            hw);
        SCI_LAUNCHED("k_proj_fwd");
        int e = w.stored ? tv_tape(Xk, q, w.phi, lambdas + k, 0, N * B, B, H, W, weight, U, Xn,
                                   w.tp + (int64_t)k * U * 2 * nbhw,
                                   w.tu + (int64_t)k * (U > 1 ? U - 1 : 1) * nbhw, s)
                         : tv_launch_flags(w.V, Xn, nullptr, N * B, H, W, hw, weight, 0.f, T,
                                           nullptr, nullptr, w.tv, w.tv_bytes, s, 0, kNoStop);
        if (e) return e;
    }
    SCI_CUDA(cudaMemsetAsync(w.loss, 0, sizeof(double), s));
    const float *XK = w.X + K * nbhw;
    const int64_t n4 = aligned16(XK) && aligned16(xt) ? nbhw / 4 : 0;
    k_mse<false><<<std::min(4u * kSMs, grid1(n4 ? n4 : nbhw, 256).x), 256, 0, s>>>(
        XK, xt, nullptr, 0.f, nbhw, n4, w.loss);
    SCI_LAUNCHED("k_mse");
    return SCI_OK;
}

// Whole forward / reverse passes run as cached CUDA graphs (sci_graph.cuh),
// keyed by every argument: the reverse pass is ~20 launches per outer
// iteration.
template <typename... T>
std::string make_key(const T &...v) {
    std::string k;
    (k.append(reinterpret_cast<const char *>(&v), sizeof(T)), ...);
    return k;
}

}  // namespace unr
}  // namespace sci

using namespace sci;
using namespace sci::unr;

extern "C" {

int sci_unrolled_workspace_bytes(int64_t N, int64_t B, int64_t H, int64_t W, int K, int tv_iters,
                                 size_t *bytes) {
    SCI_CHECK_ARG(bytes, "null bytes");
    if (int e = check(N, B, H, W, K, tv_iters, 1.f)) return e;
    *bytes = layout(N, B, H, W, K, tv_iters, nullptr, nullptr);
    return SCI_OK;
}

int sci_unrolled_fwd(const float *logits, const float *lambdas, const float *x_true, int64_t N,
                     int64_t B, int64_t H, int64_t W, int K, int tv_iters, float tv_weight,
                     double *loss, float *x_out, void *workspace, size_t workspace_bytes,
                     void *stream) {
    if (int e = check(N, B, H, W, K, tv_iters, tv_weight)) return e;
    SCI_CHECK_ARG(logits && lambdas && x_true, "sci_unrolled_fwd: null pointer");
    const size_t need = layout(N, B, H, W, K, tv_iters, nullptr, nullptr);
    SCI_CHECK_ARG(workspace && workspace_bytes >= need,
                  "sci_unrolled_fwd: workspace of %zu bytes needed, got %zu", need,
                  workspace_bytes);
    Ws w;
    layout(N, B, H, W, K, tv_iters, &w, static_cast<char *>(workspace));
    const int64_t nbhw = N * B * H * W;
    auto body = [&](cudaStream_t s) -> int {
        if (int e = forward(logits, lambdas, x_true, N, B, H, W, K, tv_iters, tv_weight, w, s))
            return e;
        if (loss)
            SCI_CUDA(cudaMemcpyAsync(loss, w.loss, sizeof(double), cudaMemcpyDeviceToDevice, s));
        if (x_out)
            SCI_CUDA(cudaMemcpyAsync(x_out, w.X + (int64_t)K * nbhw, 4 * nbhw,
                                     cudaMemcpyDeviceToDevice, s));
        return SCI_OK;
    };
    const std::string key = make_key(1, logits, lambdas, x_true, N, B, H, W, K, tv_iters,
                                     tv_weight, loss, x_out, workspace, (int)w.stored);
    return run_graph("unrolled graph capture", key, as_stream(stream), body);
}

int sci_unrolled_bwd(const float *logits, const float *lambdas, const float *x_true, int64_t N,
                     int64_t B, int64_t H, int64_t W, int K, int tv_iters, float tv_weight,
                     float grad_loss, float *grad_logits, double *grad_lambdas,
                     void *workspace, size_t workspace_bytes, void *stream) {
    if (int e = check(N, B, H, W, K, tv_iters, tv_weight)) return e;
    SCI_CHECK_ARG(logits && lambdas && x_true && grad_logits && grad_lambdas,
                  "sci_unrolled_bwd: null pointer");
    const size_t need = layout(N, B, H, W, K, tv_iters, nullptr, nullptr);
    SCI_CHECK_ARG(workspace && workspace_bytes >= need,
                  "sci_unrolled_bwd: workspace of %zu bytes needed, got %zu", need,
                  workspace_bytes);
    Ws w;
    layout(N, B, H, W, K, tv_iters, &w, static_cast<char *>(workspace));
    const std::string key = make_key(2, logits, lambdas, x_true, N, B, H, W, K, tv_iters,
                                     tv_weight, grad_loss, grad_logits, grad_lambdas, workspace,
                                     (int)w.stored);
    return run_graph("unrolled graph capture", key, as_stream(stream), [&](cudaStream_t s) -> int {
    // The checkpoints of the preceding sci_unrolled_fwd call on this
    // workspace (same arguments) are used as they are.
    const int64_t hw = H * W, nbhw = N * B * hw, nhw = N * hw, nf = N * B;
    const int T = tv_iters, U = T - 1;
    // dL/dx^K = grad_loss * 2 (x^K - x_true) / numel
    const float *XK = w.X + (int64_t)K * nbhw;
    const int64_t n4 = aligned16(XK) && aligned16(x_true) && aligned16(w.xb) ? nbhw / 4 : 0;
    k_mse<true><<<grid1(n4 ? n4 : nbhw, 256), 256, 0, s>>>(
        XK, x_true, w.xb, 2.f * grad_loss / (float)nbhw, nbhw, n4, nullptr);
    SCI_LAUNCHED("k_mse");
    SCI_CUDA(cudaMemsetAsync(w.y1c, 0, 4 * nhw, s));
    SCI_CUDA(cudaMemsetAsync(w.ybar, 0, 4 * nhw, s));
    SCI_CUDA(cudaMemsetAsync(w.phib, 0, 4 * B * hw, s));
    SCI_CUDA(cudaMemsetAsync(w.psb, 0, 4 * hw, s));
    SCI_CUDA(cudaMemsetAsync(grad_lambdas, 0, sizeof(double) * K, s));
    const bool v4 = hw % 4 == 0 && aligned16(w.phi);
    for (int k = K - 1; k >= 0; --k) {
        const float *Xk = w.X + k * nbhw, *q = w.Q + k * nhw, *lam = lambdas + k;
        // TV adjoint: fbar = d/dv^k, from the forward's tape or, some frames
        // at a time, from one recomputed from x^k and q^k
        for (int64_t f0 = 0; f0 < nf; f0 += w.frames) {
            const int64_t n = std::min(w.frames, nf - f0), o = f0 * hw;
            float *tp = w.tp, *tu = w.tu;
            if (w.stored) {
                tp += (int64_t)k * U * 2 * nbhw;
                tu += (int64_t)k * (U > 1 ? U - 1 : 1) * nbhw;
            } else if (int e = tv_tape(Xk + o, q, w.phi, lam, f0, n, B, H, W, tv_weight, U,
                                       nullptr, tp, tu, s)) {
                return e;
            }
            if (int e = tv_adjoint(Xk + o, q, w.phi, lam, f0, n, B, H, W, tv_weight, U, tp, tu,
                                   w.xb + o, w.fb + o, s))
                return e;
        }
        // projection adjoint: xbar^k
        if (v4)
            launch_proj_bwd<4>(hw, (int)N, s, w.fb, Xk, w.phi, w.ps, q, lambdas, k, w.y1c, w.ybar,
                               w.phib, w.psb, grad_lambdas, w.xb, (int)N, (int)B, hw);
        else
            launch_proj_bwd<1>(hw, (int)N, s, w.fb, Xk, w.phi, w.ps, q, lambdas, k, w.y1c, w.ybar,
                               w.phib, w.psb, grad_lambdas, w.xb, (int)N, (int)B, hw);
        SCI_LAUNCHED("k_proj_bwd");
    }
    // y1c is the last of the carries that the loop used: scratch from here on
    if (v4 && aligned16(x_true) && aligned16(grad_logits)) {
        k_init_bwd_y<4><<<grid1(nhw / 4, 256), 256, 0, s>>>(w.xb, w.phi, w.ps, w.y, w.ybar, w.y1c,
                                                            (int)N, (int)B, hw);
        k_init_bwd_phi<4><<<grid1(B * hw / 4, 256), 256, 0, s>>>(
            w.xb, x_true, w.phi, w.ps, w.y, w.ybar, w.y1c, w.phib, w.psb, grad_logits, (int)N,
            (int)B, hw);
    } else {
        k_init_bwd_y<1><<<grid1(nhw, 256), 256, 0, s>>>(w.xb, w.phi, w.ps, w.y, w.ybar, w.y1c,
                                                        (int)N, (int)B, hw);
        k_init_bwd_phi<1><<<grid1(B * hw, 256), 256, 0, s>>>(
            w.xb, x_true, w.phi, w.ps, w.y, w.ybar, w.y1c, w.phib, w.psb, grad_logits, (int)N,
            (int)B, hw);
    }
    SCI_LAUNCHED("k_init_bwd");
    return SCI_OK;
    });
}

}  // extern "C"
