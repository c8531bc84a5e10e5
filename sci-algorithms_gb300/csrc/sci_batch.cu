// Batched GAP-TV over many measurements of uneven sizes.
//
// The reference reconstructs coded-frame blocks one after another
// (admmdenoise_cacti's frame-block loop, PnP_SCI/python/pnp_sci_algo.py:498);
// here a batch of independent measurements (each with its own H x W x B and
// packed binary mask) advances together.  Every phase of an iteration is
// one launch spanning all items: the GAP residual maps, then the Chambolle
// TV pass over every item's (frame, row chunk, column band) work items, then
// the stop-test launch over the same work items (sci_batch_lean.cu).  Items
// are found from the task index through prefix tables in a device-resident
// item table.  The whole multi-iteration loop is captured once into a CUDA
// graph and replayed.  An autotuner times row-chunk heights on the batch's
// own data.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "sci_bulk.cuh"
#include "sci_graph.cuh"
#include "sci_batch.cuh"
#include "sci_tv.cuh"

namespace sci {

// bit 0: a bounded bulk-copy wait of the batched projection gave up
__device__ unsigned int g_batch_status;

namespace batch {

// x0 = At(y / Phi_sum) for every item (the start point of the GAP loop).
// Start of a solve, one pass over every item's pixels: X0, x = At(y /
// Phi_sum); Y1, the accelerated GAP's y1 = 0 (one launch instead of a
// memset node per item).
template <bool X0, bool Y1>
__global__ void __launch_bounds__(PROJ_T) k_batch_init(const Table *__restrict__ T) {
    const int g = blockIdx.x;
    if (g >= T->proj_prefix[T->n]) return;
    const int i = find_item(T->proj_prefix, T->n, g);
    const Item &I = T->it[i];
    const int64_t p = (int64_t)(g - T->proj_prefix[i]) * PROJ_T + threadIdx.x;
    if (p >= I.hw) return;
    if (Y1) I.y1[p] = 0.f;
    if (X0) {
        const uint32_t w = I.bits[p];
        const float s0 = I.y[p] / I.phisum[p];
        for (int b = 0; b < I.B; ++b) I.x[b * I.hw + p] = ((w >> b) & 1u) ? s0 : 0.f * s0;
    }
}

// GAP projection (acc: y1 += y - A x, x_p = x + lam At((y1 - A x)/Phi_sum)).
template <bool ACC>
__global__ void __launch_bounds__(PROJ_T) k_batch_proj(const Table *__restrict__ T) {
    __shared__ float xs[32 * PROJ_T];
    const int g = blockIdx.x;
    if (g >= T->proj_prefix[T->n]) return;
    const int i = find_item(T->proj_prefix, T->n, g);
    const Item &I = T->it[i];
    const int t = threadIdx.x;
    const int64_t p = (int64_t)(g - T->proj_prefix[i]) * PROJ_T + t;
    if (p >= I.hw) return;
    const int64_t hw = I.hw;
    const int B = I.B;
    const uint32_t w = __ldg(I.bits + p);
    float s = 0.f;
    for (int b = 0; b < B; ++b) {
        const float v = __ldg(I.x + b * hw + p);
        xs[b * PROJ_T + t] = v;
        s = fmaf(v, ((w >> b) & 1u) ? 1.f : 0.f, s);
    }
    const float yv = __ldg(I.y + p), ps = __ldg(I.phisum + p);
    float r;
    if (ACC) {
        const float tt = I.y1[p] + (yv - s);
        I.y1[p] = tt;
        r = __fdiv_rn(tt - s, ps);
    } else {
        r = __fdiv_rn(yv - s, ps);
    }
    for (int b = 0; b < B; ++b) {
        const float m = ((w >> b) & 1u) ? 1.f : 0.f;
        __stcs(I.xp + b * hw + p, fmaf(I.lam, r * m, xs[b * PROJ_T + t]));
    }
}

// The same projection with the tile's B rows of 256 floats staged by bulk
// copies (one mbarrier, 64 threads x 4 pixels); the default for items whose
// planes are 16-byte aligned with hw % 4 == 0 (all items of a batch, see
// check()).  Same arithmetic, bit-identical results.
template <bool ACC>
__global__ void __launch_bounds__(PROJ_T / 4) k_batch_proj_tma(const Table *__restrict__ T) {
    extern __shared__ __align__(128) float xs[];  // [B][PROJ_T]
    __shared__ __align__(8) uint64_t bar;
    const int g = blockIdx.x;
    if (g >= T->proj_prefix[T->n]) return;
    const int i = find_item(T->proj_prefix, T->n, g);
    const Item &I = T->it[i];
    const int64_t hw = I.hw;
    const int B = I.B;
    const int64_t p0 = (int64_t)(g - T->proj_prefix[i]) * PROJ_T;
    const unsigned n = (unsigned)(hw - p0 < PROJ_T ? hw - p0 : PROJ_T);
    const int tid = threadIdx.x;
    if (tid == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&bar, (unsigned)B * n * 4u);
        for (int b = 0; b < B; ++b) bulk_g2s(xs + b * PROJ_T, I.x + b * hw + p0, n * 4u, &bar);
    }
    __syncthreads();  // the barrier is initialised before anyone waits on it
    const bool ok = mbar_wait(&bar, 0);
    if (__syncthreads_or(!ok)) {
        if (tid == 0) {
            atomicOr(&g_batch_status, 1u);
            mbar_wait(&bar, 0);  // let the copies land before the block ends
        }
        return;
    }
    const int q = tid * 4;
    if ((unsigned)q >= n) return;
    const int64_t p = p0 + q;
    const uint4 w4 = __ldg(reinterpret_cast<const uint4 *>(I.bits + p));
    const uint32_t wv[4] = {w4.x, w4.y, w4.z, w4.w};
    const float4 yv = ldg4(I.y + p), psv = ldg4(I.phisum + p);
    const float yy[4] = {yv.x, yv.y, yv.z, yv.w}, pp[4] = {psv.x, psv.y, psv.z, psv.w};
    float r[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        float sacc = 0.f;
        for (int b = 0; b < B; ++b)
            sacc = fmaf(xs[b * PROJ_T + q + e], ((wv[e] >> b) & 1u) ? 1.f : 0.f, sacc);
        if (ACC) {
            const float tt = I.y1[p + e] + (yy[e] - sacc);
            I.y1[p + e] = tt;
            r[e] = __fdiv_rn(tt - sacc, pp[e]);
        } else {
            r[e] = __fdiv_rn(yy[e] - sacc, pp[e]);
        }
    }
    for (int b = 0; b < B; ++b) {
        const float4 xv = *reinterpret_cast<const float4 *>(xs + b * PROJ_T + q);
        float4 o;
        o.x = fmaf(I.lam, r[0] * (((wv[0] >> b) & 1u) ? 1.f : 0.f), xv.x);
        o.y = fmaf(I.lam, r[1] * (((wv[1] >> b) & 1u) ? 1.f : 0.f), xv.y);
        o.z = fmaf(I.lam, r[2] * (((wv[2] >> b) & 1u) ? 1.f : 0.f), xv.z);
        o.w = fmaf(I.lam, r[3] * (((wv[3] >> b) & 1u) ? 1.f : 0.f), xv.w);
        st4_cs(I.xp + b * hw + p, o);
    }
}

unsigned batch_device_status(bool clear) {
    unsigned v = 0;
    if (cudaMemcpyFromSymbol(&v, g_batch_status, sizeof(v)) != cudaSuccess) return 0;
    if (clear && v) {
        const unsigned z = 0;
        cudaMemcpyToSymbol(g_batch_status, &z, sizeof(z));
    }
    return v;
}

// TV pass (FIX = 0) or its stop-test launch (FIX = 1) over all items' tiles.
template <int FIX>
__global__ void __launch_bounds__(tv::WPB * 32, 3) k_batch_tv(const Table *__restrict__ T) {
    const int g = blockIdx.x * tv::WPB + (threadIdx.x >> 5);
    if (g >= T->tv_prefix[T->n]) return;  // warp-uniform
    const int i = find_item(T->tv_prefix, T->n, g);
    const tv::Pass &P = T->it[i].tv;
    int frame, chunk, band;
    if (!tv::decode_index(P, g - T->tv_prefix[i], frame, chunk, band)) return;
    const int lane = threadIdx.x & 31;
    if (!FIX) {
        switch (P.S) {
            case 1: tv::run_mode<1, 4, false, true, true>(P, frame, chunk, band, lane); break;
            case 2: tv::run_mode<2, 4, false, true, true>(P, frame, chunk, band, lane); break;
            case 3: tv::run_mode<3, 4, false, true, true>(P, frame, chunk, band, lane); break;
            default: tv::run_mode<4, 4, false, true, true>(P, frame, chunk, band, lane); break;
        }
        return;
    }
    const int j = tv::find_stop(P, frame);
    switch (j) {  // a = 0: j in [1, S-1] re-runs with j updates
        case 1: tv::run_mode<1, 4, false, true, false>(P, frame, chunk, band, lane); break;
        case 2: tv::run_mode<2, 4, false, true, false>(P, frame, chunk, band, lane); break;
        case 3: tv::run_mode<3, 4, false, true, false>(P, frame, chunk, band, lane); break;
        default: break;
    }
}

// --------------------------------------------------------------- host side
size_t r256(size_t b) { return (b + 255) & ~size_t(255); }

struct Layout {
    size_t table, xp, y1, energy, stop, total;
    std::vector<size_t> item_xp, item_y1, item_c, item_e, item_e1, item_stop;
};

Layout layout(const sci_batch_item *items, int n, int K) {
    Layout L;
    size_t off = 0;
    L.table = off;
    off += r256(sizeof(Table));
    for (int i = 0; i < n; ++i) {
        const int64_t hw = items[i].H * items[i].W, nn = items[i].B * hw;
        L.item_xp.push_back(off);
        off += r256(4 * (size_t)nn);
        L.item_y1.push_back(off);
        off += r256(4 * (size_t)hw);
        L.item_c.push_back(off);
        off += r256(4 * (size_t)hw);
    }
    // per item the energy sums of even and odd iterations (the generic
    // launches use the first), then its stop decisions and ticket
    L.energy = off;
    for (int i = 0; i < n; ++i) {
        const size_t eb = r256(sizeof(double) * 2 * K * (size_t)items[i].B);
        L.item_e.push_back(off - L.energy);
        L.item_e1.push_back(off + eb - L.energy);
        off += 2 * eb;
    }
    L.stop = off;
    for (int i = 0; i < n; ++i) {
        L.item_stop.push_back(off);
        off += r256(sizeof(int) * (size_t)items[i].B + sizeof(unsigned));
    }
    L.total = off;
    return L;
}

constexpr int kMinR = 8;  // least rows of a chunk
// Workspace that the wait selftest asks for, as it always has (it uses one word).
constexpr size_t kWaitBytes = 3080;

int check(const sci_batch_item *items, int n, int K) {
    SCI_CHECK_ARG(items && n >= 1 && n <= MAXI, "batch: 1..%d items (got %d)", MAXI, n);
    SCI_CHECK_ARG(K >= 2 && K <= tv::SMAX + 1, "batch: tv_iter_max must be in [2, 5]");
    for (int i = 0; i < n; ++i) {
        const sci_batch_item &it = items[i];
        SCI_CHECK_ARG(it.y && it.mask_bits && it.phisum && it.x, "batch: item %d null pointer", i);
        SCI_CHECK_ARG(it.B >= 1 && it.B <= 32 && it.H >= 1 && it.W >= 4 && it.W % 4 == 0,
                      "batch: item %d needs 1 <= B <= 32, W %% 4 == 0 (B=%lld H=%lld W=%lld)", i,
                      (long long)it.B, (long long)it.H, (long long)it.W);
        SCI_CHECK_ARG(it.tv_weight > 0.f, "batch: item %d tv_weight must be > 0", i);
        SCI_CHECK_ARG(((reinterpret_cast<uintptr_t>(it.x) | reinterpret_cast<uintptr_t>(it.y) |
                        reinterpret_cast<uintptr_t>(it.phisum)) & 15u) == 0,
                      "batch: item %d buffers must be 16-byte aligned", i);
    }
    return SCI_OK;
}

// Bands of one frame of the lean pass and the height of the chunks that R
// rows at most make of it.
int lean_bands(const sci_batch_item &s) {
    return tv::band_count((int)s.W, s.cpl == 2 ? 64 : 128, 4, 4);
}
int even_R(int64_t H, int64_t R) {
    const int64_t c = (H + R - 1) / R;
    return (int)std::max<int64_t>(kMinR, (H + c - 1) / c);
}

// The least common chunk height (kMinR or more) at which the batch makes at
// most `waves` times the work items that the GPU holds at a time: a pass
// takes as long as its longest chain of rows, and a last wave that is nearly
// empty as long as a full one.
int waves_R(const sci_batch_item *items, int n, int waves) {
    int64_t lo = kMinR, hi = kMinR;
    for (int i = 0; i < n; ++i) hi = std::max(hi, items[i].H);
    while (lo < hi) {
        const int64_t R = (lo + hi) / 2;
        int64_t c = 0;
        for (int i = 0; i < n; ++i)
            c += items[i].B * lean_bands(items[i]) * ((items[i].H + R - 1) / R);
        if (c <= (int64_t)waves * resident_warps()) hi = R;
        else lo = R + 1;
    }
    return (int)lo;
}

// For items without a chunk height: the fewest waves with chunks of at most
// 96 rows (us per iteration by waves: see sci_batch_autotune).
int default_R(const sci_batch_item *items, int n) {
    int R = 0;
    for (int w = 1; w <= 16; ++w)
        if ((R = waves_R(items, n, w)) <= 96) break;
    return R;
}

// Builds the host copy of the device table.
void build_table(const sci_batch_item *items, int n, int K, float eps, char *ws, const Layout &L,
                 Table &T) {
    memset(&T, 0, sizeof(T));
    T.n = n;
    const int R0 = default_R(items, n);
    T.proj_prefix[0] = T.tv_prefix[0] = T.qp_prefix[0] = T.tq_prefix[0] = 0;
    // longest chunks first: the last wave's are short (16 / 64 items 10.15 /
    // 82.2 ms in the caller's order, 10.05 / 81.5)
    std::vector<int> ord(n);
    for (int i = 0; i < n; ++i) ord[i] = i;
    std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) {
        return (items[a].R > 0 ? items[a].R : even_R(items[a].H, R0)) >
               (items[b].R > 0 ? items[b].R : even_R(items[b].H, R0));
    });
    for (int i = 0; i < n; ++i) {
        const int k = ord[i];  // the item's place in the caller's list
        const sci_batch_item &s = items[k];
        Item &I = T.it[i];
        I.y = s.y;
        I.bits = s.mask_bits;
        I.phisum = s.phisum;
        I.x = s.x;
        I.xp = reinterpret_cast<float *>(ws + L.item_xp[k]);
        I.y1 = reinterpret_cast<float *>(ws + L.item_y1[k]);
        I.c = reinterpret_cast<float *>(ws + L.item_c[k]);
        I.B = (int)s.B;
        I.hw = s.H * s.W;
        I.lam = s.lambda;
        tv::Pass &P = I.tv;
        P.f = I.xp;
        P.u = s.x;
        P.energy = reinterpret_cast<double *>(ws + L.energy + L.item_e[k]);
        P.fs = I.hw;
        P.nf = (int)s.B;
        P.H = (int)s.H;
        P.W = (int)s.W;
        P.K = K;
        P.a = 0;
        P.tau = 0.25f;
        P.tw = 0.25f / s.tv_weight;
        P.weight = s.tv_weight;
        P.eps = eps;
        P.cpl = 4;
        P.S = K - 1;
        P.hl = 4;
        P.hr = 4;
        P.own = 128 - 4 - 4;
        P.ht = K - 1;
        P.nbands = tv::band_count((int)s.W, 128, P.hl, P.hr);
        P.R = s.R > 0 ? s.R : even_R(s.H, R0);
        P.nchunks = (int)((s.H + P.R - 1) / P.R);
        P.vec = 1;
        P.lag = 1;
        P.frame_fast = 1;
        T.proj_prefix[i + 1] = T.proj_prefix[i] + (int)((I.hw + PROJ_T - 1) / PROJ_T);
        T.qp_prefix[i + 1] = T.qp_prefix[i] + (int)((I.hw + QP_T - 1) / QP_T);
        // the lean passes: the lean pipeline with the item's column
        // width, energies of even / odd iterations, stop decisions by ticket
        for (int par = 0; par < 2; ++par) {
            tv::Pass &Q = I.tvq[par];
            Q = P;
            // halos of 4 columns for either width: with W % 4 == 0 every
            // band window starts on a multiple of 4 columns, so that a lane
            // pair's 16-byte copies (2 columns per lane) are aligned
            const int cpl = s.cpl == 2 ? 2 : 4;
            Q.cpl = cpl;
            Q.hl = 4;
            Q.hr = 4;
            Q.own = 32 * cpl - 8;
            Q.nbands = tv::band_count((int)s.W, 32 * cpl, Q.hl, Q.hr);
            Q.energy = reinterpret_cast<double *>(ws + L.energy +
                                                  (par ? L.item_e1[k] : L.item_e[k]));
            Q.stopj = reinterpret_cast<int *>(ws + L.item_stop[k]);
            Q.ticket = reinterpret_cast<unsigned *>(ws + L.item_stop[k] + sizeof(int) * s.B);
            // the fused iteration: the TV pass loads x_k and applies
            // x_k + lam (c phi_b) (the projection's rounding), writing x_{k+1}
            Q.f = par ? I.xp : I.x;
            Q.u = par ? I.x : I.xp;
            Q.proj = 1;
            Q.bits = I.bits;
            Q.cmap = I.c;
            Q.lam = I.lam;
        }
        T.tv_prefix[i + 1] = T.tv_prefix[i] + P.nbands * P.nchunks * P.nf;
        // both parities have the same geometry
        T.tq_prefix[i + 1] =
            T.tq_prefix[i] + I.tvq[0].nbands * I.tvq[0].nchunks * I.tvq[0].nf;
    }
}

// After an odd number of lean iterations the last x is in xp: copy
// it into every item's x.
__global__ void __launch_bounds__(PROJ_T) k_batch_copy_x(const Table *__restrict__ T) {
    const int g = blockIdx.x;
    if (g >= T->proj_prefix[T->n]) return;
    const int i = find_item(T->proj_prefix, T->n, g);
    const Item &I = T->it[i];
    const int64_t p = (int64_t)(g - T->proj_prefix[i]) * PROJ_T + threadIdx.x;
    if (p >= I.hw) return;
    for (int b = 0; b < I.B; ++b) I.x[b * I.hw + p] = I.xp[b * I.hw + p];
}

// A bounded wait of a grid that another one feeds, on purpose without one:
// one warp polls a count that nothing raises at most `polls` times, then sets
// bit 1 of the batch status.
__global__ void k_wait_selftest(const unsigned *count, unsigned polls) {
    unsigned ns = 32;
    for (unsigned n = 0; n < polls; ++n) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
        if (v != 0u) return;
        __nanosleep(ns);
        if (ns < 1024) ns <<= 1;
    }
    if (threadIdx.x == 0) atomicOr(&g_batch_status, 2u);
}

int wait_selftest(unsigned polls, unsigned *count, cudaStream_t s) {
    SCI_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned), s));
    k_wait_selftest<<<1, 32, 0, s>>>(count, polls);
    SCI_LAUNCHED("k_wait_selftest");
    return SCI_OK;
}

// The lean pass unless SCI_BATCH_QUEUE=0 or a mask is off the 16-byte
// boundaries of its vector loads.
bool lean_enabled(const Table &T) {
    for (int i = 0; i < T.n; ++i)
        if (reinterpret_cast<uintptr_t>(T.it[i].bits) & 15u) return false;
    const char *e = getenv("SCI_BATCH_QUEUE");
    return !(e && atoi(e) == 0);
}

int enqueue(const Table &T, Table *dT, const Layout &L, char *ws, int n, int iters, int K,
            int accelerate, int init_x0, cudaStream_t s) {
    const int pb = T.proj_prefix[n], tb = (T.tv_prefix[n] + tv::WPB - 1) / tv::WPB;
    if (init_x0 || accelerate) {
        if (init_x0 && accelerate) k_batch_init<true, true><<<pb, PROJ_T, 0, s>>>(dT);
        else if (init_x0) k_batch_init<true, false><<<pb, PROJ_T, 0, s>>>(dT);
        else k_batch_init<false, true><<<pb, PROJ_T, 0, s>>>(dT);
        SCI_LAUNCHED("k_batch_init");
    }
    if (lean_enabled(T)) {
        // the items' stop decisions and tickets: a ticket counts the TV
        // tasks of an iteration and is reset by the last one, so it starts
        // at zero once per solve
        SCI_CUDA(cudaMemsetAsync(ws + L.stop, 0, L.total - L.stop, s));
        bool narrow = false;
        for (int i = 0; i < n; ++i)
            narrow = narrow || T.it[i].tvq[0].cpl == 2 || narrow_tail(T.it[i].tvq[0]);
        for (int k = 0; k < iters; ++k)
            if (int e = iteration_launch(T, dT, k, accelerate != 0, K - 1, narrow, s)) return e;
        if (iters & 1) {  // the last TV pass wrote xp
            k_batch_copy_x<<<pb, PROJ_T, 0, s>>>(dT);
            SCI_LAUNCHED("k_batch_copy_x");
        }
        return SCI_OK;
    }
    const size_t ebytes = L.total - L.energy;
    // bulk-copy projection unless a mask is not 16-byte aligned (the other
    // planes are checked by check(); SCI_PROJ_TMA=0 selects the plain kernel)
    int maxB = 1;
    bool bulk = true;
    for (int i = 0; i < n; ++i) {
        maxB = std::max(maxB, T.it[i].B);
        bulk = bulk && (reinterpret_cast<uintptr_t>(T.it[i].bits) & 15u) == 0;
    }
    if (const char *e = getenv("SCI_PROJ_TMA")) bulk = bulk && atoi(e) != 0;
    for (int it = 0; it < iters; ++it) {
        const size_t psm = sizeof(float) * (size_t)maxB * PROJ_T;  // <= 32 KB
        if (bulk) {
            if (accelerate) k_batch_proj_tma<true><<<pb, PROJ_T / 4, psm, s>>>(dT);
            else k_batch_proj_tma<false><<<pb, PROJ_T / 4, psm, s>>>(dT);
        } else {
            if (accelerate) k_batch_proj<true><<<pb, PROJ_T, 0, s>>>(dT);
            else k_batch_proj<false><<<pb, PROJ_T, 0, s>>>(dT);
        }
        SCI_LAUNCHED("k_batch_proj");
        SCI_CUDA(cudaMemsetAsync(ws + L.energy, 0, ebytes, s));
        k_batch_tv<0><<<tb, tv::WPB * 32, 0, s>>>(dT);
        SCI_LAUNCHED("k_batch_tv");
        if (K >= 3) {
            k_batch_tv<1><<<tb, tv::WPB * 32, 0, s>>>(dT);
            SCI_LAUNCHED("k_batch_tv fixup");
        }
    }
    return SCI_OK;
}

// The whole solve of a batch (table upload, then the loop, captured once
// into a cached CUDA graph when use_graph).
int solve(const sci_batch_item *items, int n, int iters, int tv_iter_max, float eps,
                 int accelerate, int init_x0, int use_graph, void *workspace,
                 size_t workspace_bytes, cudaStream_t s) {
    const Layout L = layout(items, n, tv_iter_max);
    SCI_CHECK_ARG(workspace && workspace_bytes >= L.total,
                  "batch: workspace of %zu bytes needed, got %zu", L.total, workspace_bytes);
    char *ws = static_cast<char *>(workspace);
    Table *hT = new Table;
    build_table(items, n, tv_iter_max, eps, ws, L, *hT);
    Table *dT = reinterpret_cast<Table *>(ws + L.table);
    // the table is small; a stream-ordered copy from this host struct needs
    // it to stay alive until the copy ran, so the copy is synchronous here
    cudaError_t ce = cudaStreamSynchronize(s);
    if (ce == cudaSuccess) ce = cudaMemcpy(dT, hT, sizeof(Table), cudaMemcpyHostToDevice);
    if (ce != cudaSuccess) {
        delete hT;
        return cuda_status(ce, "batch table upload");
    }
    int rc = SCI_OK;
    if (!use_graph) {
        rc = enqueue(*hT, dT, L, ws, n, iters, tv_iter_max, accelerate, init_x0, s);
        delete hT;
        return rc;
    }
    std::string key(reinterpret_cast<const char *>(hT), sizeof(Table));
    key_append(key, iters, accelerate, init_x0);
    rc = run_graph("batch graph capture", key, s, [&](cudaStream_t cs) {
        return enqueue(*hT, dT, L, ws, n, iters, tv_iter_max, accelerate, init_x0, cs);
    });
    delete hT;
    return rc;
}

}  // namespace batch
}  // namespace sci

using namespace sci;
using namespace sci::batch;

extern "C" {

int sci_batch_workspace_bytes(const sci_batch_item *items, int n, int tv_iter_max,
                              size_t *bytes) {
    if (int e = check(items, n, tv_iter_max)) return e;
    SCI_CHECK_ARG(bytes, "null bytes");
    *bytes = layout(items, n, tv_iter_max).total;
    return SCI_OK;
}

int sci_batch_autotune(sci_batch_item *items, int n, int iters, int tv_iter_max, float eps,
                       int accelerate, int *iters_per_launch, void *workspace,
                       size_t workspace_bytes, void *stream) {
    if (int e = check(items, n, tv_iter_max)) return e;
    const Layout L = layout(items, n, tv_iter_max);
    SCI_CHECK_ARG(workspace && workspace_bytes >= L.total, "batch: workspace too small");
    SCI_CHECK_ARG(iters >= 0, "batch: iters must be >= 0");
    cudaStream_t s = as_stream(stream);
    // Every candidate is timed on the batch itself -- a few iterations of its
    // own solve from x0 = At(y / Phi_sum) (overwriting x): chunk heights that
    // make 1, 2, 3 or 6 waves of work items of the TV pass.  Measured, us per
    // iteration at 1 / 2 / 3 / 6: 4 items of up to 256 x 256 x 24 51 / 64 / 72;
    // 6 of up to 512 x 512 x 32 185 / 186 / 193 / 230; 16 235 / 210 / 219 /
    // 259; 64 of up to 1024 x 1024 x 32 1890 (1 to 3 waves are too few) / 1716.  The
    // choice is cached per process for the batch's list of shapes.
    const int probe = std::max(1, std::min(iters, 6));
    std::string key;
    key_append(key, n, tv_iter_max, probe, accelerate);
    for (int i = 0; i < n; ++i) key_append(key, items[i].B, items[i].H, items[i].W);
    static std::mutex mu;
    static std::map<std::string, int> tuned;  // chunk height
    auto apply = [&](int R) {
        for (int i = 0; i < n; ++i) items[i].R = even_R(items[i].H, R);
    };
    for (int i = 0; i < n; ++i) items[i].cpl = 4;
    if (iters_per_launch) *iters_per_launch = 0;
    {
        std::lock_guard<std::mutex> lk(mu);
        auto f = tuned.find(key);
        if (f != tuned.end()) {
            apply(f->second);
            return SCI_OK;
        }
    }
    cudaEvent_t e0, e1;
    SCI_CUDA(cudaEventCreate(&e0));
    SCI_CUDA(cudaEventCreate(&e1));
    int rc = SCI_OK, bR = 0, last = 0;
    float best = 1e30f;
    for (int waves : {1, 2, 3, 6}) {
        const int R = waves_R(items, n, waves);
        if (R == last) continue;
        last = R;
        apply(R);
        float ms = 0.f;
        for (int rep = 0; rep <= 2 && rc == SCI_OK; ++rep) {  // the first run warms up
            cudaEventRecord(e0, s);
            rc = solve(items, n, probe, tv_iter_max, eps, accelerate, 1, 0, workspace,
                       workspace_bytes, s);
            if (rc != SCI_OK) break;
            cudaEventRecord(e1, s);
            cudaEventSynchronize(e1);
            float t = 0.f;
            cudaEventElapsedTime(&t, e0, e1);
            if (rep > 0) ms += t;
        }
        if (rc != SCI_OK) break;
        if (ms < best) {
            best = ms;
            bR = R;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc == SCI_OK) {
        apply(bR);
        std::lock_guard<std::mutex> lk(mu);
        tuned[key] = bR;
    }
    return rc;
}

int sci_batch_selftest_queue_wait(unsigned int polls, void *workspace, size_t workspace_bytes,
                                  void *stream) {
    SCI_CHECK_ARG(polls >= 1 && polls <= (1u << 20), "selftest: polls in [1, 2^20]");
    SCI_CHECK_ARG(workspace && workspace_bytes >= kWaitBytes,
                  "selftest: a workspace of %zu bytes is needed", kWaitBytes);
    return wait_selftest(polls, static_cast<unsigned *>(workspace), as_stream(stream));
}

int sci_batch_gap_tv(const sci_batch_item *items, int n, int iters, int tv_iter_max, float eps,
                     int accelerate, int init_x0, int use_graph, int iters_per_launch,
                     void *workspace, size_t workspace_bytes, void *stream) {
    if (int e = check(items, n, tv_iter_max)) return e;
    SCI_CHECK_ARG(iters >= 0, "batch: iters must be >= 0");
    SCI_CHECK_ARG(iters_per_launch >= 0, "batch: iters_per_launch must be >= 0");
    return solve(items, n, iters, tv_iter_max, eps, accelerate, init_x0, use_graph, workspace,
                 workspace_bytes, as_stream(stream));
}

}  // extern "C"
