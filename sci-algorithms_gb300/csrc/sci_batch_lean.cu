// Batched uneven GAP-TV: one iteration of every item as three launches.
//
// Residual tasks (128-pixel tiles: the GAP residual map c, as the
// single-measurement solver's fused iteration forms it), TV tasks (one
// (frame, row chunk, column band) work item of the register-lean pipeline
// each, which applies the projection x + lam (c phi_b) as it loads x) and
// stop-test tasks (the same work items) of all items; a warp finds its item
// through prefix sums.  Per item, the per-pixel arithmetic is that of the
// single-measurement solver, so each item's result is the same.
//
// What bounds it: the lean pass's issue on large batches, a work item's chain
// of rows where few are in flight.  A persistent launch whose warps took the
// tasks of all iterations from a queue, waiting for the tasks they build on,
// filled the gaps between phases but held its warps in waits and drew a stop
// test for every work item; us per iteration, queue / launches: 4
// items of up to 256 x 256 x 24 76 / 45, 8 85 / 61, 6 of up to 512 x 512 x 32
// 216 / 175, 16 257 / 201, 64 of up to 1024 x 1024 x 32 1855 / 1630.  Of the
// 201: TV 157 (the rate of one large measurement, times 1.35 in halo), maps
// 34, stop test 5 to 9.
#include "sci_batch.cuh"
#include "sci_tv_slim.cuh"

namespace sci {
namespace batch {

namespace {

constexpr int MINB = 4;  // resident blocks per SM the registers are sized for

__device__ __forceinline__ float bitf(uint32_t w, int b) { return ((w >> b) & 1u) ? 1.0f : 0.0f; }

// GAP residual map of one 128-pixel tile of item I (4 pixels per lane), the
// arithmetic of k_gap_resid_vec: yb = sum_b phi_b x_b in frame order, ACC:
// y1 += y - yb, c = (y1 - yb) / Phi_sum, else c = (y - yb) / Phi_sum, with
// x the iteration's TV input P.f.  Tile 0 also clears the energy sums the
// item's TV pass of this iteration adds to.
template <bool ACC>
__device__ __forceinline__ void resid_task(const Item &I, const tv::Pass &P, int tile, int lane) {
    if (tile == 0) {
        const int ne = P.nf * P.K * 2;
        for (int e = lane; e < ne; e += 32) P.energy[e] = 0.0;
    }
    const int64_t hw = I.hw;
    const int64_t p = (int64_t)tile * QP_T + lane * 4;
    if (p >= hw) return;  // hw % 4 == 0: all 4 pixels are inside
    const int B = I.B;
    const uint4 w = ld4(I.bits + p);
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int b = 0; b < B; ++b) {
        const float4 v = ld4(P.f + b * hw + p);
        s.x = fmaf(v.x, bitf(w.x, b), s.x);
        s.y = fmaf(v.y, bitf(w.y, b), s.y);
        s.z = fmaf(v.z, bitf(w.z, b), s.z);
        s.w = fmaf(v.w, bitf(w.w, b), s.w);
    }
    const float4 yv = ld4(I.y + p), ps = ld4(I.phisum + p);
    float4 r;
    if (ACC) {
        float4 tt = *reinterpret_cast<const float4 *>(I.y1 + p);
        tt.x = tt.x + (yv.x - s.x);
        tt.y = tt.y + (yv.y - s.y);
        tt.z = tt.z + (yv.z - s.z);
        tt.w = tt.w + (yv.w - s.w);
        st4(I.y1 + p, tt);
        r = make_float4(__fdiv_rn(tt.x - s.x, ps.x), __fdiv_rn(tt.y - s.y, ps.y),
                        __fdiv_rn(tt.z - s.z, ps.z), __fdiv_rn(tt.w - s.w, ps.w));
    } else {
        r = make_float4(__fdiv_rn(yv.x - s.x, ps.x), __fdiv_rn(yv.y - s.y, ps.y),
                        __fdiv_rn(yv.z - s.z, ps.z), __fdiv_rn(yv.w - s.w, ps.w));
    }
    st4(I.c + p, r);
}

// S updates of one work item, CPL columns per lane.
template <int S, bool ENERGY, bool N2>
__device__ __forceinline__ void run_item(const tv::Pass &P, int frame, int chunk, int band,
                                         int lane, const tv::slim::Rings &G4,
                                         const tv::slim::Rings &G2) {
    using namespace tv::slim;
    if constexpr (N2) {
        const int lo = 128 - P.hr + (P.nbands - 2) * P.own;  // of the last of 128-column bands
        const bool tail = P.cpl == 4 && band > 0 && band == P.nbands - 1 && narrow_tail(P);
        if (tail || P.cpl == 2) {
            tv::Pass Q = P;
            if (tail) {  // the last of three 64-column bands, owning from lo
                band = 2;
                Q.nbands = 3;
                Q.own = lo - (64 - P.hr);
            }
            return srun_mode<S, 2, ENERGY, 1>(Q, frame, chunk, band, lane, G2);
        }
    }
    srun_mode<S, 4, ENERGY, 1>(P, frame, chunk, band, lane, G4);
}

// The TV pass with S dual updates of one work item, or (FIX) its re-run with
// the stop index j the pass decided.
// N2: some band runs 2 columns per lane (otherwise that code is not built,
// which leaves the 4-column pipeline more registers).
template <int S, bool FIX, bool N2>
__device__ __forceinline__ void tv_task(const tv::Pass &P, int frame, int chunk, int band,
                                        int lane, const tv::slim::Rings &G4,
                                        const tv::slim::Rings &G2) {
    if (!FIX) return run_item<S, true, N2>(P, frame, chunk, band, lane, G4, G2);
    const int j = P.stopj[frame];
    if (j < 1 || j >= S) return;
    if (j == 1) return run_item<1, false, N2>(P, frame, chunk, band, lane, G4, G2);
    if constexpr (S > 2)
        if (j == 2) return run_item<2, false, N2>(P, frame, chunk, band, lane, G4, G2);
    if constexpr (S > 3) run_item<3, false, N2>(P, frame, chunk, band, lane, G4, G2);
}

// The item of task g, prefix[i] <= g < prefix[i + 1], searched by a whole warp
// in one round trip to memory for each 32 items.
__device__ __forceinline__ int warp_find(const int *prefix, int n, int g, int lane) {
    int i = 0;
    for (int q = 0; q < n; q += 32)
        i += __popc(__ballot_sync(0xffffffffu, q + lane < n && prefix[q + lane + 1] <= g));
    return i;
}

// One phase of iteration k over all items as a launch of its own.
template <bool ACC>
__global__ void __launch_bounds__(tv::WPB * 32, 4) k_batch_resid(const Table *__restrict__ T, int k) {
    grid_dep_wait();
    if (gridDim.x > kSMs * 8) grid_dep_launch();
    const int lane = threadIdx.x & 31, g = blockIdx.x * tv::WPB + (threadIdx.x >> 5);
    if (g >= T->qp_prefix[T->n]) return;
    const int i = warp_find(T->qp_prefix, T->n, g, lane);
    resid_task<ACC>(T->it[i], T->it[i].tvq[k & 1], g - T->qp_prefix[i], lane);
}

template <int S, bool FIX, bool N2>
__global__ void __launch_bounds__(tv::WPB * 32, MINB)
    k_batch_lean(const Table *__restrict__ T, int k) {
    __shared__ __align__(16) unsigned char smem[tv::slim::Smem<4, 1>::bytes];
    grid_dep_wait();
    if (gridDim.x > kSMs * MINB) grid_dep_launch();
    const int lane = threadIdx.x & 31, g = blockIdx.x * tv::WPB + (threadIdx.x >> 5);
    if (g >= T->tq_prefix[T->n]) return;
    const int i = warp_find(T->tq_prefix, T->n, g, lane);
    const tv::Pass &P = T->it[i].tvq[k & 1];
    int frame, chunk, band;
    tv::decode_index(P, g - T->tq_prefix[i], frame, chunk, band);
    constexpr int share = tv::slim::Smem<4, 1>::bytes / tv::WPB;
    tv_task<S, FIX, N2>(P, frame, chunk, band, lane, tv::slim::lane_rings<4, 1>(smem, lane, share),
                        tv::slim::lane_rings<2, 1>(smem, lane, share));
    if (!FIX) tv::decide_stops(P, lane);
}

}  // namespace

int resident_warps() { return MINB * tv::WPB * kSMs; }

int iteration_launch(const Table &T, const Table *dT, int k, bool accelerate, int S, bool narrow,
                 cudaStream_t s) {
    const dim3 t(tv::WPB * 32);
    const dim3 rg((T.qp_prefix[T.n] + tv::WPB - 1) / tv::WPB);
    const dim3 tg((T.tq_prefix[T.n] + tv::WPB - 1) / tv::WPB);
    if (accelerate) SCI_CUDA(launch_dep(k_batch_resid<true>, rg, t, 0, s, dT, k));
    else SCI_CUDA(launch_dep(k_batch_resid<false>, rg, t, 0, s, dT, k));
    SCI_LAUNCHED("k_batch_resid");
#define SCI_PHASE_CASE(SV, N2)                                                  \
    do {                                                                        \
        SCI_CUDA(launch_dep(k_batch_lean<SV, false, N2>, tg, t, 0, s, dT, k));  \
        SCI_LAUNCHED("k_batch_lean");                                           \
        if (SV < 2) break;                                                      \
        SCI_CUDA(launch_dep(k_batch_lean<SV, true, N2>, tg, t, 0, s, dT, k));   \
        SCI_LAUNCHED("k_batch_lean fix");                                       \
    } while (0)
    switch (S) {
        case 1: SCI_PHASE_CASE(1, true); break;
        case 2: SCI_PHASE_CASE(2, true); break;
        case 3: SCI_PHASE_CASE(3, true); break;
        default:
            if (narrow) SCI_PHASE_CASE(4, true);
            else SCI_PHASE_CASE(4, false);
            break;
    }
#undef SCI_PHASE_CASE
    return SCI_OK;
}

}  // namespace batch
}  // namespace sci
