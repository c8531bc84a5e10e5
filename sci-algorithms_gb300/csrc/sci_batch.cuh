// Device item table of the batched uneven GAP-TV (sci_batch.cu: the generic
// launches, autotuner and C ABI; sci_batch_lean.cu: the lean pass's).
#pragma once

#include "sci_tv.cuh"

namespace sci {
namespace batch {

constexpr int MAXI = 256;    // items per batch
constexpr int PROJ_T = 256;  // pixels per projection tile of the generic launches
constexpr int QP_T = 128;    // pixels per residual task of the lean launches (one warp)

struct Item {
    tv::Pass tv;      // generic launches: f = xp (projected stack), u = x
    tv::Pass tvq[2];  // iterations of even / odd k: the lean pass with
                      // the projection applied on load from the residual map c,
                      // the stack ping-ponging x -> xp (even k) and xp -> x (odd
                      // k), the energies of even / odd k, the item's stop decisions
    const float *y;
    const uint32_t *bits;
    const float *phisum;
    float *x, *xp, *y1, *c;  // c: residual map (H W)
    int B;
    int64_t hw;
    float lam;
};

struct Table {
    int n;
    int proj_prefix[MAXI + 1];  // 256-pixel tiles
    int qp_prefix[MAXI + 1];    // 128-pixel residual tasks (one warp each)
    int tv_prefix[MAXI + 1];    // TV work items (one warp each) of the generic passes
    int tq_prefix[MAXI + 1];    // TV work items of the lean passes (tvq geometry)
    Item it[MAXI];
};

// A last band of 128 columns that owns at most 60 runs as one of 64, at half
// the work: a third to a sixth of a pass over frames 256 to 1024 wide.
__host__ __device__ __forceinline__ bool narrow_tail(const tv::Pass &P) {
    return P.cpl == 4 && P.nbands > 1 && P.W - (128 - P.hr + (P.nbands - 2) * P.own) <= 64 - P.hl;
}

__device__ __forceinline__ int find_item(const int *prefix, int n, int g) {
    int lo = 0, hi = n;  // prefix[lo] <= g < prefix[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (prefix[mid] <= g) lo = mid;
        else hi = mid;
    }
    return lo;
}

// sci_batch_lean.cu: one iteration of every item, a launch for each phase
// (narrow: some band runs 2 columns per lane).  Returns a negative status on
// a launch error.
int iteration_launch(const Table &T, const Table *dT, int k, bool accelerate, int S, bool narrow,
                     cudaStream_t s);
int resident_warps();  // TV work items in flight on the whole GPU

}  // namespace batch
}  // namespace sci
