// Launches of the unrolled solver's TV kernels on register tiles: the
// forward that writes its tape (sci_tv_tile.cuh) and the adjoint
// (sci_tv_adjoint.cuh).
#include <algorithm>
#include <initializer_list>

#include "sci_tv_adjoint.cuh"

namespace sci {
namespace {

using namespace tv::tile;

// 1: rows aligned for vectors, 0: not, -1: a window's rows (at most 64 + 2)
// span 4 GB or more.
int access(int64_t H, int64_t W, std::initializer_list<const void *> ptrs) {
    if (std::min<int64_t>(H, 66) * W >= int64_t(1) << 30) return -1;
    for (const void *p : ptrs)
        if (reinterpret_cast<uintptr_t>(p) % 8) return 0;
    return W % 2 == 0;
}

template <int N, int NW, int MINB, typename Args>
int64_t windows(Args &P) {
    using G = Geo<2, N, NW>;
    P.nchunks = window_count(P.H, G::ROWS);
    P.nbands = window_count(P.W, G::COLS);
    const int64_t n = (int64_t)P.nbands * P.nchunks * P.nf;
    P.early = n > kSMs * MINB;
    return n;
}

template <int N, int NW, int MINB>
cudaError_t tape(tv::Pass &P, bool out, cudaStream_t s) {
    const dim3 g((unsigned)windows<N, NW, MINB>(P)), b(NW * 32);
    if (out) return launch_dep(k_tv_tile_tape<2, N, NW, MINB, true>, g, b, 0, s, P);
    return launch_dep(k_tv_tile_tape<2, N, NW, MINB, false>, g, b, 0, s, P);
}

template <int N, int NW, int MINB>
cudaError_t adjoint_pass(Adj &P, cudaStream_t s) {
    const dim3 g((unsigned)windows<N, NW, MINB>(P)), b(NW * 32);
    return launch_dep(k_tv_adjoint<2, N, NW, MINB>, g, b, 0, s, P);
}

}  // namespace

// Input frames of the two calls below: v = x + lam (q phi_b) of frames frame0
// .. frame0 + nf - 1 of a stack of scenes of B frames (x points at the first
// of them, q and phi at the whole maps, lam to the device).

// U <= 4 updates (no stop test), writing 4 p_1 .. 4 p_U to tape_p [U][nf][2]
// [H][W], u_1 .. u_{U-1} to tape_u [U-1][nf][H][W] and, when u is given, u_U.
int tv_tape(const float *x, const float *q, const float *phi, const float *lam, int64_t frame0,
            int64_t nf, int64_t B, int64_t H, int64_t W, float weight, int U, float *u,
            float *tape_p, float *tape_u, cudaStream_t s) {
    tv::Pass P{};
    P.f = x;
    P.cmap = q;
    P.phi = phi;
    P.lam_dev = lam;
    P.frame0 = (int)frame0;
    P.B = (int)B;
    P.u = u;
    P.nf = (int)nf;
    P.H = (int)H;
    P.W = (int)W;
    P.fs = H * W;
    P.S = U;
    P.tau = 0.25f;
    P.tw = 0.25f / weight;
    P.weight = weight;
    P.tape_p = tape_p;
    P.tape_u = tape_u;
    P.vec = access(H, W, {x, q, phi, u, tape_p, tape_u});
    // Windows of 64 x 32, 2 x 4 pixels per thread, 32 warps per SM: 0.20 ms of
    // a 16 x 256 x 256 x 8 iteration's 0.35 with the adjoint (2 x 8 pixels at
    // 16 warps: 11 us more; at 24 with spills: 20 us).
    SCI_CUDA((tape<2, 8, 4>(P, u != nullptr, s)));
    return SCI_OK;
}

// fbar = d/dv of <xbar, TV(v)> from the tape of tv_tape.
int tv_adjoint(const float *x, const float *q, const float *phi, const float *lam, int64_t frame0,
               int64_t nf, int64_t B, int64_t H, int64_t W, float weight, int U,
               const float *tape_p, const float *tape_u, const float *xbar, float *fbar,
               cudaStream_t s) {
    Adj P{};
    P.f = x;
    P.cmap = q;
    P.phi = phi;
    P.lam_dev = lam;
    P.frame0 = (int)frame0;
    P.B = (int)B;
    P.tape_u = tape_u;
    P.tape_p = tape_p;
    P.xbar = xbar;
    P.fbar = fbar;
    P.nf = (int)nf;
    P.H = (int)H;
    P.W = (int)W;
    P.U = U;
    P.tw = 0.25f / weight;
    P.vec = access(H, W, {x, q, phi, tape_p, tape_u, xbar, fbar});
    // The same windows at 24 warps per SM (80 registers); 64 registers spill
    // (+35 us per iteration), 2 x 8 pixels at 16 warps +14 us, 48- and 64-row
    // windows of 2 x 4 pixels +4 and +45 us.
    SCI_CUDA((adjoint_pass<2, 8, 3>(P, s)));
    return SCI_OK;
}

}  // namespace sci
