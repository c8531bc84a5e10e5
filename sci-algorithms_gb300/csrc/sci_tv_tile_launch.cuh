// Launch helpers of the register-tile TV pass, instantiated per window shape
// in sci_tv_tile.cu (64 x 48, 2 x 8 pixels per thread) and
// sci_tv_tile_small.cu (64 x 32, 2 x 4 pixels per thread).
#pragma once
#include "sci_tv_tile.cuh"

namespace sci {
namespace tv {
namespace tile {

inline int64_t pass_windows(const Pass &P) { return (int64_t)P.nbands * P.nchunks * P.nf; }

template <int C, int N, int NW, int MINB>
struct Shape {
    static int64_t windows(int64_t nf, int64_t H, int64_t W) {
        using G = Geo<C, N, NW>;
        return nf * window_count((int)H, G::ROWS) * window_count((int)W, G::COLS);
    }
    static void geometry(Pass &P) {
        using G = Geo<C, N, NW>;
        P.nchunks = window_count(P.H, G::ROWS);
        P.nbands = window_count(P.W, G::COLS);
        P.early = pass_windows(P) > kSMs * MINB;
    }
    template <bool PIN, bool OUT_U, int PROJ>
    static void main_pass(const Pass &P, cudaStream_t s) {
        (void)launch_dep(k_tv_tile<C, N, NW, MINB, PIN, OUT_U, PROJ>,
                         dim3((unsigned)pass_windows(P)), dim3(NW * 32), 0, s, P);
        // errors: the caller's cudaGetLastError
    }
    template <bool PIN, int PROJ>
    static void fix_pass(const Pass &P, cudaStream_t s) {
        (void)launch_dep(k_tv_tile_fix<C, N, NW, MINB, PIN, PROJ>,
                         dim3((unsigned)pass_windows(P)), dim3(NW * 32), 0, s, P);
    }
    // proj as launch_slim's, 5 the spectral projection
    static void launch(const Pass &P, bool pin, bool final_pass, int proj, cudaStream_t s) {
        if (proj == 3) main_pass<false, true, 3>(P, s);
        else if (proj == 2) main_pass<false, true, 4>(P, s);
        else if (proj == 5) main_pass<false, true, 5>(P, s);
        else if (proj) main_pass<false, true, 1>(P, s);
        else if (!pin && final_pass) main_pass<false, true, 0>(P, s);
        else if (!pin) main_pass<false, false, 0>(P, s);
        else if (final_pass) main_pass<true, true, 0>(P, s);
        else main_pass<true, false, 0>(P, s);
    }
    static void launch_fix(const Pass &P, bool pin, int proj, cudaStream_t s) {
        if (proj == 3) fix_pass<false, 3>(P, s);
        else if (proj == 2) fix_pass<false, 4>(P, s);
        else if (proj == 5) fix_pass<false, 5>(P, s);
        else if (proj) fix_pass<false, 1>(P, s);
        else if (pin) fix_pass<true, 0>(P, s);
        else fix_pass<false, 0>(P, s);
    }
};

}  // namespace tile
}  // namespace tv
}  // namespace sci
