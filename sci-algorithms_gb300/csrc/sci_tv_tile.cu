// Launches of the register-tile TV pass (sci_tv_tile.cuh): windows of 64
// columns x 48 rows (thread: 2 x 8 pixels, 6 warps), 4 blocks per SM.
// Window shapes measured (us per call with its stop-test launch and memset,
// 28 x 256 x 256 / 10 x 512 x 512 / 8 x 1001 x 1023 / 30 steps of 16 x 1024
// x 1024): 6 warps at 80 registers 22.6 / 24.7 / 57.6 / 602; 6 at 96 25.2 /
// 26.8 / 61.5 / 693; 8 at 80 23.0 / 24.8 / 57.5 / 607; 8 at 128 (no spills)
// 24.7 / 26.3 / 63.6 / 745; 4 at 96 23.9 / 25.6 / 59.5 / 645; 2 x 4 pixels,
// 8 warps at 64 24.7 / 26.1 / 67.1 / 719.  Warps in flight count for more
// than the last spills.
#include "sci_tv_tile.cuh"

namespace sci {
namespace tv {

namespace {
constexpr int C = 2, N = 4, NW = 6, MINB = 4;

dim3 blocks(const Pass &P) { return dim3((unsigned)tile_blocks(P)); }

template <bool PIN, bool OUT_U, int PROJ>
void main_pass(const Pass &P, cudaStream_t s) {
    (void)launch_dep(tile::k_tv_tile<C, N, NW, MINB, PIN, OUT_U, PROJ>, blocks(P), dim3(NW * 32),
                     0, s, P);  // reported by the caller's cudaGetLastError
}
template <bool PIN, int PROJ>
void fix_pass(const Pass &P, cudaStream_t s) {
    (void)launch_dep(tile::k_tv_tile_fix<C, N, NW, MINB, PIN, PROJ>, blocks(P), dim3(NW * 32), 0,
                     s, P);
}
}  // namespace

// Which calls run on tiles (slim: the lean row pipeline could run it, frames
// of nf x H x W), by the number of windows.  A tile pass costs about 10 us +
// 17 us per 1000 windows, halo and two barriers per update included; the row
// pipelines have a chain of stages per row as their fixed part, about 24 us
// (lean) and 28 us (generic), and less per pixel.  Measured, tile against
// pipeline, us (windows):
//   lean: 10 x 512 x 512 24.7 / 30.8 (1170), 16 x 512 x 512 32.9 / 37.1
//   (1872), 4 x 1024 x 1024 34.9 / 35.0 (1976), 24 x 512 x 512 45.1 / 45.2
//   (2808), 8 x 1024 x 1024 57 / 47 (3952), 24 x 2048 x 2048 560 / 310;
//   generic: 10 x 517 x 643 31 / 45 (1560), 16 x 1001 x 1023 107 / 133
//   (7600), 24 x 2045 x 2047 576 / 463 (45288); 30 steps (up to 8 passes): 10
//   x 517 x 643 161 / 259, 16 x 1024 x 1024 602 / 792, 24 x 2048 x 2048 3130
//   / 2570.
bool tile_wins(int64_t nf, int64_t H, int64_t W, bool slim) {
    using G = tile::Geo<C, N, NW>;
    return nf * tile::window_count((int)H, G::ROWS) * tile::window_count((int)W, G::COLS) <=
           (slim ? 2000 : 14000);
}

// Window counts and the pass's launches.
void tile_geometry(Pass &P) {
    using G = tile::Geo<C, N, NW>;
    P.nchunks = tile::window_count(P.H, G::ROWS);
    P.nbands = tile::window_count(P.W, G::COLS);
}
int tile_columns() { return C; }
int64_t tile_blocks(const Pass &P) { return (int64_t)P.nbands * P.nchunks * P.nf; }
int tile_resident_blocks() { return MINB; }

// proj as launch_slim's, 5 the spectral projection
void launch_tile(const Pass &P, bool pin, bool final_pass, int proj, cudaStream_t s) {
    if (proj == 3) main_pass<false, true, 3>(P, s);
    else if (proj == 2) main_pass<false, true, 4>(P, s);
    else if (proj == 5) main_pass<false, true, 5>(P, s);
    else if (proj) main_pass<false, true, 1>(P, s);
    else if (!pin && final_pass) main_pass<false, true, 0>(P, s);
    else if (!pin) main_pass<false, false, 0>(P, s);
    else if (final_pass) main_pass<true, true, 0>(P, s);
    else main_pass<true, false, 0>(P, s);
}

void launch_tile_fix(const Pass &P, bool pin, int proj, cudaStream_t s) {
    if (proj == 3) fix_pass<false, 3>(P, s);
    else if (proj == 2) fix_pass<false, 4>(P, s);
    else if (proj == 5) fix_pass<false, 5>(P, s);
    else if (proj) fix_pass<false, 1>(P, s);
    else if (pin) fix_pass<true, 0>(P, s);
    else fix_pass<false, 0>(P, s);
}

}  // namespace tv
}  // namespace sci
