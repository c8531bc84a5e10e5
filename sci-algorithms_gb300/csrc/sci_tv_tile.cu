// Launches of the register-tile TV pass (sci_tv_tile.cuh): windows of 64
// columns x 48 rows (thread: 2 x 8 pixels, 6 warps), 4 blocks per SM.
// Window shapes measured (us per call with its stop-test launch and memset,
// 28 x 256 x 256 / 10 x 512 x 512 / 8 x 1001 x 1023 / 30 steps of 16 x 1024
// x 1024): 6 warps at 80 registers 22.6 / 24.7 / 57.6 / 602; 6 at 96 25.2 /
// 26.8 / 61.5 / 693; 8 at 80 23.0 / 24.8 / 57.5 / 607; 8 at 128 (no spills)
// 24.7 / 26.3 / 63.6 / 745; 4 at 96 23.9 / 25.6 / 59.5 / 645; 2 x 4 pixels,
// 8 warps at 64 24.7 / 26.1 / 67.1 / 719.  Warps in flight count for more
// than the last spills.
#include "sci_tv_rule.cuh"
#include "sci_tv_tile_launch.cuh"

namespace sci {
namespace tv {

void tile_small_geometry(Pass &P);  // sci_tv_tile_small.cu
void launch_tile_small(const Pass &P, bool pin, bool final_pass, int proj, cudaStream_t s);
void launch_tile_small_fix(const Pass &P, bool pin, int proj, cudaStream_t s);

namespace {
using Large = tile::Shape<2, 4, 6, 4>;
static_assert(tile::Geo<2, 4, 6>::COLS == kWinCols && tile::Geo<2, 4, 6>::ROWS == kWinRows &&
                  tile::HALO == kWinHalo,
              "tile_wins counts the large windows");

// Few windows (the GPU holds 608): half the pixels per thread, so that a
// window's chain of updates is shorter and there are more warps to overlap.
// The line lies between the last size that gains and the first that does not.
// Measured (TV call with its memset and stop-test launch, large /
// small windows, us): 8 x 64 x 96 (32 windows of the large shape) 11.9 / 10.4,
// 8 x 256 x 256 (280) 14.5 / 12.6, 32 x 128 x 128 (384) 14.5 / 14.6, 12 x 256
// x 256 (420) 15.8 / 16.4, 16 x 256 x 256 (560) 16.5 / 16.7, 28 x 256 x 256
// (980) 22.3 / 22.8, 24 x 512 x 512 (2808) 41.3 / 47.4.
bool small(const Pass &P) { return Large::windows(P.nf, P.H, P.W) <= 300; }
}  // namespace

void tile_geometry(Pass &P) {
    if (small(P)) tile_small_geometry(P);
    else Large::geometry(P);
}
int tile_columns() { return 2; }

void launch_tile(const Pass &P, bool pin, bool final_pass, int proj, cudaStream_t s) {
    if (small(P)) launch_tile_small(P, pin, final_pass, proj, s);
    else Large::launch(P, pin, final_pass, proj, s);
}

void launch_tile_fix(const Pass &P, bool pin, int proj, cudaStream_t s) {
    if (small(P)) launch_tile_small_fix(P, pin, proj, s);
    else Large::launch_fix(P, pin, proj, s);
}

}  // namespace tv
}  // namespace sci
