// Launches of the register-tile TV pass (sci_tv_tile.cuh): windows of 64
// columns x 48 rows (thread: 2 x 8 pixels, 6 warps), 4 blocks per SM.
// Window shapes measured (us per call with its stop-test launch and memset,
// 28 x 256 x 256 / 10 x 512 x 512 / 8 x 1001 x 1023 / 30 steps of 16 x 1024
// x 1024): 6 warps at 80 registers 22.6 / 24.7 / 57.6 / 602; 6 at 96 25.2 /
// 26.8 / 61.5 / 693; 8 at 80 23.0 / 24.8 / 57.5 / 607; 8 at 128 (no spills)
// 24.7 / 26.3 / 63.6 / 745; 4 at 96 23.9 / 25.6 / 59.5 / 645; 2 x 4 pixels,
// 8 warps at 64 24.7 / 26.1 / 67.1 / 719.  Warps in flight count for more
// than the last spills.
#include "sci_tv_tile_launch.cuh"

namespace sci {
namespace tv {

void tile_small_geometry(Pass &P);  // sci_tv_tile_small.cu
void launch_tile_small(const Pass &P, bool pin, bool final_pass, int proj, cudaStream_t s);
void launch_tile_small_fix(const Pass &P, bool pin, int proj, cudaStream_t s);

namespace {
using Large = tile::Shape<2, 4, 6, 4>;

// Fewer windows than fill the GPU's 608 slots: half the pixels per thread, so
// that a window's chain of updates is shorter and there are more warps to
// overlap.  Measured (TV call with its memset and stop-test launch, large /
// small windows, us): 8 x 64 x 96 (32 windows of the large shape) 11.9 / 10.4,
// 8 x 256 x 256 (280) 14.5 / 12.6, 32 x 128 x 128 (384) 14.5 / 14.6, 12 x 256
// x 256 (420) 15.8 / 16.4, 16 x 256 x 256 (560) 16.5 / 16.7, 28 x 256 x 256
// (980) 22.3 / 22.8, 24 x 512 x 512 (2808) 41.3 / 47.4.
bool small(const Pass &P) { return Large::windows(P.nf, P.H, P.W) <= 300; }
}  // namespace

// Which calls run on tiles (slim: the lean row pipeline could run it, frames
// of nf x H x W), by the number of windows.  A tile pass costs about 10 us +
// 11 to 13 us per 1000 windows, halo and two barriers per update included; the
// row pipelines have a chain of stages per row as their fixed part, about 24
// us (lean) and 28 us (generic), and less per pixel -- the lean one the less
// the wider the frame, as its bands of 64 or 128 columns cover narrow frames
// badly.  Measured, tile against pipeline, us (windows):
//   lean, W <= 256: 64 x 256 x 256 32.2 / 37.4 (2240), 400 x 128 x 128 59.7 /
//   60.9 (3600), 128 x 256 x 256 59.4 / 60.8 (4480), 256 x 256 x 256 120 / 100
//   (8960); W <= 512: 20 x 384 x 384 25.3 / 33.9 (1400), 24 x 512 x 512 41.1 /
//   45.2 (2808), 32 x 512 x 512 55.3 / 53.5 (3744); wider: 4 x 1024 x 1024
//   31.0 / 34.4 (1976), 10 x 768 x 768 45.6 / 44.9 (2660, an iteration of a
//   solve), 6 x 1024 x 1024 42.0 / 39.1 (2964), 24 x 2048 x 2048 560 / 310;
//   generic: 10 x 517 x 643 31 / 45 (1560), 16 x 1001 x 1023 112 / 134
//   (7600), 32 x 1001 x 1023 211 / 203 (15200), 24 x 2045 x 2047 604 / 467
//   (45288); 30 steps (up to 8 passes): 10 x 517 x 643 161 / 259, 16 x 1024 x
//   1024 617 / 795, 32 x 1024 x 1024 1144 / 1192 (15808), 12 x 2048 x 2048
//   1614 / 1477.
bool tile_wins(int64_t nf, int64_t H, int64_t W, bool slim) {
    const int64_t lean = W <= 256 ? 4500 : W <= 512 ? 3300 : 2500;
    return Large::windows(nf, H, W) <= (slim ? lean : 14000);
}

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
