// The register-tile TV pass for few windows (see sci_tv_tile.cu): 64 x 32
// pixels, 2 x 4 per thread, 8 warps at 64 registers.
#include "sci_tv_tile_launch.cuh"

namespace sci {
namespace tv {
namespace {
using Small = tile::Shape<2, 2, 8, 4>;
}

void tile_small_geometry(Pass &P) { Small::geometry(P); }
void launch_tile_small(const Pass &P, bool pin, bool final_pass, int proj, cudaStream_t s) {
    Small::launch(P, pin, final_pass, proj, s);
}
void launch_tile_small_fix(const Pass &P, bool pin, int proj, cudaStream_t s) {
    Small::launch_fix(P, pin, proj, s);
}

}  // namespace tv
}  // namespace sci
