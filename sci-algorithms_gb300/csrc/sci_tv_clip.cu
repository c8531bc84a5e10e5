// The MATLAB clip files' single pass (up to 4 dual updates) on the lean row
// pipeline (sci_tv_slim.cuh, FORM 2), 4 columns per lane: 8 x 1080 x 1920 with
// the projection of a float mask on load 49 us, behind a residual pass of 28,
// where the generic pipeline took 82 behind a projection of 44 (bytes alone:
// 30 and 20 us).  Bound by issue, as the other lean passes; 4 blocks per SM
// need no spills.
#include "sci_tv_slim_launch.cuh"

namespace sci {
namespace tv {
namespace {
using namespace slim;
constexpr int MB = 4;

template <int PROJ>
cudaError_t launch(const Pass &P, int SG, cudaStream_t s) {
    const dim3 g(pass_blocks(P)), b(WPB * 32);
    switch (SG) {
        case 1: return launch_dep(k_tv_slim_clip<1, MB, PROJ>, g, b, 0, s, P);
        case 2: return launch_dep(k_tv_slim_clip<2, MB, PROJ>, g, b, 0, s, P);
        case 3: return launch_dep(k_tv_slim_clip<3, MB, PROJ>, g, b, 0, s, P);
        default: return launch_dep(k_tv_slim_clip<4, MB, PROJ>, g, b, 0, s, P);
    }
}
}  // namespace

// proj: 0 none, 1 packed mask, 2 float mask
void launch_clip(const Pass &P, int SG, int proj, cudaStream_t s) {
    if (proj == 2) (void)launch<2>(P, SG, s);  // reported by the caller's cudaGetLastError
    else if (proj) (void)launch<1>(P, SG, s);
    else (void)launch<0>(P, SG, s);
}
int clip_resident_blocks() { return MB; }

}  // namespace tv
}  // namespace sci
