// Which TV calls run on register tiles (sci_tv_tile.cuh) and which on the row
// pipelines: host code, free of CUDA.
//
// A tile pass of four updates costs about 10 us + 11 to 13 us per 1000 windows,
// and hardly less with fewer: its loads, stores and barriers stay. The
// pipelines have a chain of stages per row as their fixed part, which shrinks
// with the updates, and a smaller cost per pixel: the lean one the least, the
// less the wider the frame (its bands of 64 or 128 columns cover narrow frames
// badly); the generic one more, most where rows are not aligned for vectors.
// So the line is a number of windows for each pipeline, width and number of
// updates: just below where tiles become the slower pass. Measured (a TV call
// with its memset and stop-test launch, 22 sizes from 64 x 96 to 2049 x 2049, 40
// to 18000 windows), tiles / pipeline, us (windows):
//   lean: 1 update 17 x 256 x 256 8.4 / 8.7 (595), 26 x 256 x 256 10.7 / 10.1
//     (910), 4 x 1024 x 1024 16.5 / 11.5 (1976); 2 updates 5 x 512 x 512 13.3 /
//     16.3 (585), 9 x 384 x 384 16.3 / 15.9 (630), 4 x 1024 x 1024 26.7 / 20.6;
//     3 updates 26 x 256 x 256 20.1 / 20.9, 4 x 1024 x 1024 28.9 / 24.9; 4
//     updates 4 x 1024 x 1024 31.7 / 33.3, 24 x 512 x 512 41.1 / 45.2 (2808), 32
//     x 512 x 512 55.3 / 53.5 (3744), 128 x 256 x 256 59.4 / 60.8 (4480), 256 x
//     256 x 256 120 / 100 (8960), 16 x 1024 x 1024 104 / 74 (7904);
//   generic, rows aligned for vectors (a residual is asked for): 2 updates 2 x
//     1024 x 1024 18.4 / 20.5 (988), 4 x 1024 x 1024 28.0 / 24.8; 3 and 4
//     updates 16 x 1024 x 1024 99.8 / 106 and 110 / 129, an iteration of ADMM
//     with 24 such frames 273 / 261 (11856);
//   generic, other rows: 1 update 6 x 1023 x 1025 24.6 / 22.7 (2964); 4 updates
//     16 x 1001 x 1023 112 / 134 (7600), 32 x 1001 x 1023 211 / 203 (15200); of 4 k
//     + 2 columns 17 x 1508 x 1090 (12920), an iteration of a solve 211 / 242;
//   several passes, aligned: 30 steps of 22 x 1024 x 1024 1085 / 1235 (10868), of
//     36 x 1024 x 1024 9 steps 468 / 447 (17784).
#pragma once
#include <algorithm>
#include <cstdint>

namespace sci {
namespace tv {

// The large windows (64 columns x 48 rows, overlapping by 4 on each side).
constexpr int kWinCols = 64, kWinRows = 48, kWinHalo = 4;

inline int64_t rule_count(int64_t n, int64_t width) {
    const int64_t own = width - 2 * kWinHalo;
    return n <= width ? 1 : 1 + (n - width + own - 1) / own;
}

// The pipeline that would run the call instead: lean; generic with vector
// loads; generic with scalar loads, as tiles too; generic with scalar loads where
// tiles load pairs (rows of 4 k + 2 columns, wider than 512).
enum Pipeline { PIPE_LEAN = 0, PIPE_VECTOR = 1, PIPE_SCALAR = 2, PIPE_PAIRS = 3 };

// The most windows for `updates` dual updates in all, up to `most` a pass.
inline int64_t tile_line(Pipeline pipe, int64_t W, int updates, int most) {
    // one pass of 1, 2, 3, 4 updates, several passes; W <= 256, <= 512, wider
    static const int line[4][3][5] = {
        {{600, 605, 1290, 4500, 0}, {585, 585, 1330, 3400, 0}, {290, 580, 790, 2500, 0}},
        {{600, 1200, 4500, 5900, 11000}, {585, 4400, 14000, 14000, 14000}, {530, 990, 7950, 7950, 14000}},
        {{900, 1290, 3390, 5900, 7950}, {900, 2500, 4400, 6000, 14000}, {1330, 1490, 10900, 10900, 14000}},
        {{1850, 14000, 14000, 14000, 14000}, {1850, 14000, 14000, 14000, 14000}, {1850, 14000, 14000, 14000, 14000}}};
    const int w = W <= 256 ? 0 : W <= 512 ? 1 : 2;
    if (updates <= most) return line[pipe][w][updates - 1];
    // a last pass of one update, which wide aligned rows take better on the
    // pipeline, weighs when few others go before it (6 steps of 22 x 1024 x 1024:
    // tiles / pipeline 257 / 244 us; 10 steps of 24 such frames in a solve 468 /
    // 460 us an iteration)
    if (pipe == PIPE_VECTOR && w == 2 && updates % most == 1 && updates <= 2 * most + 1) return 7950;
    return line[pipe == PIPE_LEAN ? PIPE_VECTOR : pipe][w][4];
}

// Whether a call of `updates` dual updates, up to `most` a pass, runs on tiles.
inline bool tile_wins(Pipeline pipe, int64_t nf, int64_t H, int64_t W, int updates, int most) {
    const int64_t rows = rule_count(H, kWinRows), n = nf * rows * rule_count(W, kWinCols);
    // frames a little higher than a window leave most of the second one empty;
    // with few windows tiles still win (49 x 4097, 4 updates, tiles / pipeline:
    // 23 frames 45.5 / 45.6 us, 74 134 / 105)
    if (n > 3000 && 2 * rows * (kWinRows - 2 * kWinHalo) > 3 * H) return false;
    return n <= tile_line(pipe, W, updates, most);
}

// Whether a spectral solve of L bands runs its TV (1 to 4 updates) on tiles that
// apply the projection as they load x: that saves the projection kernel's pass
// too, so it pays for more windows. Measured, us an iteration with / without,
// 256 x 256 x 28 (980 windows): 1 update 15.9 / 16.1, 2 20.5 / 23.2, 4 23.8 /
// 28.0; 2 updates 512 x 512 x 28 (3276) 49.8 / 50.4, 700 x 700 x 8 (1872) 30.7 /
// 31.8, 300 x 700 x 28 (2912) 42.0 / 40.0. Rows the lean pass cannot take gain
// more: 511 x 513 x 28 (3640) 59.2 / 62.9.
inline bool spectral_tile_wins(int64_t L, int64_t H, int64_t W, int updates) {
    static const int line[3][4] = {{2100, 2100, 2100, 4500}, {3300, 3300, 3300, 3300}, {2500, 1900, 2500, 2500}};
    const int w = W <= 256 ? 0 : W <= 512 ? 1 : 2;
    const bool lean = W % (w == 2 ? 4 : 2) == 0;
    return L * rule_count(H, kWinRows) * rule_count(W, kWinCols) <= line[w][lean ? updates - 1 : 3];
}

}  // namespace tv
}  // namespace sci
