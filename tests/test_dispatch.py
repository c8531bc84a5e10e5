"""Which pipeline a TV call takes (sci_tv_rule.cuh), against measured times."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "sci-algorithms_gb300", "csrc")
# lean pass; generic, rows aligned for vectors; other rows; rows of 4 k + 2 columns
LEAN, VECTOR, SCALAR, PAIRS = 0, 1, 2, 3

# (pipeline, frames, H, W, dual updates, us on the row pipeline, us on tiles):
# for each pipeline, width and number of updates the largest call measured that
# tiles make faster by 4 % or more and the smallest that the pipeline does
MEASURED = [
    (LEAN, 70, 64, 96, 1, 8.2, 7.4),
    (LEAN, 100, 128, 128, 1, 10.3, 12.1),
    (LEAN, 8, 300, 500, 1, 8.7, 8.3),
    (LEAN, 9, 384, 384, 1, 8.9, 10.3),
    (LEAN, 1, 768, 768, 1, 8.2, 7.5),
    (LEAN, 3, 768, 768, 1, 8.9, 11.0),
    (LEAN, 67, 128, 128, 2, 18.3, 16.2),
    (LEAN, 225, 64, 96, 2, 20.6, 22.6),
    (LEAN, 5, 512, 512, 2, 16.3, 13.3),
    (LEAN, 12, 300, 500, 2, 16.5, 17.7),
    (LEAN, 2, 768, 768, 2, 15.3, 13.1),
    (LEAN, 3, 768, 768, 2, 16.1, 18.1),
    (LEAN, 100, 128, 128, 3, 24.0, 22.8),
    (LEAN, 475, 64, 96, 3, 35.4, 39.0),
    (LEAN, 19, 384, 384, 3, 24.7, 23.1),
    (LEAN, 26, 300, 500, 3, 26.8, 28.6),
    (LEAN, 2, 768, 768, 3, 18.6, 14.5),
    (LEAN, 5, 768, 768, 3, 22.3, 24.4),
    (LEAN, 378, 128, 128, 4, 63.6, 59.5),
    (LEAN, 171, 256, 256, 4, 74.0, 86.9),
    (LEAN, 29, 512, 512, 4, 51.5, 47.4),
    (LEAN, 62, 300, 500, 4, 59.8, 63.8),
    (LEAN, 4, 1024, 1024, 4, 33.3, 31.7),
    (LEAN, 3, 1080, 1920, 4, 39.0, 41.2),
    (VECTOR, 150, 64, 96, 1, 10.9, 8.3),
    (VECTOR, 26, 256, 256, 1, 11.2, 12.3),
    (VECTOR, 8, 300, 500, 1, 10.4, 9.6),
    (VECTOR, 12, 300, 500, 1, 11.0, 12.2),
    (VECTOR, 1, 1024, 1024, 1, 10.3, 8.5),
    (VECTOR, 3, 768, 768, 1, 10.3, 12.4),
    (VECTOR, 26, 256, 256, 2, 20.6, 18.6),
    (VECTOR, 650, 64, 96, 2, 44.1, 47.2),
    (VECTOR, 49, 384, 384, 2, 47.3, 45.2),
    (VECTOR, 62, 300, 500, 2, 55.6, 58.7),
    (VECTOR, 2, 1024, 1024, 2, 20.5, 18.4),
    (VECTOR, 5, 768, 768, 2, 22.1, 23.7),
    (VECTOR, 500, 128, 128, 3, 81.9, 77.2),
    (VECTOR, 1500, 64, 96, 3, 103.8, 117.1),
    (VECTOR, 200, 384, 384, 3, 187.6, 174.5),
    (VECTOR, 16, 1024, 1024, 3, 106.0, 99.8),
    (VECTOR, 22, 1024, 1024, 3, 126.7, 132.8),
    (VECTOR, 129, 256, 256, 4, 85.5, 70.2),
    (VECTOR, 1500, 64, 96, 4, 120.6, 125.5),
    (VECTOR, 200, 384, 384, 4, 205.7, 191.9),
    (VECTOR, 16, 1024, 1024, 4, 128.5, 110.0),
    (VECTOR, 22, 1024, 1024, 4, 138.8, 145.5),
    (VECTOR, 314, 256, 256, 5, 297.4, 275.7),
    (VECTOR, 3500, 64, 96, 5, 520.4, 567.6),
    (VECTOR, 200, 384, 384, 5, 376.1, 335.6),
    (VECTOR, 16, 1024, 1024, 5, 209.7, 196.8),
    (VECTOR, 22, 1024, 1024, 5, 244.3, 257.3),
    (VECTOR, 1222, 128, 128, 8, 494.9, 401.5),
    (VECTOR, 3500, 64, 96, 8, 608.5, 636.8),
    (VECTOR, 200, 384, 384, 8, 480.8, 390.4),
    (VECTOR, 28, 1024, 1024, 8, 416.2, 366.6),
    (VECTOR, 36, 1024, 1024, 8, 447.0, 468.3),
    (VECTOR, 2750, 64, 96, 29, 1932.5, 1724.4),
    (VECTOR, 200, 384, 384, 29, 1819.6, 1422.1),
    (VECTOR, 28, 1024, 1024, 29, 1528.0, 1346.2),
    (VECTOR, 36, 1024, 1024, 29, 1619.5, 1709.8),
    (SCALAR, 225, 65, 97, 1, 13.3, 10.4),
    (SCALAR, 108, 129, 129, 1, 12.5, 14.2),
    (SCALAR, 9, 385, 385, 1, 12.0, 10.3),
    (SCALAR, 37, 257, 257, 1, 12.4, 14.4),
    (SCALAR, 2, 1025, 1025, 1, 14.2, 12.4),
    (SCALAR, 3, 1025, 1025, 1, 14.4, 15.4),
    (SCALAR, 225, 65, 97, 2, 25.7, 22.6),
    (SCALAR, 650, 65, 97, 2, 43.8, 46.3),
    (SCALAR, 54, 257, 257, 2, 30.2, 28.7),
    (SCALAR, 62, 301, 501, 2, 43.3, 53.3),
    (SCALAR, 5, 769, 769, 2, 24.6, 23.5),
    (SCALAR, 2, 1081, 1921, 2, 26.7, 28.4),
    (SCALAR, 217, 129, 129, 3, 48.2, 39.9),
    (SCALAR, 850, 65, 97, 3, 60.9, 63.7),
    (SCALAR, 49, 385, 385, 3, 60.6, 48.9),
    (SCALAR, 114, 385, 385, 3, 88.8, 105.0),
    (SCALAR, 22, 1025, 1025, 3, 149.0, 135.1),
    (SCALAR, 375, 129, 129, 4, 74.9, 71.8),
    (SCALAR, 1500, 65, 97, 4, 110.8, 116.9),
    (SCALAR, 171, 257, 257, 4, 96.6, 90.5),
    (SCALAR, 114, 385, 385, 4, 105.8, 118.5),
    (SCALAR, 29, 769, 769, 4, 122.0, 116.7),
    (SCALAR, 15, 1081, 1921, 4, 189.6, 197.5),
    (SCALAR, 1500, 65, 97, 5, 352.0, 254.5),
    (SCALAR, 400, 257, 257, 5, 570.0, 379.6),
    (SCALAR, 50, 769, 769, 5, 434.8, 363.8),
    (SCALAR, 1500, 65, 97, 8, 301.1, 284.4),
    (SCALAR, 3500, 65, 97, 8, 634.8, 663.8),
    (SCALAR, 153, 301, 501, 8, 376.3, 339.4),
    (SCALAR, 50, 769, 769, 8, 476.6, 420.2),
    (SCALAR, 36, 1025, 1025, 8, 508.1, 530.0),
    (SCALAR, 1500, 65, 97, 29, 1245.7, 1056.6),
    (SCALAR, 400, 257, 257, 29, 1824.0, 1652.7),
    (SCALAR, 50, 769, 769, 29, 1759.8, 1586.3),
    (SCALAR, 36, 1025, 1025, 29, 1900.5, 2004.2),
]

MAIN = r"""
#include <cstdio>
#include "sci_tv_rule.cuh"
int main() {
    int pipe, updates;
    long long nf, H, W;
    while (std::scanf("%d %lld %lld %lld %d", &pipe, &nf, &H, &W, &updates) == 5)
        std::printf("%d\n", (int)(pipe < 0
            ? sci::tv::spectral_tile_wins(nf, H, W, updates)
            : sci::tv::tile_wins((sci::tv::Pipeline)pipe, nf, H, W, updates, 4)));
}
"""


@pytest.fixture(scope="module")
def decide(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("rule")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run([cxx, "-std=c++17", "-I" + CSRC, str(d / "main.cpp"), "-o", str(d / "main")],
                   check=True)

    def f(calls):
        text = "".join("%d %d %d %d %d\n" % c for c in calls)
        out = subprocess.run([str(d / "main")], input=text, capture_output=True, text=True,
                             check=True).stdout.split()
        return [o == "1" for o in out]
    return f


def test_calls_near_the_lines_take_the_faster_pass(decide):
    tiles = decide([m[:5] for m in MEASURED])
    for m, on_tiles in zip(MEASURED, tiles):
        assert on_tiles == (m[6] < m[5]), m


# Calls that ran slower on tiles than on the pipeline they had taken before
# (a residual, odd rows, one to three updates; several passes within a solve).
@pytest.mark.parametrize("pipe,nf,H,W,updates", [
    (LEAN, 4, 1024, 1024, 1), (LEAN, 4, 1024, 1024, 2), (LEAN, 40, 300, 300, 1),
    (LEAN, 40, 300, 300, 2), (LEAN, 10, 512, 512, 1), (LEAN, 10, 512, 512, 2),
    (LEAN, 200, 128, 128, 1), (LEAN, 200, 128, 128, 2), (LEAN, 24, 256, 256, 1),
    (LEAN, 20, 511, 300, 2), (VECTOR, 24, 1024, 1024, 2), (VECTOR, 24, 1024, 1024, 4),
    (VECTOR, 8, 1080, 1920, 2), (VECTOR, 24, 1024, 1024, 9),
    (SCALAR, 6, 1023, 1025, 1), (SCALAR, 5, 2047, 2049, 1), (SCALAR, 30, 49, 4097, 3)])
def test_calls_that_tiles_slowed_down(decide, pipe, nf, H, W, updates):
    assert decide([(pipe, nf, H, W, updates)]) == [False]


# Rows that tiles load in pairs and the pipeline one by one: tiles to the end of
# the range measured (us on the row pipeline, on tiles).
@pytest.mark.parametrize("nf,H,W,updates,pipe_us,tile_us", [
    (17, 1508, 1090, 4, 241.6, 211.2),
    (28, 1024, 1026, 3, 182.9, 152.8),
    (28, 1024, 1026, 4, 190.0, 170.6),
    (28, 1024, 1026, 8, 469.2, 368.1),
    (28, 1024, 1026, 19, 1244.8, 954.6),
    (18, 1508, 1090, 3, 186.4, 151.3),
    (18, 1508, 1090, 4, 192.8, 168.6),
    (18, 1508, 1090, 8, 475.8, 365.2),
    (18, 1508, 1090, 19, 1260.9, 947.1),
    (1, 1080, 1922, 1, 14.3, 11.4),
    (1, 1080, 1922, 2, 23.8, 17.9)])
def test_rows_of_pairs_stay_on_tiles(decide, nf, H, W, updates, pipe_us, tile_us):
    assert tile_us < pipe_us
    assert decide([(PAIRS, nf, H, W, updates)]) == [True]


# Spectral solves, projection on load or not: (bands, H, W, updates, us an
# iteration without, with).
@pytest.mark.parametrize("L,H,W,updates,apart,fused", [
    (28, 256, 256, 1, 16.1, 15.9), (28, 256, 256, 2, 23.2, 20.5), (28, 256, 256, 4, 28.0, 23.8),
    (20, 511, 300, 2, 27.7, 27.5), (16, 512, 512, 3, 40.7, 33.8), (16, 511, 513, 2, 46.8, 37.3),
    (8, 512, 800, 4, 37.4, 31.9), (28, 300, 700, 2, 40.0, 42.0), (28, 512, 800, 2, 67.8, 76.1)])
def test_spectral_solves_take_the_faster_form(decide, L, H, W, updates, apart, fused):
    assert decide([(-1, L, H, W, updates)]) == [fused < apart]
