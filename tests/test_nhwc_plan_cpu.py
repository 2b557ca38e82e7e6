"""Host arithmetic of the channels_last forward (nhwc_plan.h), compiled with the host compiler: where the bulk copies of
the raw filters end, and which problems have tiles."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ddfnet_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "nhwc_plan.h"
using namespace ddf;
// argv: OH OW columns of a tile, pixel stride, batch stride, sample -> elements from the first to behind the last one copied
int main(int, char** v) {
    NhwcPlan pl = {};
    pl.OH = atoi(v[1]); pl.OW = atoi(v[2]); pl.cols = atoi(v[3]);
    pl.sf_pixel_stride = atoll(v[4]); pl.sf_batch_stride = atoll(v[5]);
    const int b = atoi(v[6]);
    long long lo = 1ll << 60, hi = -lo;
    for (int y = 0; y < pl.OH; ++y)
        for (int x = 0; x < pl.OW; x += pl.cols) {
            const NhwcRun r = nhwc_filter_run(pl, b, y, x, pl.OW - x < pl.cols ? pl.OW - x : pl.cols);
            if (r.bytes % 16 != 0 || r.from % 8 != 0) return 1;
            if (r.from < lo) lo = r.from;
            if (r.from + r.bytes / 2 > hi) hi = r.from + r.bytes / 2;
        }
    printf("%lld %lld\n", lo, hi);
}
"""


TILES = r"""
#include <initializer_list>
#include <cstdio>
#include <cstdlib>
#include "nhwc_plan.h"
using namespace ddf;
// argv: C stride -> the problems of every width up to 600 without tiles, or whose layout is unsound
int main(int, char** v) {
    int bad = 0, n = 0;
    for (int s = atoi(v[2]), ow = 1; ow <= 600; ++ow)
        for (int oh : {1, 2, 5, 8, 56})
            for (int pixel : {32, 80})
                for (int bulk = 0; bulk <= 64; bulk += bulk ? 8 : 16) {
                    NhwcPlan pl = {};
                    pl.B = 3; pl.C = atoi(v[1]); pl.vecs = pl.C / 8;
                    pl.OH = oh; pl.OW = ow; pl.H = oh * s; pl.W = ow * s;
                    pl.sf_bulk = bulk > 0; pl.sf_pixel_stride = bulk;
                    const uint32_t smem = nhwc_tiles(pl, s, (uint32_t)pixel, 148);
                    const int cols = (pl.cols - 1) * s + 3, rows = (pl.rows - 1) * s + 3;   // of a tile's window
                    ++n;
                    bad += !(smem > 0 && smem <= kNhwcSmem && pl.cols >= 1 && pl.cols * pl.vecs <= kNhwcThreads &&
                             pl.rows >= 1 && pl.rows <= kNhwcRows && pl.tiles == 3 * pl.tiles_x * pl.tiles_y &&
                             pl.cols * pl.tiles_x >= ow && pl.cols * (pl.tiles_x - 1) < ow &&
                             pl.rows * pl.tiles_y >= oh && pl.rows * (pl.tiles_y - 1) < oh &&
                             pl.row_bytes >= (uint32_t)(cols * pl.C * 2) && pl.off_raw >= (uint32_t)rows * pl.row_bytes &&
                             pl.sf_stride >= (uint32_t)(pl.cols * (pl.rows * pixel + 16)) && pl.off_affine >= 64 + 2 * pl.sf_stride &&
                             pl.off_buf >= pl.off_affine + 8u * pl.C &&
                             pl.buf_stride >= pl.off_raw + (uint32_t)(pl.rows * pl.cols * bulk) * 2u &&
                             smem >= pl.off_buf + 2u * pl.buf_stride && pl.off_buf % 128 == 0 && pl.buf_stride % 128 == 0);
                }
    printf("%d %d\n", bad, n);
}
"""


@pytest.fixture(scope="module")
def compiled(tmp_path_factory):
    def build(text):
        d = tmp_path_factory.mktemp("nhwc_plan")
        (d / "main.cpp").write_text(text)
        subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wno-sign-compare", "-Werror", f"-I{CSRC}", str(d / "main.cpp"), "-o", str(d / "main")],
                       check=True)
        return lambda *args: [int(n) for n in subprocess.run([str(d / "main"), *map(str, args)], check=True, capture_output=True,
                                                             text=True).stdout.split()]
    return build


@pytest.fixture(scope="module")
def program(compiled):
    return compiled(PROGRAM)


@pytest.fixture(scope="module")
def tiles(compiled):
    return compiled(TILES)


@pytest.mark.parametrize("stride", [1, 2])
@pytest.mark.parametrize("C", [8 << i for i in range(9)])
def test_every_width_has_tiles_that_fit(tiles, C, stride):
    bad, n = tiles(C, stride)
    assert bad == 0 and n == 600 * 5 * 2 * 8


@pytest.mark.parametrize("oh,ow,cols", [(1, 1, 1), (5, 7, 7), (3, 9, 4), (4, 8, 3)])
@pytest.mark.parametrize("pixel", [16, 24, 64])
def test_filter_copies_end_with_the_last_pixels_values(program, oh, ow, cols, pixel):
    """One filter map for three samples, one map behind the other, interleaved, and the last sample first."""
    n = oh * ow * pixel
    for batch in (0, n, 16, -n):
        for b in range(3):
            lo, hi = program(oh, ow, cols, pixel, batch, b)
            first = b * batch
            assert lo == first
            assert hi <= first + (oh * ow - 1) * pixel + 9
