"""Host arithmetic of the channels_last forward (nhwc_plan.h), compiled with the host compiler: where the bulk copies of
the raw filters end."""
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


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("nhwc_plan")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    return lambda *args: [int(n) for n in subprocess.run([str(d / "main"), *map(str, args)], check=True, capture_output=True,
                                                         text=True).stdout.split()]


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
