"""Tiles of the channels_last forward against the float64 oracle: rows of several tiles and a narrower last one, tiles of
fewer rows at the bottom, more tiles than CTAs (both buffers used many times, samples changing on the way), one
column or row, every channel count's columns per tile; planar and channels_last filters."""
import pytest
import torch

from tests.util import DTYPES, check_close, make_inputs, oracle_forward

pytestmark = pytest.mark.gpu

# B, C, H, W, stride
SHAPES = [(2, 64, 13, 57, 1), (70, 64, 57, 45, 1), (9, 128, 30, 30, 2), (3, 8, 9, 300, 1), (2, 16, 5, 129, 1), (40, 32, 17, 70, 2),
          (3, 512, 7, 5, 1), (1, 2048, 3, 5, 1), (2, 1024, 9, 6, 2), (5, 64, 1, 31, 1), (5, 64, 31, 1, 1), (400, 64, 6, 4, 1)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("mode", ["mul", "add"])
def test_matches_oracle(shape, dt, mode):
    from ddfnet_b200.nhwc import ddf_nhwc
    B, C, H, W, s = shape
    x, cf, sf = make_inputs(B, C, H, W, 3, s, DTYPES[dt], seed=40 + sum(shape), with_go=False)
    dev = torch.device("cuda:0")
    xd, cfd = x.to(dev).contiguous(memory_format=torch.channels_last), cf.to(dev)
    want = oracle_forward(x, cf, sf, 3, 1, s, mode)
    check_close(ddf_nhwc(xd, cfd, sf.to(dev), 3, 1, s, mode), want, DTYPES[dt], f"planar {shape} {dt} {mode}")
    sf16 = torch.full((B, 16, H // s, W // s), float("nan"), dtype=DTYPES[dt])   # the maps behind the nine must be ignored
    sf16[:, :9] = sf
    sf16 = sf16.to(dev).contiguous(memory_format=torch.channels_last)
    check_close(ddf_nhwc(xd, cfd, sf16, 3, 1, s, mode), want, DTYPES[dt], f"channels_last {shape} {dt} {mode}")


@pytest.mark.parametrize("hw", [(1, 1), (1, 3), (5, 1), (7, 7), (27, 29), (28, 28), (57, 55)])
@pytest.mark.parametrize("C", [8, 256, 2048])
def test_pooled_partials(hw, C):
    """Tiles of a quarter of the image below 784 pixels, of 196 from there on."""
    from ddfnet_b200.nhwc import pool_partials
    x = torch.randn(3, C, *hw, generator=torch.Generator().manual_seed(4)).to(torch.float16)
    p = pool_partials(x.to("cuda:0").contiguous(memory_format=torch.channels_last))
    n = hw[0] * hw[1]
    tile = (n + 3) // 4 if n < 784 else 196
    assert p.shape == (3, (n + tile - 1) // tile, C)
    pixels = x.double().flatten(2).split(tile, 2)
    want = torch.stack([t.sum(2) for t in pixels], 1)
    # a chain of at most 196 float sums of values below 6: 196 * 2^-24 * 196 * 6 would be the worst case
    assert torch.allclose(p.cpu().double(), want, rtol=0, atol=1.5e-2 * tile / 196 + 1e-6)
