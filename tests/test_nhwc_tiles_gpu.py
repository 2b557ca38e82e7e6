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


@pytest.mark.parametrize("mode", ["mul", "add"])
def test_one_filter_map_for_all_samples(mode):
    """sf_batch_stride 0: what lies behind the map's last value belongs to no sample and must not matter."""
    from ddfnet_b200 import _lib
    B, C, H, W, g = 3, 64, 9, 20, 24
    x, cf, sf = make_inputs(1, C, H, W, 3, 1, torch.float16, seed=77, with_go=False)
    x, cf = (torch.cat([t * (i + 1) for i in range(B)]) for t in (x, cf))
    dev = torch.device("cuda:0")
    xd = x.to(dev).contiguous(memory_format=torch.channels_last)
    maps = torch.full((H, W, g), float("nan"), dtype=torch.float16)
    maps[..., :9] = sf[0].permute(1, 2, 0)
    buf = torch.full((H * W * g + 512,), float("nan"), dtype=torch.float16)
    buf[: (H * W - 1) * g + 9] = maps.flatten()[: (H * W - 1) * g + 9]
    buf, cfd = buf.to(dev), cf.to(dev)
    out = torch.empty_like(xd)
    rc = _lib.load().ddf_b200_forward_nhwc(xd.data_ptr(), cfd.data_ptr(), buf.data_ptr(), None, out.data_ptr(), None, None, 0, B,
                                           C, H, W, 3, 1, 1, {"mul": 0, "add": 1}[mode], 1, 0, g, 1, 0, 1.0,
                                           torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    check_close(out, oracle_forward(x, cf, sf.expand(B, -1, -1, -1), 3, 1, 1, mode), torch.float16, f"shared filter {mode}")


# B, H, W, stride, maps of the spatial filter: widths at which a row of 256 columns does not fit a CTA's shared memory
@pytest.mark.parametrize("shape", [(1, 6, 512, 2, 16), (3, 9, 1022, 2, 16), (2, 5, 480, 2, 32), (1, 3, 256, 1, 48), (1, 4, 333, 1, 64)])
@pytest.mark.parametrize("mode", ["mul", "add"])
def test_wide_rows_of_eight_channels(shape, mode):
    from ddfnet_b200.nhwc import ddf_nhwc
    B, H, W, s, g = shape
    x, cf, sf = make_inputs(B, 8, H, W, 3, s, torch.float16, seed=sum(shape), with_go=False)
    dev = torch.device("cuda:0")
    maps = torch.full((B, g, H // s, W // s), float("nan"), dtype=torch.float16)
    maps[:, :9] = sf
    out = ddf_nhwc(x.to(dev).contiguous(memory_format=torch.channels_last), cf.to(dev),
                   maps.to(dev).contiguous(memory_format=torch.channels_last), 3, 1, s, mode)
    check_close(out, oracle_forward(x, cf, sf, 3, 1, s, mode), torch.float16, f"{shape} {mode}")


@pytest.mark.parametrize("starve", [1, 2, 3])
def test_a_wait_that_runs_out(starve):
    """The CTAs leave together: tiles before the one that never completes are whole, no other element is written, and
    the context stays usable."""
    from ddfnet_b200 import _lib
    L = _lib.load()
    B, C, H, W, g = 64, 256, 56, 56, 16   # 56 rows in tiles of at most 8 by 8: more than three a CTA
    x, cf, sf = make_inputs(2, C, H, W, 3, 1, torch.float16, seed=78, with_go=False)
    dev = torch.device("cuda:0")
    xd = x.to(dev).repeat(B // 2, 1, 1, 1).contiguous(memory_format=torch.channels_last)
    cfd = cf.to(dev).repeat(B // 2, 1, 1, 1)
    maps = torch.zeros(B, H, W, g, dtype=torch.float16, device=dev)
    maps[..., :9] = sf.to(dev).permute(0, 2, 3, 1).repeat(B // 2, 1, 1, 1)
    out = torch.full_like(xd, float("nan"))

    def call(limit, starve):
        return L.ddf_b200_nhwc_waitlimit(xd.data_ptr(), cfd.data_ptr(), maps.data_ptr(), out.data_ptr(), B, C, H, W, 3, 1, 1,
                                         _lib.MUL, 1, H * W * g, g, 1, limit, starve, torch.cuda.current_stream().cuda_stream)

    assert L.ddf_b200_take_fault() == 0
    assert call(2_000_000, starve) == 0
    assert L.ddf_b200_take_fault() == 1
    assert L.ddf_b200_take_fault() == 0
    left = out.clone()
    assert call(2_000_000_000, 0) == 0
    assert L.ddf_b200_take_fault() == 0
    check_close(out[:2], oracle_forward(x, cf, sf, 3, 1, 1, "mul"), torch.float16, "after a starved launch")
    written = ~left.isnan()
    assert torch.equal(left[written], out[written])
    assert torch.equal(written, written[:, :1].expand_as(written))   # whole pixels
    share = written.float().mean().item()
    assert (share == 0) if starve == 1 else 0 < share < 1
