"""The band kernel's forward and grad-x where a thread has two channels of a unit (many units per CTA), one (few), or
two with the filters read from shared memory (k = 5): channel counts that leave the last unit without its second
channel, the split that spreads few planes over more CTAs, and inputs near bfloat16's limit."""
import pytest
import torch

from tests.util import DTYPES, check_close, make_inputs, oracle_backward, oracle_forward

pytestmark = pytest.mark.gpu

# (B, C, H, W, k, d, s)
SHAPES = [(8, 131, 50, 67, 3, 1, 1), (7, 259, 40, 70, 3, 2, 1), (17, 75, 100, 75, 3, 1, 2),    # two
          (1, 43, 50, 67, 3, 1, 1), (1, 37, 14, 13, 3, 1, 1), (3, 11, 7, 9, 3, 2, 1),            # one
          (2, 37, 50, 67, 5, 1, 1), (1, 5, 14, 13, 5, 2, 1)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("mode", ["mul", "add"])
def test_matches_oracle(shape, dt, mode):
    from ddfnet_b200 import _lib, ddf
    B, C, H, W, k, d, s = shape
    x, cf, sf, go = make_inputs(B, C, H, W, k, s, DTYPES[dt], 80 + sum(shape))
    dev = torch.device("cuda:0")
    xd = x.to(dev).requires_grad_()
    out = ddf(xd, cf.to(dev), sf.to(dev), k, d, s, mode)
    check_close(out, oracle_forward(x, cf, sf, k, d, s, mode), DTYPES[dt], f"forward {shape} {dt} {mode}")
    (gx,) = torch.autograd.grad(out, xd, go.to(dev))
    check_close(gx, oracle_backward(go, x, cf, sf, k, d, s, mode)[0], DTYPES[dt], f"grad_x {shape} {dt} {mode}")
    assert _lib.load().ddf_b200_take_fault() == 0


@pytest.mark.parametrize("shape", [SHAPES[0], SHAPES[3], SHAPES[6]])
def test_inputs_near_the_types_limit(shape):
    """x * sf leaves float's range, x * (cf * sf) does not; see the same test of the plane-ring kernel."""
    from ddfnet_b200 import ddf
    B, C, H, W, k, d, s = shape
    x, cf, sf, _ = make_inputs(B, C, H, W, k, s, torch.bfloat16, 8)
    x.view(-1)[::29] = -3.3e38
    cf, sf = (cf * 2.0 ** -8), (sf * 2.0 ** 4)
    dev = torch.device("cuda:0")
    out = ddf(x.to(dev), cf.to(dev), sf.to(dev), k, d, s, "mul").cpu().double()
    want = oracle_forward(x, cf, sf, k, d, s, "mul")
    assert torch.isfinite(want).all() and torch.isfinite(out).all()
    assert (out - want).norm() <= 4e-3 * want.norm()


@pytest.mark.parametrize("shape", [SHAPES[0], SHAPES[3], SHAPES[4], SHAPES[6]])
@pytest.mark.parametrize("large,small", [(2.0 ** 55, 2.0 ** -100), (2.0 ** 20, 2.0 ** -118)])
def test_small_factors_of_a_large_filter(shape, large, small):
    """x * sf falls below float's range, x * (cf * sf) does not: held in the 2-norm as above.  Some channels have ordinary
    filters, some samples none that are large."""
    from ddfnet_b200 import ddf
    B, C, H, W, k, d, s = shape
    x, cf, sf, go = make_inputs(B, C, H, W, k, s, torch.bfloat16, 9)
    x, go, sf = x * small, go * small, sf * (2.0 ** -5 / large)
    cf = cf * large
    cf[1::2, 1::3] = 0.25
    dev = torch.device("cuda:0")
    xd = x.to(dev).requires_grad_()
    out = ddf(xd, cf.to(dev), sf.to(dev), k, d, s, "mul")
    (gx,) = torch.autograd.grad(out, xd, go.to(dev))
    for got, want in ((out, oracle_forward(x, cf, sf, k, d, s, "mul")), (gx, oracle_backward(go, x, cf, sf, k, d, s, "mul")[0])):
        got = got.detach().cpu().double()
        assert (got - want).norm() <= 4e-3 * want.norm()


# (B, C, H, W, k, d, s), normalised in the kernel: at k = 5 straight into registers (few units a CTA) and by way of shared memory
@pytest.mark.parametrize("shape", [(2, 37, 50, 67, 5, 1, 1), (3, 160, 50, 67, 5, 2, 1), (1, 43, 50, 67, 3, 1, 1), (6, 75, 50, 37, 3, 1, 2)])
@pytest.mark.parametrize("dt", ["f32", "f16"])
@pytest.mark.parametrize("mode", ["mul", "add"])
def test_filters_normalised_in_the_kernel(shape, dt, mode):
    """The last sample's channel filters are beyond what products with padding zeros may meet: tap by tap there."""
    from ddfnet_b200.op import ddf_sfnorm, spatial_filter_norm
    B, C, H, W, k, d, s = shape
    x, cf, raw, _ = make_inputs(B, C, H, W, k, s, DTYPES[dt], 50 + sum(shape))
    raw = raw + 0.4
    big = dt == "f32" and mode == "mul"
    if big:
        cf[-1, 0] = 2e18
    dev = torch.device("cuda:0")
    out = ddf_sfnorm(x.to(dev), cf.to(dev), raw.to(dev), k, d, s, mode, 0.7).cpu()
    want = oracle_forward(x, cf, spatial_filter_norm(raw.double(), k, 0.7), k, d, s, mode)
    if big:
        got = out[-1, 0].double()
        assert (got - want[-1, 0]).norm() <= 1e-6 * want[-1, 0].norm()
        out[-1, 0], want[-1, 0] = 0.0, 0.0
    check_close(out, want, DTYPES[dt], f"sfnorm {shape} {dt} {mode}")


@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_many_units_at_k5(dt):
    """2-byte mul by way of shared memory: more than fifty units of a channel per SM."""
    from ddfnet_b200 import ddf
    x, cf, sf = make_inputs(2, 960, 200, 19, 5, 1, DTYPES[dt], 51, with_go=False)
    dev = torch.device("cuda:0")
    out = ddf(x.to(dev), cf.to(dev), sf.to(dev), 5, 1, 1, "mul")
    check_close(out, oracle_forward(x, cf, sf, 5, 1, 1, "mul"), DTYPES[dt], f"forward {dt}")
