"""The plane-ring kernel at k = 5 (2-byte types, mul, 28 and 14 columns): forward and grad-x against the float64
oracle, at planes per pass that do and do not divide the channels, heights other than the width, and one sample of
many channels (the spatial filter changes within a CTA's share, or never)."""
import pytest
import torch

from tests.util import DTYPES, check_close, make_inputs, oracle_backward, oracle_forward

pytestmark = pytest.mark.gpu

# (B, C, H, W): 28 columns take two planes a pass where the channels are even, 14 columns up to nine
SHAPES = [(3, 64, 28, 28), (37, 5, 28, 28), (1, 300, 28, 28), (5, 64, 9, 28), (12, 48, 14, 14), (60, 6, 14, 14),
          (50, 7, 14, 14), (9, 64, 20, 14)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dt", ["f16", "bf16"])
def test_matches_oracle(shape, dt):
    from ddfnet_b200 import _lib, ddf
    B, C, H, W = shape
    x, cf, sf, go = make_inputs(B, C, H, W, 5, 1, DTYPES[dt], 70 + sum(shape))
    dev = torch.device("cuda:0")
    xd = x.to(dev).requires_grad_()
    out = ddf(xd, cf.to(dev), sf.to(dev), 5, 1, 1, "mul")
    check_close(out, oracle_forward(x, cf, sf, 5, 1, 1, "mul"), DTYPES[dt], f"forward {shape} {dt}")
    (gx,) = torch.autograd.grad(out, xd, go.to(dev))
    check_close(gx, oracle_backward(go, x, cf, sf, 5, 1, 1, "mul")[0], DTYPES[dt], f"grad_x {shape} {dt}")
    assert _lib.load().ddf_b200_take_fault() == 0


@pytest.mark.parametrize("shape", [(12, 64, 28, 28), (40, 48, 14, 14)])
def test_inputs_near_the_types_limit(shape):
    """x * sf leaves float's range, x * (cf * sf) does not: at most a few such values in a window, of one sign, so the
    results are held in the 2-norm (bfloat16's rounding of each: 2^-9)."""
    from ddfnet_b200 import ddf
    B, C, H, W = shape
    x, cf, sf, _ = make_inputs(B, C, H, W, 5, 1, torch.bfloat16, 7)
    x.view(-1)[::29] = -3.3e38
    cf, sf = (cf * 2.0 ** -8), (sf * 2.0 ** 4)
    dev = torch.device("cuda:0")
    out = ddf(x.to(dev), cf.to(dev), sf.to(dev), 5, 1, 1, "mul").cpu().double()
    want = oracle_forward(x, cf, sf, 5, 1, 1, "mul")
    assert torch.isfinite(want).all() and torch.isfinite(out).all()
    assert (out - want).norm() <= 4e-3 * want.norm()


@pytest.mark.parametrize("shape", [(12, 64, 28, 28), (40, 48, 14, 14)])
@pytest.mark.parametrize("large,small", [(3.0e38, 2.0 ** -100), (2.0 ** 55, 2.0 ** -100), (2.0 ** 20, 2.0 ** -118)])
def test_small_factors_of_a_large_filter(shape, large, small):
    """x * sf falls below float's range, x * (cf * sf) does not: held in the 2-norm as above.  Some planes have ordinary
    filters, some samples none that are large."""
    from ddfnet_b200 import ddf
    B, C, H, W = shape
    x, cf, sf, go = make_inputs(B, C, H, W, 5, 1, torch.bfloat16, 9)
    x, go, sf = x * small, go * small, sf * (2.0 ** -5 / large)
    cf = cf.clamp(-1, 1) * large
    cf[1::2, 1::3] = 0.25
    dev = torch.device("cuda:0")
    xd = x.to(dev).requires_grad_()
    out = ddf(xd, cf.to(dev), sf.to(dev), 5, 1, 1, "mul")
    (gx,) = torch.autograd.grad(out, xd, go.to(dev))
    for got, want in ((out, oracle_forward(x, cf, sf, 5, 1, 1, "mul")), (gx, oracle_backward(go, x, cf, sf, 5, 1, 1, "mul")[0])):
        got = got.detach().cpu().double()
        assert (got - want).norm() <= 4e-3 * want.norm()
