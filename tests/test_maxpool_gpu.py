"""The stem's max-pooling kernel against torch's, bit for bit: one pixel, odd sizes, ends of a thread's run of
outputs, one and several channel vectors, NaN and infinities."""
import pytest
import torch
import torch.nn.functional as F

from tests.util import DTYPES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 8, 1, 1), (2, 8, 2, 3), (1, 64, 7, 9), (3, 24, 15, 16), (2, 16, 17, 18), (2, 64, 112, 112)])
@pytest.mark.parametrize("dt", ["f32", "f16", "bf16"])
def test_matches_torch(shape, dt):
    from ddfnet_b200 import _lib
    from ddfnet_b200.nhwc import StemMaxPool
    g = torch.Generator().manual_seed(sum(shape))
    x = torch.randn(shape, generator=g).to(DTYPES[dt])
    flat = x.view(-1)
    flat[::29] = float("nan")
    flat[3::31] = float("inf")
    flat[5::7] = float("-inf")
    x = x.cuda().contiguous(memory_format=torch.channels_last)
    before = _lib.load().ddf_b200_launch_count()
    with torch.no_grad():
        got = StemMaxPool()(x)
    # a tensor that is contiguous in both layouts goes to torch
    assert _lib.load().ddf_b200_launch_count() - before == (0 if x.is_contiguous() else 1)
    want = F.max_pool2d(x, 3, 2, 1)
    assert got.shape == want.shape and got.is_contiguous(memory_format=torch.channels_last)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0))


def test_gradients_stay_with_torch():
    from ddfnet_b200.nhwc import StemMaxPool
    x = torch.randn(2, 16, 9, 9, device="cuda").contiguous(memory_format=torch.channels_last).requires_grad_()
    StemMaxPool()(x).sum().backward()
    assert x.grad is not None


def test_a_traced_pooling_runs_on_new_inputs():
    from ddfnet_b200.nhwc import StemMaxPool
    a, b = (torch.randn(2, 16, 9, 11, device="cuda").contiguous(memory_format=torch.channels_last) for _ in range(2))
    with torch.no_grad():
        traced = torch.jit.trace(StemMaxPool(), (a,), check_trace=False)
        assert torch.equal(traced(b), F.max_pool2d(b, 3, 2, 1))
