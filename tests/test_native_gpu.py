"""The operator's C++ host path (csrc/native.cpp) at its seams with torch: what it hands to the autograd
functions of op.py, and what it has to do itself that torch.autograd.Function did."""
import pytest
import torch

from tests.util import DTYPES, make_inputs

pytestmark = pytest.mark.gpu

SHAPE = (2, 8, 9, 11)


def _inputs(seed, dt="f32", grad=False):
    B, C, H, W = SHAPE
    ts = [t.cuda() for t in make_inputs(B, C, H, W, 3, 1, DTYPES[dt], seed)]
    for t in ts[:3]:
        t.requires_grad_(grad)
    return ts


def _entry(fused):
    from ddfnet_b200 import ddf, ddf_sfnorm
    if fused:
        return lambda x, cf, sf: ddf_sfnorm(x, cf, sf, 3, 1, 1, "mul", 0.5)
    return lambda x, cf, sf: ddf(x, cf, sf, 3, 1, 1, "mul")


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("grad", [False, True])
def test_a_traced_call_runs_on_new_inputs(fused, grad):
    f = _entry(fused)
    a, b = _inputs(1, grad=grad)[:3], _inputs(2, grad=grad)[:3]
    traced = torch.jit.trace(lambda x, cf, sf: f(x, cf, sf) + 1, tuple(a), check_trace=False)
    assert torch.equal(traced(*b), f(*b) + 1)
    assert not torch.equal(traced(*a), traced(*b))


def test_the_autograd_functions_are_autograd_functions():
    from ddfnet_b200 import DDFFunction, DDFSpatialNormFunction, ddf
    a = _inputs(3)[:3]
    assert issubclass(DDFFunction, torch.autograd.Function) and issubclass(DDFSpatialNormFunction, torch.autograd.Function)
    assert torch.equal(DDFFunction.apply(*a), ddf(*a))

    class Doubled(DDFFunction):
        @staticmethod
        def forward(ctx, *args):
            return DDFFunction.forward(ctx, *args) * 2

    assert torch.equal(Doubled.apply(*a, 3, 1, 1, "mul"), 2 * ddf(*a))


def test_transforms_are_refused_as_for_any_autograd_function():
    from torch.autograd import forward_ad
    f = _entry(False)
    a = _inputs(4)[:3]
    with pytest.raises(RuntimeError, match="setup_context"):
        torch.func.vmap(f)(*(torch.stack((t, t)) for t in a))
    with pytest.raises(RuntimeError, match="setup_context"):
        torch.func.grad(lambda x: f(x, *a[1:]).sum())(a[0])
    with forward_ad.dual_level(), pytest.raises(RuntimeError):
        f(forward_ad.make_dual(a[0], torch.ones_like(a[0])), *a[1:])


@pytest.mark.parametrize("fused", [False, True])
def test_a_gradient_that_does_not_arrive_is_zero(fused):
    class Drop(torch.autograd.Function):
        @staticmethod
        def forward(ctx, y):
            return y.clone()

        @staticmethod
        def backward(ctx, g):
            return None

    ts = _inputs(5, grad=True)[:3]
    Drop.apply(_entry(fused)(*ts)).sum().backward()
    assert all(t.grad is not None and not t.grad.any() for t in ts)


@pytest.mark.parametrize("fused,name", [(False, "DDFFunction"), (True, "DDFSpatialNormFunction")])
def test_a_profiler_shows_the_call_and_its_backward(fused, name):
    ts = _inputs(6, grad=True)[:3]
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        _entry(fused)(*ts).sum().backward()
    seen = {e.key for e in prof.key_averages()}
    assert {name, name + "Backward"} <= seen
