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


def _gradients(ts, go, **kw):
    out = _entry(False)(*ts)
    return torch.autograd.grad(out, ts, go, **kw)


def test_backward_on_another_stream_and_in_two_threads():
    import threading
    B, C, H, W = SHAPE
    sets = [_inputs(20 + i, "f16", grad=True) for i in range(2)]
    want = [_gradients(s[:3], s[3]) for s in sets]
    torch.cuda.synchronize()
    got, errors = [None, None], []

    def work(i):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for _ in range(50):
                    got[i] = _gradients(sets[i][:3], sets[i][3])
            stream.synchronize()
        except Exception as e:  # a thread's exception would be lost
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for g, w in zip(got, want):
        assert all(torch.equal(a, b) for a, b in zip(g, w))


def test_gradients_have_their_inputs_types():
    x, cf, sf, go = _inputs(7)
    ts = [x.half().requires_grad_(), cf.requires_grad_(), sf.half().requires_grad_()]
    out = _entry(False)(*ts)
    assert out.dtype == torch.float32
    got = torch.autograd.grad(out, ts, go)
    want = _gradients([t.detach().float().requires_grad_() for t in ts], go)
    for g, t, w in zip(got, ts, want):
        assert g.dtype == t.dtype and torch.equal(g, w.to(t.dtype))


@pytest.mark.parametrize("need", [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1)])
def test_only_the_gradients_that_are_asked_for(need):
    ts = _inputs(8)
    full = _gradients([t.detach().requires_grad_() for t in ts[:3]], ts[3])
    some = [t.detach().requires_grad_(bool(n)) for t, n in zip(ts[:3], need)]
    _entry(False)(*some).backward(ts[3])
    for t, n, f in zip(some, need, full):
        assert (t.grad is None) == (not n) and (not n or torch.equal(t.grad, f))


def test_saved_tensors_pass_through_hooks():
    ts = _inputs(9, grad=True)
    want, packed = _gradients(ts[:3], ts[3]), []

    def pack(t):
        packed.append(t.shape)
        return t.cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        out = _entry(False)(*ts[:3])
    assert len(packed) == 3
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(out, ts[:3], ts[3]), want))


def test_changed_inputs_and_a_second_backward_are_noticed():
    ts = _inputs(10, grad=True)
    out = _entry(False)(*ts[:3])
    with torch.no_grad():
        ts[1].mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.sum().backward()
    out = _entry(False)(*ts[:3])
    out.sum().backward()
    with pytest.raises(RuntimeError, match="second time"):
        out.sum().backward()


def test_no_history_without_a_gradient_to_record():
    ts = _inputs(11, grad=True)
    with torch.no_grad():
        assert not _entry(False)(*ts[:3]).requires_grad
    with torch.inference_mode():
        assert _entry(False)(*ts[:3]).is_inference()
    assert not _entry(False)(*(t.detach() for t in ts[:3])).requires_grad
