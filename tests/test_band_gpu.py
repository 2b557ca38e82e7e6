"""The band kernels (planes of any height and width): forward and the three gradients against the float64
oracle at the edges of their ranges -- one row, one column, widths around a warp and at the widest band,
a last band of one row, channel counts that the planes of a pass do not divide, H and W that the stride
does not divide -- and non-finite values next to the padding."""
import pytest
import torch

from tests.util import DTYPES, check_close, check_extremes, make_inputs, oracle_backward, oracle_forward

pytestmark = pytest.mark.gpu

# (B, C, H, W, k, d, s)
SHAPES = [
    (1, 3, 1, 9, 3, 1, 1), (2, 5, 9, 1, 3, 1, 1), (1, 300, 5, 7, 3, 1, 1), (3, 37, 9, 11, 3, 2, 1),
    (2, 19, 5, 33, 5, 1, 1), (2, 7, 13, 31, 5, 2, 1), (1, 9, 7, 11, 3, 1, 2), (2, 33, 15, 29, 3, 1, 2),
    (1, 8, 201, 320, 3, 1, 1),   # the widest band, a last band of one row
    (1, 8, 200, 321, 3, 1, 1),   # wider: the generic kernels
    (2, 5, 33, 200, 3, 2, 1), (1, 5, 19, 299, 5, 2, 1),   # dilated, too wide for both residues in a band
    (1, 3, 9, 320, 3, 2, 1),     # ... and a band beyond the plane's last row
    # k = 5: the widest band of the filter gradients and of the other two, and one column more
    (1, 3, 9, 320, 5, 1, 1), (1, 3, 9, 321, 5, 2, 1), (1, 3, 13, 352, 5, 1, 1), (1, 3, 9, 353, 5, 1, 1),
    (1, 3, 11, 640, 3, 1, 2), (1, 3, 10, 641, 3, 1, 2), (1, 3, 11, 642, 3, 1, 2),   # the widest at stride 2, and wider
    (1, 70, 101, 75, 3, 2, 1), (3, 67, 50, 67, 3, 1, 1), (2, 131, 101, 75, 3, 1, 2), (1, 24, 61, 99, 5, 1, 1),
    (1, 24, 63, 101, 5, 2, 1), (1, 40, 30, 167, 5, 2, 1), (40, 75, 17, 13, 3, 1, 1),
    # both sides of where the forward and grad-x leave small planes to the generic kernels: pixels of a plane, one
    # column and few or many planes, samples and work in each
    (3, 50, 2, 4, 3, 1, 1), (3, 50, 3, 3, 3, 1, 1), (3, 20, 33, 1, 5, 1, 1), (40, 400, 33, 1, 5, 1, 1),
    (600, 10, 5, 3, 3, 2, 1), (600, 11, 5, 3, 3, 2, 1), (592, 3, 7, 6, 5, 1, 1), (593, 3, 7, 6, 5, 1, 1),
]


def _inputs(shape, dt, seed):
    B, C, H, W, k, d, s = shape
    dev = torch.device("cuda:0")
    cpu = make_inputs(B, C, H, W, k, s, DTYPES[dt], seed)
    return cpu, [t.to(dev) for t in cpu]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("mode", ["mul", "add"])
def test_matches_oracle(shape, dt, mode):
    from ddfnet_b200 import _lib, ddf
    k, d, s = shape[4:]
    (x, cf, sf, go), dev = _inputs(shape, dt, 50 + sum(shape))
    ts = [t.requires_grad_() for t in dev[:3]]
    out = ddf(*ts, k, d, s, mode)
    check_close(out, oracle_forward(x, cf, sf, k, d, s, mode), DTYPES[dt], f"forward {shape} {dt} {mode}")
    got = torch.autograd.grad(out, ts, dev[3])
    want = oracle_backward(go, x, cf, sf, k, d, s, mode)
    for name, g, w in zip(("grad_x", "grad_cf", "grad_sf"), got, want):
        check_close(g, w, DTYPES[dt], f"{name} {shape} {dt} {mode}", reduction=name != "grad_x")
    assert _lib.load().ddf_b200_take_fault() == 0


EXTREME = [(1, 70, 101, 75, 3, 2, 1), (1, 24, 63, 101, 5, 1, 1), (2, 131, 51, 75, 3, 1, 2)]


@pytest.mark.parametrize("shape", EXTREME)
@pytest.mark.parametrize("which", [0, 1, 2, 3])
@pytest.mark.parametrize("dt", ["f32", "bf16"])
@pytest.mark.parametrize("version", ["", "o"])
def test_padding_is_skipped_not_multiplied(shape, which, dt, version):
    """An infinity in one operand reaches exactly the results it reaches in the oracle, which skips taps
    outside the plane, and leaves the others as they are.  (The filter gradients' compensated sums make NaN of
    an infinity; their other values are compared.)"""
    from ddfnet_b200 import ddf
    k, d, s = shape[4:]
    for mode in ("mul", "add"):
        cpu, t = _inputs(shape, dt, 9)
        for v in (cpu[which], t[which]):
            v.view(-1)[::37] = float("inf")
            v.view(-1)[5::411] = float("-inf")
        x, cf, sf, go = cpu
        ts = [v.clone().requires_grad_() for v in t[:3]]
        out = ddf(*ts, k, d, s, mode, version)
        gx, gcf, gsf = torch.autograd.grad(out, ts, t[3])
        wx, wcf, wsf = oracle_backward(go, x, cf, sf, k, d, s, mode)
        check_extremes(out, oracle_forward(x, cf, sf, k, d, s, mode), DTYPES[dt], f"out {mode}")
        check_extremes(gx, wx, DTYPES[dt], f"grad_x {mode}")
        for name, g, w in (("grad_cf", gcf, wcf), ("grad_sf", gsf, wsf)):
            fin = torch.isfinite(w)
            assert torch.equal(torch.isfinite(g).cpu(), fin), f"{name} {mode}"
            zero = torch.zeros((), dtype=torch.float64)
            check_close(torch.where(fin, g.cpu().double(), zero), torch.where(fin, w, zero), DTYPES[dt], f"{name} {mode}",
                        reduction=True)


@pytest.mark.parametrize("shape", EXTREME + [(3, 37, 9, 11, 3, 1, 1), (1, 24, 63, 101, 5, 2, 1)])
@pytest.mark.parametrize("which", [1, 2])
@pytest.mark.parametrize("dt", ["f32", "bf16"])
@pytest.mark.parametrize("mode", ["mul", "add"])
def test_large_filter_values(shape, which, dt, mode):
    """Filter values from 1e18 on, whose products with padding zeros would be no safe zeros, take the loop that
    skips the padding: every value of it.  At most one such value in a window, so that none cancels; the filter
    gradients, sums of several, are held in the 2-norm."""
    from ddfnet_b200 import ddf
    k, d, s = shape[4:]
    cpu, t = _inputs(shape, dt, 10)
    for v in (cpu[which], t[which]):
        v.view(-1)[:: (211 if which == 1 else 1009)] = 2e18
    x, cf, sf, go = cpu
    ts = [v.clone().requires_grad_() for v in t[:3]]
    out = ddf(*ts, k, d, s, mode)
    gx, *filters = torch.autograd.grad(out, ts, t[3])
    wx, *want = oracle_backward(go, x, cf, sf, k, d, s, mode)
    check_close(out, oracle_forward(x, cf, sf, k, d, s, mode), DTYPES[dt], "out")
    check_close(gx, wx, DTYPES[dt], "grad_x")
    for g, w in zip(filters, want):
        assert (g.cpu().double() - w).norm() <= (1e-6 if dt == "f32" else 4e-3) * w.norm()


@pytest.mark.parametrize("shape", [(2, 300, 60, 63, 3, 1, 1), (300, 40, 14, 13, 3, 2, 1), (2, 300, 45, 47, 5, 1, 1), (4, 200, 61, 63, 3, 1, 2),
                                   (1, 96, 75, 301, 5, 2, 1)])
@pytest.mark.parametrize("dt", ["f32", "bf16"])
@pytest.mark.parametrize("mode", ["mul", "add"])
def test_results_do_not_change_between_runs(shape, dt, mode):
    """Every CTA walks several times more stages than its ring has slots: a value read after its slot was handed
    back would show as a difference between runs (there are no atomics: equal inputs give equal bits)."""
    from ddfnet_b200 import _lib, ddf
    k, d, s = shape[4:]
    _, t = _inputs(shape, dt, 11)
    ts = [v.requires_grad_() for v in t[:3]]

    def results():
        out = ddf(*ts, k, d, s, mode)
        return [out, *torch.autograd.grad(out, ts, t[3])]

    first = results()
    for _ in range(30):
        assert all(torch.equal(a, b) for a, b in zip(results(), first))
    assert _lib.load().ddf_b200_take_fault() == 0


def test_spatial_norm_inside_the_kernel():
    from ddfnet_b200.op import ddf_sfnorm, spatial_filter_norm
    shape = (1, 70, 101, 75, 3, 1, 1)
    (x, cf, raw, _), dev = _inputs(shape, "f32", 3)
    out = ddf_sfnorm(*dev[:3], 3, 1, 1, "mul", 0.7)
    want = oracle_forward(x, cf, spatial_filter_norm(raw.double(), 3, 0.7), 3, 1, 1, "mul")
    check_close(out, want, torch.float32, "sfnorm")


@pytest.mark.parametrize("shape", [(4, 60, 50, 67, 3, 1, 1), (16, 75, 9, 11, 3, 1, 2)])
def test_no_scratch_and_built_in_scratch(shape):
    """Without a workspace the generic kernels run, as for every problem that they cover; the entry point
    with built-in scratch gives the regular one's results."""
    from ddfnet_b200 import _lib
    L = _lib.load()
    B, C, H, W, k, d, s = shape
    (x, cf, sf, go), dev = _inputs(shape, "f32", 4)
    want = oracle_backward(go, x, cf, sf, k, d, s, "mul")
    xd, cfd, sfd, god = dev
    st = torch.cuda.current_stream().cuda_stream
    need = int(L.ddf_b200_backward_workspace(B, C, H, W, k, d, s, 0, 0, _lib.VARIANT_AUTO))
    assert need > 0
    ws = torch.empty(need, dtype=torch.uint8, device=xd.device)
    got = []
    for ptr, n in ((ws.data_ptr(), need), (None, 0)):
        g = [torch.empty_like(t) for t in dev[:3]]
        assert L.ddf_b200_backward(god.data_ptr(), xd.data_ptr(), cfd.data_ptr(), sfd.data_ptr(), *(t.data_ptr() for t in g),
                                   ptr, n, B, C, H, W, k, d, s, 0, 0, _lib.VARIANT_AUTO, st) == 0
        got.append(g)
    g = [torch.empty_like(t) for t in dev[:3]]
    assert L.ddf_b200_backward_noalloc(god.data_ptr(), xd.data_ptr(), cfd.data_ptr(), sfd.data_ptr(),
                                       *(t.data_ptr() for t in g), B, C, H, W, k, d, s, 0, 0, st) == 0
    got.append(g)
    for gs in got:
        for name, a, w in zip(("grad_x", "grad_cf", "grad_sf"), gs, want):
            check_close(a, w, torch.float32, name, reduction=name != "grad_x")
    assert all(torch.equal(a, b) for a, b in zip(got[0], got[2]))


@pytest.mark.parametrize("shape", [(2, 150, 33, 45, 3, 1, 1), (3, 37, 9, 11, 3, 2, 1), (2, 60, 31, 29, 5, 1, 1), (2, 64, 50, 67, 3, 1, 2)])
@pytest.mark.parametrize("dt", ["f32", "bf16"])
def test_wait_limit_reports_a_fault_and_the_context_survives(shape, dt):
    """Every stage is announced 16 bytes larger than what is copied, so that none completes: with a limit of
    about a millisecond the compute warps give up, the kernels return, the fault word reads 1 and the next
    calls give their results."""
    from ddfnet_b200 import _lib
    L = _lib.load()
    B, C, H, W, k, d, s = shape
    dc = {"f32": _lib.F32, "bf16": _lib.BF16}[dt]
    (x, cf, sf, go), dev = _inputs(shape, dt, 6)
    xd, cfd, sfd, god = dev
    out, gcf, gsf = torch.empty_like(god), torch.empty_like(cfd), torch.empty_like(sfd)
    ws = torch.empty(64 << 20, dtype=torch.uint8, device=xd.device)

    def call(o, filters, limit, starve):
        return L.ddf_b200_band_waitlimit(god.data_ptr(), xd.data_ptr(), cfd.data_ptr(), sfd.data_ptr(), o,
                                         *([gcf.data_ptr(), gsf.data_ptr()] if filters else [None, None]),
                                         ws.data_ptr(), ws.numel(), B, C, H, W, k, d, s, _lib.MUL, dc, limit, starve,
                                         torch.cuda.current_stream().cuda_stream)

    assert L.ddf_b200_take_fault() == 0
    for o, filters in ((out.data_ptr(), False), (None, True)):
        assert call(o, filters, 2_000_000, 1) == 0
        assert L.ddf_b200_take_fault() == 1
        assert L.ddf_b200_take_fault() == 0
    assert call(out.data_ptr(), True, 2_000_000_000, 0) == 0
    check_close(out, oracle_forward(x, cf, sf, k, d, s, "mul"), DTYPES[dt], "forward after a starved launch")
    _, wcf, wsf = oracle_backward(go, x, cf, sf, k, d, s, "mul")
    check_close(gcf, wcf, DTYPES[dt], "grad_cf after a starved launch", reduction=True)
    check_close(gsf, wsf, DTYPES[dt], "grad_sf after a starved launch", reduction=True)
    assert L.ddf_b200_take_fault() == 0


@pytest.mark.parametrize("shape", [(3, 328, 11, 7, 5, 2, 1), (3, 432, 9, 7, 5, 1, 1), (5, 64, 12, 21, 3, 2, 1), (4, 128, 50, 67, 3, 1, 1),
                                   (4, 80, 55, 69, 3, 1, 2), (1, 512, 33, 31, 3, 1, 1)])
@pytest.mark.parametrize("dt", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("mode", ["mul", "add"])
def test_filter_gradients_are_as_exact_as_the_generic_kernels(shape, dt, mode):
    """Relative error (2-norm) against 64 bits.  The final rounding is the same on both sides and most of it; a
    float32 problem's ratio scatters by 1 % from seed to seed (its sums have other orders)."""
    from ddfnet_b200 import ddf
    k, d, s = shape[4:]
    _, t = _inputs(shape, dt, 60)
    err = {}
    exact = [v.double().requires_grad_() for v in t[:3]]
    want = torch.autograd.grad(ddf(*exact, k, d, s, mode, "o"), exact[1:], t[3].double())
    for version in ("", "o"):
        ts = [v.clone().requires_grad_() for v in t[:3]]
        got = torch.autograd.grad(ddf(*ts, k, d, s, mode, version), ts[1:], t[3])
        err[version] = [((g.double() - w).norm() / w.norm()).item() for g, w in zip(got, want)]
    for a, b in zip(err[""], err["o"]):
        assert a <= b * (1.03 if dt == "f32" else 1.0001), err


@pytest.mark.parametrize("shape,dt", [((5, 60, 50, 67, 3, 1, 1), "f32"), ((3, 75, 31, 29, 5, 1, 1), "bf16"), ((7, 75, 33, 31, 3, 1, 2), "f16")])
def test_less_scratch_gives_the_same_bits(shape, dt):
    """The samples go through the scratch in slices of what it holds, down to one."""
    from ddfnet_b200 import _lib
    L = _lib.load()
    B, C, H, W, k, d, s = shape
    dc = {"f32": _lib.F32, "f16": _lib.F16, "bf16": _lib.BF16}[dt]
    _, dev = _inputs(shape, dt, 8)
    need = int(L.ddf_b200_backward_workspace(B, C, H, W, k, d, s, _lib.ADD, dc, _lib.VARIANT_AUTO))
    assert need > 0 and need % B == 0
    ws, got = torch.empty(need, dtype=torch.uint8, device="cuda"), []
    for samples in (B, B - 1, 2, 1):
        ws.fill_(0xff)
        g = [torch.empty_like(t) for t in dev[1:3]]
        before = L.ddf_b200_launch_count()
        assert L.ddf_b200_backward(dev[3].data_ptr(), *(t.data_ptr() for t in dev[:3]), None, *(t.data_ptr() for t in g),
                                   ws.data_ptr(), need // B * samples, B, C, H, W, k, d, s, _lib.ADD, dc,
                                   _lib.VARIANT_AUTO, torch.cuda.current_stream().cuda_stream) == 0
        assert L.ddf_b200_launch_count() - before == 2 * -(-B // samples)
        got.append(g)
    for g in got[1:]:
        assert torch.equal(g[0], got[0][0]) and torch.equal(g[1], got[0][1])
