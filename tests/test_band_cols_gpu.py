"""Filter gradients by a thread per tap column (2-byte types, stride 1) against the float64 oracle: planes per pass,
bands, bands shared by several CTAs, chunks that do not fill their last pass, dilated groups beyond the plane; and the
planes whose width four does not divide, which it takes from the plane-streaming form, with and without scratch."""
import pytest
import torch

from tests.util import DTYPES, check_close, make_inputs, oracle_backward

pytestmark = pytest.mark.gpu

# (B, C, H, W, k, d)
SHAPES = [(2, 9, 7, 9, 3, 1), (3, 67, 8, 11, 3, 2), (1, 130, 33, 40, 3, 1), (2, 37, 50, 67, 3, 1), (1, 9, 21, 320, 3, 1),
          (1, 6, 9, 333, 3, 2), (1, 5, 5, 700, 3, 1),            # wider than a CTA's ten warps of a column
          (2, 21, 9, 30, 5, 1), (1, 70, 17, 31, 5, 2), (1, 11, 30, 97, 5, 1), (1, 7, 19, 101, 5, 2), (1, 4, 11, 320, 5, 1)]
# many planes: 14 and 7 columns, and a width that two divides
STAGES = [(40, 24, 14, 14, 3, 1), (40, 24, 14, 14, 5, 1), (60, 36, 7, 7, 3, 1), (60, 36, 7, 7, 5, 1), (12, 40, 20, 30, 3, 2)]


def _grads(shape, dt, mode, scratch=True):
    from ddfnet_b200 import _lib
    B, C, H, W, k, d = shape
    cpu = make_inputs(B, C, H, W, k, 1, DTYPES[dt], 90 + sum(shape))
    x, cf, sf, go = (t.to("cuda:0") for t in cpu)
    L = _lib.load()
    gcf, gsf = torch.empty_like(cf), torch.empty_like(sf)
    args = (B, C, H, W, k, d, 1, {"mul": 0, "add": 1}[mode], {"f16": 1, "bf16": 2}[dt])
    need = int(L.ddf_b200_backward_workspace(*args, 0))
    ws = torch.empty(max(need, 16), dtype=torch.uint8, device="cuda:0") if scratch else None
    st = torch.cuda.current_stream().cuda_stream
    rc = L.ddf_b200_backward(go.data_ptr(), x.data_ptr(), cf.data_ptr(), sf.data_ptr(), None, gcf.data_ptr(),
                             gsf.data_ptr() if scratch else None, ws.data_ptr() if scratch else None, need if scratch else 0,
                             *args, 0, st)
    assert rc == 0
    assert L.ddf_b200_take_fault() == 0
    return cpu, gcf, gsf


@pytest.mark.parametrize("shape", SHAPES + STAGES)
@pytest.mark.parametrize("dt", ["f16", "bf16"])
@pytest.mark.parametrize("mode", ["mul", "add"])
def test_matches_oracle(shape, dt, mode):
    (x, cf, sf, go), gcf, gsf = _grads(shape, dt, mode)
    k, d = shape[4:]
    _, wcf, wsf = oracle_backward(go, x, cf, sf, k, d, 1, mode)
    check_close(gcf, wcf, DTYPES[dt], f"grad_cf {shape} {dt} {mode}", reduction=True)
    check_close(gsf, wsf, DTYPES[dt], f"grad_sf {shape} {dt} {mode}", reduction=True)


@pytest.mark.parametrize("shape", STAGES)
def test_channel_filters_alone_need_no_scratch(shape):
    (x, cf, sf, go), gcf, _ = _grads(shape, "bf16", "mul", scratch=False)
    k, d = shape[4:]
    check_close(gcf, oracle_backward(go, x, cf, sf, k, d, 1, "mul")[1], DTYPES["bf16"], f"grad_cf {shape}", reduction=True)
