"""``ddf(features, channel_filter, spatial_filter, kernel_size, dilation, stride,
kernel_combine, version)`` -- drop-in for the reference autograd op
(``DDFFunction`` / ``ddf`` in ddf/ddf.py:27-122).

Same positional signature, same assertion checks (ddf/ddf.py:32-65), same
8-tuple of gradients (ddf/ddf.py:119).  Differences, all deliberate:

* float16 and bfloat16 tensors are computed natively (float accumulation) and
  the result has the input's type; the reference up-casts float16 to float32
  (ddf/ddf.py:36-42) and cannot take bfloat16.
* inputs are saved for the backward when autograd asks for any input gradient
  (``ctx.needs_input_grad``); the reference tests ``requires_grad`` on its
  up-cast copies (ddf/ddf.py:88-89), which loses the graph under float16.
* ``version``: '' picks a kernel automatically, 'o' forces the generic kernel,
  'f' forces the plane-streaming kernel (the reference's 'o' / 'f' select its
  generic / tiled forward, ddf/ddf.py:77-84).
* non-contiguous inputs raise RuntimeError, as the reference's native
  CHECK_CONTIGUOUS does (ddf/src/cuda/ddf_mul_cuda.cpp:28-40).

The arithmetic runs in hand-written CUDA kernels reached through the C ABI of
libddf_b200.so; there is no CPU path.  The host side of a call -- argument checks, output
allocation, autograd node, launch -- is csrc/native.cpp; this file holds the checks' error texts.
"""
from __future__ import annotations

import ctypes

import torch

from . import _lib
try:
    from . import _native
except ImportError:  # not built: importing works, calling the op raises
    _native = None

_DTYPES = {torch.float32: _lib.F32, torch.float16: _lib.F16, torch.bfloat16: _lib.BF16,
           torch.float64: _lib.F64}
_VARIANT = {"": _lib.VARIANT_AUTO, "o": _lib.VARIANT_GENERIC, "f": _lib.VARIANT_STREAM}


def _common_dtype(*tensors):
    dt = tensors[0].dtype
    for t in tensors[1:]:
        dt = torch.promote_types(dt, t.dtype)
    if dt not in _DTYPES:
        raise TypeError(f"ddf: unsupported dtype {dt}")
    return dt


def _require_contiguous(t, name):
    if not t.is_contiguous():
        raise RuntimeError(f"{name} must be contiguous ")


def _check_shapes(features, channel_filter, spatial_filter, kernel_size, dilation, stride,
                  kernel_combine, version):
    """The reference's argument checks (ddf/ddf.py:32-65)."""
    assert features.is_cuda, 'input feature must be a CUDA tensor.'
    assert channel_filter.is_cuda, 'channel_filter must be a CUDA tensor.'
    assert spatial_filter.is_cuda, 'spatial_filter must be a CUDA tensor.'
    b, c, h, w = features.size()
    bc, cc, hc, wc = channel_filter.size()
    assert bc == b and cc == c, \
        "channel_filter size {} does not match feature size {}".format(
            channel_filter.size(), features.size())
    assert hc == kernel_size and wc == kernel_size, \
        "channel_filter size {} does not match kernel size {}".format(
            channel_filter.size(), kernel_size)
    bs, cs, hs, ws = spatial_filter.size()
    assert bs == b and hs == h // stride and ws == w // stride, \
        "spatial_filter size {} does not match feature size {} with stride {}".format(
            spatial_filter.size(), features.size(), stride)
    assert cs == kernel_size ** 2, \
        "spatial_filter size {} does not match kernel size {}".format(
            spatial_filter.size(), kernel_size)
    assert (kernel_size - 1) % 2 == 0 and kernel_size >= 1 and dilation >= 1 and stride >= 1
    assert kernel_combine in {'mul', 'add'}, \
        'only support mul or add combination, instead of {}'.format(kernel_combine)
    assert version in _VARIANT, "version must be '', 'o' or 'f'"
    assert channel_filter.device == features.device and spatial_filter.device == features.device


def spatial_filter_norm(raw, kernel_size, scale):
    """FilterNorm(filter_type='spatial') without running statistics (ddf/ddf.py:146-157) on a
    (B, k*k, H, W) tensor whose heads are already folded into B: each pixel's k*k values are
    centred, divided by their unbiased std + 1e-10 and multiplied by ``scale``.  Plain torch
    ops, float32 statistics for 2-byte inputs: the statement of what the fused kernels compute."""
    v = raw.float() if raw.dtype in (torch.float16, torch.bfloat16) else raw
    v = v - v.mean(dim=1, keepdim=True)
    v = v / (v.std(dim=1, keepdim=True) + 1e-10)
    return v * scale


def explain(norm, features, channel_filter, spatial_filter, kernel_size=3, dilation=1, stride=1,
            kernel_combine='mul', *rest):
    """Raises the error that fits arguments the native entry points refused."""
    version = (rest[1] if len(rest) > 1 else '') if norm else (rest[0] if rest else '')
    if len(rest) > (2 if norm else 1):
        raise TypeError(f"ddf: {7 + len(rest)} arguments given, at most {9 if norm else 8} expected")
    _check_shapes(features, channel_filter, spatial_filter, kernel_size, dilation, stride,
                  kernel_combine, version)
    if norm:
        assert kernel_size >= 3, 'the fused filter norm needs kernel_size >= 3'
        float(rest[0] if rest else 1.0)
    _common_dtype(features, channel_filter, spatial_filter)
    _require_contiguous(features, "features")
    _require_contiguous(channel_filter, "channel_filter")
    _require_contiguous(spatial_filter, "spatial_filter")
    if max(*features.shape, kernel_size, dilation, stride) > 1 << 20:
        raise _lib.DDFError(_lib.E_TOO_LARGE)


def _bind_native():
    """Hands the library's entry points to the native module (the first call does this)."""
    lib = _lib.load()
    names = ("ddf_b200_forward", "ddf_b200_forward_sfnorm", "ddf_b200_backward_workspace", "ddf_b200_backward",
             "ddf_b200_sfnorm", "ddf_b200_sfnorm_backward", "ddf_b200_take_fault")
    _native.bind({n: ctypes.cast(getattr(lib, n), ctypes.c_void_p).value for n in names}, _lib._DEBUG)


def _not_built(*_args):
    raise RuntimeError("ddfnet_b200/_native.so not found. The DDF op has no Python fallback; build it first:  "
                       "python -m ddfnet_b200.csrc.build")


if _native is not None:
    _native.hooks(_lib.DDFError, explain, _bind_native)
ddf = _native.ddf if _native is not None else _not_built
ddf_sfnorm = _native.ddf_sfnorm if _native is not None else _not_built


class DDFFunction:
    """The operator under its autograd-function name (ddf/ddf.py:27): ``DDFFunction.apply`` is ``ddf``."""

    apply = staticmethod(ddf)


class DDFSpatialNormFunction:
    """``ddf`` with the spatial FilterNorm fused into the forward kernel:
    ``ddf_sfnorm(x, cf, raw, k, d, s, combine, scale, version)`` equals
    ``ddf(x, cf, FilterNorm_spatial(raw), k, d, s, combine, version)`` with the normalised
    filter never written to memory (it is kept in float inside the kernel).  The backward
    recomputes the normalised filter with the library's ``ddf_b200_sfnorm``, runs the ordinary
    DDF backward on it and carries the filter gradient back through the normalisation with
    ``ddf_b200_sfnorm_backward``."""

    apply = staticmethod(ddf_sfnorm)
