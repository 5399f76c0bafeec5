"""Convolutions on the hand-written tcgen05 kernels.

* :func:`conv2d` - 1x1 and 3x3 convolutions (stride 1 or 2, padding (k-1)/2, channel counts multiples of 64) of
  channels-last bf16 activations: forward, data gradient and weight gradient are implicit GEMMs on tcgen05 / TMEM with
  TMA-fetched pixel boxes (``csrc/conv_igemm_tcgen05.cu``); the forward can hand the following BatchNorm its
  per-channel statistics from the epilogue, one set per stacked view.
* :func:`stem_conv` - the ResNet stem (7 x 7, stride 2, 3 -> 64 channels; ``csrc/conv_stem_tcgen05.cu``), also with
  BatchNorm statistics in the epilogue, and its weight gradient.
* :func:`conv_bn_act` - ``relu(bn(conv(x)) + residual)`` built from the two and :func:`tspipe_b200.ops.bn.bn_act`.

Reference call sites: the convolutions of the torchvision ResNet that
`benchmarks/byol/models/resnet_base_network.py:60-77` flattens (library convolutions there).
"""
from __future__ import annotations

import ctypes as _c
import os
from typing import Optional, Tuple

import torch
from torch import nn

from . import bn as _bn
from . import fused as _f
from . import gemm as _gemm

K_REAL = 147
K_PAD = 192


def is_stem_conv(m: nn.Module) -> bool:
    return (isinstance(m, nn.Conv2d) and m.in_channels == 3 and m.out_channels == 64 and m.kernel_size == (7, 7)
            and m.stride == (2, 2) and m.padding == (3, 3) and m.dilation == (1, 1) and m.groups == 1
            and m.bias is None and m.padding_mode == "zeros")


def eligible(x: torch.Tensor) -> bool:
    """Channels-last bf16 CUDA input [N, 3, H, W] with H even and W a multiple of 8 in [8, 224]."""
    if not (isinstance(x, torch.Tensor) and x.is_cuda and x.dim() == 4 and x.dtype == torch.bfloat16):
        return False
    n, c, h, w = x.shape
    if c != 3 or h % 2 or w % 8 or not (8 <= w <= 224) or h < 8:
        return False
    return x.stride() == (h * w * 3, 1, w * 3, 3) and x.data_ptr() % 16 == 0


def weight_matrix(weight: torch.Tensor) -> torch.Tensor:
    """``[64, 3, 7, 7]`` -> bf16 ``[64, 192]`` with ``k = kh * 21 + kw * 3 + c`` and zeros from k = 147."""
    wm = torch.zeros(64, K_PAD, dtype=torch.bfloat16, device=weight.device)
    wm[:, :K_REAL] = weight.detach().permute(0, 2, 3, 1).reshape(64, K_REAL)
    return wm


class _StemConv(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, want_sums, segs):
        n, _, h, w = x.shape
        y = torch.empty((n, 64, h // 2, w // 2), dtype=torch.bfloat16, device=x.device,
                        memory_format=torch.channels_last)
        sums = _f.zeroed(segs * 128, x.device) if want_sums else None
        wm = weight_matrix(weight)
        L = _f.lib()
        L.tsp_conv_stem_fwd.restype = _c.c_int
        with _f.on_device(x.device):
            code = L.tsp_conv_stem_fwd(_f._ptr(x), _f._ptr(wm), _f._ptr(y), _f._ptr(sums), _c.c_int(n), _c.c_int(h),
                                       _c.c_int(w), _c.c_int(segs), _f._ptr(_gemm._status_word(x.device)), _f._stream())
        _f._check(code, "tsp_conv_stem_fwd")
        _f._count()
        ctx.save_for_backward(x, weight)
        if sums is None:
            sums = torch.empty(0, device=x.device)
        ctx.mark_non_differentiable(sums)
        ctx.set_materialize_grads(False)   # (sums' gradient would be a tensor of zeros, allocated and filled on every call)
        return y, sums

    @staticmethod
    def backward(ctx, dy, _dsums):
        if dy is None:
            return None, None, None, None
        x, weight = ctx.saved_tensors
        dx = dw = None
        need_dx = ctx.needs_input_grad[0]
        dy = dy.to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
        if need_dx:                        # images that want a gradient themselves: the library's data gradient
            dx = torch.ops.aten.convolution_backward(dy, x, weight.to(torch.bfloat16), None, [2, 2], [3, 3], [1, 1], False,
                                                     [0, 0], 1, [True, False, False])[0]
        if ctx.needs_input_grad[1]:
            # (added in place in a recording only: an eager call may have asked for this gradient by name)
            target = _grad_target(weight) if _f.adds_in_place(weight) else None
            if target is None:
                target = torch.zeros((64, 7, 7, 3), dtype=torch.float32, device=x.device)
                dw = target.permute(0, 3, 1, 2)
            if dy.data_ptr() % 16:
                dy = dy.clone(memory_format=torch.channels_last)
            n, _, h, w = x.shape
            L = _f.lib()
            L.tsp_conv_stem_wgrad.restype = _c.c_int
            with _f.on_device(x.device):
                code = L.tsp_conv_stem_wgrad(_f._ptr(x), _f._ptr(dy), _f._ptr(target), _c.c_int(n), _c.c_int(h),
                                             _c.c_int(w), _f._ptr(_gemm._status_word(x.device)), _f._stream())
            _f._check(code, "tsp_conv_stem_wgrad")
            _f._count()
            if dw is not None and weight.dtype != torch.float32:
                dw = dw.to(weight.dtype)
        return dx, dw, None, None


def _grad_target(weight: torch.Tensor) -> Optional[torch.Tensor]:
    """The weight's fp32 gradient when a kernel can add to it in place: it lives in the layout [Cout][k][k][Cin], i.e.
    channels-last, as in the runtime's flat gradient buffer (autograd then gets nothing more to accumulate)."""
    g = weight.grad if weight.is_leaf else None
    if (_ACCUMULATE_IN_PLACE and g is not None and g.dtype == torch.float32 and g.shape == weight.shape
            and g.permute(0, 2, 3, 1).is_contiguous()):
        return g
    return None


def stem_conv(x: torch.Tensor, weight: torch.Tensor, want_sums: bool = True, segments: int = 1
              ) -> Tuple[torch.Tensor, Optional[torch.Tensor]]:
    """``(y, sums)``: y = conv2d(x, weight, stride 2, padding 3) in channels-last bf16; ``sums`` = per-channel
    [sum | sum of squares] of y over all pixels (fp32, ``[segments][128]`` flattened: one set per group of
    ``N / segments`` consecutive images) or None."""
    if x.shape[0] % segments != 0:
        segments = 1
    y, sums = _StemConv.apply(x, weight, want_sums, segments)
    return y, (sums if want_sums else None)


# -------------------------------------------------------------------------------------------------
# 1x1 / 3x3 convolutions: implicit GEMM on tcgen05 (csrc/conv_igemm_tcgen05.cu)
# -------------------------------------------------------------------------------------------------
# eligible convolutions run on the tcgen05 implicit-GEMM kernels (set_igemm(False) or TSPIPE_CONV=library: library)
_IGEMM = os.environ.get("TSPIPE_CONV", "igemm") != "library"
_W16 = {}            # id(weight) -> (weight, version, bf16 [Cout, k, k, Cin] copy); dropped at every optimizer step


def set_igemm(flag: bool) -> None:
    """Route eligible convolutions through the tcgen05 implicit-GEMM kernels (default) or the library."""
    global _IGEMM
    _IGEMM = bool(flag)


def clear_weight_cache() -> None:
    _W16.clear()


def _w16(weight: torch.Tensor) -> torch.Tensor:
    """bf16 copy of a convolution weight laid out ``[Cout][kh][kw][Cin]`` (no copy beyond the cast when the
    parameter is stored channels-last, which is how the runtime keeps 4-D parameters)."""
    if _f.IN_CAPTURE:                   # inside a CUDA graph the cast is part of the graph
        w = _f.recorded_bf16(weight).permute(0, 2, 3, 1)
        return w if w.is_contiguous() and w.data_ptr() % 16 == 0 else w.clone(memory_format=torch.contiguous_format)
    hit = _W16.get(id(weight))
    if hit is not None and hit[0] is weight and hit[1] == weight._version and hit[2].device == weight.device:
        return hit[2]
    w = weight.detach().to(torch.bfloat16).permute(0, 2, 3, 1)
    if not w.is_contiguous():
        w = w.contiguous()
    _W16[id(weight)] = (weight, weight._version, w)
    return w


def _nhwc(x: torch.Tensor) -> bool:
    n, c, h, w = x.shape
    return x.stride() == (h * w * c, 1, w * c, c) or (h * w == 1 and x.is_contiguous())


def igemm_eligible(m: nn.Module, x: torch.Tensor) -> bool:
    """Conv2d with a square 1x1 or 3x3 kernel, stride 1 or 2, padding (k-1)/2, no bias / groups / dilation, channel
    counts multiples of 64, on a channels-last bf16 CUDA activation (even height and width for stride 2)."""
    if not (isinstance(m, nn.Conv2d) and m.groups == 1 and m.bias is None and m.dilation == (1, 1)
            and m.padding_mode == "zeros"):
        return False
    k, s = m.kernel_size[0], m.stride[0]
    if m.kernel_size != (k, k) or m.stride != (s, s) or k not in (1, 3) or s not in (1, 2) \
            or m.padding != ((k - 1) // 2, (k - 1) // 2):
        return False
    if m.in_channels % 64 or m.out_channels % 64:
        return False
    if not (isinstance(x, torch.Tensor) and x.is_cuda and x.dim() == 4 and x.dtype == torch.bfloat16):
        return False
    n, c, h, w = x.shape
    if s == 2 and (h % 2 or w % 2):
        return False
    return _nhwc(x) and x.data_ptr() % 16 == 0


def _lib():
    L = _f.lib()
    if not hasattr(L, "_conv_ready"):
        for name in ("tsp_conv_fprop", "tsp_conv_dgrad", "tsp_conv_wgrad"):
            getattr(L, name).restype = _c.c_int
        L._conv_ready = True
    return L


def _geom(x: torch.Tensor, weight: torch.Tensor, stride: int):
    n, cin, h, w = x.shape
    cout, k = weight.shape[0], weight.shape[2]
    pad = (k - 1) // 2
    return n, h, w, cin, cout, k, (h + 2 * pad - k) // stride + 1, (w + 2 * pad - k) // stride + 1


def _stats_ok(n: int, ho: int, wo: int, k: int, stride: int, segs: int) -> bool:
    if n % segs:
        return False
    # Flat tiles of 128 pixels, which must not straddle two views; the rows that the last one lacks count as zeros.  Convolution,
    # statistics and normalisation on a B200, with a pass of its own for the statistics and with the epilogue's: 64 images of 7 x 7,
    # 512 -> 2048 42.4 and 36.2 us, 37 of 14 x 14, 256 -> 1024 40.2 and 34.0, one of 7 x 7, 64 -> 64 25.4 and 24.5.
    if k == 1 and stride == 1:
        return segs == 1 or (n // segs * ho * wo) % 128 == 0
    if ho * wo <= 64:                          # several images per pixel box: a box must not straddle two views
        per_box = 128 // (ho * wo)
        tiles = -(-n // per_box)
        return (n // segs) % (-(-n // tiles)) == 0
    return True


class _Conv2d(torch.autograd.Function):
    """``conv2d`` forward / backward on the implicit-GEMM kernels.  Returns ``(y, sums)``; ``sums`` (not
    differentiable) holds ``[segs][sum | sum of squares]`` per output channel when requested."""

    @staticmethod
    def forward(ctx, x, weight, stride, want_sums, segs):
        n, h, w, cin, cout, k, ho, wo = _geom(x, weight, stride)
        w16 = _w16(weight)
        y = torch.empty((n, cout, ho, wo), dtype=torch.bfloat16, device=x.device, memory_format=torch.channels_last)
        sums = _f.zeroed(segs * 2 * cout, x.device) if want_sums else None
        with _f.on_device(x.device):
            code = _lib().tsp_conv_fprop(_f._ptr(x), _f._ptr(w16), _f._ptr(y), _f._ptr(sums), _c.c_int(segs), _c.c_int(n),
                                         _c.c_int(h), _c.c_int(w), _c.c_int(cin), _c.c_int(cout), _c.c_int(k),
                                         _c.c_int(stride), _f._ptr(_gemm._status_word(x.device)), _f._stream())
        _f._check(code, "tsp_conv_fprop")
        _f._count()
        ctx.save_for_backward(x, weight)
        ctx.stride = stride
        if sums is None:
            sums = torch.empty(0, device=x.device)
        ctx.mark_non_differentiable(sums)
        ctx.set_materialize_grads(False)   # (sums' gradient would be a tensor of zeros, allocated and filled on every call)
        return y, sums

    @staticmethod
    def backward(ctx, dy, _dsums):
        return _Conv2d._backward(ctx, dy, None) if dy is not None else (None,) * 5

    @staticmethod
    def _backward(ctx, dy, addend):
        x, weight = ctx.saved_tensors
        stride = ctx.stride
        n, h, w, cin, cout, k, ho, wo = _geom(x, weight, stride)
        if dy.dtype != torch.bfloat16 or not _nhwc(dy):
            dy = dy.to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
        L = _lib()
        status = _f._ptr(_gemm._status_word(x.device))
        dx = dw = None
        with _f.on_device(x.device):
            st = _f._stream()
            if ctx.needs_input_grad[0]:
                dx = torch.empty_like(x)
                code = L.tsp_conv_dgrad(_f._ptr(dy), _f._ptr(_w16(weight)), _f._ptr(addend), _f._ptr(dx), _c.c_int(n),
                                        _c.c_int(h), _c.c_int(w), _c.c_int(cin), _c.c_int(cout), _c.c_int(k),
                                        _c.c_int(stride), status, st)
                _f._check(code, "tsp_conv_dgrad")
                _f._count(4 if stride == 2 and k == 3 else 1)
            if ctx.needs_input_grad[1]:
                target = _grad_target(weight)      # the kernel ADDS into its output
                if target is None:
                    target = torch.zeros((cout, k, k, cin), dtype=torch.float32, device=x.device)
                    dw = target.permute(0, 3, 1, 2)
                code = L.tsp_conv_wgrad(_f._ptr(x), _f._ptr(dy), _f._ptr(target), _c.c_int(n), _c.c_int(h), _c.c_int(w),
                                        _c.c_int(cin), _c.c_int(cout), _c.c_int(k), _c.c_int(stride), status, st)
                _f._check(code, "tsp_conv_wgrad")
                _f._count()
                if dw is not None and weight.dtype != torch.float32:
                    dw = dw.to(weight.dtype)
        return dx, dw, None, None, None


class _Conv2dFork(torch.autograd.Function):
    """:class:`_Conv2d` of an input that is also handed on unchanged (the other branch of a residual block): the
    gradient that comes back on that branch is added by the data-gradient kernel as it stores its result."""

    @staticmethod
    def forward(ctx, x, weight, stride, want_sums, segs):
        y, sums = _Conv2d.forward(ctx, x, weight, stride, want_sums, segs)
        return y, sums, x.view_as(x)

    @staticmethod
    def backward(ctx, dy, _dsums, dskip):
        x, _ = ctx.saved_tensors
        if dy is None:
            return dskip, None, None, None, None
        fits = (dskip is not None and dskip.dtype == x.dtype and _nhwc(dskip) and dskip.data_ptr() % 16 == 0
                and ctx.needs_input_grad[0])
        grads = _Conv2d._backward(ctx, dy, dskip if fits else None)
        if dskip is not None and not fits and grads[0] is not None:
            return (grads[0] + dskip,) + grads[1:]
        return grads


_ACCUMULATE_IN_PLACE = True


def set_accumulate_in_place(flag: bool) -> None:
    """Let the kernels of weight gradients, and in eager calls those of bias and BatchNorm gradients, add straight into an
    existing fp32 ``grad`` of matching layout (default) instead of handing autograd a fresh tensor to accumulate."""
    global _ACCUMULATE_IN_PLACE
    _ACCUMULATE_IN_PLACE = bool(flag)
    if _f._host is not None:                   # (one that is loaded later takes the setting then)
        _f._host.set_accumulate(_ACCUMULATE_IN_PLACE)


def conv2d(x: torch.Tensor, weight: torch.Tensor, stride: int = 1, want_sums: bool = False, segments: int = 1
           ) -> Tuple[torch.Tensor, Optional[torch.Tensor]]:
    """``(y, sums)``: ``y = conv2d(x, weight, stride, padding (k-1)/2)`` in channels-last bf16; ``sums`` =
    ``[segments][sum | sum of squares]`` per output channel over each group of ``N / segments`` consecutive images
    (fp32) when ``want_sums`` and the tiling allows it, else None."""
    n, h, w, cin, cout, k, ho, wo = _geom(x, weight, stride)
    want = bool(want_sums) and _stats_ok(n, ho, wo, k, stride, segments)
    y, sums = _Conv2d.apply(x, weight, stride, want, segments)
    return y, (sums if want else None)


def _eager(conv: nn.Module, bn: nn.Module, x: torch.Tensor, residual: Optional[torch.Tensor], relu: bool, fork: bool):
    """An eligible convolution and its training-mode BatchNorm as one C++ autograd function: ``(y,)``, with ``fork`` ``(y, x)``;
    None where that does not apply."""
    host = _f.eager() if type(x) is torch.Tensor else None
    if host is None:
        return None
    weight, stride = conv.weight, conv.stride[0]
    n, h, w, _, cout, k, ho, wo = _geom(x, weight, stride)
    segs = _bn.tracked_segments(bn, n * ho * wo, n, cout)
    if segs == 0:
        return None
    return host.conv_bn_act(x, weight, _w16(weight), bn.weight, bn.bias, residual, bn.sum, bn.sum_squares, bn.count,
                            bn.group.total, bn.eps, relu, stride, segs, _stats_ok(n, ho, wo, k, stride, segs), fork,
                            _gemm._status_word(x.device))


def conv_bn_act(conv: nn.Module, bn: nn.Module, x: torch.Tensor, residual: Optional[torch.Tensor] = None,
                relu: bool = False) -> torch.Tensor:
    """``relu(bn(conv(x)) + residual)``.  An eligible convolution runs on the tcgen05 implicit-GEMM kernel; in front
    of a training-mode BatchNorm its epilogue already produces the BatchNorm's statistics (one pass over the
    activation less).  Everything else is the library convolution followed by :func:`tspipe_b200.ops.bn.bn_act`."""
    if _IGEMM and torch.is_autocast_enabled() and igemm_eligible(conv, x):
        out = _eager(conv, bn, x, residual, relu, False)
        if out is not None:
            return out[0]
        want = bool(bn.training)
        segs = _bn.current_segments() if want else 1
        y, sums = conv2d(x, conv.weight, conv.stride[0], want_sums=want, segments=segs)
        return _bn.bn_act(bn, y, residual, relu, sums=sums if (sums is not None and _bn.applicable(bn, y)) else None)
    return _bn.bn_act(bn, conv(x), residual, relu)


def conv_bn_act_fork(conv: nn.Module, bn: nn.Module, x: torch.Tensor, relu: bool = False
                     ) -> Tuple[torch.Tensor, torch.Tensor]:
    """``(relu(bn(conv(x))), x)`` for the first convolution of a residual block: the second output is ``x`` for the
    block's other branch, whose gradient the convolution's data gradient takes along (see :class:`_Conv2dFork`)."""
    if not (_IGEMM and torch.is_grad_enabled() and x.requires_grad and torch.is_autocast_enabled()
            and igemm_eligible(conv, x) and (conv.kernel_size[0], conv.stride[0]) != (1, 2)):
        return conv_bn_act(conv, bn, x, relu=relu), x
    out = _eager(conv, bn, x, None, relu, True)
    if out is not None:
        return out[0], out[1]
    want = bool(bn.training)
    segs = _bn.current_segments() if want else 1
    n, h, w, _, _, k, ho, wo = _geom(x, conv.weight, conv.stride[0])
    want = want and _stats_ok(n, ho, wo, k, conv.stride[0], segs)
    y, sums, skip = _Conv2dFork.apply(x, conv.weight, conv.stride[0], want, segs)
    y = _bn.bn_act(bn, y, None, relu, sums=sums if (want and _bn.applicable(bn, y)) else None)
    return y, skip


def conv(m: nn.Module, x: torch.Tensor) -> torch.Tensor:
    """``m(x)`` for a Conv2d, on the implicit-GEMM kernel when eligible."""
    if _IGEMM and torch.is_autocast_enabled() and igemm_eligible(m, x):
        return conv2d(x, m.weight, m.stride[0])[0]
    return m(x)
