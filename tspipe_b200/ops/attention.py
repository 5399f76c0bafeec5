"""Scaled dot-product attention ``softmax(Q K^T / sqrt(d) + mask) V`` for [B, H, N, D] tensors.

The reference models run it unfused - two batched GEMMs, a softmax and a dropout
(timm ``Attention`` in `benchmarks/moco-v3/vits.py`, HF ``BertSelfAttention`` in
`benchmarks/distilbert/bert.py`).  Here it is one fused call; ``mask`` is an additive or boolean
key-padding mask broadcastable to [B, 1, 1, N] / [B, H, N, N].

Forward passes that need no gradient (the frozen teacher) with head dimension 64 and a boolean key-padding mask run on the
tcgen05 kernel of ``csrc/attn_heads_tcgen05.cu`` (:func:`heads_fwd`), but for many short sequences, a single key and calls that a
trace, a dispatch mode or autocast to another type is to see; everything else goes to the library's fused attention, which also
provides the backward.
"""
from __future__ import annotations

import ctypes as _c
import math
from typing import Optional, Tuple

import torch
import torch.nn.functional as F

# Forwards without a gradient on :func:`heads_fwd`: None = those with a mask, True = all (without a mask from 4097 keys on by
# :func:`flash_fwd`), False = none.  The library turns a
# mask into an additive matrix, which costs it more than the attention: [32, 12, 512, 64] 110 us with a padding mask and 45
# without one, the kernel 58 and 57; [64, 12, 197, 64] without a mask 32 and 40.
_TCGEN05: Optional[bool] = None
# Heads above which sequences of up to 32 tokens stay with the library: a head is an item of the kernel's there, 128 queries and keys
# whatever they hold.  Masked, [32, 16, 32, 64] 20.9 us either way, [64, 12, 32, 64] 29.1 and the library 27.0, [8, 12, 32, 64]
# 9.8 and 12.7; of 100 tokens [64, 12] 31.1 and 41.3.
_FEW_KEYS = 512


def set_tcgen05(flag: Optional[bool]) -> None:
    global _TCGEN05
    _TCGEN05 = None if flag is None else bool(flag)


_PACKED = {"state": None}     # None = not probed yet, True / False = usable or not

# How the ViT blocks form q, k, v: "packed" = one projection GEMM and the packed-qkv library attention; "split" = one
# projection GEMM whose column tiles go to three tensors (three GEMMs on slices of the weight where its blocks are not what
# the tcgen05 kernels take) and the generic fused attention: no packed tensor, hence no concatenation of dq, dk, dv in the
# backward either.
_QKV_MODE = "split"      # measured on MoCo-v3 ViT-B, 256 samples per GPU: 114.8 ms per step against 121.3 ms for "packed"


def set_qkv_mode(mode: str) -> None:
    global _QKV_MODE
    assert mode in ("packed", "split")
    _QKV_MODE = mode


def qkv_mode() -> str:
    return _QKV_MODE


def project_qkv(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], heads: int):
    """``q, k, v`` as ``[B, H, N, D]`` views from the fused projection parameters ``weight [3C, C]``, ``bias [3C]``.
    On CUDA in "split" mode this is one GEMM whose column tiles go to three tensors (three GEMMs on slices of the parameters
    where the blocks are not what the tcgen05 kernels take), so that no packed qkv tensor exists whose gradient autograd would
    have to assemble from dq, dk and dv; otherwise one GEMM and an unbind."""
    from .linear import linear, linear_qkv
    b, n, c = x.shape
    if x.is_cuda and _QKV_MODE == "split":
        qkv = linear_qkv(x, weight, bias)
        if qkv is not None:
            return tuple(t.view(b, n, heads, c // heads).transpose(1, 2) for t in qkv)
        return tuple(linear(x, weight[i * c:(i + 1) * c], None if bias is None else bias[i * c:(i + 1) * c])
                     .view(b, n, heads, c // heads).transpose(1, 2) for i in range(3))
    qkv = linear(x, weight, bias).reshape(b, n, 3, heads, c // heads)
    return tuple(qkv.permute(2, 0, 3, 1, 4))


def set_packed(flag: Optional[bool]) -> None:
    """Force (True / False) or re-probe (None) the packed-qkv library attention."""
    _PACKED["state"] = flag


def packed_attention(qkv: torch.Tensor) -> Optional[torch.Tensor]:
    """Attention on the packed projection output ``qkv [B, N, 3, H, D]`` -> ``[B, N, H, D]`` through the
    flash-attn library's packed entry point, or None when that is not usable here.  Compared with unbinding q, k, v
    for the generic fused attention this avoids two full-size copies per block and step: the concatenation of
    dq, dk, dv that autograd builds for the packed tensor, and the ``[B, H, N, D] -> [B, N, H * D]`` repacking of
    the output."""
    if _PACKED["state"] is False or not (qkv.is_cuda and qkv.dtype in (torch.bfloat16, torch.float16)):
        return None
    if qkv.shape[-1] > 256 or qkv.shape[-1] % 8:
        return None
    try:
        from flash_attn import flash_attn_qkvpacked_func
        if _PACKED["state"] is None:
            probe = torch.randn(1, 16, 3, 1, 64, device=qkv.device, dtype=torch.bfloat16)
            ref = F.scaled_dot_product_attention(*(t.transpose(1, 2) for t in probe.unbind(2))).transpose(1, 2)
            ok = torch.allclose(flash_attn_qkvpacked_func(probe).float(), ref.float(), rtol=3e-2, atol=3e-2)
            _PACKED["state"] = bool(ok)
            if not ok:
                return None
        return flash_attn_qkvpacked_func(qkv)
    except Exception:   # noqa: BLE001 - library missing or not built for this GPU: use the generic path
        _PACKED["state"] = False
        return None


def _strides3(t: torch.Tensor):
    """(row, head, batch) element strides of a [B, H, N, D] tensor as a ctypes array."""
    return (_c.c_int64 * 3)(t.stride(2), t.stride(1), t.stride(0))


def flash_eligible(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor) -> bool:
    if not (q.is_cuda and q.dtype == k.dtype == v.dtype == torch.bfloat16 and q.dim() == k.dim() == v.dim() == 4):
        return False
    d, dv = q.shape[-1], v.shape[-1]
    if (d, dv) not in ((64, 64), (256, 256)):
        return False
    if d == 256 and not (k.data_ptr() == v.data_ptr() and k.stride() == v.stride()):
        return False
    if q.shape[0] * q.shape[1] > 65535 or k.shape[2] < 1:
        return False
    for t in (q, k, v):
        if t.stride(-1) != 1 or t.data_ptr() % 16 or any(s % 8 for s in t.stride()[:-1]):
            return False
    return True


def flash_fwd(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: Optional[float] = None,
              fixed_max: Optional[float] = None, out_dtype: torch.dtype = torch.bfloat16, want_lse: bool = False
              ) -> Tuple[torch.Tensor, Optional[torch.Tensor]]:
    """``(O, lse)`` for bf16 ``q [B, H, Nq, D]``, ``k [B, H, Nk, D]``, ``v [B, H, Nk, Dv]`` (any strides with a
    contiguous last dimension).  ``O`` is returned as a ``[B, H, Nq, Dv]`` view of a ``[B, Nq, H, Dv]`` buffer, so
    the usual ``o.transpose(1, 2).reshape(B, Nq, H * Dv)`` is free.  ``fixed_max``: an upper bound of
    ``scale * q.k`` known in advance (removes the running-maximum rescaling)."""
    from . import fused as _f
    from . import gemm as _gemm
    b, h, nq, d = q.shape
    nk, dv = k.shape[2], v.shape[3]
    scale = 1.0 / math.sqrt(d) if scale is None else float(scale)
    o = torch.empty((b, nq, h, dv), dtype=out_dtype, device=q.device).transpose(1, 2)
    lse = torch.empty((b * h, nq), dtype=torch.float32, device=q.device) if want_lse else None
    L = _f.lib()
    L.tsp_attn_fwd.restype = _c.c_int
    with _f.on_device(q.device):
        code = L.tsp_attn_fwd(_f._ptr(q), _f._ptr(k), _f._ptr(v), _f._ptr(o), _f._ptr(lse), _c.c_int(b), _c.c_int(h),
                              _c.c_int(nq), _c.c_int(nk), _c.c_int(d), _c.c_int(dv), _strides3(q), _strides3(k),
                              _strides3(v), _strides3(o), _c.c_float(scale),
                              _c.c_float(0.0 if fixed_max is None else float(fixed_max)),
                              _c.c_int(0 if fixed_max is None else 1), _c.c_int(_f._dt(o)),
                              _f._ptr(_gemm._status_word(q.device)), _f._stream())
    _f._check(code, "tsp_attn_fwd")
    _f._count()
    return o, (lse.view(b, h, nq) if want_lse else None)


def _key_mask(mask: torch.Tensor, b: int, nk: int) -> Optional[torch.Tensor]:
    """``mask`` as ``[b or 1, nk]`` when it is boolean and depends on the key (and the batch) alone, else None."""
    if mask.dtype != torch.bool or mask.dim() != 4 or mask.shape[1] != 1 or mask.shape[2] != 1:
        return None
    if mask.shape[0] not in (1, b) or mask.shape[3] != nk or (nk > 1 and mask.stride(3) != 1):
        return None
    return mask[:, 0, 0]


def heads_fwd(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, mask: Optional[torch.Tensor] = None
              ) -> Optional[torch.Tensor]:
    """``softmax(q k^T / 8 + mask) v`` for bf16 ``[B, H, N, 64]`` tensors (any strides with a contiguous last dimension)
    without a gradient, as a ``[B, H, Nq, 64]`` view of a ``[B, Nq, H, 64]`` buffer; None where the kernel does not take
    them.  ``mask``: boolean, True = the key takes part, ``[B or 1, 1, 1, Nk]``; where no key does, all do.  Of keys and values
    that are off, tiles of 128 are not read: a NaN there is without effect, one in another tile is not (its probability, zero,
    times NaN)."""
    from . import fused as _f
    from . import gemm as _gemm
    ts = (q, k, v) if mask is None else (q, k, v, mask)
    if any(_f._wrapped(t) for t in ts) or torch.autograd.forward_ad._current_level >= 0:
        return None
    if q.dim() != 4 or q.shape[-1] != 64 or not flash_eligible(q, k, v) or any(t.device != q.device for t in ts):
        return None
    b, h, nq, d = q.shape
    nk = k.shape[2]
    if k.shape != (b, h, nk, d) or v.shape != k.shape or nk > 4096 or b * h * nq == 0:
        return None
    if any(s <= 0 for t in (q, k, v) for s in t.stride()):
        return None
    m = None
    if mask is not None:
        m = _key_mask(mask, b, nk)
        if m is None:
            return None
    o = torch.empty((b, nq, h, d), dtype=torch.bfloat16, device=q.device)
    L = _f.lib()
    L.tsp_attn_heads_fwd.restype = _c.c_int
    with _f.on_device(q.device):
        code = L.tsp_attn_heads_fwd(_f._ptr(q), _f._ptr(k), _f._ptr(v), _f._ptr(m),
                                    _c.c_int64(0 if m is None or m.shape[0] == 1 else m.stride(0)), _f._ptr(o), _c.c_int(b),
                                    _c.c_int(h), _c.c_int(nq), _c.c_int(nk), _strides3(q), _strides3(k), _strides3(v),
                                    _c.c_float(1.0 / math.sqrt(d)), _f._ptr(_gemm._status_word(q.device)), _f._stream())
    _f._check(code, "tsp_attn_heads_fwd")
    _f._count()
    return o.transpose(1, 2)


def _observed() -> bool:
    """Whether something other than the device is to see the call: a trace, a compilation, a dispatch mode (which a launch
    through ctypes would pass by), or autocast to another type than the kernel's."""
    return (torch.compiler.is_compiling() or torch.jit.is_tracing() or torch._C._len_torch_dispatch_stack() > 0
            or (torch.is_autocast_enabled("cuda") and torch.get_autocast_dtype("cuda") != torch.bfloat16))


def attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, mask: Optional[torch.Tensor] = None,
              dropout_p: float = 0.0) -> torch.Tensor:
    needs_grad = torch.is_grad_enabled() and (q.requires_grad or k.requires_grad or v.requires_grad)
    if ((_TCGEN05 or (_TCGEN05 is None and mask is not None)) and dropout_p == 0.0 and not needs_grad and q.is_cuda
            and not _observed() and k.shape[-2] > 1      # (a single key that is off: the library gives zeros)
            and not (k.shape[-2] <= 32 and q.shape[-2] <= 32 and q.numel() > _FEW_KEYS * q.shape[-2] * q.shape[-1])):
        o = heads_fwd(q, k, v, mask)
        if o is None and _TCGEN05 and mask is None and k.shape[-2] > 4096 and q.shape[-1] == 64 and flash_eligible(q, k, v):
            o = flash_fwd(q, k, v)[0]              # (more keys than the other kernel's masks and tiles are made for)
        if o is not None:
            return o
    return F.scaled_dot_product_attention(q, k, v, attn_mask=mask, dropout_p=dropout_p)
