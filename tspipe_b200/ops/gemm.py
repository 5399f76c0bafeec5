"""Bindings of the tcgen05 / TMEM / TMA GEMM (``csrc/gemm_tcgen05.cu``) and the ops built on it.

``matmul_nt(a, b)`` computes ``a @ b.T`` for row-major bf16 ``a [M, K]`` and ``b [N, K]`` with fp32
accumulation in tensor memory, optional fused ``+ bias`` and GELU epilogue.  ``linear`` is the autograd
wrapper used by the transformer blocks and heads: forward, ``dX = dY W`` and ``dW = dY^T X`` on the CTA-pair
tcgen05 GEMM (operands whose contraction index is the slow one are read in place as MN-major tiles, the weight
gradient is added into the fp32 gradient buffer), the bias gradient on the column-sum kernel.  ``info_nce`` is the MoCo-v3 contrastive loss
(`benchmarks/moco-v3/main.py:147-162`): row-normalised ``q @ k.T / T`` on the tcgen05 kernel followed
by the fused cross-entropy kernel (value + gradient in one launch).

The kernel bounds every barrier wait; a non-zero device status word after a launch means a wait ran
out and the output is invalid - :func:`check_status` raises in that case.
"""
from __future__ import annotations

import ctypes as _c
from typing import Optional

import torch
import torch.nn.functional as F

from . import fused as _f

_status = {}


def _status_word(device) -> torch.Tensor:
    key = (device.type, device.index)
    if key not in _status:
        _status[key] = torch.zeros(1, dtype=torch.int32, device=device)
    return _status[key]


def check_status(device=None) -> None:
    """Synchronising check of the GEMM status word (tests and debugging)."""
    for key, t in _status.items():
        code = int(t.item())
        if code != 0:
            t.zero_()
            raise RuntimeError(f"tcgen05 GEMM on {key}: bounded wait ran out in role {code} "
                               "(1 = TMA producer, 2 = MMA issuer, 3 = epilogue, 4 = MMA issuer on a free accumulator)")


def eligible(x: torch.Tensor, weight: torch.Tensor) -> bool:
    """Shapes and dtypes the tcgen05 linear path takes: bf16 compute (a bf16 input, or bf16 autocast), feature counts
    multiples of 64, at least one full tile of rows."""
    k = x.shape[-1]
    if not (x.is_cuda and weight.is_cuda and weight.dim() == 2):
        return False
    if not (x.dtype == torch.bfloat16 or (torch.is_autocast_enabled() and torch.get_autocast_dtype("cuda") == torch.bfloat16)):
        return False
    return k % 64 == 0 and weight.shape[0] % 64 == 0 and x.numel() // k >= 128 and weight.stride(1) == 1 \
        and weight.stride(0) == k


_two_cta = True     # measured faster than the one-CTA kernel on every ViT / head shape tried


def set_two_cta(on: bool) -> None:
    """Route :func:`matmul_nt` through the two-SM kernel (``cta_group::2``, one 256 x 256 tile per CTA pair)."""
    global _two_cta
    _two_cta = bool(on)


def matmul_nt(a: torch.Tensor, b: torch.Tensor, bias: Optional[torch.Tensor] = None, gelu: bool = False,
              out_dtype: torch.dtype = torch.bfloat16, two_cta: Optional[bool] = None) -> torch.Tensor:
    """``a [M, K] @ b [N, K]^T`` (bf16 operands).  ``two_cta`` picks the CTA-pair kernel for this call
    (default: the module setting, see :func:`set_two_cta`)."""
    assert a.dim() == 2 and b.dim() == 2 and a.shape[1] == b.shape[1]
    a = a if (a.dtype == torch.bfloat16 and a.is_contiguous()) else a.to(torch.bfloat16).contiguous()
    b = b if (b.dtype == torch.bfloat16 and b.is_contiguous()) else b.to(torch.bfloat16).contiguous()
    m, k = a.shape
    n = b.shape[0]
    c = torch.empty(m, n, dtype=out_dtype, device=a.device)
    bf = None if bias is None else bias.detach().float().contiguous()
    epi = 0 if bias is None else (2 if gelu else 1)
    if gelu and bias is None:
        bf, epi = torch.zeros(n, dtype=torch.float32, device=a.device), 2
    L = _f.lib()
    fn = L.tsp_gemm_bf16_tn_2cta if (_two_cta if two_cta is None else two_cta) else L.tsp_gemm_bf16_tn
    fn.restype = _c.c_int
    with _f.on_device(a.device):
        code = fn(_f._ptr(a), _f._ptr(b), _f._ptr(c), _f._ptr(bf), _c.c_int(m), _c.c_int(n), _c.c_int(k),
                  _c.c_int(k), _c.c_int(k), _c.c_int(n), _c.c_int(_f._dt(c)), _c.c_int(epi),
                  _f._ptr(_status_word(a.device)), _f._stream())
    _f._check(code, "tsp_gemm_bf16_tn")
    _f._count()
    return c


_W16 = {}        # id(parameter) -> (parameter, version, bf16 copy); dropped at every optimizer step


def clear_weight_cache() -> None:
    _W16.clear()


def _w16(weight: torch.Tensor) -> torch.Tensor:
    """bf16 copy of a weight matrix, cast once per parameter and optimizer step.  A row slice of a parameter (the q / k
    / v blocks of a fused projection) maps to the same slice of the parameter's copy.  The cache entry holds the
    parameter itself, so an address that is reused by another tensor can never alias an old entry."""
    if weight.dtype == torch.bfloat16 and weight.is_contiguous():
        return weight.detach()
    base = weight._base if weight._base is not None else weight
    if not base.is_contiguous() or base.dtype == torch.bfloat16:
        return weight.detach().to(torch.bfloat16).contiguous()
    if _f.IN_CAPTURE:                   # inside a CUDA graph the cast is part of the graph
        w = _f.recorded_bf16(weight)
        return w if w.is_contiguous() and w.data_ptr() % 16 == 0 else w.clone(memory_format=torch.contiguous_format)
    hit = _W16.get(id(base))
    if hit is None or hit[0] is not base or hit[1] != base._version:
        hit = (base, base._version, base.detach().to(torch.bfloat16))
        _W16[id(base)] = hit
    b16 = hit[2]
    if base is weight:
        return b16
    return b16.as_strided(weight.shape, weight.stride(), weight.storage_offset() - base.storage_offset())


def _column_sums(dy2: torch.Tensor, out: Optional[torch.Tensor] = None, add_to: Optional[torch.Tensor] = None
                 ) -> Optional[torch.Tensor]:
    """fp32 column sums of a matrix (the bias gradient) on the column-sum kernel, in ``out`` when given; with ``add_to``
    they are added to it and None is returned."""
    m, n = dy2.shape
    if n % 8 or n > 8192 or m < 2:
        sums = torch.sum(dy2, 0, dtype=torch.float32)
        if add_to is not None:
            add_to.add_(sums)
            return None
        return sums if out is None else out.copy_(sums)
    sums = add_to if add_to is not None else out if out is not None else \
        torch.empty(n, dtype=torch.float32, device=dy2.device)
    L = _f.lib()
    with _f.on_device(dy2.device):
        _f._check(L.tsp_col_sums(_f._ptr(dy2), _c.c_int64(m), _c.c_int(n), _c.c_int(_f._dt(dy2)), _f._ptr(sums),
                                 _c.c_int(0 if add_to is None else 1), _f._stream()), "tsp_col_sums")
    _f._count()
    return None if add_to is not None else sums


def _column_sums_of(dys, out: torch.Tensor, add: bool) -> None:
    """fp32 column sums of up to three bf16 matrices of one shape, side by side into ``out`` (``add``: on top of it)."""
    m, n = dys[0].shape
    if n % 8 or n > 8192 or m < 2:
        for i, dy in enumerate(dys):
            part = out[i * n: (i + 1) * n]
            _column_sums(dy, *((None, part) if add else (part,)))
        return
    ptrs = (_c.c_void_p * len(dys))(*(t.data_ptr() for t in dys))
    with _f.on_device(out.device):
        _f._check(_f.lib().tsp_col_sums_of(ptrs, _c.c_int(len(dys)), _c.c_int64(m), _c.c_int(n), _c.c_int(_f._dt(dys[0])),
                                           _f._ptr(out), _c.c_int(1 if add else 0), _f._stream()), "tsp_col_sums_of")
    _f._count()


def matmul_nn(a, b: torch.Tensor) -> torch.Tensor:
    """``[a_0 | a_1 | ..] @ b`` (bf16, fp32 accumulation): ``a`` = up to three ``[M, K_i]`` matrices of one width, ``b
    [K, N]`` read in place as MN-major tiles.  ``dX = dY @ W`` of a linear layer, or of layers that share their input."""
    m, n = a[0].shape[0], b.shape[1]
    c = torch.empty((m, n), dtype=torch.bfloat16, device=b.device)
    ptrs = (_c.c_void_p * len(a))(*(t.data_ptr() for t in a))
    L = _f.lib()
    with _f.on_device(b.device):
        code = L.tsp_gemm_bf16_nn_2cta(ptrs, _c.c_int(len(a)), _f._ptr(b), _f._ptr(c), _c.c_int(m), _c.c_int(n),
                                       _c.c_int(b.shape[0]), _c.c_int(a[0].shape[1]), _c.c_int(n), _c.c_int(n),
                                       _f._ptr(_status_word(b.device)), _f._stream())
    _f._check(code, "tsp_gemm_bf16_nn_2cta")
    _f._count()
    return c


def _add_weight_grad(target: torch.Tensor, dys, x2: torch.Tensor) -> None:
    """``target += [dy_0 | dy_1 | ..]^T @ x2`` (fp32 ``[N, K]``, contiguous) for up to three gradients of one width."""
    n, k = target.shape
    ptrs = (_c.c_void_p * len(dys))(*(t.data_ptr() for t in dys))
    L = _f.lib()
    with _f.on_device(x2.device):
        code = L.tsp_gemm_bf16_wgrad_2cta(ptrs, _c.c_int(len(dys)), _f._ptr(x2), _f._ptr(target), _c.c_int(n), _c.c_int(k),
                                          _c.c_int(x2.shape[0]), _c.c_int(n // len(dys)), _c.c_int(k), _c.c_int(k),
                                          _f._ptr(_status_word(x2.device)), _f._stream())
    _f._check(code, "tsp_gemm_bf16_wgrad_2cta")
    _f._count()


def _bf16_rows(t: torch.Tensor, width: int) -> torch.Tensor:
    """``t`` as a contiguous, 16-byte aligned bf16 ``[rows, width]`` matrix."""
    t2 = t.reshape(-1, width)
    if t2.dtype != torch.bfloat16 or not t2.is_contiguous():
        t2 = t2.to(torch.bfloat16).contiguous()
    return t2 if t2.data_ptr() % 16 == 0 else t2.clone()


def _grad_target(weight: torch.Tensor):
    """The fp32 buffer that a weight gradient may be added to in place, or None."""
    from . import conv as _conv
    g = weight.grad if weight.is_leaf else None
    if (_conv._ACCUMULATE_IN_PLACE and g is not None and g.dtype == torch.float32 and g.is_contiguous()
            and g.shape == weight.shape and g.data_ptr() % 16 == 0):
        return g
    return None


class _Linear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight, bias):
        x2 = x.reshape(-1, x.shape[-1])
        if x2.dtype != torch.bfloat16 or not x2.is_contiguous():
            x2 = x2.to(torch.bfloat16).contiguous()
        y = matmul_nt(x2, _w16(weight), bias)
        ctx.save_for_backward(x2, weight)
        ctx.has_bias = bias is not None
        ctx.bias = bias if _f.IN_CAPTURE else None
        ctx.in_shape = x.shape
        ctx.dtypes = (x.dtype, weight.dtype, None if bias is None else bias.dtype)
        return y.view(*x.shape[:-1], weight.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, weight = ctx.saved_tensors
        n, k = weight.shape
        dy2 = _bf16_rows(dy, n)
        dx = dw = db = None
        if ctx.needs_input_grad[0]:
            dx = matmul_nn([dy2], _w16(weight)).view(ctx.in_shape)
            if ctx.dtypes[0] != torch.bfloat16:
                dx = dx.to(ctx.dtypes[0])
        if ctx.needs_input_grad[1]:
            target = _grad_target(weight)          # the kernel adds into the existing gradient buffer
            if target is None:
                target = torch.zeros((n, k), dtype=torch.float32, device=x2.device)
                dw = target
            _add_weight_grad(target, [dy2], x2)
            if dw is not None and weight.dtype != torch.float32:
                dw = target.to(weight.dtype)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            db = _column_sums(dy2, add_to=_f.recorded_grad(ctx.bias))
            db = None if db is None else db.to(ctx.dtypes[2])
        return dx, dw, db


class _LinearQKV(torch.autograd.Function):
    """``q, k, v = (x W_i^T + b_i)`` with ``W_i``, ``b_i`` the row blocks of a fused projection: one GEMM with three
    destinations; in the backward one GEMM for dX over the three gradients side by side (fp32 accumulation across them, no sums of bf16
    partial results) and one for the fused weight's gradient."""

    @staticmethod
    def forward(ctx, x, weight, bias):
        x2 = _bf16_rows(x, x.shape[-1])
        w16 = _w16(weight)
        c = weight.shape[0] // 3
        ctx.save_for_backward(x2, weight)
        ctx.in_shape, ctx.dtypes = x.shape, (x.dtype, weight.dtype, None if bias is None else bias.dtype)
        ctx.bias = bias if _f.IN_CAPTURE else None
        m, k = x2.shape
        out = [torch.empty((m, c), dtype=torch.bfloat16, device=x2.device) for _ in range(3)]
        bf = None if bias is None else bias.detach().float().contiguous()
        ptrs = (_c.c_void_p * 3)(*(t.data_ptr() for t in out))
        with _f.on_device(x2.device):
            code = _f.lib().tsp_gemm_bf16_tn_2cta_split(_f._ptr(x2), _f._ptr(w16), ptrs, _c.c_int(3), _f._ptr(bf), _c.c_int(m),
                                                        _c.c_int(3 * c), _c.c_int(k), _c.c_int(k), _c.c_int(k), _c.c_int(c),
                                                        _f._ptr(_status_word(x2.device)), _f._stream())
        _f._check(code, "tsp_gemm_bf16_tn_2cta_split")
        _f._count()
        return tuple(t.view(*x.shape[:-1], c) for t in out)

    @staticmethod
    def backward(ctx, *dys):
        x2, weight = ctx.saved_tensors
        n, k = weight.shape
        c = n // 3
        dy2 = [_bf16_rows(dy, c) for dy in dys]
        dx = dw = db = None
        if ctx.needs_input_grad[0]:
            dx = matmul_nn(dy2, _w16(weight)).view(ctx.in_shape)
            if ctx.dtypes[0] != torch.bfloat16:
                dx = dx.to(ctx.dtypes[0])
        if ctx.needs_input_grad[1]:
            target = _grad_target(weight)
            if target is None:
                target = torch.zeros((n, k), dtype=torch.float32, device=x2.device)
                dw = target
            _add_weight_grad(target, dy2, x2)
            if dw is not None and weight.dtype != torch.float32:
                dw = target.to(weight.dtype)
        if ctx.dtypes[2] is not None and ctx.needs_input_grad[2]:
            gb = _f.recorded_grad(ctx.bias)
            if gb is None:
                db = torch.empty(n, dtype=torch.float32, device=x2.device)
            _column_sums_of(dy2, db if db is not None else gb, db is None)
            db = None if db is None else db.to(ctx.dtypes[2])
        return dx, dw, db


class _LinearGelu(torch.autograd.Function):
    """``gelu(x W^T + b)``: the GEMM's epilogue forms the activation from the rounded product, which is kept for the backward
    only.  Backward: the activation's derivative as one elementwise pass, then the linear layer's products."""

    @staticmethod
    def forward(ctx, x, weight, bias, grads):
        x2 = _bf16_rows(x, x.shape[-1])
        (m, k), n = x2.shape, weight.shape[0]
        bf = _f.param_f32(bias)
        act = torch.empty((m, n), dtype=torch.bfloat16, device=x2.device)
        h = torch.empty_like(act) if grads and any(ctx.needs_input_grad) else None
        with _f.on_device(x2.device):
            code = _f.lib().tsp_gemm_bf16_tn_gelu_2cta(_f._ptr(x2), _f._ptr(_w16(weight)), _f._ptr(h), _f._ptr(act),
                                                       _f._ptr(bf), _c.c_int(m), _c.c_int(n), _c.c_int(k), _c.c_int(k),
                                                       _c.c_int(k), _c.c_int(n), _f._ptr(_status_word(x2.device)),
                                                       _f._stream())
        _f._check(code, "tsp_gemm_bf16_tn_gelu_2cta")
        _f._count()
        if h is not None:
            ctx.save_for_backward(x2, weight, h, bf)
        ctx.in_shape, ctx.dtypes = x.shape, (x.dtype, weight.dtype, bias.dtype)
        ctx.bias = bias if _f.IN_CAPTURE else None
        return act.view(*x.shape[:-1], n)

    @staticmethod
    def backward(ctx, dy):
        x2, weight, h, bf = ctx.saved_tensors
        n, k = weight.shape
        dy2 = _bf16_rows(dy, n)
        dh = torch.empty_like(h)
        sums = db = None
        if ctx.needs_input_grad[2]:                # the bias gradient: column sums of dh, formed as it is written
            sums = _f.recorded_grad(ctx.bias)
            if sums is None:
                sums = db = torch.zeros(n, dtype=torch.float32, device=h.device)
        with _f.on_device(h.device):
            if sums is None:
                _f._check(_f.lib().tsp_gelu_bwd(_f._ptr(dy2), _f._ptr(h), _f._ptr(bf), _f._ptr(dh), _c.c_int64(h.numel()),
                                                _c.c_int(n), _c.c_int(_f._dt(h)), _f._stream()), "tsp_gelu_bwd")
            else:
                _f._check(_f.lib().tsp_gelu_bwd_sums(_f._ptr(dy2), _f._ptr(h), _f._ptr(bf), _f._ptr(dh), _f._ptr(sums),
                                                     _c.c_int64(h.shape[0]), _c.c_int(n), _c.c_int(_f._dt(h)), _f._stream()),
                          "tsp_gelu_bwd_sums")
        _f._count()
        dx = dw = None
        if ctx.needs_input_grad[0]:
            dx = matmul_nn([dh], _w16(weight)).view(ctx.in_shape)
            if ctx.dtypes[0] != torch.bfloat16:
                dx = dx.to(ctx.dtypes[0])
        if ctx.needs_input_grad[1]:
            target = _grad_target(weight)
            if target is None:
                target = torch.zeros((n, k), dtype=torch.float32, device=x2.device)
                dw = target
            _add_weight_grad(target, [dh], x2)
            if dw is not None and weight.dtype != torch.float32:
                dw = target.to(weight.dtype)
        return dx, dw, None if db is None else db.to(ctx.dtypes[2]), None


def linear_gelu(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor) -> torch.Tensor:
    """``gelu(x @ weight^T + bias)``; see :class:`_LinearGelu`."""
    return _LinearGelu.apply(x, weight, bias, torch.is_grad_enabled())


def linear_qkv(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None):
    """``(q, k, v)`` of a fused projection ``weight [3C, K]``; see :class:`_LinearQKV`."""
    return _LinearQKV.apply(x, weight, bias)


def linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    host = _f.eager() if _two_cta and type(x) is torch.Tensor else None
    if host is not None:
        y = host.linear(x, weight, _w16(weight), bias, _status_word(x.device))
        if y is not None:
            return y
    return _Linear.apply(x, weight, bias)


def info_nce(q: torch.Tensor, k: torch.Tensor, temp: float, k_all: Optional[torch.Tensor] = None,
             label_offset: int = 0) -> torch.Tensor:
    """``CE(normalize(q) @ normalize(k_all)^T / T, arange(N) + label_offset) * 2T``.  ``k_all`` defaults to
    ``k`` (single replica); with data-parallel replicas it is the concatenation of every replica's keys
    (gathered through peer memory, :func:`tspipe_b200.parallel.keys.gather_keys`)."""
    keys = k if k_all is None else k_all
    qn = F.normalize(q.float(), dim=1)
    kn = F.normalize(keys.detach().float(), dim=1)
    n = q.shape[0]
    if _fused_nce and k_all is None and label_offset == 0 and q.is_cuda and q.shape[1] == 256 and n >= 128:
        return _FusedNCE.apply(qn, kn.to(torch.bfloat16), float(temp))
    if q.is_cuda and q.shape[1] % 8 == 0 and q.shape[1] >= 64 and n >= 128 and keys.shape[0] >= 64:
        logits = _ScaledLogits.apply(qn, kn, 1.0 / temp)
    else:
        logits = qn @ kn.t() / temp
    labels = torch.arange(n, device=q.device) + label_offset
    if q.is_cuda:
        return _f.cross_entropy(logits, labels) * (2 * temp)
    return F.cross_entropy(logits, labels) * (2 * temp)


def matmul_nt_gathered(a: torch.Tensor, b_sources, rows_per_b: int, out_dtype: torch.dtype = torch.float32) -> torch.Tensor:
    """``a [M, K] @ concat(b_sources)^T`` where every source is a ``[rows_per_b, K]`` bf16 buffer that may live on
    another GPU (peer-mapped): each CTA pulls its key tile from the owning GPU with its own TMA load."""
    from ..comm.peer import pointer_table
    a = a if (a.dtype == torch.bfloat16 and a.is_contiguous()) else a.to(torch.bfloat16).contiguous()
    m, k = a.shape
    r = len(b_sources)
    c = torch.empty(m, r * rows_per_b, dtype=out_dtype, device=a.device)
    L = _f.lib()
    L.tsp_gemm_bf16_tn_gathered_b.restype = _c.c_int
    with _f.on_device(a.device):
        code = L.tsp_gemm_bf16_tn_gathered_b(_f._ptr(a), pointer_table(b_sources), _c.c_int(r), _c.c_int(rows_per_b),
                                             _f._ptr(c), _c.c_int(m), _c.c_int(k), _c.c_int(k), _c.c_int(k),
                                             _c.c_int(r * rows_per_b), _c.c_int(_f._dt(c)),
                                             _f._ptr(_status_word(a.device)), _f._stream())
    _f._check(code, "tsp_gemm_bf16_tn_gathered_b")
    _f._count()
    return c


class _GatheredLogits(torch.autograd.Function):
    """Contrastive logits against the keys of ALL replicas, read in place from the GPUs that own them."""

    @staticmethod
    def forward(ctx, qn, views, table, rows_per_b, like):
        ctx.table, ctx.r, ctx.like, ctx.adtype = table, len(views), like, qn.dtype
        return matmul_nt_gathered(qn, views, rows_per_b)

    @staticmethod
    def backward(ctx, g):
        from ..parallel.keys import gather_blocks
        k_all = gather_blocks(ctx.table, ctx.r, ctx.like)           # [R*n, D] (already scaled by 1/T)
        return matmul_nt(g, k_all.t().contiguous(), out_dtype=torch.float32).to(ctx.adtype), None, None, None, None


def info_nce_replicas(q: torch.Tensor, k: torch.Tensor, temp: float):
    """InfoNCE across data-parallel replicas with the key all-gather folded into the logit GEMM.  Returns None
    when the fused path does not apply (no replicas, CPU, shapes off the tile grid)."""
    from ..parallel.keys import exchange_for
    from ..runtime import context
    ctx = context.current()
    n, d = q.shape
    if ctx is None or ctx.topo.dp <= 1 or not q.is_cuda or d % 8 or d < 64 or n % 128:
        return None
    if _fused_nce and d == 256 and ctx.topo.dp <= 8:
        # attention-style kernel: every CTA streams key tiles from all replicas' buffers; no logits in memory
        kn16 = F.normalize(k.detach().float(), dim=1).to(torch.bfloat16).contiguous()
        ex = exchange_for(kn16, "moco_keys_bf16")
        if ex is not None:
            views, _ = ex.publish(kn16)
            return _FusedNCEGathered.apply(F.normalize(q.float(), dim=1), kn16, views, float(temp))
    kn = (F.normalize(k.detach().float(), dim=1) * (1.0 / temp)).to(torch.bfloat16).contiguous()
    ex = exchange_for(kn, "moco_keys_scaled_bf16")
    if ex is None:
        return None
    views, table = ex.publish(kn)
    qn = F.normalize(q.float(), dim=1)
    logits = _GatheredLogits.apply(qn, views, table, n, kn)
    labels = torch.arange(n, device=q.device) + n * ctx.topo.replica
    return _f.cross_entropy(logits, labels) * (2 * temp)


_fused_nce = True


def set_fused_nce(on: bool) -> None:
    """Contrastive loss through the fused attention kernel (no N x N logits in memory) when it applies."""
    global _fused_nce
    _fused_nce = bool(on)


_NCE_KEY_SPLIT = True


def set_nce_key_split(flag: bool) -> None:
    """Split the keys of the fused contrastive loss over the grid (default) or run one CTA per query tile."""
    global _NCE_KEY_SPLIT
    _NCE_KEY_SPLIT = bool(flag)


def nce_key_chunks(n_queries: int, n_keys: int, target_ctas: int = 120) -> int:
    """Into how many chunks the fused contrastive loss splits the keys so that (query tiles) x (chunks) fills the
    GPU: the smallest power of two that reaches ``target_ctas`` CTAs, as long as every chunk keeps at least two
    64-row key tiles and the keys divide evenly."""
    if not _NCE_KEY_SPLIT:
        return 1
    tiles = -(-n_queries // 128)
    c = 1
    while tiles * c < target_ctas and n_keys % (2 * c * 64) == 0 and n_keys // (2 * c) >= 128:
        c *= 2
    return c


class _FusedNCE(torch.autograd.Function):
    """``2T * mean_i(logsumexp_j(q_i.k_j / T) - q_i.k_i / T)`` for unit-norm rows, forward and backward from ONE
    pass of the fused attention kernel with V = K: ``lse`` gives the loss, ``O_i = sum_j p_ij k_j`` the gradient
    ``dL/dq_i = 2/N (O_i - k_i)``.  Cosine logits are bounded by 1/T, so the kernel runs without rescaling."""

    @staticmethod
    def forward(ctx, qn, kn16, temp):
        from .attention import flash_fwd
        n, d = qn.shape
        nk = kn16.shape[0]
        q16 = qn.to(torch.bfloat16)
        c = nce_key_chunks(n, nk)
        if c == 1:
            o, lse = flash_fwd(q16.view(1, 1, n, d), kn16.view(1, 1, -1, d), kn16.view(1, 1, -1, d), scale=1.0 / temp,
                               fixed_max=1.0 / temp, out_dtype=torch.float32, want_lse=True)
            o, lse = o.reshape(n, d), lse.view(n)
        else:
            # Keys split over the grid: chunk c of the keys is "head" c of the kernel's (query tile, head) grid, every
            # head sees the same queries.  Each CTA returns its chunk's softmax-weighted key sum and log-sum-exp
            # (exact: the scores are bounded by 1/T, so all chunks use the same fixed maximum); the chunks are then
            # merged with their softmax weights.
            q_rep = q16.unsqueeze(0).expand(c, n, d).contiguous().view(1, c, n, d)
            k_chunks = kn16.view(1, c, nk // c, d)
            o_part, lse_part = flash_fwd(q_rep, k_chunks, k_chunks, scale=1.0 / temp, fixed_max=1.0 / temp,
                                         out_dtype=torch.float32, want_lse=True)
            lse_part = lse_part.view(c, n)
            lse = torch.logsumexp(lse_part, dim=0)
            w = torch.exp(lse_part - lse)                                   # [c, n], sums to 1 over the chunks
            o = torch.einsum("cn,cnd->nd", w, o_part[0])
        pos = (q16.float() * kn16[:n].float()).sum(1) / temp
        ctx.save_for_backward(o, kn16)
        ctx.n, ctx.qdtype = n, qn.dtype
        return (lse - pos).mean() * (2 * temp)

    @staticmethod
    def backward(ctx, g):
        o, kn16 = ctx.saved_tensors
        return ((o - kn16[: ctx.n].float()) * (g * 2.0 / ctx.n)).to(ctx.qdtype), None, None


def nce_pair_chunks(n: int, target_ctas: int = 148):
    """``(rows per chunk, chunks)`` of the keys for the two-pair loss: 64-row key tiles dealt to as many chunks as bring
    (2 pairs) x (128-query tiles) x (chunks) closest below ``target_ctas`` CTAs, two tiles per chunk at least."""
    tiles_q, tiles_k = -(-n // 128), -(-n // 64)
    c = max(1, min(target_ctas // (2 * tiles_q), tiles_k // 2)) if _NCE_KEY_SPLIT else 1
    per = -(-tiles_k // c)
    return per * 64, -(-tiles_k // per)


class _NCEPair(torch.autograd.Function):
    """Both directions of the symmetric contrastive loss: unit-norm bf16 rows, the fused attention kernel with V = K over
    (pair, key chunk, query tile), and one pass that merges the chunks into the loss and the gradient with respect to the
    queries."""

    @staticmethod
    def forward(ctx, q1, q2, k1, k2, temp):
        n, d = q1.shape
        chunk, c = nce_pair_chunks(n)
        dev = q1.device
        q16 = torch.empty((2, n, d), dtype=torch.bfloat16, device=dev)
        k16 = torch.empty((2, c * chunk, d), dtype=torch.bfloat16, device=dev)
        o = torch.empty((2, c, n, d), dtype=torch.float32, device=dev)
        lse = torch.empty(2 * c * n + 4, dtype=torch.float32, device=dev)      # and the loss's 64-bit sum
        loss = torch.empty((), dtype=torch.float32, device=dev)
        gq = torch.empty((2, n, d), dtype=q1.dtype, device=dev)
        L = _f.lib()
        with _f.on_device(dev):
            code = L.tsp_nce_pair(_f._ptr(q1), _f._ptr(k1), _f._ptr(q2), _f._ptr(k2), _c.c_int(n), _c.c_int(_f._dt(q1)),
                                  _c.c_int(chunk), _c.c_int(c), _c.c_float(temp), _f._ptr(q16), _f._ptr(k16), _f._ptr(o),
                                  _f._ptr(lse), _f._ptr(loss), _f._ptr(gq), _f._ptr(_status_word(dev)), _f._stream())
        _f._check(code, "tsp_nce_pair")
        _f._count(3)
        _f.save_gradient(ctx, gq)
        return loss

    @staticmethod
    def backward(ctx, gout):
        (gq,) = ctx.saved_tensors
        g1, g2 = _f._scaled(gq, gout, ctx.own).unbind(0)
        need = ctx.needs_input_grad
        return g1 if need[0] else None, g2 if need[1] else None, None, None, None


def info_nce_pair(q1: torch.Tensor, k1: torch.Tensor, q2: torch.Tensor, k2: torch.Tensor, temp: float
                  ) -> Optional[torch.Tensor]:
    """``info_nce(q1, k1, temp) + info_nce(q2, k2, temp)`` of one replica from three launches, or None where they do not
    apply: 256 columns and at least one query tile of plain contiguous tensors, a temperature whose ``exp(-2 / T)`` is
    far from underflow."""
    if not (_fused_nce and q1.is_cuda and q1.dim() == 2 and q1.shape[1] == 256 and q1.shape[0] >= 128 and temp >= 0.05
            and q1.dtype in (torch.float32, torch.bfloat16)):
        return None
    for t in (q1, k1, q2, k2):
        if not (t.shape == q1.shape and t.dtype == q1.dtype and t.device == q1.device and t.is_contiguous()
                and t.data_ptr() % 16 == 0):
            return None
    host = _f.eager() if type(q1) is torch.Tensor and type(q2) is torch.Tensor else None
    if host is not None:
        loss = host.nce_pair(q1, q2, k1, k2, float(temp), *nce_pair_chunks(q1.shape[0]), _status_word(q1.device))
        if loss is not None:
            return loss
    k1, k2 = (t.detach() if t.requires_grad else t for t in (k1, k2))
    return _NCEPair.apply(q1, q2, k1, k2, float(temp))


class _FusedNCEGathered(torch.autograd.Function):
    """:class:`_FusedNCE` against the keys of ALL replicas, read in place from the GPUs that own them (positives
    are the local keys: row i of this replica pairs with key ``i + n * replica`` of the concatenation)."""

    @staticmethod
    def forward(ctx, qn, kn16, views, temp):
        from ..comm.peer import pointer_table
        n, d = qn.shape
        q16 = qn.to(torch.bfloat16).contiguous()
        o = torch.empty(n, d, dtype=torch.float32, device=qn.device)
        lse = torch.empty(n, dtype=torch.float32, device=qn.device)
        L = _f.lib()
        L.tsp_attn_nce_gathered.restype = _c.c_int
        with _f.on_device(qn.device):
            code = L.tsp_attn_nce_gathered(_f._ptr(q16), pointer_table(views), _c.c_int(len(views)), _c.c_int(n),
                                           _f._ptr(o), _f._ptr(lse), _c.c_int(n), _c.c_float(1.0 / temp),
                                           _c.c_float(1.0 / temp), _f._ptr(_status_word(qn.device)), _f._stream())
        _f._check(code, "tsp_attn_nce_gathered")
        _f._count()
        pos = (q16.float() * kn16.float()).sum(1) / temp
        ctx.save_for_backward(o, kn16)
        ctx.n, ctx.qdtype = n, qn.dtype
        return (lse - pos).mean() * (2 * temp)

    @staticmethod
    def backward(ctx, g):
        o, kn16 = ctx.saved_tensors
        return ((o - kn16.float()) * (g * 2.0 / ctx.n)).to(ctx.qdtype), None, None, None


class _ScaledLogits(torch.autograd.Function):
    """``scale * a @ b^T`` in fp32 on the tcgen05 kernel; gradient w.r.t. ``a`` only."""

    @staticmethod
    def forward(ctx, a, b, scale):
        bb = (b * scale).to(torch.bfloat16)
        ctx.save_for_backward(bb)
        ctx.adtype = a.dtype
        return matmul_nt(a.to(torch.bfloat16), bb, out_dtype=torch.float32)

    @staticmethod
    def backward(ctx, g):
        (bb,) = ctx.saved_tensors
        # dA = g @ (scale*b): [N, M] x [M, D] -> operands as (g, (scale*b)^T) for the TN kernel
        return matmul_nt(g, bb.t().contiguous(), out_dtype=torch.float32).to(ctx.adtype), None, None
