"""Python bindings and autograd wrappers of the sm_100a kernels in ``csrc/``.

Every wrapper runs on the current CUDA stream.  ``LAUNCHES`` counts kernel launches issued
through this module (benchmarks report it).  The module raises instead of falling back when the
library cannot be loaded on a CUDA machine.
"""
from __future__ import annotations

import ctypes
import sys
import types
import weakref
from typing import Optional, Sequence

import torch

from . import build as _build

_launches = 0         # by the functions of this package; LAUNCHES adds those of the C++ functions
_lib = None
_host = None
_c = ctypes


def available() -> bool:
    return torch.cuda.is_available()


def lib():
    global _lib
    if _lib is None:
        L = _build.load()
        for name in ("tsp_ema_update", "tsp_lars_step", "tsp_lars_step_ordered", "tsp_lars_norms", "tsp_lars_apply", "tsp_adamw_step",
                     "tsp_sgd_step", "tsp_byol_loss", "tsp_cosine_loss", "tsp_kd_ce_loss", "tsp_layernorm_fwd",
                     "tsp_layernorm_bwd", "tsp_layernorm_bwd_blocks", "tsp_gelu_fwd", "tsp_gelu_bwd"):
            getattr(L, name).restype = _c.c_int
        # declared argument types: plain numbers at a call, an object per argument less where a whole loss takes 100 us of host
        v, i, f = _c.c_void_p, _c.c_int, _c.c_float
        L.tsp_kd_ce_loss.argtypes = [v] * 4 + [i] * 4 + [f] * 3 + [v] * 4
        L.tsp_distil_loss.argtypes = [v] * 4 + [i] * 4 + [f] * 3 + [v] * 2 + [i] * 2 + [f] + [v] * 5
        L.tsp_byol_loss_pair.argtypes = [v] * 4 + [i] * 3 + [f] + [v] * 4
        L.tsp_cosine_loss.argtypes = [v] * 3 + [i] * 3 + [f] + [v] * 4
        L.tsp_scale.argtypes = [v] * 3 + [_c.c_int64, i, v]
        _lib = L
    return _lib


def set_sm_reserve(n: int) -> None:
    """Leave ``n`` SMs free of the persistent kernels (convolutions, GEMMs, attention, the vocabulary loss, the LARS step)
    so that communication kernels
    that become ready while one of them runs - NCCL sends / receives of the stage links, peer reductions on a side
    stream - find an SM at once instead of when the persistent kernel ends."""
    lib().tsp_set_sm_reserve(_c.c_int(int(n)))


def _count(n: int = 1) -> None:
    global _launches
    _launches += n


class _Counting(types.ModuleType):
    @property
    def LAUNCHES(self) -> int:
        return _launches + (0 if _host is None else _host.launches())

    @LAUNCHES.setter
    def LAUNCHES(self, n: int) -> None:
        global _launches
        _launches = n - (0 if _host is None else _host.launches())


sys.modules[__name__].__class__ = _Counting


def eager():
    """The C++ autograd functions (``csrc/host/eager.cpp``) for a call that is made eagerly; None while a stage is being
    recorded, whose backward adds small gradients in place, under a trace, which sees the calls of the Python functions, and where
    they cannot be built."""
    global _host
    if IN_CAPTURE or torch._C._get_tracing_state() is not None or torch.compiler.is_compiling():
        return None
    if _host is None:
        from . import conv
        lib()
        _host = _build.load_host()
        if _host is not None:
            _host.set_accumulate(conv._ACCUMULATE_IN_PLACE)
    return _host


def _ptr(t: Optional[torch.Tensor]):
    return _c.c_void_p(0 if t is None else t.data_ptr())


def _raw_stream() -> int:
    """Raw handle of the current stream of the current device (the launchers' last argument)."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _stream():
    return _c.c_void_p(_raw_stream())


IN_CAPTURE = 0          # > 0 while a stage is being recorded into a CUDA graph


class capturing:
    """While a stage is recorded into a CUDA graph the per-step caches of derived tensors (bf16 weight copies) are
    bypassed: what the graph needs it must compute itself at every replay."""

    def __enter__(self):
        global IN_CAPTURE
        IN_CAPTURE += 1
        self.key = _stream_key()
        self.outer = _RECORDINGS.get(self.key)
        _RECORDINGS[self.key] = _Recording()
        return self

    def __exit__(self, *exc):
        global IN_CAPTURE
        IN_CAPTURE -= 1
        if self.outer is None:
            _RECORDINGS.pop(self.key, None)
        else:
            _RECORDINGS[self.key] = self.outer
        return False


class _Recording:
    """What the launches of one recording share: bf16 copies of whole flat parameter buffers and what is left of its block of
    zeroed floats."""

    def __init__(self):
        self.copies, self.zeros = {}, None


# recordings by the stream that is being recorded: the backward's launches come from autograd's own thread, on that stream
_RECORDINGS = {}


def _stream_key():
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice()) if torch.cuda.is_available() else None


def _recording() -> Optional[_Recording]:
    return _RECORDINGS.get(_stream_key()) if IN_CAPTURE else None


def zeroed(n: int, device) -> torch.Tensor:
    """``n`` zeroed floats for a kernel that adds its sums to them.  In a recording they come from blocks that one launch
    zeroes for many layers (at every replay, before the first of them)."""
    rec = _recording()
    if rec is None or n > 8192:
        return torch.zeros(n, dtype=torch.float32, device=device)
    if rec.zeros is None or rec.zeros.numel() < n or rec.zeros.device != device:
        rec.zeros = torch.zeros(1 << 16, dtype=torch.float32, device=device)
    out = rec.zeros[:n]
    rec.zeros = rec.zeros[(n + 3) // 4 * 4:]   # 16-byte aligned pieces
    return out


_FLAT_COPY_MAX = 32 << 20
_FLAT_PARAMS = weakref.WeakValueDictionary()      # every living FlatParams of fp32, by its id


def register_flat(flat) -> None:
    """``flat`` (:class:`~tspipe_b200.runtime.state.FlatParams`) holds parameters that may be cast together."""
    _FLAT_PARAMS[id(flat)] = flat


def recorded_bf16(weight: torch.Tensor) -> torch.Tensor:
    """bf16 copy of a parameter for a graph under recording, with the parameter's strides.  The parameters of a
    ``FlatParams`` are cast together, once per recording: a cast per parameter is a launch per parameter, 2.4 us each for the
    52 convolution weights of a ResNet-50 against 21 us for the whole buffer.  The copy (two bytes a parameter, 64 MB at
    most) lives as long as the recording, where single casts are freed layer by layer.  Cast singly: larger buffers, whose
    casts are bound by memory one by one; tensors that are no parameter of such a buffer (a computed weight may be freed within
    the recording and its address used again); and a parameter written in place since the buffer was cast (by its version, as in
    the caches of eager calls)."""
    w = weight.detach()
    rec = _recording()
    owner = weight._base if weight._base is not None else weight
    if rec is None or w.dtype != torch.float32:
        return w.to(torch.bfloat16)
    store = w.untyped_storage().data_ptr()
    for ref in _FLAT_PARAMS.valuerefs():
        flat = ref()
        if flat is not None and flat.data.untyped_storage().data_ptr() == store \
                and flat.total <= _FLAT_COPY_MAX:
            if flat not in rec.copies:
                rec.copies[flat] = (flat.data.to(torch.bfloat16), {id(p): p._version for p in flat.params})
            copy, versions = rec.copies[flat]
            if versions.get(id(owner)) == owner._version:
                return copy.as_strided(w.shape, w.stride(), w.storage_offset() - flat.data.storage_offset())
    return w.to(torch.bfloat16)


def adds_in_place(p: Optional[torch.Tensor]) -> bool:
    """Whether a backward adds a parameter's gradient where it lies instead of handing it to autograd: on a stream whose
    launches are being recorded (elsewhere, also on other threads meanwhile, the gradient may have been asked for by name),
    for a leaf without hooks that want to see it."""
    return (_recording() is not None and p is not None and p.is_leaf and p.requires_grad
            and not p._backward_hooks and not p._post_accumulate_grad_hooks)


def recorded_grad(p: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """The fp32 gradient buffer of a parameter that a backward adds to in place, or None."""
    g = p.grad if adds_in_place(p) else None
    return g if g is not None and g.dtype == torch.float32 and g.is_contiguous() and g.shape == p.shape else None


class _Current:
    def __enter__(self):
        return self

    def __exit__(self, *exc):
        return False


_CURRENT = _Current()


def on_device(device):
    """``with on_device(t.device):`` makes the tensor's device current for the launches inside.  Free when it already
    is (every launch of a training step: the executor thread and autograd's device thread both run with their device
    current), so the per-launch cost of the general context manager is only paid when it does something."""
    idx = device.index
    if idx is None or torch._C._cuda_getDevice() == idx:
        return _CURRENT
    return torch.cuda.device(idx)


def _check(code: int, what: str) -> None:
    if code != 0:
        raise RuntimeError(f"{what} failed with code {code}")


def param_f32(p: torch.Tensor) -> torch.Tensor:
    """A weight or bias vector as the kernels read it: fp32, contiguous, on a 16-byte boundary (a parameter may be a slice of
    any vector)."""
    t = p.detach()
    if t.dtype != torch.float32 or not t.is_contiguous():
        t = t.float().contiguous()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _dt(t: torch.Tensor) -> int:
    if t.dtype == torch.float32:
        return 0
    if t.dtype == torch.bfloat16:
        return 1
    raise TypeError(f"unsupported dtype {t.dtype}")


# ---------------------------------------------------------------------------------------------
# flat-buffer updates
# ---------------------------------------------------------------------------------------------
@torch.no_grad()
def ema_update_(teacher: torch.Tensor, student: torch.Tensor, momentum: float,
                bf16_shadow: Optional[torch.Tensor] = None) -> None:
    """``teacher = m*teacher + (1-m)*student`` in place (fp32, contiguous).  ``student`` may be a
    view of another GPU's memory mapped into this process."""
    assert teacher.dtype == torch.float32 and student.dtype == torch.float32
    assert teacher.is_contiguous() and student.is_contiguous() and teacher.numel() == student.numel()
    if teacher.numel() == 0:
        return
    with on_device(teacher.device):
        _check(lib().tsp_ema_update(_ptr(teacher), _ptr(student), _c.c_int64(teacher.numel()),
                                    _c.c_float(momentum), _ptr(bf16_shadow), _stream()), "tsp_ema_update")
    _count()


CHUNK = 16384


def build_chunks(offsets: Sequence[int], numels: Sequence[int], device, lo: int = 0, hi: Optional[int] = None
                 ) -> torch.Tensor:
    """Chunk table ``[n_chunks, 3] = (segment, begin, length)`` restricted to flat range ``[lo, hi)``."""
    rows = []
    for s, (off, n) in enumerate(zip(offsets, numels)):
        a, b = max(off, lo), min(off + n, hi if hi is not None else off + n)
        pos = a
        while pos < b:
            ln = min(CHUNK, b - pos)
            rows.append((s, pos, ln))
            pos += ln
    if not rows:
        return torch.zeros((0, 3), dtype=torch.int64, device=device)
    return torch.tensor(rows, dtype=torch.int64, device=device)


# LARS with norms and updates in one launch (:class:`LarsOrder`): from this many chunks on over all buffers of a step
# (80 MB), i.e. where they do not stay in L2 from one step to the next.
LARS_ORDERED = 1280
# Pieces of p and g (64 KB) between the norms and the update of a piece: 50 MB of L2.  Blocks hold 592 pieces and as many
# tickets; with less between, updates wait for norms (592: 165 us where 769 takes 144), with more the time creeps up (1776: 147).
LARS_LAG, LARS_PIECE = 768, 8192


class LarsOrder:
    """The order in which one launch forms the norms and makes the updates of a LARS step, and its workspace."""

    def __init__(self, chunks: torch.Tensor, n_seg: int, device, lag: int = LARS_LAG):
        seg, begin, ln = chunks.cpu().view(-1, 3).unbind(1)
        parts = (ln + LARS_PIECE - 1) // LARS_PIECE                    # pieces per chunk
        at = torch.repeat_interleave(torch.arange(len(parts)), parts)
        past = (torch.arange(len(at)) - (parts.cumsum(0) - parts)[at]) * LARS_PIECE
        rows, need = self.plan(torch.stack([seg[at], begin[at] + past, (ln[at] - past).clamp_max(LARS_PIECE)], 1), n_seg, lag)
        self.order = torch.from_numpy(rows).to(device)
        self.need = torch.tensor(need, dtype=torch.int32, device=device)
        self.n_seg = n_seg
        # not zero once a wait in the kernel has run out; in host memory, where it is read without a synchronisation
        self.status = torch.zeros(1, dtype=torch.int32, pin_memory=torch.device(device).type == "cuda")
        # sums of squares [2 n_seg], the ticket, finished pieces per segment, whether a wait ran out
        self.work = torch.zeros(3 * n_seg + 2, dtype=torch.float32, device=device)

    @staticmethod
    def plan(chunks, n_seg: int, lag: int):
        """Rows ``(segment << 1 | update | length << 32, begin)`` from pieces ``(segment, begin, length)``: a piece's update
        comes after the norms of all pieces of its segment (what makes the kernel's waits end), at the earliest ``lag`` pieces
        after its own norms."""
        seg, begin, ln = torch.as_tensor(chunks, dtype=torch.int64).view(-1, 3).unbind(1)
        i = torch.arange(len(seg))
        last = torch.zeros(n_seg, dtype=torch.int64).scatter_reduce_(0, seg, i, "amax")
        when = torch.maximum(i + lag, last[seg]).cummax(0)[0] if len(seg) else i      # the piece whose norms the update follows
        norms = torch.stack([seg << 1 | ln << 32, begin], 1)
        updates = torch.stack([norms[:, 0] | 1, begin], 1)
        rows = torch.cat([norms, updates])[torch.cat([2 * i, 2 * when + 1]).argsort(stable=True)]
        return rows.numpy(), torch.bincount(seg, minlength=n_seg).tolist()


class Hyper(ctypes.Structure):
    """Hyperparameters of a launch (``tsp::Hyper``): a code per segment, ``group << 1 | adapt``, in device memory, and the
    groups' values, by value or as a table in device memory."""
    VALS, GROUPS = 8, 32
    _fields_ = [("seg_code", ctypes.c_void_p), ("table", ctypes.c_void_p), ("by_value", ctypes.c_float * (8 * 32))]

    @staticmethod
    def of(hp) -> "Hyper":
        """``hp`` itself, or what stands for a matrix in device memory with one row of values per segment (a fifth and last
        value: adapt), to be used on the current stream."""
        if isinstance(hp, Hyper):
            return hp
        n, k = hp.shape
        codes = torch.arange(n, dtype=torch.int32, device=hp.device) << 1
        if k == 5:
            codes |= (hp[:, 4] != 0).to(torch.int32)
        table = torch.nn.functional.pad(hp.float(), (0, Hyper.VALS - k)).contiguous()
        h = Hyper(seg_code=codes.data_ptr(), table=table.data_ptr())
        h.keep = (codes, table)
        return h


@torch.no_grad()
def lars_step_(p, g, mu, chunks, hyper, norms, grad_scale=1.0, teacher=None, ema_m=0.0) -> None:
    with on_device(p.device):
        _check(lib().tsp_lars_step(_ptr(p), _ptr(g), _ptr(mu), _ptr(chunks), _c.c_int(chunks.shape[0]), _c.byref(Hyper.of(hyper)),
                                   _c.c_float(grad_scale), _ptr(norms), _c.c_int(norms.numel() // 2), _ptr(teacher),
                                   _c.c_int64(0 if teacher is None else teacher.numel()), _c.c_float(ema_m),
                                   _stream()), "tsp_lars_step")
    _count(3)


@torch.no_grad()
def lars_step_ordered_(p, g, mu, order: LarsOrder, hyper, grad_scale=1.0, teacher=None, ema_m=0.0) -> None:
    with on_device(p.device):
        _check(lib().tsp_lars_step_ordered(_ptr(p), _ptr(g), _ptr(mu), _ptr(order.order), _c.c_int(order.order.shape[0]),
                                           _ptr(order.need), _c.byref(Hyper.of(hyper)), _c.c_float(grad_scale), _ptr(order.work),
                                           _c.c_int(order.n_seg), _ptr(teacher), _c.c_int64(0 if teacher is None else teacher.numel()),
                                           _c.c_float(ema_m), _ptr(order.status), _stream()), "tsp_lars_step_ordered")
    _count(2)


@torch.no_grad()
def lars_norms_(p, g, chunks, hyper, norms, grad_scale=1.0) -> None:
    with on_device(p.device):
        _check(lib().tsp_lars_norms(_ptr(p), _ptr(g), _ptr(chunks), _c.c_int(chunks.shape[0]), _c.byref(Hyper.of(hyper)),
                                    _c.c_float(grad_scale), _ptr(norms), _c.c_int(norms.numel() // 2), _stream()),
               "tsp_lars_norms")
    _count(2)


@torch.no_grad()
def lars_apply_(p, g, mu, chunks, hyper, norms, grad_scale=1.0, teacher=None, ema_m=0.0) -> None:
    with on_device(p.device):
        _check(lib().tsp_lars_apply(_ptr(p), _ptr(g), _ptr(mu), _ptr(chunks), _c.c_int(chunks.shape[0]), _c.byref(Hyper.of(hyper)),
                                    _c.c_float(grad_scale), _ptr(norms), _ptr(teacher),
                                    _c.c_int64(0 if teacher is None else teacher.numel()), _c.c_float(ema_m),
                                    _stream()), "tsp_lars_apply")
    _count()


@torch.no_grad()
def adamw_step_(p, g, m, v, chunks, hyper, grad_scale=1.0, teacher=None, ema_m=0.0) -> None:
    with on_device(p.device):
        _check(lib().tsp_adamw_step(_ptr(p), _ptr(g), _ptr(m), _ptr(v), _ptr(chunks), _c.c_int(chunks.shape[0]),
                                    _c.byref(Hyper.of(hyper)), _c.c_float(grad_scale), _ptr(teacher),
                                    _c.c_int64(0 if teacher is None else teacher.numel()), _c.c_float(ema_m),
                                    _stream()), "tsp_adamw_step")
    _count()


@torch.no_grad()
def sgd_step_(p, g, buf, chunks, hyper, grad_scale=1.0, teacher=None, ema_m=0.0) -> None:
    with on_device(p.device):
        _check(lib().tsp_sgd_step(_ptr(p), _ptr(g), _ptr(buf), _ptr(chunks), _c.c_int(chunks.shape[0]), _c.byref(Hyper.of(hyper)),
                                  _c.c_float(grad_scale), _ptr(teacher),
                                  _c.c_int64(0 if teacher is None else teacher.numel()), _c.c_float(ema_m), _stream()),
               "tsp_sgd_step")
    _count()


# ---------------------------------------------------------------------------------------------
# losses: forward computes value AND gradient; backward only scales
# ---------------------------------------------------------------------------------------------
def _wrapped(t: torch.Tensor) -> bool:
    """A batched or otherwise wrapped stand-in (vmap, tracing), whose memory a kernel cannot read."""
    return torch._C._functorch.is_legacy_batchedtensor(t) or torch._C._functorch.is_functorch_wrapped_tensor(t)


def _rows(t: torch.Tensor) -> torch.Tensor:
    """``t`` as a contiguous matrix of its rows (its last dimension)."""
    return t if t.dim() == 2 and t.is_contiguous() else t.reshape(-1, t.shape[-1]).contiguous()


def _address(t) -> int:
    return 0 if t is None else t.data_ptr()


def _owns_saved() -> bool:
    return torch._C._autograd._top_saved_tensors_default_hooks(False) is None


def save_gradient(ctx, g: torch.Tensor) -> None:
    """Saves a gradient that a forward has computed for :func:`_scaled`, and whether it stays this function's own: hooks on
    saved tensors may keep what they are given, or hand out the same tensor elsewhere."""
    ctx.save_for_backward(g)
    ctx.own = _owns_saved()


def _scaled(g: torch.Tensor, gout: torch.Tensor, own: bool) -> torch.Tensor:
    """``g * gout`` for a gradient ``g`` that the forward has computed and saved and the loss's gradient ``gout`` (a scalar).
    As plain ops where the product is recorded itself (``create_graph``) or ``gout`` is no plain fp32 scalar.  In place where
    ``g`` is the function's ``own`` and the graph is freed behind this backward, so that nobody else will read it (a CUDA graph
    may be replayed: not there); then ``gout = 1``, a loss that is differentiated as it is, costs no pass over the gradient."""
    if (torch.is_grad_enabled() or type(g) is not torch.Tensor or type(gout) is not torch.Tensor
            or gout.dtype != torch.float32 or gout.dim() != 0 or gout.get_device() != g.get_device()
            or not g.is_contiguous() or g.data_ptr() % 16 or _wrapped(gout) or _wrapped(g)):
        return g * gout.to(g.dtype)
    own = (own and not torch._C._autograd._get_current_graph_task_keep_graph()
           and not torch._C._cuda_isCurrentStreamCapturing())
    out = g if own else torch.empty_like(g)
    with on_device(g.device):
        _check(lib().tsp_scale(g.data_ptr(), gout.data_ptr(), out.data_ptr(), g.numel(), _dt(g), _raw_stream()), "tsp_scale")
    _count()
    return out


class _ByolPair(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, y, scale):
        x = x.contiguous()
        y = y.detach().to(x.dtype).contiguous()
        n, d = x.shape
        loss = torch.zeros((), dtype=torch.float32, device=x.device)
        gx = torch.empty_like(x)
        with on_device(x.device):
            _check(lib().tsp_byol_loss(_ptr(x), _ptr(y), _c.c_int(n), _c.c_int(d), _c.c_int(_dt(x)),
                                       _c.c_float(scale), _ptr(loss), _ptr(gx), _stream()), "tsp_byol_loss")
        _count()
        save_gradient(ctx, gx)
        return loss

    @staticmethod
    def backward(ctx, gout):
        (gx,) = ctx.saved_tensors
        return _scaled(gx, gout, ctx.own), None, None


def byol_pair_loss(x: torch.Tensor, y: torch.Tensor, scale: float) -> torch.Tensor:
    """``scale * sum_rows (2 - 2 cos(x_r, y_r))``; ``y`` (teacher) gets no gradient and may live in
    peer memory."""
    return _ByolPair.apply(x, y, scale)


class _ByolBoth(torch.autograd.Function):
    """Both directions of the symmetric loss from one launch, their gradients scaled by another."""

    @staticmethod
    def forward(ctx, x1, x2, y1, y2, scale):
        n, d = x1.shape
        loss = torch.empty((), dtype=torch.float32, device=x1.device)
        total = torch.empty(2, dtype=torch.float64, device=x1.device)
        gx = torch.empty((2, n, d), dtype=x1.dtype, device=x1.device)
        with on_device(x1.device):
            _check(lib().tsp_byol_loss_pair(x1.data_ptr(), y1.data_ptr(), x2.data_ptr(), y2.data_ptr(), n, d, _dt(x1), scale,
                                            total.data_ptr(), loss.data_ptr(), gx.data_ptr(), _raw_stream()),
                   "tsp_byol_loss_pair")
        _count()
        save_gradient(ctx, gx)
        return loss

    @staticmethod
    def backward(ctx, gout):
        (gx,) = ctx.saved_tensors
        g1, g2 = _scaled(gx, gout, ctx.own).unbind(0)
        need = ctx.needs_input_grad
        return g1 if need[0] else None, g2 if need[1] else None, None, None, None


def byol_loss(o1, o2, t1, t2) -> torch.Tensor:
    host = eager() if type(o1) is torch.Tensor and type(o2) is torch.Tensor else None
    if host is not None:
        loss = host.byol_pair(o1, o2, t2, t1)
        if loss is not None:
            return loss
    n = o1.shape[0]
    if all(t.dim() == 2 and t.shape == o1.shape and t.dtype == o1.dtype and t.device == o1.device
           and t.is_contiguous() for t in (o1, o2, t1, t2)) and o1.dtype in (torch.float32, torch.bfloat16) and n > 0:
        t1, t2 = (t.detach() if t.requires_grad else t for t in (t1, t2))
        return _ByolBoth.apply(o1, o2, t2, t1, 1.0 / n)
    return byol_pair_loss(o1, t2, 1.0 / n) + byol_pair_loss(o2, t1, 1.0 / n)


def _mask_bytes(row_mask: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """A row mask as the kernels read it: a byte per row, zero where a row is off (a bool is one already)."""
    if row_mask is None:
        return None
    m = row_mask.reshape(-1)
    return (m.view(torch.uint8) if m.dtype == torch.bool else m.to(torch.uint8)).contiguous()


def _labels(labels: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    if labels is not None and not (labels.dim() == 1 and labels.dtype == torch.int64 and labels.is_contiguous()):
        labels = labels.reshape(-1).to(torch.int64).contiguous()
    return labels


class _KdCe(torch.autograd.Function):
    @staticmethod
    def forward(ctx, s, t, labels, row_mask, temp, w_ce, w_kd):
        s2 = _rows(s)
        t2 = _rows(t) if isinstance(t, torch.Tensor) else t      # None, or a peer-mapped matrix read in place over NVLink
        n, c = s2.shape
        loss = torch.empty((), dtype=torch.float32, device=s2.device)
        total = torch.empty(3, dtype=torch.float64, device=s2.device)
        gs = torch.empty_like(s2)
        lab, msk = _labels(labels), _mask_bytes(row_mask)
        with on_device(s2.device):
            _check(lib().tsp_kd_ce_loss(s2.data_ptr(), _address(t2), _address(lab), _address(msk), n, c, _dt(s2),
                                        0 if t2 is None else _dt(t2), temp, w_ce, w_kd, total.data_ptr(),
                                        loss.data_ptr(), gs.data_ptr(), _raw_stream()), "tsp_kd_ce_loss")
        _count(2)
        save_gradient(ctx, gs)
        ctx.shape = s.shape
        return loss

    @staticmethod
    def backward(ctx, gout):
        (gs,) = ctx.saved_tensors
        g = _scaled(gs, gout, ctx.own)
        return g if g.shape == ctx.shape else g.view(ctx.shape), None, None, None, None, None, None


def kd_ce_loss(s, t, labels, temp: float, w_ce: float, w_kd: float, row_mask=None) -> torch.Tensor:
    """``w_ce * sum CE(s, label) + w_kd * T^2 * sum KL(softmax(t/T) || softmax(s/T))`` over rows
    (weights carry the normalisation); labels < 0 are ignored for the CE term."""
    return _KdCe.apply(s, t, labels, row_mask, temp, w_ce, w_kd)


def kd_soft_target_loss(s, t, labels, temp: float, w_ce: float = 1.0, w_kd: float = 1.0) -> torch.Tensor:
    """``w_ce * CE(s, labels) + w_kd * T^2 * KL(softmax(t/T) || softmax(s/T))``, both batch means."""
    n = s.shape[0]
    return kd_ce_loss(s, t, labels, temp, w_ce / n, w_kd / n)


def cross_entropy(s, labels) -> torch.Tensor:
    n = s.reshape(-1, s.shape[-1]).shape[0]
    return kd_ce_loss(s, None, labels, 1.0, 1.0 / n, 0.0)


class _Cosine(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, y, row_mask, scale):
        x2 = _rows(x)
        y2 = _rows(y).to(x2.dtype)
        n, d = x2.shape
        loss = torch.empty((), dtype=torch.float32, device=x2.device)
        total = torch.empty((), dtype=torch.float64, device=x2.device)
        gx = torch.empty_like(x2)
        msk = _mask_bytes(row_mask)
        with on_device(x2.device):
            _check(lib().tsp_cosine_loss(x2.data_ptr(), y2.data_ptr(), _address(msk), n, d, _dt(x2), scale,
                                         total.data_ptr(), loss.data_ptr(), gx.data_ptr(), _raw_stream()),
                   "tsp_cosine_loss")
        _count(2)
        save_gradient(ctx, gx)
        ctx.shape = x.shape
        return loss

    @staticmethod
    def backward(ctx, gout):
        (gx,) = ctx.saved_tensors
        g = _scaled(gx, gout, ctx.own)
        return g if g.shape == ctx.shape else g.view(ctx.shape), None, None, None


def cosine_embedding_loss(x, y, scale: float, row_mask=None) -> torch.Tensor:
    return _Cosine.apply(x, y, row_mask, scale)


class _Distil(torch.autograd.Function):
    """:func:`kd_ce_loss` and :func:`cosine_embedding_loss` over the same rows, their terms in one sum."""

    @staticmethod
    def forward(ctx, s, x, t, y, labels, row_mask, temp, w_ce, w_kd, scale):
        s2, t2, x2, y2 = _rows(s), _rows(t), _rows(x), _rows(y)
        (n, c), d = s2.shape, x2.shape[1]
        loss = torch.empty((), dtype=torch.float32, device=s2.device)
        total = torch.empty(3, dtype=torch.float64, device=s2.device)
        gs, gx = torch.empty_like(s2), torch.empty_like(x2)
        lab, msk = _labels(labels), _mask_bytes(row_mask)
        with on_device(s2.device):
            _check(lib().tsp_distil_loss(s2.data_ptr(), t2.data_ptr(), _address(lab), _address(msk), n, c, _dt(s2), _dt(t2),
                                         temp, w_ce, w_kd, x2.data_ptr(), y2.data_ptr(), d, _dt(x2), scale,
                                         total.data_ptr(), loss.data_ptr(), gs.data_ptr(), gx.data_ptr(), _raw_stream()),
                   "tsp_distil_loss")
        _count(3)
        ctx.save_for_backward(gs, gx)
        ctx.own = _owns_saved()
        ctx.shapes = s.shape, x.shape
        return loss

    @staticmethod
    def backward(ctx, gout):
        out = []
        for g, shape, need in zip(ctx.saved_tensors, ctx.shapes, ctx.needs_input_grad):
            g = _scaled(g, gout, ctx.own) if need else None
            out.append(g if g is None or g.shape == shape else g.view(shape))
        return (*out, None, None, None, None, None, None, None, None)


def distil_loss(s, t, labels, temp: float, w_ce: float, w_kd: float, x, y, scale: float, row_mask=None) -> torch.Tensor:
    """``kd_ce_loss(s, t, ...) + cosine_embedding_loss(x, y, scale)`` under one row mask."""
    ts = (s, t, x, y)
    if all(type(v) is torch.Tensor and v.dim() > 1 and v.numel() > 0 and v.dtype in (torch.float32, torch.bfloat16)
           and v.device == s.device and not _wrapped(v) for v in ts) and y.dtype == x.dtype \
            and s.shape == t.shape and x.shape == y.shape and s.shape[:-1] == x.shape[:-1]:
        return _Distil.apply(s, x, t, y, labels, row_mask, temp, w_ce, w_kd, scale)
    return kd_ce_loss(s, t, labels, temp, w_ce, w_kd, row_mask) + cosine_embedding_loss(x, y, scale, row_mask)


def info_nce_loss(q: torch.Tensor, k: torch.Tensor, temp: float) -> torch.Tensor:
    """InfoNCE of MoCo-v3: ``CE(normalize(q) @ normalize(k)^T / T, arange(N)) * 2T``."""
    from . import gemm
    return gemm.info_nce(q, k, temp)


# ---------------------------------------------------------------------------------------------
# LayerNorm / GELU
# ---------------------------------------------------------------------------------------------
class _LayerNorm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, b, eps):
        d = x.shape[-1]
        x2 = x.reshape(-1, d).contiguous()
        rows = x2.shape[0]
        y = torch.empty_like(x2)
        mean = torch.empty(rows, dtype=torch.float32, device=x.device)
        rstd = torch.empty(rows, dtype=torch.float32, device=x.device)
        wf, bf = param_f32(w), param_f32(b)
        with on_device(x.device):
            _check(lib().tsp_layernorm_fwd(_ptr(x2), _ptr(wf), _ptr(bf), _ptr(y), _ptr(mean), _ptr(rstd),
                                           _c.c_int(rows), _c.c_int(d), _c.c_float(eps), _c.c_int(_dt(x2)), _stream()),
                   "tsp_layernorm_fwd")
        _count()
        ctx.save_for_backward(x2, wf, mean, rstd)
        ctx.shape = x.shape
        ctx.wdtype = w.dtype
        ctx.owners = (w, b) if IN_CAPTURE else (None, None)
        return y.view(x.shape)

    @staticmethod
    def backward(ctx, dy):
        return _LayerNorm._backward(ctx, dy, None)

    @staticmethod
    def _backward(ctx, dy, skip):
        x2, wf, mean, rstd = ctx.saved_tensors
        rows, d = x2.shape
        dy2 = dy.reshape(rows, d).to(x2.dtype).contiguous()
        dx = torch.empty_like(x2)
        gw, gb = (recorded_grad(p) for p in ctx.owners)
        add = gw is not None and gb is not None
        dw = gw if add else torch.empty(d, dtype=torch.float32, device=x2.device)
        db = gb if add else torch.empty(d, dtype=torch.float32, device=x2.device)
        nb = lib().tsp_layernorm_bwd_blocks(_c.c_int(rows))
        partial = torch.empty(nb * 2 * d, dtype=torch.float32, device=x2.device)
        with on_device(x2.device):
            _check(lib().tsp_layernorm_bwd_add(_ptr(dy2), _ptr(x2), _ptr(skip), _ptr(wf), _ptr(mean), _ptr(rstd), _ptr(dx),
                                               _ptr(dw), _ptr(db), _ptr(partial), _c.c_int(rows), _c.c_int(d),
                                               _c.c_int(_dt(x2)), _c.c_int(1 if add else 0), _stream()),
                   "tsp_layernorm_bwd")
        _count(2)
        if add:
            return dx.view(ctx.shape), None, None, None
        return dx.view(ctx.shape), dw.to(ctx.wdtype), db.to(ctx.wdtype), None


class _AddLayerNorm(torch.autograd.Function):
    """``(s, layer_norm(s))`` with ``s = x + a``, or ``s = x`` where ``a`` is None (a residual connection that starts here):
    the gradient that comes back for ``s`` is added as the LayerNorm's own is stored."""

    @staticmethod
    def forward(ctx, x, a, w, b, eps, need_sum):
        ctx.set_materialize_grads(False)
        if a is None:
            return x.view_as(x), _LayerNorm.forward(ctx, x, w, b, eps)
        d = x.shape[-1]
        rows = x.numel() // d
        s = torch.empty_like(x) if need_sum or any(ctx.needs_input_grad) else None
        y = torch.empty_like(x)
        mean = torch.empty(rows, dtype=torch.float32, device=x.device)
        rstd = torch.empty(rows, dtype=torch.float32, device=x.device)
        wf, bf = param_f32(w), param_f32(b)
        with on_device(x.device):
            _check(lib().tsp_add_layernorm_fwd(_ptr(x), _ptr(a), _ptr(s), _ptr(wf), _ptr(bf), _ptr(y), _ptr(mean), _ptr(rstd),
                                               _c.c_int(rows), _c.c_int(d), _c.c_float(eps), _c.c_int(_dt(x)), _stream()),
                   "tsp_add_layernorm_fwd")
        _count()
        if s is not None:
            ctx.save_for_backward(s.view(rows, d), wf, mean, rstd)
        ctx.shape, ctx.wdtype = x.shape, w.dtype
        ctx.owners = (w, b) if IN_CAPTURE else (None, None)
        return s, y

    @staticmethod
    def backward(ctx, ds, dy):
        if dy is None:
            return ds, (ds if ctx.needs_input_grad[1] else None), None, None, None, None
        x2 = ctx.saved_tensors[0]
        fits = ds is not None and ds.dtype == x2.dtype and ds.is_contiguous() and ds.data_ptr() % 16 == 0
        dx, dw, db, _ = _LayerNorm._backward(ctx, dy, ds if fits else None)
        if ds is not None and not fits:
            dx = dx + ds
        return dx, (dx if ctx.needs_input_grad[1] else None), dw, db, None, None


def add_layer_norm(x: torch.Tensor, a: Optional[torch.Tensor], weight: torch.Tensor, bias: torch.Tensor, eps: float = 1e-5,
                   need_sum: bool = True):
    """``(s, layer_norm(s))`` for ``s = x + a`` (``s = x`` without ``a``), in one pass each way where the kernels apply.
    Without ``need_sum`` the first may be None (it is not written then)."""
    d = x.shape[-1]
    if (x.is_cuda and d % 8 == 0 and d <= 1024 and x.dtype in (torch.float32, torch.bfloat16) and x.is_contiguous()
            and x.data_ptr() % 16 == 0 and x.numel() > 0
            and (a is None or (a.dtype == x.dtype and a.shape == x.shape and a.device == x.device and a.is_contiguous()
                               and a.data_ptr() % 16 == 0))):
        return _AddLayerNorm.apply(x, a, weight, bias, eps, need_sum)
    s = x if a is None else x + a
    return s, layer_norm(s, weight, bias, eps)


def layer_norm(x: torch.Tensor, weight: torch.Tensor, bias: torch.Tensor, eps: float = 1e-5) -> torch.Tensor:
    d = x.shape[-1]
    if not x.is_cuda or d % 8 != 0 or d > 1024 or x.dtype not in (torch.float32, torch.bfloat16):
        return torch.nn.functional.layer_norm(x, (d,), weight, bias, eps)
    return _LayerNorm.apply(x, weight, bias, eps)


class _Gelu(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, bias):
        x = x.contiguous()
        d = x.shape[-1]
        y = torch.empty_like(x)
        bf = None if bias is None else param_f32(bias)
        with on_device(x.device):
            _check(lib().tsp_gelu_fwd(_ptr(x), _ptr(bf), _ptr(y), _c.c_int64(x.numel()), _c.c_int(d), _c.c_int(_dt(x)),
                                      _stream()), "tsp_gelu_fwd")
        _count()
        ctx.save_for_backward(x, bf if bf is not None else x.new_empty(0))
        ctx.has_bias = bias is not None
        ctx.bdtype = None if bias is None else bias.dtype
        ctx.bias = bias if IN_CAPTURE else None
        return y

    @staticmethod
    def backward(ctx, dy):
        x, bf = ctx.saved_tensors
        dy = dy.contiguous()
        dx = torch.empty_like(x)
        d = x.shape[-1]
        with on_device(x.device):
            _check(lib().tsp_gelu_bwd(_ptr(dy), _ptr(x), _ptr(bf if ctx.has_bias else None), _ptr(dx),
                                      _c.c_int64(x.numel()), _c.c_int(d), _c.c_int(_dt(x)), _stream()), "tsp_gelu_bwd")
        _count()
        db = None
        if ctx.has_bias:
            from .gemm import _column_sums
            db = _column_sums(dx.reshape(-1, d), add_to=recorded_grad(ctx.bias))
            db = None if db is None else db.to(ctx.bdtype)
        return dx, db


def gelu(x: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``gelu(x + bias)`` (erf form)."""
    if not x.is_cuda or x.numel() % 8 != 0 or x.dtype not in (torch.float32, torch.bfloat16) or \
            (bias is not None and x.shape[-1] % 8 != 0):
        return torch.nn.functional.gelu(x if bias is None else x + bias)
    return _Gelu.apply(x, bias)


# ---------------------------------------------------------------------------------------------
# data-parallel reduce-scatter + sharded step + all-gather over peer-mapped buffers (csrc/peer.cu)
# ---------------------------------------------------------------------------------------------
@torch.no_grad()
def dp_reduce_norms_(grad_ptrs, n_peers, scale, g_out, p, chunks, hyper, norms) -> None:
    L = lib()
    L.tsp_dp_reduce_norms.restype = _c.c_int
    with on_device(p.device):
        _check(L.tsp_dp_reduce_norms(grad_ptrs, _c.c_int(n_peers), _c.c_float(scale), _ptr(g_out), _ptr(p),
                                     _ptr(chunks), _c.c_int(chunks.shape[0]), _c.byref(Hyper.of(hyper)), _ptr(norms),
                                     _c.c_int(norms.numel() // 2), _stream()), "tsp_dp_reduce_norms")
    _count(2)


@torch.no_grad()
def publish_norms_(table_ptrs, n_peers, self_idx, norms) -> None:
    """This rank's partial LARS norms into slot ``self_idx`` of every replica's table (peer stores)."""
    L = lib()
    L.tsp_publish_norms.restype = _c.c_int
    with on_device(norms.device):
        _check(L.tsp_publish_norms(table_ptrs, _c.c_int(n_peers), _c.c_int(self_idx), _ptr(norms),
                                   _c.c_int(norms.numel()), _stream()), "tsp_publish_norms")
    _count()


@torch.no_grad()
def sum_norms_(table, n_peers, norms) -> None:
    """``norms = sum_r table[r]`` over the replicas' slots."""
    L = lib()
    L.tsp_sum_norms.restype = _c.c_int
    with on_device(norms.device):
        _check(L.tsp_sum_norms(_ptr(table), _c.c_int(n_peers), _c.c_int(norms.numel()), _ptr(norms), _stream()),
               "tsp_sum_norms")
    _count()


@torch.no_grad()
def dp_lars_apply_(param_ptrs, n_peers, self_idx, g, mu, chunks, hyper, norms) -> None:
    L = lib()
    L.tsp_dp_lars_apply.restype = _c.c_int
    with on_device(g.device):
        _check(L.tsp_dp_lars_apply(param_ptrs, _c.c_int(n_peers), _c.c_int(self_idx), _ptr(g), _ptr(mu), _ptr(chunks),
                                   _c.c_int(chunks.shape[0]), _c.byref(Hyper.of(hyper)), _ptr(norms), _stream()),
               "tsp_dp_lars_apply")
    _count()


@torch.no_grad()
def dp_adamw_step_(grad_ptrs, param_ptrs, n_peers, self_idx, scale, m, v, chunks, hyper) -> None:
    L = lib()
    L.tsp_dp_adamw_step.restype = _c.c_int
    with on_device(m.device):
        _check(L.tsp_dp_adamw_step(grad_ptrs, param_ptrs, _c.c_int(n_peers), _c.c_int(self_idx), _c.c_float(scale),
                                   _ptr(m), _ptr(v), _ptr(chunks), _c.c_int(chunks.shape[0]), _c.byref(Hyper.of(hyper)),
                                   _stream()), "tsp_dp_adamw_step")
    _count()
