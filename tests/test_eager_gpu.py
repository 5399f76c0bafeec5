"""Eager calls as C++ autograd functions (``csrc/host/eager.cpp``) against the Python functions of the same layers."""
import contextlib

import pytest
import torch
from torch import nn

from tspipe_b200.batchnorm import BatchNormGroup, DeferredBatchNorm
from tspipe_b200.ops import fused

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _cl(*shape, dtype=torch.bfloat16):
    return torch.randn(*shape, device=DEV).to(dtype).contiguous(memory_format=torch.channels_last)


def _both(monkeypatch, make, call, taken=True):
    """``call(*make())`` with the C++ functions and with the Python ones; the first have run where the call is one for them (``taken``)."""
    outs = []
    for native in (True, False):
        torch.manual_seed(0)
        with monkeypatch.context() as m:
            if not native:
                m.setattr(fused, "eager", lambda: None)
            args = make()
            before = 0 if fused._host is None else fused._host.launches()
            outs.append(call(*args))
            assert ((0 if fused._host is None else fused._host.launches()) > before) == (native and taken)
    return outs


def _same(a, b, tol=2e-3):
    assert (a is None) == (b is None)
    if a is not None:
        assert a.shape == b.shape and a.dtype == b.dtype
        a, b = a.double(), b.double()
        assert float((a - b).norm()) <= tol * float(b.norm()) + 1e-12


def _conv_block(k, stride, cin, cout, n, side, views, res, fork, dtype=torch.bfloat16):
    conv = nn.Conv2d(cin, cout, k, stride=stride, padding=(k - 1) // 2, bias=False).to(DEV, memory_format=torch.channels_last)
    bn = DeferredBatchNorm(cout).to(DEV)
    group = BatchNormGroup(bn, chunks=10)
    with torch.no_grad():
        bn.weight.uniform_(0.5, 1.5)
        bn.bias.normal_()
    so = (side + 2 * ((k - 1) // 2) - k) // stride + 1
    x = _cl(n, cin, side, side).requires_grad_()
    r = _cl(n, cout, so, so, dtype=dtype).requires_grad_() if res else None
    gy, gx = _cl(n, cout, so, so), _cl(n, cin, side, side)
    return conv, bn, group, x, r, gy, gx, views, fork


def _run_conv(conv, bn, group, x, r, gy, gx, views, fork):
    from tspipe_b200.ops import bn as fbn
    from tspipe_b200.ops import conv as fconv
    leaves = [x, conv.weight, bn.weight, bn.bias] + ([r] if r is not None else [])
    with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False), fbn.segments(views):
        if fork:
            y, skip = fconv.conv_bn_act_fork(conv, bn, x, relu=True)
        else:
            y, skip = fconv.conv_bn_act(conv, bn, x, residual=r, relu=True), None
    fconv.clear_weight_cache()
    out = [y] + ([skip] if fork else [])
    grads = torch.autograd.grad(out, leaves, [gy] + ([gx] if fork else []), retain_graph=True)
    again = torch.autograd.grad(out, leaves, [gy] + ([gx] if fork else []))
    only = None
    return [y.detach(), group._acc, *grads, *again], only


@pytest.mark.parametrize("k,stride,cin,cout,n,side,views,res,fork",
                         [(1, 1, 64, 64, 4, 8, 1, False, False), (1, 1, 64, 256, 4, 8, 2, True, False),
                          (3, 1, 64, 64, 3, 14, 1, False, False), (3, 2, 128, 64, 5, 8, 1, False, False),
                          (1, 2, 64, 128, 2, 10, 2, False, False), (1, 1, 256, 64, 6, 7, 2, False, True),
                          (3, 1, 64, 64, 2, 9, 1, False, True), (1, 1, 64, 64, 3, 5, 3, False, False)])
def test_convolution_and_batchnorm(monkeypatch, k, stride, cin, cout, n, side, views, res, fork):
    """Strides, taps, residuals, forks, views, statistics from the epilogue and from a pass of their own (7 x 7 images of two
    views); three views are no case for the convolution's function: their BatchNorms run one after the other."""
    a, b = _both(monkeypatch, lambda: _conv_block(k, stride, cin, cout, n, side, views, res, fork), lambda *v: _run_conv(*v)[0])
    for p, q in zip(a, b):
        _same(p, q)


def test_convolution_gradients_in_place_by_name_and_with_hooks(monkeypatch):
    """The weight's gradient goes to an existing buffer only when it is asked for; BatchNorm's through its hooks."""
    def call(conv, bn, group, x, r, gy, gx, views, fork):
        from tspipe_b200.ops import conv as fconv
        conv.weight.grad = torch.ones_like(conv.weight)
        bn.weight.grad, bn.bias.grad = torch.ones_like(bn.weight), torch.ones_like(bn.bias)
        seen = []
        bn.weight.register_hook(lambda g: seen.append(1) or 2 * g)
        with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False):
            y = fconv.conv_bn_act(conv, bn, x, relu=True)
        (dw,) = torch.autograd.grad(y, [bn.bias], gy, retain_graph=True)
        assert torch.equal(conv.weight.grad, torch.ones_like(conv.weight)) and not seen
        y.backward(gy)
        assert seen == [1]
        return [dw, conv.weight.grad, bn.weight.grad, bn.bias.grad, x.grad]
    a, b = _both(monkeypatch, lambda: _conv_block(3, 1, 64, 128, 2, 8, 1, False, False), call)
    for p, q in zip(a, b):
        _same(p, q)


@pytest.mark.parametrize("watch", ["nothing", "post", "node", "no_buffer", "by_name"])
def test_vector_gradients_in_place_only_where_nobody_watches(monkeypatch, watch):
    """BatchNorm's and a linear layer's bias gradients go to the parameter's own buffer in a plain backward(); a hook behind the
    accumulation, one on its node, a parameter without a buffer and a backward over named inputs get them as before."""
    def make():
        lin = nn.Linear(64, 128).to(DEV)
        bn = DeferredBatchNorm(128).to(DEV)
        return lin, bn, BatchNormGroup(bn, chunks=10), torch.randn(256, 64, device=DEV).bfloat16(), torch.randn(256, 128, device=DEV).bfloat16()

    def call(lin, bn, group, x, g):
        from tspipe_b200.ops import bn as fbn
        from tspipe_b200.ops import gemm
        ps = [lin.weight, lin.bias, bn.weight, bn.bias]
        for p in ps:
            p.grad = None if watch == "no_buffer" else torch.ones_like(p)
        seen = []
        if watch == "post":
            for p in ps[1:]:
                p.register_post_accumulate_grad_hook(lambda p: seen.append(p.shape))
        nodes = [p.expand_as(p).grad_fn.next_functions[0][0] for p in ps[1:]]
        if watch == "node":
            for node in nodes:
                node.register_hook(lambda *a: seen.append(1))
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = fbn.bn_act(bn, gemm.linear(x, lin.weight, lin.bias), None, True)
        if watch == "by_name":
            y.backward(g, inputs=ps[2:])
            assert torch.equal(lin.bias.grad, torch.ones_like(lin.bias))
        else:
            y.backward(g, retain_graph=True)
            y.backward(g)
        assert len(seen) == (6 if watch in ("post", "node") else 0)
        return [p.grad for p in (ps[2:] if watch == "by_name" else ps)]
    a, b = _both(monkeypatch, make, call)
    # (the bias in front of a BatchNorm has a gradient of zero, of which the rounding is left)
    for p, q in zip(a, b):
        if watch in ("by_name",) or p is not a[1]:
            _same(p, q)
        else:
            assert float((p - q).abs().max()) < 0.1


@pytest.mark.parametrize("mode", ["no_grad", "inference", "cpu_hooks", "written", "fp32_residual"])
def test_convolution_under_other_modes(monkeypatch, mode):
    from tspipe_b200.ops import conv as fconv

    def call(conv, bn, group, x, r, gy, gx, views, fork):
        ctx = {"no_grad": torch.no_grad, "inference": torch.inference_mode,
               "cpu_hooks": torch.autograd.graph.save_on_cpu}.get(mode, contextlib.nullcontext)
        with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False), ctx():
            y = fconv.conv_bn_act(conv, bn, x, residual=r, relu=True)
        if mode in ("no_grad", "inference"):
            assert not y.requires_grad
            return [y.clone()]
        if mode == "written":                   # a weight changed in place between forward and backward is refused
            with torch.no_grad():
                conv.weight.mul_(2)
            with pytest.raises(RuntimeError, match="modified by an inplace operation"):
                y.backward(gy)
            return [y.detach()]
        return [y.detach(), *torch.autograd.grad(y, [x, conv.weight, bn.weight, bn.bias, r], gy)]
    make = lambda: _conv_block(1, 1, 64, 64, 4, 8, 1, True, False,                      # noqa: E731
                               torch.float32 if mode == "fp32_residual" else torch.bfloat16)
    a, b = _both(monkeypatch, make, call, taken=mode != "fp32_residual")        # (which the Python function converts)
    for p, q in zip(a, b):
        _same(p, q)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape,views,res,relu", [((128, 64), 1, False, True), ((256, 4096), 2, False, True),
                                                  ((64, 72), 2, True, True), ((4, 64, 6, 5), 2, True, False)])
def test_batchnorm(monkeypatch, shape, views, res, relu, dtype):
    from tspipe_b200.ops import bn as fbn

    def make():
        bn = DeferredBatchNorm(shape[1]).to(DEV)
        return (bn, BatchNormGroup(bn, chunks=10), *((_cl if len(shape) == 4 else lambda *s, dtype: torch.randn(*s, device=DEV).to(dtype))
                                                     (*shape, dtype=dtype) for _ in range(3)))

    def call(bn, group, x, r, g):
        x.requires_grad_()
        r.requires_grad_()
        with fbn.segments(views):
            y = fbn.bn_act(bn, x, r if res else None, relu)
        return [y.detach(), group._acc, *torch.autograd.grad(y, [x, bn.weight, bn.bias] + ([r] if res else []), g)]
    a, b = _both(monkeypatch, make, call)
    for p, q in zip(a, b):
        _same(p, q, 2e-3 if dtype == torch.bfloat16 else 1e-5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,k,n,bias,grad", [((128,), 64, 64, True, False), ((4, 50), 128, 192, False, True),
                                                ((300,), 256, 64, True, True), ((2, 100), 64, 8256, True, False)])
def test_linear(monkeypatch, rows, k, n, bias, grad, dtype):
    """With and without a bias and a gradient buffer, a bias wider than the column-sum kernel takes."""
    from tspipe_b200.ops import gemm

    def make():
        m = nn.Linear(k, n, bias=bias).to(DEV)
        if grad:
            m.weight.grad = torch.ones_like(m.weight)
        return m, torch.randn(*rows, k, device=DEV).to(dtype).requires_grad_(), torch.randn(*rows, n, device=DEV).bfloat16()

    def call(m, x, g):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = gemm.linear(x, m.weight, m.bias)
        gemm.clear_weight_cache()
        y.backward(g)
        return [y.detach(), x.grad, m.weight.grad, m.bias.grad if bias else None]
    a, b = _both(monkeypatch, make, call)
    for p, q in zip(a, b):
        _same(p, q)


@pytest.mark.parametrize("kind", ["byol", "nce"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_pair_losses(monkeypatch, kind, dtype):
    """Value and gradients, differentiated as it is, scaled, twice, with a recorded product, under hooks, for one input."""
    from tspipe_b200.ops import gemm

    def make():
        base = [torch.randn(160, 256, device=DEV) for _ in range(2)]
        ts = [(base[i % 2] + 0.7 * torch.randn(160, 256, device=DEV)).to(dtype) for i in range(4)]
        return [t.requires_grad_() for t in ts]

    def call(o1, o2, t1, t2):
        def loss():
            return fused.byol_loss(o1, o2, t1, t2) if kind == "byol" else gemm.info_nce_pair(o1, t2, o2, t1, 0.2)
        l0 = loss()
        out = [l0.detach(), *torch.autograd.grad(l0, [o1, o2])]
        l1 = loss()
        out += torch.autograd.grad(3 * l1, [o1, o2], retain_graph=True)
        out += torch.autograd.grad(l1, [o1, o2])
        out += torch.autograd.grad(loss(), [o2])
        scale = torch.ones((), device=DEV, requires_grad=True)
        (g,) = torch.autograd.grad(loss() * scale, o1, create_graph=True)
        out += torch.autograd.grad(g.float().sum(), scale)
        with torch.autograd.graph.save_on_cpu():
            l2 = loss()
        out += torch.autograd.grad(2 * l2, [o1])
        out.append(torch.autograd.grad(loss(), [o1], torch.full((), 2.0, device=DEV))[0])
        return out
    a, b = _both(monkeypatch, make, call)
    for p, q in zip(a, b):
        _same(p, q, 1e-5)
    ts = make()
    with pytest.raises(RuntimeError, match="appears to not have been used in the graph"):       # (teachers have no gradient)
        torch.autograd.grad(fused.byol_loss(*ts) if kind == "byol" else gemm.info_nce_pair(ts[0], ts[3], ts[1], ts[2], 0.2), [ts[2]])


def _additions(call):
    """In-place additions that autograd has made during ``call`` (a gradient that a kernel adds itself is none)."""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        call()
    return sum(e.count for e in prof.key_averages() if e.key == "aten::add_")


def _three_layers():
    """A linear layer, a BatchNorm and a convolution with one, with gradient buffers: forward of all, parameters, gradients."""
    from tspipe_b200.ops import bn as fbn
    from tspipe_b200.ops import conv as fconv
    from tspipe_b200.ops import gemm
    lin, conv = nn.Linear(64, 128).to(DEV), nn.Conv2d(64, 64, 1, bias=False).to(DEV, memory_format=torch.channels_last)
    bns = nn.ModuleList([DeferredBatchNorm(128), DeferredBatchNorm(64)]).to(DEV)
    group = BatchNormGroup(bns, chunks=100)
    xs = torch.randn(256, 64, device=DEV).bfloat16(), torch.randn(256, 128, device=DEV).bfloat16(), _cl(4, 64, 8, 8)
    gs = torch.randn(256, 128, device=DEV).bfloat16(), torch.randn(256, 128, device=DEV).bfloat16(), _cl(4, 64, 8, 8)
    ps = [*lin.parameters(), *conv.parameters(), *bns.parameters()]
    for p in ps:
        p.grad = torch.ones_like(p)

    def forward():
        with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False):
            return [gemm.linear(xs[0], lin.weight, lin.bias), fbn.bn_act(bns[0], xs[1], None, True),
                    fconv.conv_bn_act(conv, bns[1], xs[2], relu=True)]
    return forward, ps, gs, group


@pytest.mark.parametrize("where", ["here", "side", "held", "both"])
def test_gradients_of_layers_on_other_streams(monkeypatch, where):
    """A kernel adds to a gradient itself only on the stream of the accumulation: not where the accumulating nodes were made on
    another one than the layer's (``held``), and of two uses on two streams in one graph (``both``) on one of them.  The caller's stream
    reads the gradients behind backward() without a wait of its own, while the side stream is busy."""
    def call(forward, ps, gs, group):
        here, native = torch.cuda.current_stream(), fused.eager() is not None
        side = torch.cuda.Stream() if native else here          # (the reference on one stream)
        held = [p.expand_as(p).grad_fn.next_functions[0][0] for p in ps] if where == "held" else None
        ys = forward() if where in ("here", "both") else []
        side.wait_stream(here)
        if where != "here":
            with torch.cuda.stream(side):
                ys += forward()
                here.wait_stream(side)
                torch.cuda._sleep(10_000_000)
        outs = []

        def backward():
            torch.autograd.backward(ys, gs * (len(ys) // 3))
            outs.extend(p.grad.clone() for p in ps)
        added = _additions(backward)
        torch.cuda.synchronize()
        if native:
            assert added == {"here": 0, "side": 0, "held": len(ps), "both": len(ps)}[where]
        del held
        return outs
    a, b = _both(monkeypatch, _three_layers, call)
    for p, q in zip(a, b):
        _same(p, q)


def test_every_gradient_goes_to_autograd_where_in_place_addition_is_off(monkeypatch):
    from tspipe_b200.ops import conv as fconv

    def call(forward, ps, gs, group):
        native = fused.eager() is not None
        fconv.set_accumulate_in_place(False)
        try:
            ys = forward()
            added = _additions(lambda: torch.autograd.backward(ys, gs))
        finally:
            fconv.set_accumulate_in_place(True)
        assert added == len(ps) or not native
        return [p.grad for p in ps]
    a, b = _both(monkeypatch, _three_layers, call)
    for p, q in zip(a, b):
        _same(p, q)


@pytest.mark.parametrize("anomaly", [False, True])
def test_vector_gradients_in_place_count_as_written(anomaly):
    """A gradient that a graph has saved is refused behind a backward() that added to it, and a search for NaN sees all of them."""
    forward, ps, gs, group = _three_layers()
    vectors = [p for p in ps if p.dim() == 1]
    kept = [p.grad * torch.ones_like(p, requires_grad=True) for p in vectors]
    ys = forward()
    if anomaly:
        with pytest.raises(RuntimeError, match="returned nan values"), torch.autograd.detect_anomaly():
            ys[0].backward(torch.full_like(gs[0], float("nan")))
    else:
        torch.autograd.backward(ys, gs)
        for k in kept:
            with pytest.raises(RuntimeError, match="modified by an inplace operation"):
                k.sum().backward()


@pytest.mark.parametrize("fmt", [torch.channels_last, torch.contiguous_format])
def test_fork_of_single_pixels_takes_the_other_gradient_along(monkeypatch, fmt):
    """Images of one pixel are channels-last in either format: the data gradient adds the other branch's, in one rounding."""
    from tspipe_b200.ops import conv as fconv

    def call(conv, bn, group, x, r, gy, gx, views, fork):
        native = fused.eager() is not None
        gx = gx.clone(memory_format=fmt)
        with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False):
            y, skip = fconv.conv_bn_act_fork(conv, bn, x, relu=True)
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
            dx, dw = torch.autograd.grad([y, skip], [x, conv.weight], [gy, gx])
        assert not native or not any(e.key == "aten::add" for e in prof.key_averages())
        return [dx, dw]
    a, b = _both(monkeypatch, lambda: _conv_block(1, 1, 64, 64, 64, 1, 1, False, True), call)
    for p, q in zip(a, b):
        _same(p, q)


@pytest.mark.parametrize("kind,res", [("conv", False), ("conv", True), ("fork", False), ("rows", False), ("rows", True)])
@pytest.mark.parametrize("views", [1, 2])
def test_gradients_added_twice_to_buffers(monkeypatch, views, res, kind):
    """Two plain backward() calls into filled buffers, which the kernels add to, over views, residuals and forks."""
    from tspipe_b200.ops import bn as fbn
    from tspipe_b200.ops import conv as fconv

    def call(conv, bn, group, x, r, gy, gx, views, fork):
        native = fused.eager() is not None
        ps = [bn.weight, bn.bias] + ([conv.weight] if kind != "rows" else [])
        for p in ps:
            p.grad = torch.ones_like(p)

        def step():
            with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False), fbn.segments(views):
                if fork:
                    torch.autograd.backward(fconv.conv_bn_act_fork(conv, bn, x, relu=True), [gy, gx])
                elif kind == "conv":
                    fconv.conv_bn_act(conv, bn, x, residual=r, relu=True).backward(gy)
                else:
                    fbn.bn_act(bn, x, r, True).backward(gy)
        step()
        x.grad = None
        if r is not None:
            r.grad = None
        added = _additions(step)
        assert added == 0 or not native
        return [p.grad for p in ps + [x] + ([r] if r is not None else [])]
    a, b = _both(monkeypatch, lambda: _conv_block(1, 1, 64, 64, 4, 8, views, res, kind == "fork"), call)
    for p, q in zip(a, b):
        _same(p, q)


@pytest.mark.parametrize("frozen", ["convolution", "vectors", "input"])
@pytest.mark.parametrize("buffers", [False, True])
def test_convolution_with_frozen_parts(monkeypatch, frozen, buffers):
    from tspipe_b200.ops import conv as fconv

    def call(conv, bn, group, x, r, gy, gx, views, fork):
        conv.weight.requires_grad_(frozen != "convolution")
        bn.weight.requires_grad_(frozen != "vectors")
        x.requires_grad_(frozen != "input")
        ps = [p for p in (conv.weight, bn.weight, bn.bias) if p.requires_grad]
        for p in ps:
            p.grad = torch.ones_like(p) if buffers else None
        with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False):
            fconv.conv_bn_act(conv, bn, x, relu=True).backward(gy)
        assert all(t.grad is None for t in (conv.weight, bn.weight, x) if not t.requires_grad)
        return [t.grad for t in ps + ([x] if frozen != "input" else [])]
    a, b = _both(monkeypatch, lambda: _conv_block(3, 1, 64, 64, 2, 8, 1, False, False), call)
    for p, q in zip(a, b):
        _same(p, q)


def test_graph_kept_under_saved_tensor_hooks(monkeypatch):
    from tspipe_b200.ops import conv as fconv

    def call(conv, bn, group, x, r, gy, gx, views, fork):
        with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False), torch.autograd.graph.save_on_cpu():
            y = fconv.conv_bn_act(conv, bn, x, residual=r, relu=True)
        for keep in (True, True, False):
            y.backward(gy, retain_graph=keep)
        with pytest.raises(RuntimeError, match="second time"):
            y.backward(gy)
        return [t.grad for t in (x, conv.weight, bn.weight, bn.bias, r)]
    a, b = _both(monkeypatch, lambda: _conv_block(1, 1, 64, 64, 4, 8, 1, True, False), call)
    for p, q in zip(a, b):
        _same(p, q)


def test_output_of_a_convolution_is_let_go_within_the_backward():
    """In the backward's peak its memory has become that of dx; with a graph that is kept it stays, and the graph can be used again."""
    from tspipe_b200.ops import conv as fconv
    conv, bn, group, x, _, gy, _, _, _ = _conv_block(1, 1, 64, 64, 64, 64, 1, False, False)
    size = x.numel() * 2
    with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False):
        y = fconv.conv_bn_act(conv, bn, x, relu=True)
    peaks, grads = [], []
    for keep in (True, False):
        x.grad = conv.weight.grad = None
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        y.backward(gy, retain_graph=keep)
        peaks.append(torch.cuda.max_memory_allocated() - before)
        grads.append(x.grad)
    assert size * 0.9 < peaks[0] - peaks[1] < size * 1.1
    _same(*grads)


def test_layers_on_two_threads(monkeypatch):
    """Forwards and backwards of two threads, each on a stream of its own, at the same time: as one after the other."""
    import threading

    def run(forward, ps, gs, group):
        for _ in range(20):
            torch.autograd.backward(forward(), gs)
        torch.cuda.current_stream().synchronize()

    def call(first, second):
        if fused.eager() is None:
            run(*first)
            run(*second)
        else:
            torch.cuda.synchronize()

            def on_a_stream(args):
                with torch.cuda.stream(torch.cuda.Stream()):
                    run(*args)
            threads = [threading.Thread(target=on_a_stream, args=(a,)) for a in (first, second)]
            for t in threads:
                t.start()
            for t in threads:
                t.join()
        return [p.grad for a in (first, second) for p in a[1]]
    a, b = _both(monkeypatch, lambda: (_three_layers(), _three_layers()), call)
    for p, q in zip(a, b):
        _same(p, q)
