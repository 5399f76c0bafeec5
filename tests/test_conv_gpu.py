"""tcgen05 convolutions (stem 7 x 7 / 2, implicit-GEMM 1x1 / 3x3) and fused partition execution against plain PyTorch
in fp32."""
import copy
import math

import pytest
import torch
import torch.nn.functional as F
from torch import nn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w", [(2, 64, 64), (3, 224, 224), (5, 96, 40), (1, 8, 8), (150, 16, 16)])
def test_stem_conv_matches_fp32_reference(n, h, w):
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(0)
    dev = torch.device("cuda", 0)
    x = torch.randn(n, 3, h, w, device=dev).to(dtype=torch.bfloat16, memory_format=torch.channels_last)
    weight = (torch.randn(64, 3, 7, 7, device=dev) * 0.1).requires_grad_()
    assert conv.eligible(x)
    y, sums = conv.stem_conv(x, weight)
    gemm.check_status()
    wr = weight.detach().bfloat16().float().requires_grad_()
    ref = F.conv2d(x.float(), wr, stride=2, padding=3)
    assert y.shape == ref.shape and y.is_contiguous(memory_format=torch.channels_last)
    torch.testing.assert_close(y.float(), ref, rtol=2e-2, atol=2e-2)
    yf = y.float()
    torch.testing.assert_close(sums[:64], yf.sum((0, 2, 3)), rtol=1e-3, atol=1e-2)
    torch.testing.assert_close(sums[64:], (yf * yf).sum((0, 2, 3)), rtol=1e-3, atol=1e-2)
    g = torch.randn_like(y)
    y.backward(g)
    ref.backward(g.float())
    torch.testing.assert_close(weight.grad, wr.grad, rtol=5e-2, atol=5e-2 * wr.grad.abs().max().item())


@pytest.mark.parametrize("n,h,w", [(1, 8, 8), (2, 10, 16), (3, 50, 200), (37, 18, 224), (1, 600, 24), (250, 18, 40), (372, 10, 16)])
def test_stem_conv_rows_and_runs(n, h, w):
    """Widths whose rows end inside a product, odd numbers of output rows, CTAs that begin and end inside an image; infinite and
    NaN pixels reach the outputs whose window holds them and no other."""
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(5)
    dev = torch.device("cuda", 0)
    x = torch.randn(n, 3, h, w, device=dev).to(dtype=torch.bfloat16, memory_format=torch.channels_last)
    weight = (torch.randn(64, 3, 7, 7, device=dev) * 0.1)
    weight[3, 1, 2, 3] = 0.0
    for bad in (False, True):
        if bad:
            x[0, 1, h // 2, w // 2], x[-1, 0, 0, 0], x[-1, 2, h - 1, w - 1] = math.inf, -math.inf, math.nan
        y, sums = conv.stem_conv(x, weight, segments=n if n < 4 else 1)
        gemm.check_status()
        ref = F.conv2d(x.double(), weight.bfloat16().double(), stride=2, padding=3)
        assert torch.equal(y.isnan(), ref.isnan()) and torch.equal(y.isinf(), ref.isinf())
        ok = ref.isfinite()
        # 147 products in fp32 and one rounding to bf16
        assert float((y.double() - ref)[ok].norm() / ref[ok].norm()) < 2 ** -8
        if not bad:
            part = y.float().view(n if n < 4 else 1, -1, 64, h // 2, w // 2)
            want = torch.stack([part.sum((1, 3, 4)), part.square().sum((1, 3, 4))], 1).view(sums.shape)
            torch.testing.assert_close(sums, want, rtol=1e-4, atol=1e-4 * float(want.abs().max()))


@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan, 9.2e-41, 1.2e-38, 3e38])
def test_stem_conv_weights_that_cannot_be_halved_blindly(value):
    """The middle tap of a row is in two products with half its weight each: infinite, NaN, subnormal (odd) and large weights."""
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(6)
    dev = torch.device("cuda", 0)
    x = torch.randn(2, 3, 12, 24, device=dev).to(dtype=torch.bfloat16, memory_format=torch.channels_last)
    weight = torch.zeros(64, 3, 7, 7, device=dev)
    for c in range(3):
        weight[5 + c, c, 2, 3] = value
        weight[20, c, 6, 2 + c] = value
    scale = 2.0 ** 126 if abs(value) < 1e-30 else 2.0 ** -20 if value == 3e38 else 1.0
    x = (x.double() * scale).to(torch.bfloat16)
    y, _ = conv.stem_conv(x, weight, want_sums=False)
    gemm.check_status()
    ref = F.conv2d(x.double(), weight.bfloat16().double(), stride=2, padding=3)
    assert torch.equal(y.isnan(), ref.isnan()) and torch.equal(y.isinf(), ref.isinf())
    ok = ref.isfinite()
    assert ((y.double() - ref)[ok].abs() <= 2.0 ** -8 * ref[ok].abs()).all() and (math.isfinite(value) == bool(ok.all()))


def test_fused_partition_matches_plain_sequential():
    """conv1 -> bn1 -> relu -> maxpool -> linear head -> bn1d -> relu run through FusedSequential give the same
    outputs, gradients and BatchNorm statistics as the plain modules."""
    from tspipe_b200.batchnorm import DeferredBatchNorm
    from tspipe_b200.ops import gemm
    from tspipe_b200.ops.pool import MaxPool3x3s2
    from tspipe_b200.runtime.fuse import FusedSequential, fuse_partition
    torch.manual_seed(1)
    dev = torch.device("cuda", 0)

    def build():
        return nn.Sequential(nn.Conv2d(3, 64, 7, stride=2, padding=3, bias=False), DeferredBatchNorm(64, chunks=10 ** 9),
                             nn.ReLU(), MaxPool3x3s2(), nn.AdaptiveAvgPool2d(1), nn.Flatten(), nn.Linear(64, 32),
                             DeferredBatchNorm(32, chunks=10 ** 9), nn.ReLU()).to(dev).to(memory_format=torch.channels_last)
    plain = build()
    fused = copy.deepcopy(plain)
    fuse_partition(fused)
    assert isinstance(fused, FusedSequential) and list(fused.state_dict()) == list(plain.state_dict())
    x = torch.randn(16, 3, 64, 64, device=dev).to(dtype=torch.bfloat16, memory_format=torch.channels_last)
    outs = []
    for net in (plain, fused):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = net(x)
        y.float().square().mean().backward()
        outs.append(y)
    gemm.check_status()
    torch.testing.assert_close(outs[1].float(), outs[0].float(), rtol=3e-2, atol=3e-2)
    for (k, p), q in zip(plain.named_parameters(), fused.parameters()):
        torch.testing.assert_close(q.grad, p.grad, rtol=5e-2, atol=5e-2 * max(p.grad.abs().max().item(), 1e-3), msg=k)
    torch.testing.assert_close(fused[1].sum, plain[1].sum, rtol=1e-2, atol=1.0)
    torch.testing.assert_close(fused[1].sum_squares, plain[1].sum_squares, rtol=1e-2, atol=1.0)


def test_stem_conv_statistics_per_group_of_images():
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(2)
    dev = torch.device("cuda", 0)
    x = torch.randn(6, 3, 32, 32, device=dev).to(dtype=torch.bfloat16, memory_format=torch.channels_last)
    x[3:] *= 3.0
    weight = torch.randn(64, 3, 7, 7, device=dev) * 0.1
    y, sums = conv.stem_conv(x, weight, segments=2)
    gemm.check_status()
    yf = y.float()
    sums = sums.view(2, 128)
    for g, part in enumerate((yf[:3], yf[3:])):
        torch.testing.assert_close(sums[g, :64], part.sum((0, 2, 3)), rtol=1e-3, atol=1e-2)
        torch.testing.assert_close(sums[g, 64:], (part * part).sum((0, 2, 3)), rtol=1e-3, atol=1e-2)


# (input shape NCHW, cout, kernel, stride, segments)
IGEMM_CASES = [
    ((4, 64, 16, 16), 256, 1, 1, 1),      # 1x1: plain GEMM over 1024 pixels
    ((8, 256, 8, 8), 64, 1, 1, 2),        # narrow output, two view segments
    ((3, 128, 10, 10), 64, 1, 1, 1),      # 300 pixels: ragged last tile (no statistics possible)
    ((4, 64, 14, 14), 64, 3, 1, 2),       # 3x3: boxes of 14 x 7 pixels, odd number of (tap, ci) blocks
    ((2, 64, 9, 9), 128, 3, 1, 1),        # odd width: 81-pixel boxes (zero rows in the weight-gradient K loop)
    ((8, 128, 7, 7), 128, 3, 1, 2),       # 7 x 7 images: two images per box
    ((2, 64, 12, 12), 128, 3, 2, 1),      # stride 2 through the parity views
    ((2, 128, 56, 56), 128, 3, 2, 2),     # ResNet-50 layer2 shape: 28 x 4 boxes
    ((2, 128, 8, 8), 256, 1, 2, 1),       # 1x1 stride 2 (downsample branch)
    ((2, 256, 56, 56), 64, 1, 1, 2),      # ResNet-50 layer1 conv1
    ((2, 512, 16, 8), 1024, 1, 1, 2),
    ((1, 64, 130, 6), 64, 3, 1, 1),       # wider than one box
]


@pytest.mark.parametrize("shape,cout,k,stride,segs", IGEMM_CASES)
def test_igemm_convolution_forward_backward_and_statistics(shape, cout, k, stride, segs):
    """Implicit-GEMM convolution on tcgen05: output, per-segment channel statistics, data and weight gradient against
    F.conv2d in fp32 (same bf16-rounded operands)."""
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(3)
    dev = torch.device("cuda", 0)
    x = torch.randn(shape, device=dev).to(dtype=torch.bfloat16, memory_format=torch.channels_last).requires_grad_()
    m = nn.Conv2d(shape[1], cout, k, stride=stride, padding=(k - 1) // 2, bias=False).to(dev)
    m = m.to(memory_format=torch.channels_last)
    assert conv.igemm_eligible(m, x)
    conv.clear_weight_cache()
    y, sums = conv.conv2d(x, m.weight, stride, want_sums=True, segments=segs)
    gemm.check_status()
    xr = x.detach().float().requires_grad_()
    wr = m.weight.detach().bfloat16().float().requires_grad_()
    ref = F.conv2d(xr, wr, stride=stride, padding=(k - 1) // 2)
    assert y.shape == ref.shape and y.is_contiguous(memory_format=torch.channels_last)
    torch.testing.assert_close(y.float(), ref, rtol=2e-2, atol=2e-2)
    yf = y.float()
    if sums is not None:
        sums = sums.view(segs, 2, cout)
        for g, part in enumerate(yf.chunk(segs)):
            torch.testing.assert_close(sums[g, 0], part.sum((0, 2, 3)), rtol=1e-3, atol=2e-2)
            torch.testing.assert_close(sums[g, 1], (part * part).sum((0, 2, 3)), rtol=1e-3, atol=2e-2)
    else:
        pixels = shape[0] // segs * ref.shape[2] * ref.shape[3]
        assert k == 1 and stride == 1 and pixels % 128 != 0     # the only case without statistics: ragged 1x1 tiles
    g = torch.randn_like(y)
    y.backward(g)
    gemm.check_status()
    ref.backward(g.float())
    torch.testing.assert_close(x.grad.float(), xr.grad, rtol=3e-2, atol=3e-2 * max(xr.grad.abs().max().item(), 1.0))
    torch.testing.assert_close(m.weight.grad, wr.grad, rtol=5e-2, atol=5e-2 * wr.grad.abs().max().item())
    # a second backward ADDS into the existing fp32 gradient (the kernel accumulates in place)
    y2, _ = conv.conv2d(x, m.weight, stride)
    y2.backward(g)
    gemm.check_status()
    torch.testing.assert_close(m.weight.grad, 2 * wr.grad, rtol=5e-2, atol=1e-1 * wr.grad.abs().max().item())


@pytest.mark.parametrize("n,h,w,cin,cout", [(1, 1, 1, 64, 64), (1, 7, 7, 64, 128), (3, 10, 10, 128, 64), (37, 14, 14, 256, 1024),
                                            (64, 7, 7, 512, 2048), (64, 7, 7, 2048, 512)])
def test_statistics_of_one_group_with_a_ragged_last_tile(n, h, w, cin, cout):
    """1x1: the rows that the last tile of 128 pixels lacks count as zeros, also where a weight is infinite."""
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(43)
    dev = torch.device("cuda", 0)
    x = torch.rand(n, cin, h, w, device=dev).add(0.5).to(dtype=torch.bfloat16, memory_format=torch.channels_last)
    weight = (torch.randn(cout, cin, 1, 1, device=dev) / cin ** 0.5).to(memory_format=torch.channels_last)
    weight[3, 5] = float("inf")
    conv.clear_weight_cache()
    y, sums = conv.conv2d(x, weight, 1, want_sums=True)
    gemm.check_status()
    terms = y.double()
    assert terms[:, 3].eq(float("inf")).all()
    for got, part in zip(sums.view(2, cout).double(), (terms, terms * terms)):
        want, size = part.sum((0, 2, 3)), part.abs().sum((0, 2, 3))
        assert got[3] == float("inf")
        keep = torch.arange(cout, device=dev) != 3
        assert ((got - want).abs() <= 2.0 ** -16 * size)[keep].all()     # fp32 sums of some hundred terms each, added up


# (images, height, width, cin, cout, kernel): the pixel tiles around the numbers where the channel tile changes its width (74
# tiles of 256 channels run at once in halves on 148 SMs, 37 in quarters), and grids of several tiles per block
TILE_CASES = [(37, 16, 16, 256, 256, 1), (75, 16, 8, 256, 256, 1), (37, 16, 8, 256, 256, 1), (19, 16, 16, 256, 256, 3),
              (37, 16, 16, 256, 256, 3), (38, 16, 16, 256, 256, 3), (74, 7, 7, 128, 256, 3), (148, 7, 7, 128, 256, 3),
              (150, 7, 7, 128, 256, 3), (16, 56, 56, 64, 256, 1), (16, 56, 56, 64, 128, 1), (16, 56, 56, 128, 64, 1),
              (16, 56, 56, 512, 128, 1), (8, 56, 56, 128, 128, 3), (64, 14, 14, 448, 512, 1)]


@pytest.mark.parametrize("n,h,w,cin,cout,k", TILE_CASES)
def test_convolution_channel_tiles_and_epilogue_warps(n, h, w, cin, cout, k):
    """Output, statistics of one and of several image groups, and the data gradient: fp32 sums, rounded once to bf16."""
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(31)
    dev = torch.device("cuda", 0)
    x = torch.randn(n, cin, h, w, device=dev).to(dtype=torch.bfloat16, memory_format=torch.channels_last).requires_grad_()
    weight = (torch.randn(cout, cin, k, k, device=dev) / (k * cin ** 0.5)).to(memory_format=torch.channels_last).requires_grad_()
    conv.clear_weight_cache()
    wr = weight.detach().bfloat16().double()
    want = F.conv2d(x.detach().double(), wr, padding=(k - 1) // 2)
    size = F.conv2d(x.detach().double().abs(), wr.abs(), padding=(k - 1) // 2)
    for segs in (1, 2 if n % 4 == 0 else 1):
        y, sums = conv.conv2d(x, weight, 1, want_sums=True, segments=segs)
        gemm.check_status()
        # a product rounds once to 8 bits; its fp32 sum over k * k * cin terms errs by 2^-22 of the terms' sizes at most
        assert ((y.double() - want).abs() <= want.abs() * 2.0 ** -8 + size * 2.0 ** -20).all()
        if sums is None:
            assert k == 1 and (n // segs * h * w) % 128
            continue
        for s, part in zip(sums.view(segs, 2, cout).double(), y.detach().double().chunk(segs)):
            for got, terms in zip(s, (part, part * part)):
                bound = 2.0 ** -16 * terms.abs().sum((0, 2, 3))       # fp32 sums of some hundred terms each, added up
                assert ((got - terms.sum((0, 2, 3))).abs() <= bound).all()
    g = torch.randn(y.shape, device=dev).to(dtype=torch.bfloat16, memory_format=torch.channels_last)
    (dx,) = torch.autograd.grad(y, x, g)
    gemm.check_status()
    want = torch.nn.grad.conv2d_input(x.shape, wr, g.double(), padding=(k - 1) // 2)
    size = torch.nn.grad.conv2d_input(x.shape, wr.abs(), g.double().abs(), padding=(k - 1) // 2)
    assert ((dx.double() - want).abs() <= want.abs() * 2.0 ** -8 + size * 2.0 ** -20).all()


def test_bottleneck_on_igemm_convolutions_matches_library_path():
    from tspipe_b200.batchnorm import DeferredBatchNorm
    from tspipe_b200.models.resnet import Bottleneck
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(4)
    dev = torch.device("cuda", 0)
    down = nn.Sequential(nn.Conv2d(256, 512, 1, stride=2, bias=False), nn.BatchNorm2d(512))
    blk = DeferredBatchNorm.convert_deferred_batch_norm(Bottleneck(256, 128, 2, down), chunks=10 ** 9).to(dev)
    blk = blk.to(memory_format=torch.channels_last)
    x = torch.randn(8, 256, 16, 16, device=dev).to(dtype=torch.bfloat16, memory_format=torch.channels_last)
    outs, grads = [], []
    for flag in (False, True):
        conv.set_igemm(flag)
        conv.clear_weight_cache()
        try:
            xi = x.clone().requires_grad_()
            blk.zero_grad()
            with torch.autocast("cuda", dtype=torch.bfloat16):
                y = blk(xi)
            y.float().square().mean().backward()
        finally:
            conv.set_igemm(True)
        outs.append(y.float())
        grads.append([xi.grad.float()] + [p.grad.clone() for p in blk.parameters()])
    gemm.check_status()
    torch.testing.assert_close(outs[1], outs[0], rtol=3e-2, atol=3e-2)
    for a, b in zip(grads[1], grads[0]):
        torch.testing.assert_close(a, b, rtol=5e-2, atol=5e-2 * max(b.abs().max().item(), 1e-3))


@pytest.mark.parametrize("mode", ["stream", "side stream", "graph", "forked graph"])
def test_kernels_that_start_early_wait_for_what_they_read(mode):
    """Convolutions and products in a chain whose every launch overwrites what the next one reads, beside library kernels, a
    memset and a second stream: the same bits as with a synchronisation after each launch."""
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(41)
    dev = torch.device("cuda", 0)
    x0 = torch.randn(8, 64, 28, 28, device=dev).to(dtype=torch.bfloat16, memory_format=torch.channels_last)
    w1 = (torch.randn(256, 64, 1, 1, device=dev) * 0.2).to(memory_format=torch.channels_last)
    w2 = (torch.randn(64, 256, 1, 1, device=dev) * 0.1).to(memory_format=torch.channels_last)
    w3 = (torch.randn(64, 64, 3, 3, device=dev) * 0.08).to(memory_format=torch.channels_last)
    lin = (torch.randn(64, 64, device=dev) * 0.2).bfloat16()
    buf, side_out = torch.empty_like(x0), torch.empty_like(x0)
    side = torch.cuda.Stream()

    def chain(wait, fork):
        buf.copy_(x0)
        for i in range(6):
            y = conv.conv2d(buf, w1, 1)[0]
            wait()
            z = conv.conv2d(y, w2, 1)[0]
            wait()
            if fork:
                side.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(side):
                    side_out.copy_(conv.conv2d(z, w3, 1)[0])
                torch.cuda.current_stream().wait_stream(side)
            buf.zero_()
            t = conv.conv2d(z, w3, 1)[0]
            wait()
            buf.add_(t)
            rows = buf.permute(0, 2, 3, 1).reshape(-1, 64)
            p = gemm.matmul_nt(rows, lin)
            wait()
            rows.copy_(p.to(rows.dtype) / (p.float().abs().max() + 1))
        return buf

    with torch.no_grad():
        want = chain(torch.cuda.synchronize, False).clone()
        for _ in range(3):
            if mode == "stream":
                got = chain(lambda: None, False)
            elif mode == "side stream":
                with torch.cuda.stream(side):
                    side.wait_stream(torch.cuda.default_stream())
                    got = chain(lambda: None, False)
            else:
                graph = torch.cuda.CUDAGraph()
                torch.cuda.synchronize()
                with torch.cuda.graph(graph):
                    got = chain(lambda: None, mode == "forked graph")
                graph.replay()
                graph.replay()
            torch.cuda.synchronize()
            assert torch.isfinite(want).all() and torch.equal(got, want)
    gemm.check_status()


def _module_of_early_kernels(kind, dev):
    """A fused block and its input: what convolutions and products follow directly, and their gradients."""
    from tspipe_b200.batchnorm import BatchNormGroup, DeferredBatchNorm
    from tspipe_b200.models.resnet import Bottleneck, mlp_head_children
    from tspipe_b200.models.vit import Block, ViTConfig
    from tspipe_b200.runtime.fuse import fuse_partition
    torch.manual_seed(43)
    if kind == "vit block":
        m, x = Block(ViTConfig(embed_dim=384, num_heads=6)), torch.randn(16, 65, 384, device=dev).bfloat16()
    elif kind == "head":
        m, x = nn.Sequential(mlp_head_children(512, 1024, 256)), torch.randn(512, 512, device=dev).bfloat16()
    else:                                     # the addend of the first data gradient: on a flat pixel grid, on a strided one
        down = None if kind == "block" else nn.Sequential(nn.Conv2d(256, 512, 1, stride=2, bias=False), nn.BatchNorm2d(512))
        m = nn.Sequential(Bottleneck(256, 64, 1, None) if down is None else Bottleneck(256, 128, 2, down))
        x = torch.randn(16, 256, 28, 28, device=dev).to(dtype=torch.bfloat16, memory_format=torch.channels_last)
    m = fuse_partition(DeferredBatchNorm.convert_deferred_batch_norm(m.to(dev).to(memory_format=torch.channels_last), chunks=1))
    return m, BatchNormGroup(m, chunks=1), x


@pytest.mark.parametrize("mode", ["stream", "graph"])
@pytest.mark.parametrize("kind", ["block", "strided block", "head", "vit block"])
def test_kernels_that_start_early_behind_normalisations(kind, mode, monkeypatch):
    """Forward and backward of blocks in which normalisations and GELU let convolutions, products and weight gradients start
    as soon as they are placed themselves, on one input buffer that every pass overwrites: what a run with a synchronisation
    after each call gives.  Sums that atomics add up differ in their last bits, and a value next to a ReLU's corner may take its gradient
    along; a tile that was read too early is a share of some 10^-2 of a tensor's elements, far off."""
    from tspipe_b200.ops import bn, conv, fused, gemm
    from tspipe_b200.runtime.stage_graph import capture
    dev = torch.device("cuda", 0)
    m, group, x0 = _module_of_early_kernels(kind, dev)
    buf, params = torch.empty_like(x0).requires_grad_(), list(m.parameters())
    g = None

    def chain():
        nonlocal g
        out = []
        for i in range(3):
            with torch.no_grad():
                buf.copy_(x0.roll(i, 0) * (i + 1))
            with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False), bn.segments(2):
                y = m(buf)
            if g is None:
                g = torch.randn(y.shape, device=dev).to(y.dtype)
                g = g.to(memory_format=torch.channels_last) if g.dim() == 4 else g
            grads = torch.autograd.grad(y, [buf] + params, g)
            # (without the gradient of a bias in front of a BatchNorm, which is rounding alone)
            out += [y.detach()] + [t for j, t in enumerate(grads) if (kind, j) != ("head", 2)]
        return out

    count = fused._count
    with monkeypatch.context() as patch:
        patch.setattr(fused, "_count", lambda *a: (count(*a), torch.cuda.synchronize())[0])
        chain()
        want = [t.clone() for t in chain()]
    torch.cuda.synchronize()
    for _ in range(3):
        conv.clear_weight_cache()
        gemm.clear_weight_cache()
        if mode == "stream":
            got = chain()
        else:
            graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
            got = capture(graph, stream, torch.cuda.graph_pool_handle(), chain)
            graph.replay()
            graph.replay()
        torch.cuda.synchronize()
        gemm.check_status()
        for a, b in zip(got, want):
            rms = b.float().square().mean().sqrt()
            off = ((a.float() - b.float()).abs() > 0.5 * rms).float().mean()
            assert b.isfinite().all() and float(rms) > 0 and float(off) < 2e-3, (kind, tuple(b.shape), float(off))
