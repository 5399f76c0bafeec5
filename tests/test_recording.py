"""What the launches of a stage under recording share, and where they take other ways than eager ones."""
import threading

import pytest
import torch
from torch import nn

from tspipe_b200.ops import fused
from tspipe_b200.runtime.state import FlatParams


def _flat(*shapes):
    torch.manual_seed(0)
    ps = [nn.Parameter(torch.randn(*s)) for s in shapes]
    ps = [nn.Parameter(p.detach().to(memory_format=torch.channels_last)) if p.dim() == 4 else p for p in ps]
    return ps, FlatParams(ps, torch.device("cpu"), with_grad=True)


def test_recorded_copies_of_a_flat_buffer():
    """One cast for all parameters, each copy with its parameter's strides; row slices map to the same slice."""
    ps, flat = _flat((8, 16, 3, 3), (24, 40), (5,))
    with fused.capturing():
        for p in ps:
            c = fused.recorded_bf16(p)
            assert c.stride() == p.stride() and torch.equal(c, p.detach().bfloat16())
        assert torch.equal(fused.recorded_bf16(ps[1][8:16]), ps[1][8:16].detach().bfloat16())
        assert len(fused._recording().copies) == 1


def test_recorded_copy_of_a_computed_weight_is_its_own():
    """A computed weight's memory may be given back within the recording and be the next one's."""
    with fused.capturing():
        for value in range(1, 9):
            w = torch.full((2, 512, 512), float(value))
            assert torch.equal(fused.recorded_bf16(w[0]), torch.full((512, 512), float(value)).bfloat16())
            del w


def test_recorded_copy_follows_a_parameter_written_in_place():
    ps, flat = _flat((16, 16), (32, 16))
    with fused.capturing(), torch.no_grad():
        fused.recorded_bf16(ps[0])
        ps[1].mul_(3.0)                                 # a layer that renormalises its weight before it uses it
        assert torch.equal(fused.recorded_bf16(ps[1]), ps[1].bfloat16())
        assert torch.equal(fused.recorded_bf16(ps[0]), ps[0].bfloat16())


def test_gradients_are_added_in_place_only_where_they_are_recorded(monkeypatch):
    """Not on another thread's stream while one is recorded, and not past a parameter's hooks."""
    ps, flat = _flat((7,), (9,), (11,))
    ps[1].register_hook(lambda g: 2 * g)
    ps[2].register_post_accumulate_grad_hook(lambda p: None)
    monkeypatch.setattr(fused, "_stream_key", threading.get_ident)       # a stream of its own per thread
    seen = []
    with fused.capturing():
        assert fused.recorded_grad(ps[0]) is ps[0].grad
        assert fused.recorded_grad(ps[1]) is None and fused.recorded_grad(ps[2]) is None
        t = threading.Thread(target=lambda: seen.append(fused.recorded_grad(ps[0])))
        t.start()
        t.join()
    assert seen == [None] and fused.recorded_grad(ps[0]) is None


# ---- on the GPU ---------------------------------------------------------------------------------------------------
def _stage(kind):
    """``(children, input, output gradient's shape, views)`` of a small stage of each kind."""
    from tspipe_b200.models.bert import BertConfig, EncoderLayer
    from tspipe_b200.models.resnet import Bottleneck, mlp_head_children, resnet_trunk_children
    from tspipe_b200.models.vit import Block, ViTConfig
    dev = torch.device("cuda", 0)

    def image(n, c, s):
        return torch.randn(n, s, s, c, device=dev).bfloat16().permute(0, 3, 1, 2)
    if kind == "vit":
        return [Block(ViTConfig(embed_dim=128, num_heads=2))], torch.randn(4, 65, 128, device=dev).bfloat16(), (4, 65, 128), 1
    if kind == "bert":
        x = {"hidden": torch.randn(4, 48, 128, device=dev).bfloat16(), "mask": torch.ones(4, 48, dtype=torch.int64, device=dev)}
        x["mask"][1, 30:] = 0
        return [EncoderLayer(BertConfig(hidden=128, heads=2, ffn=256, dropout=0.0))], x, (4, 48, 128), 1
    if kind == "head":
        return list(mlp_head_children(256, 512, 128).values()), torch.randn(256, 256, device=dev).bfloat16(), (256, 128), 2
    if kind == "stem":
        ch = resnet_trunk_children("resnet18")
        return [ch[k] for k in ("conv1", "bn1", "relu", "maxpool")], image(4, 3, 32), (4, 64, 8, 8), 2
    if kind == "bottleneck":
        return [Bottleneck(256, 64, 1, None)], image(4, 256, 14), (4, 256, 14, 14), 2
    down = nn.Sequential(nn.Conv2d(128, 256, 1, stride=2, bias=False), nn.BatchNorm2d(256))
    return [Bottleneck(128, 64, 2, down)], image(4, 128, 14), (4, 256, 7, 7), 2


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["vit", "bert", "head", "stem", "bottleneck", "strided"])
def test_recorded_stage_adds_the_eager_gradients(kind, monkeypatch):
    """A stage's recorded forward and backward, replayed twice without clearing, leave twice the eager gradient in every
    parameter, one-dimensional ones and one with a hook included.  A replay runs the eager launches on the same values; only
    atomic sums come in another order, so that a bf16 rounding may fall the other way here and there: 2 % of a gradient's norm
    (a missing or doubled one is off by half), and of the typical norm where a gradient is a sum that cancels."""
    from tspipe_b200.batchnorm import BatchNormGroup, DeferredBatchNorm
    from tspipe_b200.ops import bn, gemm
    from tspipe_b200.runtime.fuse import fuse_partition
    from tspipe_b200.runtime.stage_graph import StudentStageGraphs
    torch.manual_seed(3)
    dev = torch.device("cuda", 0)
    children, x, oshape, views = _stage(kind)
    m = nn.Sequential(*children).to(dev).to(memory_format=torch.channels_last)
    with torch.no_grad():
        for p in m.parameters():
            if p.dim() == 1:
                p.add_(0.2 * torch.randn_like(p))
    m = fuse_partition(DeferredBatchNorm.convert_deferred_batch_norm(m, chunks=10))
    BatchNormGroup(m, chunks=10)
    flat = FlatParams(list(m.parameters()), dev, with_grad=True)
    one_d = [p for p in flat.params if p.dim() == 1]
    one_d[-1].register_hook(lambda g: 3 * g)
    xs = x if isinstance(x, torch.Tensor) else x["hidden"]
    xs.requires_grad_(kind != "stem")
    g = torch.randn(oshape, device=dev).bfloat16() * 1e-2
    g = g.contiguous(memory_format=torch.channels_last) if g.dim() == 4 else g

    def eager():
        flat.zero_grad()
        with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False), bn.segments(views):
            y = m(x)
        y = y if isinstance(y, torch.Tensor) else y["hidden"]
        y.backward(g)
        flat.collect_stray_grads()
        return y.detach(), flat.grad.clone()
    y, want = eager()
    in_place = []
    plain = fused.recorded_grad
    monkeypatch.setattr(fused, "recorded_grad", lambda p: in_place.append(plain(p)) or in_place[-1])
    stage = StudentStageGraphs(m, flat, True, dev)
    out, slot = None, None
    for _ in range(3):
        out, slot = stage.forward(0, x, views)
    assert slot is not None and any(t is not None for t in in_place)
    flat.zero_grad()
    stage.backward(slot, [g])
    _, slot = stage.forward(0, x, views)
    dx = stage.backward(slot, [g])
    gemm.check_status()
    out = out if isinstance(out, torch.Tensor) else out["hidden"]
    assert float((out.detach() - y).float().norm()) <= 1e-2 * float(y.float().norm())
    typical = float((want.norm() / want.count_nonzero().sqrt()))
    for i, p in enumerate(flat.params):
        a, b = flat._view(flat.grad, i, p.data), 2 * flat._view(want, i, p.data)
        assert float((a - b).norm()) <= 0.02 * (float(b.norm()) + typical * p.numel() ** 0.5), (kind, i, tuple(p.shape))
    if kind != "stem":
        assert float((dx[0] - xs.grad).float().norm()) <= 0.02 * float(xs.grad.float().norm())
