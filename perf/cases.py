"""The work that a user of the framework has it do, as cases that can be timed and checked.

A case is one pass through a public entry point, at a size from the benchmark workloads (BYOL ResNet-50, MoCo-v3 ViT,
DistilBERT, soft-target KD) or from the range around them:

``byol_loss`` / ``moco_loss`` / ``kd_loss`` / ``distil_loss``  loss value and student gradients (``losses.py``)
``lars`` / ``adamw`` / ``sgd``  one optimizer step over a partition's flat parameters with the momentum-teacher update
``head``       a BYOL projector (Linear, BatchNorm, ReLU, Linear), forward and backward
``stem``       the ResNet stem (7x7 convolution, BatchNorm, ReLU, max-pool), forward and backward
``bottleneck`` one ResNet bottleneck block, forward and backward
``vit_block``  one ViT transformer block, forward and backward, or the teacher's forward alone
``bert_layer`` one BERT encoder layer with a padding mask: the frozen teacher's forward
``trunk``      the whole ResNet trunk of a target network, forward with batch statistics

Modules compute in bf16 under autocast with fp32 parameters in flat buffers, as the runtime keeps them: gradients are
added into the flat gradient buffer.  With ``graph`` the module's forward and backward are recorded into CUDA graphs
and replayed, which is how the executor runs a stage after its first calls; without it they run eagerly, and the bf16
weight copies live for one step (they are dropped after every pass, as the executor does after every optimizer step).  Tolerances are about four times the errors measured against 64-bit
arithmetic on a B200.
"""
from __future__ import annotations

import contextlib
import math
from types import SimpleNamespace

import torch
import torch.nn.functional as F
from torch import nn

DEV = "cuda"


# -------------------------------------------------------------------------------------------------------------------
# the cases
# -------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the loss of one BYOL step at a small per-GPU batch: launches and latency only
        dict(name="byol_loss_128", kind="byol_loss", rows=128, dim=256, dtype="bf16"),
        # contrastive loss of MoCo-v3 with a whole global batch of keys on one GPU
        dict(name="moco_loss_4096", kind="moco_loss", rows=4096, dim=256, dtype="bf16"),
        # DistilBERT objective over the vocabulary, 16 sequences of 512 tokens
        dict(name="distil_loss_16x512", kind="distil_loss", batch=16, length=512, vocab=30528, hidden=768),
        # LARS with the momentum update over ResNet-50 sized parameters
        dict(name="lars_25m", kind="lars", params=25_557_032, ema=True),
        # AdamW with the momentum update over ViT-B sized parameters
        dict(name="adamw_86m", kind="adamw", params=86_567_656, ema=True),
        # BYOL projector at the batch of two stacked views of 128 images
        dict(name="head_256", kind="head", rows=256, din=2048, hidden=4096, dout=256, views=2, graph=False),
        # the stem on two stacked views of 64 images, the head of the headline benchmark's network
        dict(name="stem_128", kind="stem", images=128, side=224, views=2, graph=True),
        # largest residual block of ResNet-50 (layer 1) on two stacked views of 128 images
        dict(name="layer1_256", kind="bottleneck", images=256, side=56, cin=256, planes=64, stride=1, views=2,
             graph=True),
        # strided block with a projection shortcut at an odd batch
        dict(name="layer3_down_37", kind="bottleneck", images=37, side=28, cin=512, planes=256, stride=2, views=1,
             graph=False),
        # student block of ViT-B, 197 tokens
        dict(name="vit_b_train_64", kind="vit_block", batch=64, tokens=197, dim=768, heads=12, train=True, graph=True),
        # frozen BERT-base teacher, 32 sequences of 512 tokens with padding
        dict(name="bert_teacher_32x512", kind="bert_layer", batch=32, length=512, hidden=768, heads=12, ffn=3072,
             graph=True),
        # whole trunk of BYOL's target network on one microbatch
        dict(name="resnet50_target_64", kind="trunk", arch="resnet50", images=64, side=224, graph=True),
    ]


def _log_int(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))
    return max(lo, min(hi, int(v) // step * step))


def draw(rng):
    case = _draw(rng)
    if case["kind"] not in _LOSSES + _OPTIMS:
        case["graph"] = rng.random() < 0.75
    return case


def _draw(rng):
    kind = rng.choice(["byol_loss", "moco_loss", "kd_loss", "distil_loss", "lars", "adamw", "sgd", "head", "stem",
                       "bottleneck", "bottleneck", "bottleneck", "vit_block", "vit_block", "bert_layer", "trunk"])
    if kind == "byol_loss":
        return dict(kind=kind, rows=_log_int(rng, 16, 2048), dim=rng.choice([128, 256, 512]),
                    dtype=rng.choice(["bf16", "fp32"]))
    if kind == "moco_loss":
        return dict(kind=kind, rows=rng.choice([_log_int(rng, 128, 4096, 128), _log_int(rng, 33, 3000)]), dim=256,
                    dtype=rng.choice(["bf16", "fp32"]))
    if kind == "kd_loss":
        return dict(kind=kind, rows=_log_int(rng, 16, 4096), classes=rng.choice([10, 100, 1000, 1000, 1001, 21841]),
                    dtype=rng.choice(["bf16", "fp32"]))
    if kind == "distil_loss":
        return dict(kind=kind, batch=_log_int(rng, 1, 16), length=rng.choice([64, 128, 200, 384, 512]), vocab=30528,
                    hidden=768)
    if kind in ("lars", "adamw", "sgd"):
        return dict(kind=kind, params=_log_int(rng, 500_000, 86_000_000), ema=rng.random() < 0.6)
    if kind == "head":
        views = rng.choice([1, 2])
        return dict(kind=kind, rows=_log_int(rng, 64, 1024) * views, din=rng.choice([256, 512, 2048]), hidden=4096,
                    dout=256, views=views)
    if kind == "stem":
        views = rng.choice([1, 2])
        return dict(kind=kind, images=_log_int(rng, 8, 64) * views, side=rng.choice([96, 160, 192, 224]), views=views)
    if kind == "bottleneck":
        views = rng.choice([1, 2])
        layer = rng.choice([1, 2, 3, 4])
        planes, side = 32 * 2 ** layer, 112 // 2 ** layer
        first = rng.random() < 0.35
        stride = 2 if first and layer > 1 else 1
        cin = (64 if layer == 1 else 2 * planes) if first else 4 * planes
        return dict(kind=kind, images=_log_int(rng, 8, 96) * views, side=side * stride, cin=cin, planes=planes,
                    stride=stride, views=views)
    if kind == "vit_block":
        dim, heads = rng.choice([(384, 12), (768, 12), (768, 12), (1024, 16)])
        tokens = rng.choice([65, 145, 197, 197, 257])
        most = min(64, 64 * 197 * 768 * 768 // (tokens * dim * dim))       # the work of the largest listed block
        return dict(kind=kind, batch=_log_int(rng, 4, most), tokens=tokens, dim=dim, heads=heads,
                    train=rng.random() < 0.6)
    if kind == "bert_layer":
        return dict(kind=kind, batch=_log_int(rng, 2, 32), length=rng.choice([64, 128, 250, 384, 512]), hidden=768,
                    heads=12, ffn=3072)
    return dict(kind=kind, arch=rng.choice(["resnet18", "resnet50"]), images=_log_int(rng, 8, 64),
                side=rng.choice([96, 160, 224]))


# -------------------------------------------------------------------------------------------------------------------
# inputs, from the seed alone
# -------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(0x5EED ^ (int(seed) * 2654435761 % (1 << 31)))


def _randn(g, *shape, scale=1.0):
    return torch.randn(*shape, generator=g, device=DEV) * scale


def _dt(case):
    return torch.float32 if case.get("dtype") == "fp32" else torch.bfloat16


def _image_like(g, n, c, h, w, relu=False):
    x = torch.randn(n, h, w, c, generator=g, device=DEV, dtype=torch.bfloat16)
    return (x.relu_() if relu else x).permute(0, 3, 1, 2)          # channels-last


def _grad_like(g, n, c, h, w):
    """An output gradient of random sign and bounded magnitude, channels-last."""
    x = torch.rand(n, h, w, c, generator=g, device=DEV, dtype=torch.float32) * 2 - 1
    return ((x + 0.5 * x.sign()) * 1e-2).to(torch.bfloat16).permute(0, 3, 1, 2)


def _loss_inputs(case, seed):
    g = _gen(seed)
    if case["kind"] in ("byol_loss", "moco_loss"):
        base = [_randn(g, case["rows"], case["dim"]) for _ in range(2)]
        ts = [(base[i % 2] + 0.7 * _randn(g, case["rows"], case["dim"])).to(_dt(case)) for i in range(4)]
        return dict(o1=ts[0], o2=ts[1], t1=ts[2], t2=ts[3])
    if case["kind"] == "kd_loss":
        n, c = case["rows"], case["classes"]
        return dict(s=_randn(g, n, c, scale=2.0).to(_dt(case)), t=_randn(g, n, c, scale=2.0).to(_dt(case)),
                    labels=torch.randint(0, c, (n,), generator=g, device=DEV))
    b, l, v, h = case["batch"], case["length"], case["vocab"], case["hidden"]
    s = torch.randn(b, l, v, generator=g, device=DEV, dtype=torch.bfloat16) * 1.5
    t = torch.randn(b, l, v, generator=g, device=DEV, dtype=torch.bfloat16) * 1.5
    sh, th = _randn(g, b, l, h).bfloat16(), _randn(g, b, l, h).bfloat16()
    lens = torch.randint(max(1, l // 2), l + 1, (b, 1), generator=g, device=DEV)
    attn = (torch.arange(l, device=DEV)[None] < lens).to(torch.int64)
    labels = torch.randint(0, v, (b, l), generator=g, device=DEV)
    masked = (torch.rand(b, l, generator=g, device=DEV) < 0.15) & (attn > 0)
    labels = torch.where(masked, labels, torch.full_like(labels, -100))
    return dict(s=s, t=t, sh=sh, th=th, labels=labels, attn=attn, n_lab=int((labels >= 0).sum()),
                n_sel=int(attn.sum()))


def _param_shapes(total):
    """Tensors of a network with about ``total`` parameters: matrices of growing width with their vectors, and one odd
    remainder matrix."""
    shapes, left, i = [], total, 0
    while left > 0:
        d = (256, 512, 1024, 2048)[i % 4]
        m = (d, min(4 * d, 2048))
        if m[0] * m[1] + m[0] > left:
            rows = max(left // 257, 1)
            shapes += [(rows, 257)] if left >= 257 else [(left,)]
            break
        shapes += [m, (m[0],)]
        left -= m[0] * m[1] + m[0]
        i += 1
    return shapes


_HP = {"lars": dict(lr=0.2, weight_decay=1e-6, momentum=0.9), "adamw": dict(lr=1e-3, weight_decay=0.1),
       "sgd": dict(lr=0.05, momentum=0.9, weight_decay=1e-4)}
_EMA = 0.99


def _optim_inputs(case, seed):
    g = _gen(seed)
    shapes = _param_shapes(case["params"])
    ps = [_randn(g, *s, scale=0.05) for s in shapes]
    gs = [_randn(g, *s, scale=0.01) for s in shapes]
    st = [_randn(g, *s, scale=0.01) for s in shapes]
    v = [_randn(g, *s, scale=0.01).square_() for s in shapes] if case["kind"] == "adamw" else None
    ts = [p + _randn(g, *s, scale=0.001) for p, s in zip(ps, shapes)] if case["ema"] else None
    return dict(p=ps, g=gs, m=st, v=v, t=ts)


def _init(module, g):
    """Weights of a network in training: LeCun-scaled matrices, norm scales around one, small biases.  BatchNorm biases
    are around a half, so that fewer activations sit within a rounding error of a ReLU's corner (each one that falls on
    the other side takes its whole gradient along)."""
    with torch.no_grad():
        for p in module.parameters():
            if p.dim() > 1:
                p.copy_(torch.randn(p.shape, generator=g, device=DEV) / math.sqrt(p[0].numel()))
        for m in module.modules():
            if isinstance(m, (nn.BatchNorm1d, nn.BatchNorm2d, nn.LayerNorm)):
                m.weight.copy_(1 + 0.1 * torch.randn(m.weight.shape, generator=g, device=DEV))
                m.bias.copy_(0.1 * torch.randn(m.bias.shape, generator=g, device=DEV))
                if not isinstance(m, nn.LayerNorm):
                    m.bias.add_(0.5)
            elif isinstance(m, nn.Linear) and m.bias is not None:
                m.bias.copy_(0.1 * torch.randn(m.bias.shape, generator=g, device=DEV))
    return module


def _build(case, g):
    """The module of a case with its weights, before the runtime's preparation."""
    kind = case["kind"]
    if kind == "head":
        from tspipe_b200.models.resnet import mlp_head_children
        m = nn.Sequential(mlp_head_children(case["din"], case["hidden"], case["dout"]))
    elif kind == "stem":
        from tspipe_b200.models.resnet import resnet_trunk_children
        ch = resnet_trunk_children("resnet18")
        m = nn.Sequential(*(ch[k] for k in ("conv1", "bn1", "relu", "maxpool")))
    elif kind == "bottleneck":
        from tspipe_b200.models.resnet import Bottleneck
        down = None
        if case["stride"] != 1 or case["cin"] != 4 * case["planes"]:
            down = nn.Sequential(nn.Conv2d(case["cin"], 4 * case["planes"], 1, stride=case["stride"], bias=False),
                                 nn.BatchNorm2d(4 * case["planes"]))
        m = nn.Sequential(Bottleneck(case["cin"], case["planes"], case["stride"], down))
    elif kind == "vit_block":
        from tspipe_b200.models.vit import Block, ViTConfig
        m = nn.Sequential(Block(ViTConfig(embed_dim=case["dim"], num_heads=case["heads"])))
    elif kind == "bert_layer":
        from tspipe_b200.models.bert import BertConfig, EncoderLayer
        m = nn.Sequential(EncoderLayer(BertConfig(hidden=case["hidden"], heads=case["heads"], ffn=case["ffn"])))
    else:
        from tspipe_b200.models.resnet import resnet_trunk_children
        m = nn.Sequential(resnet_trunk_children(case["arch"]))
    return _init(m.to(DEV), g)


def _module_inputs(case, seed):
    """``(module, inputs, output gradient or None)``."""
    g = _gen(seed)
    m = _build(case, g)
    kind = case["kind"]
    if kind == "head":
        return m, _randn(g, case["rows"], case["din"]).bfloat16(), _randn(g, case["rows"], case["dout"], scale=1e-2).bfloat16()
    if kind == "stem":
        n, s = case["images"], case["side"]
        return m, _image_like(g, n, 3, s, s), _grad_like(g, n, 64, s // 4, s // 4)
    if kind == "bottleneck":
        n, s, so = case["images"], case["side"], case["side"] // case["stride"]
        return m, _image_like(g, n, case["cin"], s, s, relu=True), _grad_like(g, n, 4 * case["planes"], so, so)
    if kind == "vit_block":
        shape = (case["batch"], case["tokens"], case["dim"])
        x = _randn(g, *shape).bfloat16()
        return m, x, (_randn(g, *shape, scale=1e-2).bfloat16() if case["train"] else None)
    if kind == "bert_layer":
        b, l = case["batch"], case["length"]
        lens = torch.randint(max(1, l // 2), l + 1, (b, 1), generator=g, device=DEV)
        mask = (torch.arange(l, device=DEV)[None] < lens).to(torch.int64)
        return m.eval(), {"hidden": _randn(g, b, l, case["hidden"]).bfloat16(), "mask": mask}, None
    return m, _image_like(g, case["images"], 3, case["side"], case["side"]), None


_LOSSES = ("byol_loss", "moco_loss", "kd_loss", "distil_loss")
_OPTIMS = ("lars", "adamw", "sgd")


def _trains(case):
    return case["kind"] in ("head", "stem", "bottleneck") or (case["kind"] == "vit_block" and case["train"])


def prepare(case, seed):
    kind = case["kind"]
    if kind in _LOSSES:
        x = _loss_inputs(case, seed)
        for k in ("o1", "o2", "s", "sh"):
            if k in x:
                x[k].requires_grad_(True)
        return dict(case=case, x=x)
    if kind in _OPTIMS:
        from tspipe_b200.optim import SGD, AdamW, LARS
        from tspipe_b200.runtime.state import FlatParams
        x = _optim_inputs(case, seed)
        ps = [nn.Parameter(p) for p in x["p"]]
        flat = FlatParams(ps, torch.device(DEV), with_grad=True)
        for p, g in zip(ps, x["g"]):
            p.grad.copy_(g)
        opt = {"lars": LARS, "adamw": AdamW, "sgd": SGD}[kind](ps, **_HP[kind])
        opt.bind_flat(flat, use_kernel=True)

        def like(ts):
            buf = torch.zeros_like(flat.data)
            for i, t in enumerate(ts):
                flat._view(buf, i, ps[i].data).copy_(t)
            return buf
        names = {"lars": ["mu"], "adamw": ["exp_avg", "exp_avg_sq"], "sgd": ["momentum_buffer"]}[kind]
        opt.load_state_dict(dict(opt.state_dict(), tspipe_flat=dict(
            flat={n: like(x[k]) for n, k in zip(names, "mv")}, steps=1)))
        if case["ema"]:
            opt.teacher_flat, opt.ema_momentum = like(x["t"]), _EMA
        return dict(case=case, opt=opt, flat=flat, bufs=[opt._buf(n) for n in names])
    from tspipe_b200.batchnorm import BatchNormGroup, DeferredBatchNorm
    from tspipe_b200.runtime.fuse import fuse_partition
    from tspipe_b200.runtime.state import FlatParams
    m, x, gy = _module_inputs(case, seed)
    m = m.to(memory_format=torch.channels_last)
    m = fuse_partition(DeferredBatchNorm.convert_deferred_batch_norm(m, chunks=1))
    group = BatchNormGroup(m, chunks=1)
    flat = FlatParams(list(m.parameters()), torch.device(DEV), with_grad=_trains(case))
    if not _trains(case):
        for p in m.parameters():
            p.requires_grad_(False)
    elif kind != "stem":                # the images themselves need no gradient
        x.requires_grad_(True)
    state = dict(case=case, m=m, x=x, gy=gy, flat=flat, group=group)
    if case["graph"]:
        _record(state)
    return state


def _forward(state):
    from tspipe_b200.ops import bn
    case = state["case"]
    with contextlib.nullcontext() if _trains(case) else torch.no_grad(), \
            torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False), bn.segments(case.get("views", 1)):
        y = state["m"](state["x"])
    return y if isinstance(y, torch.Tensor) else y["hidden"]


def _record(state):
    """The forward and the backward as a pair of CUDA graphs after two eager passes, as the executor records a stage."""
    from tspipe_b200.runtime.stage_graph import capture
    case, x, group = state["case"], state["x"], state["group"]
    train, params = _trains(case), list(state["m"].parameters())
    for _ in range(2):
        y = _forward(state)
        if train:
            y.backward(state["gy"])
    del y
    x = x if isinstance(x, torch.Tensor) else x["hidden"]
    x.grad = None
    if group.layers:                    # forget the statistics of the eager passes
        group.step()
        group.running_mean.zero_()
        group.running_var.fill_(1.0)
    stream, pool = torch.cuda.Stream(), torch.cuda.graph_pool_handle()
    state["fwd"], state["bwd"] = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph() if train else None
    y = capture(state["fwd"], stream, pool, lambda: _forward(state))

    def backward():
        leaves = ([x] if x.requires_grad else []) + params
        gs = torch.autograd.grad(y, leaves, state["gy"], allow_unused=True)
        for p, g in zip(params, gs[-len(params):]):
            if g is not None:
                p.grad.add_(g)
        return gs[0] if x.requires_grad else None
    if train:
        state["dx"] = capture(state["bwd"], stream, pool, backward)
    state["y"] = y.detach()


# -------------------------------------------------------------------------------------------------------------------
# one pass
# -------------------------------------------------------------------------------------------------------------------
def _layer_grads(state):
    """The gradients of each layer of a head as one range of the flat buffer, weight and bias together (the bias in
    front of a BatchNorm has a gradient of zero, of which only the rounding would be left to compare)."""
    flat, n = state["flat"], len(state["flat"].params)
    ends = [flat.offsets[i] for i in range(2, n, 2)] + [flat.offsets[-1] + flat.numels[-1]]
    return [flat.grad[flat.offsets[2 * i]: e] for i, e in enumerate(ends)]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in _LOSSES:
        from tspipe_b200 import losses
        x = state["x"]
        if kind in ("byol_loss", "moco_loss"):
            loss = getattr(losses, kind)(x["o1"], x["o2"], x["t1"], x["t2"])
            gs = torch.autograd.grad(loss, [x["o1"], x["o2"]])
        elif kind == "kd_loss":
            loss = losses.soft_target_kd(x["s"], x["t"], x["labels"])
            gs = torch.autograd.grad(loss, [x["s"]])
        else:
            loss = losses.distil_loss((x["s"], x["sh"]), (x["t"], x["th"]),
                                      (x["labels"], x["attn"], x["n_lab"], x["n_sel"]))
            gs = torch.autograd.grad(loss, [x["s"], x["sh"]])
        return dict(loss=loss.detach(), grads=list(gs))
    if kind in _OPTIMS:
        state["opt"].step()
        flat, opt = state["flat"], state["opt"]
        return dict(p=flat.data, state=state["bufs"], teacher=opt.teacher_flat)
    from tspipe_b200.ops import conv, gemm
    m, x, flat = state["m"], state["x"], state["flat"]
    train = _trains(case)
    if case["graph"]:
        state["fwd"].replay()
        out = dict(y=state["y"])
        if train:
            flat.zero_grad()
            state["bwd"].replay()
            dx = state["dx"]
    else:
        y = _forward(state)
        out = dict(y=y.detach())
        if train:
            flat.zero_grad()
            x.grad = None
            y.backward(state["gy"])
            dx = x.grad
        conv.clear_weight_cache()
        gemm.clear_weight_cache()
    if train:
        out["grads"] = _layer_grads(state) if kind == "head" else [p.grad for p in m.parameters()]
        if dx is not None:
            out["dx"] = dx
    if kind == "trunk":                 # a whole mini-batch has passed: its statistics are committed
        state["group"].step()
        out["running"] = [state["group"].running_mean, state["group"].running_var]
    return out


# -------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# -------------------------------------------------------------------------------------------------------------------
def _conv_flops(images, so, cin, planes, stride):
    per = cin * planes * stride * stride + 9 * planes * planes + 4 * planes * planes
    if stride != 1 or cin != 4 * planes:
        per += cin * 4 * planes
    return 2.0 * images * so * so * per, cin * planes + 13 * planes * planes + (
        cin * 4 * planes if (stride != 1 or cin != 4 * planes) else 0)


_TRUNK = {"resnet18": (1.82e9, 11.2e6), "resnet50": (4.09e9, 23.5e6)}      # multiply-adds of an image at 224, weights


def work(case):
    k = case["kind"]
    e = 4 if case.get("dtype") == "fp32" else 2
    if k in ("byol_loss", "moco_loss"):
        n, d = case["rows"], case["dim"]
        fl = 12.0 * n * d if k == "byol_loss" else 2 * 4.0 * n * n * d
        return dict(bytes=6.0 * n * d * e, flops=fl)
    if k == "kd_loss":
        return dict(bytes=3.0 * case["rows"] * case["classes"] * e + 8 * case["rows"], flops=20.0 * case["rows"] * case["classes"])
    if k == "distil_loss":
        n = case["batch"] * case["length"]
        return dict(bytes=3.0 * 2 * n * (case["vocab"] + case["hidden"]) + 16 * n, flops=20.0 * n * case["vocab"])
    if k in _OPTIMS:
        n = float(case["params"])
        # read p, g and the state once, write p and the state; the teacher is read and written
        rw = {"lars": 5, "sgd": 5, "adamw": 7}[k] + (2 if case["ema"] else 0)
        return dict(bytes=4 * rw * n, flops=15 * n)
    if k == "head":
        n, a, b, c = case["rows"], case["din"], case["hidden"], case["dout"]
        w = a * b + b * c
        return dict(bytes=2.0 * n * (2 * a + 2 * c) + 8.0 * w, flops=6.0 * n * w)
    if k == "stem":
        n, s = case["images"], case["side"]
        return dict(bytes=2.0 * n * (3 * s * s + 2 * 64 * (s // 4) ** 2), flops=2 * 2.0 * n * (s // 2) ** 2 * 64 * 147)
    if k == "bottleneck":
        n, s, so = case["images"], case["side"], case["side"] // case["stride"]
        fl, w = _conv_flops(n, so, case["cin"], case["planes"], case["stride"])
        return dict(bytes=2.0 * n * (2 * case["cin"] * s * s + 8 * case["planes"] * so * so) + 8.0 * w, flops=3 * fl)
    if k == "vit_block":
        t, d = case["batch"] * case["tokens"], case["dim"]
        f = 2.0 * t * 12 * d * d + 4.0 * t * case["tokens"] * d
        return dict(bytes=2.0 * t * d * (4 if case["train"] else 2) + 12.0 * d * d * (8 if case["train"] else 4),
                    flops=f * (3 if case["train"] else 1))
    if k == "bert_layer":
        t, d, f = case["batch"] * case["length"], case["hidden"], case["ffn"]
        w = 4 * d * d + 2 * d * f
        return dict(bytes=2.0 * t * d * 2 + 4.0 * w, flops=2.0 * t * w + 4.0 * t * case["length"] * d)
    fl, w = _TRUNK[case["arch"]]
    n, s = case["images"], case["side"]
    return dict(bytes=2.0 * n * 3 * s * s + 4.0 * w, flops=2.0 * n * fl * (s / 224) ** 2)


def tolerance(case):
    kind = case["kind"]
    if kind in _OPTIMS or case.get("dtype") == "fp32":
        return {"rel": 2e-6 if kind != "moco_loss" else 1e-2}
    if kind in _LOSSES:
        return {"rel": 1e-2}
    if kind == "bert_layer":
        return {"rel": 1.6e-2}
    # several bf16 layers with rounding in between.  Behind a ReLU the gradient of a unit whose sign a rounding
    # changes is off by its whole value, hence "max" (the output gradients have even magnitude)
    return {"rel": 3e-2} if kind == "vit_block" else {"rel": 3e-2, "max": 0.99}


# -------------------------------------------------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# -------------------------------------------------------------------------------------------------------------------
def _bn64(x, w, b, eps, views, relu=False, res=None):
    dims = [0] + list(range(2, x.dim()))
    shape = [1, -1] + [1] * (x.dim() - 2)
    parts = []
    for v in x.chunk(views):
        mu = v.mean(dims, keepdim=True)
        var = ((v - mu) ** 2).mean(dims, keepdim=True)
        parts.append((v - mu) / torch.sqrt(var + eps) * w.view(shape) + b.view(shape))
    y = torch.cat(parts) if views > 1 else parts[0]
    y = y if res is None else y + res
    return torch.relu(y) if relu else y


def _conv64(x, w, stride, pad):
    """A 1x1 convolution as a matrix product, the others by the library in 64 bits."""
    if w.shape[2] == 1:
        x = x[:, :, ::stride, ::stride]
        n, c, h, wd = x.shape
        y = x.permute(0, 2, 3, 1).reshape(-1, c) @ w.view(w.shape[0], c).t()
        return y.view(n, h, wd, -1).permute(0, 3, 1, 2)
    return F.conv2d(x, w, stride=stride, padding=pad)


def _bottleneck64(x, P, stride, views):
    bn = lambda v, i, **kw: _bn64(v, P[f"{i}.weight"], P[f"{i}.bias"], 1e-5, views, **kw)      # noqa: E731
    ident = x
    if "downsample.0.weight" in P:
        ident = bn(_conv64(x, P["downsample.0.weight"], stride, 0), "downsample.1")
    h = bn(_conv64(x, P["conv1.weight"], 1, 0), "bn1", relu=True)
    h = bn(_conv64(h, P["conv2.weight"], stride, 1), "bn2", relu=True)
    return bn(_conv64(h, P["conv3.weight"], 1, 0), "bn3", relu=True, res=ident)


def _heads(t, heads):
    b, n, c = t.shape
    return t.view(b, n, heads, c // heads).transpose(1, 2)


def _attn64(x, w, b, heads, mask=None):
    q, k, v = (_heads(t, heads) for t in F.linear(x, w, b).chunk(3, dim=-1))
    s = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    if mask is not None:
        s = s.masked_fill(~mask[:, None, None, :].bool(), float("-inf"))
    o = s.softmax(-1) @ v
    return o.transpose(1, 2).reshape(x.shape)


def _forward64(case, P, x):
    kind = case["kind"]
    views = case.get("views", 1)
    if kind == "head":
        h = F.linear(x, P["proj_fc1.weight"], P["proj_fc1.bias"])
        h = _bn64(h, P["proj_bn.weight"], P["proj_bn.bias"], 1e-5, views, relu=True)
        return F.linear(h, P["proj_fc2.weight"], P["proj_fc2.bias"])
    if kind == "stem":
        h = _bn64(_conv64(x, P["0.weight"], 2, 3), P["1.weight"], P["1.bias"], 1e-5, views, relu=True)
        return F.max_pool2d(h, 3, 2, 1)
    if kind == "bottleneck":
        return _bottleneck64(x, {k[2:]: v for k, v in P.items()}, case["stride"], views)
    P = {k[2:]: v for k, v in P.items()}
    if kind == "vit_block":
        ln = lambda v, i: F.layer_norm(v, v.shape[-1:], P[i + ".weight"], P[i + ".bias"], 1e-6)     # noqa: E731
        a = _attn64(ln(x, "norm1"), P["attn.qkv.weight"], P["attn.qkv.bias"], case["heads"])
        x = x + F.linear(a, P["attn.proj.weight"], P["attn.proj.bias"])
        h = F.gelu(F.linear(ln(x, "norm2"), P["mlp.fc1.weight"], P["mlp.fc1.bias"]))
        return x + F.linear(h, P["mlp.fc2.weight"], P["mlp.fc2.bias"])
    h, mask = x
    ln = lambda v, i: F.layer_norm(v, v.shape[-1:], P[i + ".weight"], P[i + ".bias"], 1e-12)        # noqa: E731
    a = _attn64(h, P["qkv.weight"], P["qkv.bias"], case["heads"], mask)
    h = ln(h + F.linear(a, P["out.weight"], P["out.bias"]), "norm1")
    f = F.linear(F.gelu(F.linear(h, P["fc1.weight"], P["fc1.bias"])), P["fc2.weight"], P["fc2.bias"])
    return ln(h + f, "norm2")


def _trunk64(case, m, x):
    """Forward of a plain trunk in 64 bits; returns the output and every BatchNorm's (mean, biased variance)."""
    stats = []

    def bn(v, mod, relu=False, res=None):
        dims = [0] + list(range(2, v.dim()))
        mu = v.mean(dims)
        stats.append((mu, v.var(dims, unbiased=False)))
        return _bn64(v, mod.weight.double(), mod.bias.double(), mod.eps, 1, relu, res)

    def conv(v, mod):
        return _conv64(v, mod.weight.double(), mod.stride[0], mod.padding[0])
    for name, c in m.named_children():
        if name == "conv1":
            x = conv(x, c)
        elif name == "bn1":
            x = bn(x, c, relu=True)
        elif name == "maxpool":
            x = F.max_pool2d(x, 3, 2, 1)
        elif name.startswith("layer"):
            # statistics are listed in the order of the module tree, where the shortcut comes last
            ident, tail = x, None
            if c.downsample is not None:
                ident = bn(conv(x, c.downsample[0]), c.downsample[1])
                tail = stats.pop()
            if hasattr(c, "conv3"):
                h = bn(conv(x, c.conv1), c.bn1, relu=True)
                h = bn(conv(h, c.conv2), c.bn2, relu=True)
                x = bn(conv(h, c.conv3), c.bn3, relu=True, res=ident)
            else:
                h = bn(conv(x, c.conv1), c.bn1, relu=True)
                x = bn(conv(h, c.conv2), c.bn2, relu=True, res=ident)
            if tail is not None:
                stats.append(tail)
        elif name == "avgpool":
            x = x.mean((2, 3))
    return x, stats


def _loss64(case, x):
    if case["kind"] == "byol_loss":
        n = lambda t: F.normalize(t, dim=1)                                                    # noqa: E731
        r = lambda a, b: 2 - 2 * (n(a) * n(b)).sum(-1)                                          # noqa: E731
        return (r(x["o1"], x["t2"]) + r(x["o2"], x["t1"])).mean()
    if case["kind"] == "moco_loss":
        def nce(q, k):
            lo = F.normalize(q, dim=1) @ F.normalize(k, dim=1).t() / 0.2
            return F.cross_entropy(lo, torch.arange(q.shape[0], device=q.device)) * 0.4
        return nce(x["o1"], x["t2"]) + nce(x["o2"], x["t1"])
    kl = lambda s, t, T: F.kl_div(F.log_softmax(s / T, -1), F.softmax(t / T, -1), reduction="batchmean") * T * T  # noqa: E731
    if case["kind"] == "kd_loss":
        return F.cross_entropy(x["s"], x["labels"]) + kl(x["s"], x["t"], 4.0)
    sel = x["attn"].bool()
    loss = 5.0 * kl(x["s"][sel], x["t"][sel], 2.0)
    loss = loss + 2.0 * F.cross_entropy(x["s"].flatten(0, 1), x["labels"].flatten(), ignore_index=-100)
    return loss + (1 - F.cosine_similarity(x["sh"][sel], x["th"][sel], dim=-1)).mean()


def _optim64(case, seed):
    from_ = _optim_inputs(case, seed)
    hp = _HP[case["kind"]]
    out = {k: [] for k in ("p", "a", "b", "t")}
    for i, p in enumerate(from_["p"]):
        matrix = p.dim() > 1
        p, g, m = p.double(), from_["g"][i].double(), from_["m"][i].double()
        if case["kind"] == "lars":
            if matrix:
                g = g + hp["weight_decay"] * p
                g = g * (0.001 * p.norm() / g.norm())
            m = 0.9 * m + g
            p = p - hp["lr"] * m
        elif case["kind"] == "sgd":
            m = 0.9 * m + g + hp["weight_decay"] * p
            p = p - hp["lr"] * m
        else:
            p = p * (1 - hp["lr"] * hp["weight_decay"])
            m = 0.9 * m + 0.1 * g
            v = 0.999 * from_["v"][i].double() + 0.001 * g * g
            p = p - hp["lr"] / (1 - 0.9 ** 2) * m / (torch.sqrt(v) / math.sqrt(1 - 0.999 ** 2) + 1e-8)
            out["b"].append(v)
        out["p"].append(p)
        out["a"].append(m)
        if case["ema"]:
            out["t"].append(_EMA * from_["t"][i].double() + (1 - _EMA) * p)
    pad = lambda ts: torch.cat([F.pad(t.reshape(-1), (0, -t.numel() % 64)) for t in ts]) if ts else None     # noqa: E731
    return dict(p=pad(out["p"]), state=[pad(out["a"])] + ([pad(out["b"])] if out["b"] else []), teacher=pad(out["t"]))


def exact(case, seed):
    kind = case["kind"]
    if kind in _OPTIMS:
        return _optim64(case, seed)
    if kind in _LOSSES:
        x = {k: v.double() if isinstance(v, torch.Tensor) and v.is_floating_point() else v
             for k, v in _loss_inputs(case, seed).items()}
        leaves = [x[k].requires_grad_(True) for k in ("o1", "o2", "s", "sh") if k in x]
        loss = _loss64(case, x)
        return dict(loss=loss.detach(), grads=list(torch.autograd.grad(loss, leaves)))
    m, x, gy = _module_inputs(case, seed)
    if kind == "trunk":
        with torch.no_grad():
            y, stats = _trunk64(case, m, x.double())
        mean, var = (torch.cat([s[i] for s in stats]) for i in (0, 1))
        return dict(y=y, running=[0.1 * mean, 0.9 + 0.1 * var])
    if kind == "bert_layer":
        with torch.no_grad():
            P = {k: v.double() for k, v in m.named_parameters()}
            return dict(y=_forward64(case, P, (x["hidden"].double(), x["mask"])))
    P = {k: v.detach().double().requires_grad_(gy is not None) for k, v in m.named_parameters()}
    x = x.double()
    if gy is None:
        with torch.no_grad():
            return dict(y=_forward64(case, P, x))
    if kind != "stem":
        x.requires_grad_(True)
    y = _forward64(case, P, x)
    gs = torch.autograd.grad(y, list(P.values()) + ([x] if kind != "stem" else []), gy.double())
    out = dict(y=y.detach(), grads=list(gs[:len(P)]))
    if kind == "stem":
        out["grads"][0] = None          # max-pool windows tie in bf16 and not in 64 bits: the gradient takes other routes
    if kind == "bottleneck":            # BatchNorm gradients are sums that cancel but for what rounding leaves of them
        out["grads"] = [g if P[k].dim() > 1 else None for k, g in zip(P, out["grads"])]
    if kind == "head":
        out["grads"] = [torch.cat([w.flatten(), b]) for w, b in zip(gs[:len(P):2], gs[1:len(P):2])]
    if kind != "stem":
        out["dx"] = gs[-1]
    return out
