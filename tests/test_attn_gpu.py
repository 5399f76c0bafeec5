"""Fused attention forward on tcgen05 (and the contrastive loss built on it) against plain PyTorch in fp32."""
import math

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _ref(q, k, v, scale):
    s = (q.float() @ k.float().transpose(-1, -2)) * scale
    return torch.softmax(s, -1) @ v.float(), torch.logsumexp(s, -1)


@pytest.mark.parametrize("b,h,nq,nk", [(2, 3, 197, 197), (1, 2, 64, 64), (1, 1, 128, 128), (2, 2, 300, 520), (3, 12, 50, 197)])
def test_flash_forward_head_dim_64(b, h, nq, nk):
    """Interleaved qkv layout as the ViT blocks produce it ([B, N, 3, H, 64] viewed as [B, H, N, 64])."""
    from tspipe_b200.ops import attention, gemm
    torch.manual_seed(0)
    dev = torch.device("cuda", 0)
    n = max(nq, nk)
    qkv = (torch.randn(b, n, 3, h, 64, device=dev) * 1.5).bfloat16()
    q, k, v = qkv.permute(2, 0, 3, 1, 4)
    q, k, v = q[:, :, :nq], k[:, :, :nk], v[:, :, :nk]
    assert attention.flash_eligible(q, k, v)
    o, lse = attention.flash_fwd(q, k, v, want_lse=True)
    gemm.check_status()
    ro, rl = _ref(q, k, v, 1 / math.sqrt(64))
    assert o.shape == (b, h, nq, 64)
    assert o.transpose(1, 2).reshape(b, nq, h * 64).is_contiguous()
    torch.testing.assert_close(o.float(), ro, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(lse, rl, rtol=1e-3, atol=1e-2)


@pytest.mark.parametrize("b,h,nq,nk", [(2, 3, 197, 197), (1, 1, 1, 1), (1, 2, 128, 127), (2, 2, 257, 129), (3, 12, 50, 500),
                                       (40, 12, 300, 512), (1, 1, 64, 4096)])
@pytest.mark.parametrize("masked", ["none", "padding", "holes", "one for all"])
def test_heads_forward(b, h, nq, nk, masked):
    """Edges of the tiles of queries and keys, one item to several per SM, tiles of keys that are switched off at the end and in
    between; maxima that grow from tile to tile.  Rounding: P and the output in bf16, sums in fp32."""
    from tspipe_b200.ops import attention, gemm
    torch.manual_seed(0)
    dev = torch.device("cuda", 0)
    n = max(nq, nk)
    qkv = (torch.randn(b, n, 3, h, 64, device=dev) * 1.5).bfloat16()
    qkv[:, :, 1] *= torch.linspace(0.2, 2, n, device=dev).bfloat16()[None, :, None, None]
    q, k, v = qkv.permute(2, 0, 3, 1, 4)
    q, k, v = q[:, :, :nq], k[:, :, :nk], v[:, :, :nk]
    at = torch.arange(nk, device=dev)
    mask = {"none": None, "padding": at[None] < torch.randint(1, nk + 1, (b, 1), device=dev),
            "holes": ((at[None] // 128 % 2 == 1) & (torch.rand(b, nk, device=dev) < 0.5)) | (at[None] == nk - 1),
            "one for all": (at % 3 != 1)[None] | (at == 0)[None]}[masked]
    mask = None if mask is None else mask[:, None, None, :]
    o = attention.heads_fwd(q, k, v, mask)
    gemm.check_status()
    assert o.shape == (b, h, nq, 64) and o.transpose(1, 2).is_contiguous()
    s = (q.double() @ k.double().transpose(-1, -2)) / 8
    want = torch.softmax(s if mask is None else s.masked_fill(~mask, -math.inf), -1) @ v.double()
    assert float((o.double() - want).norm() / want.norm()) < 2 * 2 ** -8
    if mask is not None and nk > 1:
        attention.set_tcgen05(None)
        with torch.no_grad():
            assert torch.equal(attention.attention(q, k, v, mask), o)


def test_heads_forward_without_any_key():
    from tspipe_b200.ops import attention
    dev = torch.device("cuda", 0)
    q, k, v = (torch.randn(3, 2, 300, 64, device=dev).bfloat16() for _ in range(3))
    mask = torch.rand(3, 1, 1, 300, device=dev) < 0.5
    mask[1] = False
    assert torch.equal(attention.heads_fwd(q, k, v, mask)[1], attention.heads_fwd(q, k, v)[1])


@pytest.mark.parametrize("nq,nk", [(300, 300), (64, 64), (40, 2), (1, 384), (128, 127), (40, 1)])
@pytest.mark.parametrize("packed", [False, True])
def test_attention_without_any_key_is_what_the_library_gives(nq, nk, packed):
    """Forwards with a gradient go to the library, those without one to the kernel: a batch entry whose keys are all off gives
    the same in both."""
    from tspipe_b200.ops import attention
    torch.manual_seed(6)
    dev = torch.device("cuda", 0)
    n = max(nq, nk)
    q, k, v = (torch.randn(3, n, 3, 2, 64, device=dev).bfloat16().permute(2, 0, 3, 1, 4) if packed else
               torch.randn(3, 3, 2, n, 64, device=dev).bfloat16())
    q, k, v = q[:, :, :nq], k[:, :, :nk], v[:, :, :nk]
    mask = torch.rand(3, 1, 1, nk, device=dev) < 0.5
    mask[..., -1] = True
    mask[1] = False
    want = F.scaled_dot_product_attention(q, k, v, attn_mask=mask)
    with torch.no_grad():
        got = attention.attention(q, k, v, mask)
    grad = attention.attention(q.detach().requires_grad_(), k, v, mask).detach()
    assert float((grad.double() - want.double()).norm()) <= 2 * 2 ** -8 * float(want.double().norm())
    for a, b in zip(got.double(), want.double()):
        assert float((a - b).norm()) <= 2 * 2 ** -8 * float(b.norm())       # (zeros: equal)


@pytest.mark.parametrize("nk", [4096, 4097, 9000])
def test_attention_on_request_at_any_number_of_keys(nk, monkeypatch):
    from tspipe_b200.ops import attention, gemm
    torch.manual_seed(8)
    dev = torch.device("cuda", 0)
    q, k, v = (torch.randn(2, 3, n, 64, device=dev).bfloat16() for n in (130, nk, nk))
    kernel, calls = {}, []
    for name in ("heads_fwd", "flash_fwd"):
        kernel[name] = getattr(attention, name)
        monkeypatch.setattr(attention, name, lambda *a, name=name: [calls.append(name), kernel[name](*a)][1])
    attention.set_tcgen05(True)
    try:
        with torch.no_grad():
            o = attention.attention(q, k, v)
    finally:
        attention.set_tcgen05(None)
    gemm.check_status()
    assert calls == (["heads_fwd"] if nk <= 4096 else ["heads_fwd", "flash_fwd"])
    want = torch.softmax(q.double() @ k.double().transpose(-1, -2) / 8, -1) @ v.double()
    assert float((o.double() - want).norm() / want.norm()) < 2 * 2 ** -8


@pytest.mark.parametrize("b,n,kernel", [(2, 32, True), (64, 8, False), (64, 32, False), (64, 33, True), (42, 32, True)])
def test_attention_of_many_short_sequences_stays_with_the_library(b, n, kernel, monkeypatch):
    from tspipe_b200.ops import attention
    torch.manual_seed(9)
    dev = torch.device("cuda", 0)
    q, k, v = torch.randn(b, n, 3, 12, 64, device=dev).bfloat16().permute(2, 0, 3, 1, 4)
    mask = (torch.arange(n, device=dev)[None] < torch.randint(1, n + 1, (b, 1), device=dev))[:, None, None]
    heads_fwd, calls = attention.heads_fwd, []
    monkeypatch.setattr(attention, "heads_fwd", lambda *a: [calls.append(1), heads_fwd(*a)][1])
    with torch.no_grad():
        o = attention.attention(q, k, v, mask)
    assert bool(calls) == kernel
    want = torch.softmax((q.double() @ k.double().transpose(-1, -2) / 8).masked_fill(~mask, -math.inf), -1) @ v.double()
    assert float((o.double() - want).norm() / want.norm()) < 2 * 2 ** -8


def test_attention_is_seen_by_traces_modes_and_autocast():
    from torch.utils.flop_counter import FlopCounterMode
    from tspipe_b200.ops import attention
    dev = torch.device("cuda", 0)
    q, k, v = (torch.randn(2, 3, 40, 64, device=dev).bfloat16() for _ in range(3))
    mask = torch.arange(40, device=dev)[None, None, None] < torch.tensor([40, 17], device=dev).view(2, 1, 1, 1)
    call = lambda q, k, v, mask: attention.attention(q, k, v, mask)      # noqa: E731
    want = F.scaled_dot_product_attention(v, q, k, attn_mask=mask)
    with torch.no_grad():
        traced = torch.jit.trace(call, (q, k, v, mask), check_trace=False)
        assert torch.equal(traced(v, q, k, mask), want)
        compiled = torch.compile(call, backend="eager", fullgraph=True)
        assert torch.equal(compiled(v, q, k, mask), want)
        with FlopCounterMode(display=False) as flops:
            call(q, k, v, mask)
        assert flops.get_total_flops() > 0
        with torch.autocast("cuda", dtype=torch.float16):
            assert call(q, k, v, mask).dtype == torch.float16
        with torch.autocast("cuda", dtype=torch.bfloat16):
            assert torch.equal(call(q, k, v, mask), attention.heads_fwd(q, k, v, mask))


def test_heads_forward_leaves_the_rest_to_the_library():
    from tspipe_b200.ops import attention
    dev = torch.device("cuda", 0)
    q = torch.randn(2, 3, 40, 64, device=dev).bfloat16()
    full = torch.ones(2, 3, 40, 40, dtype=torch.bool, device=dev)
    assert attention.heads_fwd(q, q, q, full) is None                             # per query
    assert attention.heads_fwd(q, q, q, torch.zeros(2, 1, 1, 40, device=dev)) is None      # additive
    assert attention.heads_fwd(q.float(), q.float(), q.float()) is None
    assert attention.heads_fwd(q[..., :32], q[..., :32], q[..., :32]) is None
    assert attention.heads_fwd(q, q[:1].expand(2, -1, -1, -1), q) is None         # a stride of zero
    assert attention.heads_fwd(q, q[:, :, :30], q) is None
    assert attention.heads_fwd(q[:, :, 1:], q, q) is not None
    assert torch.vmap(lambda t: attention.attention(t, t, t))(q[None]).shape == (1, 2, 3, 40, 64)


def test_attention_dispatch_and_vit_block_without_grad():
    """A ViT block gives the same result through the three attention paths: tcgen05 kernel (no gradient needed, without a
    mask on request), the library's fused attention on unbound q / k / v, and the packed-qkv library entry point."""
    from tspipe_b200.models.vit import CONFIGS, Block
    from tspipe_b200.ops import attention, gemm
    torch.manual_seed(1)
    dev = torch.device("cuda", 0)
    blk = Block(CONFIGS["vit_base"]).to(dev)
    x = torch.randn(4, 197, 768, device=dev)
    try:
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            attention.set_qkv_mode("packed")
            attention.set_packed(False)
            attention.set_tcgen05(True)
            y = blk(x)                                   # tcgen05 attention
            attention.set_tcgen05(False)
            y_ref = blk(x)                               # library attention on unbound q, k, v
            attention.set_packed(None)
            y_packed = blk(x)                            # packed entry point when the library supports this GPU
            attention.set_qkv_mode("split")
            y_split = blk(x)                             # three projection GEMMs + library attention
    finally:
        attention.set_tcgen05(None)
        attention.set_packed(None)
        attention.set_qkv_mode("split")
    gemm.check_status()
    torch.testing.assert_close(y.float(), y_ref.float(), rtol=3e-2, atol=3e-2)
    torch.testing.assert_close(y_packed.float(), y_ref.float(), rtol=3e-2, atol=3e-2)
    torch.testing.assert_close(y_split.float(), y_ref.float(), rtol=3e-2, atol=3e-2)
    grads = {}
    for mode in ("split", "packed"):                      # with gradients, both ways of forming q, k, v
        attention.set_qkv_mode(mode)
        try:
            xg = x.clone().requires_grad_()
            blk.zero_grad()
            with torch.autocast("cuda", dtype=torch.bfloat16):
                blk(xg).float().sum().backward()
            grads[mode] = (xg.grad.clone(), blk.attn.qkv.weight.grad.clone())
        finally:
            attention.set_qkv_mode("split")
    for a, b in zip(grads["split"], grads["packed"]):
        torch.testing.assert_close(a, b, rtol=5e-2, atol=5e-2 * b.abs().max().item())


@pytest.mark.parametrize("recorded", [False, True])
@pytest.mark.parametrize("b,l", [(3, 50), (2, 300), (9, 128)])
def test_encoder_layer_of_a_frozen_teacher(b, l, recorded):
    """A BERT layer with heads of 64 and a padding mask, without a gradient, eagerly and replayed on new inputs: attention runs on
    the kernel and differs from the library's as one rounding of the attention does from another."""
    from tspipe_b200.models.bert import BertConfig, EncoderLayer
    from tspipe_b200.ops import attention, fused, gemm
    from tspipe_b200.runtime.stage_graph import capture
    torch.manual_seed(7)
    dev = torch.device("cuda", 0)
    m = EncoderLayer(BertConfig(hidden=256, heads=4, ffn=1024)).to(dev).eval()

    def inputs():
        lens = torch.randint(max(1, l // 3), l + 1, (b, 1), device=dev)
        return torch.randn(b, l, 256, device=dev).bfloat16(), (torch.arange(l, device=dev)[None] < lens).long()

    def run(x, mask):
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False):
            return m({"hidden": x, "mask": mask})["hidden"]

    x, mask = inputs()
    counts = {}
    try:
        for flag in (None, False):
            attention.set_tcgen05(flag)
            run(x, mask)
            before = fused.LAUNCHES
            run(x, mask)
            counts[flag] = fused.LAUNCHES - before
        want_in = inputs()
        want = run(*want_in)                                # the library's attention
    finally:
        attention.set_tcgen05(None)
    assert counts[None] == counts[False] + 1
    if recorded:
        graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        got = capture(graph, stream, torch.cuda.graph_pool_handle(), lambda: run(x, mask))
        x.copy_(want_in[0])
        mask.copy_(want_in[1])
        graph.replay()
    else:
        got = run(*want_in)
    gemm.check_status()
    assert float((got.double() - want.double()).norm() / want.double().norm()) < 2 * 2 ** -8


def test_patch_embedding_as_gemm_matches_convolution():
    from tspipe_b200.models.vit import CONFIGS, PatchEmbed
    torch.manual_seed(5)
    dev = torch.device("cuda", 0)
    pe = PatchEmbed(CONFIGS["vit_base"]).to(dev)
    for fmt in (torch.contiguous_format, torch.channels_last):
        x = torch.randn(3, 3, 224, 224, device=dev).contiguous(memory_format=fmt).requires_grad_()
        y = pe(x)
        ref = pe.proj(x).flatten(2).transpose(1, 2)
        torch.testing.assert_close(y, ref, rtol=2e-3, atol=2e-3)     # TF32 may be on for either path
        g = torch.randn_like(y)
        gw = torch.autograd.grad(y, pe.proj.weight, g, retain_graph=True)[0]
        gw_ref = torch.autograd.grad(ref, pe.proj.weight, g)[0]
        torch.testing.assert_close(gw, gw_ref, rtol=2e-3, atol=2e-3 * gw_ref.abs().max().item())


@pytest.mark.parametrize("n", [128, 1024, 4096])
def test_fused_contrastive_loss_matches_cross_entropy(n):
    """Loss value and gradient from one fused pass (V = K, scores bounded by 1/T) vs normalize + matmul + CE."""
    from tspipe_b200.ops import fused, gemm
    torch.manual_seed(2)
    dev = torch.device("cuda", 0)
    temp = 0.2
    q = torch.randn(n, 256, device=dev, requires_grad=True)
    k = torch.randn(n, 256, device=dev)
    k[: n // 2] += 0.5 * q.detach()[: n // 2]        # some positives that actually align
    loss = fused.info_nce_loss(q, k, temp)
    loss.backward()
    gemm.check_status()
    qr = q.detach().clone().requires_grad_()
    logits = F.normalize(qr, dim=1) @ F.normalize(k, dim=1).t() / temp
    ref = F.cross_entropy(logits, torch.arange(n, device=dev)) * (2 * temp)
    ref.backward()
    torch.testing.assert_close(loss, ref, rtol=5e-3, atol=5e-3)
    torch.testing.assert_close(q.grad, qr.grad, rtol=5e-2, atol=5e-2 * qr.grad.abs().max().item())
    gemm.set_fused_nce(False)
    try:
        q2 = q.detach().clone().requires_grad_()
        unfused = fused.info_nce_loss(q2, k, temp)
    finally:
        gemm.set_fused_nce(True)
    torch.testing.assert_close(loss, unfused, rtol=5e-3, atol=5e-3)
