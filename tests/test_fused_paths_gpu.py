"""Kernels that fold several passes into one, at the sizes where their dispatch or their tiling changes, against plain
PyTorch in fp32 or fp64 (tolerances: the rounding of the result's type, times the length of a sum where there is one)."""
import math

import pytest
import torch
import torch.nn.functional as F
from torch import nn

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
EPS = {torch.float32: 2 ** -23, torch.bfloat16: 2 ** -8}


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


def _cl(*shape, dtype=torch.bfloat16):
    n, c, h, w = shape
    return torch.randn(n, h, w, c, device=DEV).to(dtype).permute(0, 3, 1, 2)


# ---- losses -------------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,c", [(3, 7), (5, 8), (4, 776), (3, 1001), (2, 4104), (2, 16400)])
def test_kd_ce_rows_vectorised_and_not(n, c, dtype):
    """Row lengths on both sides of every block size, 8 elements per access or one; a masked row, rows without a label,
    classes switched off by the type's lowest value, and by -inf under cross-entropy alone."""
    from tspipe_b200.ops import fused
    torch.manual_seed(0)
    s = (torch.randn(n, c, device=DEV) * 3).to(dtype)
    t = (torch.randn(n, c, device=DEV) * 3).to(dtype)
    s[0, : c // 2] = torch.finfo(dtype).min
    t[0, : c // 2] = torch.finfo(dtype).min
    y = torch.randint(c // 2 + 1, c, (n,), device=DEV)
    y[1] = -100
    on = torch.ones(n, dtype=torch.bool, device=DEV)
    on[-1] = n < 3
    s = s.requires_grad_()
    loss = fused.kd_ce_loss(s, t, y, 2.0, 0.5, 0.25, row_mask=on)
    (g,) = torch.autograd.grad(loss * 3.0, s)
    r = s.detach().double().requires_grad_()
    ls, lt = F.log_softmax(r / 2, 1), F.log_softmax(t.double() / 2, 1)
    term = torch.where(lt.exp() > 0, lt.exp() * (lt - ls), torch.zeros_like(ls))
    ref = 0.25 * 4 * term[on].sum() + 0.5 * F.cross_entropy(r[on], y[on], ignore_index=-100, reduction="sum")
    (gr,) = torch.autograd.grad(ref * 3.0, r)
    assert abs(float(loss.detach()) - float(ref.detach())) <= 1e-5 * abs(float(ref.detach()))
    assert _rel(g, gr) < max(2 * EPS[dtype], 1e-5)
    assert not g[~on].any()
    s = s.detach().clone()
    s[0, : c // 2] = -math.inf
    s.requires_grad_()
    (g,) = torch.autograd.grad(fused.kd_ce_loss(s, None, y, 1.0, 1.0, 0.0), s)
    r = s.detach().double().requires_grad_()
    (gr,) = torch.autograd.grad(F.cross_entropy(r, y, ignore_index=-100, reduction="sum"), r)
    assert _rel(g, gr) < max(2 * EPS[dtype], 1e-5)


@pytest.mark.parametrize("n,c", [(1, 30528), (1023, 24584), (1024, 24576), (1024, 28664), (1024, 28672), (1024, 24584), (1025, 30528), (1100, 30720),
                                 (1024, 30728), (591, 24584), (592, 24584), (592, 24576), (592, 30720)])
def test_kd_ce_long_rows(n, c):
    """Either side of the limits of the kernel that keeps a row on the chip (592 rows, 24584 to 30720 elements), with masked
    rows, a row without a label, one with classes switched off."""
    from tspipe_b200.ops import fused
    torch.manual_seed(0)
    s, t = ((torch.randn(n, c, device=DEV) * 3).bfloat16() for _ in range(2))
    s[0, : c // 2] = t[0, : c // 2] = torch.finfo(torch.bfloat16).min
    y = torch.randint(c // 2 + 1, c, (n,), device=DEV)
    on = torch.arange(n, device=DEV) % 5 != 3
    y[n // 2] = -100 if n > 1 else c - 1
    s.requires_grad_()
    for row_mask, keep in ((on, on), (None, torch.ones_like(on))):
        loss = fused.kd_ce_loss(s, t, y, 2.0, 0.5, 0.25, row_mask=row_mask)
        (g,) = torch.autograd.grad(loss, s)
        want, err, norm = 0.0, 0.0, 0.0
        for rows in torch.arange(n, device=DEV).split(64):
            r = s.detach()[rows].double().requires_grad_()
            ls, lt = F.log_softmax(r / 2, 1), F.log_softmax(t[rows].double() / 2, 1)
            term = torch.where(lt.exp() > 0, lt.exp() * (lt - ls), torch.zeros_like(ls))[keep[rows]]
            ref = term.sum() + 0.5 * F.cross_entropy(r[keep[rows]], y[rows][keep[rows]], ignore_index=-100, reduction="sum")
            (gr,) = torch.autograd.grad(ref, r)
            want += float(ref.detach())
            err += float((g[rows].double() - gr).square().sum())
            norm += float(gr.square().sum())
        assert abs(float(loss.detach()) - want) <= 1e-5 * abs(want)
        assert math.sqrt(err / norm) < 2 * EPS[torch.bfloat16]
        assert not g[~keep].any()
    t[n - 1 if keep[n - 1] else 0, 9] = math.nan
    assert fused.kd_ce_loss(s, t, y, 2.0, 0.5, 0.25).isnan()


def test_kd_ce_long_rows_with_maxima_that_grow_along_a_row():
    """Logits that rise from vector to vector, in steps that stay with a warp's reference and in steps that move it, for the
    student, the teacher and both, in labelled rows and others."""
    from tspipe_b200.ops import fused
    torch.manual_seed(4)
    n, c = 600, 30528
    part = torch.arange(c, device=DEV) // 6144
    s, t = (torch.randn(n, c, device=DEV) for _ in range(2))
    rise = torch.tensor([0.0, 1.5, 3.0, 10.0, 60.0], device=DEV).repeat_interleave(n // 5)[:, None] * part
    s[::3] += rise[::3]
    t[1::3] += rise[1::3]
    s[2::3] += rise[2::3]
    t[2::3] += 0.5 * rise[2::3]
    s, t = s.bfloat16().requires_grad_(), t.bfloat16()
    y = torch.where(torch.arange(n, device=DEV) % 2 == 0, torch.randint(0, c, (n,), device=DEV), -100)
    loss = fused.kd_ce_loss(s, t, y, 2.0, 0.5, 0.25)
    (g,) = torch.autograd.grad(loss, s)
    r = s.detach().double().requires_grad_()
    ls, lt = F.log_softmax(r / 2, 1), F.log_softmax(t.double() / 2, 1)
    ref = (lt.exp() * (lt - ls)).sum() + 0.5 * F.cross_entropy(r, y, ignore_index=-100, reduction="sum")
    (gr,) = torch.autograd.grad(ref, r)
    assert abs(float(loss.detach()) - float(ref.detach())) <= 1e-6 * abs(float(ref.detach()))
    for i in range(n):                                  # every row by itself: bf16's rounding
        assert _rel(g[i], gr[i]) < 2 * EPS[torch.bfloat16]


@pytest.mark.parametrize("n,c,dtype,mask", [(40, 1000, torch.float32, None), (40, 1001, torch.bfloat16, torch.int64),
                                            (600, 30528, torch.bfloat16, torch.bool)])
def test_distil_loss_equals_its_terms(n, c, dtype, mask):
    """One call for both terms, above and below the limits of the kernel for long rows: value, gradients, scaled backward."""
    from tspipe_b200.ops import fused
    torch.manual_seed(5)
    s, t = ((torch.randn(n // 4, 4, c, device=DEV) * 2).to(dtype) for _ in range(2))
    x, y = (torch.randn(n // 4, 4, 72, device=DEV).to(dtype) for _ in range(2))
    lab = torch.randint(-1, c, (n // 4, 4), device=DEV)
    on = None if mask is None else (torch.arange(n, device=DEV).view(-1, 4) % 3 != 1).to(mask)
    s.requires_grad_()
    x.requires_grad_()
    one = fused.distil_loss(s, t, lab, 2.0, 0.5, 0.25, x, y, 0.125, row_mask=on)
    two = fused.kd_ce_loss(s, t, lab, 2.0, 0.5, 0.25, row_mask=on) + fused.cosine_embedding_loss(x, y, 0.125, row_mask=on)
    assert abs(float(one.detach()) - float(two.detach())) <= 3e-7 * abs(float(two.detach()))
    for a, b in zip(torch.autograd.grad(3 * one, [s, x]), torch.autograd.grad(3 * two, [s, x])):
        assert a.shape == b.shape and _rel(a, b) < 1e-6
    (only,) = torch.autograd.grad(fused.distil_loss(s.detach(), t, lab, 2.0, 0.5, 0.25, x, y, 0.125, row_mask=on), x)
    assert _rel(only, torch.autograd.grad(fused.cosine_embedding_loss(x, y, 0.125, row_mask=on), x)[0]) < 1e-6


@pytest.mark.parametrize("reserve", [0, 8])
def test_kd_ce_long_rows_leave_reserved_sms(reserve):
    from tspipe_b200.ops import fused as f
    n, c = 1024, 30528
    s = torch.randn(n, c, device=DEV).bfloat16()
    total, loss = torch.empty(3, dtype=torch.float64, device=DEV), torch.empty((), device=DEV)
    f.set_sm_reserve(reserve)
    try:
        assert f.lib().tsp_kd_ce_loss(s.data_ptr(), s.data_ptr(), None, None, n, c, 1, 1, 2.0, 0.0, 1.0, total.data_ptr(),
                                      loss.data_ptr(), None, f._raw_stream()) == 0
    finally:
        f.set_sm_reserve(0)
    tickets, blocks = total[1:2].view(torch.int32).tolist()
    assert blocks == torch.cuda.get_device_properties(DEV).multi_processor_count - reserve and tickets == n + blocks
    assert abs(float(loss)) < 1e-4


@pytest.mark.parametrize("reserve", [0, 8])
def test_kd_ce_long_rows_from_four_per_usable_sm(reserve):
    from tspipe_b200.ops import fused as f
    usable, c = torch.cuda.get_device_properties(DEV).multi_processor_count - reserve, 24584
    s = torch.randn(4 * usable, c, device=DEV).bfloat16()
    total, loss = torch.empty(3, dtype=torch.float64, device=DEV), torch.empty((), device=DEV)
    for n in (4 * usable - 1, 4 * usable):
        f.set_sm_reserve(reserve)
        try:
            assert f.lib().tsp_kd_ce_loss(s.data_ptr(), s.data_ptr(), None, None, n, c, 1, 1, 2.0, 0.0, 1.0, total.data_ptr(),
                                          loss.data_ptr(), None, f._raw_stream()) == 0
        finally:
            f.set_sm_reserve(0)
        tickets, blocks = total[1:2].view(torch.int32).tolist()          # (none drawn by the kernel for fewer rows)
        assert (tickets, blocks) == ((n + usable, usable) if n == 4 * usable else (0, 0))
        assert abs(float(loss)) < 1e-4


@pytest.mark.parametrize("off", [-math.inf, torch.finfo(torch.bfloat16).min])
def test_kd_ce_long_rows_with_classes_switched_off_for_the_student_alone(off):
    """Many rows give what few rows do, whose kernel forms the divergence from the probabilities: where the student's lowest
    values meet the teacher's best classes (the largest float, times a mass of one), and where what the teacher gives them
    vanishes in steps along the row."""
    from tspipe_b200.ops import fused
    torch.manual_seed(3)
    n, c, step = 1100, 30528, 6144
    s, t = ((torch.randn(n, c, device=DEV) * 3).bfloat16() for _ in range(2))
    if off != -math.inf:
        s[3, ::2] = off
    t[5, :step] -= 320
    t[5, step: 2 * step] -= 160
    s[5, :step] = off
    t[n - 1, 7::9] = s[n - 1, 7::9] = off
    y = torch.randint(0, c, (n,), device=DEV)
    y[3] = y[5] = y[n - 1] = -100
    s.requires_grad_()
    loss = fused.kd_ce_loss(s, t, y, 2.0, 0.5, 0.25)
    (g,) = torch.autograd.grad(loss, s)
    parts = [fused.kd_ce_loss(s[i:j], t[i:j], y[i:j], 2.0, 0.5, 0.25) for i, j in ((0, 4), (4, 512), (512, n))]
    (want_g,) = torch.autograd.grad(sum(parts), s)
    want = sum(p.detach().double() for p in parts)
    assert want.isfinite() and abs(float(loss.detach()) - float(want)) <= 1e-5 * abs(float(want))
    assert _rel(g, want_g) < 2 * EPS[torch.bfloat16]
    with torch.no_grad():                               # without the row whose value hides the others'
        loss, part = fused.kd_ce_loss(s[4:], t[4:], y[4:], 2.0, 0.5, 0.25), fused.kd_ce_loss(s[4:512], t[4:512], y[4:512], 2.0, 0.5, 0.25)
        want = part.double() + fused.kd_ce_loss(s[512:], t[512:], y[512:], 2.0, 0.5, 0.25).double()
    assert want.isfinite() and abs(float(loss) - float(want)) <= 1e-5 * abs(float(want))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("temp", [0.5, 1.0, 1.4, 2.0])
def test_kd_with_classes_switched_off_at_every_temperature(temp, dtype):
    """Classes that the type's lowest value, or -inf, switches off in the teacher, or in the teacher and the student, add
    nothing to the divergence on either side of T = log2(e) = 1.44; a NaN still shows."""
    from tspipe_b200.ops import fused
    torch.manual_seed(18)
    low = torch.finfo(dtype).min
    for off, in_student in ((low, False), (low, True), (-math.inf, False), (-math.inf, True)):
        s, t = ((torch.randn(4, 264, device=DEV) * 2).to(dtype) for _ in range(2))
        t[:, :100] = off
        if in_student:
            s[:, :100] = off
        s.requires_grad_()
        loss = fused.kd_ce_loss(s, t, None, temp, 0.0, 1.0)
        (g,) = torch.autograd.grad(loss, s)
        r, t6 = s.detach().double().requires_grad_(), t.double()
        ls, lt = F.log_softmax(r / temp, 1), F.log_softmax(t6 / temp, 1)
        ref = temp ** 2 * (lt.exp() * (lt - ls))[:, 100:].sum()
        (gr,) = torch.autograd.grad(ref, r)
        assert abs(float(loss.detach()) - float(ref.detach())) <= 1e-5 * abs(float(ref.detach()))
        assert _rel(g, torch.nan_to_num(gr, nan=0.0)) < max(2 * EPS[dtype], 1e-5)
    t[1, 200] = math.nan
    assert fused.kd_ce_loss(s, t, None, temp, 0.0, 1.0).isnan()


def test_losses_of_many_rows_lose_nothing_in_their_sum():
    """20000 terms added one by one in fp32 would be some 1e-6 to 1e-5 off; the terms' own roundings cancel to below 2^-24."""
    from tspipe_b200.ops import fused
    torch.manual_seed(17)
    s, t = torch.randn(20000, 16, device=DEV) * 2, torch.randn(20000, 16, device=DEV) * 2
    y = torch.randint(0, 16, (20000,), device=DEV)
    s6, t6 = s.double(), t.double()
    kd = F.kl_div(F.log_softmax(s6 / 2, 1), F.log_softmax(t6 / 2, 1), reduction="sum", log_target=True)
    for got, want in ((fused.kd_ce_loss(s, t, y, 2.0, 0.5, 0.25), 0.25 * 4 * kd + 0.5 * F.cross_entropy(s6, y, reduction="sum")),
                      (fused.cosine_embedding_loss(s, t, 0.5), 0.5 * (1 - F.cosine_similarity(s6, t6)).sum())):
        assert got.dtype == torch.float32 and abs(float(got) - float(want)) <= 4e-7 * abs(float(want))


@pytest.mark.parametrize("n,d", [(1, 8), (2048, 256), (20000, 16)])
def test_byol_loss_of_many_rows_loses_nothing_in_its_sum(n, d):
    """Both directions' terms go into one 64-bit sum; every term is right to some 2^-22 and the roundings cancel."""
    from tspipe_b200.ops import fused
    torch.manual_seed(27)
    o1, o2, t1, t2 = (torch.randn(n, d, device=DEV) for _ in range(4))
    want = sum((2 - 2 * F.cosine_similarity(a.double(), b.double())).mean() for a, b in ((o1, t2), (o2, t1)))
    for _ in range(2):                                 # (scratch of an earlier call)
        got = fused.byol_loss(o1, o2, t1, t2)
        assert got.dtype == torch.float32 and abs(float(got) - float(want)) <= (4e-7 if n == 1 else 2e-7) * abs(float(want))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n,d", [(1, 8), (7, 256), (130, 100)])
def test_byol_pair_equals_two_single_losses(n, d, dtype):
    from tspipe_b200.ops import fused
    torch.manual_seed(1)
    o1, o2, t1, t2 = (torch.randn(n, d, device=DEV).to(dtype) for _ in range(4))
    o1, o2 = o1.requires_grad_(), o2.requires_grad_()
    gs = torch.autograd.grad(fused.byol_loss(o1, o2, t1, t2), [o1, o2])
    ref = fused.byol_pair_loss(o1, t2, 1.0 / n) + fused.byol_pair_loss(o2, t1, 1.0 / n)
    for a, b in zip(gs, torch.autograd.grad(ref, [o1, o2])):
        assert torch.equal(a, b)
    # a recorded or batched product goes through plain ops
    (g,) = torch.autograd.grad(fused.byol_loss(o1, o2, t1, t2), o1, torch.ones((), device=DEV, requires_grad=True),
                               create_graph=True)
    assert g.requires_grad and torch.equal(g.detach(), gs[0])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [128, 129, 200, 1000, 1184, 1185, 2048])
def test_nce_pair_matches_cross_entropy(n, dtype):
    """Ragged query tiles, key chunks whose last one is short."""
    from tspipe_b200.losses import moco_loss
    from tspipe_b200.ops import gemm
    torch.manual_seed(2)
    q1, q2, k1, k2 = ((torch.randn(n, 256, device=DEV) * 2).to(dtype) for _ in range(4))
    q1, q2 = (q1 + k2).requires_grad_(), (q2 + k1).requires_grad_()
    chunk, c = gemm.nce_pair_chunks(n)
    assert chunk % 64 == 0 and (c - 1) * chunk < n <= c * chunk
    assert gemm.info_nce_pair(q1, k2, q2, k1, 0.2) is not None
    loss = moco_loss(q1, q2, k1, k2)
    g = torch.autograd.grad(loss, [q1, q2])
    gemm.check_status()
    r = [t.detach().double().requires_grad_() for t in (q1, q2)]
    lab = torch.arange(n, device=DEV)
    ref = sum(0.4 * F.cross_entropy(F.normalize(a, dim=1) @ F.normalize(b.double(), dim=1).t() / 0.2, lab)
              for a, b in zip(r, (k2, k1)))
    assert abs(float(loss.detach()) - float(ref.detach())) < 2e-3 * abs(float(ref.detach()))       # unit rows and probabilities in bf16
    for a, b in zip(g, torch.autograd.grad(ref, r)):
        assert _rel(a, b) < 8e-3


@pytest.mark.parametrize("noise", [0.05, 0.7])
@pytest.mark.parametrize("n,dtype", [(128, torch.float32), (512, torch.float32), (512, torch.bfloat16)])
def test_nce_pair_does_not_round_its_value_to_16_bits(n, dtype, noise):
    """Rounding rows to bf16 moves a score by some 2^-9 / sqrt(256) / T, 6e-4; the mean over n rows of either direction by 6e-4 /
    sqrt(2 n) = 4e-5 at 128.  Corrected to first order what is left is second order and fp32 sums: a tenth of that at most."""
    from tspipe_b200.ops import gemm
    torch.manual_seed(26)
    base = [torch.randn(n, 256, device=DEV) for _ in range(2)]
    q1, q2, k1, k2 = ((base[i % 2] + noise * torch.randn(n, 256, device=DEV)).to(dtype) for i in range(4))
    loss = gemm.info_nce_pair(q1, k1, q2, k2, 0.2)
    lab = torch.arange(n, device=DEV)
    ref = sum(0.4 * F.cross_entropy(F.normalize(a.double(), dim=1) @ F.normalize(b.double(), dim=1).t() / 0.2, lab)
              for a, b in ((q1, k1), (q2, k2)))
    assert abs(float(loss) - float(ref)) < 4e-6 * max(1.0, float(ref))


# ---- optimizers ---------------------------------------------------------------------------------------------------
@pytest.mark.parametrize("name", ["adamw", "sgd"])
@pytest.mark.parametrize("shift", [0, 1])
def test_vectorised_optimizer_on_an_unaligned_teacher(name, shift):
    """A teacher buffer off the 16-byte grid, and one whose end cuts a vector, take the scalar loop."""
    from tspipe_b200.optim import SGD, AdamW
    from tspipe_b200.runtime.state import FlatParams
    torch.manual_seed(3)
    ps = [nn.Parameter(torch.randn(37, 53, device=DEV)), nn.Parameter(torch.randn(130, device=DEV))]
    ref = [nn.Parameter(p.detach().clone()) for p in ps]
    mk = (lambda q: AdamW(q, lr=1e-2, weight_decay=0.1)) if name == "adamw" else \
        (lambda q: SGD(q, lr=0.05, momentum=0.9, weight_decay=1e-3))
    flat = FlatParams(ps, DEV, with_grad=True)
    opt, ropt = mk(ps), mk(ref)
    opt.bind_flat(flat, use_kernel=True)
    n = flat.total - 64 + shift * 2                 # shift 1: an end inside the last parameter's vectors
    teacher = torch.zeros(flat.total + 8, device=DEV)[shift: shift + n]
    opt.teacher_flat, opt.ema_momentum = teacher, 0.5
    for p, q in zip(ps, ref):
        q.grad = torch.randn_like(q)
        p.grad.copy_(q.grad)
    opt.step()
    ropt.step()
    for p, q in zip(ps, ref):
        torch.testing.assert_close(p.detach(), q.detach(), rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(teacher, 0.5 * flat.data[:n], rtol=1e-6, atol=1e-7)


# ---- elementwise and row passes -----------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("m,n", [(2, 8), (77, 24), (1000, 768), (300, 4096), (130, 5120)])
def test_column_sums(m, n, dtype):
    from tspipe_b200.ops import gemm
    torch.manual_seed(4)
    x = torch.randn(m, n, device=DEV).to(dtype)
    want = x.double().sum(0)
    torch.testing.assert_close(gemm._column_sums(x).double(), want, rtol=0, atol=1e-5 * math.sqrt(m) * 4)
    base = torch.full((n,), 2.0, device=DEV)
    assert gemm._column_sums(x, add_to=base) is None
    torch.testing.assert_close(base.double() - 2, want, rtol=0, atol=1e-5 * math.sqrt(m) * 4)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("m,c,res", [(16, 4096, False), (64, 4096, True), (37, 24, True), (515, 1000, False),
                                     (4099, 64, True), (9, 2056, False)])
def test_batchnorm_passes_at_odd_widths(m, c, res, dtype):
    """Channel counts whose vectors do and do not divide a block, from one row per thread to several trips."""
    from tspipe_b200.ops import bn as fbn
    torch.manual_seed(5)
    mod = nn.BatchNorm1d(c).to(DEV)
    with torch.no_grad():
        mod.weight.normal_(1, 0.2)
        mod.bias.normal_(0.3, 0.2)
    x = (torch.randn(m, c, device=DEV) + 0.5).to(dtype).requires_grad_()
    r = torch.randn(m, c, device=DEV).to(dtype).requires_grad_() if res else None
    g = torch.randn(m, c, device=DEV).to(dtype)
    y = fbn.bn_act(mod, x, r, True)
    got = torch.autograd.grad(y, [x, mod.weight, mod.bias] + ([r] if res else []), g)
    x6, w6, b6 = x.detach().double().requires_grad_(), mod.weight.detach().double().requires_grad_(), \
        mod.bias.detach().double().requires_grad_()
    r6 = r.detach().double().requires_grad_() if res else None
    z = F.batch_norm(x6, None, None, w6, b6, True)
    z = z + r6 if res else z
    assert _rel(y, F.relu(z)) < 2 * EPS[dtype] + 1e-6
    z = z * (y.double() > 0)                           # the kernel's own mask: roundings at the corner are not at issue
    want = torch.autograd.grad(z, [x6, w6, b6] + ([r6] if res else []), g.double())
    for a, b in zip(got, want):
        assert _rel(a, b) < 4 * EPS[dtype] + 2e-5


@pytest.mark.parametrize("train,relu,res", [(True, True, False), (True, False, False), (True, True, True), (False, False, False),
                                            (False, True, False)])
def test_batchnorm_with_parameters_anywhere_in_a_vector(train, relu, res):
    """Weight and bias as slices of one vector, off the 16-byte grid, give what aligned ones give."""
    from tspipe_b200.batchnorm import BatchNormGroup, DeferredBatchNorm
    from tspipe_b200.ops import bn as fbn
    c = 64
    torch.manual_seed(19)
    x, r, g = (_cl(4, c, 6, 10) for _ in range(3))
    vec = torch.cat([torch.zeros(1, device=DEV), torch.randn(2 * c, device=DEV)])
    outs = []
    for off in (0, 1):
        mod = DeferredBatchNorm(c).to(DEV).train(train)
        BatchNormGroup(mod, chunks=10)
        flat = vec[1:].clone() if off == 0 else vec
        torch.nn.utils.vector_to_parameters(flat[off:], mod.parameters())
        assert (mod.weight.data_ptr() % 16 != 0) == (off != 0)
        xi = x.clone(memory_format=torch.preserve_format).requires_grad_()
        y = fbn.bn_act(mod, xi, r if res else None, relu)
        out = [y, *torch.autograd.grad(y, [xi, mod.weight, mod.bias], g)]
        if train and relu and not res:
            z = fbn.bn_relu_pool(mod, xi)
            out += [z, *torch.autograd.grad(z, [xi, mod.weight, mod.bias], _cl(*z.shape).fill_(1.0))]
        outs.append(out)
    for a, b in zip(*outs):
        assert _rel(a, b) < 1e-3                       # the sums' additions come in any order: a rounding here and there


def test_layer_norm_and_gelu_with_parameters_anywhere_in_a_vector():
    """Weights and biases as slices of a vector, off the 16-byte grid, give what aligned ones give."""
    from tspipe_b200.ops import fused
    torch.manual_seed(20)
    d = 72
    x, a, g = (torch.randn(9, d, device=DEV) for _ in range(3))
    x.requires_grad_()
    vec = torch.randn(3 * d + 1, device=DEV)
    outs = []
    for w, b, c in (vec[1:].view(3, d).unbind(0), vec[1:].clone().view(3, d).unbind(0)):
        w, b, c = (t.detach().requires_grad_() for t in (w, b, c))
        ys = [fused.layer_norm(x, w, b), *fused.add_layer_norm(x, a, w, b), fused.gelu(x, c)]
        outs.append([t for y in ys for t in (y, *torch.autograd.grad(y, [x], g, retain_graph=True))])
    for p, q in zip(*outs):
        assert torch.equal(p, q)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gelu_special_values_and_wide_bias(dtype):
    from tspipe_b200.ops import fused
    x = torch.tensor([math.inf, -1e30, 0.0, -0.0, 40.0, -40.0, math.nan, 1.0], device=DEV).to(dtype)
    y = fused.gelu(x).float()
    assert y[0] == math.inf and y[1] == 0 and y[2] == 0 and y[4] == 40 and y[5] == 0 and y[6].isnan()
    torch.manual_seed(6)
    for rows, d in ((3, 8), (5, 24), (300, 5120)):
        v = (torch.randn(rows, d, device=DEV) * 3).to(dtype).requires_grad_()
        b = torch.randn(d, device=DEV, requires_grad=True)
        out = fused.gelu(v, b)
        g = torch.randn_like(out)
        gv, gb = torch.autograd.grad(out, [v, b], g)
        v6, b6 = v.detach().double().requires_grad_(), b.detach().double().requires_grad_()
        ref = F.gelu(v6 + b6)
        rv, rb = torch.autograd.grad(ref, [v6, b6], g.double())
        for a, w in ((out, ref), (gv, rv), (gb, rb)):
            assert _rel(a, w) < 2 * EPS[dtype] + 1e-6


@pytest.mark.parametrize("res", [False, True])
def test_batchnorm_apply_on_both_sides_of_the_cache_size(res):
    """The rows that a tensor of 126 MB and one above it have in common, which are read with and without hints."""
    from tspipe_b200.ops import bn
    torch.manual_seed(42)
    c, m = 64, (126 << 20) // 128
    x = torch.randn(m + 8, c, device=DEV).bfloat16()
    r = torch.randn_like(x) if res else None
    w, b, mean, var = (torch.rand(c, device=DEV) + 0.5 for _ in range(4))

    def apply(n):
        y, f = torch.empty_like(x[:n]), bn._f
        k = f._c
        fixed = torch.cat([mean, var])
        assert f.lib().tsp_bn_apply(f._ptr(x), f._ptr(r), f._ptr(y), None, f._ptr(fixed), f._ptr(w), f._ptr(b), None, None, None, None,
                                    k.c_int64(0), k.c_int64(n), k.c_int(c), k.c_float(1e-5), k.c_int(1), k.c_int(f._dt(x)), k.c_int(1),
                                    f._stream()) == 0
        return y
    small, large = apply(m), apply(m + 8)
    assert torch.equal(small, large[:m])
    want = (x[-4096:].double() - mean) * (var.double() + 1e-5).rsqrt() * w + b + (r[-4096:].double() if res else 0)
    # a rounding to bf16 behind a handful in fp32 of terms below 32
    assert ((large[-4096:].double() - want.relu()).abs() <= want.abs() * 2.0 ** -8 + 32 * 2.0 ** -21).all()


@pytest.mark.parametrize("shift", [0, 1])
def test_gelu_of_every_bf16_argument(shift):
    """Two values share an instruction: each is its own GELU, in either place, over all arguments with a finite result."""
    from tspipe_b200.ops import fused
    x = torch.arange(-32768, 32768, device=DEV).to(torch.int16).view(torch.bfloat16)
    x = x[x.isfinite()]
    x = x[: x.numel() // 8 * 8].roll(shift)
    y, swapped = fused.gelu(x.view(-1, 8)).view(-1).double(), fused.gelu(x.flip(0).contiguous().view(-1, 8)).view(-1).flip(0).double()
    assert torch.equal(y, swapped)
    v = x.double()
    ref = v * torch.special.ndtr(v)
    # the rounding to bf16; the tail's rational form, 0.75e-7 absolute (Abramowitz & Stegun 7.1.26 has 1.5e-7 for erf), which is
    # an exact zero behind |x| = 16; its fp32 arithmetic and approximate exponential, whose argument is rounded at up to 2^7; a
    # subnormal flushed
    tail = torch.special.ndtr(-v.abs())
    err = (y - ref).abs() - ref.abs() * 2.0 ** -8 - v.abs().clamp_max(16) * (0.75e-7 + tail * 2.0 ** -16) - 2.0 ** -126
    assert err.max() <= 0


@pytest.mark.parametrize("shift", [0, 1])
def test_gelu_gradient_of_every_bf16_argument(shift):
    """As above for the derivative, times one: within a bf16 rounding and the tail's error, also where a gradient of two follows."""
    from tspipe_b200.ops import fused
    x = torch.arange(-32768, 32768, device=DEV).to(torch.int16).view(torch.bfloat16)
    x = x[x.isfinite()]
    x = x[: x.numel() // 8 * 8].roll(shift)

    def grad(v, g):
        v = v.reshape(-1, 8).clone().requires_grad_()
        return torch.autograd.grad(fused.gelu(v), v, torch.full_like(v, g))[0].view(-1)
    g = grad(x, 1.0)
    assert torch.equal(g, grad(x.flip(0), 1.0).flip(0)) and torch.equal(grad(x, 2.0), 2 * g)
    v = x.double()
    density = torch.exp(-0.5 * v * v) * 0.3989422804014327
    ref = torch.special.ndtr(v) + v * density
    # the rounding to bf16; the tail's rational form, 0.75e-7 absolute; its fp32 arithmetic and the approximate exponential, whose argument
    # is rounded at up to 2^7 (2^-17 times ln 2 of it, and as much for its product with the constants); a subnormal flushed
    tail = torch.special.ndtr(-v.abs())
    err = (g.double() - ref).abs() - ref.abs() * 2.0 ** -8 - 0.75e-7 - (tail + v.abs() * density) * 2.0 ** -16 - 2.0 ** -126
    assert err.max() <= 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,d", [(1, 8), (17, 256), (16, 264), (4800, 520), (33, 776), (5000, 1024)])
def test_layer_norm_widths(rows, d, dtype):
    from tspipe_b200.ops import fused
    torch.manual_seed(7)
    x = (torch.randn(rows, d, device=DEV) + 1).to(dtype).requires_grad_()
    w, b = torch.randn(d, device=DEV, requires_grad=True), torch.randn(d, device=DEV, requires_grad=True)
    y = fused.layer_norm(x, w, b, 1e-6)
    g = torch.randn_like(y)
    got = torch.autograd.grad(y, [x, w, b], g)
    leaves = [t.detach().double().requires_grad_() for t in (x, w, b)]
    ref = F.layer_norm(leaves[0], (d,), leaves[1], leaves[2], 1e-6)
    assert _rel(y, ref) < EPS[dtype] + 1e-6
    for a, r in zip(got, torch.autograd.grad(ref, leaves, g.double())):
        assert _rel(a, r) < 2 * EPS[dtype] + 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,d,with_a", [(1, 8, True), (33, 264, True), (700, 768, True), (700, 768, False), (19, 1024, False)])
def test_add_layer_norm_equals_the_separate_passes(rows, d, with_a, dtype):
    from tspipe_b200.ops import fused
    torch.manual_seed(14)
    x, a = ((torch.randn(rows, d, device=DEV)).to(dtype).requires_grad_() for _ in range(2))
    w, b = torch.randn(d, device=DEV, requires_grad=True), torch.randn(d, device=DEV, requires_grad=True)
    gs, gy = torch.randn(rows, d, device=DEV).to(dtype), torch.randn(rows, d, device=DEV).to(dtype)
    leaves = [x, w, b] + ([a] if with_a else [])
    s, y = fused.add_layer_norm(x, a if with_a else None, w, b, 1e-6)
    got = torch.autograd.grad([s, y], leaves, [gs, gy])
    s2 = x + a if with_a else x
    y2 = fused.layer_norm(s2, w, b, 1e-6)
    want = torch.autograd.grad([s2, y2] if with_a else [y2], leaves, [gs, gy] if with_a else [gy])
    if not with_a:
        want = (want[0] + gs,) + want[1:]
    for p, q in zip((s, y) + tuple(got), (s2, y2) + tuple(want)):
        assert _rel(p, q) < 1e-6                       # bit-equal in bf16; fp32 products may be contracted differently
    (only,) = torch.autograd.grad(fused.add_layer_norm(x, a if with_a else None, w, b, 1e-6)[1], x, gy)     # no gradient for s
    assert _rel(only, torch.autograd.grad(fused.layer_norm(s2, w, b, 1e-6), x, gy)[0]) < 1e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape,views", [((2, 64, 8, 8), 2), ((3, 8, 5, 7), 1), ((4, 24, 9, 2), 2), ((2, 64, 30, 16), 1),
                                         ((1, 512, 2, 3), 1), ((2, 64, 18, 33), 2), ((1, 2056, 3, 5), 1),
                                         ((8, 64, 137, 139), 1), ((16, 64, 137, 139), 2)])
def test_batchnorm_relu_maxpool_equals_the_separate_passes(shape, views, dtype):
    """Odd extents (last window of two rows or columns), strips of one, two and four rows that end early, channel counts off
    the block size, more channels than a block takes.  Both sides are handed the same statistics, with sums of zero, whose variance
    is one product however it is contracted: their activations are the same bits, and ties are the same ties."""
    from tspipe_b200.batchnorm import BatchNormGroup, DeferredBatchNorm
    from tspipe_b200.ops import bn as fbn
    from tspipe_b200.ops.pool import MaxPool3x3s2
    torch.manual_seed(8)
    n, c, h, w = shape
    x = _cl(*shape, dtype=dtype).requires_grad_()
    variance = torch.linspace(0.5, 4, c, device=DEV)
    stats = torch.stack([torch.zeros_like(variance), variance * (n // views * h * w)]).repeat(views, 1, 1).reshape(-1)
    outs = []
    for fused in (True, False):
        mod = DeferredBatchNorm(c).to(DEV)
        with torch.no_grad():
            mod.weight.copy_(torch.linspace(-1, 2, c))
            mod.bias.copy_(torch.linspace(0.5, -0.5, c))
        group = BatchNormGroup(mod, chunks=10)
        with fbn.segments(views):
            if fused:
                y = fbn.bn_relu_pool(mod, x, stats.clone())
                _, idx, won = y.grad_fn.saved_tensors[:3]
            else:
                act = fbn.bn_act(mod, x, None, True, stats.clone())
                y = MaxPool3x3s2()(act)
        torch.manual_seed(9)
        g = _cl(*y.shape, dtype=dtype)
        outs.append([y.detach(), *torch.autograd.grad(y, [x, mod.weight, mod.bias] + ([] if fused else [act]), g), group._acc])
    (y, dx, dw, db, acc), (y2, dx2, dw2, db2, dact, acc2) = outs
    assert torch.equal(y, y2) and torch.equal(acc, acc2)
    # the winners: x and the activation at the tap that the code names (a code is larger for an earlier tap)
    code = idx.view(n, y.shape[2], y.shape[3], c).permute(0, 3, 1, 2).long()
    live = code != 255
    assert torch.equal(live, y > 0)
    code = code.where(live, torch.full_like(code, 5))                   # (any tap that exists)
    iy = 2 * torch.arange(y.shape[2], device=DEV).view(-1, 1) - 1 + 2 - code // 4
    ix = 2 * torch.arange(y.shape[3], device=DEV) - 1 + 2 - code % 4
    assert bool(((iy >= 0) & (iy < h) & (ix >= 0) & (ix < w))[live].all())
    at = iy * w + ix

    def taken(t):
        return t.detach().reshape(n, c, h * w).gather(2, at.reshape(n, c, -1)).view_as(y)
    assert torch.equal(taken(x)[live], won[live]) and torch.equal(taken(act)[live], y[live])
    # dx = A (dact - mean(dact) - xhat mean(dact xhat)) with A = weight / std: dact and dx are rounded to the type, on one side perhaps to
    # the neighbour of the other's (two units of 2^-8 or 2^-23); the means are of the rounded dact on one side and of what its windows
    # give on the other; terms add up in another order
    per = lambda t: t.double().reshape(views, n // views, c, h, w)                                      # noqa: E731
    a = (torch.linspace(-1, 2, c, device=DEV).abs() * variance.rsqrt()).view(-1, 1, 1)
    xhat, d = per(x.detach()).abs() * variance.rsqrt().view(-1, 1, 1), per(dact).abs()
    means = d.mean((1, 3, 4), True) + xhat * (d * xhat).mean((1, 3, 4), True)
    off = (per(dx) - per(dx2)).abs() - EPS[dtype] * (2 * per(dx2).abs() + a * (2 * d + means))
    assert float(off.max()) <= 1e-5
    for p, q in ((dw, dw2), (db, db2)):
        assert _rel(p, q) < EPS[dtype] + 1e-5


@pytest.mark.parametrize("widths", [(8,), (64, 8, 256, 2048)])
@pytest.mark.parametrize("chunks", [1, 2, 3])
def test_statistics_commit_equals_the_library_ops(chunks, widths):
    """Steps of one and two views, commits behind the first and the second view, a layer that has seen nothing."""
    from tspipe_b200.batchnorm import BatchNormGroup, DeferredBatchNorm
    torch.manual_seed(22)
    groups = [BatchNormGroup(torch.nn.Sequential(*(DeferredBatchNorm(c, momentum=0.1 + 0.2 * i, chunks=chunks)
                                                   for i, c in enumerate(widths))).to(dev)) for dev in ("cpu", DEV)]
    for step, segs in enumerate((1, 2, 2, 1, 2)):
        acc = torch.rand(3, 2, sum(widths)) * 4
        acc[1] += acc[0].square()
        acc[2] = torch.randint(2, 50, acc[2].shape)
        acc[:, segs:] = 0
        acc[:, :, : widths[0]] *= (step > 2)
        for g in groups:
            g._acc += acc.to(g._acc.device)
            g.step(segments=segs)
    groups[1].commit()
    groups[0].commit()
    for name in ("running_mean", "running_var", "_acc", "nbt"):
        a, b = (getattr(g, name).double().cpu() for g in groups)
        assert _rel(b, a) < 1e-6, name
    assert groups[0].tracked == groups[1].tracked


# ---- tensor-core products -----------------------------------------------------------------------------------------
@pytest.mark.parametrize("m,n,k", [(128, 64, 64), (300, 192, 128), (12608, 768, 64), (257, 4096, 192), (5000, 1024, 64)])
def test_linear_products_at_every_tile_width(m, n, k):
    """The widths that ``pick_bn`` chooses between: full and ragged last tiles in every direction, k tails in the weight
    gradient (rows that are no multiple of 64)."""
    from tspipe_b200.ops import gemm
    torch.manual_seed(10)
    x, w, dy = torch.randn(m, k, device=DEV).bfloat16(), torch.randn(n, k, device=DEV).bfloat16(), \
        torch.randn(m, n, device=DEV).bfloat16()
    assert _rel(gemm.matmul_nt(x, w), x.double() @ w.double().t()) < EPS[torch.bfloat16]
    assert _rel(gemm.matmul_nn([dy], w), dy.double() @ w.double()) < EPS[torch.bfloat16]
    dw = torch.ones(n, k, device=DEV)
    gemm._add_weight_grad(dw, [dy], x)
    gemm.check_status()
    assert _rel(dw - 1, dy.double().t() @ x.double()) < 1e-5


@pytest.mark.parametrize("m,n,k", [(6400, 768, 320), (6376, 760, 64), (4864, 1000, 200), (9344, 768, 128), (12608, 768, 768),
                                   (18950, 256, 72)])
def test_products_with_a_nearly_empty_last_round(m, n, k):
    """One, two or more tiles past whole rounds of 74 pairs: their columns are dealt to the idle pairs."""
    from tspipe_b200.ops import gemm
    torch.manual_seed(29)
    a, b = torch.randn(m, k, device=DEV).bfloat16(), torch.randn(n, k, device=DEV).bfloat16()
    bias = torch.randn(n, device=DEV)
    exact, size = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()

    def close(got, want, ulp, slack=0.0):      # fp32 sums of k terms err by less than 2^-20 of the terms' sizes
        assert ((got.double() - want).abs() <= want.abs() * ulp + (size + bias.abs()) * 2.0 ** -20 + slack).all()

    close(gemm.matmul_nt(a, b, bias, out_dtype=torch.float32), exact + bias.double(), 2.0 ** -22)
    close(gemm.matmul_nt(a, b), exact, 2.0 ** -8)
    if k % 64 == 0:
        close(gemm.matmul_nn([a], b.t().contiguous()), exact, 2.0 ** -8)
    if n % 64 == 0:                            # the activation of the rounded product, rounded once more
        with torch.no_grad():
            got = gemm.linear_gelu(a, b, bias)
        h = exact.bfloat16().double() + bias.double()
        close(got, F.gelu(h), 2.0 ** -7, exact.abs().max().item() * 2.0 ** -7)
    gemm.check_status()


@pytest.mark.parametrize("bias", [True, False])
@pytest.mark.parametrize("rows,c,heads", [((2, 65), 192, 3), ((3, 197), 768, 12)])
def test_fused_qkv_projection_matches_three_linears(rows, c, heads, bias):
    from tspipe_b200.ops import gemm
    from tspipe_b200.ops.attention import project_qkv
    torch.manual_seed(11)
    x = torch.randn(*rows, c, device=DEV).bfloat16().requires_grad_()
    w = (torch.randn(3 * c, c, device=DEV) / math.sqrt(c)).requires_grad_()
    b = torch.randn(3 * c, device=DEV, requires_grad=True) if bias else None
    qkv = project_qkv(x, w, b, heads)
    g = [torch.randn_like(t) for t in qkv]
    leaves = [x, w] + ([b] if bias else [])
    got = torch.autograd.grad(qkv, leaves, g)
    gemm.check_status()
    ref_leaves = [x.detach().double().requires_grad_(), w.detach().bfloat16().double().requires_grad_()] + \
        ([b.detach().double().requires_grad_()] if bias else [])
    ref = F.linear(*ref_leaves).view(*rows, 3, heads, c // heads).permute(2, 0, 3, 1, 4).unbind(0)
    for a, r in zip(qkv, ref):
        assert _rel(a, r) < EPS[torch.bfloat16]
    for a, r in zip(got, torch.autograd.grad(ref, ref_leaves, [t.double() for t in g])):
        assert _rel(a, r) < EPS[torch.bfloat16]


@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("m,n,k", [(128, 64, 64), (300, 192, 128), (1000, 3072, 768)])
def test_linear_gelu_epilogue_equals_the_separate_kernel(m, n, k, grad):
    from tspipe_b200.ops import fused, gemm
    torch.manual_seed(16)
    x = torch.randn(m, k, device=DEV).bfloat16().requires_grad_(grad)
    w = (torch.randn(n, k, device=DEV) * 2 / math.sqrt(k)).requires_grad_(grad)
    b = torch.randn(n, device=DEV, requires_grad=grad)
    y, ref = gemm.linear_gelu(x, w, b), fused.gelu(gemm.linear(x, w, None), b)
    gemm.check_status()
    assert _rel(y, ref) < 1e-4                         # the same roundings
    if grad:
        g = torch.randn_like(y)
        for p, q in zip(torch.autograd.grad(y, [x, w, b], g), torch.autograd.grad(ref, [x, w, b], g)):
            assert _rel(p, q) < 1e-4
        gemm.check_status()


@pytest.mark.parametrize("m,n,k", [(1, 64, 8), (33, 128, 72), (257, 320, 64), (300, 448, 200), (9733, 512, 64)])
def test_linear_gelu_at_the_edges_of_tiles_and_blocks(m, n, k):
    """The epilogue's 32 x 32 blocks past the last row, in a cut tile and in pieces of tiles (the last case): bit for bit."""
    from tspipe_b200.ops import fused, gemm
    torch.manual_seed(41)
    x, w = torch.randn(m, k, device=DEV).bfloat16(), torch.randn(n, k, device=DEV) / math.sqrt(k)
    b = torch.randn(n, device=DEV)
    h = gemm.linear(x, w, None)
    assert torch.equal(gemm.linear_gelu(x, w, b), fused.gelu(h, b))
    y = gemm.linear_gelu(x.clone().requires_grad_(), w, b)          # which keeps h as well
    gemm.check_status()
    assert torch.equal(y.detach(), fused.gelu(h, b))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,d", [(1, 8), (17, 264), (16, 256), (128, 3072), (5000, 1000), (20000, 8200)])
def test_gelu_backward_with_the_bias_gradient(rows, d, dtype):
    """dx as the separate pass writes it, and its column sums added to what is there."""
    from tspipe_b200.ops import fused as f
    torch.manual_seed(25)
    dy, x = ((torch.randn(rows, d, device=DEV) * 2).to(dtype) for _ in range(2))
    b = torch.randn(d, device=DEV)
    dx, want, sums = torch.empty_like(x), torch.empty_like(x), torch.ones(d, device=DEV)
    c = f._c
    assert f.lib().tsp_gelu_bwd(f._ptr(dy), f._ptr(x), f._ptr(b), f._ptr(want), c.c_int64(x.numel()), c.c_int(d), c.c_int(f._dt(x)),
                                f._stream()) == 0
    assert f.lib().tsp_gelu_bwd_sums(f._ptr(dy), f._ptr(x), f._ptr(b), f._ptr(dx), f._ptr(sums), c.c_int64(rows), c.c_int(d),
                                     c.c_int(f._dt(x)), f._stream()) == 0
    assert torch.equal(dx, want)
    # fp32 sums of up to 20000 terms, in groups of some twenty
    torch.testing.assert_close((sums - 1).double(), dx.double().sum(0), rtol=0, atol=2e-6 * float(dx.double().abs().sum(0).max()))


def test_products_on_a_thread_that_has_made_no_runtime_call():
    """Autograd's worker may enter the library with no device context bound: tensor maps have to be made all the same."""
    import threading
    from tspipe_b200.ops import gemm
    a = torch.randn(256, 128, device=DEV).bfloat16()
    b = torch.randn(128, 192, device=DEV).bfloat16()
    target = torch.zeros(128, 128, device=DEV)
    want = gemm.matmul_nn([a], b)
    out, errors = [], []

    def work():
        try:
            gemm._add_weight_grad(target, [a], a)
            out.append(gemm.matmul_nn([a], b))
        except Exception as e:                         # noqa: BLE001
            errors.append(e)

    torch.cuda.synchronize()
    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not errors, errors
    assert torch.equal(out[0], want) and _rel(target, a.double().t() @ a.double()) < 1e-5


def test_forward_kernels_on_threads_that_have_made_no_runtime_call():
    """A forward that autograd's worker computes again (a checkpoint), for the kernels with maps of their own."""
    import threading
    from tspipe_b200.ops import attention, conv, gemm
    f = conv._f
    torch.manual_seed(24)
    a = torch.randn(256, 128, device=DEV).bfloat16()
    q = torch.randn(1, 2, 128, 64, device=DEV).bfloat16()
    x, wm = _cl(2, 3, 16, 16), conv.weight_matrix(torch.randn(64, 3, 7, 7, device=DEV) * 0.1)
    y, word = _cl(2, 64, 8, 8), gemm._status_word(DEV)
    runs = {"gemm": lambda: gemm.matmul_nt(a, a, two_cta=False), "attention": lambda: attention.flash_fwd(q, q, q),
            "stem": lambda: f.lib().tsp_conv_stem_fwd(f._ptr(x), f._ptr(wm), f._ptr(y), None, 2, 16, 16, 1, f._ptr(word), f._stream())}
    for run in runs.values():
        run()                                          # (memory for the outputs is cached from here on)
    torch.cuda.synchronize()
    errors = {}
    for name, run in runs.items():
        def work():
            try:
                code = run()
                if isinstance(code, int) and code != 0:
                    errors[name] = code
            except Exception as e:                     # noqa: BLE001
                errors[name] = e
        t = threading.Thread(target=work)
        t.start()
        t.join()
    gemm.check_status()
    assert not errors, errors


@pytest.mark.parametrize("n,h,w", [(1, 8, 8), (3, 10, 24), (2, 32, 224), (5, 64, 96)])
def test_stem_weight_gradient(n, h, w):
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(12)
    x = _cl(n, 3, h, w)
    weight = (torch.randn(64, 3, 7, 7, device=DEV) * 0.1).requires_grad_()
    y, _ = conv.stem_conv(x, weight, want_sums=False)
    g = _cl(*y.shape)
    want = torch.autograd.grad(F.conv2d(x.double(), (w6 := weight.detach().double().requires_grad_()), stride=2, padding=3),
                               w6, g.double())[0]
    (dw,) = torch.autograd.grad(y, weight, g, retain_graph=True)
    assert _rel(dw, want) < 1e-5
    weight.grad = torch.ones_like(weight).to(memory_format=torch.channels_last)
    y.backward(g)                                      # added in place to an existing gradient
    gemm.check_status()
    assert _rel(weight.grad - 1, want) < 1e-5


@pytest.mark.parametrize("n,h,w", [(1, 8, 8), (3, 10, 24), (2, 22, 200), (1, 14, 224)])
def test_stem_weight_gradient_of_infinite_pixels(n, h, w):
    """Infinite and NaN pixels at the corners, beside the row's end and in an image's last rows reach the taps that pair them
    with a gradient, and no other: what the products read past the rows' ends and of missing rows stays out."""
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(13)
    for at, value in (((0, 1, h - 1, w - 1), math.inf), ((n - 1, 0, 0, w - 2), -math.inf), ((n - 1, 2, h - 2, 0), math.nan)):
        x = _cl(n, 3, h, w)
        x[at] = value
        weight = (torch.randn(64, 3, 7, 7, device=DEV) * 0.1).requires_grad_()
        y, _ = conv.stem_conv(x, weight, want_sums=False)
        g = _cl(*y.shape)
        (dw,) = torch.autograd.grad(y, weight, g)
        gemm.check_status()
        patches, g6 = F.unfold(x.double(), 7, padding=3, stride=2), g.double().flatten(2)
        # (a tap's pixels outside the image are no terms of its sum: zeros times finite gradients)
        want = torch.stack([(g6[i, :, None] * patches[i][None]).sum(-1) for i in range(n)]).sum(0).view(64, 3, 7, 7)
        ok = want.isfinite()
        assert not ok.all() and ok.any() and torch.equal(dw.isfinite(), ok) and torch.equal(dw.isnan(), want.isnan())
        assert _rel(dw[ok], want[ok]) < 1e-5


@pytest.mark.parametrize("n,h,w", [(1, 8, 8), (3, 10, 24), (2, 22, 200), (2, 16, 224)])
def test_stem_weight_gradient_of_infinite_gradients(n, h, w):
    """An infinite or NaN gradient reaches all taps of its channel, those outside the image as a product with zero padding, and
    no other channel; beside an infinite pixel too."""
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(14)
    for at, value in (((0, 5, 0, 0), math.inf), ((n - 1, 63, h // 2 - 1, w // 2 - 1), -math.inf), ((n - 1, 0, h // 4, w // 4), math.nan)):
        for bad_pixel in (False, True):
            x = _cl(n, 3, h, w)
            if bad_pixel:
                x[0, 2, h - 1, w - 1] = math.inf
            weight = (torch.randn(64, 3, 7, 7, device=DEV) * 0.1).requires_grad_()
            y, _ = conv.stem_conv(x, weight, want_sums=False)
            g = _cl(*y.shape)
            g[at] = value
            (dw,) = torch.autograd.grad(y, weight, g)
            gemm.check_status()
            patches, g6 = F.unfold(x.double(), 7, padding=3, stride=2), g.double().flatten(2)
            want = torch.stack([(g6[i, :, None] * patches[i][None]).sum(-1) for i in range(n)]).sum(0).view(64, 3, 7, 7)
            ok = want.isfinite()
            assert ok.any() and not ok[at[1]].any() and torch.equal(dw.isfinite(), ok) and torch.equal(dw.isnan(), want.isnan())
            assert _rel(dw[ok], want[ok]) < 1e-5


@pytest.mark.parametrize("h,w", [(224, 224), (218, 216)])
def test_stem_weight_gradient_of_nan_takes_no_longer(h, w):
    """A gradient of NaN alone, over images of which some hundred rows fall to a CTA.  Where zeros of dY meet pixels the sums are
    formed twice, the second time by threads: 4 to 6 ms."""
    from tspipe_b200.ops import conv
    x = _cl(128, 3, h, w)
    weight = (torch.randn(64, 3, 7, 7, device=DEV) * 0.1).requires_grad_()
    y, _ = conv.stem_conv(x, weight, want_sums=False)
    times = {}
    for name, g in (("finite", _cl(*y.shape)), ("nan", torch.full_like(y, math.nan))):
        for _ in range(3):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            (dw,) = torch.autograd.grad(y, weight, g, retain_graph=True)
            b.record()
            b.synchronize()
            times[name] = min(times.get(name, math.inf), a.elapsed_time(b))
        assert dw.isnan().all() if name == "nan" else dw.isfinite().all()
    assert times["nan"] < (3 * times["finite"] + 0.2 if w % 32 == 0 else 10), times


def test_stem_weight_gradient_by_name_and_past_hooks():
    """Eagerly the gradient goes to autograd, also where a channels-last one is there already: whoever asks for it by name
    gets it, and hooks see it."""
    from tspipe_b200.ops import conv
    torch.manual_seed(21)
    x, g = _cl(2, 3, 16, 16), _cl(2, 64, 8, 8)
    weight = (torch.randn(64, 3, 7, 7, device=DEV) * 0.1).to(memory_format=torch.channels_last).requires_grad_()
    want = torch.autograd.grad(conv.stem_conv(x, weight)[0], weight, g)[0]
    weight.grad = torch.ones_like(weight)
    (got,) = torch.autograd.grad(conv.stem_conv(x, weight)[0], weight, g)
    assert _rel(got, want) < 1e-6 and torch.equal(weight.grad, torch.ones_like(weight))
    weight.register_hook(lambda t: 2 * t)
    conv.stem_conv(x, weight)[0].backward(g)
    assert _rel(weight.grad - 1, 2 * want) < 1e-5


@pytest.mark.parametrize("n,h,w,cin,cout,k", [(1, 8, 16, 64, 256, 1), (3, 10, 10, 128, 256, 1), (2, 7, 7, 512, 512, 1),
                                              (1, 8, 8, 64, 64, 3), (3, 13, 9, 64, 64, 3), (2, 5, 61, 64, 64, 3),
                                              (2, 56, 56, 64, 64, 3), (1, 64, 2, 64, 64, 3), (200, 8, 8, 64, 64, 3)])
def test_convolution_weight_gradient_paths(n, h, w, cin, cout, k):
    """1x1 as a linear layer on the CTA-pair GEMM and 64 to 64 channels 3x3 with the bordered box resident: the fp32 sums of
    exact bf16 products, against float64."""
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(14)
    x = _cl(n, cin, h, w)
    weight = (torch.randn(cout, cin, k, k, device=DEV) * 0.1).to(memory_format=torch.channels_last).requires_grad_()
    y, _ = conv.conv2d(x, weight)
    g = _cl(*y.shape)
    want = torch.autograd.grad(F.conv2d(x.double(), (w6 := weight.detach().double().requires_grad_()), padding=k // 2),
                               w6, g.double())[0]
    for twice in (1, 2):                               # the second one is added to the gradient that is there
        y.backward(g, retain_graph=True)
        gemm.check_status()
        assert _rel(weight.grad, twice * want) < 1e-5


@pytest.mark.parametrize("n,h,w", [(1, 13, 9), (2, 5, 61), (3, 56, 56), (1, 66, 2)])
def test_infinities_stay_in_the_taps_that_they_meet(n, h, w):
    """3x3 weight gradient with the bordered box resident: infinite and NaN activations in the corners and along the borders
    of an image, against the taps' sums over the zero-padded activation one by one."""
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(25)
    x, g = _cl(n, 64, h, w), _cl(n, 64, h, w)
    for c, (i, j, v) in enumerate([(0, 0, math.inf), (h - 1, w - 1, math.nan), (h // 2, 0, -math.inf), (h // 2, w - 1, math.inf),
                                   (0, w // 2, math.nan), (h - 1, w // 2, math.inf), (h - 1, 0, math.inf)]):
        x[n - 1, 8 * c, i, j] = v
    weight = (torch.randn(64, 64, 3, 3, device=DEV) * 0.1).to(memory_format=torch.channels_last).requires_grad_()
    conv.conv2d(x, weight)[0].backward(g)
    gemm.check_status()
    xp, g6 = F.pad(x.double(), (1, 1, 1, 1)), g.double()
    want = torch.stack([torch.stack([torch.einsum("nohw,nihw->oi", g6, xp[:, :, i: i + h, j: j + w]) for j in range(3)], -1)
                        for i in range(3)], -2)
    got, fin = weight.grad.double(), torch.isfinite(want)
    assert not fin.all() and torch.equal(fin, torch.isfinite(got)) and torch.equal(want.isnan(), got.isnan())
    assert torch.equal(want[want.isinf()], got[want.isinf()]) and _rel(got[fin], want[fin]) < 1e-5


@pytest.mark.parametrize("block,cin,planes,stride,side", [("bottleneck", 256, 64, 1, 14), ("bottleneck", 128, 64, 2, 10),
                                                          ("basic", 64, 64, 1, 9), ("basic", 64, 128, 2, 8)])
def test_residual_gradient_rides_in_the_data_gradient(block, cin, planes, stride, side):
    """The gradient of a block's input with the skip branch added by the first convolution's data gradient (1x1, 3x3 and
    3x3 / 2 kernels, ragged pixel tiles) against the sum that autograd forms: the same roundings."""
    from tspipe_b200.models.resnet import BasicBlock, Bottleneck
    from tspipe_b200.ops import conv, gemm
    cls = Bottleneck if block == "bottleneck" else BasicBlock
    out = planes * cls.expansion
    down = nn.Sequential(nn.Conv2d(cin, out, 1, stride=stride, bias=False), nn.BatchNorm2d(out)) \
        if stride != 1 or cin != out else None
    torch.manual_seed(13)
    blk = cls(cin, planes, stride, down).to(DEV).to(memory_format=torch.channels_last)
    x = _cl(3, cin, side, side)
    x1, x2 = x.clone(memory_format=torch.preserve_format).requires_grad_(), x.clone(memory_format=torch.preserve_format).requires_grad_()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y, skip = conv.conv_bn_act_fork(blk.conv1, blk.bn1, x1, relu=True)
        z = conv.conv_bn_act(blk.conv1, blk.bn1, x2, relu=True)
    g, gs = _cl(*y.shape), _cl(*x.shape)
    assert skip.grad_fn is not None
    (a,) = torch.autograd.grad([y, skip], x1, [g, gs])
    (b,) = torch.autograd.grad(z, x2, g)
    assert _rel(a, b + gs) < 1e-3                      # bit-equal but for the order of the BatchNorm sums
    (c,) = torch.autograd.grad(conv.conv2d(x1, blk.conv1.weight, blk.conv1.stride[0])[0], x1, _cl(*y.shape), retain_graph=True)
    assert c.shape == x.shape
    with torch.autocast("cuda", dtype=torch.bfloat16):
        blk(x1).float().square().mean().backward()
    gemm.check_status()
    assert torch.isfinite(x1.grad).all()


def test_loss_gradient_scaling_in_place_and_not():
    """A retained graph gives the same gradient again, with any factor; a freed one takes the buffer over."""
    from tspipe_b200.ops import fused
    torch.manual_seed(15)
    s = torch.randn(9, 1000, device=DEV).bfloat16().requires_grad_()
    y = torch.randint(0, 1000, (9,), device=DEV)
    loss = fused.cross_entropy(s, y)
    one = torch.autograd.grad(loss, s, retain_graph=True)[0].clone()
    (half,) = torch.autograd.grad(loss, s, torch.tensor(0.5, device=DEV), retain_graph=True)
    (again,) = torch.autograd.grad(loss, s, retain_graph=True)
    assert torch.equal(one, again) and torch.equal(half.float(), one.float() * 0.5)
    (last,) = torch.autograd.grad(loss, s, torch.tensor(2.0, device=DEV))
    assert torch.equal(last.float(), one.float() * 2)


def test_loss_gradient_scaling_leaves_what_saved_tensor_hooks_keep():
    from tspipe_b200 import losses
    from tspipe_b200.ops import fused
    torch.manual_seed(22)
    o1, o2, t1, t2 = (torch.randn(128, 256, device=DEV) for _ in range(4))
    o1.requires_grad_()
    y = torch.randint(0, 256, (128,), device=DEV)
    for loss in (lambda: losses.byol_loss(o1, o2, t1, t2), lambda: losses.moco_loss(o1, o2, t1, t2),
                 lambda: fused.cross_entropy(o1, y), lambda: fused.cosine_embedding_loss(o1, t1, 1.0),
                 lambda: fused.byol_pair_loss(o1, t1, 1.0)):
        kept = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: kept.append(t) or t, lambda t: t):
            value = loss()
        before = [t.clone() for t in kept]
        (g,) = torch.autograd.grad(value, o1, torch.tensor(3.0, device=DEV))
        assert kept and all(torch.equal(a, b) for a, b in zip(kept, before))
        assert _rel(g, 3 * torch.autograd.grad(loss(), o1)[0]) < 1e-6


def test_weight_gradients_add_nothing_after_a_wait_that_ran_out():
    """The status word as a wait that gave up leaves it: every role leaves, gradients that are there stay as they are, and the
    next check reports it."""
    from tspipe_b200.ops import conv, gemm
    torch.manual_seed(23)
    word = gemm._status_word(DEV)
    a = torch.randn(300, 128, device=DEV).bfloat16()
    target = torch.ones(128, 128, device=DEV)
    layers = [(_cl(2, cin, 12, 12), (torch.randn(cout, cin, 3, 3, device=DEV) * 0.1).to(memory_format=torch.channels_last))
              for cin, cout in ((64, 64), (64, 128))]
    ys = []
    for x, w in layers:
        w.requires_grad_().grad = torch.ones_like(w)
        ys.append(conv.conv2d(x, w)[0])
    gs = [_cl(*y.shape) for y in ys]
    gemm.check_status()
    word.fill_(7)
    gemm._add_weight_grad(target, [a], a)
    torch.autograd.backward(ys, gs)
    x, dw, dy = _cl(2, 3, 16, 16), torch.ones(64, 147, device=DEV), _cl(2, 64, 8, 8)
    assert conv._f.lib().tsp_conv_stem_wgrad(conv._f._ptr(x), conv._f._ptr(dy), conv._f._ptr(dw), 2, 16, 16, conv._f._ptr(word),
                                             conv._f._stream()) == 0
    with pytest.raises(RuntimeError, match="role 7"):
        gemm.check_status()
    for t in [target, dw] + [w.grad for _, w in layers]:
        assert torch.equal(t, torch.ones_like(t))
    gemm._add_weight_grad(target, [a], a)              # the context stays usable
    gemm.check_status()
    assert _rel(target - 1, a.double().t() @ a.double()) < 1e-5
