"""Flat optimizer steps with hyperparameters that change from step to step, by value and as a table."""
import pytest
import torch
from torch import nn

from tspipe_b200.optim import LARS, SGD, AdamW
from tspipe_b200.runtime.state import FlatParams

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)
MAKE = {"lars": lambda gs: LARS(gs, lr=0.1, weight_decay=1e-3), "adamw": lambda gs: AdamW(gs, lr=1e-2, weight_decay=0.1),
        "sgd": lambda gs: SGD(gs, lr=0.05, momentum=0.9, weight_decay=1e-3)}


def _params(n):
    torch.manual_seed(0)
    return [nn.Parameter(torch.randn(*((33, 17 + i % 5) if i % 3 else (41,)), device=DEV)) for i in range(n)]


def _groups(ps, k):
    return [dict(params=ps[i::k], lr=0.01 * (1 + i % 5), weight_decay=1e-3 * (i % 3)) for i in range(k)]


def _same(ps, ref, steps):
    """A step rounds values no larger than the largest parameter (or update) some four times, on either side."""
    for p, q in zip(ps, ref):
        atol = 2 * 4 * steps * 2 ** -24 * max(1.0, float(q.detach().abs().max()))
        torch.testing.assert_close(p.detach(), q.detach(), rtol=0, atol=atol)


@pytest.mark.parametrize("name", sorted(MAKE))
@pytest.mark.parametrize("groups", [1, 3, 32, 33, 40])
def test_groups_with_a_schedule_match_the_step_per_tensor(name, groups):
    """One group to more than travel by value, every group with its own and a new learning rate in every step."""
    ps, ref = _params(80), _params(80)
    opt, ropt = MAKE[name](_groups(ps, groups)), MAKE[name](_groups(ref, groups))
    flat = FlatParams(ps, DEV, with_grad=True)
    opt.bind_flat(flat, use_kernel=True)
    for step in range(3):
        torch.manual_seed(step)
        for p, q in zip(ps, ref):
            q.grad = torch.randn_like(q)
            p.grad.copy_(q.grad)
        for o in (opt, ropt):
            for i, g in enumerate(o.param_groups):
                g["lr"] *= 0.9 + 0.002 * i
            o.step()
    _same(ps, ref, 3)


@pytest.mark.parametrize("lag", [0, 1, 7, 1000])
@pytest.mark.parametrize("ema", [False, True])
def test_lars_norms_and_updates_in_one_launch(lag, ema):
    """Tensors of less than a chunk to many, one with an odd length, at distances between norms and update from none to all
    of the work; two steps, the second on the counters that the first has left."""
    from tspipe_b200.ops import fused
    torch.manual_seed(0)
    shapes = [(33, 17), (41,), (700, 257), (3, 16384), (5,), (16384,), (900, 1024), (16385, 1)]
    ps = [nn.Parameter(torch.randn(*s, device=DEV)) for s in shapes]
    ref = [nn.Parameter(p.detach().clone()) for p in ps]
    flat = FlatParams(ps, DEV, with_grad=True)
    opt, ropt = MAKE["lars"](ps), MAKE["lars"](ref)
    opt.bind_flat(flat, use_kernel=True)
    order = fused.LarsOrder(opt._chunks, len(ps), DEV, lag=lag)
    teacher = flat.data.clone() if ema else None
    mu = torch.zeros_like(flat.data)
    want = [p.detach().clone() for p in ref]
    for step in range(2):
        for p, q in zip(ps, ref):
            q.grad = torch.randn_like(q)
            p.grad.copy_(q.grad)
        rows = [[g["lr"], g["weight_decay"], g["momentum"], g["trust_coefficient"]] for g in opt._groups]
        fused.lars_step_ordered_(flat.data, flat.grad, mu, order, opt._hyper_of(rows), 1.0, teacher, 0.9)
        ropt.step()
        want = [0.9 * w + 0.1 * q.detach() for w, q in zip(want, ref)]
    assert int(order.status) == 0
    _same(ps, ref, 2)
    if ema:
        _same([flat._view(teacher, i, p.data) for i, p in enumerate(ps)], want, 2)


def test_lars_wait_that_runs_out_is_raised():
    """A tensor whose norms are never all in (an order that asks for a piece too many): the step ends, that tensor is NaN, the
    others are stepped, and neither a step nor a checkpoint follows until a state is loaded."""
    shapes = [(600, 4096), (513, 4096), (41,), (700, 4096)]
    torch.manual_seed(0)
    ps = [nn.Parameter(torch.randn(*s, device=DEV)) for s in shapes]
    ref = [nn.Parameter(p.detach().clone()) for p in ps]
    flat = FlatParams(ps, DEV, with_grad=True)
    opt, ropt = MAKE["lars"](ps), MAKE["lars"](ref)
    opt.bind_flat(flat, use_kernel=True)
    assert opt._order is not None
    for p, q in zip(ps, ref):
        q.grad = torch.randn_like(q)
        p.grad.copy_(q.grad)
    opt._buf("mu")
    state = opt.state_dict()
    before = flat.data.clone()
    opt._order.need[3] += 1
    opt.step()
    ropt.step()
    torch.cuda.synchronize()
    _same(ps[:3], ref[:3], 1)
    assert ps[3].isnan().all()
    for use in (opt.step, opt.state_dict):
        with pytest.raises(RuntimeError, match="ran out"):
            use()
    flat.data.copy_(before)
    opt._order.need[3] -= 1
    opt.load_state_dict(state)
    opt.step()
    _same(ps, ref, 1)
    opt.state_dict()


@pytest.mark.parametrize("reserve", [0, 8])
def test_lars_in_one_launch_leaves_reserved_sms(reserve):
    """Every block draws a ticket more than it has rows of work."""
    from tspipe_b200.ops import fused
    ps = [nn.Parameter(torch.randn(3000, 2048, device=DEV)), nn.Parameter(torch.randn(77, device=DEV))]
    flat = FlatParams(ps, DEV, with_grad=True)
    opt = MAKE["lars"](ps)
    opt.bind_flat(flat, use_kernel=True)
    order = fused.LarsOrder(opt._chunks, 2, DEV)
    fused.set_sm_reserve(reserve)
    try:
        fused.lars_step_ordered_(flat.data, flat.grad, torch.zeros_like(flat.data), order, opt._hyper_of([[0.1, 0.0, 0.9, 1e-3]]))
    finally:
        fused.set_sm_reserve(0)
    tickets, sms = int(order.work.view(torch.int32)[4]), torch.cuda.get_device_properties(0).multi_processor_count
    assert order.order.shape[0] > 4 * sms and tickets - order.order.shape[0] == 4 * (sms - reserve)


def test_a_recorded_step_repeats_its_values_and_refuses_new_ones():
    ps, qs = _params(5), _params(5)
    lars, adam = MAKE["lars"](ps), MAKE["adamw"](qs)
    for o, x in ((lars, ps), (adam, qs)):
        o.bind_flat(FlatParams(x, DEV, with_grad=True), use_kernel=True)
        o.step()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        lars.step()                                   # nothing has changed since the last step
    with pytest.raises(RuntimeError, match="cannot be recorded"):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            adam.step()                               # the bias corrections have
    for p in ps:
        p.grad.fill_(0.5)
    before = [p.detach().clone() for p in ps]
    g.replay()
    assert all(not torch.equal(p, b) for p, b in zip(ps, before))


@pytest.mark.parametrize("name", ["lars", "adamw"])
@pytest.mark.parametrize("groups,rows", [(2, False), (40, False), (2, True)])
def test_data_parallel_kernels_on_the_same_values(name, groups, rows):
    """The replicas' kernels, which do not wait for one another, with two replicas' buffers on one GPU: each updates its half
    of the range in both, from the mean of both gradients; with the optimizer's values or a row of them per segment."""
    from tspipe_b200.comm.peer import pointer_table
    from tspipe_b200.ops import fused
    ps, ref = _params(80), _params(80)
    opt, ropt = MAKE[name](_groups(ps, groups)), MAKE[name](_groups(ref, groups))
    flat = FlatParams(ps, DEV, with_grad=True, pad_to=2)
    opt.bind_flat(flat, use_kernel=True)
    torch.manual_seed(1)
    for p, q in zip(ps, ref):
        p.grad.normal_()
        q.grad = p.grad.clone()
    data2, grad2 = flat.data.clone(), flat.grad.clone()
    flat.grad.mul_(0.5)
    grad2.mul_(1.5)                                   # the mean is the reference's gradient
    grads, params = pointer_table([flat.grad, grad2]), pointer_table([flat.data, data2])
    ropt.step()
    half = flat.total // 2
    chunks = [fused.build_chunks(flat.offsets, flat.numels, DEV, r * half, (r + 1) * half) for r in (0, 1)]
    if name == "lars":
        vals = [[g["lr"], g["weight_decay"], g["momentum"], g["trust_coefficient"]] for g in opt._groups]
        hp = torch.tensor([vals[i % groups] + [float(p.ndim > 1)] for i, p in enumerate(ps)], device=DEV) if rows \
            else opt._hyper_of(vals)
        g_out, mu, norms = torch.zeros_like(flat.grad), torch.zeros_like(flat.grad), []
        for r in (0, 1):
            norms.append(torch.zeros_like(opt._norms))
            fused.dp_reduce_norms_(grads, 2, 0.5, g_out, flat.data, chunks[r], hp, norms[r])
        for r in (0, 1):
            fused.dp_lars_apply_(params, 2, r, g_out, mu, chunks[r], hp, norms[0] + norms[1])
    else:
        vals = [[g["lr"], *g["betas"], g["eps"], g["weight_decay"], 1 - g["betas"][0], 1 - g["betas"][1]] for g in opt._groups]
        hp = torch.tensor([vals[i % groups] for i in range(len(ps))], device=DEV) if rows else opt._hyper_of(vals)
        m, v = torch.zeros_like(flat.grad), torch.zeros_like(flat.grad)
        for r in (0, 1):
            fused.dp_adamw_step_(grads, params, 2, r, 0.5, m, v, chunks[r], hp)
    assert torch.equal(flat.data, data2)
    _same(ps, ref, 1)
