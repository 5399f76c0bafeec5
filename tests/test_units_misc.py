"""Host-side units: run log and throughput meter, message layout of the peer links, wire forms of channels-last
tensors, key chunking of the fused contrastive loss, parameter routes of a momentum teacher in split placement."""
import pytest
import torch
from torch import nn


def test_throughput_meter_overall_and_recent():
    from tspipe_b200.run_log import ThroughputMeter
    m = ThroughputMeter(window=3)
    assert m.overall() == 0.0 and m.recent() == 0.0
    for i in range(6):
        m.add(100, now=10.0 + i)           # one batch of 100 samples per second
    assert m.samples == 600 and m.batches == 6
    assert m.overall(now=16.0) == pytest.approx(100.0)
    assert m.recent() == pytest.approx(100.0)
    m.add(400, now=16.0)                   # a burst shows in the window, less in the overall rate
    assert m.recent() > m.overall(now=16.0)


def test_run_log_writes_scalars_and_model(tmp_path):
    from tspipe_b200.run_log import RunLog, join_partitions

    class FakePipe:
        def state_dicts(self):
            return ({0: {"a.weight": torch.ones(2)}, 1: {"b.weight": torch.zeros(3)}}, {0: {"a.weight": torch.ones(2) * 2}})
    lin = nn.Linear(2, 2)
    opt = torch.optim.SGD(lin.parameters(), lr=0.1)
    log = RunLog(str(tmp_path), tensorboard=False)
    log.scalar("loss", 1.5, 1)
    log.scalar("loss", 1.25, 2)
    path = log.save_final(FakePipe(), opt)
    log.close()
    rows = (tmp_path / "scalars.csv").read_text().splitlines()
    assert rows[0] == "wall_time,step,tag,value" and rows[1].endswith(",1,loss,1.5") and len(rows) == 3
    sd = torch.load(path, weights_only=False)
    assert list(sd["online_network_state_dict"]) == ["a.weight", "b.weight"]
    assert torch.equal(sd["target_network_state_dict"]["a.weight"], torch.full((2,), 2.0))
    assert "param_groups" in sd["optimizer_state_dict"]
    with pytest.raises(KeyError):
        join_partitions({0: {"k": torch.ones(1)}, 1: {"k": torch.ones(1)}})
    off = RunLog(str(tmp_path / "none"), enabled=False)
    off.scalar("loss", 1.0, 1)
    assert off.save_final(FakePipe(), opt) is None and not (tmp_path / "none").exists()


def test_peer_link_message_layout_is_aligned_and_ordered():
    from tspipe_b200.comm.peer_link import _layout, _nbytes
    specs = [((3, 5), torch.bfloat16), ((), torch.float32), ((7,), torch.int64), ((0, 4), torch.float32)]
    offs, need = _layout(specs)
    assert all(o % 256 == 0 for o in offs) and need % 256 == 0
    for (shape, dtype), a, b in zip(specs, offs, offs[1:] + [need]):
        assert b - a >= _nbytes(shape, dtype)
    assert _layout([]) == ([], 256)


@pytest.mark.parametrize("channels_last", [False, True])
def test_wire_form_round_trip(channels_last):
    from tspipe_b200.comm.links import wire_empty, wire_form
    x = torch.randn(2, 6, 3, 5).contiguous(memory_format=torch.channels_last)
    w = wire_form(x, channels_last)
    assert w.is_contiguous()
    if channels_last:
        assert w.data_ptr() == x.data_ptr() and w.shape == (2, 3, 5, 6)          # a view, no transpose
    buf, t = wire_empty(tuple(x.shape), x.dtype, None, channels_last)
    buf.copy_(w)
    assert t.shape == x.shape and torch.equal(t, x)
    assert t.is_contiguous(memory_format=torch.channels_last) == channels_last or not channels_last
    v = torch.randn(4, 9)
    assert wire_form(v, channels_last) is v


def test_contrastive_loss_key_chunks():
    from tspipe_b200.ops import gemm
    assert gemm.nce_key_chunks(4096, 4096) == 4            # 32 query tiles x 4 chunks = 128 CTAs
    assert gemm.nce_key_chunks(128, 128) == 1              # one key tile pair cannot be split
    assert gemm.nce_key_chunks(4096, 4160) == 1            # keys do not divide into 128-row chunks
    for n, nk in [(512, 4096), (1024, 1024), (256, 256), (8192, 8192)]:
        c = gemm.nce_key_chunks(n, nk)
        assert c >= 1 and nk % c == 0 and (c == 1 or (nk // c) % 64 == 0 and nk // c >= 128)
    gemm.set_nce_key_split(False)
    try:
        assert gemm.nce_key_chunks(4096, 4096) == 1
    finally:
        gemm.set_nce_key_split(True)


@pytest.mark.parametrize("cut_on,cut_tg", [([2, 2, 1], [3, 1]), ([5], [2, 2]), ([1, 4], [4])])
def test_split_placement_routes_cover_every_teacher_parameter_once(cut_on, cut_tg):
    from tspipe_b200.runtime.ema_plan import build_ema_plans, layout_offsets, split_placement_routes
    torch.manual_seed(0)
    layers = [nn.Linear(8, 8) for _ in range(4)]
    student = layers + [nn.Linear(8, 3)]                    # the last student layer has no teacher counterpart
    teacher = [nn.Linear(8, 8) for _ in range(4)]

    def cut(mods, sizes):
        out, i = [], 0
        for s in sizes:
            out.append(nn.Sequential(*mods[i:i + s]))
            i += s
        return out
    parts_on, parts_tg = cut(student, cut_on), cut(teacher, cut_tg)
    sources, dests = split_placement_routes(build_ema_plans(parts_on, parts_tg), len(parts_tg), len(parts_on))
    flat_s = []
    for part in parts_on:                                   # flat student buffers as the runtime lays them out
        ps = list(part.parameters())
        offs = layout_offsets(ps)
        buf = torch.zeros((offs[-1] + ps[-1].numel() + 63) // 64 * 64 if ps else 64)
        for p, o in zip(ps, offs):
            buf[o:o + p.numel()] = p.detach().reshape(-1)
        flat_s.append(buf)
    want = [p for l in layers for p in l.parameters()]     # teacher parameter i <-> student parameter i
    i = 0
    for jt, part in enumerate(parts_tg):
        ps = list(part.parameters())
        offs = layout_offsets(ps)
        got = torch.full(((offs[-1] + ps[-1].numel() + 63) // 64 * 64,), float("nan"))
        for js, runs in sources[jt].items():
            packed = torch.cat([flat_s[js][o:o + n] for o, n in dests[js][jt]])      # what the student rank sends
            pos = 0
            for t_off, _, n in runs:
                got[t_off:t_off + n] = packed[pos:pos + n]
                pos += n
            assert pos == packed.numel()
        for p, o in zip(ps, offs):
            assert torch.equal(got[o:o + p.numel()], want[i].detach().reshape(-1))
            i += 1
    assert i == len(want)


def test_bench_cuts_and_grids_are_consistent():
    """The benchmark's ResNet-50 cuts cover the 30 student / 26 teacher children, cut both networks at the same
    children (so that the momentum update stays local to a stage), and its pipelined grids use every GPU."""
    import itertools
    import os
    import sys
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    import bench
    from tspipe_b200.models.resnet import byol_networks
    online, target, predictor = byol_networks("resnet50", 64, 32)
    n_on, n_tg = len(online) + len(predictor), len(target)
    for pp, (on, tg) in bench.BYOL_SPLITS.items():
        assert len(on) == len(tg) == pp and sum(on) == n_on and sum(tg) == n_tg and min(on + tg) >= 1
        assert list(itertools.accumulate(on))[:-1] == list(itertools.accumulate(tg))[:-1]
        assert on[0] >= 4                      # conv1, bn1, relu, maxpool stay together (they run as one fused stem)
    for world in (1, 2, 4, 8):
        for pp, dp, ub in bench.pipeline_grids(world, "byol"):
            assert pp * dp == world and pp in bench.BYOL_SPLITS and (128 * world // dp) % ub == 0
    assert bench.pipeline_grids(8, "moco") == []


def test_hooks_on_all_modules_see_the_norms_of_a_block_and_the_pooling_of_a_stem():
    """A hook registered for every module (a profiler's, a module tracker's) is called for the modules whose work a fused pass
    would otherwise take over."""
    import torch
    from torch.nn.modules.module import register_module_forward_hook
    from tspipe_b200.models.vit import Block, LayerNorm, ViTConfig
    from tspipe_b200.ops.pool import MaxPool3x3s2
    from tspipe_b200.runtime.fuse import has_hooks
    blk, x, seen = Block(ViTConfig(embed_dim=64, num_heads=2)), torch.randn(2, 5, 64), []
    ref = blk(x)
    handle = register_module_forward_hook(lambda m, args, out: seen.append(m))
    try:
        assert torch.equal(blk(x), ref)
        assert has_hooks(MaxPool3x3s2())
    finally:
        handle.remove()
    assert [m for m in seen if isinstance(m, LayerNorm)] == [blk.norm1, blk.norm2]
    assert not has_hooks(MaxPool3x3s2())


def test_hyperparameters_of_a_launch():
    """A code per segment (group and whether the trust ratio applies), the groups' values by value; only a change rewrites
    them; more groups than travel by value go through a table."""
    import torch
    from torch import nn
    from tspipe_b200.ops import fused
    from tspipe_b200.optim import LARS
    from tspipe_b200.runtime.state import FlatParams
    for n in (2, 33):
        ps = [nn.Parameter(torch.randn(4, 3) if i % 2 else torch.randn(5)) for i in range(2 * n)]
        opt = LARS([dict(params=ps[i::n], lr=0.5 + i) for i in range(n)], weight_decay=0.25)
        flat = FlatParams(ps, torch.device("cpu"), with_grad=True)
        opt.bind_flat(flat, use_kernel=True)
        assert opt._codes.tolist() == [(i % n) << 1 | i % 2 for i in range(2 * n)]
        rows = [[g["lr"], g["weight_decay"]] for g in opt._groups]
        if n <= fused.Hyper.GROUPS:
            h = opt._hyper_of(rows)
            assert not h.table and h.by_value[8:10] == [1.5, 0.25]
            h.by_value[8] = 7.0
            assert opt._hyper_of([list(r) for r in rows]).by_value[8] == 7.0         # unchanged: not written again
            assert opt._hyper_of([[2.5, 0.0], [3.5, 1.0]]).by_value[8] == 3.5
        else:
            assert opt._hyper_of(rows).table == opt._hyper_table.data_ptr()
            assert opt._hyper_table[32, :2].tolist() == [32.5, 0.25]


def test_learning_rate_set_after_loading_a_state_is_used():
    """Loading replaces the optimizer's group dicts; a step on the flat buffers reads the new ones."""
    import torch
    from torch import nn
    from tspipe_b200.optim import SGD
    from tspipe_b200.runtime.state import FlatParams
    ps = [nn.Parameter(torch.ones(5)), nn.Parameter(torch.ones(3))]
    opt = SGD([dict(params=ps[:1]), dict(params=ps[1:], lr=0.5)], lr=0.25)
    opt.bind_flat(FlatParams(ps, torch.device("cpu"), with_grad=True), use_kernel=False)
    opt.load_state_dict(opt.state_dict())
    opt.param_groups[0]["lr"] = 0.125
    for p in ps:
        p.grad.fill_(1.0)
    opt.step()
    assert torch.equal(ps[0].detach(), torch.full((5,), 0.875)) and torch.equal(ps[1].detach(), torch.full((3,), 0.5))
    assert [g is h for g, h in zip(opt._groups, opt.param_groups)] == [True, True]


@pytest.mark.parametrize("lag", [0, 3, 50, 10_000])
def test_lars_order_updates_after_the_norms_of_the_whole_tensor(lag):
    """Every chunk's norms and update once each, an update after all norms of its tensor (the wait in the kernel ends by this
    order alone) and no earlier than ``lag`` chunks after its own."""
    from tspipe_b200.ops import fused
    numels = [5, 3 * fused.CHUNK, 100 * fused.CHUNK + 1, 64, 7 * fused.CHUNK - 1]
    offsets = [sum((n + 63) // 64 * 64 for n in numels[:i]) for i in range(len(numels))]
    chunks = fused.build_chunks(offsets, numels, "cpu").tolist()
    rows, need = fused.LarsOrder.plan(chunks, len(numels), lag)
    assert need == [-(-n // fused.CHUNK) for n in numels] and len(rows) == 2 * len(chunks)
    at = [{}, {}]
    for pos, (word, begin) in enumerate(rows):
        seg, update, length = (word & 0xFFFFFFFF) >> 1, word & 1, word >> 32
        assert begin not in at[update]
        at[update][begin] = (pos, seg, length)
    norms = [p for p, _, _ in sorted(at[0].values())]
    for seg, begin, length in chunks:
        assert at[0][begin][1:] == at[1][begin][1:] == (seg, length)
        pos = at[1][begin][0]
        assert pos > max(p for p, s, _ in at[0].values() if s == seg)
        mine = norms.index(at[0][begin][0])
        assert pos > norms[min(mine + lag, len(norms) - 1)]


def test_in_place_setting_loads_nothing_and_reaches_the_extension(monkeypatch):
    """The setting is kept for an extension that is loaded later, and passed on to one that is there."""
    from tspipe_b200.ops import build, conv, fused

    class Host:
        seen = []

        def set_accumulate(self, on):
            self.seen.append(on)

    def unavailable():
        raise RuntimeError("no compiler")
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(build, "load", unavailable)
    monkeypatch.setattr(build, "load_host", unavailable)
    monkeypatch.setattr(fused, "_host", None)
    try:
        conv.set_accumulate_in_place(False)
        monkeypatch.setattr(build, "load_host", Host)
        monkeypatch.setattr(fused, "lib", lambda: None)
        assert isinstance(fused.eager(), Host) and Host.seen == [False]
        conv.set_accumulate_in_place(True)
        assert Host.seen == [False, True]
    finally:
        conv.set_accumulate_in_place(True)


@pytest.mark.parametrize("left", ["nothing", "a stale module", "a compiler that fails"])
def test_eager_calls_go_on_without_the_extension(monkeypatch, tmp_path, left):
    """Without a module that fits, or a compiler, the Python functions take the calls, which is said once."""
    import subprocess
    import warnings

    from tspipe_b200.ops import build, fused
    path = tmp_path / "tspipe_eager.so"
    if left == "a stale module":
        path.write_bytes(b"of another torch")
        (tmp_path / "tspipe_eager.so.srchash").write_text("0")
    monkeypatch.setattr(build, "HOST_PATH", str(path))
    monkeypatch.setattr(build, "load", lambda: None)
    monkeypatch.setattr(build, "build", lambda: None)
    monkeypatch.setattr(build, "_host", None)
    monkeypatch.setattr(build, "_no_host", False, raising=False)
    monkeypatch.setattr(build.shutil, "which", lambda name: None if left != "a compiler that fails" else name)
    monkeypatch.setattr(build.subprocess, "run", lambda cmd, **k: subprocess.CompletedProcess(cmd, 1, "", "no header"))
    monkeypatch.setattr(fused, "_host", None)
    monkeypatch.setattr(fused, "lib", lambda: None)
    with pytest.warns(RuntimeWarning, match="Python functions"):
        assert fused.eager() is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert fused.eager() is None
