"""What the launches of a stage under recording share, and where they take other ways than eager ones."""
import threading

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
