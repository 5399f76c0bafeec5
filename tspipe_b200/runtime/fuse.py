"""Peephole fusion of a stage partition's children.

A partition is an ``nn.Sequential`` whose child granularity is part of the user-facing contract
(``model_split`` counts children, checkpoints are keyed by child names), so the modules stay as they
are; only the way the partition *runs* them changes.  :class:`FusedSequential` executes the same
children in order but lets neighbouring ones share a kernel:

* ``BatchNorm -> ReLU``                      one fused normalise + activation pass (``ops.bn.bn_act``);
* ``Conv2d(3, 64, 7, stride 2) -> BatchNorm`` the tcgen05 stem convolution, whose epilogue already produces the
  BatchNorm statistics (``ops.conv.stem_conv``), so the statistics pass over the activation disappears;
* that stem convolution's ``BatchNorm -> ReLU -> MaxPool 3x3/2`` one pass forward and two backward
  (``ops.bn.bn_relu_pool``): the normalised activation is never written;
* ``Linear`` children (the MLP heads)        the tcgen05 GEMM path of ``ops.linear.linear``, forward and backward.

The reference runs these layers one library call at a time
(`benchmarks/byol/models/resnet_base_network.py`, `tspipe/tspipe.py:553-580` for the child granularity).
"""
from __future__ import annotations

from typing import Any, List

import torch
from torch import nn
from torch.nn.modules.batchnorm import _BatchNorm
from torch.nn.modules.module import _has_any_global_hook


def has_hooks(m: nn.Module) -> bool:
    """Whether something watches calls of ``m``: hooks of its own, or ones on all modules (profilers, module trackers)."""
    return bool(m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks
                or _has_any_global_hook())


class FusedSequential(nn.Sequential):
    """Same children, same parameters and state-dict keys as the ``nn.Sequential`` it replaces."""

    def forward(self, x: Any) -> Any:  # type: ignore[override]
        from ..ops import bn as _bn
        from ..ops import conv as _conv
        from ..ops import linear as _linear
        from ..ops.pool import MaxPool3x3s2
        mods: List[nn.Module] = list(self._modules.values())
        i, n = 0, len(mods)
        while i < n:
            m = mods[i]
            nxt = mods[i + 1] if i + 1 < n else None
            if _conv.is_stem_conv(m) and _conv.eligible(x) and torch.is_autocast_enabled():
                bn_next = isinstance(nxt, _BatchNorm) and nxt.training
                segs = _bn.current_segments() if x.shape[0] % _bn.current_segments() == 0 else 1
                bn_next = bn_next and (segs == _bn.current_segments())
                y, sums = _conv.stem_conv(x, m.weight, want_sums=bn_next, segments=segs)
                if bn_next and _bn.applicable(nxt, y):
                    relu = i + 2 < n and isinstance(mods[i + 2], nn.ReLU)
                    if relu and i + 3 < n and type(mods[i + 3]) is MaxPool3x3s2 and not has_hooks(mods[i + 3]):
                        z = _bn.bn_relu_pool(nxt, y, sums=sums)
                        if z is not None:
                            x, i = z, i + 4
                            continue
                    x = _bn.bn_act(nxt, y, relu=relu, sums=sums)
                    i += 3 if relu else 2
                else:
                    x = y
                    i += 1
                continue
            if isinstance(m, _BatchNorm) and isinstance(nxt, nn.ReLU) and isinstance(x, torch.Tensor) \
                    and _bn.applicable(m, x):
                x = _bn.bn_act(m, x, relu=True)
                i += 2
                continue
            if type(m) is nn.Linear and isinstance(x, torch.Tensor):
                x = _linear.linear(x, m.weight, m.bias)
                i += 1
                continue
            x = m(x)
            i += 1
        return x


def fuse_partition(module: nn.Module) -> nn.Module:
    """Switch a plain ``nn.Sequential`` partition to fused execution (in place; no-op for anything else)."""
    if type(module) is nn.Sequential:
        module.__class__ = FusedSequential
    return module
