"""Whether a model may do a module's work itself instead of calling the module."""
from __future__ import annotations

import torch.nn as nn
from torch.nn.modules.module import _has_any_global_hook


def untouched(m: nn.Module, cls: type) -> bool:
    """`m` is a `cls`, and calling it does what `cls.forward` does: no hook waits for the call (its own or a global one), it
    was not replaced, wrapped or parametrised (which gives it another class), and has no `forward` of its own."""
    return (type(m) is cls and not m._forward_hooks and not m._forward_pre_hooks and not m._backward_hooks
            and not m._backward_pre_hooks and "forward" not in m.__dict__ and not _has_any_global_hook())


def plain_embedding(m: nn.Module) -> bool:
    """An untouched table whose rows are looked up and whose gradient is the plain sum."""
    return (untouched(m, nn.Embedding) and m.padding_idx is None and m.max_norm is None and not m.scale_grad_by_freq
            and not m.sparse)


def dropout(m: nn.Module, x):
    """`m(x)`, without the call where an untouched `nn.Dropout` drops nothing."""
    return x if untouched(m, nn.Dropout) and (m.p == 0.0 or not m.training) else m(x)
