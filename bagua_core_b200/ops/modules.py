"""Whether a model may do a module's work itself instead of calling the module."""
from __future__ import annotations

import torch.nn as nn
from torch.nn.modules import module as _module

_GLOBAL_HOOKS = (_module._global_forward_hooks, _module._global_forward_pre_hooks, _module._global_backward_hooks,
                 _module._global_backward_pre_hooks)


def untouched(m, cls: type) -> bool:
    """`m` is a `cls`, and calling it does what `cls.forward` does: no hook waits for the call (its own or a global one), it
    was not replaced, wrapped or parametrised (which gives it another class), and has no `forward` of its own.
    (Asked a dozen times in a small model's step, so through the instance's dictionary.)"""
    if type(m) is not cls:
        return False
    d = m.__dict__
    g = _GLOBAL_HOOKS
    return not (d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"]
                or "forward" in d or g[0] or g[1] or g[2] or g[3])


def plain_embedding(m) -> bool:
    """An untouched table whose rows are looked up and whose gradient is the plain sum."""
    return (untouched(m, nn.Embedding) and m.padding_idx is None and m.max_norm is None and not m.scale_grad_by_freq
            and not m.sparse)


def drops_nothing(m) -> bool:
    """An untouched `nn.Dropout` that hands its input on."""
    return untouched(m, nn.Dropout) and (m.p == 0.0 or not m.training)
