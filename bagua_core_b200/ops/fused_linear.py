"""`nn.Linear` that reads its weight from the optimizer's bf16 copy.

Drop-in for `nn.Linear`: unless the call is inside a bf16 autocast region and either an optimizer
maintains a bf16 copy of the weight (`bagua_core_b200.ops.shadow`) or in-place weight-gradient
accumulation is switched on (`bagua_core_b200.ops.wgrad`), it is `nn.Linear`.
Otherwise forward and backward run the same
three GEMMs as the framework's own bf16 linear layer — y = x Wᵀ + b, dx = dy W, dW = dyᵀ x, library
calls — but on the optimizer's copy of W instead of a fresh cast of the fp32 master weight (for
VGG-16's first classifier layer alone that cast moves 0.6 GB per step), and, with `wgrad.enabled`,
with the dW GEMM adding its product straight into the fp32 `weight.grad` instead of handing a bf16
matrix to autograd for a cast and a separate accumulation.  The bias gradient is this package's column
sum.  The autograd function is native (`csrc/trainer/autograd_ops.cc`).
"""
from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

from .._native import C as _C
from . import shadow as _shadow
from . import wgrad as _wgrad


_ACTIVATIONS = {"gelu": (1, F.gelu), "relu": (2, F.relu)}


class ShadowLinear(nn.Linear):
    # False: the weight gradient goes through autograd, rounded to bf16 as `nn.Linear`'s, whatever `wgrad.enabled` says
    accumulate_in_place = True

    def forward(self, x: torch.Tensor, activation: str = "") -> torch.Tensor:
        """`activation` ("gelu", "relu"): applied to the result, in the same autograd function where the layer runs
        natively."""
        code, act = _ACTIVATIONS[activation] if activation else (0, None)
        dev = x.device.type
        managed = getattr(self.weight, "_bagua_bf16", None) is not None  # an optimizer keeps a bf16 copy
        if ((managed or _wgrad.enabled) and torch.is_autocast_enabled(dev)
                and torch.get_autocast_dtype(dev) == torch.bfloat16):
            # the copy when it is current, a fresh cast otherwise: the same code path either way
            if code and _C.activation_fusable(x, self.out_features):
                act = None
            else:
                code = 0
            y = _C.linear(x, self.weight, self.bias, _shadow.autocast_copy(self.weight),
                          self.accumulate_in_place and _wgrad.active(), code)
        else:
            y = super().forward(x)
        return y if act is None else act(y)
