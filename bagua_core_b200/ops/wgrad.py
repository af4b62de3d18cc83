"""Weight gradients accumulated by the GEMM that computes them.

Under bf16 autocast a linear layer's weight gradient takes three passes over memory: the GEMM
dW = dyᵀ x writes it in bf16, autograd casts it to the fp32 of the master weight, and the
accumulation step adds it to `weight.grad` (here a view of a flat gradient bucket).  That is 18
bytes of traffic per weight after the GEMM; for VGG-16, whose classifier holds 124 M of the model's
138 M parameters, about 2 GB per step.  The library GEMM can instead read and write the fp32
gradient itself (`C = A B + C` with bf16 A, B and fp32 C): 8 bytes per weight, no cast, no separate
accumulation, and the product is never rounded to bf16.

The native linear function (`csrc/trainer/autograd_ops.cc`) does that for a parameter whose `.grad` is an
fp32 tensor, and gives autograd no gradient for the weight, so autograd has nothing to cast or add; the
convolution blocks add their bf16 weight gradient to the fp32 one in one pass, and both add their bias
gradients with the kernel that reduces them.  The parameter's post-accumulate-grad hooks still run: autograd
runs them when it reaches the parameter even without a gradient.  The ordinary path is taken whenever the
shortcut would change what the user sees:

* the feature is off (`enabled`, default False), autograd turns out not to run the hooks of a parameter that got
  no gradient (`active`), or a higher-order graph is being built;
* the backward pass returns the gradient instead of accumulating it (`torch.autograd.grad`);
* `.grad` is missing, not fp32, not contiguous or of another shape;
* the parameter has tensor hooks (`register_hook`), which autograd would apply to the gradient;
* the same parameter takes part in the graph more than once: autograd would add the uses' gradients first
  and accumulate once, so all uses take the ordinary path.

Module attributes `accumulated` and `declined` count the weight gradients of linear layers that were added in
place and those that were not; `cuda_mode` says which library call accumulates on CUDA: "addmm" (one GEMM reads
and writes the fp32 gradient), "mm_add" (GEMM with fp32 output, then an in-place add), "off" (neither is
available) or None (no call yet).

Reference: the reference engine is told about finished gradients per tensor
(bagua-core-internal/src/lib.rs:300-319); how the trainer produces them is outside it.
"""
from __future__ import annotations

from typing import Optional

import torch

from .._native import C as _C

# Off by default.
enabled = False


def active() -> bool:
    """Whether gradients may be added in place: `enabled`, and a bucket would still learn of them."""
    return enabled and (_hooks_run_anyway or _autograd_runs_hooks_without_a_gradient())


def __getattr__(name):
    if name in ("accumulated", "declined"):
        return _C.op_stats()[name]
    if name == "cuda_mode":
        return _C.op_stats()["gemm_mode"] or None
    raise AttributeError(f"module {__name__!r} has no attribute {name!r}")


_hooks_run_anyway: Optional[bool] = None


def _autograd_runs_hooks_without_a_gradient() -> bool:
    """Whether autograd runs a parameter's post-accumulate-grad hooks when the backward of its only
    consumer returned None for it.  torch 2.11 does (the hooks then run when autograd reaches the
    parameter, once, however many uses it had), and in-place accumulation relies on it.
    Found out once, on a three-element graph on the host."""
    global _hooks_run_anyway
    if _hooks_run_anyway is None:
        fired = []

        class _Probe(torch.autograd.Function):
            @staticmethod
            def forward(ctx, x, w):
                return x * w.detach()

            @staticmethod
            def backward(ctx, dy):
                return dy, None

        try:
            with torch.inference_mode(False), torch.enable_grad():
                w = torch.nn.Parameter(torch.ones(3, device="cpu"))
                w.grad = torch.zeros(3, device="cpu")
                handle = w.register_post_accumulate_grad_hook(lambda p: fired.append(1))
                x = torch.ones(3, device="cpu", requires_grad=True)
                _Probe.apply(x, w).sum().backward()
                handle.remove()
        except RuntimeError:  # a transform of torch.func is looking on: not found out yet
            return False
        _hooks_run_anyway = bool(fired)
    return _hooks_run_anyway
