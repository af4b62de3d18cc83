"""Convolution block with the element-wise tail fused: conv → (bias + ReLU) in one in-place pass,
and in the backward one pass that applies the ReLU mask and reduces the bias gradient.

The convolution itself stays a library call (cuDNN through `at::convolution` /
`at::convolution_backward`), but for the weight gradient of 3 x 3 convolutions with bf16 parameters
(`csrc/kernels/conv_wgrad.cu`, where its rule takes it).  What the framework would run around it — a bias add, a clamp, a
ReLU-mask kernel and a separate column reduction for the bias gradient — is replaced by the
sm_100a kernels of `csrc/kernels/model_ops.cu`; the autograd functions are native
(`csrc/trainer/autograd_ops.cc`).  The fused path needs a block computed in bf16
(bf16 autocast on CUDA, or bf16 parameters and inputs); anything else takes the plain PyTorch
composition, so `ConvBiasReLU` is a drop-in for `Conv2d` followed by `ReLU`.  bf16 tensors on the
CPU run the same path against a host restatement of the kernels
(`csrc/kernels/model_ops_cpu.cc`), which is how the glue is tested without a GPU.
"""
from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

from .._native import C as _C
from . import shadow as _shadow
from . import wgrad as _wgrad


# Kernels launched so far in this process by the functions of this file and of `fused_linear`
# (benchmarks report it as `launches`).
_pool_launches = 0


def __getattr__(name):
    if name == "launches":
        return _pool_launches + _C.op_stats()["launches"]
    raise AttributeError(f"module {__name__!r} has no attribute {name!r}")


def _stream(t: torch.Tensor) -> int:
    return _C.current_stream(t)


def _count(n: int) -> None:
    global _pool_launches
    _pool_launches += n


class _ConvBiasReLUFn:
    """Runs in the autocast dtype where autocast is on (parameters stay fp32 outside; autograd
    casts the gradients back to the parameters' dtype).  With `wgrad.enabled` the backward adds the
    gradients of weight and bias to an fp32 `.grad` itself, with the bits autograd would produce."""

    @staticmethod
    def apply(x, weight, bias, stride, padding, dilation, groups):
        return _C.conv_bias_relu(x, weight, bias, stride, padding, dilation, groups, False,
                                 _shadow.autocast_copy(weight), _wgrad.active())


class _ConvBiasReLUPoolFn:
    """conv → bias + ReLU → 2x2 max pooling.  The full-resolution activation is never written: the
    backward, which produces the convolution's output gradient and the bias gradient in one pass,
    routes the gradient by four bits per pooled value that the forward leaves."""

    @staticmethod
    def apply(x, weight, bias, stride, padding, dilation, groups):
        return _C.conv_bias_relu(x, weight, bias, stride, padding, dilation, groups, True,
                                 _shadow.autocast_copy(weight), _wgrad.active())


class _MaxPool2x2Fn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        n, c, h, w = x.shape
        y = torch.empty((n, c, h // 2, w // 2), dtype=x.dtype, device=x.device, memory_format=torch.channels_last)
        _C.k_maxpool2x2_forward(x, y, _stream(x))
        _count(1)
        ctx.save_for_backward(x)
        return y

    @staticmethod
    def backward(ctx, dy):
        (x,) = ctx.saved_tensors
        dy = dy.contiguous(memory_format=torch.channels_last)
        dx = torch.empty_like(x, memory_format=torch.channels_last)
        _C.k_maxpool2x2_backward(x, dy, dx, _stream(x))
        _count(1)
        return dx


class MaxPool2x2(nn.Module):
    """`nn.MaxPool2d(2, 2)`.  Channels-last CUDA bf16 inputs with even height and width go through
    this package's kernels: no index tensor in the forward, and a backward that recomputes the
    arg-max and writes the whole input gradient in one pass (no zero-fill)."""

    def forward(self, x):
        if (x.dtype == torch.bfloat16 and x.dim() == 4
                and x.is_contiguous(memory_format=torch.channels_last)
                and _C.k_maxpool2x2_supported(x.shape[0], x.shape[2], x.shape[3], x.shape[1])):
            return _MaxPool2x2Fn.apply(x)
        return F.max_pool2d(x, 2, 2)


def _computes_in_bf16(x: torch.Tensor, weight: torch.Tensor) -> bool:
    if torch.is_autocast_enabled(x.device.type):
        return torch.get_autocast_dtype(x.device.type) == torch.bfloat16
    return x.dtype == torch.bfloat16 and weight.dtype == torch.bfloat16


class ConvBiasReLU(nn.Conv2d):
    """`nn.Conv2d` (with bias) followed by ReLU, with the same parameters and state dict as the
    convolution alone."""

    def forward(self, x):
        fusable = (self.bias is not None and not isinstance(self.padding, str) and self.padding_mode == "zeros"
                   and x.dim() == 4 and _computes_in_bf16(x, self.weight)
                   and _C.k_bias_relu_supported(1, self.out_channels))
        if not fusable:
            return F.relu(super().forward(x))
        return _ConvBiasReLUFn.apply(x, self.weight, self.bias, self.stride, self.padding, self.dilation,
                                     self.groups)


class ConvBiasReLUPool(nn.Conv2d):
    """`nn.Conv2d` (with bias) followed by ReLU and `MaxPool2d(2, 2)`, with the convolution's
    parameters and state dict.  On the fused path the pooling is folded into the bias + ReLU pass
    in both directions, so the full-resolution activation is read once on the way forward and its
    gradient is written once on the way back."""

    def forward(self, x):
        fusable = (self.bias is not None and not isinstance(self.padding, str) and self.padding_mode == "zeros"
                   and x.dim() == 4 and _computes_in_bf16(x, self.weight)
                   and _C.k_bias_relu_supported(1, self.out_channels))
        if fusable:
            # the convolution's output size decides whether the 2x2 windows tile it exactly
            h = (x.shape[2] + 2 * self.padding[0] - self.dilation[0] * (self.kernel_size[0] - 1) - 1) // self.stride[0] + 1
            w = (x.shape[3] + 2 * self.padding[1] - self.dilation[1] * (self.kernel_size[1] - 1) - 1) // self.stride[1] + 1
            fusable = _C.k_maxpool2x2_supported(x.shape[0], h, w, self.out_channels)
        if not fusable:
            return F.max_pool2d(F.relu(super().forward(x)), 2, 2)
        return _ConvBiasReLUPoolFn.apply(x, self.weight, self.bias, self.stride, self.padding,
                                         self.dilation, self.groups)
