"""Quantized linear layer: the autograd surface of the reference's cuda/QLinear.py (Qlinear_func,
Qlinear_func_reduce, QgemmNT_func, QLinear) on top of the tcgen05 int8 GEMMs."""
from __future__ import annotations

import torch
import torch.nn as nn
from torch.autograd.function import Function

from . import _native, config, kernels


# The few most recently quantized activations: (tensor kept alive so its address cannot be recycled, version, key,
# Xq, sX), newest last.  Four entries cover HGT's interleaved k / attn / v / msg / q projections.
_shared_input = []
_SHARED_SLOTS = 4


def clear_shared_input() -> None:
    _shared_input.clear()


def _input_key(X, mode):
    return (X.data_ptr(), tuple(X.shape), tuple(X.stride()), X.device, mode, config.seed())


def _linear(X, W, b, want_scale, copies=None):
    """Forward of cuda/QLinear.py:28-35,52-60 (absmax scales of X and W, quantize, GEMM, optional output scale) with its
    native autograd node, which keeps the quantized operands for the backward pass (cuda/QLinear.py:37-47,62-72: dY
    quantized to nearest, dX and dW by int8 GEMMs, bias gradient in fp32).  With config.share_quantized_inputs() a layer
    whose input is the tensor a previous layer just quantized (same memory, same version) re-uses that int8 copy.
    `copies` (a dict that the layers of one forward pass hand to each other) does the same for layers that are known to
    read the same X."""
    if copies is not None:
        Y, sY, copies["Xq"], copies["sX"] = _native.call(_native.ops.qlinear, X, W, b, want_scale, copies.get("Xq"),
                                                         copies.get("sX"))
        return (Y, sY) if want_scale else Y
    share = config.sharing_quantized_inputs() and config.mode_for("gemm_fwd") != kernels.ROUND_STOCHASTIC
    Xq = sX = None
    if share:
        key = _input_key(X, config.mode_for("gemm_fwd"))
        for ent in _shared_input:
            if ent[1] == X._version and ent[2] == key:
                Xq, sX = ent[3], ent[4]
    Y, sY, Xq_used, sX_used = _native.call(_native.ops.qlinear, X, W, b, want_scale, Xq, sX)
    if share and Xq is None:
        _shared_input.append((X, X._version, key, Xq_used, sX_used))
        del _shared_input[:-_SHARED_SLOTS]
    return (Y, sY) if want_scale else Y


class Qlinear_func:
    @staticmethod
    def apply(X, W, b=None):
        return _linear(X, W, b, False)


class Qlinear_func_reduce:
    """Also returns max|Y|/127 computed in the GEMM epilogue, so the consumer can skip its own absmax pass."""

    @staticmethod
    def apply(X, W, b=None):
        return _linear(X, W, b, True)


class QgemmNT_func(Function):
    """A . B^T with both operands quantized per call (cuda/QLinear.py:9-23, the reference's legacy cuBLAS path)."""

    @staticmethod
    def forward(ctx, A, B):
        ctx.save_for_backward(A, B)
        return kernels.cuda_kernels.QgemmNT(A, B)

    @staticmethod
    def backward(ctx, grad_output):
        A, B = ctx.saved_tensors
        gA = kernels.cuda_kernels.QgemmNN(grad_output, B) if ctx.needs_input_grad[0] else None
        gB = kernels.cuda_kernels.QgemmTN(grad_output, A) if ctx.needs_input_grad[1] else None
        return gA, gB


class QLinear(nn.Linear):
    """nn.Linear whose matmuls run as int8 GEMMs (cuda/QLinear.py:75-93).  The reference requires K % 4 == 0; any K
    is accepted here because the quantized operands are stored with rows padded to 16 bytes."""

    def __init__(self, in_features, out_features, bias=True):
        super().__init__(in_features, out_features, bias)
        self.isReduce = False

    def enable_reduce(self):
        self.isReduce = True

    def forward(self, input, copies=None):
        t = input.reshape(-1, input.size(-1))
        out_shape = input.shape[:-1] + (self.weight.size(0),)
        out = _linear(t, self.weight, self.bias, self.isReduce, copies)
        if self.isReduce:
            return out[0].reshape(out_shape), out[1]
        return out.reshape(out_shape)


def _hooked(m) -> bool:
    """True when calling the module does more than its forward: hooks that want to see its input and output."""
    own = (m._forward_hooks, m._forward_pre_hooks, m._backward_hooks, m._backward_pre_hooks)
    return any(own) or torch.nn.modules.module._has_any_global_hook() or "forward" in m.__dict__


def linear_group(layers, input):
    """Yields the outputs of up to three QLinear layers that read the same input, whose absmax pass and int8 copy they
    share; with config.share_quantized_inputs() the weights are quantized in the same launch as well.  Bit-identical to
    calling the layers one by one, which is what happens with stochastic rounding (every layer draws its own numbers, in
    the order in which the outputs are asked for)."""
    plain = not _native.transformed() and all(type(m) is QLinear and not m.isReduce and not _hooked(m) for m in layers)
    if not plain or config.mode_for("gemm_fwd") == kernels.ROUND_STOCHASTIC:
        yield from (m(input) for m in layers)
    elif config.sharing_quantized_inputs():
        out = _native.ops.qlinear_group(input.reshape(-1, input.size(-1)), [m.weight for m in layers],
                                        [m.bias for m in layers])
        yield from (y.reshape(input.shape[:-1] + (y.size(1),)) for y in out)
    else:
        copies = {}
        yield from (m(input, copies) for m in layers)
