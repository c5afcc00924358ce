"""Quantized aggregation operators: the autograd surface of the reference's cuda/SPMM.py.  The operators and their
autograd nodes are native (csrc/torch_autograd.cpp); `apply` has the arguments of the reference's Functions."""
from __future__ import annotations

from . import _native
from .kernels import *  # noqa: F401,F403  (the reference's module re-exports its kernels the same way)


class spmm_copy_u:
    """out[v] = sum of the int8-quantized features of v's in-neighbours (cuda/SPMM.py:8-24); the gradient is the same
    sum over the out-edges of the int8-quantized dZ."""

    @staticmethod
    def apply(g, N, scaleN=None):
        return _native.call(_native.ops.spmm_copy_u, _native.graph(g), N, scaleN)


class _WithScaleSwitch(type):
    """The class attribute `compat_dn_scale` is handed to the host layer, whose backward pass reads it."""

    _compat_dn_scale = False

    @property
    def compat_dn_scale(cls) -> bool:
        return cls._compat_dn_scale

    @compat_dn_scale.setter
    def compat_dn_scale(cls, value) -> None:
        _WithScaleSwitch._compat_dn_scale = bool(value)
        _native.setting("set_compat_dn_scale", bool(value))

    @compat_dn_scale.deleter
    def compat_dn_scale(cls) -> None:
        cls.compat_dn_scale = False


class spmm_u_mul_e(metaclass=_WithScaleSwitch):
    """out[v,h,:] = sum_e E[e,h] * N[src(e),h,:] with both operands int8 (cuda/SPMM.py:36-62).

    `spmm_u_mul_e.compat_dn_scale = True` reproduces the reference's backward, which scales dN with the forward product
    s(N)*s(E) (cuda/SPMM.py:52,56) instead of s(dZ)*s(E); the default uses the consistent scale.  What counts is its value
    when the backward pass runs."""

    @staticmethod
    def apply(g, N, E, scaleE_=None):
        return _native.call(_native.ops.spmm_u_mul_e, _native.graph(g), N, E, scaleE_)
