"""Quantized edge-score operators: the autograd surface of the reference's cuda/SDDMM.py, plus `sddmm_u_dot_v`,
which the reference's HGT and link-prediction scripts call (evaluation/test_HGT.py:58) but never define.  Native, as in
SPMM.py."""
from __future__ import annotations

from . import _native
from .kernels import *  # noqa: F401,F403  (the reference's module re-exports its kernels the same way)


class sddmm_u_add_v:
    """e[k] = U[src(k)] + V[dst(k)] on int8 operands (cuda/SDDMM.py:10-32); the gradients are the sums of dZ over
    the out-edges (dU) and in-edges (dV) of each node."""

    @staticmethod
    def apply(g, U, V, scaleU_=None, scaleV_=None):
        return _native.call(_native.ops.sddmm_u_add_v, _native.graph(g), U, V, scaleU_, scaleV_)


class sddmm_u_dot_v:
    """e[k,h] = <U[src(k),h,:], V[dst(k),h,:]> on int8 operands.  Backward: dU[u] = sum over out-edges of
    dZ[k] * V[dst(k)], dV[v] = sum over in-edges of dZ[k] * U[src(k)], both as int8 weighted SpMMs."""

    @staticmethod
    def apply(g, U, V):
        return _native.call(_native.ops.sddmm_u_dot_v, _native.graph(g), U, V)
