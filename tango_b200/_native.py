"""The native host layer (lib/_torch_ops.so, from csrc/torch_*.cpp): the operators over torch tensors with autograd nodes
in C++.  Prebuilt in-tree like the CUDA library, for one version of torch with CUDA.  It is loaded when the first operator is
called, so that graphs, partitions and settings can be used where it cannot be (a CPU build of torch); an operator there, or
with a build that is missing or belongs to another torch, raises ImportError."""
from __future__ import annotations

import importlib.machinery
import importlib.util
import os
import sys

import torch
from torch.autograd.function import Function, once_differentiable

from . import _lib, build

PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "lib", "_torch_ops.so")


def _load():
    if not os.path.exists(PATH):
        raise ImportError(f"{PATH} is missing: build it first with `python tango_b200/build.py`")
    built, here = build.built_tag(), build.host_tag()
    if built not in ("", here):
        raise ImportError(f"{PATH} was built for {built}, not for {here}: build it anew with `python tango_b200/build.py`")
    loader = importlib.machinery.ExtensionFileLoader("_torch_ops", PATH)
    module = importlib.util.module_from_spec(importlib.util.spec_from_file_location("_torch_ops", PATH, loader=loader))
    # the extension names its exception class by the package it belongs to, under whatever name that was imported
    sys.modules.setdefault("tango_b200._lib", _lib)
    loader.exec_module(module)
    return module


class _NotLoaded:
    """Takes the place of the extension until something of it is asked for."""

    def __getattr__(self, name):
        return getattr(load(), name)


ops = _NotLoaded()
_settings = {}        # setter of the extension -> its arguments, for settings made before it is loaded


def load():
    """The extension; raises ImportError where it cannot be loaded."""
    global ops
    if isinstance(ops, _NotLoaded):
        module = _load()
        for name, args in _settings.items():
            getattr(module, name)(*args)
        ops = module
    return ops


def setting(name, *args) -> None:
    """ops.<name>(*args) for a setter, now or when the extension is loaded."""
    _settings[name] = args
    if not isinstance(ops, _NotLoaded):
        getattr(ops, name)(*args)


def transformed() -> bool:
    """True under tracing, forward-mode differentiation or a functorch transform."""
    return (torch._C._get_tracing_state() is not None or torch.autograd.forward_ad._current_level >= 0
            or torch._C._are_functorch_transforms_active())


class _Opaque(Function):
    """An operator as a Python autograd Function around its native node.  Tracing, forward mode and the functorch
    transforms know only what passes through the dispatcher or a Function: a call to the extension would leave a constant in
    the trace and drop a tangent without a word.  Through a Function it is recorded, or refused with an error."""

    @staticmethod
    def forward(ctx, op, *args):
        leaf = {id(a): a.detach().requires_grad_(a.requires_grad) for a in args if isinstance(a, torch.Tensor)}
        ctx.args = [leaf.get(id(a), a) for a in args]      # one tensor given twice stays one
        with torch.enable_grad():
            out = op(*ctx.args)
        single = not isinstance(out, tuple)
        ctx.outs = (out,) if single else out
        res = [o.detach() if isinstance(o, torch.Tensor) else o for o in ctx.outs]
        ctx.mark_non_differentiable(*[r for r, o in zip(res, ctx.outs) if isinstance(o, torch.Tensor) and not o.requires_grad])
        return res[0] if single else tuple(res)

    @staticmethod
    @once_differentiable
    def backward(ctx, *grads):
        outs = [(o, g) for o, g in zip(ctx.outs, grads) if isinstance(o, torch.Tensor) and o.requires_grad and g is not None]
        leaf = {id(a): a for a in ctx.args if isinstance(a, torch.Tensor) and a.requires_grad}
        found = torch.autograd.grad([o for o, _ in outs], list(leaf.values()), [g for _, g in outs], retain_graph=True,
                                    allow_unused=True) if outs and leaf else ()
        grad = dict(zip(leaf, found))
        return (None, *(grad.pop(id(a), None) for a in ctx.args))      # the first of two places takes the whole gradient


def call(op, *args):
    """op(*args) for an operator of `ops` whose tensors are differentiable."""
    return _Opaque.apply(op, *args) if transformed() else op(*args)


class LaunchCounter:
    """`counter[0]`: kernels of this library launched so far (benchmarks report it per step)."""

    def __getitem__(self, _):
        return ops.launches()

    def __setitem__(self, _, value):
        ops.set_launches(int(value))


def _direction(g, fmt: str, hub):
    indptr, indices, edge_ids = g.adj_csr if fmt == "csr" else g.adj_csc
    ident = getattr(g, "_identity", None)
    if ident is not None and ident.get(fmt, False):
        edge_ids = None          # slot k holds edge k: the kernels skip the indirection
    plans = getattr(g, "_plans", None)
    sched = None
    if plans is not None:
        if fmt not in plans:
            from .graph import SpmmSchedule
            plans[fmt] = SpmmSchedule(indptr)
        sched = plans[fmt]
    return ops.Direction((indptr, indices, edge_ids), sched, hub)


class _Kept:
    """The view of a graph that is kept on the graph object, and the objects it was built from.  A copied or unpickled graph
    gets an empty one."""
    __slots__ = ("made_from", "handle")

    def __init__(self, made_from=None, handle=None):
        self.made_from, self.handle = made_from, handle

    def __reduce__(self):
        return _Kept, ()


def graph(g):
    """The host layer's view of a graph object, built once and kept on it; built anew when the object's index bundles
    or hub regions are other objects than the ones it was built from."""
    csc, csr = g.adj_csc, g.adj_csr
    hubs = getattr(g, "_hubs", None)
    hub_csc, hub_csr = (hubs.get("csc"), hubs.get("csr")) if hubs else (None, None)
    made_from = (csc, csr, hub_csc, hub_csr)
    kept = getattr(g, "_native", None)
    if isinstance(kept, _Kept) and kept.made_from is not None and all(a is b for a, b in zip(kept.made_from, made_from)):
        return kept.handle
    src, dst = g.coo
    handle = ops.Graph(_direction(g, "csc", hub_csc), _direction(g, "csr", hub_csr), src, dst, g.num_nodes())
    try:
        g._native = _Kept(made_from, handle)
    except AttributeError:       # an object without room for it: rebuilt on every call
        pass
    return handle
