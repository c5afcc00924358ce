"""The native host layer (lib/_torch_ops.so, from csrc/torch_*.cpp): the operators over torch tensors with autograd nodes
in C++.  Prebuilt in-tree like the CUDA library; importing fails loudly when it is missing."""
from __future__ import annotations

import importlib.machinery
import importlib.util
import os
import sys

from . import _lib

PATH = os.path.join(os.path.dirname(os.path.abspath(__file__)), "lib", "_torch_ops.so")


def _load():
    if not os.path.exists(PATH):
        raise ImportError(f"{PATH} is missing: build it first with `python tango_b200/build.py`")
    import torch  # noqa: F401  (its libraries have to be loaded before the extension)
    loader = importlib.machinery.ExtensionFileLoader("_torch_ops", PATH)
    module = importlib.util.module_from_spec(importlib.util.spec_from_file_location("_torch_ops", PATH, loader=loader))
    # the extension names its exception class by the package it belongs to, under whatever name that was imported
    sys.modules.setdefault("tango_b200._lib", _lib)
    loader.exec_module(module)
    return module


ops = _load()


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


def graph(g):
    """The host layer's view of a graph object, built once and kept on it; built anew when the object's index bundles
    or hub regions are other objects than the ones it was built from."""
    csc, csr = g.adj_csc, g.adj_csr
    hubs = getattr(g, "_hubs", None)
    hub_csc, hub_csr = (hubs.get("csc"), hubs.get("csr")) if hubs else (None, None)
    kept = getattr(g, "_native", None)
    if kept is not None and kept[0] is csc and kept[1] is csr and kept[2] is hub_csc and kept[3] is hub_csr:
        return kept[4]
    src, dst = g.coo
    handle = ops.Graph(_direction(g, "csc", hub_csc), _direction(g, "csr", hub_csr), src, dst, g.num_nodes())
    try:
        g._native = (csc, csr, hub_csc, hub_csr, handle)
    except AttributeError:       # an object without room for it: rebuilt on every call
        pass
    return handle
