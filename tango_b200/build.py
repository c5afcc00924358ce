"""Builds the sm_100a shared library in-tree (tango_b200/lib/libtango_b200.so) with nvcc.

nvcc cross-compiles without a GPU.  The explicit -gencode pair is required: tcgen05 kind::i8 only assembles for the
architecture-specific target compute_100a/sm_100a.  --fmad=false keeps every fp32 epilogue a sequence of single
IEEE operations so results are bit-reproducible against the CPU checker.

The host layer (csrc/torch_*.cpp -> lib/_torch_ops.so) is a Python extension over the torch C++ headers, compiled with
g++ and linked against the library above, which it finds beside itself.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from importlib import metadata
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
HEADER = os.path.join(ROOT, "include", "tango_b200.h")
CUDA_HOME = os.environ.get("CUDA_HOME") or "/usr/local/cuda"
LIB_PATH = os.path.join(LIB_DIR, "libtango_b200.so")
SOURCES = ["quantize.cu", "quantize_fused.cu", "spmm.cu", "sddmm.cu", "gat_softmax.cu", "gat_project.cu", "igemm_tcgen05.cu", "peer.cu"]
HOST_SOURCES = ["torch_ops.cpp", "torch_autograd.cpp", "torch_bind.cpp"]
HOST_LIB_PATH = os.path.join(LIB_DIR, "_torch_ops.so")
HOST_TAG_PATH = os.path.join(LIB_DIR, "_torch_ops.tag")     # what the host layer was built for
# measurement aid of the benchmark, a library of its own (not part of the product ABI)
PROBE_SRC = os.path.join(CSRC, "bench", "row_gather_probe.cu")
PROBE_LIB_PATH = os.path.join(LIB_DIR, "libtango_bench_probe.so")


def _nvcc() -> str:
    cand = os.environ.get("NVCC") or "/usr/local/cuda/bin/nvcc"
    return cand if os.path.exists(cand) else "nvcc"


def _newer(target: str, deps) -> bool:
    return not os.path.exists(target) or any(os.path.getmtime(d) > os.path.getmtime(target) for d in deps)


def _run(cmd, what: str):
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        sys.stderr.write(res.stdout + res.stderr)
        raise RuntimeError(f"{os.path.basename(cmd[0])} failed building {what}")
    return res


def _sources(*suffixes):
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(suffixes)] + [HEADER]


def host_tag() -> str:
    """The versions that the host layer depends on: it is compiled against torch's C++ headers for one interpreter."""
    return f"torch {metadata.version('torch')} {sysconfig.get_config_var('SOABI')}"


def built_tag() -> str:
    try:
        with open(HOST_TAG_PATH) as f:
            return f.read().strip()
    except OSError:
        return ""


def _host_outdated() -> bool:
    return built_tag() != host_tag() or _newer(HOST_LIB_PATH, _sources(".cpp", "torch_ops.h", "torch_autograd.h"))


def needs_build() -> bool:
    return _newer(LIB_PATH, _sources(".cu", ".cuh")) or _newer(PROBE_LIB_PATH, [PROBE_SRC]) or _host_outdated()


def _build_host() -> None:
    """g++ over the torch headers (no nvcc: the host layer holds no device code)."""
    from torch.utils.cpp_extension import include_paths, library_paths
    import torch
    if torch.version.cuda is None:
        sys.stderr.write("the host layer is not built: this torch has no CUDA (graphs and settings work, operators do not)\n")
        return
    flags = ["-O2", "-fPIC", "-std=c++17", "-fvisibility=hidden", "-DTORCH_API_INCLUDE_EXTENSION_H",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-I" + os.path.dirname(HEADER),
             "-I" + os.path.join(CUDA_HOME, "include"), "-I" + sysconfig.get_paths()["include"]]
    flags += ["-isystem" + p for p in include_paths()]
    objects = [os.path.join(LIB_DIR, os.path.splitext(s)[0] + ".o") for s in HOST_SOURCES]
    with ThreadPoolExecutor() as pool:
        list(pool.map(lambda so: _run(["g++", *flags, "-c", os.path.join(CSRC, so[0]), "-o", so[1]], so[0]),
                      zip(HOST_SOURCES, objects)))
    link = ["g++", "-shared", "-o", HOST_LIB_PATH, *objects, "-L" + LIB_DIR, "-ltango_b200", "-Wl,-rpath,$ORIGIN"]
    link += [f for p in library_paths() for f in ("-L" + p, "-Wl,-rpath," + p)]
    _run(link + ["-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-lc10", "-lc10_cuda"], "_torch_ops.so")
    for o in objects:
        os.remove(o)
    with open(HOST_TAG_PATH, "w") as f:
        f.write(host_tag() + "\n")


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(LIB_DIR, exist_ok=True)
    nvcc = [_nvcc(), "-shared", "-Xcompiler", "-fPIC", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3",
            "-std=c++17"]
    if force or _newer(LIB_PATH, _sources(".cu", ".cuh")):
        cmd = nvcc + ["--fmad=false", "-diag-suppress", "128", "-I", os.path.dirname(HEADER), "--threads", "0",
                      "-Xlinker", "-soname=libtango_b200.so", "-o", LIB_PATH] + [os.path.join(CSRC, s) for s in SOURCES]
        if verbose:
            cmd[1:1] = ["-Xptxas", "-v"]
        res = _run(cmd, "libtango_b200.so")
        if verbose:
            sys.stderr.write(res.stderr)
    if force or _newer(PROBE_LIB_PATH, [PROBE_SRC]):
        _run(nvcc + ["-o", PROBE_LIB_PATH, PROBE_SRC], "libtango_bench_probe.so")
    if force or _host_outdated():
        _build_host()
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
