"""Builds the C-ABI shared library (libb200moe.so) from csrc/ with nvcc for sm_100a.

    python -m llm_kernels_b200.build          # build if sources are newer than the library

The library lands next to this file (llm_kernels_b200/libb200moe.so) so it travels
with the source tree; there is no JIT cache and no install step.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libb200moe.so")
# Python module over the library and torch's C++ API (csrc/calls.cpp); belongs to one build of torch and one Python, which it names
CALLS = os.path.join(HERE, "_calls.so")
SOURCES = ["api.cu", "quant.cu", "router.cu", "route.cu", "permute.cu", "gemm_fp8.cu", "gemm_fp8_rows.cu", "gemm_w4a8.cu", "gemm_w4a16.cu", "bitpack.cu", "w4.cu", "wquant.cu", "ep_fused.cu", "layer.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put it on PATH")


def _older(target: str, names) -> bool:
    """target is missing or older than a source, the header or this file."""
    if not os.path.exists(target):
        return True
    deps = [os.path.join(CSRC, f) for f in names] + [os.path.join(HERE, "..", "include", "b200moe.h"), os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > os.path.getmtime(target) for d in deps)


def _library_sources():
    return [f for f in os.listdir(CSRC) if f != "calls.cpp"]


def calls_stamp() -> str:
    """The torch and the Python that the compiled calls must have been built for."""
    import torch
    return f"built for torch {torch.__version__}, {sys.implementation.cache_tag}"


def calls_fit() -> bool:
    """Whether the compiled calls are there and belong to this torch and this Python.  Looked up in the file: a module of another
    torch may not even load."""
    if not os.path.exists(CALLS):
        return False
    with open(CALLS, "rb") as f:
        return calls_stamp().encode() + b"\0" in f.read()


def _calls_possible() -> bool:
    """Whether there is a torch with CUDA and its headers to build the compiled calls against.  The library needs neither."""
    try:
        import torch
    except ImportError:
        return False
    return torch.version.cuda is not None and os.path.exists(os.path.join(_torch_include(torch), "torch", "csrc", "Exceptions.h"))


def _torch_include(torch) -> str:
    return os.path.join(os.path.dirname(torch.__file__), "include")


def _calls_due() -> bool:
    return _calls_possible() and (_older(CALLS, ["calls.cpp"]) or not calls_fit())


def needs_build() -> bool:
    return _older(LIB, _library_sources()) or _calls_due()


def _build_calls() -> None:
    import sysconfig
    import torch
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    include = _torch_include(torch)
    includes = [include, os.path.join(include, "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"],
                os.path.join(cuda, "include")]
    subprocess.check_call([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
                           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DCALLS_STAMP="{calls_stamp()}"',
                           *[f"-I{d}" for d in includes], os.path.join(CSRC, "calls.cpp"), "-o", CALLS, LIB,
                           f"-L{os.path.join(os.path.dirname(include), 'lib')}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python",
                           "-Wl,-rpath,$ORIGIN"])


def build(force: bool = False, verbose: bool = False) -> str:
    if force or _older(LIB, _library_sources()):
        _build_library(verbose)
        force = True
    if force and not _calls_possible():
        sys.stderr.write("no torch with CUDA and its headers: the library is built, the compiled calls are left out\n")
    elif force or _calls_due():
        _build_calls()
    return LIB


def _build_library(verbose: bool) -> None:
    nvcc = _nvcc()
    objs = []
    procs = []
    bdir = os.path.join(HERE, "build")
    os.makedirs(bdir, exist_ok=True)
    for src in SOURCES:
        obj = os.path.join(bdir, src.replace(".cu", ".o"))
        objs.append(obj)
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        log, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(f"--- {src}\n{log}\n")
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    subprocess.check_call([nvcc, "-arch=sm_100a", "-shared", "-Xlinker", "-soname=libb200moe.so", "-o", LIB, *objs])


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
