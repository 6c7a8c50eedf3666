"""Builds ``libortho_b200.so`` (the C-ABI CUDA library) in-tree with nvcc for sm_100a.

    python -m libortho_b200.build [--force] [--verbose]

Takes the place of the reference's ``setup.py`` CUDAExtension build (``setup.py:112-130``):
one target architecture, ``-O3 -lineinfo``, static CUDA runtime, no Python headers.  The forward's host path
``_fastcall.so`` is a CPython extension beside it, compiled against the installed torch and rebuilt when that
or the interpreter changes.
"""
from __future__ import annotations

import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB_PATH = os.path.join(HERE, "libortho_b200.so")
SOURCES = ["api.cu", "plan.cu", "decode.cu", "decode_stream.cu", "mid.cu", "wide.cu", "prefill.cu", "transpose.cu", "longrows.cu", "static_scratch.cu", "comm.cu", "pack.cu", "sieve.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--use_fast_math",
    "-cudart", "static",
]
# the forward's host path as a CPython extension (csrc/fastcall.cpp), compiled against the installed torch
FAST_SOURCE = os.path.join(CSRC, "fastcall.cpp")
FAST_PATH = os.path.join(HERE, "_fastcall.so")
FAST_STAMP = os.path.join(HERE, "build", "fastcall.txt")       # what the extension was compiled against


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _deps() -> list:
    out = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))]
    out.append(os.path.join(INCLUDE, "ortho_b200.h"))
    return out


def _fast_against() -> str:
    """What ties the extension to the installation: torch's version and place, the interpreter's ABI."""
    import sysconfig

    import torch
    return "\n".join((torch.__version__, os.path.dirname(torch.__file__), str(sysconfig.get_config_var("SOABI"))))


def needs_build_fast() -> bool:
    deps = [FAST_SOURCE, os.path.join(INCLUDE, "ortho_b200.h")]
    if not os.path.exists(FAST_PATH) or any(os.path.getmtime(d) > os.path.getmtime(FAST_PATH) for d in deps):
        return True
    try:
        with open(FAST_STAMP) as f:
            return f.read() != _fast_against()
    except FileNotFoundError:
        return True


def build_fast(force: bool = False) -> str:
    if not force and not needs_build_fast():
        return FAST_PATH
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    inc = cpp_extension.include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include"), INCLUDE]
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-w", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f'-DORTHO_TORCH_VERSION="{torch.__version__}"',
           *[f"-I{d}" for d in inc], FAST_SOURCE, "-o", FAST_PATH, f"-L{lib}", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", "-ltorch"]
    out = subprocess.run(cmd, capture_output=True, text=True)
    if out.returncode != 0:
        raise RuntimeError("g++ failed on fastcall.cpp:\n" + out.stdout + out.stderr)
    os.makedirs(os.path.dirname(FAST_STAMP), exist_ok=True)
    with open(FAST_STAMP, "w") as f:
        f.write(_fast_against())
    return FAST_PATH


def needs_build() -> bool:
    if not os.path.exists(LIB_PATH):
        return True
    t = os.path.getmtime(LIB_PATH)
    return any(os.path.getmtime(d) > t for d in _deps())


def build(force: bool = False, verbose: bool = False) -> str:
    build_fast(force)
    if not force and not needs_build():
        return LIB_PATH
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    nvcc = _nvcc()
    procs = []
    objs = []
    for src in SOURCES:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        objs.append(obj)
        cmd = [nvcc, *NVCC_FLAGS, "-I", INCLUDE, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            failed = True
            sys.stderr.write(f"--- nvcc failed on {src}\n{out}\n")
        elif verbose:
            sys.stderr.write(out)
    if failed:
        raise RuntimeError("nvcc failed; see output above")
    link = [nvcc, "-shared", "-cudart", "static", "-gencode", "arch=compute_100a,code=sm_100a",
            "-Xcompiler", "-fPIC", "-o", LIB_PATH, *objs]
    out = subprocess.run(link, capture_output=True, text=True)
    if out.returncode != 0:
        raise RuntimeError("link failed:\n" + out.stdout + out.stderr)
    return LIB_PATH


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
