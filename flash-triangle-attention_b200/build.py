"""Build libfta.so (the C-ABI CUDA library, nvcc for sm_100a) and _fta_torch.so (the torch extension
behind ``attention()``, plain C++ linked against libfta.so) in-tree.

    python flash-triangle-attention_b200/build.py [--force]

The shared objects land next to this file so that they travel with the source tree.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libfta.so")
SOURCES = ["api.cu", "fwd_sm100.cu", "fwd_quad_sm100.cu", "bwd_sm100.cu", "stream_kernels.cu", "noalloc.cu"]
HEADERS = ["tc05.cuh", "tmap.h", "fta_kernels.h", "schedule.h", "native_api.h", os.path.join("..", "..", "include", "fta.h")]
TORCH_EXT = os.path.join(HERE, "_fta_torch.so")
TORCH_SOURCE = "torch_binding.cpp"
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]


def _sources():
    return [s for s in SOURCES if os.path.exists(os.path.join(CSRC, s))]


def _stale(target, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def needs_build() -> bool:
    return _stale(LIB, [os.path.join(CSRC, s) for s in _sources() + HEADERS] + [os.path.abspath(__file__)])


def _torch_command():
    from torch.utils import cpp_extension  # include and library folders of the installed torch
    inc = [f"-I{d}" for d in cpp_extension.include_paths("cuda") + [sysconfig.get_paths()["include"]]]
    lib = cpp_extension.library_paths("cuda")
    return (["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-fvisibility=hidden", "-DTORCH_API_INCLUDE_EXTENSION_H",
             "-DTORCH_EXTENSION_NAME=_fta_torch"] + inc + [os.path.join(CSRC, TORCH_SOURCE), "-o", TORCH_EXT]
            + [f"-L{d}" for d in lib + [HERE]] + ["-Wl,-rpath,$ORIGIN"] + [f"-Wl,-rpath,{d}" for d in lib]
            + ["-l:libfta.so", "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"])


def build_torch_ext(force: bool = False) -> str:
    deps = [os.path.join(CSRC, s) for s in (TORCH_SOURCE, "native_api.h", os.path.join("..", "..", "include", "fta.h"))]
    if force or _stale(TORCH_EXT, deps + [os.path.abspath(__file__)]):
        subprocess.run(_torch_command(), check=True)
    return TORCH_EXT


def build(force: bool = False, verbose: bool = False) -> str:
    if force or needs_build():
        _build_lib(verbose)
    build_torch_ext(force)
    return LIB


def _build_lib(verbose: bool) -> None:
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    objs = []
    procs = []
    for s in _sources():
        obj = os.path.join(CSRC, s.replace(".cu", ".o"))
        cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", os.path.join(CSRC, s), "-o", obj]
        procs.append((s, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    for s, pr in procs:
        out, _ = pr.communicate()
        if verbose or pr.returncode != 0:
            sys.stderr.write(out)
        if pr.returncode != 0:
            raise RuntimeError(f"nvcc failed on {s}")
    subprocess.run([nvcc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"], check=True)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
