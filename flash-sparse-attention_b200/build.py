"""Build libfsa_sm100.so (sm_100a only) in-tree with nvcc.

    python flash-sparse-attention_b200/build.py [--force]

The library lands in flash-sparse-attention_b200/fsa/lib/libfsa_sm100.so and the native host code
(csrc/host, a Python extension on torch's C++ API) beside it; nvcc cross-compiles without a GPU.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT_DIR = os.path.join(HERE, "fsa", "lib")
LIB = os.path.join(OUT_DIR, "libfsa_sm100.so")
HOST_SRC = os.path.join(CSRC, "host")
HOST_LIB = os.path.join(OUT_DIR, "_fsa_host.so")
OBJ_DIR = os.path.join(HERE, "build")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC", "-DFSA_BUILD",
]


def sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def host_sources():
    return sorted(f for f in os.listdir(HOST_SRC) if f.endswith(".cpp"))


HEADER = os.path.join(os.path.dirname(HERE), "include", "fsa_sm100.h")


def _newest(paths):
    return max(os.path.getmtime(p) for p in paths)


def _files(d, *ends):
    return [os.path.join(d, f) for f in os.listdir(d) if f.endswith(ends)]


def _run(cmd, what, verbose=False):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"{what} failed:\n{r.stdout}\n{r.stderr}")
    if verbose:
        sys.stderr.write(r.stderr)


def _fresh(obj, inputs, force):
    return not force and os.path.exists(obj) and os.path.getmtime(obj) >= _newest(inputs)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OUT_DIR, exist_ok=True)
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = _files(CSRC, ".cuh", ".h") + [HEADER]
    host_headers = _files(HOST_SRC, ".h") + [HEADER]

    def compile_one(job):
        src, obj, is_host = job
        if _fresh(obj, [src] + (host_headers if is_host else headers), force or verbose):
            return False
        if is_host:
            import torch
            from torch.utils import cpp_extension

            inc = [f"-I{p}" for p in cpp_extension.include_paths("cuda") + [sysconfig.get_paths()["include"]]]
            _run(["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_fsa_host",
                  f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *inc, "-c", src, "-o", obj], f"g++ {src}")
        else:
            _run([NVCC, *(["-Xptxas=-v"] if verbose else []), *FLAGS, "-c", src, "-o", obj], f"nvcc {src}", verbose)
        return True

    cuda = [(os.path.join(CSRC, f), os.path.join(OBJ_DIR, f[:-3] + ".o"), False) for f in sources()]
    host = [(os.path.join(HOST_SRC, f), os.path.join(OBJ_DIR, "host_" + f[:-4] + ".o"), True) for f in host_sources()]
    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        list(ex.map(compile_one, cuda + host))
    objs = [o for _, o, _ in cuda]
    if not _fresh(LIB, objs, force):
        _run([NVCC, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "shared",
              "-Xlinker", "-rpath=/usr/local/cuda/lib64"], "link")
    hobjs = [o for _, o, _ in host]
    if not _fresh(HOST_LIB, hobjs + [LIB], force):
        from torch.utils import cpp_extension

        dirs = cpp_extension.library_paths("cuda")
        _run(["g++", "-shared", "-o", HOST_LIB, *hobjs, f"-L{OUT_DIR}", "-l:libfsa_sm100.so", *[f"-L{d}" for d in dirs], "-lc10", "-lc10_cuda",
              "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-Wl,-rpath,$ORIGIN"], "link")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
