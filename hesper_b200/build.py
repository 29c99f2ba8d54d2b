"""Builds libhesper_b200.so (CUDA kernels + C ABI) in-tree with nvcc for sm_100a, and
_binding.so (the layer API's calls as C++ over torch and the C ABI) with g++.

Run as ``python -m hesper_b200.build``.  nvcc cross-compiles without a GPU.  The
shared object carries a static CUDA runtime, so it needs only the driver.
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libhesper_b200.so")
BINDING = os.path.join(HERE, "_binding.so")
BINDING_TAG = os.path.join(OBJ, "_binding.tag")  # the Python and torch it was built against

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
]


def sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _binding_tag() -> str:
    import torch
    return f"{sys.version} | torch {torch.__version__} in {os.path.dirname(torch.__file__)}"


def binding_stale() -> bool:
    """Whether _binding.so is missing, older than its sources or built against another Python or torch
    than those that would load it."""
    if _stale(BINDING, [os.path.join(CSRC, "py_binding.cpp"), os.path.join(HERE, "..", "include", "hesper_b200.h")]):
        return True
    try:
        with open(BINDING_TAG) as f:
            return f.read() != _binding_tag()
    except OSError:
        return True


def build_binding(force: bool = False) -> str:
    """_binding.so, linked against the library beside it and the torch that is installed."""
    if not (force or binding_stale()):
        return BINDING
    src = os.path.join(CSRC, "py_binding.cpp")
    import sysconfig

    import torch
    from torch.utils import cpp_extension
    tdir = os.path.dirname(torch.__file__)
    nvcc = shutil.which(os.environ.get("HB200_NVCC", "nvcc"))
    cuda = cpp_extension.CUDA_HOME or (os.path.dirname(os.path.dirname(nvcc)) if nvcc else "/usr/local/cuda")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-Wno-deprecated-declarations",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           "-I" + sysconfig.get_paths()["include"], "-I" + os.path.join(cuda, "include")]
    cmd += ["-I" + p for p in cpp_extension.include_paths()]
    cmd += [src, "-o", BINDING, "-L" + HERE, "-l:libhesper_b200.so", "-Wl,-rpath,$ORIGIN",
            "-L" + os.path.join(tdir, "lib"), "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed: " + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    with open(BINDING_TAG, "w") as f:
        f.write(_binding_tag())
    return BINDING


def build(force: bool = False, verbose: bool = False) -> str:
    nvcc = os.environ.get("HB200_NVCC", "nvcc")
    os.makedirs(OBJ, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(HERE, "..", "include", "hesper_b200.h"))
    jobs = []
    objs = []
    for src in sources():
        s = os.path.join(CSRC, src)
        o = os.path.join(OBJ, src[:-3] + ".o")
        objs.append(o)
        if force or _stale(o, [s] + headers):
            extra = os.environ.get("HB200_NVCC_EXTRA", "").split()
            cmd = [nvcc] + NVCC_FLAGS + extra + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed: " + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stderr

    if jobs:
        with ThreadPoolExecutor(max_workers=min(8, len(jobs))) as ex:
            for out in ex.map(run, jobs):
                if verbose and out:
                    sys.stderr.write(out)
    if jobs or force or _stale(LIB, objs):
        link = [nvcc, "-shared", "-o", LIB] + objs + ["-cudart", "static", "-ldl",
                "-gencode", "arch=compute_100a,code=sm_100a"]
        run(link)
    build_binding(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
