"""Build the sm_100a shared library in-tree with nvcc.

    python -m worldattention_b200.build            # incremental
    python -m worldattention_b200.build --force    # rebuild everything

The results, both loaded by `_lib.py`: `worldattention_b200/libwa_b200.so` (the kernels, a plain C ABI) and
`worldattention_b200/_host.so` (the Python module that makes the per-forward calls, built against PyTorch's headers).
"""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libwa_b200.so")
HOST_SRC = os.path.join(CSRC, "host", "wa_host.cpp")
HOST = os.path.join(HERE, "_host.so")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-Xptxas", "-v", "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or install the CUDA toolkit")


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    sources = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    headers += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE) if f.endswith(".h")]
    nvcc = _nvcc()

    def compile_one(src: str):
        obj = os.path.join(OBJ, src[:-3] + ".o")
        path = os.path.join(CSRC, src)
        if not force and not _stale(obj, [path] + headers):
            return obj, ""
        cmd = [nvcc, *NVCC_FLAGS, "-c", path, "-o", obj]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{res.stdout}\n{res.stderr}")
        return obj, res.stderr

    with ThreadPoolExecutor(max_workers=min(8, len(sources) + 1)) as pool:
        host = pool.submit(build_host, force, headers)
        results = list(pool.map(compile_one, sources))
    objs = [o for o, _ in results]
    if verbose:
        for (_, log), src in zip(results, sources):
            if log:
                print(f"---- {src}\n{log}")
    if force or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
        res = subprocess.run(cmd, capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    host.result()
    return LIB


def build_host(force: bool, headers) -> str:
    """The host module: plain C++ against PyTorch's headers (no nvcc)."""
    if not force and not _stale(HOST, [HOST_SRC] + headers):
        return HOST
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    include = [f"-I{os.path.join(root, 'include')}", f"-I{os.path.join(root, 'include', 'torch', 'csrc', 'api', 'include')}",
               f"-I{os.path.join(cuda, 'include')}", f"-I{sysconfig.get_paths()['include']}"]
    cmd = [os.environ.get("CXX") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           *include, HOST_SRC, "-o", HOST, f"-L{os.path.join(root, 'lib')}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda", "-ltorch_cuda"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"building the host module failed:\n{res.stdout}\n{res.stderr}")
    return HOST


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv or "--verbose" in sys.argv))
