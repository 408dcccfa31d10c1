"""Build ``libmtcuda.so`` in-tree with nvcc for sm_100a (``python -m metaltile_b200.build``).

Every ``csrc/*.cu`` is compiled to an object file (in parallel) and linked into
``metaltile_b200/libmtcuda.so``.  The library depends on the CUDA runtime only.  ``csrc/binding.cpp`` becomes
``metaltile_b200/_native.so``, the Python binding of the typed ops over that library (it alone knows about torch).
"""
from __future__ import annotations

import concurrent.futures as cf
import glob
import hashlib
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libmtcuda.so")
NATIVE = os.path.join(HERE, "_native.so")        # the Python binding of the typed ops (csrc/binding.cpp)

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xptxas", "-v",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _digest(paths) -> str:
    h = hashlib.sha256(" ".join(NVCC_FLAGS).encode())
    for p in sorted(paths):
        with open(p, "rb") as f:
            h.update(p.encode() + b"\0" + f.read())
    return h.hexdigest()


def _compile(nvcc, src, obj, log, headers):
    """One object file; left alone when neither its source nor a header nor the flags changed."""
    stamp, digest = obj + ".stamp", _digest([src, *headers])
    if os.path.exists(obj) and os.path.exists(stamp) and open(stamp).read() == digest:
        return obj
    cmd = [nvcc, *NVCC_FLAGS, "-c", src, "-o", obj]
    env = dict(os.environ)
    env.pop("CC", None)
    env.pop("CXX", None)
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, env=env)
    with open(log, "w") as f:
        f.write(" ".join(cmd) + "\n" + r.stdout)
    if r.returncode != 0:
        raise RuntimeError(f"nvcc failed on {src}:\n{r.stdout[-6000:]}")
    with open(stamp, "w") as f:
        f.write(digest)
    return obj


def _compile_native(log):
    """csrc/binding.cpp -> _native.so with the host compiler, against the installed PyTorch's headers and libmtcuda.so."""
    import sysconfig

    from torch.utils import cpp_extension

    import torch
    cxx = shutil.which("g++") or "c++"
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", "-I", sysconfig.get_paths()["include"]]
    for inc in cpp_extension.include_paths("cuda"):
        cmd += ["-isystem", inc]
    cmd += [os.path.join(CSRC, "binding.cpp"), "-o", NATIVE, "-L", HERE, "-l:libmtcuda.so", "-Wl,-rpath,$ORIGIN", "-L", libs,
            "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    with open(log, "w") as f:
        f.write(" ".join(cmd) + "\n" + r.stdout)
    if r.returncode != 0:
        raise RuntimeError(f"{cxx} failed on binding.cpp:\n{r.stdout[-6000:]}")


def build(force: bool = False, verbose: bool = False) -> str:
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    deps = srcs + [os.path.join(CSRC, "binding.cpp")] + headers
    stamp = os.path.join(OBJ, "stamp")
    digest = _digest(deps)
    if not force and os.path.exists(LIB) and os.path.exists(NATIVE) and os.path.exists(stamp) and open(stamp).read() == digest:
        return LIB
    if force:
        shutil.rmtree(OBJ, ignore_errors=True)
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()
    objs = []
    with cf.ThreadPoolExecutor(max_workers=min(8, len(srcs))) as ex:
        futs = []
        for s in srcs:
            base = os.path.splitext(os.path.basename(s))[0]
            futs.append(ex.submit(_compile, nvcc, s, os.path.join(OBJ, base + ".o"), os.path.join(OBJ, base + ".log"), headers))
        for f in futs:
            objs.append(f.result())
    env = dict(os.environ)
    env.pop("CC", None)
    env.pop("CXX", None)
    cmd = [nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "static"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, env=env)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n" + r.stdout)
    _compile_native(os.path.join(OBJ, "binding.log"))
    with open(stamp, "w") as f:
        f.write(digest)
    if verbose:
        print("built", LIB)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
