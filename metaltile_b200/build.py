"""Build ``libmtcuda.so`` in-tree with nvcc for sm_100a (``python -m metaltile_b200.build``).

Every ``csrc/*.cu`` is compiled to an object file (in parallel) and linked into
``metaltile_b200/libmtcuda.so``.  The library depends on the CUDA runtime only.  ``csrc/dispatch_binding.cpp`` becomes
``metaltile_b200/_dispatch.so``, the Python binding of the name-keyed call on host buffers, and ``csrc/binding.cpp``
``metaltile_b200/_native.so``, that of the typed ops on tensors: it alone needs PyTorch, and is left out where there is none.
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
DISPATCH = os.path.join(HERE, "_dispatch.so")    # the Python binding of the name-keyed call (csrc/dispatch_binding.cpp)
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


def _torch():
    """PyTorch, or None where it is not installed."""
    try:
        import torch
        return torch
    except ImportError:
        return None


def _extension(source, out, log, extra_flags=(), extra_libs=()):
    """A CPython extension over libmtcuda.so with the host compiler."""
    import sysconfig

    cxx = shutil.which("g++") or "c++"
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-I", sysconfig.get_paths()["include"], *extra_flags, os.path.join(CSRC, source),
           "-o", out, "-L", HERE, "-l:libmtcuda.so", "-Wl,-rpath,$ORIGIN", *extra_libs]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    with open(log, "w") as f:
        f.write(" ".join(cmd) + "\n" + r.stdout)
    if r.returncode != 0:
        raise RuntimeError(f"{cxx} failed on {source}:\n{r.stdout[-6000:]}")


def native_digest(torch=None) -> str:
    """What _native.so is tied to: its sources, the library's interface, and the PyTorch and the Python whose headers it is
    compiled against (another PyTorch has another ABI: an extension left from the one before must not pass for current)."""
    torch = torch or _torch()
    tied = [torch.__version__, str(torch.version.git_version), str(torch._C._GLIBCXX_USE_CXX11_ABI), sys.version]
    sources = [os.path.join(CSRC, "binding.cpp"), *glob.glob(os.path.join(HERE, "..", "include", "*.h"))]
    return _digest(sources) + hashlib.sha256("\0".join(tied).encode()).hexdigest()


def _compile_native(torch, log):
    """csrc/binding.cpp -> _native.so against the installed PyTorch's headers."""
    from torch.utils import cpp_extension

    flags = [f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DMTC_TORCH_VERSION="{torch.__version__}"']
    for inc in cpp_extension.include_paths("cuda"):
        flags += ["-isystem", inc]
    libs = os.path.join(os.path.dirname(torch.__file__), "lib")
    _extension("binding.cpp", NATIVE, log, flags,
               ["-L", libs, "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda"])


def _stamp(path, digest):
    with open(path, "w") as f:
        f.write(digest)


def build(force: bool = False, verbose: bool = False) -> str:
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    headers = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    deps = srcs + [os.path.join(CSRC, "dispatch_binding.cpp")] + headers
    torch = _torch()
    # the C library and the binding that needs it alone; the extension over PyTorch has a stamp of its own
    stamps = [(os.path.join(OBJ, "stamp"), _digest(deps) + sys.version, (LIB, DISPATCH))]
    if torch:
        stamps.append((os.path.join(OBJ, "native.stamp"), native_digest(torch), (NATIVE,)))
    stale = [force or not all(map(os.path.exists, outs)) or not os.path.exists(path) or open(path).read() != digest
             for path, digest, outs in stamps]
    if not any(stale):
        return LIB
    if not stale[0]:                                     # only the extension over PyTorch
        _compile_native(torch, os.path.join(OBJ, "binding.log"))
        _stamp(*stamps[1][:2])
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
    _extension("dispatch_binding.cpp", DISPATCH, os.path.join(OBJ, "dispatch_binding.log"))
    if torch:
        _compile_native(torch, os.path.join(OBJ, "binding.log"))
    else:
        print("PyTorch is not installed: _native.so (the typed ops on tensors) is not built")
    for path, digest, _ in stamps:
        _stamp(path, digest)
    if verbose:
        print("built", LIB)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True)
