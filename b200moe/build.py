"""In-tree build of the sm_100a extension.

Every ``csrc/*.cu`` is compiled with nvcc for ``compute_100a/sm_100a`` and linked
into ``b200moe/_C/libb200moe.so``, which ``b200moe.ops.native`` loads through
ctypes.  The sources use only the CUDA runtime (the one driver entry point they
need, ``cuTensorMapEncodeTiled``, is resolved at run time), so the library
builds on a machine without a GPU or a driver.
"""
from __future__ import annotations

import hashlib
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "csrc")
# B200MOE_DEBUG=1 selects the checked build: -DB200MOE_DEBUG (range checks on data-dependent indices, see
# csrc/debug.cuh), its own object directory and library name, loaded by b200moe.ops.native under the same variable.
DEBUG = os.environ.get("B200MOE_DEBUG", "0") not in ("", "0")
OUT = os.path.join(HERE, "_C", "debug") if DEBUG else os.path.join(HERE, "_C")
LIB = os.path.join(OUT, "libb200moe_debug.so" if DEBUG else "libb200moe.so")
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-Xptxas", "-v"] + (["-DB200MOE_DEBUG"] if DEBUG else [])


def nvcc() -> str:
    found = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(found):
        raise RuntimeError("nvcc not found")
    return found


def _sources():
    return sorted(f for f in os.listdir(SRC) if f.endswith(".cu"))


def _digest(path: str, flags=tuple(NVCC_FLAGS)) -> str:
    """Of a source, the headers and what it is compiled with."""
    h = hashlib.sha256()
    for name in sorted(os.listdir(SRC)):
        if name.endswith((".cuh", ".h")) or os.path.join(SRC, name) == path:
            with open(os.path.join(SRC, name), "rb") as f:
                h.update(f.read())
    h.update(" ".join(flags).encode())
    return h.hexdigest()


def _compile(name: str, verbose: bool) -> str:
    src = os.path.join(SRC, name)
    obj = os.path.join(OUT, name[:-3] + ".o")
    stamp = obj + ".sha"
    digest = _digest(src)
    if os.path.exists(obj) and os.path.exists(stamp) and open(stamp).read() == digest:
        return obj
    cmd = [nvcc(), *NVCC_FLAGS, "-c", src, "-o", obj]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    log = obj[:-2] + ".ptxas.log"
    with open(log, "w") as f:
        f.write(proc.stdout + proc.stderr)
    if proc.returncode:
        sys.stderr.write(proc.stdout + proc.stderr)
        raise RuntimeError(f"nvcc failed for {name}")
    with open(stamp, "w") as f:
        f.write(digest)
    if verbose:
        print(f"[b200moe.build] compiled {name}")
    return obj


def _build_nodes(verbose: bool) -> None:
    """The C++ autograd nodes (csrc/nodes.cpp), compiled against the installed PyTorch; one file for both libraries, which
    it binds to at run time.  The package does without (the nodes in Python issue the same launches): skipped where PyTorch
    is not there; where they cannot be built this says so, leaves none of an earlier build and raises nothing."""
    try:
        import torch
        from torch.utils import cpp_extension
    except ImportError:
        if verbose:
            print("[b200moe.build] no PyTorch here: C++ autograd nodes not built")
        return
    target = os.path.join(HERE, "_C", "b200moe_nodes.so")
    stamp = target + ".sha"
    try:
        source = os.path.join(SRC, "nodes.cpp")
        digest = _digest(source, [torch.__version__, sys.version])
        if os.path.exists(target) and os.path.exists(stamp) and open(stamp).read() == digest:
            return
        import sysconfig
        lib = os.path.join(os.path.dirname(torch.__file__), "lib")
        cuda = os.path.dirname(os.path.dirname(nvcc()))
        include = [*cpp_extension.include_paths(), os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
        os.makedirs(os.path.dirname(target), exist_ok=True)
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-DTORCH_API_INCLUDE_EXTENSION_H",
               "-DTORCH_EXTENSION_NAME=b200moe_nodes", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
               *(f"-I{path}" for path in include), source, "-o", target, f"-L{lib}", "-lc10", "-lc10_cuda", "-ltorch",
               "-ltorch_cpu", "-ltorch_python", "-ldl"]
        proc = subprocess.run(cmd, capture_output=True, text=True)
        if proc.returncode:
            raise RuntimeError(f"g++ failed for nodes.cpp\n{proc.stdout}{proc.stderr}")
    except Exception as error:
        for stale in (target, stamp):
            if os.path.exists(stale):
                os.unlink(stale)
        sys.stderr.write(f"[b200moe.build] C++ autograd nodes not built, the nodes in Python stand for them: {error}\n")
        return
    with open(stamp, "w") as f:
        f.write(digest)
    if verbose:
        print("[b200moe.build] compiled nodes.cpp")


def build_all(verbose: bool = False, force: bool = False) -> str:
    os.makedirs(OUT, exist_ok=True)
    if force:
        for name in os.listdir(OUT):
            if name.endswith((".o", ".sha", ".so")):
                os.unlink(os.path.join(OUT, name))
    names = _sources()
    with ThreadPoolExecutor(max_workers=min(8, len(names) or 1)) as pool:
        nodes = pool.submit(_build_nodes, verbose)
        objects = list(pool.map(lambda n: _compile(n, verbose), names))
        nodes.result()
    newest = max(os.path.getmtime(o) for o in objects)
    if not os.path.exists(LIB) or os.path.getmtime(LIB) < newest:
        cmd = [nvcc(), "-shared", "-o", LIB, *objects, "-Xcompiler", "-fPIC", "-lcudart"]
        proc = subprocess.run(cmd, capture_output=True, text=True)
        if proc.returncode:
            sys.stderr.write(proc.stdout + proc.stderr)
            raise RuntimeError("link failed")
        if verbose:
            print(f"[b200moe.build] linked {LIB}")
    return LIB


if __name__ == "__main__":
    build_all(verbose=True, force="--force" in sys.argv)
