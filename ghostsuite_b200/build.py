"""Builds libghost_b200.so (sm_100a only) in-tree with nvcc, and _ghost_torch.so, the torch binding on
top of it, with g++.  The library itself sees no torch header: it is a plain C-ABI shared object."""
from __future__ import annotations

import importlib.util
import os
import re
import shutil
import subprocess
import sys
import sysconfig

from ._lib import binding_built_for

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libghost_b200.so")
SOURCES = ["common.cu", "ghost_gram.cu", "ghost_gram_pair.cu", "xty_gemm.cu", "xty_gemm_pair.cu", "tile_dot.cu", "rowwise.cu", "pass_reduce.cu", "dense_small.cu", "conv_tokens.cu", "embedding.cu", "gradproj.cu", "proj_extras.cu", "workload_loss.cu"]
BINDING = os.path.join(HERE, "_ghost_torch.so")
BINDING_SOURCE = os.path.join("host", "torch_ops.cpp")
HEADERS = ["common.cuh", "gram_operands.cuh", "sm100_ptx.cuh", "mma_sync.cuh", "xty_colsum.cuh", "xty_operands.cuh", "xty_store.cuh", "launch_rules.h", os.path.join("..", "..", "include", "ghost_b200.h")]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found; set NVCC or put /usr/local/cuda/bin on PATH")


def _stale(target: str, sources) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    deps = [os.path.join(CSRC, s) for s in sources] + [os.path.abspath(__file__)]
    return any(os.path.getmtime(d) > t for d in deps)


def _torch():
    """``(installation root, version)`` of torch, without importing it."""
    spec = importlib.util.find_spec("torch")
    if spec is None:
        raise RuntimeError("torch is not importable: its headers are needed for _ghost_torch.so")
    root = os.path.dirname(spec.origin)
    with open(os.path.join(root, "version.py")) as f:
        return root, re.search(r"__version__\s*=\s*['\"]([^'\"]+)", f.read()).group(1)


def _binding_stale() -> bool:
    return _stale(BINDING, [BINDING_SOURCE] + HEADERS[-2:]) or not binding_built_for(_torch()[1], BINDING)


def _start_binding():
    """Start compiling the torch binding; it needs the library's header only, so it runs beside nvcc."""
    root, version = _torch()
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    obj = os.path.join(HERE, "build", "torch_ops.o")
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", f'-DGHOST_TORCH_VERSION="{version}"',
           "-c", os.path.join(CSRC, BINDING_SOURCE), "-o", obj]
    cmd += [f"-I{d}" for d in include]
    link = ["g++", "-shared", obj, "-o", BINDING, f"-L{HERE}", "-l:libghost_b200.so", f"-L{os.path.join(root, 'lib')}",
            "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    return subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True), link


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile every .cu under csrc/ for sm_100a and link libghost_b200.so next to this file, then the
    torch binding."""
    lib_stale = force or _stale(LIB, SOURCES + HEADERS)
    binding_stale = lib_stale or _binding_stale()
    if not lib_stale and not binding_stale:
        return LIB
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    binding = _start_binding()
    if lib_stale:
        _build_library(verbose)
    proc, link = binding
    out, _ = proc.communicate()
    if proc.returncode != 0:
        sys.stderr.write(f"--- g++ failed on {BINDING_SOURCE}\n{out}\n")
        raise RuntimeError("building _ghost_torch.so failed")
    subprocess.run(link, check=True)
    return LIB


def _build_library(verbose: bool) -> None:
    nvcc = _nvcc()
    objdir = os.path.join(HERE, "build")
    flags = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
             "-Xcompiler", "-fPIC"]
    if verbose:
        flags += ["-Xptxas", "-v"]
    objs = []
    procs = []
    for src in SOURCES:
        obj = os.path.join(objdir, src.replace(".cu", ".o"))
        objs.append(obj)
        cmd = [nvcc] + flags + ["-c", os.path.join(CSRC, src), "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            failed = True
            sys.stderr.write(f"--- nvcc failed on {src}\n{out}\n")
        elif verbose or out.strip():
            sys.stderr.write(f"--- {src}\n{out}\n")
    if failed:
        raise RuntimeError("building libghost_b200.so failed")
    link = [nvcc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"]
    subprocess.run(link, check=True)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
