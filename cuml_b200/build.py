"""Build recipe of libb2fil.so (nvcc for sm_100a) and of the torch call path beside it; in-tree
output under cuml_b200/lib/.

`python -m cuml_b200.build [--force] [--verbose]` (also called by `__graft_entry__.build()`).
The register / shared-memory report of ptxas is written to cuml_b200/lib/ptxas.log.
"""
from __future__ import annotations

import importlib.metadata
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB = os.path.join(LIB_DIR, "libb2fil.so")
SOURCES = ["api.cu", "kernels.cu", "kernels_q_top6.cu", "kernels_q_plain6.cu", "kernels_q_plain4.cu",
           "kernels_q_cat.cu", "kernels_q_generic.cu", "kernels_q_narrow.cu", "kernels_q_pair.cu",
           "kernels_q_leafg.cu", "kernels_q_vec.cu", "kernels_q_top_vec.cu", "kernels_q_top_out.cu",
           "kernels_sparse_c.cu",
           "pack.cpp", "blocks.cpp"]
HEADERS = ["each_tree.hpp", "forest.hpp", "host_pool.hpp", "kernels.hpp", "kernels_q.hpp", "device_common.cuh", "dense_q.cuh",
           os.path.join("..", "..", "include", "b2fil.h")]


# Native call path for torch tensors: a CPython module compiled against the installed torch, whose
# version is part of the file name (another torch needs another build).
TORCH_SOURCE = os.path.join(SRC, "torch_call.cpp")


def torch_module_path():
    """Path of the compiled torch module, or None where torch is not installed."""
    try:
        return os.path.join(LIB_DIR, f"b2fil_torch-{importlib.metadata.version('torch')}.so")
    except importlib.metadata.PackageNotFoundError:
        return None


def _torch_command(out: str) -> list:
    root = os.path.dirname(importlib.util.find_spec("torch").origin)  # without importing torch
    inc, lib = os.path.join(root, "include"), os.path.join(root, "lib")
    cuda = os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")
    dirs = [inc, os.path.join(inc, "torch", "csrc", "api", "include"), cuda,
            sysconfig.get_paths()["include"]]
    return (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-Wall"] + ["-I" + d for d in dirs] +
            [TORCH_SOURCE, "-o", out, "-L" + lib, "-lc10", "-lc10_cuda", "-ltorch_cpu",
             "-ltorch_cuda", "-ltorch_python", "-ltorch"])


def _nvcc() -> str:
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libb2fil.so cannot be built")
    return exe


def _newer(target: str, deps: list) -> bool:
    if not os.path.exists(target):
        return False
    t = os.path.getmtime(target)
    return all((not os.path.exists(d)) or os.path.getmtime(d) <= t for d in deps)


def _lib_up_to_date() -> bool:
    deps = [os.path.join(SRC, s) for s in SOURCES + HEADERS] + [os.path.abspath(__file__)]
    return _newer(LIB, deps)


def _torch_module_settled() -> bool:
    """Built, not needed, or tried and failed (the log of a failed try is kept as <module>.failed)."""
    module = torch_module_path()
    deps = [TORCH_SOURCE, os.path.abspath(__file__)]
    return module is None or _newer(module, deps) or _newer(module + ".failed", deps)


def up_to_date() -> bool:
    return _lib_up_to_date() and _torch_module_settled()


def _build_torch_module() -> str:
    """Compile the torch module and return the log.  Not an error when that fails: device calls then go
    through ctypes, a few microseconds slower."""
    module = torch_module_path()
    failed = module + ".failed"
    try:
        cmd = _torch_command(module + ".tmp")
        proc = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        text, ok = " ".join(cmd) + "\n" + proc.stdout, proc.returncode == 0
    except (OSError, RuntimeError, AttributeError) as e:  # no compiler, no CUDA headers, no torch
        text, ok = f"torch call path: {e!r}\n", False
    if ok:
        os.replace(module + ".tmp", module)
        if os.path.exists(failed):
            os.remove(failed)
    else:
        with open(failed, "w") as fh:
            fh.write(text)
        if os.path.exists(module):
            os.remove(module)  # older than its source
        sys.stderr.write(f"{text}\nthe torch call path could not be built; device calls go through ctypes\n")
    return text


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and up_to_date():
        return LIB
    if force or not _torch_module_settled():
        os.makedirs(LIB_DIR, exist_ok=True)
        if torch_module_path():
            log = _build_torch_module()
            if verbose:
                print(log)
    if not force and _lib_up_to_date():
        return LIB
    if not all(os.path.exists(os.path.join(SRC, s)) for s in SOURCES):
        raise RuntimeError("kernel sources missing; cannot build libb2fil.so")
    os.makedirs(LIB_DIR, exist_ok=True)
    # one nvcc per translation unit, all at once (the kernel families are split over several
    # files for exactly this), then one link step
    obj_dir = os.path.join(LIB_DIR, "obj")
    os.makedirs(obj_dir, exist_ok=True)
    base = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
            "-Xcompiler", "-fPIC,-Wall", "-Xptxas", "-v"]
    jobs = []
    for src in SOURCES:
        obj = os.path.join(obj_dir, os.path.splitext(src)[0] + ".o")
        cmd = base + ["-c", os.path.join(SRC, src), "-o", obj]
        out = open(obj + ".log", "w+")  # a file, not a pipe: nothing blocks while others run
        jobs.append((cmd, obj, subprocess.Popen(cmd, stdout=out, stderr=subprocess.STDOUT), out))
    log, failed = [], False
    for cmd, obj, proc, out in jobs:
        proc.wait()
        out.seek(0)
        log.append(" ".join(cmd) + "\n" + out.read())
        out.close()
        failed |= proc.returncode != 0
    if not failed:
        cmd = [_nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", LIB]
        cmd += [obj for _, obj, _, _ in jobs]
        proc = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        log.append(" ".join(cmd) + "\n" + proc.stdout)
        failed = proc.returncode != 0
    text = "\n".join(log)
    with open(os.path.join(LIB_DIR, "ptxas.log"), "w") as fh:
        fh.write(text)
    if failed:
        sys.stderr.write(text)
        raise RuntimeError("nvcc failed building libb2fil.so")
    if verbose:
        print(text)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
