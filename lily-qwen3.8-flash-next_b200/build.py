"""Builds the CUDA library and the Python call layer in-tree for sm_100a.

    python lily-qwen3.8-flash-next_b200/build.py [--force]

liblily_sampler.so beside this file exports the C ABI of include/lily_sampler.h
(nvcc cross-compiles without a GPU); _lily_calls.so is the extension module that fills
its argument blocks from torch tensors (csrc/python_ext.cpp). One compiler process per
source file, side by side; a file is compiled again when it or a header is newer.
"""
from __future__ import annotations

import os
import re
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "liblily_sampler.so")
CALLS = os.path.join(HERE, "_lily_calls.so")
CALLS_SOURCE = os.path.join(CSRC, "python_ext.cpp")
HEAD_SOURCE = os.path.join(CSRC, "lmhead.cu")

ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]
NVCC_FLAGS = [*ARCH_FLAGS, "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC"]


def sources():
    out = []
    for name in sorted(os.listdir(CSRC)):
        path = os.path.join(CSRC, name)
        if name.endswith((".cu", ".cpp")) and path != CALLS_SOURCE:
            out.append(path)
    return out


def _headers():
    deps = [os.path.join(INCLUDE, n) for n in os.listdir(INCLUDE)]
    return deps + [os.path.join(CSRC, n) for n in os.listdir(CSRC) if n.endswith((".cuh", ".h"))]


def _newest(paths) -> float:
    return max(os.path.getmtime(p) for p in paths)


def _older(target: str, t: float) -> bool:
    return not os.path.exists(target) or os.path.getmtime(target) < t


def stale() -> bool:
    headers = _newest(_headers())
    return _older(LIB, max(headers, _newest(sources()))) or _older(CALLS, max(headers, os.path.getmtime(CALLS_SOURCE)))


def _run(cmd, verbose=False):
    proc = subprocess.run(cmd, capture_output=True, text=True)
    if proc.returncode != 0:
        raise RuntimeError(" ".join(cmd[:1]) + " failed:\n" + proc.stdout + proc.stderr)
    if verbose:
        sys.stderr.write(proc.stderr)
    return proc.stderr


def check_head_registers(report: str) -> None:
    """Refuses a head kernel that the compiler did not give the registers its warps share out
    (Shape::REGS in lmhead_kernel.cuh): it would wait for registers it does not have, and
    the library would refuse to launch it. `report`: what ptxas -v said."""
    found = re.findall(r"Compiling entry function '\w*lmhead_kernelILj(\d+)ELi(\d)E\w*'.*?Used (\d+) registers", report,
                       re.S)
    if len(found) != 9:
        raise RuntimeError(f"the compiler reported {len(found)} of the LM head's 9 kernels")
    for tokens, fmt, used in found:
        want = 80 if tokens == "64" and fmt != "0" else 64
        if int(used) != want:
            raise RuntimeError(f"lmhead_kernel<{tokens}, {fmt}> was compiled for {used} registers a thread instead of {want} "
                               "(another compiler, or flags in LILY_NVCC_EXTRA?): its shares have to be cut anew")


def _calls_command():
    """g++ for the extension module: torch's headers and libraries, the library beside it (by its
    soname, so that a package that was moved or copied finds its own)."""
    import sysconfig

    import torch

    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    abi = int(torch._C._GLIBCXX_USE_CXX11_ABI)
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", f"-D_GLIBCXX_USE_CXX11_ABI={abi}",
            "-I", os.path.join(root, "include"), "-I", os.path.join(root, "include", "torch", "csrc", "api", "include"),
            "-I", os.path.join(cuda, "include"), "-I", sysconfig.get_paths()["include"], CALLS_SOURCE,
            "-L", os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda",
            "-L", HERE, "-l:" + os.path.basename(LIB), "-Wl,-rpath,$ORIGIN", "-o", CALLS]


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and not stale():
        return LIB
    nvcc = os.environ.get("NVCC", "nvcc")
    extra = os.environ.get("LILY_NVCC_EXTRA", "").split()  # extra nvcc flags, e.g. -Xptxas -v
    if verbose:
        extra += ["-Xptxas", "-v"]
    os.makedirs(OBJ, exist_ok=True)
    headers = _newest(_headers())
    jobs, objects = [], []
    for src in sources():
        obj = os.path.join(OBJ, os.path.basename(src) + ".o")
        objects.append(obj)
        if force or _older(obj, max(headers, os.path.getmtime(src))):
            report = ["-Xptxas", "-v"] if src == HEAD_SOURCE and not verbose else []
            jobs.append([nvcc, *NVCC_FLAGS, *extra, *report, "-I", INCLUDE, "-c", "-o", obj, src])
    with ThreadPoolExecutor(max_workers=max(1, len(jobs))) as pool:
        for cmd, said in zip(jobs, pool.map(lambda cmd: _run(cmd, verbose), jobs)):
            if cmd[-1] == HEAD_SOURCE:
                try:
                    check_head_registers(said)
                except RuntimeError:
                    os.unlink(cmd[-2])
                    raise
    _run([nvcc, *ARCH_FLAGS, "-shared", "-Xcompiler", "-fPIC", "-Xlinker", "-soname=" + os.path.basename(LIB), "-o", LIB,
          *objects])
    if force or _older(CALLS, max(headers, os.path.getmtime(CALLS_SOURCE))):
        _run(_calls_command())
    else:
        os.utime(CALLS)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
