"""Builds libb200_qlinear.so (the C-ABI library) and libb200_qlinear.a (the same objects as a static archive, for hosts
that link statically) from csrc/*.cu with nvcc, for sm_100a only, then _host_ops.so, the CPython extension behind
linear.py's hot calls. The libraries need nvcc and nothing else; the extension needs torch and is left out, with a note, where
torch cannot be imported (a Rust or C host), or with --c-only. The name differs on purpose from the reference's own static
library `gpu_kernels`, which keeps supplying every symbol this library does not replace.

The GEMM uses tcgen05.mma kind::i8, which exists on sm_100a and not on sm_103a or sm_120: no other -gencode
may be added. No fast-math: the rounding points of the quantizer and of the epilogue are part of the contract.
"""
from __future__ import annotations

import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libb200_qlinear.so")
ARCHIVE = os.path.join(HERE, "libb200_qlinear.a")
HOST_OPS = os.path.join(HERE, "_host_ops.so")      # linear.py's hot calls (csrc/host_ops.cpp), linked against LIB and torch
UNITS = ["quant_rows", "gemm_i8", "gemm_skinny", "weight_pack"]
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
         "-Xcompiler", "-fPIC,-fvisibility=hidden", "-I" + CSRC, "-I" + os.path.join(os.path.dirname(HERE), "include")]


def _stale(target: str, deps: list[str]) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _host_ops_stamp(torch) -> str:
    """What an extension is bound to: the interpreter's ABI and the very torch it was linked against."""
    return "\n".join([sys.implementation.cache_tag, torch.__version__, os.path.dirname(os.path.abspath(torch.__file__)),
                      f"cxx11_abi={int(torch.compiled_with_cxx11_abi())}"])


def _host_ops(force: bool, verbose: bool) -> None:
    """csrc/host_ops.cpp -> HOST_OPS, against the headers and libraries of the torch that will import it."""
    try:
        import torch
    except ImportError as e:
        sys.stderr.write(f"{os.path.basename(HOST_OPS)} left out: torch cannot be imported ({e}); {LIB} does not need it\n")
        return
    src = os.path.join(CSRC, "host_ops.cpp")
    stamp = os.path.join(OBJ, "host_ops.torch")
    bound = _host_ops_stamp(torch)
    fresh = os.path.exists(stamp) and open(stamp).read() == bound
    if not force and fresh and not _stale(HOST_OPS, [src, os.path.abspath(__file__), os.path.join(os.path.dirname(HERE), "include", "gpu_kernels.h")]):
        return
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(NVCC))
    dirs = [os.path.join(os.path.dirname(HERE), "include"), os.path.join(root, "include"),
            os.path.join(root, "include", "torch", "csrc", "api", "include"), os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    cmd = ["g++", "-shared", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", src, "-o", HOST_OPS]
    cmd += [f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"] + ["-I" + d for d in dirs]
    cmd += ["-L" + HERE, "-l:" + os.path.basename(LIB), "-Wl,-rpath,$ORIGIN", "-L" + os.path.join(root, "lib"), "-ltorch_python", "-ltorch_cpu",
            "-lc10", "-lc10_cuda"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode:
        sys.stderr.write(r.stdout + r.stderr)
    if r.returncode:
        raise RuntimeError("g++ failed on host_ops.cpp")
    with open(stamp, "w") as f:
        f.write(bound)


def build(force: bool = False, verbose: bool = False, c_only: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h", ".inl"))]
    headers.append(os.path.abspath(__file__))

    def compile_unit(u: str) -> str:
        src, obj = os.path.join(CSRC, u + ".cu"), os.path.join(OBJ, u + ".o")
        if force or _stale(obj, [src] + headers):
            cmd = [NVCC, "-c", src, "-o", obj] + FLAGS + (["-Xptxas", "-v"] if verbose else [])
            r = subprocess.run(cmd, capture_output=True, text=True)
            if verbose or r.returncode:
                sys.stderr.write(r.stdout + r.stderr)
            if r.returncode:
                raise RuntimeError(f"nvcc failed on {u}.cu")
        return obj

    with ThreadPoolExecutor(max_workers=len(UNITS)) as ex:
        objs = list(ex.map(compile_unit, UNITS))
    if force or _stale(LIB, objs):
        subprocess.check_call([NVCC, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"])
    if force or _stale(ARCHIVE, objs):
        if os.path.exists(ARCHIVE):
            os.remove(ARCHIVE)
        subprocess.check_call(["ar", "rcs", ARCHIVE] + objs)
    if not c_only:
        _host_ops(force, verbose)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv, c_only="--c-only" in sys.argv))
