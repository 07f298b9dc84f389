"""Builds ``lisa_b200/lib/liblisa_cuda.so`` from ``lisa_b200/csrc`` with nvcc for sm_100a, and beside it
``_lisa_torch.so``, the compiled host side of ``lisa_b200.ops``.

The library is plain CUDA C++ behind the C ABI of ``include/lisa_cuda.h``: no torch, no
Python in it.  nvcc cross-compiles without a GPU.  Run as ``python -m lisa_b200.build``.
"""
from __future__ import annotations

import concurrent.futures as cf
import hashlib
import os
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIBDIR = os.path.join(PKG, "lib")
OBJDIR = os.path.join(PKG, "build")
LIB = os.path.join(LIBDIR, "liblisa_cuda.so")

TORCH_LIB = os.path.join(LIBDIR, "_lisa_torch.so")
TORCH_SOURCE = "torch_ops.cpp"

SOURCES = ["api.cu", "qmv_affine.cu", "qmv_tc.cu", "qmv_dp.cu", "qmv_mm.cu", "qmv_i8.cu", "qmm_affine.cu", "qmm_pair.cu", "dequantize.cu", "gather_qmm.cu", "gguf_matvec.cu", "gguf_dp.cu", "gguf_mm.cu",
           "moe.cu", "moe_decode.cu", "moe_dp.cu", "moe_mm.cu", "norm.cu", "typed.cu", "ep.cu", "tensor_map.cu", "files.cpp"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "include"), "-I", CSRC]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _stamp(paths) -> str:
    """What the two libraries are made of: sources, flags, and for the torch extension the torch and Python whose ABI it uses.  The
    folder of the checkout is left out: a copy of a built tree is built."""
    import sysconfig

    import torch

    h = hashlib.sha256()
    for p in sorted(paths):
        with open(p, "rb") as f:
            h.update(os.path.relpath(p, ROOT).encode())
            h.update(f.read())
    line = " ".join([*NVCC_FLAGS, torch.__version__, sysconfig.get_config_var("SOABI") or "", *_torch_command()])
    h.update(line.replace(ROOT, "").encode())
    return h.hexdigest()


def _compile(src: str, verbose: bool) -> str:
    obj = os.path.join(OBJDIR, os.path.splitext(src)[0] + ".o")
    cmd = [_nvcc(), *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{res.stdout}\n{res.stderr}")
    if verbose:
        sys.stderr.write(res.stderr)
    return obj


def _torch_command() -> list[str]:
    """g++ over csrc/torch_ops.cpp against torch's headers; links liblisa_cuda.so from its own folder."""
    import sysconfig

    import torch
    from torch.utils import cpp_extension

    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           os.path.join(CSRC, TORCH_SOURCE), "-o", TORCH_LIB, "-I", os.path.join(ROOT, "include"), "-isystem", sysconfig.get_paths()["include"],
           "-isystem", "/usr/local/cuda/include"]
    for path in cpp_extension.include_paths():
        cmd += ["-isystem", path]
    for path in cpp_extension.library_paths():
        cmd += ["-L", path]
    cmd += ["-L", LIBDIR, "-l:liblisa_cuda.so", "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python",
            "-Wl,-rpath,$ORIGIN"]
    return cmd


def _torch_extension() -> str:
    res = subprocess.run(_torch_command(), capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"g++ failed for {TORCH_SOURCE}:\n{res.stdout}\n{res.stderr}")
    return TORCH_LIB


def _refuse_if_loaded() -> None:
    """A process that has loaded a library keeps it: built anew under it, its calls would go on running the old code."""
    cabi = sys.modules.get(f"{os.path.basename(PKG)}._cabi")
    if cabi is not None and cabi._lib is not None:
        raise RuntimeError(f"{LIB} is out of date, and this process has already loaded it: build it in a process of its own "
                           "(`python -m lisa_b200.build`) and start again")


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(LIBDIR, exist_ok=True)
    os.makedirs(OBJDIR, exist_ok=True)
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC)] + [os.path.join(ROOT, "include", f) for f in os.listdir(os.path.join(ROOT, "include"))]
    stamp = _stamp(deps)
    stamp_file = os.path.join(OBJDIR, "stamp")
    if not force and os.path.exists(LIB) and os.path.exists(TORCH_LIB) and os.path.exists(stamp_file) and open(stamp_file).read() == stamp:
        return LIB
    _refuse_if_loaded()
    with cf.ThreadPoolExecutor(max_workers=min(8, len(SOURCES))) as ex:
        objs = list(ex.map(lambda s: _compile(s, verbose), SOURCES))
    cmd = [_nvcc(), "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a", "-cudart", "static"]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError(f"link failed:\n{res.stdout}\n{res.stderr}")
    _torch_extension()
    with open(stamp_file, "w") as f:
        f.write(stamp)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
