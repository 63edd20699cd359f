"""Build the CUDA library in-tree: nvcc for sm_100a only, one shared object `libdm_b200.so` next to this file, and the
Python extension `_dm_native.so` (csrc/dm_torch.cpp: the eager route of the attention functions against torch's C++ API).

    python -m delta_matching_b200.build [--force] [--verbose]

The library exports the C ABI declared in include/dm_b200.h and links only against the CUDA runtime (the driver entry
point for tensor-map encoding is resolved at run time), so it builds on a machine without a GPU.
"""
from __future__ import annotations

import hashlib
import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libdm_b200.so")
SOURCES = ("dm_abi.cu", "dm_quant.cu", "dm_fwd.cu", "dm_fwd_teams.cu", "dm_delta.cu", "dm_bwd_kv.cu", "dm_bwd_pipe.cu", "dm_bwd_tiles.cu", "dm_bwd.cu", "dm_bwd_p2.cu", "dm_probe.cu", "dm_static_scratch.cu")
NATIVE = os.path.join(HERE, "_dm_native.so")
NATIVE_SOURCE = "dm_torch.cpp"
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.sep not in cand or os.path.isfile(cand)):
            return cand
    return "nvcc"


def source_files():
    out = []
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h", ".cpp")):
            out.append(os.path.join(CSRC, f))
    out.append(os.path.join(os.path.dirname(HERE), "include", "dm_b200.h"))
    return out


def code_sha() -> str:
    """12 hex characters of a hash over the kernel sources (the stamp kernel_version() reports)."""
    h = hashlib.sha256()
    for f in source_files():
        if os.path.isfile(f):
            h.update(os.path.basename(f).encode())
            h.update(open(f, "rb").read())
    return h.hexdigest()[:12]


def _build_native(verbose: bool) -> None:
    """g++ against the installed torch's headers; the module finds torch's libraries already loaded (it is imported behind
    torch) and takes the kernel library's entry points as addresses, so it links neither by path.

    The C++ runtime is named as the shared library that torch uses: a compiler without a libstdc++.so of its own links the
    static one, and an exception that leaves the module's copy for torch's autograd engine ends the process."""
    import sysconfig
    import torch
    from torch.utils import cpp_extension
    inc = [f for d in (*cpp_extension.include_paths(), sysconfig.get_path("include"), "/usr/local/cuda/include") for f in ("-isystem", d)]
    lib_dir = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", *inc, os.path.join(CSRC, NATIVE_SOURCE), "-o", NATIVE,
           f"-L{lib_dir}", "-ltorch_python", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-lc10", "-lc10_cuda",
           "-nostdlib++", "-l:libstdc++.so.6", "-lm"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"g++ failed for {NATIVE_SOURCE}:\n{r.stdout}\n{r.stderr[-6000:]}")
    if verbose:
        sys.stderr.write(r.stderr)


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile and link (skipped when a stamp says that the libraries come from these sources and this recipe)."""
    obj_dir = OBJ
    lib = LIB
    os.makedirs(obj_dir, exist_ok=True)
    stamp = os.path.join(obj_dir, "stamp.txt")
    sha = code_sha() + " " + hashlib.sha256(open(__file__, "rb").read()).hexdigest()[:12]
    if not force and os.path.isfile(lib) and os.path.isfile(NATIVE) and os.path.isfile(stamp) and open(stamp).read().strip() == sha:
        return lib
    srcs = list(SOURCES)
    nvcc = _nvcc()
    flags = NVCC_FLAGS

    def compile_one(src):
        obj = os.path.join(obj_dir, src[:-3] + ".o")
        cmd = [nvcc, *flags, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed for {src}:\n{r.stdout}\n{r.stderr}")
        if verbose:
            sys.stderr.write(r.stderr)
        return obj

    with ThreadPoolExecutor(max_workers=min(8, len(srcs) + 1)) as ex:
        native = ex.submit(_build_native, verbose)
        objs = list(ex.map(compile_one, srcs))
        native.result()
    r = subprocess.run([nvcc, "-shared", "-o", lib, *objs, "-lcudart"], capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    with open(stamp, "w") as fh:
        fh.write(sha + "\n")
    return lib


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
