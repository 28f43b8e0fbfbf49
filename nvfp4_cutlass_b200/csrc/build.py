"""Ahead-of-time build of libnvfp4_b200.so for sm_100a (no JIT, no other arch).

    python nvfp4_cutlass_b200/csrc/build.py [--force] [--verbose]

Each .cu is compiled to an object with nvcc, then linked into one shared library
next to the Python package (nvfp4_cutlass_b200/lib/libnvfp4_b200.so).  Objects are
rebuilt only when a source or header is newer.  binding.cpp becomes a CPython module
beside it (lib/_binding-torch<version>.<Python's ABI>.so), compiled with g++ against torch's headers.
The library itself needs the CUDA toolkit alone: where there is no torch with CUDA, or the module does not compile, the build says
so and goes on without it (a Python caller's GEMM calls then go through ctypes).
"""
from __future__ import annotations

import importlib.machinery
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.dirname(HERE)
OUT_DIR = os.path.join(PKG, "lib")
OBJ_DIR = os.path.join(HERE, "build")
LIB = os.path.join(OUT_DIR, "libnvfp4_b200.so")
SOURCES = ["abi.cu", "gemm_normal.cu", "gemm_cluster.cu", "gemm_split.cu", "gemm_swap.cu", "gemm_stream.cu", "moe_glue.cu", "quantize_weight.cu", "checkpoint_loader.cu", "debug_kernels.cu"]
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
HEADER = os.path.join(os.path.dirname(PKG), "include", "nvfp4_b200.h")
FLAGS = ["-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
         "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr",
         "-ccbin", "/usr/bin/g++"]


def _newest_header() -> float:
    hdrs = [os.path.join(HERE, f) for f in os.listdir(HERE) if f.endswith((".cuh", ".hpp"))]
    hdrs.append(HEADER)
    return max(os.path.getmtime(h) for h in hdrs)


def binding_path():
    """Where the module for this interpreter and the installed torch belongs: it reads tensors through both's C interfaces, so
    its name says which, and after an upgrade of either there is none until the next build (_C.py looks for the same name).
    None where there is no torch with CUDA to compile it against."""
    try:
        import torch
    except (ImportError, OSError):
        return None
    if torch.version.cuda is None:
        return None
    return os.path.join(OUT_DIR, f"_binding-torch{torch.__version__}{importlib.machinery.EXTENSION_SUFFIXES[0]}")


def _binding_command() -> list:
    import torch
    from torch.utils import cpp_extension

    include = [f"-I{d}" for d in (*cpp_extension.include_paths(), sysconfig.get_paths()["include"],
                                  os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include"))]
    libs = [f"-L{d}" for d in cpp_extension.library_paths()]      # loaded by torch before the module is imported
    return ["/usr/bin/g++", "-std=c++17", "-O2", "-fPIC", "-shared", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", *include, *libs,
            os.path.join(HERE, "binding.cpp"), "-o", binding_path(), "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OUT_DIR, exist_ok=True)
    os.makedirs(OBJ_DIR, exist_ok=True)
    hdr_time = _newest_header()
    jobs = []
    for src in SOURCES:
        s = os.path.join(HERE, src)
        o = os.path.join(OBJ_DIR, src.replace(".cu", ".o"))
        if force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), hdr_time):
            jobs.append((s, o))

    link = bool(jobs) or not os.path.exists(LIB)
    binding = os.path.join(HERE, "binding.cpp")
    target = binding_path()
    if target is None:
        print("no torch with CUDA: built without binding.cpp's module", file=sys.stderr)
    elif force or not os.path.exists(target) or os.path.getmtime(target) < max(os.path.getmtime(binding), os.path.getmtime(HEADER)):
        if os.path.exists(target):
            os.remove(target)                        # one that calls the library by an older header must not outlive a failed compile
        jobs.append((binding, target))

    def compile_one(job):
        s, o = job
        cmd = _binding_command() if s == binding else [NVCC, *FLAGS, *( ["-Xptxas", "-v"] if verbose else []), "-c", s, "-o", o]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0 and s == binding:
            print(f"built without binding.cpp's module, which did not compile:\n{r.stdout}\n{r.stderr}", file=sys.stderr)
        elif r.returncode != 0:
            raise RuntimeError(f"{cmd[0]} failed on {s}:\n{r.stdout}\n{r.stderr}")
        return r.stderr

    with ThreadPoolExecutor(max_workers=len(SOURCES) + 1) as ex:
        for log in ex.map(compile_one, jobs):
            if verbose and log:
                print(log)
    objs = [os.path.join(OBJ_DIR, s.replace(".cu", ".o")) for s in SOURCES]
    if link:
        cmd = [NVCC, "-shared", "-o", LIB, *objs, "-ccbin", "/usr/bin/g++", "-Xlinker", "--exclude-libs,ALL"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
