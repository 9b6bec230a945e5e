"""Builds liblbk.so (the CUDA kernels and their C ABI) in-tree with nvcc for sm_100a, and held_arrays, a small extension module
of the Python package."""
import os
import re
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB = os.path.join(HERE, "liblbk.so")
SOURCES = ["context.cu", "proposals.cu", "quantise.cu", "histogram.cu", "split.cu", "partition.cu",
           "predict.cu", "predict_ranked.cu", "update_tree.cu", "objective.cu", "exchange.cu", "small_tree.cu", "build_tree.cu"]
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
         "-Xcompiler", "-fPIC", "-fmad=false", "-I", INCLUDE, "-I", CSRC]


def _newer(target, deps):
    if not os.path.exists(target):
        return False
    t = os.path.getmtime(target)
    return all(os.path.getmtime(d) <= t for d in deps)


def module_name(torch_version=None) -> str:
    """Name of held_arrays as built for a version of torch (this one's).  The module uses torch's C++ classes, whose layout is
    compiled in: another torch, and by the file's suffix another Python, has a module of its own and never loads this one."""
    if torch_version is None:
        import torch

        torch_version = torch.__version__
    return "held_arrays_torch_" + re.sub(r"\W", "_", str(torch_version))


def module_path(torch_version=None) -> str:
    return os.path.join(HERE, module_name(torch_version) + sysconfig.get_config_var("EXT_SUFFIX"))


def build(force: bool = False, verbose: bool = False) -> str:
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".h", ".cuh"))]
    headers.append(os.path.join(INCLUDE, "lbk.h"))
    objs = []
    jobs = []
    for src in SOURCES:
        s = os.path.join(CSRC, src)
        o = os.path.join(CSRC, src.replace(".cu", ".o"))
        objs.append(o)
        if force or not _newer(o, [s] + headers):
            cmd = [NVCC] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("the build failed:\n" + " ".join(cmd) + "\n" + r.stdout + r.stderr)
        return r.stderr

    if jobs:
        with ThreadPoolExecutor(max_workers=8) as ex:
            for out in ex.map(run, jobs):
                if verbose and out:
                    print(out)
    if jobs or not os.path.exists(LIB):
        run([NVCC, "-shared", "-o", LIB] + objs + ["-lcudart", "-ldl"])
    source = os.path.join(CSRC, "held_arrays.cpp")
    if force or not _newer(module_path(), [source]):
        from torch.utils import cpp_extension

        # (torch has loaded the libraries it names before it is imported)
        run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", source, "-o", module_path()]
            + ["-DLBK_MODULE=" + module_name()]
            + ["-I" + d for d in cpp_extension.include_paths() + [sysconfig.get_paths()["include"]]]
            + ["-L" + d for d in cpp_extension.library_paths()] + ["-ltorch_python", "-ltorch_cpu", "-lc10"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
