"""Builds libsbattn.so (sm_100a only, nvcc) and _binding.so (the PyTorch layer's native host path, g++) next to this file.
Usage: python -m stickbreaking_attention_b200.build"""
import glob
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
LIB = os.path.join(HERE, "libsbattn.so")
BINDING = os.path.join(HERE, "_binding.so")
BINDING_SRC = os.path.join(HERE, "csrc", "sb_torch.cpp")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "--use_fast_math",
         "-Xcompiler", "-fPIC"]
# the kernels of float32 precision, which need accurate exponentials, denormal numbers and IEEE division: compiled without --use_fast_math
PRECISE = {"sb_f32.cu", "sb_f32_tc.cu", "sb_weights.cu"}


def sources():
    return sorted(glob.glob(os.path.join(HERE, "csrc", "*.cu")))


def stale():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = sources() + glob.glob(os.path.join(HERE, "csrc", "*.cuh")) + glob.glob(
        os.path.join(HERE, "..", "include", "*.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def built_for():
    """What _binding.so depends on besides its sources: the PyTorch and Python it was compiled against (compiled into it)."""
    import sysconfig
    import torch
    return f"sbattn binding for torch {torch.__version__}, python {sysconfig.get_config_var('SOABI')}, " \
           f"cxx11 abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)}."


def binding_stale():
    if not os.path.exists(BINDING):
        return True
    with open(BINDING, "rb") as f:
        if built_for().encode() not in f.read():
            return True
    t = os.path.getmtime(BINDING)
    return any(os.path.getmtime(d) > t for d in [BINDING_SRC] + glob.glob(os.path.join(HERE, "..", "include", "*.h")))


def build_binding():
    """_binding.so refers to libsbattn.so by name, so that has been built before, and finds it beside itself ($ORIGIN)."""
    import sysconfig
    import torch
    from torch.utils.cpp_extension import CUDA_HOME, include_paths
    libdir = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = CUDA_HOME or "/usr/local/cuda"
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_binding",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DSBATTN_BUILT_FOR="{built_for()}"']
    cmd += [f"-isystem{d}" for d in include_paths() + [sysconfig.get_paths()["include"], os.path.join(cuda, "include")]]
    cmd += [BINDING_SRC, "-o", BINDING, f"-L{libdir}", "-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python",
            "-L" + HERE, "-l:libsbattn.so", "-Wl,-rpath,$ORIGIN"]
    pr = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if pr.returncode != 0:
        sys.stderr.write(pr.stdout)
        raise RuntimeError("g++ failed")


def build(force=False, verbose=False):
    if force or stale():
        build_library(verbose)
    if force or binding_stale():
        build_binding()
    return LIB


def build_library(verbose):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: cannot build libsbattn.so")
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    objs = []
    procs = []
    for src in sources():
        obj = os.path.join(objdir, os.path.basename(src)[:-3] + ".o")
        flags = [f for f in FLAGS if not (f == "--use_fast_math" and os.path.basename(src) in PRECISE)]
        cmd = [nvcc] + flags + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    failed = False
    for src, pr in procs:
        out, _ = pr.communicate()
        if verbose or pr.returncode != 0:
            sys.stderr.write(out)
        failed |= pr.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    subprocess.check_call([nvcc, "-shared", "-Xlinker", "-soname=libsbattn.so", "-o", LIB] + objs)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
