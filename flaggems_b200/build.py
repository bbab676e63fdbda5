"""Build the C-ABI shared library with nvcc for sm_100a, and the native host module over it.

    python -m flaggems_b200.build [--force] [--verbose]

Produces ``flaggems_b200/lib/libflaggems_b200.so`` and ``lib/_fg_host.<python and torch>.so`` next to the
sources (in-tree, git-ignored).  nvcc cross-compiles without a GPU.  No fast-math flags: the
quantisation kernels rely on IEEE fp32 semantics.
"""
import argparse
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "lib")
LIB_PATH = os.path.join(LIB_DIR, "libflaggems_b200.so")
SOURCES = ["api.cu", "quant.cu", "moe_glue.cu", "moe_layer.cu", "router.cu", "gemm_fp8_sm100.cu"]
ARCH_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a"]


def _nvcc():
    cand = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(cand):
        raise RuntimeError("nvcc not found; the CUDA toolkit is required to build flaggems_b200")
    return cand


def _stale(path, sources):
    if not os.path.exists(path):
        return True
    deps = [os.path.join(CSRC, f) for f in sources]
    deps.append(os.path.join(os.path.dirname(HERE), "include", "flaggems_b200.h"))
    return any(os.path.getmtime(d) > os.path.getmtime(path) for d in deps)


def host_path():
    """File of the native host module for the running Python and torch: it is bound to the C++ interfaces of both,
    so another version of either needs a module of its own."""
    import torch

    return os.path.join(LIB_DIR, f"_fg_host.{sysconfig.get_config_var('SOABI')}.torch-{torch.__version__}"
                                 f".abi{int(torch._C._GLIBCXX_USE_CXX11_ABI)}.so")


def build(force=False, verbose=False):
    if force or _stale(LIB_PATH, [f for f in os.listdir(CSRC) if f != "host.cpp"]):
        build_library(verbose)
    if force or _stale(host_path(), ["host.cpp"]):
        build_host()
    return LIB_PATH


def build_host():
    """The CPython module over the library, against the headers of the installed torch."""
    import torch

    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    cxx = os.environ.get("CXX") or shutil.which("g++") or "c++"
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           f"-I{os.path.join(root, 'include')}", f"-I{os.path.join(root, 'include', 'torch', 'csrc', 'api', 'include')}",
           f"-I{os.path.join(cuda, 'include')}", f"-I{sysconfig.get_paths()['include']}",
           os.path.join(CSRC, "host.cpp"), "-o", host_path(), f"-L{os.path.join(root, 'lib')}",
           "-ltorch", "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-lc10", "-lc10_cuda",
           f"-L{LIB_DIR}", "-lflaggems_b200", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError("the native host module failed to build:\n" + r.stdout)


def build_library(verbose=False):
    os.makedirs(LIB_DIR, exist_ok=True)
    objs = []
    procs = []
    for src in SOURCES:
        obj = os.path.join(LIB_DIR, src.replace(".cu", ".o"))
        cmd = [_nvcc(), *ARCH_FLAGS, "-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC",
               "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas")
            cmd.insert(2, "-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            failed = True
            sys.stderr.write(f"--- nvcc failed on {src}\n{out}\n")
        elif verbose or out.strip():
            sys.stderr.write(f"--- {src}\n{out}\n")
    if failed:
        raise RuntimeError("nvcc compilation failed")
    link = [_nvcc(), *ARCH_FLAGS, "-shared", "-o", LIB_PATH, *objs]
    r = subprocess.run(link, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n" + r.stdout)


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
