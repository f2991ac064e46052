"""Ahead-of-time build of the CUDA library: nvcc, sm_100a only, in tree.

    python -m pariskv_b200.build [--force]

produces ``pariskv_b200/libpariskv_b200.so`` from every source under ``csrc/`` and its CPython binding
``pariskv_b200/_native.so`` from ``csrc_py/bind.cpp``.  nvcc cross-compiles without a GPU, so this also runs on a build
machine.
"""
import glob
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libpariskv_b200.so")
NATIVE = os.path.join(HERE, "_native.so")
NATIVE_SRC = os.path.join(HERE, "csrc_py", "bind.cpp")
HEADER = os.path.join(HERE, "..", "include", "pariskv_b200.h")

NVCC_FLAGS = [
    "-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-O3",
]


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cpp")))


def _stale():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + [HEADER]
    return any(os.path.getmtime(d) > t for d in deps)


def _native_stale():
    return not os.path.exists(NATIVE) or any(os.path.getmtime(d) > os.path.getmtime(NATIVE) for d in (NATIVE_SRC, HEADER))


def _build_native():
    """The binding against the installed torch; needs libpariskv_b200.so to link to."""
    import sysconfig

    import torch
    home = os.path.dirname(torch.__file__)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(nvcc)))
    inc = [os.path.join(home, "include"), os.path.join(home, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda, "include"), sysconfig.get_paths()["include"]]
    subprocess.check_call(
        ["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden",
         f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}"] + [f"-I{i}" for i in inc] +
        [NATIVE_SRC, "-o", NATIVE, "-L" + HERE, "-lpariskv_b200", "-L" + os.path.join(home, "lib"), "-lc10", "-lc10_cuda",
         "-ltorch_cpu", "-ltorch_cuda", "-ltorch_python", "-Wl,-rpath,$ORIGIN"])


def build(force: bool = False, verbose: bool = False) -> str:
    """Compile what is missing or older than its sources; returns the path of the CUDA library."""
    if force or _stale():
        _build_lib(verbose)
    if force or _native_stale():
        _build_native()
    return LIB


def _build_lib(verbose):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found: cannot build libpariskv_b200.so")
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    procs = []
    objs = []
    for src in sources():
        obj = os.path.join(objdir, os.path.basename(src) + ".o")
        objs.append(obj)
        cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-x", "cu", "-c", src, "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}")
    subprocess.check_call([nvcc, "-shared", "-o", LIB] + objs + ["-lpthread", "-Xlinker", "-soname=libpariskv_b200.so"])


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
