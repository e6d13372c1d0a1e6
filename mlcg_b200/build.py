"""Compile the CUDA sources of this package into ``libmlcg_b200.so`` (sm_100a only, in-tree).

``python -m mlcg_b200.build`` builds if anything is out of date; ``--force`` rebuilds. nvcc
cross-compiles without a GPU, so the build also runs on a CPU-only machine.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libmlcg_b200.so")
NATIVE, NATIVE_SRC = os.path.join(HERE, "_native.so"), os.path.join(CSRC, "host.cpp")      # host side (torch's C++ interface, no device code)
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "--use_fast_math=false",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-O3"]
NVCC_FLAGS = [f for f in NVCC_FLAGS if f != "--use_fast_math=false"]


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _deps():
    hdrs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    return sources() + hdrs + [os.path.join(os.path.dirname(HERE), "include", "mlcg_b200.h")]


def _native_up_to_date() -> bool:
    deps = [NATIVE_SRC, os.path.join(os.path.dirname(HERE), "include", "mlcg_b200.h")]
    return os.path.exists(NATIVE) and all(os.path.getmtime(NATIVE) >= os.path.getmtime(p) for p in deps)


def _native_command():
    import sysconfig

    import torch
    root = os.path.dirname(torch.__file__)
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"), sysconfig.get_paths()["include"],
               os.path.join(os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"))), "include")]
    libs = os.path.join(root, "lib")
    return (["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-DTORCH_API_INCLUDE_EXTENSION_H", "-DTORCH_EXTENSION_NAME=_native",
             f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}"] + [f"-I{d}" for d in include] +
            [NATIVE_SRC, "-o", NATIVE, f"-L{libs}", f"-Wl,-rpath,{libs}", "-ltorch", "-ltorch_cpu", "-ltorch_python", "-lc10"])


def up_to_date() -> bool:
    return _native_up_to_date() and os.path.exists(LIB) and all(os.path.getmtime(LIB) >= os.path.getmtime(p) for p in _deps())


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and up_to_date():
        return LIB
    nvcc = os.environ.get("NVCC", "nvcc")
    objdir = os.path.join(HERE, "build")
    os.makedirs(objdir, exist_ok=True)
    procs, objs = [], []
    if force or not _native_up_to_date():
        procs.append((NATIVE_SRC, subprocess.Popen(_native_command(), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for src in sources():
        obj = os.path.join(objdir, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        if not force and os.path.exists(obj) and all(os.path.getmtime(obj) >= os.path.getmtime(p) for p in [src] + [d for d in _deps() if not d.endswith(".cu")]):
            continue
        cmd = [nvcc] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            sys.stderr.write(out)
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("the compiler failed")
    subprocess.check_call([nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB] + objs + ["-lcudart"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
