"""Build libniti_b200.so in-tree with nvcc for sm_100a (cross-compiles without a GPU), and _torch_ops.so, the native
torch front end over it, with g++ against torch's headers.

    python -m niti_b200.build            # rebuild if any source is newer than the library
    python -m niti_b200.build --force
"""
import os
import shutil
import subprocess
import sys
import sysconfig
from importlib import metadata

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libniti_b200.so")
OPS = os.path.join(PKG, "_torch_ops.so")
SOURCES = ["api.cu", "umma_kernels.cu", "simt_kernels.cu", "head_kernels.cu"]
NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden", "--expt-relaxed-constexpr"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the CUDA kernels of niti_b200 cannot be built")


def _stale(target, deps):
    return not os.path.exists(target) or any(os.path.getmtime(d) > os.path.getmtime(target) for d in deps)


def needs_build():
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))]
    return _stale(LIB, deps + [os.path.join(os.path.dirname(PKG), "include", "niti_b200.h")])


def build(force=False, verbose=False):
    if force or needs_build():
        nvcc = _nvcc()
        objs = []
        for src in SOURCES:
            obj = os.path.join(CSRC, src.replace(".cu", ".o"))
            cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
            if verbose:
                cmd.insert(1, "-Xptxas=-v")
            subprocess.run(cmd, check=True)
            objs.append(obj)
        subprocess.run([nvcc, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"], check=True)
    build_ops(force)
    return LIB


def ops_tag():
    """What the front end is tied to besides its source: torch's C++ classes and the interpreter's ABI."""
    return f"torch {metadata.version('torch')}, {sysconfig.get_config_var('SOABI')}"


def ops_stale():
    """Whether _torch_ops.so has to be built: no file, older than its sources, or built for another torch or interpreter (the
    tag is compiled into the module's docstring, so a torch that was exchanged underneath is noticed without loading it)."""
    if _stale(OPS, [os.path.join(CSRC, "torch_ops.cpp"), os.path.join(os.path.dirname(PKG), "include", "niti_b200.h")]):
        return True
    with open(OPS, "rb") as f:
        return f"({ops_tag()})\0".encode() not in f.read()


def build_ops(force=False):
    """The CPython module niti_b200._torch_ops: links against the library beside it (rpath $ORIGIN) and the installed torch."""
    src = os.path.join(CSRC, "torch_ops.cpp")
    if not force and not ops_stale():
        return OPS
    import torch
    base = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    incs = [os.path.join(base, "include"), os.path.join(base, "include", "torch", "csrc", "api", "include"),
            sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wno-interference-size", "-fPIC", "-shared", "-fvisibility=hidden",
                    f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", f'-DNITI_OPS_TAG="{ops_tag()}"', *["-I" + d for d in incs], src, "-o", OPS,
                    "-L" + PKG, "-l:libniti_b200.so", "-L" + os.path.join(base, "lib"), "-lc10", "-ltorch_cpu", "-ltorch_python",
                    "-lc10_cuda", "-ltorch_cuda", "-Wl,-rpath,$ORIGIN"], check=True)
    return OPS


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
