"""Builds librwkvb200.so (the C-ABI library) in-tree with nvcc for sm_100a, and _native.so, the host side of the
training classes that sits between PyTorch and that library.

    python rwkv-cuda_b200/build.py [--force] [--verbose]

The library has no dependency on PyTorch (it links the CUDA runtime only); _native.so links both.
"""
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
CSRC_PY = os.path.join(HERE, "csrc_py")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "librwkvb200.so")
NATIVE = os.path.join(HERE, "_native.so")

ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
COMMON = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]
# per-file extras; the fp32-tolerance operators are built without fast-math
EXTRA = {
    "wkv4.cu": [],
    "timex.cu": [],
}


def sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _nvcc():
    return shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def _stamp(roots=(CSRC, os.path.join(HERE, "..", "include")), extra=()):
    h = hashlib.sha256()
    for root in roots:
        for f in sorted(os.listdir(root)):
            if f.endswith((".cu", ".cuh", ".h", ".cpp")):
                h.update(f.encode())
                h.update(open(os.path.join(root, f), "rb").read())
    h.update(repr((ARCH, COMMON, EXTRA, extra)).encode())
    return h.hexdigest()


def build_native(force=False):
    """g++ csrc_py/native.cpp against the installed PyTorch -> _native.so (finds librwkvb200.so beside itself)."""
    import torch
    from torch.utils.cpp_extension import include_paths, library_paths
    stamp_file = os.path.join(OBJ, "stamp_native")
    stamp = _stamp((CSRC_PY, os.path.join(HERE, "..", "include")), (torch.__version__, sysconfig.get_path("include")))
    if not force and os.path.exists(NATIVE) and os.path.exists(stamp_file) and open(stamp_file).read() == stamp:
        return
    libs = [f"-L{d}" for d in library_paths("cuda")] + [f"-Wl,-rpath,{library_paths('cuda')[0]}"]
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_native",
                    f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
                    *[f"-isystem{d}" for d in (*include_paths("cuda"), sysconfig.get_path("include"))],
                    os.path.join(CSRC_PY, "native.cpp"), "-o", NATIVE, LIB, "-Wl,-rpath,$ORIGIN", *libs,
                    "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python"], check=True)
    open(stamp_file, "w").write(stamp)


def build(force=False, verbose=False):
    """Compile every .cu under csrc/, link librwkvb200.so and build _native.so; each is skipped when its sources are unchanged."""
    _build_library(force, verbose)
    build_native(force)
    return LIB


def _build_library(force, verbose):
    os.makedirs(OBJ, exist_ok=True)
    stamp_file = os.path.join(OBJ, "stamp")
    stamp = _stamp()
    if not force and os.path.exists(LIB) and os.path.exists(stamp_file) and open(stamp_file).read() == stamp:
        return
    nvcc = _nvcc()
    procs = []
    objs = []
    for src in sources():
        obj = os.path.join(OBJ, src[:-3] + ".o")
        objs.append(obj)
        cmd = [nvcc, *ARCH, *COMMON, *EXTRA.get(src, []), "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd), flush=True)
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0 or verbose:
            print(f"---- {src} ----\n{out}", flush=True)
        failed |= p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    cmd = [nvcc, *ARCH, "-shared", "-Xlinker", "-soname=librwkvb200.so", "-o", LIB, *objs, "-lcudart"]
    subprocess.run(cmd, check=True)
    open(stamp_file, "w").write(stamp)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
