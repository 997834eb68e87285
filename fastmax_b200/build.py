"""Builds the native parts of fastmax_b200 in-tree for sm_100a.

``python -m fastmax_b200.build`` compiles

* ``fastmax_b200/libfastmax_b200.so`` -- the CUDA kernels and the C ABI declared
  in ``include/fastmax_b200.h`` (plain nvcc, no torch dependency), and
* with ``--torch-ext`` (they need the torch headers and take a minute), the torch
  C++ extensions ``fastmax_cuda*.so``, which exposes the reference's
  ``forwardpass`` / ``backwardpass`` entry points on top of that C ABI, and
  ``fastmax_b200/_host*.so``, the host side of the package's frequent calls.

nvcc cross-compiles without a GPU, so the build runs anywhere the CUDA toolkit
is installed.
"""
from __future__ import annotations

import glob
import os
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
LIB = os.path.join(PKG, "libfastmax_b200.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC,
]


def _newer(target: str, sources) -> bool:
    if not os.path.exists(target):
        return False
    t = os.path.getmtime(target)
    return all(os.path.getmtime(s) <= t for s in sources)


def build_library(force: bool = False, verbose: bool = False) -> str:
    """Compile every ``csrc/*.cu`` into the shared library; returns its path."""
    cus = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    deps = cus + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(ROOT, "include", "*.h"))
    if not force and _newer(LIB, deps):
        return LIB
    objs = []
    procs = []
    os.makedirs(os.path.join(PKG, "build"), exist_ok=True)
    for cu in cus:
        obj = os.path.join(PKG, "build", os.path.basename(cu)[:-3] + ".o")
        objs.append(obj)
        if not force and _newer(obj, [cu] + deps[len(cus):]):
            continue
        cmd = ["nvcc"] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", cu, "-o", obj]
        procs.append((cu, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    for cu, pr in procs:
        out, _ = pr.communicate()
        if verbose or pr.returncode:
            sys.stderr.write(out)
        if pr.returncode:
            raise RuntimeError(f"nvcc failed on {cu}")
    subprocess.check_call(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-o", LIB]
                          + objs + ["-lcudart", "-lcuda"])
    return LIB


def build_torch_extension(force: bool = False) -> str:
    """Compile the ``fastmax_cuda`` extension next to the package and ``_host`` inside it; returns the former's path."""
    import sysconfig

    build_library()
    suffix = sysconfig.get_config_var("EXT_SUFFIX")
    targets = [("torch_binding.cpp", "fastmax_cuda", ROOT, "$ORIGIN/fastmax_b200"), ("host_binding.cpp", "_host", PKG, "$ORIGIN")]
    procs = []
    for source, name, folder, rpath in targets:
        src, target = os.path.join(CSRC, source), os.path.join(folder, name + suffix)
        if force or not _newer(target, [src, os.path.join(ROOT, "include", "fastmax_b200.h")]):
            procs.append(subprocess.Popen(_extension_command(src, name, target, rpath)))
    for pr in procs:
        if pr.wait():
            raise subprocess.CalledProcessError(pr.returncode, pr.args)
    return os.path.join(ROOT, "fastmax_cuda" + suffix)


def _extension_command(src: str, name: str, target: str, rpath: str):
    import sysconfig

    import torch
    from torch.utils import cpp_extension

    inc = cpp_extension.include_paths("cuda")
    tlib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", f"-DTORCH_EXTENSION_NAME={name}",
           "-DTORCH_API_INCLUDE_EXTENSION_H", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
           "-I" + os.path.join(ROOT, "include"), "-I" + sysconfig.get_paths()["include"]]
    cmd += ["-I" + p for p in inc]
    return cmd + [src, "-o", target, "-L" + tlib, "-L" + PKG, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
                  "-ltorch", "-ltorch_python", "-l:libfastmax_b200.so", "-L/usr/local/cuda/lib64", "-lcudart",
                  "-Wl,-rpath," + rpath, "-Wl,-rpath," + tlib]


if __name__ == "__main__":
    force = "--force" in sys.argv
    print(build_library(force=force, verbose="-v" in sys.argv))
    if "--torch-ext" in sys.argv:
        print(build_torch_extension(force=force))
