"""In-tree build of libnvfp4_b200.so (hand-written sm_100a CUDA + the C ABI).

``python -m blackwell_diffusion_rtx6000_5090_i2v_b200.build`` compiles every
``csrc/*.cu`` with nvcc for ``sm_100a`` only and links one shared library next
to this file.  nvcc cross-compiles, so no GPU is needed to build.
"""
from __future__ import annotations

import glob
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libnvfp4_b200.so")
HOST = os.path.join(HERE, "_host_calls.so")     # the Python layer's native calls into LIB

NVCC_FLAGS = [
    "-std=c++17", "-O3", "-lineinfo",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-Xcompiler", "-fPIC", "-Xcompiler", "-fvisibility=hidden",
    "--expt-relaxed-constexpr",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found: the NVFP4 library cannot be built")


def _host_cxx() -> list[str]:
    # some images export CC/CXX pointing at a toolchain without its runtime specs
    return ["-ccbin", "/usr/bin/g++"] if os.path.exists("/usr/bin/g++") else []


def sources() -> list[str]:
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def is_stale() -> bool:
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + \
        [os.path.join(HERE, "..", "include", "nvfp4_b200.h")]
    return any(os.path.getmtime(d) > t for d in deps if os.path.exists(d))


def host_built_for() -> str:
    """What the extension module is bound to; it carries this text."""
    import torch
    return f"torch {torch.__version__}, Python {sys.version_info[0]}.{sys.version_info[1]}"


def host_is_stale() -> bool:
    deps = [os.path.join(CSRC, "host_calls.cpp"), os.path.join(HERE, "..", "include", "nvfp4_b200.h")]
    if not os.path.exists(HOST) or any(os.path.getmtime(d) > os.path.getmtime(HOST) for d in deps if os.path.exists(d)):
        return True
    with open(HOST, "rb") as f:
        return host_built_for().encode() not in f.read()


def build_host(force: bool = False) -> str:
    """The extension module that the Python layer calls the library through (needs torch's headers)."""
    if not force and not host_is_stale():
        return HOST
    src = os.path.join(CSRC, "host_calls.cpp")
    import sysconfig

    import torch
    from torch.utils import cpp_extension as ext
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else os.environ.get("CXX", "g++")
    include = [*ext.include_paths(), sysconfig.get_paths()["include"],
               os.path.join(os.path.dirname(os.path.dirname(_nvcc())), "include")]
    cmd = [cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           "-DTORCH_EXTENSION_NAME=_host_calls", "-DTORCH_API_INCLUDE_EXTENSION_H",
           f'-DNVFP4_BUILT_FOR="{host_built_for()}"',
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}",
           *[f for d in include for f in ("-isystem", d)], src, "-o", HOST,
           "-L", HERE, "-l:libnvfp4_b200.so", "-Wl,-rpath,$ORIGIN",
           *[f for d in ext.library_paths() for f in ("-L", d)],
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
    subprocess.run(cmd, check=True)
    return HOST


def build_library(force: bool = False, verbose: bool = False) -> str:
    if force or is_stale():
        _build_cuda(verbose)
    build_host(force)
    return LIB


def _build_cuda(verbose: bool) -> None:
    nvcc = _nvcc()
    objs = []
    for src in sources():
        obj = os.path.join(CSRC, os.path.basename(src)[:-3] + ".o")
        cmd = [nvcc, *_host_cxx(), *NVCC_FLAGS, "-c", src, "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
            print(" ".join(cmd), file=sys.stderr)
        subprocess.run(cmd, check=True)
        objs.append(obj)
    cmd = [nvcc, *_host_cxx(), "-shared", "-o", LIB, *objs, "-cudart", "static"]
    subprocess.run(cmd, check=True)


if __name__ == "__main__":
    print(build_library(force="--force" in sys.argv, verbose="-v" in sys.argv))
