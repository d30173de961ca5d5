"""Compile the CUDA sources into `deconver_b200/libndc_b200.so` for sm_100a with nvcc, and the
layer's native host path (`csrc/ndc_torch.cpp`, on that library and PyTorch's C++ API) into
`deconver_b200/_ndc_torch.so` with the host compiler.

Both are built in-tree (next to this file) so that they travel with the source tree.
nvcc cross-compiles without a GPU.  The marching kernels are compiled as six translation units
(forward / backward of volumes / backward of images, each for float32 and bfloat16) and the tile
kernels as two, next to the ABI unit and those of the instance norm, the bias passes, the projection
and the tensor-core kernels, in parallel, then linked.  Run as `python -m deconver_b200._build [--force]`.
"""

import importlib.metadata
import os
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

PKG = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(PKG)
CSRC = os.path.join(PKG, "csrc")
INCLUDE = os.path.join(ROOT, "include")
LIB = os.path.join(PKG, "libndc_b200.so")
EXT = os.path.join(PKG, "_ndc_torch.so")
EXT_SRC = os.path.join(CSRC, "ndc_torch.cpp")
EXT_KEY = os.path.join(PKG, "_ndc_torch.key")     # what the extension was built for; travels with it
OBJ = os.path.join(PKG, "_obj")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "-Xfatbin=-compress-all",
]

# (object name, source, extra defines)
UNITS = [("abi", "ndc_abi.cu", []), ("inorm", "ndc_inorm.cu", []), ("bias", "ndc_bias.cu", []),
         ("proj", "ndc_proj.cu", []), ("tc", "ndc_tc.cu", [])] + [
    ("tile_t%d" % t, "ndc_tile_inst.cu", ["-DNDC_TILE_T=%d" % t]) for t in (0, 1)] + [
    ("dw4_p%d_t%d" % (part, t), "ndc_dw4_inst.cu", ["-DNDC_DW4_PART=%d" % part, "-DNDC_DW4_T=%d" % t])
    for part in (1, 2, 0) for t in (0, 1)   # the longest units first
]


def sources():
    deps = [os.path.join(CSRC, f) for f in sorted(os.listdir(CSRC))
            if f.endswith((".cu", ".cuh", ".h"))]
    deps.append(os.path.join(INCLUDE, "ndc_b200.h"))
    return deps


def _older(target, deps):
    if not os.path.exists(target):
        return True
    built = os.path.getmtime(target)
    return any(os.path.getmtime(s) > built for s in deps)


def is_stale():
    return _older(LIB, sources())


def ext_target():
    """The PyTorch and Python that an extension built now is for: it uses their C++ interfaces, which
    hold for one version only."""
    try:
        version = importlib.metadata.version("torch")
    except importlib.metadata.PackageNotFoundError:      # a source tree on the path
        version = "of unknown version"
    return "torch %s, %s" % (version, sys.implementation.cache_tag)


def ext_built_for():
    """The same of the extension that is there; None where that was not written down."""
    try:
        with open(EXT_KEY) as f:
            return f.read().strip()
    except FileNotFoundError:
        return None


def ext_is_stale():
    return _older(EXT, [EXT_SRC, os.path.join(INCLUDE, "ndc_b200.h"), os.path.abspath(__file__)]) or ext_built_for() != ext_target()


def _compile_ext():
    """Object of the host extension, and the command that links it once the library is there."""
    import torch

    root = os.path.dirname(torch.__file__)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    obj = os.path.join(OBJ, "ndc_torch.o")
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden",
           "-DTORCH_EXTENSION_NAME=_ndc_torch", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
           "-I", INCLUDE, "-I", os.path.join(root, "include"),
           "-I", os.path.join(root, "include", "torch", "csrc", "api", "include"),
           "-I", os.path.join(cuda, "include"), "-I", sysconfig.get_paths()["include"], "-c", EXT_SRC, "-o", obj]
    link = [cmd[0], "-shared", obj, "-o", EXT, "-L", os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu",
            "-ltorch_cuda", "-ltorch", "-ltorch_python", "-L", PKG, "-l:" + os.path.basename(LIB), "-Wl,-rpath,$ORIGIN",
            # The C++ runtime that PyTorch uses.  A compiler that comes with the archive alone would put a second
            # one into the extension, and the first exception thrown there would crash the process.
            "-l:libstdc++.so.6"]
    return subprocess.run(cmd, cwd=ROOT, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True), link


def build_library(force=False, verbose=False, extra_flags=()):
    """Build the shared library and the host extension if missing or older than a source file; the
    extension also where it was built for another PyTorch or Python."""
    if not (force or is_stale() or ext_is_stale()):
        return LIB
    os.makedirs(OBJ, exist_ok=True)
    with ThreadPoolExecutor(max_workers=1) as pool:   # the extension compiles next to the library
        ext = pool.submit(_compile_ext) if force or ext_is_stale() else None
        if force or is_stale():
            _build_cuda(verbose, extra_flags)
        if ext is not None:
            res, link = ext.result()
            if res.stdout and (verbose or res.returncode):
                print(res.stdout, end="", flush=True)
            if res.returncode:
                raise subprocess.CalledProcessError(res.returncode, res.args)
            if verbose:
                print(" ".join(link), flush=True)
            subprocess.check_call(link, cwd=ROOT)
            with open(EXT_KEY, "w") as f:
                f.write(ext_target() + "\n")
    return LIB


def _build_cuda(verbose, extra_flags):
    nvcc = os.environ.get("NVCC", "nvcc")

    def compile_unit(unit):
        name, src, defines = unit
        obj = os.path.join(OBJ, name + ".o")
        cmd = [nvcc, *NVCC_FLAGS, *extra_flags, *defines, "-I", INCLUDE, "-I", CSRC, "-c",
               os.path.join(CSRC, src), "-o", obj]
        if verbose:
            print(" ".join(cmd), flush=True)
        res = subprocess.run(cmd, cwd=ROOT, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
        return obj, res

    with ThreadPoolExecutor(max_workers=min(len(UNITS), os.cpu_count() or 1)) as pool:
        results = list(pool.map(compile_unit, UNITS))
    for _, res in results:
        if res.stdout and (verbose or res.returncode):
            print(res.stdout, end="", flush=True)
    failed = [res for _, res in results if res.returncode]
    if failed:
        raise subprocess.CalledProcessError(failed[0].returncode, failed[0].args)
    link = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", LIB] + [o for o, _ in results]
    if verbose:
        print(" ".join(link), flush=True)
    subprocess.check_call(link, cwd=ROOT)


if __name__ == "__main__":
    flags = ["-Xptxas", "-v"] if "--ptxas" in sys.argv else []
    print(build_library(force="--force" in sys.argv, verbose=True, extra_flags=flags))
