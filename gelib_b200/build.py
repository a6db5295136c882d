"""Builds ``libgelib_b200.so`` (the C-ABI library with the sm_100a kernels) in-tree with nvcc.

    python -m gelib_b200.build [--force] [--verbose]

The library is a plain shared object (no Python or torch dependency); it is what a GElib build
links instead of its own ``cuda/`` objects, and what ``gelib_b200._lib`` loads through ctypes.
``_native.so``, built beside it, is the Python package's own: it links the library and torch, and the
package runs without it.
"""
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(CSRC, "build")
LIB = os.path.join(HERE, "libgelib_b200.so")
NATIVE = os.path.join(HERE, "_native.so")  # host side of the Python products (csrc/host.cpp), against torch's C++ library
SOURCES = ["bank.cu", "plan.cu", "cg_fwd.cu", "cg_fwd_tc.cu", "cg_bwd.cu", "cg_bwd_pair.cu", "cg_bwd_tc.cu", "cg_narrow.cu", "cg_narrow1_bwd.cu", "cg_strided.cu", "col_plan.cu", "col_fwd.cu", "col_bwd.cu", "col_bwd_x.cu", "col_bwd_y.cu", "col_bwd_owned.cu", "mir_fwd.cu", "mir_bwd.cu", "diag.cu", "diag_fwd.cu", "diag_bwd.cu", "spharm.cu", "probe.cu", "gather_apply.cu", "mix.cu", "cabi.cu"]
HEADERS = ["common.h", "plan.h", "tc_common.h", "tma_maps.h", "col.h", "col_device.h", "mir.h", "f32x2.h", "col_bwd.cuh", os.path.join("..", "..", "include", "gelib_b200.h")]
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-Xcompiler", "-fPIC",
         "--expt-relaxed-constexpr"] + os.environ.get("GELIB_NVCC_FLAGS", "").split()
# spharm.cu keeps the reference's rounding points: no FMA contraction there
PER_FILE = {"spharm.cu": ["-fmad=false"]}


def _newest(paths):
    return max(os.path.getmtime(p) for p in paths)


def _digest(path):
    with open(path, "rb") as f:
        return hashlib.sha256(f.read()).hexdigest()


def build_library(force=False, verbose=False):
    srcs = [os.path.join(CSRC, s) for s in SOURCES]
    deps = srcs + [os.path.join(CSRC, h) for h in HEADERS] + [os.path.abspath(__file__)]
    if not force and os.path.exists(LIB) and os.path.getmtime(LIB) >= _newest(deps):
        return LIB
    os.makedirs(OBJ, exist_ok=True)
    hdr_time = _newest(deps[len(srcs):])

    def compile_one(name):
        src = os.path.join(CSRC, name)
        obj = os.path.join(OBJ, name.replace(".cu", ".o"))
        if not force and os.path.exists(obj) and os.path.getmtime(obj) >= max(os.path.getmtime(src), hdr_time):
            return obj, ""
        cmd = [NVCC] + FLAGS + PER_FILE.get(name, []) + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed for %s:\n%s\n%s" % (name, r.stdout, r.stderr))
        return obj, r.stderr

    with ThreadPoolExecutor(max_workers=min(8, len(SOURCES))) as ex:
        results = list(ex.map(compile_one, SOURCES))
    if verbose:
        for _, log in results:
            sys.stderr.write(log)
    objs = [o for o, _ in results]
    cmd = [NVCC, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n%s\n%s" % (r.stdout, r.stderr))
    return LIB


def _cuda_include():
    """Beside the compiler, wherever NVCC names it: by path, by name, or through a link."""
    found = shutil.which(NVCC) or NVCC
    roots = [os.path.dirname(os.path.dirname(p)) for p in (found, os.path.realpath(found))]
    places = [os.path.join(r, "include") for r in roots]
    return next((p for p in places if os.path.exists(os.path.join(p, "cuda_runtime_api.h"))), places[0])


def _native_lacks():
    """What this machine lacks to build the native host side; None when it can."""
    try:
        import torch
    except ImportError:
        return "torch"
    if torch.version.cuda is None:
        return "a torch with CUDA"
    include = os.path.join(os.path.dirname(os.path.abspath(torch.__file__)), "include")
    for header, place in (("ATen/ATen.h", include), ("cuda_runtime_api.h", _cuda_include()), ("Python.h", sysconfig.get_paths()["include"])):
        if not os.path.exists(os.path.join(place, header)):
            return "%s in %s" % (header, place)
    return None


def build_native(force=False, verbose=False):
    src, header = os.path.join(CSRC, "host.cpp"), os.path.join(HERE, "..", "include", "gelib_b200.h")
    import torch
    root = os.path.dirname(os.path.abspath(torch.__file__))
    include = [os.path.join(root, "include"), os.path.join(root, "include", "torch", "csrc", "api", "include"),
               _cuda_include(), sysconfig.get_paths()["include"]]
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden"]
    cmd += ["-DGELIB_TORCH_VERSION=\"%s\"" % torch.__version__, "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI]
    cmd += ["-I" + i for i in include] + [src, "-o", NATIVE]
    cmd += ["-L" + os.path.join(root, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"]
    cmd += ["-L" + HERE, "-l:" + os.path.basename(LIB), "-Wl,-rpath,$ORIGIN"]
    # The file is tied to this torch and this Python; what it was made with, and its own digest, are kept beside the objects.
    stamp, made_with = os.path.join(OBJ, "native.stamp"), "\n".join([sys.version] + cmd)
    if not force and os.path.exists(NATIVE) and os.path.getmtime(NATIVE) >= _newest([src, header, LIB, os.path.abspath(__file__)]):
        if os.path.exists(stamp) and open(stamp).read() == made_with + "\n" + _digest(NATIVE):
            return NATIVE
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed for host.cpp:\n%s\n%s" % (r.stdout, r.stderr))
    os.makedirs(OBJ, exist_ok=True)
    with open(stamp, "w") as f:
        f.write(made_with + "\n" + _digest(NATIVE))
    return NATIVE


def build(force=False, verbose=False):
    """The library, which needs neither torch nor Python's headers, and the native host side where they are there."""
    path = build_library(force, verbose)
    lacks = _native_lacks()
    if lacks is None:
        build_native(force, verbose)
    else:
        sys.stderr.write("gelib_b200: %s is not built, for want of %s; products run without it, with more host time per call.\n"
                         % (os.path.basename(NATIVE), lacks))
    return path


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
