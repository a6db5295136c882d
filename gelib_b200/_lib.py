"""ctypes binding of ``libgelib_b200.so`` (declared in ``include/gelib_b200.h``).

Torch is used only to own device memory and to supply the current stream; what crosses into
the library are raw pointers, sizes and strides.  There is no CPU or pure-PyTorch fallback: if
the shared library is missing, importing a product fails with instructions to build it, and a
product on CPU tensors raises.
"""
import contextlib
import ctypes
import importlib
import os
import struct
import sys
import warnings

import torch

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_HERE, "libgelib_b200.so")

GELIB_OK, GELIB_SKIPPED, GELIB_INVALID, GELIB_CUDA_ERROR = 0, 1, 2, 3
GELIB_OVERWRITE = 1
GELIB_FP64 = 2
GELIB_MAX_PARTS = 16


class Tensor5(ctypes.Structure):
    """``gelib_tensor5``: 5-D canonical view (batch, grid0, grid1, 2l+1, channels), strides in floats."""
    _fields_ = [("base", ctypes.c_void_p), ("dims", ctypes.c_int32 * 5), ("strides", ctypes.c_int64 * 5)]


_P5 = ctypes.POINTER(Tensor5)
_lib = None

# name -> (restype, argtypes); every symbol include/gelib_b200.h declares
_PART3 = [_P5, _P5, _P5, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
_PART5 = [_P5, _P5, _P5, _P5, _P5, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
_VEC3 = [ctypes.c_int, _P5, ctypes.c_int, _P5, ctypes.c_int, _P5, ctypes.c_int, ctypes.c_void_p]
_VEC5 = [ctypes.c_int, _P5, ctypes.c_int, _P5, ctypes.c_int, _P5, _P5, _P5, ctypes.c_int, ctypes.c_void_p]
_IP = ctypes.POINTER(ctypes.c_int)
SYMBOLS = {
    "gelib_version": (ctypes.c_char_p, []),
    "gelib_last_error": (ctypes.c_char_p, []),
    "gelib_status_string": (ctypes.c_char_p, [ctypes.c_int]),
    "gelib_CGcoefficient": (ctypes.c_double, [ctypes.c_int] * 5),
    "gelib_CGmatrix": (ctypes.c_int, [ctypes.c_int] * 3 + [ctypes.c_void_p]),
    "gelib_SO3type_CGproduct": (ctypes.c_int, [ctypes.c_int, _IP, _IP, ctypes.c_int, _IP, _IP, ctypes.c_int,
                                               ctypes.c_int, ctypes.c_int, _IP, _IP]),
    "gelib_SO3vec_CGproduct_schedule": (ctypes.c_int, [ctypes.c_int, _IP, _IP, ctypes.c_int, _IP, _IP, ctypes.c_int,
                                                       _IP, ctypes.c_int, ctypes.c_int, _IP]),
    "gelib_SO3part_addCGproduct": (ctypes.c_int, _PART3),
    "gelib_SO3part_addCGproduct_back0": (ctypes.c_int, _PART3),
    "gelib_SO3part_addCGproduct_back1": (ctypes.c_int, _PART3),
    "gelib_SO3part_addCGproduct_back01": (ctypes.c_int, _PART5),
    "gelib_SO3part_addDiagCGproduct": (ctypes.c_int, _PART3),
    "gelib_SO3part_addDiagCGproduct_back0": (ctypes.c_int, _PART3),
    "gelib_SO3part_addDiagCGproduct_back1": (ctypes.c_int, _PART3),
    "gelib_SO3part_addDiagCGproduct_back01": (ctypes.c_int, _PART5),
    "gelib_SO3part_addSPharm": (ctypes.c_int, [_P5, _P5, ctypes.c_int, ctypes.c_void_p]),
    "gelib_SO3vec_addCGproduct": (ctypes.c_int, _VEC3),
    "gelib_SO3vec_addCGproduct_static": (ctypes.c_int, _VEC3),
    "gelib_SO3vec_addCGproduct_back0": (ctypes.c_int, _VEC3),
    "gelib_SO3vec_addCGproduct_back1": (ctypes.c_int, _VEC3),
    "gelib_SO3vec_addCGproduct_back01": (ctypes.c_int, _VEC5),
    "gelib_SO3vec_addDiagCGproduct": (ctypes.c_int, _VEC3),
    "gelib_SO3vec_addDiagCGproduct_back0": (ctypes.c_int, _VEC3),
    "gelib_SO3vec_addDiagCGproduct_back1": (ctypes.c_int, _VEC3),
    "gelib_SO3vec_addDiagCGproduct_back01": (ctypes.c_int, _VEC5),
    "gelib_SO3vec_addSPharm": (ctypes.c_int, [ctypes.c_int, _P5, _P5, ctypes.c_int, ctypes.c_void_p]),
    "gelib_SO3vec_addCGproduct_spharm": (ctypes.c_int, [ctypes.c_int, _P5, _P5, ctypes.c_int, ctypes.c_int, _P5, ctypes.c_int,
                                                        ctypes.c_void_p]),
    "gelib_SO3vec_addCGproduct_spharm_back1": (ctypes.c_int, [ctypes.c_int, _P5, ctypes.c_int, _P5, _P5, ctypes.c_int,
                                                              ctypes.c_int, ctypes.c_void_p]),
    "gelib_add_gather": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int, ctypes.c_int,
                                        ctypes.c_longlong, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]),
    "gelib_SO3part_mix": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int,
                                         ctypes.c_int, ctypes.c_int, ctypes.c_void_p]),
    "gelib_SO3part_mix_back_w": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_longlong,
                                                ctypes.c_int, ctypes.c_int, ctypes.c_void_p]),
    "gelib_SO3irrep_matrix": (ctypes.c_int, [ctypes.c_int, ctypes.c_double, ctypes.c_double, ctypes.c_double, ctypes.c_void_p]),
    "gelib_SO3part_apply": (ctypes.c_int, [_P5, _P5, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]),
    "gelib_kernel_launch_count": (ctypes.c_longlong, []),
    "gelib_set_option": (ctypes.c_int, [ctypes.c_char_p, ctypes.c_char_p]),
    "gelib_async_status": (ctypes.c_int, []),
    "gelib_probe_fp32_tflops": (ctypes.c_double, [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]),
}


def lib():
    """The loaded library.  Raises (never falls back) when it has not been built."""
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise RuntimeError(
                "gelib_b200: %s not found. Build it with `python -m gelib_b200.build` (needs nvcc); "
                "there is no CPU fallback." % LIB_PATH)
        L = ctypes.CDLL(LIB_PATH)
        for name, (res, args) in SYMBOLS.items():
            f = getattr(L, name)
            f.restype = res
            f.argtypes = args
        _lib = L
    return _lib


_native = None


class _Declines:
    """Stands in for the native host side: every function leaves the call to the Python code."""

    def __getattr__(self, name):
        return lambda *args: None


def native():
    """The native host side of the products (csrc/host.cpp).  It only saves host time, so where it cannot be had -- no Python
    headers to build it with, or made for another torch -- the Python code does its part, after a warning."""
    global _native
    if _native is None:
        lib()
        why = None
        try:
            module = importlib.import_module(__package__ + "._native")
            if module.torch_version != torch.__version__:
                why = "built for torch %s, this is %s" % (module.torch_version, torch.__version__)
        except ImportError as e:
            why = e
        if why is not None:
            warnings.warn("gelib_b200: %s cannot be used (%s); products take more host time.  `python -m gelib_b200.build` builds it."
                          % (os.path.join(_HERE, "_native.so"), why), RuntimeWarning, stacklevel=2)
            module = _Declines()
        _native = module
    return _native


def last_error():
    return lib().gelib_last_error().decode()


def set_option(name, value):
    """Pins the kernel choice ("fwd", "bwd") or a test switch ("inject_timeout"); see include/gelib_b200.h."""
    check(lib().gelib_set_option(name.encode(), str(value).encode()))


def async_status():
    """Raises if a kernel with bounded waits gave up since the last check (call after synchronising)."""
    check(lib().gelib_async_status())


def check(status):
    """Maps a status code onto the reference's behaviour: a GELIB_SKIP prints its message and the call
    returns without computing (include/GElib_base.hpp:36); everything else raises RuntimeError, as the
    reference's std::runtime_error does through pybind11."""
    if status == GELIB_OK:
        return True
    msg = last_error()
    if status == GELIB_SKIPPED:
        sys.stderr.write(msg + "\n")
        return False
    raise RuntimeError(msg)


# ---- descriptors -----------------------------------------------------------------------------------


def _fuse(dims, strides):
    """Fuses grid dimensions into one if their strides allow it (core/Gpart.hpp:462-468)."""
    dims, strides = list(dims), list(strides)
    keep = [(d, s) for d, s in zip(dims, strides) if d != 1]
    if not keep:
        return 1, 0
    for (d0, s0), (d1, s1) in zip(keep[:-1], keep[1:]):
        if s0 != s1 * d1:
            raise RuntimeError("GElib error: grid dimensions cannot be fused into the 5-D canonical form.")
    n = 1
    for d, _ in keep:
        n *= d
    return n, keep[-1][1]


# One gelib_tensor5 in native layout.  Packing it in one call and reading the tensor's attributes once is what the cost of
# a small product is made of: a field-by-field ctypes structure took 8 us per tensor, this takes about 1.
_TENSOR5 = struct.Struct("@P5i5q")
assert _TENSOR5.size == ctypes.sizeof(Tensor5)


_pack_into = _TENSOR5.pack_into
_COMPLEX = torch.complex64


def _resolved(buf, t, written):
    """t.conj() only marks a view, and the kernels read memory.  The descriptor keeps the copy until the call has been issued;
    after that the allocator hands its memory out in stream order."""
    if written:
        raise RuntimeError("GElib error: a conjugated view cannot be written to.")
    t = t.resolve_conj()
    buf.__dict__.setdefault("copies", []).append(t)
    return t


def _pack(buf, at, t, real, written):
    if not t.is_cuda:
        raise RuntimeError("gelib_b200 computes on CUDA tensors only (this build has no CPU path); got a %s tensor"
                           % t.device.type)
    D = t.shape
    d = len(D)
    if d == 3 and not real and t.dtype is _COMPLEX:
        if t.is_conj():
            t = _resolved(buf, t, written)
        b, m, n = D
        sb, sm, sn = t.stride()
        _pack_into(buf, at, t.data_ptr(), b, 1, 1, m, n, 2 * sb, 0, 0, 2 * sm, 2 * sn)
        return
    if real:
        if t.dtype != torch.float32:
            raise RuntimeError("expected a float32 tensor")
        scale = 1
    else:
        if t.dtype != _COMPLEX:
            raise RuntimeError("expected a complex64 tensor (an SO3part)")
        scale = 2
        if t.is_conj():
            t = _resolved(buf, t, written)
    if d < 3:
        raise RuntimeError("an SO3part has at least 3 dimensions (batch, 2l+1, channels)")
    S = [scale * s for s in t.stride()]
    if d == 3:
        D = (D[0], 1, 1, D[1], D[2])
        S = (S[0], 0, 0, S[1], S[2])
    elif d == 4:
        D = (D[0], D[1], 1, D[2], D[3])
        S = (S[0], S[1], 0, S[2], S[3])
    elif d > 5:
        g, s = _fuse(D[1:d - 2], S[1:d - 2])
        D = (D[0], g, 1, D[d - 2], D[d - 1])
        S = (S[0], s, 0, S[d - 2], S[d - 1])
    _pack_into(buf, at, t.data_ptr(), *D, *S)


def descriptor(t, real=False, written=False):
    """``gelib_tensor5`` of a torch tensor in the reference's 5-D canonical form (core/Gpart.hpp:450-469).

    Complex tensors (b, [grid...], 2l+1, n) are viewed as interleaved floats, so strides double
    (cuda/GPUtensor.hpp:31-38).  ``real=True`` is for the (b, [grid...], 3, n) float input of spharm, ``written=True`` for
    a tensor that the call adds to or overwrites.
    """
    out = Tensor5()
    with torch._C.DisableTorchFunctionSubclass():
        _pack(out, 0, t, real, written)
    return out


def descriptor_array(tensors, real=False, written=False):
    arr = (Tensor5 * max(1, len(tensors)))()
    at = 0
    with torch._C.DisableTorchFunctionSubclass():
        for t in tensors:
            _pack(arr, at, t, real, written)
            at += _TENSOR5.size
    return arr


_SAME_DEVICE = contextlib.nullcontext()


def device_guard(t):
    """Context manager making t's device current; raises for anything that is not a CUDA tensor."""
    with torch._C.DisableTorchFunctionSubclass():
        if not t.is_cuda:
            raise RuntimeError("gelib_b200 computes on CUDA tensors only (this build has no CPU path); got a %s tensor"
                               % t.device.type)
        index = t.get_device()
    return _SAME_DEVICE if torch.cuda.current_device() == index else torch.cuda.device(index)


def stream_of(t):
    with torch._C.DisableTorchFunctionSubclass():
        return ctypes.c_void_p(torch._C._cuda_getCurrentRawStream(t.get_device()))
