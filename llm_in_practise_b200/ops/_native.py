"""ctypes binding to ``libb200ops.so`` (C ABI declared in ``include/b200_ops.h``).

The library is built in-tree by ``llm_in_practise_b200._build`` and loaded lazily. On a machine
with a GPU a missing library is an error (the CUDA path must be the one that runs); on a CPU-only
machine the ops fall back to their plain-PyTorch reference implementations, which are also the
numerical oracles of the GPU tests.
"""
from __future__ import annotations

import ctypes
import importlib.util
import os
import sysconfig
from pathlib import Path

import torch

_LIBDIR = Path(__file__).resolve().parent.parent / "_lib"
_lib = None
_host_lib = None
# the mapping behind os.environ, whose own look-up encodes the key each time (0.5 us, once or twice an op)
_environ = getattr(os.environ, "_data", os.environ)
_FORCE_KEY, _FORCE_ON = ("B200_FORCE_TORCH", "1") if _environ is os.environ else (os.environ.encodekey("B200_FORCE_TORCH"), os.environ.encodevalue("1"))
launch_count = 0  # number of kernel launches issued through this binding (bench.py reports it)

DT_BF16, DT_FP16, DT_FP32 = 0, 1, 2
_DT = {torch.bfloat16: DT_BF16, torch.float16: DT_FP16, torch.float32: DT_FP32}

_ERRORS = {
    10001: "bad shape", 10002: "bad alignment (pointers and strides must be 16-byte multiples)",
    10003: "CUDA driver entry point unavailable", 10004: "cuTensorMapEncodeTiled failed",
    10005: "size beyond the supported maximum", 10006: "unsupported argument combination",
}


ERR_UNSUPPORTED = 10006


class NativeError(RuntimeError):
    pass


def has(name: str) -> bool:
    """True when the loaded library exports ``name`` (a library linked from a subset of the kernel sources lacks some)."""
    return hasattr(lib(), name)


def dtype_code(dt: torch.dtype) -> int:
    try:
        return _DT[dt]
    except KeyError:
        raise TypeError(f"unsupported dtype {dt}") from None


def lib_path() -> Path:
    return _LIBDIR / "libb200ops.so"


def available() -> bool:
    """True when the CUDA kernels can run: library built and a CUDA device visible."""
    return torch.cuda.is_available() and lib_path().exists()


def use_native(*tensors) -> bool:
    """Dispatch rule shared by all ops: CUDA tensors go to the native kernels (and a missing
    library is fatal there); CPU tensors go to the PyTorch reference path."""
    if not tensors or not tensors[0].is_cuda:
        return False
    if _environ.get(_FORCE_KEY) == _FORCE_ON:
        return False
    if _lib is None:
        lib()  # raises if missing
    return True


def lib() -> ctypes.CDLL:
    global _lib, _make_entry
    if _lib is None:
        p = lib_path()
        if not p.exists():
            raise NativeError(
                f"{p} is missing: run `python -m llm_in_practise_b200._build` (or __graft_entry__.build()) first")
        _lib = ctypes.CDLL(str(p))
        _declare(_lib)
        if _make_entry is None:              # built since this module was imported (_build.ensure_built)
            _make_entry = _fastcall()
    return _lib


def host_lib() -> ctypes.CDLL | None:
    global _host_lib
    if _host_lib is None:
        p = _LIBDIR / "libb200host.so"
        if not p.exists():
            return None
        _host_lib = ctypes.CDLL(str(p))
    return _host_lib


def check(rc: int, what: str = "") -> None:
    if rc == 0:
        return
    if rc >= 10000:
        msg = _ERRORS.get(rc, "unknown error")
    else:
        msg = f"CUDA error {rc}"
        try:
            msg += " (" + torch.cuda.cudart().cudaGetErrorString(rc) + ")"  # type: ignore[attr-defined]
        except Exception:
            pass
    raise NativeError(f"b200 {what}: {msg}")


# Handles go to the entry points as plain integers: every prototype declares its pointers (``proto``), and building a c_void_p, or a
# ``torch.cuda.Stream`` object to read its handle from, takes longer than the rest of a launch (five launches of a decode step's
# recurrent mixer: 90 us with them, 70 without).
def stream() -> int:
    """Handle of the current device's current stream."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def ptr(t: torch.Tensor | None) -> int:
    return 0 if t is None else t.data_ptr()


_sm_counts: dict = {}


def sm_count(device: torch.device) -> int:
    """Multiprocessors of a CUDA device (cached: the property query is slow on a hot path)."""
    key = device.index if device.index is not None else torch.cuda.current_device()
    if key not in _sm_counts:
        _sm_counts[key] = torch.cuda.get_device_properties(key).multi_processor_count
    return _sm_counts[key]


def count_launch(n: int = 1) -> None:
    global launch_count
    launch_count += n


class GemmArgs(ctypes.Structure):
    _fields_ = [
        ("A", ctypes.c_void_p), ("B", ctypes.c_void_p), ("D", ctypes.c_void_p), ("bias", ctypes.c_void_p),
        ("A2", ctypes.c_void_p), ("B2", ctypes.c_void_p),
        ("M", ctypes.c_int32), ("N", ctypes.c_int32), ("K", ctypes.c_int32), ("K2", ctypes.c_int32),
        ("batch", ctypes.c_int32), ("nb0", ctypes.c_int32), ("b_div", ctypes.c_int32), ("bias_dtype", ctypes.c_int32),
        ("a_rs", ctypes.c_int64), ("a_bs0", ctypes.c_int64), ("a_bs1", ctypes.c_int64),
        ("b_rs", ctypes.c_int64), ("b_bs0", ctypes.c_int64), ("b_bs1", ctypes.c_int64),
        ("d_rs", ctypes.c_int64), ("d_bs0", ctypes.c_int64), ("d_bs1", ctypes.c_int64),
        ("a2_rs", ctypes.c_int64), ("b2_rs", ctypes.c_int64),
        ("a_mn", ctypes.c_int32), ("b_mn", ctypes.c_int32), ("in_dtype", ctypes.c_int32), ("out_dtype", ctypes.c_int32),
        ("alpha", ctypes.c_float), ("beta", ctypes.c_float),
        ("workspace", ctypes.c_void_p), ("workspace_bytes", ctypes.c_int64),
        ("beta_rows", ctypes.c_void_p),
        ("ar", ctypes.c_void_p),
        ("b_map", ctypes.c_void_p), ("b_count", ctypes.c_int32), ("bias_bs", ctypes.c_int64),
    ]


class GemmAllReduce(ctypes.Structure):
    """``b200_gemm_allreduce`` (include/b200_ops.h): all-reduce of D over tensor-parallel ranks inside the GEMM launch."""
    _fields_ = [
        ("d_mc", ctypes.c_void_p), ("d_ptrs", ctypes.c_void_p), ("tile_flag_ptrs", ctypes.c_void_p), ("sync_flag_ptrs", ctypes.c_void_p),
        ("ticket", ctypes.c_void_p),
        ("world", ctypes.c_int32), ("rank", ctypes.c_int32), ("channel", ctypes.c_int32), ("epoch", ctypes.c_uint32),
        ("max_tiles", ctypes.c_int64),
    ]


def _declare(L: ctypes.CDLL) -> None:
    vp, i32, i64, f32 = ctypes.c_void_p, ctypes.c_int32, ctypes.c_int64, ctypes.c_float
    L.b200_gemm.argtypes = [ctypes.POINTER(GemmArgs), vp]
    L.b200_gemm.restype = ctypes.c_int
    # remaining prototypes are declared next to their Python wrappers via `proto`


_KINDS = {ctypes.c_void_p: "p", ctypes.c_float: "f", **{t: "i" for t in (ctypes.c_int, ctypes.c_longlong, ctypes.c_int32, ctypes.c_int64,
                                                                              ctypes.c_uint32, ctypes.c_uint64, ctypes.c_ulonglong)}}


def _fastcall():
    """``make`` of the extension that calls the C ABI (csrc/host/python/fastcall.cpp), or None: calls then go through ctypes."""
    # the name says for which Python it was built: the module uses its object layouts, and a loader by path does not check them
    p = _LIBDIR / ("_b200_fastcall" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))
    if not p.exists():
        return None
    try:
        spec = importlib.util.spec_from_file_location("_b200_fastcall", p)
        module = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(module)
        return module.make
    except ImportError:                      # not a module, or one for another system
        return None


_make_entry = _fastcall()


def proto(name: str, argtypes):
    """An entry point of the library as a callable with these argument types; made once per library. The ctypes function, or where all
    its arguments are numbers and pointers a callable without ctypes' 2 us a call, which falls back on it for any other argument."""
    L = _lib if _lib is not None else lib()
    made = L.__dict__.get("_b200_entries")
    if made is None:
        made = L._b200_entries = {}
    fn = made.get(name)
    if fn is None:
        fn = getattr(L, name)
        fn.argtypes = argtypes
        fn.restype = ctypes.c_int
        if _make_entry is not None and all(t in _KINDS for t in argtypes):
            fn = _make_entry(ctypes.cast(fn, ctypes.c_void_p).value, "".join(_KINDS[t] for t in argtypes), fn) or fn
        made[name] = fn
    return fn
