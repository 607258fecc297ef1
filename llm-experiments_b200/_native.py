"""ctypes binding of ``libb2kv.so``, the C-ABI CUDA library (declared in include/b2kv.h).

The library is the only compute path of this package.  If it is missing the import of
this module fails with instructions to build it: there is no CPU or PyTorch fallback.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import pathlib
import struct
import sysconfig

_PKG = pathlib.Path(__file__).resolve().parent
LIB_PATH = _PKG / "libb2kv.so"
# Calls without ctypes' conversions (csrc/calls.c), for this interpreter; where it is not built ctypes makes them.
CALLS_PATH = _PKG / ("b2kv_calls" + sysconfig.get_config_var("EXT_SUFFIX"))
SERVE_LIB_PATH = _PKG / "libb2kv_serve.so"  # the part models are served with (build.py --serve), where that is all there is

DTYPE_F32 = 0
DTYPE_BF16 = 1

ERR_BAD_ARG = -1
ERR_ALIGN = -2
ERR_UNSUPPORTED = -3
ERR_WORKSPACE = -4
ERR_CUDA = -5
ERR_STATIC_LIMIT = -6
STATIC_SCRATCH_BYTES = 32 << 20

DEV_STATUS_TEXT = {
    1: "a block-table entry points outside the pool",
    2: "an append position lies outside the cache",
    3: "a bounded wait on a barrier ran out",
    4: "a token id lies outside the embedding table",
}

_vp = ctypes.c_void_p
_i = ctypes.c_int
_i64 = ctypes.c_int64
_sz = ctypes.c_size_t

_f = ctypes.c_float

SEG_STORE, SEG_F32, SEG_GLU_SILU, SEG_GLU_CLAMP, SEG_RELU2, SEG_SOFTCAP, SEG_DECAY = 0, 1, 2, 3, 4, 5, 6
MAX_SEGMENTS = 3
LINEAR_AHEAD = 1


class Segment(ctypes.Structure):
    """``b2kv_segment``: where a range of output columns of a linear layer goes."""

    _fields_ = [("out", _vp), ("ld", _i64), ("group", _i64), ("end", ctypes.c_int32), ("kind", ctypes.c_int32)]


class LinearArgs(ctypes.Structure):
    """``b2kv_linear_args``."""

    _fields_ = [("x", _vp), ("w", _vp), ("residual", _vp), ("bias", _vp), ("group_rows", _vp), ("ld_x", _i64), ("group_x", _i64),
                ("ld_w", _i64), ("group_w", _i64), ("ld_residual", _i64), ("seg", Segment * MAX_SEGMENTS),
                ("rows", ctypes.c_int32), ("K", ctypes.c_int32), ("N", ctypes.c_int32), ("groups", ctypes.c_int32),
                ("max_group_rows", ctypes.c_int32), ("n_seg", ctypes.c_int32), ("dtype", ctypes.c_int32),
                ("path", ctypes.c_int32), ("limit", _f)]


class LinearOptions(ctypes.Structure):
    """``b2kv_linear_options``."""

    _fields_ = [("group_x_rows", _vp), ("x_rows", ctypes.c_int32), ("flags", ctypes.c_int32)]


class GlaArgs(ctypes.Structure):
    """``b2kv_gla_args``."""

    _fields_ = [("y", _vp), ("alpha", _vp), ("norm", _vp), ("state", _vp), ("out", _vp), ("segments", _vp), ("row_pos", _vp), ("workspace", _vp),
                ("workspace_bytes", _sz),
                ("ld_y", _i64), ("ld_alpha", _i64), ("ld_out", _i64), ("q_col", ctypes.c_int32), ("k_col", ctypes.c_int32),
                ("v_col", ctypes.c_int32), ("g_col", ctypes.c_int32), ("H", ctypes.c_int32), ("dim", ctypes.c_int32),
                ("vdim", ctypes.c_int32), ("n_segments", ctypes.c_int32), ("max_n", ctypes.c_int32), ("rows", ctypes.c_int32),
                ("n_slots", ctypes.c_int32), ("dtype", ctypes.c_int32), ("path", ctypes.c_int32), ("q_scale", _f),
                ("eps", _f)]


# name -> (restype, argtypes); kept in the order of include/b2kv.h
SIGNATURES = {
    "b2kv_strerror": (ctypes.c_char_p, [_i]),
    "b2kv_last_cuda_error": (ctypes.c_char_p, []),
    "b2kv_version": (_i, []),
    "b2kv_append": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i64, _i64, _i64, _i, _vp, _vp]),
    "b2kv_append_paged": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _vp, _i, _i, _i, _i, _i, _i, _i64, _i64, _i64, _i,
                               _vp, _vp]),
    "b2kv_append_rows_paged": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _i, _i64, _i64, _i64, _i, _vp, _vp]),
    "b2kv_advance_lengths": (_i, [_vp, _i, _i, _vp]),
    "b2kv_gather": (_i, [_vp, _vp, _vp, _i, _i, _i, _i, _i, _i64, _i64, _i64, _i, _vp]),
    "b2kv_gather_paged": (_i, [_vp, _vp, _vp, _i, _vp, _i, _i, _i, _i, _i, _i, _i, _i64, _i64, _i64, _i, _vp, _vp]),
    "b2kv_decode_workspace_bytes": (_sz, [_i, _i, _i, _i, _i]),
    "b2kv_decode": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i64, _i64, _i64, _i, _vp, _sz, _vp, _vp]),
    "b2kv_decode_paged": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _vp, _i, _i, _i, _i, _i, _i, _i, _i64, _i64, _i64,
                               _i, _vp, _sz, _vp, _vp]),
    "b2kv_decode_allgather": (_i, [_vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i64, _i64, _i64, _i, _vp, _sz, _vp, _vp,
                                   _vp, _vp, ctypes.c_uint32, _i, _i, _i, ctypes.c_uint32, _vp, _vp]),
    "b2kv_decode_partial": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i64, _i64, _i64, _i, _vp, _sz, _vp,
                                 _vp]),
    "b2kv_merge_partials": (_i, [_vp, _i, _i, _i, _i, _vp, _i, _vp]),
    "b2kv_decode_static": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i64, _i64, _i64, _i, _vp, _vp]),
    "b2kv_prefill": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _i, _i, _i, _i, _i, _i, _vp, _vp]),
    "b2kv_prefill_workspace_bytes": (_sz, [_i, _i, _i, _i, _i]),
    "b2kv_prefill_ws": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i64, _i64, _i64, _i, _i, _i, _i, _i, _i, _vp, _sz,
                             _vp, _vp]),
    "b2kv_prefill_paged": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i64, _i64, _i64, _i, _i, _i, _i, _i,
                                _vp, _vp]),
    "b2kv_layernorm": (_i, [_vp, _vp, _vp, _vp, _i64, _i, ctypes.c_float, _vp]),
    "b2kv_layernorm_bf16": (_i, [_vp, _vp, _vp, _vp, _i64, _i, ctypes.c_float, _vp]),
    "b2kv_extract_last_tokens": (_i, [_vp, _vp, _i, _i, _i, _vp]),
    "b2kv_softmax": (_i, [_vp, _vp, _i64, _i, _vp]),
    "b2kv_argmax": (_i, [_vp, _vp, _i, _i, _vp]),
    "b2kv_extract_last_tokens_bf16": (_i, [_vp, _vp, _i, _i, _i, _vp]),
    "b2kv_argmax_bf16": (_i, [_vp, _vp, _i, _i, _vp]),
    "b2kv_embedding": (_i, [_vp, _vp, _vp, _vp, _i, _vp, _i, _i, _i, _i, _i, _i, _vp, _vp]),
    "b2kv_qkv_append": (_i, [_vp, _vp, _vp, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i64, _i64, _i64, _i, _vp, _vp]),
    "b2kv_matmul_rows": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _vp]),
    "b2kv_matmul": (_i, [_vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _vp, _vp]),
    "b2kv_embed_rows": (_i, [_vp, _vp, _vp, _vp, _f, _i, _i, _i, _i, _vp, _vp]),
    "b2kv_layernorm_rows": (_i, [_vp, _i64, _vp, _vp, _vp, _vp, _i64, _vp, _i64, _i, _i, _f, _i, _vp]),
    "b2kv_rmsnorm": (_i, [_vp, _i64, _vp, _vp, _f, _vp, _i64, _i, _i, _f, _i, _vp]),
    "b2kv_linear": (_i, [ctypes.POINTER(LinearArgs), _vp, _vp]),
    "b2kv_linear_opt": (_i, [ctypes.POINTER(LinearArgs), ctypes.POINTER(LinearOptions), _vp, _vp]),
    "b2kv_linear_ws": (_i, [ctypes.POINTER(LinearArgs), ctypes.POINTER(LinearOptions), _vp, _sz, _vp, _vp]),
    "b2kv_linear_workspace_bytes": (_sz, [ctypes.POINTER(LinearArgs)]),
    "b2kv_latent_append": (_i, [_vp, _i64, _i, _i, _i, _i, _vp, _i, _i, _vp, _f, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp, _vp]),
    "b2kv_latent_decode_workspace_bytes": (_sz, [_i, _i, _i, _i, _i]),
    "b2kv_latent_decode": (_i, [_vp, _vp, _i64, _i, _vp, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _i, _f, _i, _i, _vp,
                                _sz, _vp, _vp]),
    "b2kv_latent_prefill_supported": (_i, [_i, _i, _i, _i, _i]),
    "b2kv_latent_prefill": (_i, [_vp, _i64, _vp, _vp, _i64, _vp, _i64, _vp, _i64, _vp, _i, _i, _i, _i, _i, _i, _i, _i, _i, _f, _i,
                                 _vp, _vp]),
    "b2kv_gqa_append": (_i, [_vp, _i64, _i, _i, _i, _i, _vp, _vp, _f, _f, _i, _vp, _vp, _vp, _vp, _i, _i, _i, _i, _vp, _vp]),
    "b2kv_gqa_decode_workspace_bytes": (_sz, [_i, _i, _i, _i, _i, _i]),
    "b2kv_gqa_decode": (_i, [_vp, _i64, _vp, _vp, _vp, _i64, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _i, _f, _i, _i, _vp, _sz,
                             _vp, _vp]),
    "b2kv_gqa_decode_runs": (_i, [_vp, _i64, _vp, _vp, _vp, _i64, _vp, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _i, _f, _i, _i, _i, _vp, _sz,
                             _vp, _vp]),
    "b2kv_gqa_prefill_supported": (_i, [_i, _i, _i]),
    "b2kv_gqa_prefill": (_i, [_vp, _i64, _vp, _vp, _i64, _vp, _i64, _vp, _vp, _i, _i, _i, _i, _i, _i, _i, _f, _i, _vp, _vp]),
    "b2kv_gla_workspace_bytes": (_sz, [_i, _i, _i, _i, _i, _i, _i]),
    "b2kv_gla": (_i, [ctypes.POINTER(GlaArgs), _vp, _vp]),
    "b2kv_route": (_i, [_vp, _i64, _i, _i, _i, _i, _i, _vp, _vp, _vp, _vp]),
    "b2kv_moe_plan": (_i, [_vp, _vp, _i, _i, _i, _vp, _vp, _vp, _i64, _vp, _i64, _i, _i, _vp]),
    "b2kv_moe_combine": (_i, [_vp, _i64, _vp, _i64, _vp, _vp, _i, _i, _i, _i, _vp]),
    "b2kv_tune": (_i, [ctypes.c_char_p, _i]),
}


class B2KVError(RuntimeError):
    """A C-ABI call returned a negative status."""

    def __init__(self, status: int, text: str):
        super().__init__(f"b2kv error {status}: {text}")
        self.status = status


def _not_built(name: str):
    def call(*_):
        raise ImportError(f"{name} is not part of {SERVE_LIB_PATH.name}; build the whole library with {_PKG.name}/build.py")

    return call


_TYPES = {_vp: "p", _i: "i", _i64: "l", _sz: "l", _f: "f", ctypes.c_uint32: "i", ctypes.c_char_p: None}


def _calls():
    """The extension module of ``csrc/calls.c``, or None."""
    if not CALLS_PATH.exists():
        return None
    loader = importlib.machinery.ExtensionFileLoader("b2kv_calls", str(CALLS_PATH))
    try:
        module = importlib.util.module_from_spec(importlib.util.spec_from_loader("b2kv_calls", loader))
        loader.exec_module(module)
    except ImportError:  # of another machine
        return None
    return module


class Library:
    """The entry points: what ``csrc/calls.c`` can call, and ctypes functions for the rest (texts)."""

    def __init__(self, lib: ctypes.CDLL, calls):
        self.cdll = lib
        for name, (restype, argtypes) in SIGNATURES.items():
            fn = getattr(lib, name)
            kinds = ["p" if issubclass(t, ctypes._Pointer) else _TYPES[t] for t in argtypes]
            if calls is not None and None not in kinds and restype in (_i, _sz) and hasattr(fn, "argtypes"):
                fn = calls.bind(ctypes.cast(fn, _vp).value, "".join(kinds), "i" if restype is _i else "z", fn)
            setattr(self, name, fn)

    def __getattr__(self, name: str):  # what SIGNATURES does not list
        return getattr(self.cdll, name)


def _load() -> Library:
    path = LIB_PATH if LIB_PATH.exists() or not SERVE_LIB_PATH.exists() else SERVE_LIB_PATH
    if not path.exists():
        raise ImportError(
            f"{LIB_PATH} is missing. Build the CUDA library first: "
            f"`python {_PKG.name}/build.py` (needs nvcc with sm_100a support). "
            "This package has no CPU fallback."
        )
    lib = ctypes.CDLL(str(path))
    for name, (restype, argtypes) in SIGNATURES.items():
        if path == SERVE_LIB_PATH and not hasattr(lib, name):
            setattr(lib, name, _not_built(name))
            continue
        fn = getattr(lib, name)  # AttributeError here means header and library disagree
        fn.restype = restype
        fn.argtypes = argtypes
    return Library(lib, calls)


calls = _calls()
lib = _load()

# The structures as bytes, which calls.c passes on as they are (a ctypes structure takes longer to fill than its call).
_LINEAR_ARGS = struct.Struct("5P5q" + "P2q2i" * MAX_SEGMENTS + "8if4x")
_LINEAR_OPTIONS = struct.Struct("P2i")
assert _LINEAR_ARGS.size == ctypes.sizeof(LinearArgs) and _LINEAR_OPTIONS.size == ctypes.sizeof(LinearOptions)
_NO_SEGMENT = (0, 0, 0, 0, 0)


def _structure(cls, packed: bytes):
    return packed if calls is not None else ctypes.byref(cls.from_buffer_copy(packed))


def linear_args(x, w, residual, bias, group_rows, ld_x, group_x, ld_w, group_w, ld_residual, segments, rows, k, n, groups, max_group_rows, dtype,
                path, limit):
    """``b2kv_linear_args`` for ``lib``; ``segments``: (out, ld, group, end, kind) of each."""
    if len(segments) > MAX_SEGMENTS:
        raise IndexError(f"at most {MAX_SEGMENTS} segments")
    flat = [v for s in segments for v in s] + [v for _ in range(MAX_SEGMENTS - len(segments)) for v in _NO_SEGMENT]
    return _structure(LinearArgs, _LINEAR_ARGS.pack(x, w, residual, bias, group_rows, ld_x, group_x, ld_w, group_w, ld_residual, *flat, rows, k, n,
                                                    groups, max_group_rows, len(segments), dtype, path, limit))


def linear_options(group_x_rows: int, x_rows: int, flags: int):
    """``b2kv_linear_options`` for ``lib``."""
    return _structure(LinearOptions, _LINEAR_OPTIONS.pack(group_x_rows, x_rows, flags))


def check(status: int) -> None:
    """Raise for a negative status of a C-ABI call."""
    if status == 0:
        return
    text = lib.b2kv_strerror(status).decode()
    if status == ERR_CUDA:
        text += ": " + lib.b2kv_last_cuda_error().decode()
    raise B2KVError(status, text)


def tune(name: str, value: int) -> None:
    check(lib.b2kv_tune(name.encode(), int(value)))
