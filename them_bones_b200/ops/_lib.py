"""ctypes binding of the native library ``them_bones_b200/lib/libbones_b200.so``.

The library is plain C ABI: every entry point takes raw device pointers, sizes and the CUDA stream, launches
asynchronously and returns 0 or an error code.  It is built in-tree by ``csrc/build.py`` (nvcc, sm_100a) and is
required on a GPU: a missing or unloadable library raises here rather than letting a GPU run continue on a fallback.
"""
from __future__ import annotations

import ctypes
import os

import torch

_LIB = None
DEBUG_BOUNDS = os.environ.get("BONES_DEBUG_BOUNDS", "0") not in ("0", "", "false")
# BONES_LIB: path of another build of the library (for instance one compiled with a measuring define)
_PATH = os.environ.get("BONES_LIB") or os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lib",
                                                    "libbones_b200_dbg.so" if DEBUG_BOUNDS else "libbones_b200.so")


def lib_path() -> str:
    return _PATH


_P, _I, _L, _F = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
_GEMM = [_P] * 4 + [_I] * 4 + [_L] * 8 + [_I] * 3 + [_F] * 2
# Entry points called with plain Python numbers (converted by ctypes itself: building two dozen argument objects in Python was
# a third of a GEMM's host time).  Everything else passes ctypes objects.
SIGNATURES = {
    "bones_gemm_bf16": _GEMM + [_I] * 3 + [_P],                     # ..., force_bn, splits, atomic, stream
    "bones_gemm_bf16_pair": _GEMM + [_I] * 2 + [_P],
    "bones_gemm_bf16_auto": _GEMM + [_I] * 2 + [_P],
    "bones_mlp_bf16_fwd": [_P] * 6 + [_I] * 4 + [_L] * 4 + [_I, _P],     # ..., GEMM_MODE, stream
    "bones_mlp_bf16_bwd": [_P] * 9 + [_I] * 4 + [_L] * 4 + [_I, _P],
    "bones_attention_fwd": [_P] * 8 + [_I] * 4 + [_F, _I, _P],
    "bones_attention_bwd": [_P] * 13 + [_I] * 4 + [_F, _I, _P],
    "bones_mx2_quant": [_P, _L, _P, _P, _I, _P, _P, _I, _L, _L, _I, _P],
    "bones_gemm_mxfp8_pair": [_P] * 8 + [_I] + [_P] * 2 + [_I] * 5 + [_L] * 8 + [_I] * 3 + [_F] * 2 + [_I] * 3 + [_P],
}


def load():
    global _LIB
    if _LIB is None:
        if not os.path.exists(_PATH):
            raise RuntimeError(f"native library missing: {_PATH}; run `python -m them_bones_b200.csrc.build` "
                               "(or __graft_entry__.build()) first")
        lib = ctypes.CDLL(_PATH)
        for name, types in SIGNATURES.items():
            getattr(lib, name).argtypes = types
        _LIB = lib
    return _LIB


def available() -> bool:
    try:
        load()
        return True
    except (RuntimeError, OSError):
        return False


def raw_stream() -> int:
    """The current stream's handle as a number, for the entry points of ``SIGNATURES``."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def ptr(t):
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def stream():
    """The current stream's handle, without building a ``torch.cuda.Stream`` object (4 us of a 10 us launch)."""
    return ctypes.c_void_p(raw_stream())


LAUNCHES = [0]        # native kernel launches issued by this process (`launches`: an entry point with more than one kernel)


def call(name: str, *args, launches: int = 1):
    LAUNCHES[0] += launches
    rc = getattr(_LIB or load(), name)(*args)
    if rc != 0:
        raise RuntimeError(f"{name} failed with code {rc}")


def check_error_word():
    """Raises if any kernel on the current device gave up on a bounded wait since the last check.  Synchronises."""
    rc = load().bones_error_read_clear()
    if rc != 0:
        raise RuntimeError(f"a native kernel reported error code {rc} (bounded wait expired or bad argument)")
    if DEBUG_BOUNDS:
        hits = bounds_hits()
        if hits:
            raise RuntimeError(f"debug-bounds build: out-of-range indices were caught and skipped: {hits}")


def bounds_hits() -> dict:
    """Debug-bounds library only: ``{source file: (count, offending index, source line)}`` of the index checks that
    failed since the last call (read and cleared; synchronises)."""
    out = {}
    lib = load()
    for tu in ("elementwise", "comm", "tables"):
        fn = getattr(lib, f"bones_bounds_hits_{tu}", None)
        if fn is None:
            continue
        last = (ctypes.c_longlong * 2)()
        n = fn(last)
        if n:
            out[tu] = (int(n), int(last[0]), int(last[1]))
    return out


EPI_BF16, EPI_BF16_RES, EPI_RELU2, EPI_ACC_F32, EPI_MUL_2SQRT, EPI_F32, EPI_F32_RES, EPI_SOFTCAP = range(8)


PAIR_MODE = os.environ.get("BONES_GEMM_PAIR", "auto")      # auto | 0 | 1
GEMM_MODE = {"auto": 0, "1": 1}.get(PAIR_MODE, 2)


def gemm(a, b, d, *, m, n, k, lda, ldb, ldd, a_major=0, b_major=0, epi=EPI_BF16, r=None, ldr=0, alpha=1.0, beta=1.0,
         batch=1, stride_a=0, stride_b=0, stride_d=0, stride_r=0, force_bn=0, splits=0, pair=None, d_ptr=None, atomic=False):
    """``d = epilogue(alpha * a @ b^T, r)``; see csrc/gemm_bf16.cu for operand layouts.  ``pair=None``: CTA
    pairs (csrc/gemm_bf16_2cta.cu) or single CTAs by the rule of ``bones_gemm_bf16_auto``."""
    auto = pair is None and PAIR_MODE == "auto" and force_bn == 0
    if pair is None:
        pair = PAIR_MODE == "1" and force_bn == 0
    # d_ptr: raw device address used instead of ``d`` (e.g. the same buffer in another GPU's memory); atomic: fp32
    # accumulation by vector atomics even without split-K, for outputs several GPUs add into at once
    dp = d.data_ptr() if d_ptr is None else int(d_ptr)
    rp = r.data_ptr() if r is not None else 0
    st = raw_stream()
    if auto or pair:
        call("bones_gemm_bf16_auto" if auto else "bones_gemm_bf16_pair", a.data_ptr(), b.data_ptr(), dp, rp, m, n, k, batch, lda, ldb, ldd, ldr,
             stride_a, stride_b, stride_d, stride_r, a_major, b_major, epi, alpha, beta, splits, int(atomic), st)
        return
    call("bones_gemm_bf16", a.data_ptr(), b.data_ptr(), dp, rp, m, n, k, batch, lda, ldb, ldd, ldr, stride_a, stride_b, stride_d, stride_r, a_major,
         b_major, epi, alpha, beta, force_bn, splits, int(atomic), st)
