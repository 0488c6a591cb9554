"""Loading of libbi8.so (declared in include/bi8.h), through ctypes, and of the extension that calls it for the functional
operations.

There is no fallback: if the library cannot be loaded, or a call returns an error status, an
exception is raised.  Tensors are passed as raw device pointers plus sizes; the current torch
CUDA stream is passed to every call.
"""
from __future__ import annotations

import ctypes
import os

import torch

_HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(_HERE, "libbi8.so")

BI8_BF16, BI8_F32, BI8_F16 = 0, 1, 2
GEMM_DEFAULT, GEMM_FORCE_GENERIC, GEMM_FORCE_TC, GEMM_NO_SEED, GEMM_FORCE_SMALLM, GEMM_FORCE_SKINNY = 0, 1, 2, 4, 8, 16
GEMM_QUANT_IN_KERNEL = 32

_DTYPE_CODE = {torch.bfloat16: BI8_BF16, torch.float32: BI8_F32, torch.float16: BI8_F16}

EXPORTS = [
    "bi8_version", "bi8_last_error_string", "bi8_device_status", "bi8_quantize_rowwise", "bi8_quantize_colwise", "bi8_quantize_dual", "bi8_peer_allreduce", "bi8_peer_allreduce_buffer_bytes", "bi8_row_parallel_linear",
    "bi8_dequantize_rowwise", "bi8_gemm_dequant", "bi8_gemm_workspace_bytes", "bi8_gemm_workspace_used", "bi8_quantize_many", "bi8_quantize_many_fits", "bi8_quantize_dual_sum", "bi8_quantize_dual_sum_workspace_bytes", "bi8_gemm_block_partials",
    "bi8_gemm_dequant_fused_quant", "bi8_mma_peak_probe", "bi8_gemm_dequant_static", "bi8_gemm_static_scratch_bytes",
    "bi8_gemm_wait_selftest", "bi8_stream_capture_id", "bi8_quantize_rowwise_pre", "bi8_gemm_dequant_fused_pre",
    "bi8_row_parallel_linear_pre", "bi8_peer_allreduce_large", "bi8_peer_allreduce_large_buffer_bytes",
    "bi8_peer_allreduce_large_partial_offset", "bi8_peer_allreduce_large_out_offset", "bi8_rope_cache_append",
    "bi8_gemm_dequant_residual", "bi8_quantize_rowwise_pitched", "bi8_quantize_colwise_pitched", "bi8_quantize_dual_pitched",
    "bi8_quantize_rowwise_pre_pitched", "bi8_dequantize_rowwise_pitched", "bi8_column_sum", "bi8_column_sum_workspace_bytes",
    "bi8_copy_rows",
]
ADDEND_FULL = 0x100
PRE_NONE, PRE_RMSNORM, PRE_SILU_MUL = 0, 1, 2

_lib = None
_native = None


class Bi8Error(RuntimeError):
    """A libbi8 entry point returned a non-zero status."""


def lib() -> ctypes.CDLL:
    global _lib
    if _lib is None:
        if not os.path.exists(LIB_PATH):
            raise ImportError(
                f"{LIB_PATH} is missing: build it with `python -m blockwise_int8_linear_b200.build` "
                "(there is no non-CUDA fallback)")
        L = ctypes.CDLL(LIB_PATH)
        c = ctypes
        vp, i64, i32, sz = c.c_void_p, c.c_int64, c.c_int, c.c_size_t
        L.bi8_version.restype = i32
        L.bi8_last_error_string.restype = c.c_char_p
        L.bi8_device_status.argtypes = [c.POINTER(i32)]
        L.bi8_quantize_rowwise.argtypes = [vp, i32, i64, vp, vp, i64, i64, i32, vp]
        L.bi8_quantize_colwise.argtypes = [vp, i32, i64, vp, vp, i64, i64, i32, vp]
        L.bi8_quantize_dual.argtypes = [vp, i32, i64, vp, vp, vp, vp, i64, i64, i32, vp]
        L.bi8_dequantize_rowwise.argtypes = [vp, vp, vp, i32, i64, i64, i32, vp]
        L.bi8_gemm_dequant_residual.argtypes = [vp, i64, vp, i64, vp, vp, vp, i32, vp, i64, vp, i64, i32, i64, i64, i64, i32, vp, sz, i32, vp]
        L.bi8_quantize_rowwise_pitched.argtypes = [vp, i32, i64, vp, i64, vp, i64, i64, i32, vp]
        L.bi8_quantize_colwise_pitched.argtypes = [vp, i32, i64, vp, i64, vp, i64, i64, i32, vp]
        L.bi8_quantize_dual_pitched.argtypes = [vp, i32, i64, vp, i64, vp, vp, i64, vp, i64, i64, i32, vp]
        L.bi8_quantize_rowwise_pre_pitched.argtypes = [i32, vp, vp, i32, i64, vp, c.c_float, vp, i64, vp, i64, i64, i32, vp]
        L.bi8_copy_rows.argtypes = [vp, i64, vp, i64, i64, i64, vp]
        L.bi8_column_sum.argtypes = [vp, i32, i64, vp, i64, i64, vp, sz, vp]
        L.bi8_column_sum_workspace_bytes.argtypes = [i64, i64]
        L.bi8_column_sum_workspace_bytes.restype = sz
        L.bi8_dequantize_rowwise_pitched.argtypes = [vp, i64, vp, vp, i32, i64, i64, i32, vp]
        L.bi8_peer_allreduce_buffer_bytes.argtypes = [i32, i64]
        L.bi8_peer_allreduce_buffer_bytes.restype = sz
        L.bi8_row_parallel_linear.argtypes = [vp, i32, i64, vp, vp, vp, i64, vp, vp, i64, i64, i64, i32, vp, sz, c.POINTER(vp), i32, i32,
                                              i64, vp, i32, vp, i32, c.c_uint, i32, vp]
        L.bi8_row_parallel_linear_pre.argtypes = [i32, vp, vp, i32, i64, vp, c.c_float, vp, vp, vp, i64, vp, vp, i64, i64, i64, i32, vp, sz,
                                                  c.POINTER(vp), i32, i32, i64, vp, i32, vp, i32, c.c_uint, i32, vp]
        L.bi8_peer_allreduce_large.argtypes = [c.POINTER(vp), i32, i32, i64, i64, i64, vp, i32, i32, c.c_uint, vp]
        L.bi8_peer_allreduce_large_buffer_bytes.argtypes = [i32, i64]
        L.bi8_peer_allreduce_large_buffer_bytes.restype = sz
        L.bi8_peer_allreduce_large_partial_offset.argtypes = []
        L.bi8_peer_allreduce_large_partial_offset.restype = sz
        L.bi8_peer_allreduce_large_out_offset.argtypes = [i64]
        L.bi8_peer_allreduce_large_out_offset.restype = sz
        L.bi8_rope_cache_append.argtypes = [vp, i32, vp, vp, vp, vp, vp, i64, i64, i64, i64, vp]
        L.bi8_peer_allreduce.argtypes = [c.POINTER(vp), i32, i32, i64, vp, i64, i64, vp, i32, vp, i32, c.c_uint, vp]
        L.bi8_gemm_dequant.argtypes = [vp, i64, vp, i64, vp, vp, vp, i32, vp, i64, i32, i64, i64, i64, i32, vp, sz, i32, vp]
        L.bi8_gemm_workspace_bytes.argtypes = [i64, i64, i64, i32]
        L.bi8_gemm_workspace_bytes.restype = sz
        L.bi8_gemm_workspace_used.argtypes = [i64, i64, i64, i32]
        L.bi8_gemm_workspace_used.restype = sz
        L.bi8_quantize_dual_sum.argtypes = [vp, i32, i64, vp, i64, vp, vp, i64, vp, vp, i64, i64, i32, vp, sz, vp]
        L.bi8_quantize_dual_sum_workspace_bytes.argtypes = [i32, i64, i64, i32]
        L.bi8_quantize_dual_sum_workspace_bytes.restype = sz
        L.bi8_quantize_many.argtypes = [vp, i32, i32, vp]
        L.bi8_quantize_many_fits.argtypes = [vp, i32, i32]
        L.bi8_gemm_block_partials.argtypes = [vp, i64, vp, i64, vp, i64, i64, i64, i32, i32, vp]
        L.bi8_gemm_dequant_fused_quant.argtypes = [vp, i32, i64, vp, vp, vp, i64, vp, vp, i32, vp, i64, i32, i64, i64, i64, i32, vp,
                                                   sz, i32, vp]
        L.bi8_quantize_rowwise_pre.argtypes = [i32, vp, vp, i32, i64, vp, c.c_float, vp, vp, i64, i64, i32, vp]
        L.bi8_gemm_dequant_fused_pre.argtypes = [i32, vp, vp, i32, i64, vp, c.c_float, vp, vp, vp, i64, vp, vp, i32, vp, i64, vp, i64, i32,
                                                 i64, i64, i64, i32, vp, sz, i32, vp]
        L.bi8_gemm_wait_selftest.argtypes = [vp, i64, vp, i64, vp, vp, vp, i64, i32, i64, i64, i64, i32, c.c_uint, i32, vp]
        L.bi8_stream_capture_id.argtypes = [vp, c.POINTER(c.c_ulonglong)]
        L.bi8_mma_peak_probe.argtypes = [i32, c.POINTER(c.c_float), c.POINTER(i32)]
        for name in EXPORTS:
            fn = getattr(L, name)
            if name not in ("bi8_last_error_string", "bi8_gemm_workspace_bytes", "bi8_gemm_workspace_used", "bi8_quantize_dual_sum_workspace_bytes", "bi8_gemm_static_scratch_bytes",
                            "bi8_peer_allreduce_buffer_bytes", "bi8_peer_allreduce_large_buffer_bytes", "bi8_column_sum_workspace_bytes",
                            "bi8_peer_allreduce_large_partial_offset", "bi8_peer_allreduce_large_out_offset"):
                fn.restype = i32
        _lib = L
    return _lib


def native():
    """The extension module that runs the functional operations (``csrc/torch_ops.cpp``)."""
    global _native
    if _native is None:
        lib()
        if not os.path.exists(os.path.join(_HERE, "_native.so")):
            raise ImportError(
                f"{os.path.join(_HERE, '_native.so')} is missing: build it with `python -m blockwise_int8_linear_b200.build` "
                "(there is no non-CUDA fallback)")
        from . import _native as module
        from . import block_linear_config
        module.bind(Bi8Error, block_linear_config)
        _native = module
    return _native


def check(status: int, what: str) -> None:
    if status != 0:
        msg = lib().bi8_last_error_string().decode(errors="replace")
        raise Bi8Error(f"{what} failed with status {status}: {msg}")


def dtype_code(dtype: torch.dtype) -> int:
    try:
        return _DTYPE_CODE[dtype]
    except KeyError:
        raise ValueError(f"unsupported dtype {dtype}: expected bfloat16, float16 or float32") from None


def ptr(t) -> ctypes.c_void_p:
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def stream_ptr() -> ctypes.c_void_p:
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def device_status() -> int:
    """Synchronises and returns the device-side status word (0 = clean); raises on a recorded timeout."""
    detail = ctypes.c_int(0)
    rc = lib().bi8_device_status(ctypes.byref(detail))
    check(rc, "bi8_device_status")
    return rc
