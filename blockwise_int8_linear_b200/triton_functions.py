"""Functional operations of the blockwise-int8 linear layer.

Same names, signatures, return values and layouts as the reference's ``triton_functions.py``
(``quantize_block_rowwise`` 411-423, ``dequantize_block_rowwise`` 492-500,
``int8_matmul_block64_rowwise_dequantize`` 142-168, ``fast_matmulT`` 511-514); the module keeps
the reference's name although nothing here uses Triton: every function is one call into the extension
``_native`` (``csrc/torch_ops.cpp``), which validates the operands, allocates the outputs with torch and calls
``libbi8.so`` on the current CUDA stream.  There is no CPU path and no fallback.

Layouts: quantized tensors are int8 ``[rows, K]``; block scales ("state") are float32
``[ceil(K/block), rows]``.  ``block`` is ``block_linear_config.GROUP_SIZE`` read at call time
unless ``fblock_size`` is given.
"""
from __future__ import annotations

import torch

from . import _lib
from . import block_linear_config

__all__ = [
    "ceil_div", "quantize_block_rowwise", "quantize_block_colwise", "quantize_block_dual", "dequantize_block_rowwise",
    "int8_matmul_block64_rowwise_dequantize", "quantize_matmul_block_rowwise_dequantize", "int8_matmul_block_partials",
    "fast_matmulT", "rmsnorm_quantize_block_rowwise", "silu_mul_quantize_block_rowwise", "pre_quantize_matmul_block_rowwise_dequantize",
]


def ceil_div(n, d):
    return -(n // -d)


def _block(fblock_size=None) -> int:
    b = int(fblock_size or block_linear_config.GROUP_SIZE)
    if b < 1:
        raise ValueError(f"block size must be positive, got {b}")
    return b


def _scale_dtype():
    if block_linear_config.SHARED_EXP_TORCH_TYPE != torch.float32:
        raise ValueError("block scales are float32 only (block_linear_config.SHARED_EXP_TORCH_TYPE)")
    return torch.float32


_native = _lib.native


def quantize_block_rowwise(x: torch.Tensor, fblock_size=None):
    """Quantize each row of ``x [M, K]`` in blocks of ``block`` elements (``triton_functions.py:411-423``).

    Returns ``(q, state)``: ``q`` int8 ``[M, K]``; ``state`` float32 ``[ceil(K/block), M]`` holding
    ``max|x|`` of each block.  ``q = rint(127 * (x / state))`` (fp32 divide, fp32 multiply, round half to
    even); an all-zero block gives state 0 and q 0.  ``q`` is dense, except for a large 16-bit ``x`` (4 M elements, 256 on
    each side) whose ``K`` is not a multiple of 16: there it is a view of a buffer with a row pitch that is (same
    values), which the GEMM takes without a copy; call ``.contiguous()`` where a dense tensor is needed."""
    _scale_dtype()
    return _native().quantize_rowwise(x, _block(fblock_size), False)


def quantize_block_colwise(x: torch.Tensor, fblock_size=None):
    """``quantize_block_rowwise(x.t().contiguous())`` without materialising the transpose
    (the pattern at ``block_linear.py:93-94`` and ``100-103``).  ``x`` is ``[R, C]``; returns int8 ``[C, R]``
    and state ``[ceil(R/block), C]``, bit-identical to the two-step form (``q`` is laid out as there)."""
    _scale_dtype()
    return _native().quantize_colwise(x, _block(fblock_size), False)


def quantize_block_dual(x: torch.Tensor, fblock_size=None):
    """``quantize_block_rowwise(x)`` and ``quantize_block_colwise(x)`` from one read of ``x`` ``[R, C]``: returns
    ``(q_row [R, C], state_row [ceil(C/block), R], q_col [C, R], state_col [ceil(R/block), C])``, each bit-identical to its
    single-purpose function.  The layer needs both for its input (forward GEMM and weight gradient,
    ``block_linear.py:78, 100-101``) and for the output gradient (``block_linear.py:92, 102-103``)."""
    _scale_dtype()
    return _native().quantize_dual(x, _block(fblock_size))


def dequantize_block_rowwise(x: torch.Tensor, state_x: torch.Tensor, fblock_size=None):
    """``(state * q) * (1/127)`` cast to ``INPUT_OUTPUT_TORCH_TYPE`` (``triton_functions.py:492-500``)."""
    return _native().dequantize(x, state_x, _block(fblock_size), block_linear_config.INPUT_OUTPUT_TORCH_TYPE)


def int8_matmul_block64_rowwise_dequantize(a, b, state_x, state_w, bias=None, *, flags: int = 0):
    """Block GEMM with fused dequantize (``triton_functions.py:142-168``).

    ``a`` int8 ``[M, K]``; ``b`` int8 ``[K, N]`` (on the layer's path the ``.t()`` view of a row-major
    ``[N, K]`` tensor); ``state_x [ceil(K/block), M]``, ``state_w [ceil(K/block), N]`` float32; optional
    ``bias [N]``.  Returns a new ``[M, N]`` tensor of ``INPUT_OUTPUT_TORCH_TYPE``:
    ``sum_j state_w[j,n] * state_x[j,m] * (a_j . b_j) / 127**2`` accumulated in fp32, cast, then
    ``+ bias`` in the output type.  ``flags`` selects a kernel variant (see ``include/bi8.h``)."""
    return _native().gemm(a, b, state_x, state_w, bias, _block(), block_linear_config.INPUT_OUTPUT_TORCH_TYPE, flags)


def quantize_matmul_block_rowwise_dequantize(x, b, state_w, bias=None, *, flags: int = 0):
    """``int8_matmul_block64_rowwise_dequantize(*quantize_block_rowwise(x), ...)`` in one library call: the two steps
    of the layer's forward (``block_linear.py:141-143``).  ``x [M, K]`` floating point, ``b [K, N]`` int8 (the ``.t()``
    view of the ``[N, K]`` weights), ``state_w [ceil(K/block), N]``.  For ``M <= 64`` a decode quantizer runs
    overlapped with the start of the weight-streaming GEMM; the result is bit-identical to the two separate calls either way."""
    return _native().matmul(_lib.PRE_NONE, x, b, state_w, bias, None, None, 0.0, None, None, _block(),
                            block_linear_config.INPUT_OUTPUT_TORCH_TYPE, flags)


_PRE_CODE = {"none": _lib.PRE_NONE, "rmsnorm": _lib.PRE_RMSNORM, "silu_mul": _lib.PRE_SILU_MUL}


def _pre_code(op: str) -> int:
    code = _PRE_CODE.get(op)
    if code is None:
        raise ValueError(f"unknown producer step {op!r}: expected 'none', 'rmsnorm' or 'silu_mul'")
    return code


def rmsnorm_quantize_block_rowwise(x: torch.Tensor, eps: float = 1e-5, weight: torch.Tensor = None, fblock_size=None):
    """``quantize_block_rowwise(y)`` for ``y = (x * rsqrt(mean(x^2, -1) + eps) [* weight]).to(x.dtype)`` without writing
    ``y``: the normalisation in front of a layer's q/k/v and gate/up projections fused into their quantizer (the
    reference quantizes a tensor another kernel stored just before, ``block_linear.py:141``).  fp32 arithmetic, one
    rounding to ``x.dtype``, then the quantizer's own arithmetic; the row's sum of squares is taken in a fixed order."""
    _scale_dtype()
    return _native().quantize_pre(_lib.PRE_RMSNORM, x, None, weight, eps, _block(fblock_size))


def silu_mul_quantize_block_rowwise(gate: torch.Tensor, up: torch.Tensor, fblock_size=None):
    """``quantize_block_rowwise(F.silu(gate) * up)`` without writing the product (the gated activation in front of a
    layer's down projection): ``silu`` in fp32 rounded to the activation type, the product rounded again, as the two
    separate kernels would, then quantized; bit-identical to the three-step form."""
    _scale_dtype()
    return _native().quantize_pre(_lib.PRE_SILU_MUL, gate, up, None, 0.0, _block(fblock_size))


def pre_quantize_matmul_block_rowwise_dequantize(op: str, x, b, state_w, bias=None, *, x2=None, norm_weight=None, eps: float = 1e-5,
                                                 residual=None, out=None, flags: int = 0):
    """``quantize_matmul_block_rowwise_dequantize`` with the producer step ``op`` ('none', 'rmsnorm', 'silu_mul') fused
    in front of the quantizer and an optional ``residual [M, N]`` (of the output type) added to the result in the output
    type, the way a transformer layer's ``x + proj(act(...))`` does.  ``out`` may be given (it may be ``residual``
    itself: updated in place, directly on the decode path, through a temporary elsewhere).  For ``M <= 64`` this is
    quantizer + weight-streaming GEMM (+ its reduction), with the residual added by the kernel that writes the result."""
    return _native().matmul(_pre_code(op), x, b, state_w, bias, x2, norm_weight, eps, residual, out, _block(),
                            block_linear_config.INPUT_OUTPUT_TORCH_TYPE, flags)


def int8_matmul_block_partials(a, b, fblock_size=None, *, flags: int = 0):
    """Exact int32 block partial sums ``P[j] = a[:, jB:(j+1)B] @ b[jB:(j+1)B, :]`` as ``[ceil(K/B), M, N]``,
    produced by the same loads and tensor-core instructions as the GEMM (``triton_functions.py:115``)."""
    return _native().block_partials(a, b, _block(fblock_size), flags)


def fast_matmulT(a, b):
    """``a [M, K] @ b[N, K]^T`` with both operands quantized on the fly (``triton_functions.py:511-514``)."""
    _scale_dtype()
    a_int8, a_state = _native().quantize_rowwise(a, _block(), True)
    b_int8, b_state = _native().quantize_rowwise(b, _block(), True)
    return int8_matmul_block64_rowwise_dequantize(a_int8, b_int8.t(), a_state, b_state)
