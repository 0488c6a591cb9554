"""Model-side helpers for a decode step that sit between two of the library's kernels (the reference has no model code).

``rope_cache_append`` takes what a fused q/k/v ``BlockInt8Linear`` leaves for one new token per sequence, rotates q and k by
the position's angle and appends k and v to the caches in one launch (``bi8_rope_cache_append``); written with tensor
operations the same step is five launches per layer.
"""
from __future__ import annotations

import torch

from . import _lib

__all__ = ["rope_cache_append"]


def rope_cache_append(qkv: torch.Tensor, cis: torch.Tensor, pos: torch.Tensor, kcache: torch.Tensor, vcache: torch.Tensor) -> torch.Tensor:
    """``qkv [B, 3, H, D]`` (bf16 / fp16, contiguous): q, k, v of one new token per sequence.  ``cis [D/2]`` complex64 (or
    ``[D/2, 2]`` float32: cos, sin) of the step's position, ``pos`` an int64 device tensor with one element (the cache row),
    ``kcache`` / ``vcache [B, H, max_len, D]`` contiguous.  Returns the rotated q as ``[B, H, 1, D]``; row ``pos`` of the caches
    receives the rotated k and v.  Feature pairs are (even, odd) neighbours: ``(x0 + i x1) * cis``."""
    return _lib.native().rope_cache_append(qkv, cis, pos, kcache, vcache)
