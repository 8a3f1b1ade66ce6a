"""Rotary position embedding of a layer's query and key heads in one CUDA launch.

The reference's adapters call HF's `apply_rotary_pos_emb(q, k, cos, sin)` right before they compress the keys
(src/transformers_turboquant/families/llama.py:98): four elementwise torch kernels and a concatenation per
tensor.  `rope` does the same arithmetic, to the bit, reading and writing every element once."""

from __future__ import annotations

import torch

from . import _lib
from .compressors import _require_cuda


def rope_applies(q: torch.Tensor, k: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor) -> bool:
    """Whether `rope` covers these tensors: CUDA, one dtype the kernels know, rotary width = head_dim (a multiple
    of 32), cos/sin shaped [B or 1, S, d] with contiguous rows."""
    return _lib.host.rope_covers(q, k, cos, sin)


def rope(q: torch.Tensor, k: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor):
    """(q * cos + rotate_half(q) * sin, k * cos + rotate_half(k) * sin) for q [B, Hq, S, d], k [B, Hkv, S, d] (any
    strides with contiguous rows) and cos, sin [B or 1, S, d]; returns new contiguous tensors."""
    _require_cuda(q, "q")
    out = _lib.host.rope(q, k, cos, sin)
    if out is None:
        raise ValueError(f"rope: unsupported arguments q {tuple(q.shape)} {q.dtype}, k {tuple(k.shape)} {k.dtype}, "
                         f"cos {tuple(cos.shape)} {cos.dtype}")
    return out
