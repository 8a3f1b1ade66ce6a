"""A persistent compressed KV cache on the device, in the library's wire format.

The reference patches models with `use_cache = False` and recompresses the whole prefix for every
generated token (src/transformers_turboquant/patch.py:80-81); its cache exists as a concept only
(src/turboquant_pytorch/turboquant.py:199-286: append compressed entries, score queries against
them).  `CompressedKVCache` is that concept on the CUDA kernels: packed buffers with room for
`capacity` tokens per (batch, KV head), `append` compresses new tokens behind the ones in use, and
`attend` runs compressed attention of new queries over everything stored -- the split-KV kernel reads
the buffers in place, so a decode step touches each packed byte once and copies nothing.
"""

from __future__ import annotations

import torch

from . import _lib
from .compressors import (_attend, _require_cuda, TurboQuantCompressorMSE, TurboQuantCompressorV2, prepared_constants,
                          resolve_mode)


class CompressedKVCache:
    """Packed keys and values of `batch` sequences and `kv_heads` KV heads, up to `capacity` tokens each.

    Buffers (row (b, h, t)): key indices u8 [.., d*(bits-1)/8], key sign bits u8 [.., d/8], key vector and
    residual norms fp16, value indices u8 [.., d*bits/8], value vector norms fp16 -- the layout
    `compress()` returns, with a token stride of `capacity` instead of the current length.
    """

    def __init__(self, key_compressor: TurboQuantCompressorV2, val_compressor: TurboQuantCompressorMSE,
                 batch: int, kv_heads: int, capacity: int, device="cuda"):
        if key_compressor.bits != val_compressor.bits or key_compressor.head_dim != val_compressor.head_dim:
            raise ValueError("key and value compressors must share bit width and head_dim")
        if capacity < 1:
            raise ValueError("capacity must be positive")
        self.key_compressor, self.val_compressor = key_compressor, val_compressor
        self.batch, self.kv_heads, self.capacity = int(batch), int(kv_heads), int(capacity)
        self.head_dim, self.bits = key_compressor.head_dim, key_compressor.bits
        d, kb, vb = self.head_dim, key_compressor.mse_bits, val_compressor.bits
        dev = torch.device(device)
        shape = (self.batch, self.kv_heads, self.capacity)
        self.key_indices = torch.zeros(shape + (d * kb // 8,), dtype=torch.uint8, device=dev)
        self.key_signs = torch.zeros(shape + (d // 8,), dtype=torch.uint8, device=dev)
        self.key_norms = torch.zeros(shape, dtype=torch.float16, device=dev)
        self.key_residual_norms = torch.zeros(shape, dtype=torch.float16, device=dev)
        self.value_indices = torch.zeros(shape + (d * vb // 8,), dtype=torch.uint8, device=dev)
        self.value_norms = torch.zeros(shape, dtype=torch.float16, device=dev)
        self.length = 0

    def __len__(self) -> int:
        return self.length

    def nbytes(self) -> int:
        """Bytes the tokens in use occupy (what a decode step reads)."""
        d, kb, vb = self.head_dim, self.key_compressor.mse_bits, self.val_compressor.bits
        per_token = d * kb // 8 + d // 8 + 4 + d * vb // 8 + 2
        return self.batch * self.kv_heads * self.length * per_token

    def reset(self) -> None:
        self.length = 0

    def append(self, keys: torch.Tensor, values: torch.Tensor) -> None:
        """Compress [B, Hkv, S_new, D] keys and values and store them behind the tokens in use."""
        B, H, S, D = keys.shape
        if values.shape != keys.shape or (B, H, D) != (self.batch, self.kv_heads, self.head_dim):
            raise ValueError(f"expected [{self.batch}, {self.kv_heads}, S, {self.head_dim}] keys and values, got "
                             f"{tuple(keys.shape)} and {tuple(values.shape)}")
        if self.length + S > self.capacity:
            raise ValueError(f"cache holds {self.length} of {self.capacity} tokens; cannot append {S}")
        _require_cuda(keys, "keys")
        kc, vc = self.key_compressor, self.val_compressor
        kc._check_device(keys)
        vc._check_device(keys)
        # one launch compresses both sides straight behind the tokens in use: no scratch, no copies
        _lib.host.append(keys, values, prepared_constants(kc, vc), kc.bits, resolve_mode(keys.dtype, kc.mode), self.key_indices,
                         self.key_signs, self.key_norms, self.key_residual_norms, self.value_indices, self.value_norms,
                         self.capacity, self.length)
        self.length += S

    def attend(self, q: torch.Tensor, causal: bool = True, sm_scale: float | None = None,
               attention_mask: torch.Tensor | None = None) -> torch.Tensor:
        """softmax(scores * sm_scale) @ V_hat of q [B, Hq, Sq, D] over the tokens in use; with `causal` the
        queries are the last Sq positions (append their keys first).  Returns [B, Hq, Sq, D] in q.dtype.

        `attention_mask` is an optional additive mask broadcastable to [B, 1, Sq, tokens in use] (padding).
        The cache is read in place, whatever the number of queries and the arithmetic mode."""
        _require_cuda(q, "q")
        B, Hq, Sq, D = q.shape
        if (B, D) != (self.batch, self.head_dim) or Hq % self.kv_heads != 0:
            raise ValueError(f"queries {tuple(q.shape)} do not match the cache")
        if self.length == 0:
            raise ValueError("attention over an empty cache is undefined")
        kc, vc = self.key_compressor, self.val_compressor
        kc._check_device(q)
        vc._check_device(q)
        # The prefill kernels follow the token stride of the cache as the split-KV kernel does: dense copies of the
        # prefix are six strided copies per call (a 300-token chunk behind 8 000 tokens: 149 us with them, 115 us
        # without; a step of a GPT-2-shaped layer over 700 tokens: 140 and 55 us).
        packed = (self.key_indices, self.key_signs, self.key_norms, self.key_residual_norms, self.value_indices,
                  self.value_norms)
        return _attend(q, self.kv_heads, self.length, self.capacity, packed, kc, vc, sm_scale, causal, attention_mask,
                       resolve_mode(q.dtype, kc.mode))
