"""Key / value compressors backed by the sm_100a CUDA library.

`TurboQuantCompressorV2` and `TurboQuantCompressorMSE` keep the constructor signature,
attribute names (`Pi, PiT, S, centroids, boundaries, bits, mse_bits, head_dim, device`)
and methods (`compress`, `asymmetric_attention_scores`, `decompress`) of the reference
classes (src/turboquant_pytorch/compressors.py:36-317) and always produce its bit-packed
result layout (compressors.py:132-138, :281-285).  Inputs must live on a CUDA device; there
is no CPU path.  `fused_attention` is the entry the family adapters call: compressed causal
attention without the score matrix or decompressed K/V.
"""

from __future__ import annotations

import math
import os

import torch

from . import _lib
from .codebook import lloyd_max_centroids, midpoints

_DTYPES = {torch.float32: _lib.TQ_F32, torch.bfloat16: _lib.TQ_BF16, torch.float16: _lib.TQ_F16}
_MODES = {"fp32": _lib.TQ_MODE_FP32, "bf16": _lib.TQ_MODE_BF16}


def resolve_mode(dtype: torch.dtype, mode: str | None = None) -> int:
    """Arithmetic mode of a call.  Explicit `mode`, else the TQ_B200_MODE environment
    variable ("fp32" | "bf16"), else by input type: fp32 inputs run the fp32 parity
    kernels, 16-bit inputs the tensor-core kernels."""
    mode = mode or os.environ.get("TQ_B200_MODE") or "auto"
    if mode == "auto":  # (types the kernels do not know are read as fp32)
        return _lib.TQ_MODE_BF16 if dtype in (torch.bfloat16, torch.float16) else _lib.TQ_MODE_FP32
    if mode not in _MODES:
        raise ValueError(f"mode must be 'fp32', 'bf16' or 'auto', got {mode!r}")
    return _MODES[mode]


def _stream_ptr(device) -> int:
    return torch.cuda.current_stream(device).cuda_stream


def _require_cuda(t: torch.Tensor, what: str) -> None:
    if not t.is_cuda:
        raise RuntimeError(f"{what} must be a CUDA tensor: turboquant_b200 has no CPU path")


_KEY_ARRAYS = ("packed_key_indices", "packed_qjl_signs", "vec_norms", "residual_norm")
_VALUE_ARRAYS = ("packed_indices", "vec_norms")


def _dense_packed(compressed: dict, keys: tuple) -> dict:
    """The packed arrays of a compressed dictionary as the kernels read them: dense rows, one per (b, h, s) in that
    order.  A strided view (a slice of a larger buffer) is copied; a wrong row count is refused, not read past."""
    B, H, S, _ = compressed["shape"]
    out = dict(compressed)
    for name in keys:
        t = compressed[name]
        rows = t.numel() // max(t.shape[-1], 1) if name.startswith("packed") else t.numel()  # packed: [..., bytes]
        if rows != B * H * S:
            raise ValueError(f"{name} holds {tuple(t.shape)} entries for a compressed shape {compressed['shape']}")
        out[name] = t if t.is_contiguous() else t.contiguous()
    return out


def _haar_rotation(d: int, seed: int) -> torch.Tensor:
    """Seeded random rotation: Q factor of a Gaussian matrix with the sign convention
    diag(R) > 0 (compressors.py:50-56).  Generated on the CPU generator so that a seed
    means the same matrix everywhere."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    q, r = torch.linalg.qr(torch.randn(d, d, generator=g))
    s = torch.sign(torch.diagonal(r))
    s[s == 0] = 1.0
    return q * s


class _Constants:
    """Device-resident fp32 constants of a compressor and their movement between devices."""

    _tensor_attrs: tuple[str, ...] = ()

    def __setattr__(self, name, value):
        # Replacing a constant (tests overwrite them with the oracle's) invalidates the operand images prepared
        # from it.  In-place edits of a constant tensor are not seen: assign a new tensor instead.
        if name in self._tensor_attrs:
            self.__dict__["_version"] = self.__dict__.get("_version", 0) + 1
        object.__setattr__(self, name, value)

    def to(self, device):
        device = torch.device(device)
        for name in self._tensor_attrs:
            setattr(self, name, getattr(self, name).to(device=device, dtype=torch.float32).contiguous())
        self.device = str(device)
        return self

    def _check_device(self, t: torch.Tensor) -> None:
        if self.Pi.device != t.device:
            self.to(t.device)


_PAD = {}


def _zeros16(dev) -> torch.Tensor:
    """Stand-in for the codebook of a side that a one-sided constants buffer does not have."""
    key = str(dev)
    if key not in _PAD:
        _PAD[key] = torch.zeros(16, dtype=torch.float32, device=dev)
    return _PAD[key]


def _prepare(kc, vc, bits: int, d: int, dev) -> torch.Tensor:
    """One constants buffer (tq_prepare_constants) for a key compressor, a value compressor or both; the missing
    side is filled with stand-ins that no call reads."""
    pad = _zeros16(dev)
    any_pi = (kc or vc).Pi
    args = [kc.Pi if kc else any_pi, kc.S_eff if kc else any_pi, kc.centroids if kc else pad,
            kc.boundaries if kc else pad, vc.Pi if vc else any_pi, vc.centroids if vc else pad,
            vc.boundaries if vc else pad]
    nbytes = _lib.lib.tq_constants_bytes(d, bits)
    buf = torch.empty(nbytes, dtype=torch.uint8, device=dev)
    _lib.check(_lib.lib.tq_prepare_constants(*[t.data_ptr() for t in args], bits, d, buf.data_ptr(), nbytes,
                                             _stream_ptr(dev)))
    return buf


def prepared_constants(kc=None, vc=None) -> torch.Tensor:
    """The device buffer of operand images and fp32 constants for this compressor pair (or one compressor),
    built on first use and kept until one of the constants is replaced or moved."""
    owner = kc if kc is not None else vc
    key = (id(kc) if kc else 0, id(vc) if vc else 0)
    ver = (kc._version if kc else 0, vc._version if vc else 0)
    cache = owner.__dict__.setdefault("_prepared", {})
    hit = cache.get(key)
    if hit is None or hit[0] != ver:
        if kc is not None and vc is not None and (kc.bits != vc.bits or kc.head_dim != vc.head_dim):
            raise ValueError("key and value compressors must share bit width and head_dim")
        cache[key] = hit = (ver, _prepare(kc, vc, owner.bits, owner.head_dim, owner.Pi.device))
    return hit[1]


def compress_kv(keys, values, key_compressor=None, val_compressor=None):
    """Compress keys and values [B, H, S, D] in ONE launch (either may be None): what the family adapters do with
    `key_compressor.compress(k)` and `val_compressor.compress(v)` back to back (families/llama.py:103-104 of
    the reference).  Returns (compressed_keys, compressed_values) in the packed layout of `compress`."""
    kc, vc = (key_compressor if keys is not None else None), (val_compressor if values is not None else None)
    ref = keys if keys is not None else values
    if ref is None or (kc is None and vc is None):
        raise ValueError("nothing to compress")
    _require_cuda(ref, "states")
    for comp in (kc, vc):
        if comp is not None:
            comp._check_device(ref)
    B, H, S, D = ref.shape
    owner = kc or vc
    if D != owner.head_dim or (keys is not None and values is not None and values.shape != keys.shape):
        raise ValueError(f"expected [B, H, S, {owner.head_dim}] keys and values of one shape")
    ki, ks, rn, vn, vi, vv = _lib.host.compress(keys if kc is not None else None, values if vc is not None else None,
                                                prepared_constants(kc, vc), owner.bits, resolve_mode(ref.dtype, owner.mode))
    ck = cv = None
    if kc is not None:
        ck = {"packed_key_indices": ki, "packed_qjl_signs": ks, "residual_norm": rn, "vec_norms": vn, "shape": (B, H, S, D)}
    if vc is not None:
        cv = {"packed_indices": vi, "vec_norms": vv, "shape": (B, H, S, D)}
    return ck, cv


class TurboQuantCompressorV2(_Constants):
    """Key compressor: (bits-1)-bit Lloyd-Max indices of the rotated unit vector plus a
    1-bit QJL sketch of the residual (compressors.py:36-224)."""

    _tensor_attrs = ("Pi", "PiT", "S", "S_eff", "centroids", "boundaries")

    def __init__(self, head_dim: int, bits: int, seed: int, device: str = "cuda", use_triton: bool = True,
                 mode: str | None = None):
        if head_dim not in (64, 128):
            raise ValueError(f"head_dim {head_dim} unsupported by the CUDA kernels (64 or 128)")
        if bits not in (2, 3, 4):
            raise ValueError(f"bits must be 2, 3 or 4, got {bits}")
        self.head_dim, self.bits, self.mse_bits = head_dim, bits, max(bits - 1, 1)
        self.use_triton = use_triton  # accepted for call compatibility; there is one backend
        self.mode = mode
        self.Pi = _haar_rotation(head_dim, seed)
        self.PiT = self.Pi.T.contiguous()
        self.centroids = lloyd_max_centroids(head_dim, self.mse_bits)
        self.boundaries = midpoints(self.centroids)
        g = torch.Generator(device="cpu").manual_seed(seed + 10000)
        self.S = torch.randn(head_dim, head_dim, generator=g)
        self.S_eff = self.S @ self.Pi.T  # sketch matrix in rotated coordinates
        self.to(device)

    def compress(self, states: torch.Tensor) -> dict:
        """[B, H, S, D] -> packed dict (one fused kernel)."""
        if states.dim() != 4 or states.shape[-1] != self.head_dim:
            raise ValueError(f"expected [B, H, S, {self.head_dim}] states, got {tuple(states.shape)}")
        return compress_kv(states, None, key_compressor=self)[0]

    def asymmetric_attention_scores(self, queries: torch.Tensor, compressed: dict) -> torch.Tensor:
        """Unscaled, unmasked estimator scores fp32 [B, Hq, Sq, Sk] (compressors.py:163-224).
        Materialises the whole matrix; the adapters use `fused_attention` instead."""
        _require_cuda(queries, "queries")
        self._check_device(queries)
        B, Hq, Sq, D = queries.shape
        Bk, Hkv, Sk, Dk = compressed["shape"]
        if (Bk, Dk) != (B, D) or D != self.head_dim:
            raise ValueError(f"queries {tuple(queries.shape)} do not match compressed keys {compressed['shape']}")
        compressed = _dense_packed(compressed, _KEY_ARRAYS)
        return _lib.host.scores(queries, Hkv, Sk, *[compressed[n] for n in ("packed_key_indices", "packed_qjl_signs", "vec_norms",
                                                                            "residual_norm")],
                                self.Pi, self.S_eff, self.centroids, self.bits)


class TurboQuantCompressorMSE(_Constants):
    """Value compressor: `bits`-bit Lloyd-Max indices of the rotated unit vector
    (compressors.py:227-317)."""

    _tensor_attrs = ("Pi", "PiT", "centroids", "boundaries")

    def __init__(self, head_dim: int, bits: int, seed: int, device: str = "cuda", use_triton: bool = True,
                 mode: str | None = None):
        if head_dim not in (64, 128):
            raise ValueError(f"head_dim {head_dim} unsupported by the CUDA kernels (64 or 128)")
        if bits not in (2, 3, 4):
            raise ValueError(f"bits must be 2, 3 or 4, got {bits}")
        self.head_dim, self.bits = head_dim, bits
        self.use_triton = use_triton
        self.mode = mode
        self.Pi = _haar_rotation(head_dim, seed)
        self.PiT = self.Pi.T.contiguous()
        self.centroids = lloyd_max_centroids(head_dim, bits)
        self.boundaries = midpoints(self.centroids)
        self.to(device)

    def compress(self, states: torch.Tensor) -> dict:
        if states.dim() != 4 or states.shape[-1] != self.head_dim:
            raise ValueError(f"expected [B, H, S, {self.head_dim}] states, got {tuple(states.shape)}")
        return compress_kv(None, states, val_compressor=self)[1]

    def decompress(self, compressed: dict) -> torch.Tensor:
        """packed dict -> fp32 [B, H, S, D] (compressors.py:296-317)."""
        B, H, S, D = compressed["shape"]
        compressed = _dense_packed(compressed, _VALUE_ARRAYS)
        idx = compressed["packed_indices"]
        _require_cuda(idx, "compressed values")
        self._check_device(idx)
        return _lib.host.decompress(idx, compressed["vec_norms"], self.Pi, self.centroids, self.bits, B, H, S, D)


def _mask_rows(attention_mask: torch.Tensor, B: int, Sq: int, Sk: int, dev):
    """A mask broadcastable to [B, 1, Sq, Sk] as a [1 or B, Sq, Sk] tensor with unit inner stride and its kind.

    Floating-point masks are additive (0 = visible, large negative = hidden), as HF's eager path builds them.
    Boolean masks mean True = visible, which is what HF's sdpa path hands over for padded batches; the kernels
    read their bytes.  Integer masks are refused: their meaning would be a guess."""
    mk = attention_mask
    if mk.dim() == 4:
        if mk.shape[1] != 1:
            raise ValueError("per-head masks are not supported; expected [B, 1, Sq, Sk]")
        mk = mk[:, 0]
    elif mk.dim() == 2:
        mk = mk.unsqueeze(0)
    if mk.dtype == torch.bool:
        mk, kind = mk.to(device=dev), _lib.TQ_MASK_BOOL
    elif mk.dtype.is_floating_point:
        mk, kind = mk.to(device=dev, dtype=torch.float32), _lib.TQ_MASK_ADDITIVE
    else:
        raise TypeError(f"attention mask of dtype {mk.dtype} is ambiguous: pass a bool mask (True = visible) or an "
                        "additive floating-point mask")
    if mk.shape[-2:] != (Sq, Sk) or mk.shape[0] not in (1, B):
        raise ValueError(f"mask shape {tuple(attention_mask.shape)} does not broadcast to [B,1,{Sq},{Sk}]")
    if mk.stride(-1) != 1:
        mk = mk.contiguous()
    return mk, kind


def _attend(q: torch.Tensor, Hkv: int, Sk: int, capacity: int, packed: tuple, kc, vc, sm_scale, causal: bool,
            attention_mask, mode: int) -> torch.Tensor:
    """One attention call over `packed` = (key indices, signs, norms, residual norms, value indices, norms)."""
    B, _, Sq, D = q.shape
    mk, kind = (None, 0) if attention_mask is None else _mask_rows(attention_mask, B, Sq, Sk, q.device)
    return _lib.host.attend(q, Hkv, Sk, capacity, packed, prepared_constants(kc, vc), kc.bits,
                            float(sm_scale) if sm_scale is not None else 1.0 / math.sqrt(D), 1 if causal else 0, mode, mk, kind)


def fused_attention(q: torch.Tensor, compressed_k: dict, compressed_v: dict,
                    key_compressor: TurboQuantCompressorV2, val_compressor: TurboQuantCompressorMSE,
                    causal: bool = True, attention_mask: torch.Tensor | None = None,
                    sm_scale: float | None = None, mode: str | None = None) -> torch.Tensor:
    """softmax(scores * sm_scale + mask) @ V_hat from packed K and V: the attention core of
    the family adapters (families/llama.py:100-114 of the reference) as one fused pass.

    q [B, Hq, Sq, D]; the compressed tensors hold Hkv heads with Hq % Hkv == 0 (query head h
    reads KV head h // (Hq // Hkv), the `repeat_interleave` grouping).  `attention_mask` is an
    optional additive mask broadcastable to [B, 1, Sq, Sk].  Returns [B, Hq, Sq, D] in q.dtype (stored
    position-major, i.e. contiguous after `.transpose(1, 2)`).
    """
    _require_cuda(q, "q")
    key_compressor._check_device(q)
    val_compressor._check_device(q)
    B, Hq, Sq, D = q.shape
    Bk, Hkv, Sk, Dk = compressed_k["shape"]
    if compressed_v["shape"] != compressed_k["shape"] or (Bk, Dk) != (B, D):
        raise ValueError("q, compressed keys and compressed values disagree on shape")
    if key_compressor.bits != val_compressor.bits:
        raise ValueError("key and value compressors must use the same bit width")
    compressed_k, compressed_v = _dense_packed(compressed_k, _KEY_ARRAYS), _dense_packed(compressed_v, _VALUE_ARRAYS)
    packed = (*[compressed_k[n] for n in ("packed_key_indices", "packed_qjl_signs", "vec_norms", "residual_norm")],
              *[compressed_v[n] for n in ("packed_indices", "vec_norms")])
    return _attend(q, Hkv, Sk, Sk, packed, key_compressor, val_compressor, sm_scale, causal, attention_mask,
                   resolve_mode(q.dtype, mode or key_compressor.mode))


def device_fault_count(device=None) -> int:
    """Expired bounded device-side waits since the library was loaded (0 when healthy)."""
    import ctypes

    n = ctypes.c_int64(0)
    dev = torch.device(device if device is not None else "cuda")
    with torch.cuda.device(dev):  # the counter read is the one call that goes by the current device
        _lib.check(_lib.lib.tq_device_fault_count(_stream_ptr(dev), ctypes.byref(n)))
    return int(n.value)
