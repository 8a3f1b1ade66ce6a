"""Helpers shared by the GPU parity tests: oracle parameters, their twins on the device,
and thin wrappers that call the C ABI through ctypes with torch tensors as buffers."""

from __future__ import annotations

import numpy as np
import torch

from oracle import tq_oracle as orc

_PARAM_CACHE: dict = {}


def oracle_params(d: int, bits: int, key_seed: int = 42, val_seed: int = 10042):
    key = (d, bits, key_seed, val_seed)
    if key not in _PARAM_CACHE:
        _PARAM_CACHE[key] = (orc.make_key_params(d, bits, key_seed), orc.make_value_params(d, bits, val_seed))
    return _PARAM_CACHE[key]


def device_compressors(d: int, bits: int, key_seed: int = 42, val_seed: int = 10042, mode=None):
    """Product compressors whose constants are overwritten with the oracle's, so that both
    sides work from identical matrices and codebooks."""
    from turboquant_b200 import TurboQuantCompressorMSE, TurboQuantCompressorV2

    kp, vp = oracle_params(d, bits, key_seed, val_seed)
    kc = TurboQuantCompressorV2(d, bits, key_seed, device="cuda", mode=mode)
    vc = TurboQuantCompressorMSE(d, bits, val_seed, device="cuda", mode=mode)
    # .contiguous(): the Q factor of torch.linalg.qr comes back column-major
    kc.Pi, kc.S, kc.S_eff = kp.Pi.contiguous().cuda(), kp.S.contiguous().cuda(), kp.S_eff.contiguous().cuda()
    kc.PiT = kc.Pi.T.contiguous()
    kc.centroids, kc.boundaries = kp.centroids.contiguous().cuda(), kp.boundaries.contiguous().cuda()
    vc.Pi, vc.PiT = vp.Pi.contiguous().cuda(), vp.Pi.T.contiguous().cuda()
    vc.centroids, vc.boundaries = vp.centroids.contiguous().cuda(), vp.boundaries.contiguous().cuda()
    return kc, vc


def oracle_key_dict_to_device(ck: dict) -> dict:
    """The oracle's packed bytes and fp16 norms as the dict the product consumes."""
    B, H, S, D = ck["shape"]
    return {"packed_key_indices": torch.from_numpy(ck["packed_key_indices"]).cuda(),
            "packed_qjl_signs": torch.from_numpy(ck["packed_qjl_signs"]).cuda(),
            "residual_norm": ck["residual_norm"].cuda().contiguous(),
            "vec_norms": ck["vec_norms"].cuda().contiguous(), "shape": (B, H, S, D)}


def oracle_value_dict_to_device(cv: dict) -> dict:
    return {"packed_indices": torch.from_numpy(cv["packed_indices"]).cuda(),
            "vec_norms": cv["vec_norms"].cuda().contiguous(), "shape": cv["shape"]}


def unpack_fields(packed: torch.Tensor, bits: int, d: int) -> torch.Tensor:
    """Packed rows [..., d * bits / 8] as whole numbers [..., d] (fields LSB first), without the package's kernels."""
    rows = packed.reshape(-1, d * bits // 8)
    stream = (rows[:, :, None] >> torch.arange(8, dtype=torch.uint8, device=rows.device)) & 1
    weights = 1 << torch.arange(bits, device=rows.device)
    return (stream.reshape(-1, d, bits).long() * weights).sum(-1).reshape(*packed.shape[:-1], d)


def values64(packed: torch.Tensor, norms: torch.Tensor, vc) -> torch.Tensor:
    """Decoded values [..., d] in fp64 from packed rows and their norms."""
    dev = packed.device
    centroids, pi = vc.centroids.double().to(dev), vc.Pi.double().to(dev)
    return centroids[unpack_fields(packed, vc.bits, vc.head_dim)] @ pi * norms.double()[..., None]


def scores64(q: torch.Tensor, ck: dict, kc) -> torch.Tensor:
    """Unscaled estimator scores [B, Hq, Sq, Sk] in fp64 from packed keys."""
    B, Hkv, Sk, d = ck["shape"]
    rows = lambda t: t.reshape(B, Hkv, Sk, -1).repeat_interleave(q.shape[1] // Hkv, dim=1)
    cen = kc.centroids.double()[unpack_fields(rows(ck["packed_key_indices"]), kc.bits - 1, d)]
    sign = 2.0 * unpack_fields(rows(ck["packed_qjl_signs"]), 1, d).double() - 1.0
    rot = q.double() @ kc.Pi.double().T
    sketch = rot @ kc.S_eff.double().T * ((torch.pi / 2) ** 0.5 / d)
    return (rot @ cen.transpose(2, 3)) * rows(ck["vec_norms"].double())[..., 0][:, :, None] \
        + (sketch @ sign.transpose(2, 3)) * rows(ck["residual_norm"].double())[..., 0][:, :, None]


def contiguous_prefix(cache) -> tuple[dict, dict]:
    """The tokens in use of a CompressedKVCache as dense compressed dictionaries."""
    n, shape = cache.length, (cache.batch, cache.kv_heads, cache.length, cache.head_dim)
    packed = lambda t: t[:, :, :n].reshape(-1, t.shape[-1]).contiguous()
    ck = {"packed_key_indices": packed(cache.key_indices), "packed_qjl_signs": packed(cache.key_signs),
          "residual_norm": cache.key_residual_norms[:, :, :n].contiguous(), "vec_norms": cache.key_norms[:, :, :n].contiguous(),
          "shape": shape}
    return ck, {"packed_indices": packed(cache.value_indices), "vec_norms": cache.value_norms[:, :, :n].reshape(-1).contiguous(),
                "shape": shape}


def rel_err(a: torch.Tensor, b: torch.Tensor) -> float:
    """Norm-wise relative error ||a-b|| / ||b||."""
    a, b = a.double().cpu(), b.double().cpu()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


def oracle_attention_from_packed(q, ck, cv, kp, vp, causal=True, mask=None):
    """fp32 attention output computed on the CPU from the oracle's packed bytes:
    softmax(scores/sqrt(d) + mask) @ V_hat, with GQA grouping of heads."""
    B, Hq, Sq, D = q.shape
    Hkv, Sk = ck["shape"][1], ck["shape"][2]
    g = Hq // Hkv
    out = torch.empty(B, Hq, Sq, D)
    vals = orc.values_from_packed(cv["packed_indices"], cv["vec_norms"], vp, cv["shape"])
    idx = ck["packed_key_indices"].reshape(B, Hkv, Sk, -1)
    sgn = ck["packed_qjl_signs"].reshape(B, Hkv, Sk, -1)
    for h in range(Hq):
        j = h // g
        sc = orc.scores_from_packed(q[:, h:h + 1].float(), idx[:, j:j + 1], sgn[:, j:j + 1],
                                    ck["vec_norms"][:, j:j + 1], ck["residual_norm"][:, j:j + 1],
                                    kp, (B, 1, Sk, D))
        sc = sc / D ** 0.5
        if causal:
            sc = sc + orc.causal_mask(Sq, Sk)
        if mask is not None:
            sc = sc + mask
        out[:, h:h + 1] = torch.softmax(sc, dim=-1) @ vals[:, j:j + 1]
    return out
