"""Attention over expanded keys and values under masks that hide whole key tiles from every query: in front of a chunk of
queries such tiles are neither expanded nor read.  Scratch is filled with fp16 NaN beforehand, so a tile that is read but was not written shows.

Reference: the fp32 kernels on the same packed bytes; tolerances of test_gpu_dense.py."""

import math

import pytest
import torch

from helpers import rel_err
from test_gpu_dense import TOLERANCE, _inputs

pytestmark = pytest.mark.gpu


def _call(q, ck, cv, kc, vc, mask):
    """Output of the C entry under a boolean mask [1 or B, Sq, Sk], and its scratch as int16."""
    from turboquant_b200 import _lib as L
    from turboquant_b200.compressors import prepared_constants

    (B, Hq, Sq, d), (_, Hkv, Sk, _) = q.shape, ck["shape"]
    need = L.lib.tq_attention_masked_workspace_bytes(B, Hq, Sq, Hkv, Sk, Sk, d, L.TQ_MODE_BF16, mask.shape[0])
    ws = torch.full((need // 2,), -1, dtype=torch.int16, device="cuda")
    out = torch.empty_like(q)
    mask = mask.contiguous()
    consts = prepared_constants(kc, vc)
    L.check(L.lib.tq_attention_fwd_masked(
        q.data_ptr(), L.TQ_BF16, B, Hq, Sq, d, *q.stride()[:3], Hkv, Sk, Sk, ck["packed_key_indices"].data_ptr(),
        ck["packed_qjl_signs"].data_ptr(), ck["vec_norms"].data_ptr(), ck["residual_norm"].data_ptr(), cv["packed_indices"].data_ptr(),
        cv["vec_norms"].data_ptr(), consts.data_ptr(), kc.bits, 1.0 / math.sqrt(d), 1, mask.data_ptr(), L.TQ_MASK_BOOL, mask.shape[0],
        Sq * Sk, Sk, out.data_ptr(), *out.stride()[:3], ws.data_ptr(), need, L.TQ_MODE_BF16, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return out, ws


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("kind", ["window", "left", "shared", "blind", "all"])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk", [(1, 32, 8, 300, 8300),    # split over the keys
                                            (4, 64, 16, 350, 2100),   # more tiles than CTAs
                                            (2, 32, 8, 40, 6001),     # three groups of rows, ragged
                                            (12, 64, 16, 257, 2050),  # two rounds of expansion at head_dim 128
                                            (32, 16, 16, 513, 513)])  # a prompt: all tiles are expanded
def test_hidden_tiles_are_not_touched(B, Hq, Hkv, Sq, Sk, d, kind):
    from turboquant_b200 import fused_attention

    q, ck, cv, kc, vc = _inputs(B, Hq, Hkv, Sq, Sk, d, 3, torch.bfloat16)
    at, row = torch.arange(Sk, device="cuda"), torch.arange(Sq, device="cuda")[:, None] + Sk - Sq
    if kind == "window":  # leading tiles hidden where the prefix is long
        mask = (at > row - 40).expand(1, Sq, Sk)
    elif kind == "left":  # a padding of its own for every sequence
        g = torch.Generator(device="cuda").manual_seed(3)
        pad = torch.randint(0, Sk - Sq + 1, (B, 1, 1), generator=g, device="cuda")
        pad[0] = Sk - Sq
        mask = (at >= pad).expand(B, Sq, Sk)
    elif kind == "shared":  # the first keys and the chunk itself
        mask = ((at < 5) | (at >= Sk - Sq)).expand(1, Sq, Sk)
    elif kind == "blind":  # one row of the last sequence sees nothing and averages its range
        mask = (at >= Sk - Sq).expand(B, Sq, Sk).clone()
        mask[B - 1, Sq // 2] = False
    else:
        mask = torch.ones(1, Sq, Sk, dtype=torch.bool, device="cuda")
    out, ws = _call(q, ck, cv, kc, vc, mask)
    ref = fused_attention(q.float(), ck, cv, kc, vc, mode="fp32", attention_mask=mask[:, None])
    worst = ((out.float() - ref).norm(dim=-1) / ref.norm(dim=-1)).max()
    assert rel_err(out, ref) < TOLERANCE[torch.bfloat16] and float(worst) < 4 * TOLERANCE[torch.bfloat16]

    T = (Sk + 127) // 128
    if B * Hkv * T * 512 * d > 128 << 20:
        return  # (several rounds share the scratch)
    tiles = torch.nn.functional.pad(mask.any(1), (0, 128 * T - Sk)).reshape(-1, T, 128).any(-1)  # some query sees a key
    tiles = tiles | ~(mask & (at <= row)).any(-1).all(-1)[:, None]                              # ... or averages all of them
    tiles = tiles | (Sk < 6 * Sq or B * Hkv * T * d < 300 * 128 or T < 16)  # (all are expanded)
    tiles = tiles.expand(B, T)[:, None].expand(B, Hkv, T).reshape(-1)
    written = (ws[:B * Hkv * T * 256 * d].reshape(B * Hkv * T, -1) != -1).all(-1)
    assert torch.equal(written, tiles)
