"""Attention over keys and values expanded to fp16 rows: edges of its tiles, splits, masks and groups of KV heads.

Reference: the fp32 kernels on the same packed bytes.  Queries (exactly, but for values 2^-28 below their row's largest),
expanded keys, probabilities and expanded values are rounded to fp16, each by at most 2^-11 of a value and independently:
about sqrt(3) 2^-11 / sqrt(3) = 5e-4 of the output in the mean, twice that beside a score of ten (a relative error of a key
moves the exponent by as much of the score).  The output's own rounding is at most 2^-9 (bf16) or 2^-12 (fp16) of a value."""

import pytest
import torch

from helpers import device_compressors, rel_err

pytestmark = pytest.mark.gpu

TOLERANCE = {torch.bfloat16: 2.0**-9 + 2e-3, torch.float16: 2e-3}


def _inputs(B, Hq, Hkv, Sq, Sk, d, bits, dtype):
    from turboquant_b200 import _lib as L, compress_kv

    need = L.lib.tq_attention_prepared_workspace_bytes(B, Hq, Sq, Hkv, Sk, Sk, d, L.TQ_MODE_BF16)
    tile = 2 * 128 * d * 2
    assert need >= min(B * Hkv * ((Sk + 127) // 128) * tile, 60 << 20)  # served by expansion
    g = torch.Generator(device="cuda").manual_seed(Sq + 3 * Sk + d)
    kc, vc = device_compressors(d, bits)
    gain = torch.ones(d, device="cuda")
    gain[1::d // 4] = 8.0
    k, v = (torch.randn(B, Hkv, Sk, d, generator=g, device="cuda") for _ in range(2))
    q = torch.randn(B, Sq, Hq, d, generator=g, device="cuda").to(dtype).transpose(1, 2)
    return q, *compress_kv((k * gain).to(dtype), v.to(dtype), kc, vc), kc, vc


def _check(q, ck, cv, kc, vc, **kw):
    from turboquant_b200 import fused_attention

    ref = fused_attention(q.float(), ck, cv, kc, vc, mode="fp32", **kw)
    out = fused_attention(q, ck, cv, kc, vc, **kw)
    assert rel_err(out, ref) < TOLERANCE[q.dtype]
    worst = ((out.float() - ref).norm(dim=-1) / ref.norm(dim=-1)).max()  # no row is off
    assert float(worst) < 4 * TOLERANCE[q.dtype]


# rows of a group around one tile (128), two (a CTA) and three; groups of 1, 3 and 7 heads; ragged ends of the keys
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk", [(32, 12, 12, 127, 127), (32, 16, 4, 32, 129), (16, 16, 16, 257, 257),
                                            (16, 12, 4, 85, 130), (16, 14, 2, 55, 1000), (8, 16, 4, 700, 900)])
@pytest.mark.parametrize("causal", [True, False])
def test_edges_of_tiles(B, Hq, Hkv, Sq, Sk, d, causal):
    _check(*_inputs(B, Hq, Hkv, Sq, Sk, d, 3, torch.bfloat16), causal=causal)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d,bits", [(128, 2), (128, 4), (64, 2), (64, 4)])
def test_bits_and_types(d, bits, dtype):
    _check(*_inputs(4, 16, 8, 600, 600, d, bits, dtype))


# few blocks of many key tiles: partial results merged, the last split of a block without keys of its first rows
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("Hq,Hkv,Sq,Sk", [(32, 8, 300, 8300), (16, 2, 5, 30001), (32, 8, 40, 20000)])
@pytest.mark.parametrize("causal", [True, False])
def test_splits_of_the_keys(Hq, Hkv, Sq, Sk, d, causal):
    _check(*_inputs(1, Hq, Hkv, Sq, Sk, d, 3, torch.bfloat16), causal=causal)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk", [(32, 12, 4, 200, 333), (1, 32, 8, 300, 8300)])  # unsplit, split
@pytest.mark.parametrize("kind", ["padding", "scattered", "additive"])
def test_masks(B, Hq, Hkv, Sq, Sk, d, kind):
    q, ck, cv, kc, vc = _inputs(B, Hq, Hkv, Sq, Sk, d, 3, torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(1)
    at = torch.arange(Sk, device="cuda")
    if kind == "padding":  # whole tiles hidden
        mask = (at >= torch.randint(0, Sk - Sq, (B, 1, 1), generator=g, device="cuda")).expand(B, Sq, Sk)[:, None]
    elif kind == "scattered":
        mask = torch.rand(B, 1, Sq, Sk, generator=g, device="cuda") > 0.4
        mask[..., 0] = True
        mask[:, :, 3] = False  # a row that sees nothing averages its causal range
    else:
        mask = torch.randn(B, 1, Sq, Sk, generator=g, device="cuda")
        mask[mask > 1.5] = float("-inf")
        mask[..., 0] = 0.0
    _check(q, ck, cv, kc, vc, attention_mask=mask)


def test_more_kv_heads_than_are_expanded_at_a_time():
    # 528 KV heads x 256 KB of expanded rows (128 MB at a time), in two rounds
    _check(*_inputs(44, 12, 12, 1024, 1024, 64, 3, torch.bfloat16))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_queries_of_any_size(dtype):
    q, ck, cv, kc, vc = _inputs(16, 16, 8, 300, 300, 128, 3, dtype)
    scale = torch.logspace(-3, 2, 300, device="cuda")[None, None, :, None]  # one row in 1e-3, one in 100 standard deviations
    from turboquant_b200 import fused_attention

    q = (q.float() * scale).to(dtype)
    ref = fused_attention(q.float(), ck, cv, kc, vc, mode="fp32")
    out = fused_attention(q, ck, cv, kc, vc)
    assert bool(out.isfinite().all())
    small = scale.flatten() < 1.0  # (larger scores: a softmax of one key, which a rounding may choose)
    assert rel_err(out[:, :, small], ref[:, :, small]) < TOLERANCE[dtype]
    zero = torch.zeros_like(q)  # equal scores: the mean of the visible values
    assert rel_err(fused_attention(zero, ck, cv, kc, vc), fused_attention(zero.float(), ck, cv, kc, vc, mode="fp32")) < TOLERANCE[dtype]
