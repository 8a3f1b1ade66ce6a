"""Masks through their summary (visibility bits, skipped tiles) against a dense evaluation of the same bytes."""

import pytest
import torch

from helpers import device_compressors, rel_err, scores64, values64

pytestmark = pytest.mark.gpu


def _dense(q, ck, cv, kc, vc, mask, causal):
    """softmax(scores / sqrt(d) + mask) @ decoded values in fp64, from the packed bytes alone; rows whose causal range is all
    hidden average it."""
    B, Hq, Sq, d = q.shape
    _, Hkv, Sk, _ = ck["shape"]
    s = scores64(q, ck, kc) / d ** 0.5
    add = torch.where(mask, 0.0, -1e30).double()[:, None] if mask.dtype == torch.bool else mask.double()[:, None]
    s = torch.maximum(s + add, torch.tensor(-60000.0 * 0.6931471805599453, dtype=torch.float64, device=q.device))
    if causal:
        i = torch.arange(Sq, device=q.device)[:, None] + (Sk - Sq)
        s = s.masked_fill(torch.arange(Sk, device=q.device) > i, float("-inf"))
    v = values64(cv["packed_indices"], cv["vec_norms"].reshape(-1), vc).reshape(B, Hkv, Sk, d).repeat_interleave(Hq // Hkv, dim=1)
    return torch.softmax(s, -1) @ v


def _mask(kind, B, Sq, Sk, g):
    """Padding on the left, on the right, or random holes; the last query rows of the holed one see nothing."""
    k = torch.arange(Sk)
    if kind == "holes":
        m = torch.rand(B, Sq, Sk, generator=g) < 0.6
        m[:, -1] = False
        return m
    n = torch.randint(1, Sk + 1, (B, 1, 1), generator=g)
    m = (k >= Sk - n) if kind == "left" else (k < n)
    return m.expand(B, Sq, Sk)


@pytest.mark.parametrize("kind", ["left", "right", "holes"])
@pytest.mark.parametrize("d,Hq,Hkv,Sq,Sk", [(128, 4, 2, 1, 1), (128, 4, 2, 1, 127), (128, 4, 2, 1, 1029), (128, 2, 2, 3, 640),
                                            (128, 8, 1, 2, 4099), (128, 4, 2, 129, 129), (128, 3, 3, 300, 301),
                                            (128, 2, 1, 40, 1500), (64, 2, 2, 1, 260), (64, 4, 2, 257, 385)])
def test_masks_against_a_dense_evaluation(d, Hq, Hkv, Sq, Sk, kind):
    from turboquant_b200 import compress_kv, fused_attention

    g = torch.Generator().manual_seed(Sk + Sq)
    B = 3
    kc, vc = device_compressors(d, 3)
    k, v = (torch.randn(B, Hkv, Sk, d, generator=g).cuda().bfloat16() for _ in range(2))
    q = torch.randn(B, Hq, Sq, d, generator=g).cuda().bfloat16()
    ck, cv = compress_kv(k, v, kc, vc)
    mask = _mask(kind, B, Sq, Sk, g).cuda()
    want = _dense(q, ck, cv, kc, vc, mask, True)
    out = fused_attention(q, ck, cv, kc, vc, attention_mask=mask[:, None])
    assert rel_err(out, want) < 1e-2  # 16-bit operands and output
    # additive masks in the two values HF uses, and rows at any alignment of a larger tensor
    add = torch.zeros(mask.shape, device="cuda").masked_fill_(~mask, torch.finfo(torch.bfloat16).min)
    assert torch.equal(fused_attention(q, ck, cv, kc, vc, attention_mask=add[:, None]), out)
    wide = torch.zeros(B, Sq, Sk + 5, dtype=torch.bool, device="cuda")
    wide[:, :, 3:3 + Sk] = mask
    assert torch.equal(fused_attention(q, ck, cv, kc, vc, attention_mask=wide[:, None, :, 3:3 + Sk]), out)
    # one mask for the whole batch, and other additive values (read from the mask itself)
    one = fused_attention(q, ck, cv, kc, vc, attention_mask=mask[:1])
    assert rel_err(one, _dense(q, ck, cv, kc, vc, mask[:1], True)) < 1e-2
    bias = torch.where(mask, torch.randn(mask.shape, generator=g).cuda(), torch.full((), -3e38, device="cuda"))
    biased = fused_attention(q, ck, cv, kc, vc, attention_mask=bias[:, None])
    assert rel_err(biased, _dense(q, ck, cv, kc, vc, bias, True)) < 1e-2
    # fp32 kernels read the same bits
    f32 = fused_attention(q.float(), ck, cv, kc, vc, attention_mask=mask[:, None], mode="fp32")
    assert rel_err(f32, want) < 1e-4


@pytest.mark.parametrize("d,Sq,Sk", [(128, 3, 127), (128, 40, 128), (64, 70, 129), (128, 40, 132), (64, 300, 512), (128, 130, 515)])
@pytest.mark.parametrize("pitch,first", [(0, 0), (4, 0), (4, 1), (3, 2)])  # elements added to a row, and before the first
def test_additive_values_at_any_alignment(d, Sq, Sk, pitch, first):
    """Masks of arbitrary values: with and without a summary (up to 128 keys they are read as they are), rows that can and
    rows that cannot be loaded four columns at a time."""
    from turboquant_b200 import compress_kv, fused_attention

    g = torch.Generator().manual_seed(Sk + pitch)
    kc, vc = device_compressors(d, 3)
    k, v = (torch.randn(2, 2, Sk, d, generator=g).cuda().bfloat16() for _ in range(2))
    q = torch.randn(2, 4, Sq, d, generator=g).cuda().bfloat16()
    ck, cv = compress_kv(k, v, kc, vc)
    row = Sk + pitch + (-Sk) % 4 * (pitch == 4)
    mask = torch.randn(2 * Sq * row + 8, generator=g).cuda()[first:first + 2 * Sq * row].view(2, Sq, row)[:, :, :Sk]
    want = _dense(q, ck, cv, kc, vc, mask, True)
    assert rel_err(fused_attention(q, ck, cv, kc, vc, attention_mask=mask[:, None]), want) < 1e-2  # 16-bit operands and output
    assert rel_err(fused_attention(q.float(), ck, cv, kc, vc, attention_mask=mask[:, None], mode="fp32"), want) < 1e-4
