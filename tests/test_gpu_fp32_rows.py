"""fp32 attention of few query rows over a strided cache against a dense evaluation of the same bytes in fp64."""

import pytest
import torch

from helpers import contiguous_prefix, device_compressors, rel_err
from test_gpu_masks import _dense, _mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mask", [None, "left", "holes"])
@pytest.mark.parametrize("d,bits", [(128, 2), (128, 3), (128, 4), (64, 2), (64, 3), (64, 4)])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk", [(1, 1, 1, 1, 1), (2, 2, 2, 1, 33), (1, 4, 2, 1, 700), (2, 8, 2, 1, 1031), (1, 6, 2, 5, 64),
                                            (3, 4, 4, 16, 130), (1, 2, 1, 9, 300)])
def test_few_rows_in_fp32(B, Hq, Hkv, Sq, Sk, d, bits, mask):
    from turboquant_b200 import CompressedKVCache

    g = torch.Generator().manual_seed(Sk + 7 * Sq + bits)
    kc, vc = device_compressors(d, bits)
    k, v = (torch.randn(B, Hkv, Sk, d, generator=g).cuda() for _ in range(2))
    k[..., 3] *= 8
    q = torch.randn(B, Sq, Hq, d, generator=g).cuda().transpose(1, 2)
    cache = CompressedKVCache(kc, vc, B, Hkv, Sk + 13)
    cache.append(k, v)
    ck, cv = contiguous_prefix(cache)
    m = torch.ones(B, Sq, Sk, dtype=torch.bool) if mask is None else _mask(mask, B, Sq, Sk, g)
    m = m.cuda()
    want = _dense(q, ck, cv, kc, vc, m, True)
    # fp32 scores of size ~10 (2^-24 x sqrt(2 d) each) through an exponential of 2^-21, averaged: a few 1e-6
    assert rel_err(cache.attend(q, attention_mask=None if mask is None else m[:, None]), want) < 2e-5
    if mask is not None:
        add = torch.zeros(m.shape, device="cuda").masked_fill_(~m, torch.finfo(torch.float32).min)
        assert rel_err(cache.attend(q, attention_mask=add[:, None]), want) < 2e-5


@pytest.mark.parametrize("d,B,Hq,Hkv,Sq,Sk", [(128, 8, 32, 32, 8, 64), (128, 8, 32, 32, 12, 64), (128, 32, 32, 32, 16, 65), (64, 32, 12, 12, 16, 64),
                                              (64, 32, 12, 12, 8, 70)])
def test_many_rows_over_few_keys(d, B, Hq, Hkv, Sq, Sk):
    """Both sides of the line between the few-rows and the tile kernel where the heads fill the chip."""
    from turboquant_b200 import compress_kv, fused_attention

    g = torch.Generator().manual_seed(Sq + Sk)
    kc, vc = device_compressors(d, 3)
    k, v = (torch.randn(B, Hkv, Sk, d, generator=g).cuda() for _ in range(2))
    q = torch.randn(B, Hq, Sq, d, generator=g).cuda()
    ck, cv = compress_kv(k, v, kc, vc)
    m = torch.ones(B, Sq, Sk, dtype=torch.bool, device="cuda")
    assert rel_err(fused_attention(q, ck, cv, kc, vc), _dense(q, ck, cv, kc, vc, m, True)) < 2e-5  # as above
