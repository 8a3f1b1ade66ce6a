"""Chunks of queries behind long prefixes: the SM-pair kernel split over the keys, against a dense evaluation in fp64."""

import pytest
import torch

from helpers import device_compressors, rel_err
from test_gpu_masks import _dense, _mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mask", [None, "left", "holes", "bias"])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("d,bits,B,Hq,Hkv,Sq,Sk", [(128, 3, 1, 4, 2, 17, 6500), (128, 2, 2, 3, 3, 200, 5177), (128, 4, 1, 8, 2, 129, 4099),
                                                   (64, 3, 1, 2, 2, 1, 5100), (64, 2, 2, 4, 2, 300, 6500), (128, 3, 1, 2, 1, 128, 9152)])
def test_split_chunks(d, bits, B, Hq, Hkv, Sq, Sk, causal, mask):
    from turboquant_b200 import compress_kv, fused_attention

    g = torch.Generator().manual_seed(Sk + Sq + bits)
    kc, vc = device_compressors(d, bits)
    k, v = (torch.randn(B, Hkv, Sk, d, generator=g).cuda().bfloat16() for _ in range(2))
    q = torch.randn(B, Sq, Hq, d, generator=g).cuda().bfloat16().transpose(1, 2)
    ck, cv = compress_kv(k, v, kc, vc)
    if mask == "bias":
        m = torch.randn(B, Sq, Sk, generator=g).cuda()
    else:
        m = (torch.ones(B, Sq, Sk, dtype=torch.bool) if mask is None else _mask(mask, B, Sq, Sk, g)).cuda()
    got = fused_attention(q, ck, cv, kc, vc, causal=causal, attention_mask=None if mask is None else m[:, None])
    assert rel_err(got, _dense(q, ck, cv, kc, vc, m, causal)) < 1e-2  # 16-bit operands and output
