"""fp32 attention whose keys are cut into chunks: against a dense evaluation in fp64, and against the unsplit kernel."""

import pytest
import torch

from helpers import device_compressors, rel_err
from test_gpu_masks import _dense, _mask

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mask", [None, "right", "holes"])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("d,bits", [(128, 3), (64, 2), (64, 4)])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk", [(1, 1, 1, 64, 64), (1, 2, 2, 65, 129), (2, 4, 2, 130, 700), (1, 12, 12, 300, 300),
                                            (2, 8, 8, 17, 1100), (1, 3, 1, 256, 256)])
def test_split_tiles_in_fp32(B, Hq, Hkv, Sq, Sk, d, bits, causal, mask):
    from turboquant_b200 import compress_kv, fused_attention

    g = torch.Generator().manual_seed(Sk + 3 * Sq + bits)
    kc, vc = device_compressors(d, bits)
    k, v = (torch.randn(B, Hkv, Sk, d, generator=g).cuda() for _ in range(2))
    q = torch.randn(B, Hq, Sq, d, generator=g).cuda()
    ck, cv = compress_kv(k, v, kc, vc)
    m = torch.ones(B, Sq, Sk, dtype=torch.bool) if mask is None else _mask(mask, B, Sq, Sk, g)
    m = m.cuda()
    got = fused_attention(q, ck, cv, kc, vc, causal=causal, attention_mask=None if mask is None else m[:, None])
    # as for few rows: fp32 scores of size ~10 through an exponential of 2^-21, averaged
    assert rel_err(got, _dense(q, ck, cv, kc, vc, m, causal)) < 2e-5
