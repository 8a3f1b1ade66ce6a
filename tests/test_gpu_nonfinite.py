"""Queries and keys that are not finite: the rows they reach come out not finite, the others do not notice, whether a call
merges partial results or not."""

import pytest
import torch

from helpers import device_compressors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("mode,Hq,Hkv,Sq,Sk", [("bf16", 4, 2, 129, 129),    # SM-pair kernel, one cluster per tile
                                               ("bf16", 4, 2, 40, 6500),    # ... split over the keys
                                               ("bf16", 3, 3, 300, 5300),
                                               ("bf16", 4, 2, 2, 1029),     # split-KV kernel (head_dim 128)
                                               ("fp32", 4, 2, 40, 100),     # tile kernel, all keys in one chunk
                                               ("fp32", 4, 2, 40, 1500),    # ... in several
                                               ("fp32", 4, 2, 2, 1029)])    # few rows, split
@pytest.mark.parametrize("bad_key", [False, True])
def test_rows_that_meet_nan_or_inf(d, mode, Hq, Hkv, Sq, Sk, bad_key):
    from turboquant_b200 import compress_kv, fused_attention

    g = torch.Generator().manual_seed(Sq + Sk)
    B, dtype = 2, torch.float32 if mode == "fp32" else torch.bfloat16
    kc, vc = device_compressors(d, 3)
    k, v = (torch.randn(B, Hkv, Sk, d, generator=g).cuda().to(dtype) for _ in range(2))
    q = torch.randn(B, Sq, Hq, d, generator=g).cuda().to(dtype).transpose(1, 2)
    bad = torch.zeros(B, Hq, Sq, dtype=torch.bool)
    if bad_key:
        at = Sk - Sq + Sq // 2  # seen by the later half of the queries of the last group's heads
        k[1, Hkv - 1, at, 5] = float("nan")
        bad[1, (Hkv - 1) * (Hq // Hkv):, Sq // 2:] = True
    else:
        q[0, 1, Sq - 1, 3] = float("nan")
        q[1, 0, 0] = float("inf")
        bad[0, 1, Sq - 1] = bad[1, 0, 0] = True
    ck, cv = compress_kv(k, v, kc, vc)
    out = fused_attention(q, ck, cv, kc, vc)
    assert torch.equal(~out.isfinite().all(-1).cpu(), bad)
    assert torch.equal(~out.isfinite().any(-1).cpu(), bad)
