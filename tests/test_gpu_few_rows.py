"""Query preparation and estimator scores of few query rows against a dense evaluation in fp64."""

import numpy as np
import pytest
import torch

from helpers import device_compressors, scores64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d,bits", [(128, 2), (128, 3), (128, 4), (64, 2), (64, 3), (64, 4)])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk", [(1, 1, 1, 1, 1), (1, 2, 2, 1, 65), (2, 6, 2, 3, 63), (1, 4, 2, 4, 300), (1, 2, 1, 5, 128),
                                            (3, 32, 8, 40, 70)])
def test_scores_of_few_rows(B, Hq, Hkv, Sq, Sk, d, bits, dtype):
    g = torch.Generator().manual_seed(Sk * Sq + bits)
    kc, vc = device_compressors(d, bits)
    ck = kc.compress(torch.randn(B, Hkv, Sk, d, generator=g).cuda())
    q = torch.randn(B, Sq, Hq, d, generator=g).cuda().to(dtype).transpose(1, 2)
    got = kc.asymmetric_attention_scores(q, ck)
    want = scores64(q, ck, kc)
    # A single score may cancel, so its error is held against the size of the terms it sums, |q| |k|: fp32 sums of
    # d + d + 2 d products, a few times 2^-24 sqrt(4 d).
    size = q.double().norm(dim=-1)[..., None] * ck["vec_norms"].double().repeat_interleave(Hq // Hkv, dim=1)[:, :, None]
    assert float(((got - want).abs() / size).max()) < 4 * 2.0 ** -24 * (4 * d) ** 0.5


@pytest.mark.parametrize("d", [64, 128])
def test_query_rows_are_summed_in_a_fixed_order(d):
    """The order of a sum decides which way the 16-bit copy of a query coordinate is rounded, so it is part of the kernel's
    contract: groups of four columns from the last to the first, then halves folded onto each other."""
    from turboquant_b200 import _lib as L

    wide = np.longdouble  # holds the product of two floats exactly

    def fma(a, b, c):
        return (a.astype(wide) * b.astype(wide) + c.astype(wide)).astype(np.float32)

    def project(x, w):
        x, w = x.reshape(-1, 1, d // 4, 4), w.reshape(1, d, d // 4, 4)
        g = (x[..., 3].astype(wide) * w[..., 3].astype(wide)).astype(np.float32)
        for c in (2, 1, 0):
            g = fma(x[..., c], w[..., c], g)
        while g.shape[-1] > 1:
            h = g.shape[-1] // 2
            g = g[..., :h] + g[..., h:]
        return g[..., 0]

    kc, _ = device_compressors(d, 3)
    q = torch.randn(1, 3, 2, d, generator=torch.Generator().manual_seed(d)).cuda()
    got = torch.empty(6, 2 * d, device="cuda")
    L.check(L.lib.tq_prepare_queries(q.data_ptr(), L.TQ_F32, 1, 3, 2, d, q.stride(0), q.stride(1), q.stride(2), kc.Pi.data_ptr(),
                                     kc.S_eff.data_ptr(), got.data_ptr(), None, 0, L.TQ_MODE_FP32,
                                     torch.cuda.current_stream().cuda_stream))
    rot = project(q.reshape(-1, d).cpu().numpy(), kc.Pi.cpu().numpy())
    coeff = np.sqrt(np.float32(np.pi / 2)) / np.float32(d)
    want = np.concatenate([rot, coeff * project(rot, kc.S_eff.cpu().numpy())], axis=1)
    assert np.array_equal(got.cpu().numpy(), want)
