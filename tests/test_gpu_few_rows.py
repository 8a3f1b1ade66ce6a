"""Query preparation and estimator scores of few query rows against a dense evaluation in fp64."""

import pytest
import torch

from helpers import device_compressors

pytestmark = pytest.mark.gpu


def _unpack(packed, b, d):
    from turboquant_b200.kernels import unpack_bits
    return unpack_bits(packed, b, d).long()


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
    rows = lambda t: t.double().reshape(B, Hkv, Sk, -1).repeat_interleave(Hq // Hkv, dim=1)
    cen = rows(kc.centroids[_unpack(ck["packed_key_indices"], bits - 1, d)])
    sign = rows(2.0 * _unpack(ck["packed_qjl_signs"], 1, d) - 1.0)
    rot = q.double() @ kc.Pi.double().T
    sketch = rot @ kc.S_eff.double().T * ((torch.pi / 2) ** 0.5 / d)
    want = (rot @ cen.transpose(2, 3)) * rows(ck["vec_norms"])[..., 0][:, :, None] \
        + (sketch @ sign.transpose(2, 3)) * rows(ck["residual_norm"])[..., 0][:, :, None]
    # A single score may cancel, so its error is held against the size of the terms it sums, |q| |k|: fp32 sums of
    # d + d + 2 d products, a few times 2^-24 sqrt(4 d).
    size = q.double().norm(dim=-1)[..., None] * rows(ck["vec_norms"])[..., 0][:, :, None]
    assert float(((got - want).abs() / size).max()) < 4 * 2.0 ** -24 * (4 * d) ** 0.5
