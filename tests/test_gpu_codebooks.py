"""Codebooks that a caller replaced: boundaries without the symmetry of the Lloyd-Max ones."""

import pytest
import torch

from helpers import device_compressors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shift", ["both", "one"])  # all boundaries moved, or only the lowest
@pytest.mark.parametrize("d,bits", [(128, 2), (128, 3), (128, 4), (64, 2), (64, 3), (64, 4)])
def test_boundaries_are_counted_as_given(d, bits, shift, dtype):
    from turboquant_b200 import compress_kv

    def shifted(c):
        step = 0.3 * float(c.boundaries.abs().max().clamp_min(0.05))
        bnd = c.boundaries + step
        if shift == "one":
            bnd = c.boundaries.clone()
            bnd[0] -= step
        c.boundaries = bnd

    g = torch.Generator().manual_seed(bits + d)
    k, v = (torch.randn(2, 3, 400, d, generator=g).cuda().to(dtype) for _ in range(2))
    pairs = [device_compressors(d, bits, mode=mode) for mode in (None, "fp32")]
    for kc, vc in pairs:
        shifted(kc)
        shifted(vc)
    ck, cv = compress_kv(k, v, *pairs[0])
    fk, fv = pairs[1][0].compress(k), pairs[1][1].compress(v)
    for a, b, differ in ((ck["packed_key_indices"], fk["packed_key_indices"], 3e-4), (cv["packed_indices"], fv["packed_indices"], 3e-4),
                         (ck["packed_qjl_signs"], fk["packed_qjl_signs"], 2e-3)):
        if dtype == torch.float16:  # open coordinates are decided as the fp32 kernels decide them
            assert torch.equal(a, b)
        else:  # coordinates within rounding of a boundary may move (about 2e-5 of the index bytes, 3e-4 of the sign bytes)
            assert float((a != b).float().mean()) <= differ
