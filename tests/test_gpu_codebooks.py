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


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d,bits", [(128, 3), (64, 4)])
@pytest.mark.parametrize("scale", [2.0 ** 11, 2.0 ** -12])
def test_rotations_of_any_size(d, bits, scale, dtype):
    """The fp16 operand images follow the size of the matrices: a rotation times a power of two with a codebook times the
    same power gives the same indices and signs, and the residual's norm times that power."""
    from turboquant_b200 import compress_kv

    g = torch.Generator().manual_seed(bits)
    k, v = (torch.randn(1, 2, 300, d, generator=g).cuda().to(dtype) for _ in range(2))
    plain, scaled = device_compressors(d, bits), device_compressors(d, bits)
    for c in scaled:
        c.Pi, c.centroids, c.boundaries = c.Pi * scale, c.centroids * scale, c.boundaries * scale
    (pk, pv), (sk, sv) = compress_kv(k, v, *plain), compress_kv(k, v, *scaled)
    for name in ("packed_key_indices", "packed_qjl_signs", "vec_norms"):
        assert torch.equal(pk[name], sk[name]), name
    assert torch.equal(pv["packed_indices"], sv["packed_indices"])
    assert torch.allclose(sk["residual_norm"].double(), pk["residual_norm"].double() * scale, rtol=2.0 ** -10, atol=2.0 ** -24)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("scale", [2.0 ** 10, 2.0 ** -10])
def test_rotation_and_codebook_of_different_size(d, scale):
    """... and a rotation that its codebook does not fit gives what the fp32 kernels give."""
    from turboquant_b200 import compress_kv

    k = torch.randn(1, 2, 300, d, generator=torch.Generator().manual_seed(d)).cuda().half()
    got = []
    for mode in (None, "fp32"):
        kc, _ = device_compressors(d, 3, mode=mode)
        kc.Pi = kc.Pi * scale
        got.append(compress_kv(k, None, kc, None)[0])
    for name in ("packed_key_indices", "packed_qjl_signs"):
        assert torch.equal(got[0][name], got[1][name]), name


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("scale", [2.0 ** 18, 2.0 ** -18])
def test_fp16_sketches_of_any_size(scale, dtype):
    """Only signs of the sketch are read, so its size does not matter: not of the matrix, not of a single row."""
    from turboquant_b200 import compress_kv

    for d in (64, 128):
        k = torch.randn(1, 2, 300, d, generator=torch.Generator().manual_seed(d)).cuda().to(dtype)
        kc, _ = device_compressors(d, 3)
        want = compress_kv(k, None, kc, None)[0]["packed_qjl_signs"]
        kc.S_eff = kc.S_eff * scale
        assert torch.equal(compress_kv(k, None, kc, None)[0]["packed_qjl_signs"], want)
        kc.S_eff = kc.S_eff * torch.cat([torch.ones(d // 2, 1), torch.full((d // 2, 1), 1.0 / scale)]).cuda()
        assert torch.equal(compress_kv(k, None, kc, None)[0]["packed_qjl_signs"], want)
