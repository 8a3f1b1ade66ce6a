"""Value decompression against an evaluation in fp64 made on the host from the packed bytes alone."""

import numpy as np
import pytest
import torch

from helpers import device_compressors, values64

pytestmark = pytest.mark.gpu


def _packed(n, d, bits, seed):
    g = torch.Generator().manual_seed(seed)
    idx = torch.randint(0, 256, (n, d * bits // 8), dtype=torch.uint8, generator=g)
    norms = (torch.randn(n, generator=g).abs() * 12).half()
    return idx, norms


def _decompress(vc, idx, norms, d):
    return vc.decompress({"packed_indices": idx.cuda(), "vec_norms": norms.cuda(), "shape": (1, 1, idx.shape[0], d)})[0, 0]


# A coordinate is a sum of d products; fp32 sums of random sign lose about 2^-24 sqrt(d) / 2 of the size of their terms.  The
# bound is twice that for the mean, and 6 standard deviations of it for the largest.
@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000, 40001])  # 40001: every CTA of a 148-SM device walks on to further tiles
@pytest.mark.parametrize("d,bits", [(128, 2), (128, 3), (128, 4), (64, 2), (64, 3), (64, 4)])
def test_decompress_to_fp32_accuracy(n, d, bits):
    _, vc = device_compressors(d, bits)
    idx, norms = _packed(n, d, bits, n + d + bits)
    want = values64(idx, norms, vc)
    err = (_decompress(vc, idx, norms, d).double().cpu() - want).abs()
    size = want.norm(dim=-1, keepdim=True).clamp_min(1e-30) / d ** 0.5  # of a typical coordinate of the vector
    assert float((err ** 2).mean().sqrt() / (size ** 2).mean().sqrt()) < 2.0 ** -24 * d ** 0.5
    assert float((err / size).max()) < 6 * 2.0 ** -24 * d ** 0.5


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_packed_rows_may_start_anywhere(offset):
    from turboquant_b200 import _lib as L

    _, vc = device_compressors(128, 3)
    idx, norms = _packed(300, 128, 3, offset)
    buf = torch.zeros(idx.numel() + 8, dtype=torch.uint8, device="cuda")
    buf[offset:offset + idx.numel()] = idx.cuda().reshape(-1)
    out = torch.empty(300, 128, device="cuda")
    vn = norms.cuda()
    L.check(L.lib.tq_decompress_values(buf.data_ptr() + offset, vn.data_ptr(), 300, 128, vc.Pi.data_ptr(), vc.centroids.data_ptr(), 3,
                                       out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    assert torch.equal(out, _decompress(vc, idx, norms, 128))


@pytest.mark.parametrize("d,bits", [(128, 2), (128, 4), (64, 3)])
@pytest.mark.parametrize("pi_scale,cen_scale", [(2.0 ** 12, 1.0), (2.0 ** -30, 1.0), (1.0, 2.0 ** 11), (1.0, 2.0 ** -20), (2.0 ** 60, 2.0 ** -60),
                                                (2.0 ** -9, 2.0 ** 9)])
def test_constants_of_any_size(d, bits, pi_scale, cen_scale):
    """The entry point takes any fp32 matrix and codebook: powers of two move the result by exactly that factor."""
    _, vc = device_compressors(d, bits)
    idx, norms = _packed(200, d, bits, bits)
    vc.Pi, vc.centroids = vc.Pi * pi_scale, vc.centroids * cen_scale
    want = values64(idx, norms, vc)
    err = (_decompress(vc, idx, norms, d).double().cpu() - want).abs()
    size = want.norm(dim=-1, keepdim=True).clamp_min(1e-300) / d ** 0.5
    assert float((err / size).max()) < 6 * 2.0 ** -24 * d ** 0.5


def test_columns_of_different_size():
    _, vc = device_compressors(128, 3)
    idx, norms = _packed(200, 128, 3, 0)
    vc.Pi = vc.Pi * torch.logspace(-9, 2, 128, device="cuda")
    want = values64(idx, norms, vc)
    err = (_decompress(vc, idx, norms, 128).double().cpu() - want).abs()
    # per column: the size of its terms is |centroid| |column|
    size = norms.double()[:, None] * vc.Pi.double().cpu().norm(dim=0) * float(vc.centroids.double().pow(2).mean().sqrt())
    assert float((err / size.clamp_min(1e-300)).max()) < 8 * 2.0 ** -24 * 128 ** 0.5
