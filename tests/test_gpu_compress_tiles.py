"""Tiles of the fused compression kernel that hold short sequences of several heads and batch elements, both 16-bit input
types and both head dimensions, against the fp32 kernels on the same data."""

import pytest
import torch

from helpers import device_compressors

pytestmark = pytest.mark.gpu


def _bits_differ(a, b):
    x = (a ^ b).to(torch.int32)
    return float(sum(((x >> i) & 1).sum() for i in range(8))) / (8 * a.numel())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d,bits", [(128, 2), (128, 4), (64, 2), (64, 3), (64, 4)])
@pytest.mark.parametrize("B,H,S", [(1, 1, 1), (3, 5, 1), (16, 32, 1), (2, 200, 1), (5, 3, 7), (3, 7, 30), (2, 3, 64), (2, 3, 65),
                                   (1, 2, 128), (2, 2, 129), (1, 3, 700)])
def test_short_sequences_share_tiles(B, H, S, d, bits, dtype):
    from turboquant_b200 import CompressedKVCache, compress_kv

    g = torch.Generator().manual_seed(B * H + S + d)
    # rows as a fused projection leaves them: heads side by side, keys and values interleaved
    x = torch.randn(B, S, 2, H, d, generator=g)
    x[0, 0, :, 0] = 0.0
    k, v = (t.transpose(1, 2) for t in x.cuda().to(dtype).unbind(2))
    kc, vc = device_compressors(d, bits)
    ck, cv = compress_kv(k, v, kc, vc)
    kf, vf = device_compressors(d, bits, mode="fp32")
    fk, fv = kf.compress(k), vf.compress(v)
    # bf16: operands of 16 mantissa bits, coordinates within rounding of a boundary may move; an index
    # that moved moves its residual, and with it a few signs of that row
    n = k.numel()
    tight = dtype == torch.float16
    # (fp16 coordinates too close to call are decided by the fp32 arithmetic: the same bytes)
    if tight:
        for a, b in ((ck["packed_key_indices"], fk["packed_key_indices"]), (cv["packed_indices"], fv["packed_indices"]), (ck["packed_qjl_signs"], fk["packed_qjl_signs"])):
            assert torch.equal(a, b)
    assert _bits_differ(ck["packed_key_indices"], fk["packed_key_indices"]) <= 3e-5 + 4 / n
    assert _bits_differ(cv["packed_indices"], fv["packed_indices"]) <= 3e-5 + 4 / n
    assert _bits_differ(ck["packed_qjl_signs"], fk["packed_qjl_signs"]) <= 2e-4 + 40 / n
    for a, b in ((ck["vec_norms"], fk["vec_norms"]), (ck["residual_norm"], fk["residual_norm"]), (cv["vec_norms"], fv["vec_norms"])):
        assert int((a.view(torch.int16).int() - b.view(torch.int16).int()).abs().max()) <= 1
    # the same rows behind others in a cache, one token short of its end
    cache = CompressedKVCache(kc, vc, B, H, S + 4)
    cache.length = 3
    cache.append(k, v)
    for buf, ref in ((cache.key_indices, ck["packed_key_indices"]), (cache.key_signs, ck["packed_qjl_signs"]),
                     (cache.key_norms, ck["vec_norms"]), (cache.key_residual_norms, ck["residual_norm"]),
                     (cache.value_indices, cv["packed_indices"]), (cache.value_norms, cv["vec_norms"])):
        assert torch.equal(buf[:, :, 3:3 + S].reshape(-1), ref.reshape(-1))
        assert not buf[:, :, :3].any() and not buf[:, :, 3 + S:].any()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d,bits", [(128, 2), (128, 3), (128, 4), (64, 2), (64, 3), (64, 4)])
@pytest.mark.parametrize("B,H,S", [(1, 1, 1), (1, 3, 1), (4, 7, 1), (2, 3, 99), (2, 12, 28), (3, 32, 32)])
def test_few_vectors_give_the_tile_kernels_bytes(B, H, S, d, bits, dtype):
    """fp32 mode: up to 3072 vectors go to the few-vectors kernel, the same vectors among more of them to the tile kernel."""
    from turboquant_b200 import compress_kv

    g = torch.Generator().manual_seed(B * H + S + bits)
    k, v = (torch.randn(B, S, H, d, generator=g).cuda().to(dtype).transpose(1, 2) for _ in range(2))
    k[0, 0, 0] = 0.0
    k[..., 5] *= 8
    more = torch.randn(3073 // (H * S) + 1, H, S, d, generator=g).cuda().to(dtype)
    kc, vc = device_compressors(d, bits, mode="fp32")
    few, many = compress_kv(k, v, kc, vc), compress_kv(torch.cat([k, more]), torch.cat([v, more]), kc, vc)
    n = B * H * S
    for a, b in zip(few, many):
        for name, t in a.items():
            if name != "shape":
                assert torch.equal(t.reshape(n, -1), b[name].reshape(-1, t.numel() // n)[:n]), name
