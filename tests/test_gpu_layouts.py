"""Compression of views: the orders and strides that the fused kernel's tiles of several heads and batch elements meet, against
the same numbers in dense rows."""

import pytest
import torch

from helpers import device_compressors

pytestmark = pytest.mark.gpu


def _views(kind, B, H, S, d, g, dtype):
    n = lambda *shape: torch.randn(*shape, generator=g).cuda().to(dtype)
    if kind == "one head for all":        # stride 0, as keys expanded for a kernel without grouped heads
        return [n(B, 1, S, d).expand(B, H, S, d) for _ in range(2)]
    if kind == "one sequence for all":
        return [n(1, H, S, d).expand(B, H, S, d) for _ in range(2)]
    if kind == "positions first":
        return [n(S, B, H, d).permute(1, 2, 0, 3) for _ in range(2)]
    if kind == "heads first":
        return [n(H, S, B, d).permute(2, 0, 1, 3) for _ in range(2)]
    if kind == "wide rows":               # a slice of rows that hold more than one head
        return [n(B, H, S, d + 40)[..., 24:24 + d] for _ in range(2)]
    return list(n(B, S, H, 2, d).permute(3, 0, 2, 1, 4))  # "interleaved": keys and values side by side


@pytest.mark.parametrize("kind", ["one head for all", "one sequence for all", "positions first", "heads first", "wide rows", "interleaved"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("B,H,S", [(3, 5, 1), (2, 3, 37), (2, 2, 131), (3, 8, 150)])
def test_views_give_the_bytes_of_dense_rows(B, H, S, d, dtype, kind):
    from turboquant_b200 import compress_kv

    k, v = _views(kind, B, H, S, d, torch.Generator().manual_seed(S + d), dtype)
    kc, vc = device_compressors(d, 3)
    got, want = compress_kv(k, v, kc, vc), compress_kv(k.contiguous(), v.contiguous(), kc, vc)
    for a, b in zip(got, want):
        for name, t in a.items():
            assert name == "shape" or torch.equal(t, b[name]), name
