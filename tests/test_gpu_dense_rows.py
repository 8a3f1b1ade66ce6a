"""Attention over expanded keys and values: query rows of any size under masks.

Reference: the fp32 kernels on the same packed bytes; tolerances as in test_gpu_dense.py, whose fp16 roundings are the same
ones.  Rows too small for any score to differ from 0 in fp32 are averages of the visible values, weighted by the mask."""

import pytest
import torch

from helpers import rel_err
from test_gpu_dense import TOLERANCE, _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sm_scale", [None, 1e-20])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk", [(32, 12, 4, 200, 333), (1, 32, 8, 300, 8300)])  # unsplit, split
@pytest.mark.parametrize("kind", ["boolean", "additive"])
def test_small_rows_under_masks(B, Hq, Hkv, Sq, Sk, kind, dtype, sm_scale):
    from turboquant_b200 import fused_attention

    q, ck, cv, kc, vc = _inputs(B, Hq, Hkv, Sq, Sk, 128, 3, dtype)
    # neighbours of a tile of rows, and the rows of a warp, differ by factors of 2^60
    scale = torch.tensor([1.0, 1e-18, 1e-25, 1e-30, 1e-33, 1e-35, 1e-37], device="cuda")[torch.arange(Sq, device="cuda") % 7]
    q = (q.float() * scale[None, None, :, None]).to(dtype)
    g = torch.Generator(device="cuda").manual_seed(2)
    if kind == "boolean":
        mask = torch.rand(B, 1, Sq, Sk, generator=g, device="cuda") > 0.4
        mask[..., 0] = True
        mask[:, :, 21:28] = False  # rows that see nothing average their causal range, one of each size
    else:
        mask = torch.randn(B, 1, Sq, Sk, generator=g, device="cuda")
        mask[mask > 1.5] = float("-inf")
        mask[..., 0] = 0.0
    ref = fused_attention(q.float(), ck, cv, kc, vc, mode="fp32", attention_mask=mask, sm_scale=sm_scale)
    out = fused_attention(q, ck, cv, kc, vc, mode="bf16", attention_mask=mask, sm_scale=sm_scale)
    tolerance = TOLERANCE.get(dtype, TOLERANCE[torch.float16])
    worst = (out.float() - ref).norm(dim=-1) / ref.norm(dim=-1)
    assert bool(out.isfinite().all()) and float(worst.max()) < 4 * tolerance
    assert rel_err(out, ref) < tolerance
