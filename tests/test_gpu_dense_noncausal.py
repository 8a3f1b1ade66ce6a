"""Attention over expanded keys and values with more queries than keys (never causal), against the fp32 kernels on the same
packed bytes; tolerances of test_gpu_dense.py."""

import pytest
import torch

from test_gpu_dense import _check, _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk", [(4, 16, 4, 2048, 500), (1, 12, 12, 5026, 2), (3, 7, 1, 2692, 353), (2, 27, 9, 1300, 257)])
@pytest.mark.parametrize("masked", [False, True])
def test_more_queries_than_keys(B, Hq, Hkv, Sq, Sk, d, masked):
    mask = None
    if masked:
        g = torch.Generator(device="cuda").manual_seed(4)
        mask = torch.rand(B, 1, Sq, Sk, generator=g, device="cuda") > 0.4
        mask[..., 0] = True
        mask[:, :, 17] = False  # a row that sees nothing averages all keys
    _check(*_inputs(B, Hq, Hkv, Sq, Sk, d, 3, torch.bfloat16), causal=False, attention_mask=mask)
