"""Prepared prefill calls that expand keys and values, with less scratch than that takes: served from the packed bytes."""

import math

import pytest
import torch

from helpers import rel_err
from test_gpu_workspace import TQ_ERR_WORKSPACE, _Call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("Hq,Hkv,Sq,Sk", [(32, 8, 1100, 1100), (27, 9, 2000, 2300)])  # the SM-pair kernel would not be split
def test_masked_calls_need_the_summary_alone(Hq, Hkv, Sq, Sk, d):
    call = _Call("bf16", Hq, Hkv, Sq, Sk, d)
    mask = (torch.arange(Sk, device="cuda") >= 150).expand(Sq, Sk).contiguous()
    need = call.L.lib.tq_attention_masked_workspace_bytes(1, Hq, Sq, Hkv, Sk, Sk, d, call.mode, 1)
    summary = need - call.need
    assert call.need >= Hkv * ((Sk + 127) // 128) * 512 * d  # expanded rows
    st, full = call(need, mask)
    assert st == 0
    st, alone = call(summary, mask)
    assert st == 0
    # the SM-pair kernel's 16-bit operands and rotated outputs beside the expansion's: 5e-3 of the output at most
    assert rel_err(alone, full) < 1e-2
    for nbytes in (summary + 256, need // 2, need - 256):
        st, out = call(nbytes, mask)
        assert st == 0 and torch.equal(out, alone)
    for nbytes in (0, summary - 256):
        st, out = call(nbytes, mask)
        assert st == TQ_ERR_WORKSPACE and bool(out.isnan().all())


@pytest.mark.parametrize("off", [0, 8])
def test_scratch_off_its_boundary_is_not_used(off):
    call = _Call("bf16", 32, 8, 1100, 1100, 128)
    L, q, ck, cv = call.L, call.q, call.ck, call.cv
    (B, Hq, Sq, Hkv, Sk), d = call.dims, call.d
    ws = torch.full((call.need + 512,), 0xA5, dtype=torch.uint8, device="cuda")
    out = torch.full_like(q, float("nan"))
    st = L.lib.tq_attention_fwd_prepared(
        q.data_ptr(), L.TQ_BF16, B, Hq, Sq, d, *q.stride()[:3], Hkv, Sk, Sk, ck["packed_key_indices"].data_ptr(),
        ck["packed_qjl_signs"].data_ptr(), ck["vec_norms"].data_ptr(), ck["residual_norm"].data_ptr(), cv["packed_indices"].data_ptr(),
        cv["vec_norms"].data_ptr(), call.consts.data_ptr(), 3, 1.0 / math.sqrt(d), 1, None, 0, 0, out.data_ptr(), *out.stride()[:3],
        ws.data_ptr() + off, call.need, call.mode, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert st == 0
    assert torch.equal(out, call(0 if off else call.need)[1])
    assert bool((ws == 0xA5).all()) == (off != 0)
