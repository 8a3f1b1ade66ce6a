"""Prepared attention calls through the C entry with all, some and none of the scratch that partial results take."""

import math

import pytest
import torch

from helpers import device_compressors, rel_err

pytestmark = pytest.mark.gpu

TQ_ERR_WORKSPACE = 4


class _Call:
    def __init__(self, mode, Hq, Hkv, Sq, Sk, d):
        from turboquant_b200 import _lib as L, compress_kv
        from turboquant_b200.compressors import prepared_constants

        g = torch.Generator().manual_seed(Sq + Sk)
        self.L, self.dims, self.d = L, (1, Hq, Sq, Hkv, Sk), d
        self.mode = L.TQ_MODE_FP32 if mode == "fp32" else L.TQ_MODE_BF16
        dtype = torch.float32 if mode == "fp32" else torch.bfloat16
        self.kc, self.vc = device_compressors(d, 3)
        k, v = (torch.randn(1, Hkv, Sk, d, generator=g).cuda().to(dtype) for _ in range(2))
        self.q = torch.randn(1, Hq, Sq, d, generator=g).cuda().to(dtype)
        self.ck, self.cv = compress_kv(k, v, self.kc, self.vc)
        self.consts = prepared_constants(self.kc, self.vc)
        self.need = L.lib.tq_attention_prepared_workspace_bytes(1, Hq, Sq, Hkv, Sk, Sk, d, self.mode)

    def __call__(self, nbytes, mask=None):
        """(status, output) with `nbytes` of scratch between guard bytes; 0: a NULL pointer."""
        L, q, (B, Hq, Sq, Hkv, Sk) = self.L, self.q, self.dims
        out = torch.full_like(q, float("nan"))
        ws = torch.full((256 + nbytes + 256,), 0xA5, dtype=torch.uint8, device="cuda")
        ck, cv = self.ck, self.cv
        head = (q.data_ptr(), L.TQ_F32 if q.dtype == torch.float32 else L.TQ_BF16, B, Hq, Sq, self.d, *q.stride()[:3], Hkv, Sk, Sk,
                ck["packed_key_indices"].data_ptr(), ck["packed_qjl_signs"].data_ptr(), ck["vec_norms"].data_ptr(),
                ck["residual_norm"].data_ptr(), cv["packed_indices"].data_ptr(), cv["vec_norms"].data_ptr(), self.consts.data_ptr(),
                3, 1.0 / math.sqrt(self.d), 1)
        tail = (out.data_ptr(), *out.stride()[:3], ws.data_ptr() + 256 if nbytes else None, nbytes, self.mode,
                torch.cuda.current_stream().cuda_stream)
        if mask is None:
            st = L.lib.tq_attention_fwd_prepared(*head, None, 0, 0, *tail)
        else:
            st = L.lib.tq_attention_fwd_masked(*head, mask.data_ptr(), L.TQ_MASK_BOOL, 1, Sq * Sk, Sk, *tail)
        torch.cuda.synchronize()
        assert bool((ws[:256] == 0xA5).all()) and bool((ws[256 + nbytes:] == 0xA5).all())
        return st, out


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("Hq,Hkv,Sq,Sk", [(4, 2, 40, 6500), (3, 3, 300, 5300)])
def test_sm_pair_kernel_without_room_is_unsplit(Hq, Hkv, Sq, Sk, d):
    call = _Call("bf16", Hq, Hkv, Sq, Sk, d)
    assert call.need > 0  # a shape that is split
    st, full = call(call.need)
    assert st == 0
    for nbytes in (0, 256, call.need - 256):
        st, out = call(nbytes)
        assert st == 0
        assert torch.equal(out, call(0)[1])
        # the same arithmetic but for where the running maximum starts: 16-bit probabilities and outputs
        assert 0 < rel_err(out, full) < 5e-3


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("Hq,Hkv,Sq,Sk", [(4, 2, 40, 1500), (4, 2, 2, 1500)])  # the tile kernel, the few-rows kernel
def test_fp32_mode_with_room_for_queries_alone_is_unsplit(Hq, Hkv, Sq, Sk, d):
    call = _Call("fp32", Hq, Hkv, Sq, Sk, d)
    queries = (Hq * Sq * 2 * d * 4 + 255) & ~255
    assert call.need > queries
    st, full = call(call.need)
    assert st == 0
    for nbytes in (queries, call.need - 256):
        st, out = call(nbytes)
        assert st == 0
        assert 0 < rel_err(out, full) < 4e-6  # fp32 sums in another order
    for nbytes in (0, queries - 256):
        st, out = call(nbytes)
        assert st == TQ_ERR_WORKSPACE and bool(out.isnan().all())


@pytest.mark.parametrize("mode,Sq", [("bf16", 2), ("bf16", 40), ("fp32", 40)])
def test_masked_calls_need_their_scratch(mode, Sq):
    call = _Call(mode, 4, 2, Sq, 6500, 128)
    mask = torch.ones(Sq, 6500, dtype=torch.bool, device="cuda")
    need = call.L.lib.tq_attention_masked_workspace_bytes(1, 4, Sq, 2, 6500, 6500, 128, call.mode, 1)
    assert need > call.need
    st, out = call(need, mask)
    assert st == 0 and rel_err(out, call(call.need)[1]) < 5e-3
    for nbytes in (0, call.need, need - 256):
        st, out = call(nbytes, mask)
        assert st == TQ_ERR_WORKSPACE and bool(out.isnan().all())


def test_split_kv_kernel_needs_its_scratch():
    call = _Call("bf16", 4, 2, 2, 1500, 128)
    assert call(call.need)[0] == 0
    for nbytes in (0, call.need - 256):
        st, out = call(nbytes)
        assert st == TQ_ERR_WORKSPACE and bool(out.isnan().all())
