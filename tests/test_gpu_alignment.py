"""Packed outputs of the compression entry points at addresses that wide stores cannot reach."""

import pytest
import torch

from helpers import device_compressors

pytestmark = pytest.mark.gpu


def _call(L, k, v, consts, bits, outs):
    B, H, S, d = k.shape
    dt = {torch.bfloat16: L.TQ_BF16, torch.float16: L.TQ_F16}[k.dtype]
    return L.lib.tq_compress_kv(k.data_ptr(), v.data_ptr(), dt, B, H, S, d, *k.stride()[:3], *v.stride()[:3], consts.data_ptr(),
                                bits, *outs, S, 0, L.TQ_MODE_BF16, torch.cuda.current_stream().cuda_stream)


def _outputs(n, d, bits, off):
    """Guarded buffers for key indices, signs, norms, residual norms, value indices and norms, and their addresses."""
    sizes = [n * d * (bits - 1) // 8, n * d // 8, 2 * n, 2 * n, n * d * bits // 8, 2 * n]
    bufs = [torch.full((s + 64,), 0xA5, dtype=torch.uint8, device="cuda") for s in sizes]
    offs = [16 + (off if i in (0, 1, 4) else 0) for i in range(6)]
    return bufs, offs, sizes, [b.data_ptr() + o for b, o in zip(bufs, offs)]


@pytest.mark.parametrize("off", [1, 2, 4, 8])
@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("H,S", [(3, 5), (8, 400)])  # the few-vectors kernel and the tile kernel behind the fused one
def test_fp16_rows_may_start_anywhere(H, S, d, bits, off):
    from turboquant_b200 import _lib as L
    from turboquant_b200.compressors import prepared_constants

    g = torch.Generator().manual_seed(S + bits)
    kc, vc = device_compressors(d, bits)
    consts = prepared_constants(kc, vc)
    k, v = (torch.randn(1, H, S, d, generator=g).cuda().half() for _ in range(2))
    n = H * S
    got = []
    for o in (0, off):
        bufs, offs, sizes, ptrs = _outputs(n, d, bits, o)
        L.check(_call(L, k, v, consts, bits, ptrs))
        for b, at, size in zip(bufs, offs, sizes):
            assert bool((b[:at] == 0xA5).all()) and bool((b[at + size:] == 0xA5).all())
        got.append([b[at:at + size].clone() for b, at, size in zip(bufs, offs, sizes)])
    for i, (a, b) in enumerate(zip(*got)):
        if i in (0, 1, 4):  # open coordinates are decided as the fp32 kernels decide them: the same bytes
            assert torch.equal(a, b)
        else:  # norms: the order of a sum, one fp16 step
            assert int((a.view(torch.int16).int() - b.view(torch.int16).int()).abs().max()) <= 1


@pytest.mark.parametrize("bits", [2, 3, 4])
def test_bf16_rows_that_do_not_fit_are_refused(bits):
    from turboquant_b200 import _lib as L
    from turboquant_b200.compressors import prepared_constants

    kc, vc = device_compressors(128, bits)
    consts = prepared_constants(kc, vc)
    k, v = (torch.randn(1, 2, 3, 128).cuda().bfloat16() for _ in range(2))
    for which, step in ((0, 4 if bits == 3 else 2), (1, 2), (4, {2: 4, 3: 2, 4: 8}[bits]), (2, 1), (3, 1), (5, 1)):
        bufs, offs, sizes, ptrs = _outputs(6, 128, bits, 0)
        ptrs[which] += step
        assert _call(L, k, v, consts, bits, ptrs) == 1  # TQ_ERR_INVALID_ARG
        # ... and by the entry point of that side alone
        st = torch.cuda.current_stream().cuda_stream
        if which < 4:
            s = L.lib.tq_compress_keys(k.data_ptr(), L.TQ_BF16, 1, 2, 3, 128, *k.stride()[:3], kc.Pi.data_ptr(), kc.S_eff.data_ptr(),
                                       kc.centroids.data_ptr(), kc.boundaries.data_ptr(), bits, *ptrs[:4], L.TQ_MODE_BF16, st)
        else:
            s = L.lib.tq_compress_values(v.data_ptr(), L.TQ_BF16, 1, 2, 3, 128, *v.stride()[:3], vc.Pi.data_ptr(),
                                         vc.boundaries.data_ptr(), bits, *ptrs[4:], L.TQ_MODE_BF16, st)
        assert s == 1
        torch.cuda.synchronize()
        assert all(bool((b == 0xA5).all()) for b in bufs)
