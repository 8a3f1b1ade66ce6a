"""Bf16-mode attention refuses packed rows at addresses that its kernels' loads cannot reach, on the host: a misaligned wide load
is a fault of the device.  Nothing here is launched, so no GPU is needed."""

import ctypes

import pytest

TQ_OK, TQ_ERR_INVALID_ARG = 0, 1


def _status(B, Hq, Sq, Hkv, Sk, d, bits, entry, offs, scratch=True):
    """Status and message of a bf16-mode call whose key indices, signs, value indices and norms start `offs` bytes behind a
    256-byte boundary.  Pointers are of host memory: what passes the checks of the arguments ends in a CUDA error."""
    from turboquant_b200 import _lib as L

    buf = ctypes.create_string_buffer(4096)
    p = (ctypes.addressof(buf) + 255) & ~255
    rows = (p + offs[0], p + offs[1], p + offs[3], p + offs[3], p + offs[2], p + offs[3])
    head = (p, L.TQ_BF16, B, Hq, Sq, d, Hq * Sq * d, Sq * d, d, Hkv, Sk)
    out = (p, Hq * Sq * d, Sq * d, d)
    if entry == "prepared":
        need = L.lib.tq_attention_prepared_workspace_bytes(B, Hq, Sq, Hkv, Sk, Sk, d, L.TQ_MODE_BF16) if scratch else 0
        st = L.lib.tq_attention_fwd_prepared(*head, Sk, *rows, p, bits, 0.1, 1, None, 0, 0, *out, p if scratch else None, need,
                                             L.TQ_MODE_BF16, None)
    else:
        need = L.lib.tq_attention_workspace_bytes(B, Hq, Sq, d, L.TQ_MODE_BF16)
        st = L.lib.tq_attention_fwd(*head, *rows, p, p, p, p, p, bits, 0.1, 1, None, 0, 0, *out, p, need, L.TQ_MODE_BF16, None)
    assert st != TQ_OK
    return st, L.last_error()


@pytest.mark.parametrize("entry", ["prepared", "plain"])
@pytest.mark.parametrize("d,bits,Sq,Sk,boundary", [(128, 3, 1, 3000, (16, 16, 16)),  # split-KV kernel
                                                   (128, 2, 40, 40, (8, 8, 8)),      # SM-pair kernel
                                                   (64, 4, 40, 40, (8, 8, 8)),
                                                   (64, 3, 40, 40, (8, 8, 4))])
def test_rows_off_the_boundary_are_refused(entry, d, bits, Sq, Sk, boundary):
    for which in range(3):
        for step in (1, 2, 4, 8):
            offs = [0, 0, 0, 0]
            offs[which] = step
            st, message = _status(1, 4, Sq, 2, Sk, d, bits, entry, offs)
            assert (st == TQ_ERR_INVALID_ARG and "packed rows" in message) == (step % boundary[which] != 0), (which, step, message)
    st, message = _status(1, 4, Sq, 2, Sk, d, bits, entry, [0, 0, 0, 1])
    assert st == TQ_ERR_INVALID_ARG and "norms" in message


def test_expansion_reads_words():
    shape = (16, 16, 700, 8, 700, 128, 3)  # many queries per key
    for step in (1, 2, 4, 8):
        for which in range(3):
            offs = [0, 0, 0, 0]
            offs[which] = step
            st, message = _status(*shape, "prepared", offs)
            assert (st == TQ_ERR_INVALID_ARG) == (step < 4), (which, step, message)
            st, message = _status(*shape, "prepared", offs, scratch=False)  # the SM-pair kernel
            assert (st == TQ_ERR_INVALID_ARG) == (step < 8), (which, step, message)
