"""Which prefill kernel the sizes of a call ask for, read from its scratch: no GPU needed (148 SMs are assumed without one)."""

import pytest


def _need(B, Hq, Hkv, Sq, Sk, d):
    from turboquant_b200 import _lib as L

    return L.lib.tq_attention_prepared_workspace_bytes(B, Hq, Sq, Hkv, Sk, Sk, d, L.TQ_MODE_BF16)


@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk,d", [(8, 32, 8, 8192, 512, 128), (4, 16, 16, 4000, 300, 64), (1, 12, 12, 5026, 2, 128),
                                              (3, 7, 1, 2692, 353, 128), (16, 16, 2, 4791, 824, 128), (8, 32, 8, 2048, 1000, 128)])
def test_many_more_queries_than_keys_expand_them(B, Hq, Hkv, Sq, Sk, d):
    assert _need(B, Hq, Hkv, Sq, Sk, d) >= B * Hkv * ((Sk + 127) // 128) * 512 * d


@pytest.mark.parametrize("B,Hq,Hkv,Sq,Sk,d", [(1, 32, 8, 100, 100, 128), (1, 32, 8, 64, 64, 128), (1, 12, 12, 200, 333, 64)])
def test_small_calls_do_not(B, Hq, Hkv, Sq, Sk, d):
    assert _need(B, Hq, Hkv, Sq, Sk, d) == 0
