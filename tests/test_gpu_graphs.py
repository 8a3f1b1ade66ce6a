"""Attention calls of several launches captured in a graph and replayed on other data."""

import pytest
import torch

from helpers import device_compressors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("dtype,d,Hq,Hkv,Sq,Sk", [(torch.bfloat16, 128, 8, 2, 1, 3000),   # split-KV kernel
                                                  (torch.float16, 128, 4, 2, 200, 500),   # SM-pair kernel
                                                  (torch.bfloat16, 64, 4, 2, 40, 6500),   # ... split over the keys
                                                  (torch.float32, 128, 4, 2, 2, 1500),    # few rows in fp32
                                                  (torch.float32, 64, 4, 2, 100, 1500)])  # fp32 tiles in chunks
def test_replay_follows_the_buffers(dtype, d, Hq, Hkv, Sq, Sk, masked):
    from turboquant_b200 import CompressedKVCache

    kc, vc = device_compressors(d, 3)
    g = torch.Generator().manual_seed(Sk)
    draw = lambda *shape: torch.randn(*shape, generator=g).cuda().to(dtype)
    q, k, v = draw(2, Hq, Sq, d), draw(2, Hkv, Sk, d), draw(2, Hkv, Sk, d)
    mask = torch.zeros(2, 1, Sq, Sk, dtype=torch.bool, device="cuda")
    cache = CompressedKVCache(kc, vc, 2, Hkv, Sk + 9)

    def step():
        cache.reset()
        cache.append(k, v)
        return cache.attend(q, attention_mask=mask if masked else None)

    def fill():
        q.copy_(draw(*q.shape)); k.copy_(draw(*k.shape)); v.copy_(draw(*v.shape))
        live = torch.randint(Sk // 2, Sk, (2, 1, 1, 1), generator=g).cuda()
        mask.copy_((torch.arange(Sk, device="cuda") >= Sk - live).expand(2, 1, Sq, Sk))

    fill()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        step()
    torch.cuda.current_stream().wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    for _ in range(3):
        fill()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, step())
