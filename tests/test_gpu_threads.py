"""Calls from several threads, each on a stream of its own, give what they give one after the other."""

import threading

import pytest
import torch

from helpers import device_compressors

pytestmark = pytest.mark.gpu

_SHAPES = [(torch.bfloat16, 128, 1, 8, 2, 1, 3000), (torch.bfloat16, 128, 2, 4, 2, 300, 700), (torch.float32, 64, 1, 4, 4, 200, 900),
           (torch.float16, 64, 2, 6, 3, 20, 5200), (torch.float32, 128, 1, 8, 2, 2, 1500), (torch.bfloat16, 64, 3, 2, 2, 5, 130)]


class _Work:
    def __init__(self, seed, dtype, d, B, Hq, Hkv, Sq, Sk):
        g = torch.Generator().manual_seed(seed)
        self.kc, self.vc = device_compressors(d, 3)
        self.k, self.v = (torch.randn(B, Hkv, Sk, d, generator=g).cuda().to(dtype) for _ in range(2))
        self.q = torch.randn(B, Sq, Hq, d, generator=g).cuda().to(dtype).transpose(1, 2)
        # a key visible to every row, so that no row averages
        self.mask = (torch.rand(B, 1, Sq, Sk, generator=g) < 0.7).cuda()
        self.mask[..., 0] = True

    def __call__(self):
        from turboquant_b200 import CompressedKVCache, compress_kv, fused_attention

        B, Hkv, Sk, _ = self.k.shape
        ck, cv = compress_kv(self.k, self.v, self.kc, self.vc)
        cache = CompressedKVCache(self.kc, self.vc, B, Hkv, Sk + 5)
        cache.append(self.k, self.v)
        return [fused_attention(self.q, ck, cv, self.kc, self.vc), cache.attend(self.q), cache.attend(self.q, attention_mask=self.mask),
                self.vc.decompress(cv), self.kc.asymmetric_attention_scores(self.q[:, :, -2:], ck), ck["packed_qjl_signs"]]


def test_threads_with_streams_of_their_own():
    work = [_Work(i, *shape) for i, shape in enumerate(_SHAPES)]
    want = [w() for w in work]
    torch.cuda.synchronize()
    wrong, start = [], threading.Barrier(len(work))

    def run(i):
        try:
            stream = torch.cuda.Stream()
            start.wait()
            with torch.cuda.stream(stream):
                for _ in range(25):
                    got = work[i]()
                    stream.synchronize()
                    if not all(torch.equal(a, b) for a, b in zip(got, want[i])):
                        wrong.append(i)
        except Exception as e:  # a thread's exception would go unseen
            wrong.append((i, e))

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(work))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_two_streams_of_one_thread_without_waiting():
    a, b = _Work(10, *_SHAPES[0]), _Work(11, *_SHAPES[1])
    want = a(), b()
    torch.cuda.synchronize()
    sa, sb = torch.cuda.Stream(), torch.cuda.Stream()
    got = []
    for _ in range(10):
        with torch.cuda.stream(sa):
            ga = a()
        with torch.cuda.stream(sb):
            gb = b()
        got.append((ga, gb))
    torch.cuda.synchronize()
    for ga, gb in got:
        assert all(torch.equal(x, y) for x, y in zip(ga, want[0]))
        assert all(torch.equal(x, y) for x, y in zip(gb, want[1]))
