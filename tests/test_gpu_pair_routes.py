"""The routes of bf16-mode prefill: keys and values expanded (split over the keys or not), the SM-pair kernel split over the keys,
and the SM-pair kernel unsplit, which calls without scratch take.  Each test says which route its shapes are for and checks it by
the scratch they ask for."""

import threading

import pytest
import torch

from helpers import device_compressors, rel_err
from test_gpu_dense import TOLERANCE, _inputs
from test_gpu_masks import _dense, _mask
from test_gpu_threads import _Work
from test_gpu_workspace import _Call

pytestmark = pytest.mark.gpu

# batch, query heads, KV heads, queries, keys, head_dim
SPLIT_PAIRS = [(3, 6, 6, 1, 6202, 64), (4, 6, 6, 130, 5465, 64), (4, 12, 6, 1, 4623, 64),           # one position block, two; pairs
               (2, 3, 3, 19, 12994, 128), (1, 6, 6, 154, 12130, 128), (2, 12, 6, 136, 10302, 128), (3, 24, 6, 6, 14682, 128)]
EXPANDED = [(16, 12, 4, 200, 333, 64), (2, 32, 8, 700, 900, 128), (1, 27, 9, 1500, 1600, 128)]
EXPANDED_SPLIT = [(1, 32, 8, 300, 8300, 128), (2, 16, 4, 40, 6001, 64)]


def _route(B, Hq, Hkv, Sq, Sk, d):
    from turboquant_b200 import _lib as L

    need = L.lib.tq_attention_prepared_workspace_bytes(B, Hq, Sq, Hkv, Sk, Sk, d, L.TQ_MODE_BF16)
    rows = B * Hkv * ((Sk + 127) // 128) * 512 * d                       # expanded rows, one round
    partial = B * Hq * ((Sq + 127) // 128) * 128 * (d + 2) * 4           # of the SM-pair kernel, per split
    if need >= rows:
        return "expanded" if need < rows + 256 else "expanded and split"
    return "split pairs" if need % partial == 0 and need // partial > 1 else "pairs"


def _packed(B, Hq, Hkv, Sq, Sk, d, bits=3, dtype=torch.bfloat16, seed=0):
    from turboquant_b200 import compress_kv

    g = torch.Generator().manual_seed(Sk + Sq + seed)
    kc, vc = device_compressors(d, bits)
    k, v = (torch.randn(B, Hkv, Sk, d, generator=g).cuda().to(dtype) for _ in range(2))
    q = torch.randn(B, Sq, Hq, d, generator=g).cuda().to(dtype).transpose(1, 2)
    return q, *compress_kv(k, v, kc, vc), kc, vc, g


@pytest.mark.parametrize("mask", [None, "left", "holes", "bias"])
@pytest.mark.parametrize("shape", SPLIT_PAIRS)
def test_sm_pair_kernel_split_over_the_keys(shape, mask):
    from turboquant_b200 import fused_attention

    assert _route(*shape) == "split pairs"
    B, Sq, Sk = shape[0], shape[3], shape[4]
    for bits, causal in ((3, True), (2, False), (4, True)):
        q, ck, cv, kc, vc, g = _packed(*shape, bits=bits)
        if mask == "bias":
            m = torch.randn(B, Sq, Sk, generator=g).cuda()
        else:
            m = (torch.ones(B, Sq, Sk, dtype=torch.bool) if mask is None else _mask(mask, B, Sq, Sk, g)).cuda()
        got = fused_attention(q, ck, cv, kc, vc, causal=causal, attention_mask=None if mask is None else m[:, None])
        assert rel_err(got, _dense(q, ck, cv, kc, vc, m, causal)) < 1e-2  # 16-bit operands and output


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("Hq,Hkv,Sq,Sk", [(12, 12, 200, 30000), (25, 25, 100, 9000)])
def test_sm_pair_kernel_without_room_for_partial_results(Hq, Hkv, Sq, Sk, d):
    assert _route(1, Hq, Hkv, Sq, Sk, d) == "split pairs"
    call = _Call("bf16", Hq, Hkv, Sq, Sk, d)
    st, full = call(call.need)
    assert st == 0
    for nbytes in (0, 256, call.need - 256):
        st, out = call(nbytes)
        assert st == 0 and torch.equal(out, call(0)[1])
        assert 0 < rel_err(out, full) < 5e-3  # the same arithmetic but for where the running maximum starts


@pytest.mark.parametrize("Hq,Hkv,Sq,Sk,d", [(8, 2, 4096, 8192, 128), (4, 4, 2500, 9000, 64), (9, 3, 3000, 3333, 128)])
def test_long_calls_of_the_sm_pair_kernel(Hq, Hkv, Sq, Sk, d):
    # without scratch: its rings wrap around many times
    from turboquant_b200 import fused_attention

    call = _Call("bf16", Hq, Hkv, Sq, Sk, d)
    st, out = call(0)
    ref = fused_attention(call.q.float(), call.ck, call.cv, call.kc, call.vc, mode="fp32")
    assert st == 0 and rel_err(out, ref) < 1e-2  # 16-bit operands and output
    worst = ((out.float() - ref).norm(dim=-1) / ref.norm(dim=-1)).max()
    assert float(worst) < 4e-2


@pytest.mark.parametrize("bits", [2, 3, 4])
@pytest.mark.parametrize("shape", EXPANDED + EXPANDED_SPLIT)
def test_fp32_queries_over_expanded_rows(shape, bits):
    assert _route(*shape) == ("expanded" if shape in EXPANDED else "expanded and split")
    from turboquant_b200 import fused_attention

    q, ck, cv, kc, vc = _inputs(*shape, bits, torch.float32)
    assert not q.is_contiguous()
    ref = fused_attention(q, ck, cv, kc, vc, mode="fp32")
    out = fused_attention(q, ck, cv, kc, vc, mode="bf16")
    assert out.dtype == torch.float32
    worst = ((out - ref).norm(dim=-1) / ref.norm(dim=-1)).max()
    # (fp16 queries beside fp32 ones: their rounding is among those of the bound; the output is not rounded)
    assert rel_err(out, ref) < TOLERANCE[torch.float16] and float(worst) < 4 * TOLERANCE[torch.float16]


@pytest.mark.parametrize("shape", EXPANDED + EXPANDED_SPLIT + SPLIT_PAIRS[1::2])
@pytest.mark.parametrize("bad_key", [False, True])
def test_rows_that_meet_nan_or_inf(shape, bad_key):
    from turboquant_b200 import compress_kv, fused_attention

    B, Hq, Hkv, Sq, Sk, d = shape
    assert _route(*shape) != "pairs"
    g = torch.Generator().manual_seed(Sq + Sk)
    kc, vc = device_compressors(d, 3)
    k, v = (torch.randn(B, Hkv, Sk, d, generator=g).cuda().bfloat16() for _ in range(2))
    q = torch.randn(B, Sq, Hq, d, generator=g).cuda().bfloat16().transpose(1, 2)
    bad = torch.zeros(B, Hq, Sq, dtype=torch.bool)
    if bad_key:
        at = Sk - Sq + Sq // 2  # seen by the later half of the queries of the last group's heads
        k[B - 1, Hkv - 1, at, 5] = float("nan")
        bad[B - 1, (Hkv - 1) * (Hq // Hkv):, Sq // 2:] = True
    else:
        q[0, 1, Sq - 1, 3] = float("nan")
        q[B - 1, 0, 0] = float("inf")
        bad[0, 1, Sq - 1] = bad[B - 1, 0, 0] = True
    ck, cv = compress_kv(k, v, kc, vc)
    out = fused_attention(q, ck, cv, kc, vc)
    assert torch.equal(~out.isfinite().all(-1).cpu(), bad)
    assert torch.equal(~out.isfinite().any(-1).cpu(), bad)


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("dtype,shape", [(torch.bfloat16, EXPANDED[1]), (torch.float16, EXPANDED[0]), (torch.float16, EXPANDED_SPLIT[0]),
                                         (torch.bfloat16, SPLIT_PAIRS[1]), (torch.float16, SPLIT_PAIRS[5])])
def test_replay_follows_the_buffers(dtype, shape, masked):
    from turboquant_b200 import CompressedKVCache

    B, Hq, Hkv, Sq, Sk, d = shape
    kc, vc = device_compressors(d, 3)
    g = torch.Generator().manual_seed(Sk)
    draw = lambda *dims: torch.randn(*dims, generator=g).cuda().to(dtype)
    q, k, v = draw(B, Hq, Sq, d), draw(B, Hkv, Sk, d), draw(B, Hkv, Sk, d)
    mask = torch.zeros(B, 1, Sq, Sk, dtype=torch.bool, device="cuda")
    cache = CompressedKVCache(kc, vc, B, Hkv, Sk + 9)

    def step():
        cache.reset()
        cache.append(k, v)
        return cache.attend(q, attention_mask=mask if masked else None)

    def fill():
        q.copy_(draw(*q.shape)); k.copy_(draw(*k.shape)); v.copy_(draw(*v.shape))
        live = torch.randint(Sq, Sk, (B, 1, 1, 1), generator=g).cuda()
        mask.copy_((torch.arange(Sk, device="cuda") >= Sk - live).expand(B, 1, Sq, Sk))

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


def test_threads_with_streams_of_their_own():
    shapes = [(torch.bfloat16, EXPANDED[1]), (torch.float16, EXPANDED[0]), (torch.bfloat16, EXPANDED_SPLIT[0]), (torch.float16, SPLIT_PAIRS[1]),
              (torch.bfloat16, SPLIT_PAIRS[5])]
    work = [_Work(i, dtype, s[5], s[0], s[1], s[2], s[3], s[4]) for i, (dtype, s) in enumerate(shapes)]
    want = [w() for w in work]
    torch.cuda.synchronize()
    wrong, start = [], threading.Barrier(len(work))

    def run(i):
        try:
            stream = torch.cuda.Stream()
            start.wait()
            with torch.cuda.stream(stream):
                for _ in range(10):
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
