"""Streamed decode attention with rings of two to eight stages (what the step's table bounds, and four in front of a product that reads its weights
straight from memory), pairs in as many pieces as the last arriver reads at once and more, and chains: one in which the products around it start
early, and one in which the attention does too (with its preparation in the same launch), each against the same calls one by one."""
import math
from types import SimpleNamespace

import pytest
import torch

from arle_b200 import ops
from arle_b200.engine import Workspace
from launched import kernels
from test_kernels_gpu import _fast_setup, _ref_attn

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _stream_decode(q, out, kc, vc, qi, kv, bt, nq, nkv, hd, ps, window, ctas, scratch=None, product=None):
    R = kv.numel()
    slots = (ctas + R * nkv) * (nq // nkv)
    if scratch is None:
        scratch = (torch.zeros(slots * hd, device=DEV), torch.zeros(slots * 2, device=DEV), torch.zeros(R * nkv, dtype=torch.int32, device=DEV))
    ops.paged_attention_decode_stream(q, out, kc, vc, qi, kv, bt, nq, nkv, hd, ps, 1 / math.sqrt(hd), window, *scratch, ctas, product=product)
    return scratch


@pytest.mark.parametrize("nq,nkv,lens", [
    (16, 8, [64]), (16, 8, [1153]), (16, 8, [1400] * 2), (16, 8, [2100] * 2), (16, 8, [300] * 8), (16, 8, [2100] * 8), (16, 8, [700, 1, 2300, 65] * 3),
    (32, 8, [700]), (32, 8, [2100] * 3), (16, 8, [16500] * 3), (2, 1, [64 * 16]), (2, 1, [64 * 16 + 1]), (2, 1, [64 * 10]), (2, 1, [64 * 11]), (2, 1, [64 * 20]), (2, 1, [64 * 21]), (2, 1, [64 * 33]), (4, 2, [64 * 50 + 7])])
@pytest.mark.parametrize("behind", [None, 1024])           # columns of the product that follows
def test_rings_and_pieces(nq, nkv, lens, behind):
    product = None if behind is None else (torch.empty(behind, nq * 128, dtype=torch.bfloat16, device=DEV), None)
    q, kc, vc, pos, rows, bt, qi, kv = _fast_setup(nq, nkv, 128, 16, lens, [1] * len(lens), seed=4)
    out = torch.zeros(len(lens), nq * 128, dtype=torch.bfloat16, device=DEV)
    want = _ref_attn(q, kc, vc, pos, rows, bt, nq, nkv, 128, 16, None)
    scratch = None
    for _ in range(2):
        out.zero_()
        scratch = _stream_decode(q, out, kc, vc, qi, kv, bt, nq, nkv, 128, 16, None, 148, scratch, product)
        torch.testing.assert_close(out.float().cpu(), want, rtol=2e-2, atol=1e-2)      # P is rounded to bfloat16
        assert scratch[2].abs().sum().item() == 0


def test_a_chain_with_products_in_front_and_behind():
    nq, nkv, hidden, lens = 16, 8, 1024, [900, 130]
    q, kc, vc, pos, rows, bt, qi, kv = _fast_setup(nq, nkv, 128, 16, lens, [1] * 2, seed=6)
    g = torch.Generator(device=DEV).manual_seed(1)
    w_q = (torch.randn(nq * 128, hidden, generator=g, device=DEV) * 0.03).bfloat16()
    w_o = (torch.randn(hidden, nq * 128, generator=g, device=DEV) * 0.03).bfloat16()
    x0 = torch.randn(2, hidden, generator=g, device=DEV).bfloat16()
    slots = (148 + 2 * nkv) * (nq // nkv)
    scratch = (torch.zeros(slots * 128, device=DEV), torch.zeros(slots * 2, device=DEV), torch.zeros(2 * nkv, dtype=torch.int32, device=DEV))
    xs = [x0] + [torch.empty_like(x0) for _ in range(12)]
    qs, outs = torch.empty_like(q), torch.empty_like(q)

    def chain(wait):
        for a, b in zip(xs, xs[1:]):
            for step in (lambda: ops.gemm(a, w_q, qs), lambda: ops.paged_attention_decode_stream(
                    qs, outs, kc, vc, qi, kv, bt, nq, nkv, 128, 16, 1 / math.sqrt(128), None, *scratch, 148), lambda: ops.gemm(outs, w_o, b)):
                step()
                if wait:
                    torch.cuda.synchronize()
        torch.cuda.synchronize()
        return torch.stack(xs[1:])

    want = chain(True)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for a, b in zip(xs, xs[1:]):
            ops.gemm(a, w_q, qs)
            ops.paged_attention_decode_stream(qs, outs, kc, vc, qi, kv, bt, nq, nkv, 128, 16, 1 / math.sqrt(128), None, *scratch, 148)
            ops.gemm(outs, w_o, b)
    assert want.isfinite().all() and want.abs().max() > 0
    for _ in range(5):
        assert torch.equal(chain(False), want)
        for x in xs[1:]:
            x.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(torch.stack(xs[1:]), want)


@pytest.mark.parametrize("nq,hidden,sums,room", [
    (16, 1024, True, True), (16, 2048, True, True), (32, 2560, True, True), (32, 4096, False, True),
    (16, 4096, True, False), (32, 4096, True, False), (64, 5120, True, False), (16, None, False, False)])
def test_room_is_left_in_front_of_products_without_a_ring_alone(nq, hidden, sums, room):
    """``sums``: the product adds into the residual.  A step of 8 requests of 2,048 tokens: rings of six stages, four where room is left."""
    nkv, lens = 8, [2048] * 8
    q, kc, vc, pos, rows, bt, qi, kv = _fast_setup(nq, nkv, 128, 16, lens, [1] * 8, seed=4)
    out = torch.zeros(8, nq * 128, dtype=torch.bfloat16, device=DEV)
    product = None if hidden is None else (torch.empty(hidden, nq * 128, dtype=torch.bfloat16, device=DEV), object() if sums else None)
    scratch = _stream_decode(q, out, kc, vc, qi, kv, bt, nq, nkv, 128, 16, None, 148)
    shared, = [p.sharedMemBytes for name, p in kernels(lambda: _stream_decode(q, out, kc, vc, qi, kv, bt, nq, nkv, 128, 16, None, 148, scratch, product))
               if "decode_stream_kernel" in name]
    assert shared // 32768 in ((4,) if room else (5, 6)), shared         # 32 KB a stage, and less than one for the rest


@pytest.mark.parametrize("memo", [False, True])            # with a plan of the step, which the first layer's call makes
@pytest.mark.parametrize("nq,nkv,hidden,lens", [(16, 8, 1024, [900, 130]), (16, 8, 1024, [4000, 1, 64]), (4, 1, 256, [33 * 64])])
def test_a_chain_in_which_the_attention_starts_early(nq, nkv, hidden, lens, memo):
    R, layers, hd, ps = len(lens), 6, 128, 16
    _, kc0, vc0, pos, rows, bt, qi, kv = _fast_setup(nq, nkv, hd, ps, lens, [1] * R, seed=6)
    last = kv.long() - 1
    slots = (bt[torch.arange(R, device=DEV), last // ps].long() * ps + last % ps).to(torch.int32)
    g = torch.Generator(device=DEV).manual_seed(1)
    w_qkv = [(torch.randn((nq + 2 * nkv) * hd, hidden, generator=g, device=DEV) * 0.03).bfloat16() for _ in range(layers)]
    w_o = [(torch.randn(hidden, nq * hd, generator=g, device=DEV) * 0.05).bfloat16() for _ in range(layers)]
    norm = torch.rand(hd, generator=g, device=DEV) + 0.5
    inv_freq = torch.pow(torch.tensor(1e4), -torch.arange(hd // 2, dtype=torch.float32) * 2 / hd).to(DEV)
    xs = [torch.randn(R, hidden, generator=g, device=DEV).bfloat16()] + [torch.empty(R, hidden, dtype=torch.bfloat16, device=DEV) for _ in range(layers)]
    caches = [(kc0.clone(), vc0.clone()) for _ in range(layers)]
    qkv = torch.empty(R, (nq + 2 * nkv) * hd, dtype=torch.bfloat16, device=DEV)
    attn = torch.empty(R, nq * hd, dtype=torch.bfloat16, device=DEV)
    batch = SimpleNamespace(max_q_len=1, num_rows=R, ws=Workspace(DEV), q_indptr=qi, kv_lens=kv)       # scratch and counters of all layers

    def chain(wait):
        if memo:
            batch.memo = {}
        for i in range(layers):
            k, v = caches[i]
            for step in (lambda: ops.gemm(xs[i], w_qkv[i], qkv),
                         lambda: ops.decode_attention_with_prep(qkv, attn, k, v, slots, norm, norm, 1e-6, inv_freq, bt, nq, nkv, hd, ps, 1 / math.sqrt(hd),
                                                                None, batch, product=(w_o[i], None)),
                         lambda: ops.gemm(attn, w_o[i], xs[i + 1])):
                step()
                if wait:
                    torch.cuda.synchronize()

    def clear():
        for t in (*xs[1:], qkv, attn):
            t.fill_(float("nan"))
        for k, v in caches:
            k.copy_(kc0), v.copy_(vc0)
        torch.cuda.synchronize()

    def result():
        torch.cuda.synchronize()
        ops.check_errors(DEV)
        return [t.clone() for t in (*xs[1:], *(t for pair in caches for t in pair))]

    clear()
    chain(True)
    want = result()
    assert all(t.isfinite().all() for t in want[:layers]) and want[layers - 1].abs().max() > 0
    assert not torch.equal(want[layers], kc0)              # the new keys are in the cache
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(False)
    for _ in range(4):
        for run in (lambda: chain(False), graph.replay):
            clear()
            run()
            assert all(torch.equal(a, b) for a, b in zip(result(), want))
