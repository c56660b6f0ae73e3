"""Streamed decode attention with rings of two to eight stages (what the step's table bounds, and four in front of a product that reads its weights
straight from memory), pairs in as many pieces as the last arriver reads at once and more, and a chain in which the products around it start early."""
import math

import pytest
import torch

from arle_b200 import ops
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
    (32, 8, [700]), (32, 8, [2100] * 3), (16, 8, [16500] * 3), (2, 1, [64 * 16]), (2, 1, [64 * 16 + 1]), (2, 1, [64 * 33]), (4, 2, [64 * 50 + 7])])
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
