"""The float32 attention on tiles against float64: rows just below and at the least length, at and past a tile of 32 queries and 64 keys,
behind contexts, windows shorter and longer than a tile, grouped heads, sinks larger and smaller than the scores, gates, pages that no tile
boundary falls on; and a token's bits do not depend on how its prompt was cut, into single tokens, short rows or long ones."""
import math

import pytest
import torch

from arle_b200 import ops
from arle_b200.cache import CacheManager
from arle_b200.engine import StepEntry
from arle_b200.engine.batch import StepContext, Workspace
from arle_b200.parts.base import CacheNeed

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _setup(rows, nkv, hd, page, window, g):
    kvs = [n + s for n, s in rows]
    cm = CacheManager([CacheNeed(nkv, hd, window)], [], page, sum(-(-k // page) for k in kvs) + 3, len(rows), max(kvs), torch.float32, DEV)
    for i in range(len(rows)):
        cm.add_request(i)
    for i, (_, s) in enumerate(rows):
        if s:
            cm.append([(i, s)])
    cm.append([(i, n) for i, (n, _) in enumerate(rows)])
    for a in cm.groups[0].arrays:
        a.normal_(generator=g)
    ctx = StepContext(cm, Workspace(DEV)).build([StepEntry(i, [0] * n) for i, (n, _) in enumerate(rows)], [s for _, s in rows])
    return cm, ctx, ctx.cache_view(0)


@pytest.mark.parametrize("nq,nkv,hd,page", [(4, 2, 64, 16), (3, 1, 128, 5), (2, 2, 128, 64)])
@pytest.mark.parametrize("rows,window", [([(8, 0)], None), ([(7, 30), (33, 0), (1, 70), (64, 65)], None), ([(100, 130), (8, 9)], 40),
                                          ([(70, 3)], 1), ([(301, 0), (3, 200)], 128)], ids=["least", "mixed", "window40", "window1", "window128"])
@pytest.mark.parametrize("tail", [False, True])
def test_against_float64(nq, nkv, hd, page, rows, window, tail):
    g = torch.Generator(device=DEV).manual_seed(nq + hd + len(rows))
    cm, ctx, view = _setup(rows, nkv, hd, page, window, g)
    T = sum(n for n, _ in rows)
    q = torch.randn(T, nq * hd + 4, generator=g, device=DEV)[:, : nq * hd]
    sink = torch.linspace(-3.0, 9.0, nq, device=DEV) if tail else None
    gate = torch.randn(T, nq, generator=g, device=DEV) if tail else None
    out = torch.full((T, nq * hd), 7.0, device=DEV)
    ops.paged_attention(q, out, view.k, view.v, ctx.positions, ctx.row_of_token, view.block_table, nq, nkv, hd, page, hd ** -0.5, window,
                        batch=ctx, sink=sink, gate=gate)
    at = 0
    for i, (n, s) in enumerate(rows):
        slots = torch.from_numpy(cm.slot_mapping(0, i, 0, n + s)).long().to(DEV)
        k, v = (a[slots // page, :, slots % page].double().repeat_interleave(nq // nkv, 1) for a in (view.k, view.v))
        sc = torch.einsum("thd,jhd->htj", q[at: at + n].reshape(n, nq, hd).double(), k) * hd ** -0.5
        p, j = torch.arange(s, s + n, device=DEV)[:, None], torch.arange(n + s, device=DEV)[None]
        sc = sc.masked_fill(~((j <= p) & ((j > p - window) if window else True)), -math.inf)
        if tail:
            sc = torch.cat([sc, sink.double()[:, None, None].expand(nq, n, 1)], -1)
        w = sc.softmax(-1)[..., : n + s]
        o = torch.einsum("htj,jhd->thd", w, v)
        if tail:
            o = o * torch.sigmoid(gate[at: at + n].double())[..., None]
        # scores of size 1 summed over hd terms, weights that sum to one: a few dozen roundings of 2^-24 of values of size 1 to 4
        assert (out[at: at + n].double() - o.reshape(n, -1)).abs().max() < 1e-5
        at += n


@pytest.mark.parametrize("window", [None, 70, 1])
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("tail", [False, True])
def test_result_does_not_depend_on_the_cutting(window, hd, tail):
    g = torch.Generator(device=DEV).manual_seed(3)
    nq, nkv, page, n = 4, 2, 16, 330
    cm, ctx, view = _setup([(n, 0)], nkv, hd, page, None, g)
    q = torch.randn(n, nq * hd, generator=g, device=DEV)
    sink = torch.linspace(-3.0, 9.0, nq, device=DEV) if tail else None
    gate = torch.randn(n, nq, generator=g, device=DEV) if tail else None

    def run(a, b, c):
        out = torch.empty(b - a, nq * hd, device=DEV)
        ops.paged_attention(q[a:b].contiguous(), out, view.k, view.v, c.positions, c.row_of_token, view.block_table, nq, nkv, hd, page, hd ** -0.5,
                            window, batch=c, sink=sink, gate=gate[a:b] if tail else None)
        return out

    whole = run(0, n, ctx)
    ends = [1, 8, 15, 41, 42, 75, 83, 150, 157, 200, 201, 208, 320, 327, n]      # portions of 1 and 7 tokens, of 8 and more
    for a, b in list(zip([0] + ends, ends)) + [(p, p + 1) for p in (256, 255, 192, 191, 128, 127, 64, 63)]:
        cm.truncate(0, a)
        cm.append([(0, b - a)])
        part = StepContext(cm, Workspace(DEV)).build([StepEntry(0, [0] * (b - a))], [a])
        assert torch.equal(run(a, b, part), whole[a:b]), (a, b)


@pytest.mark.parametrize("which", ["q", "out", "k", "v"])
def test_arrays_off_their_boundaries_take_the_general_kernel(which):
    g = torch.Generator(device=DEV).manual_seed(5)
    nq, nkv, hd, page, n = 4, 2, 64, 16, 70
    cm, ctx, view = _setup([(n, 0)], nkv, hd, page, None, g)

    def moved(name, t):                                            # the same numbers one float further on
        if name != which:
            return t
        wide = torch.empty(t.numel() + 1, device=DEV)
        return wide[1:].view(t.shape).copy_(t)

    q = torch.randn(n, nq * hd, generator=g, device=DEV)
    k, v = moved("k", view.k.contiguous()), moved("v", view.v.contiguous())
    out, general = moved("out", torch.empty(n, nq * hd, device=DEV)), torch.empty(n, nq * hd, device=DEV)
    args = (ctx.positions, ctx.row_of_token, view.block_table, nq, nkv, hd, page, hd ** -0.5, None)
    ops.paged_attention(moved("q", q), out, k, v, *args, batch=ctx)
    ops.paged_attention(q, general, view.k, view.v, *args)
    assert torch.equal(out, general)
