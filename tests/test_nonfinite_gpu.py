"""An infinity or a NaN stays with the tokens that see it: tokens in front of it, tokens whose window has passed it and other requests of the
step get what they get without it.  (In the kernels on tiles a masked place is a weight of zero, and zero times infinity is not zero.)"""
import math

import pytest
import torch

from arle_b200 import ops
from arle_b200.cache import CacheManager
from arle_b200.engine import StepEntry
from arle_b200.engine.batch import StepContext, Workspace
from arle_b200.parts.base import CacheNeed, StateNeed

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF = torch.bfloat16
INF = math.inf


def _step(need, lens, dtype, page=16):
    state = isinstance(need, StateNeed)
    cm = CacheManager([] if state else [need], [need] if state else [], page, sum(-(-n // page) for n in lens) + 2, len(lens) + 1, 4096, dtype, DEV)
    for i in range(len(lens)):
        cm.add_request(i)
    cm.append([(i, n) for i, n in enumerate(lens)])
    ctx = StepContext(cm, Workspace(DEV)).build([StepEntry(i, [0] * n) for i, n in enumerate(lens)], [0] * len(lens))
    return cm, ctx


def _slots(cm, lens):
    return [torch.from_numpy(cm.slot_mapping(0, i, 0, n)).long().to(DEV) for i, n in enumerate(lens)]


@pytest.mark.parametrize("dn,dr,rank", [(128, 64, 512), (64, 32, 256), (128, 0, 128), (64, 0, 64)])
@pytest.mark.parametrize("window", [None, 64])
def test_latent_prefill(dn, dr, rank, window):
    heads, kd, lens = 40, rank + dr, [300, 200, 270, 70]          # 320 blocks: a CTA runs several requests' blocks
    g = torch.Generator(device=DEV).manual_seed(dn + dr)
    cm, ctx = _step(CacheNeed(streams=((1, kd),), window=window), lens, BF)
    cm.groups[0].arrays[0].normal_(generator=g)
    view, slots, T = ctx.cache_view(0), _slots(cm, lens), sum(lens)
    q = torch.empty(T, heads * (dn + dr), device=DEV, dtype=BF).normal_(generator=g)
    w = torch.empty(2 * heads * dn, rank, device=DEV, dtype=BF).normal_(0.0, rank ** -0.5, generator=g)
    places = ops.latent_built_places(ctx, q, dn, dr, dn, rank, 16, window)

    def run():
        out = torch.empty(T, heads * dn, device=DEV, dtype=BF)
        ops.latent_prefill(q, out, view.streams[0], ctx, view.block_table, w, heads, places, dr, rank, 16, (dn + dr) ** -0.5, window)
        return out

    clean = run()
    flat = view.streams[0].view(-1, kd)
    flat[slots[0][2:], 3] = INF                                    # all but two tokens of the first request
    flat[slots[1][100], rank - 1] = math.nan
    flat[slots[2][150], 0] = -INF
    hit = torch.zeros(T, dtype=torch.bool, device=DEV)
    reach = window or T
    hit[2: 300] = True
    hit[300 + 100: min(300 + 100 + reach, 500)] = True
    hit[500 + 150: min(500 + 150 + reach, 770)] = True
    out = run()
    assert torch.equal(out[~hit], clean[~hit])
    assert out[hit].isnan().all()
    ops.check_errors(DEV)


@pytest.mark.parametrize("window", [None, 32])
def test_prefill_attention_of_another_request(window):
    nq, nkv, hd, lens = 32, 8, 128, [600, 600, 600, 70, 300, 33]
    g = torch.Generator(device=DEV).manual_seed(1)
    cm, ctx = _step(CacheNeed(nkv, hd, window), lens, BF)
    for a in cm.groups[0].arrays:
        a.normal_(generator=g)
    view, slots, T = ctx.cache_view(0), _slots(cm, lens), sum(lens)
    q = torch.empty(T, nq * hd, device=DEV, dtype=BF).normal_(generator=g)

    def run():
        out = torch.empty(T, nq * hd, device=DEV, dtype=BF)
        ops.paged_attention(q, out, view.k, view.v, ctx.positions, ctx.row_of_token, view.block_table, nq, nkv, hd, 16, hd ** -0.5, window, batch=ctx)
        return out

    clean = run()
    for s in slots[:3]:
        view.v[s // 16, :, s % 16] = INF
    out = run()
    assert torch.equal(out[1800:], clean[1800:])
    ops.check_errors(DEV)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("window", [None, 40])
@pytest.mark.parametrize("lens", [[150, 8], [40, 3, 100]], ids=["150-8", "40-3-100"])
def test_float32_attention(hd, window, lens):
    nq, nkv = 4, 2
    g = torch.Generator(device=DEV).manual_seed(hd)
    cm, ctx = _step(CacheNeed(nkv, hd, window), lens, torch.float32)
    for a in cm.groups[0].arrays:
        a.normal_(generator=g)
    view, slots, T = ctx.cache_view(0), _slots(cm, lens), sum(lens)
    q = torch.randn(T, nq * hd, generator=g, device=DEV)

    def run(batch):
        out = torch.empty(T, nq * hd, device=DEV)
        ops.paged_attention(q, out, view.k, view.v, ctx.positions, ctx.row_of_token, view.block_table, nq, nkv, hd, 16, hd ** -0.5, window, batch=batch)
        return out

    clean = run(ctx)
    s = slots[0][[20, 37]]
    view.v[s[0] // 16, 0, s[0] % 16, 5] = INF
    view.v[s[1] // 16, 1, s[1] % 16, 7] = math.nan
    view.k[s[1] // 16, 1, s[1] % 16, 9] = math.nan
    out, general = run(ctx), run(None)                             # the general kernel takes a token at a time
    assert torch.equal(out.isfinite(), general.isfinite())
    hit = torch.zeros(T, dtype=torch.bool, device=DEV)
    hit[20: min(lens[0], 37 + window if window else T)] = True
    assert torch.equal(out[~hit], clean[~hit]) and not out[hit].isfinite().all()
    same = out.isfinite() & hit[:, None]
    assert torch.equal(out[same], clean[same])


@pytest.mark.parametrize("dim,vdim,ones", [(64, 64, True), (128, 64, False), (256, 32, False)])
def test_decay_memories(dim, vdim, ones):
    H, G, lens, vcols = 4, 2, [130, 70], vdim + int(ones)
    T = sum(lens)
    g = torch.Generator(device=DEV).manual_seed(dim)
    _, ctx = _step(StateNeed((H * vcols * dim,), torch.float32), lens, BF)
    wide = torch.empty(T, 2 * G * dim + H * vdim, device=DEV, dtype=BF).normal_(generator=g)
    q, k, v = wide.split([G * dim, G * dim, H * vdim], 1)
    a = 1 - 0.05 * torch.rand(T, H, generator=g, device=DEV)
    b = torch.rand(T, H, generator=g, device=DEV)
    state0 = torch.randn(3, H * vcols * dim, generator=g, device=DEV)

    def run(fn):
        st, out = state0.clone(), torch.empty(T, H, vcols, device=DEV)
        if fn is ops.decay_scan:
            fn(q, k, v, a, b, st, ctx.q_indptr, ctx.state_slots, out, H, G, dim, vdim, ones, 0.3)
        else:
            fn(q, k, v, a, b, st, ctx, out, H, G, dim, vdim, ones, 0.3)
        return out, st

    clean, _ = run(ops.decay_memories)
    v[70 + 9, 3] = INF                                             # head 0, column 3: inside a tile of 16 tokens
    k[100, dim] = -INF                                             # the second group's heads, every column
    a[71, 1] = math.nan                                            # head 1, the second token of a pair
    b[64, 0] = INF
    (out, st), (scan, scan_st) = run(ops.decay_memories), run(ops.decay_scan)
    assert torch.equal(out.isfinite(), scan.isfinite())
    assert torch.equal(st.isfinite(), scan_st.isfinite())
    ok = out.isfinite()
    assert torch.equal(out[:64], clean[:64])
    assert (out[ok] - scan[ok]).norm() <= 1e-5 * scan[ok].norm()


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("page", [16, 32])
@pytest.mark.parametrize("window", [None, 40])
@pytest.mark.parametrize("rows", [[(1, 70), (1, 300), (1, 0), (1, 31)], [(1, 517)]], ids=["four", "one"])
def test_decoded_tokens_do_not_see_other_slots_of_a_page(hd, page, window, rows):
    """What a page's former owner left behind the last token, and what lies in front of the window."""
    _other_slots(hd, page, window, rows, window)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("page,window", [(16, None), (32, 40), (64, 300)])
@pytest.mark.parametrize("rows", [[(70, 0), (300, 5), (33, 0), (256, 0)], [(1, 70), (45, 3), (16, 0), (2, 126)], [(513, 130)]], ids=["rows", "mixed", "one"])
@pytest.mark.parametrize("form", ["softmax", "cap", "kept", "sigmoid"])
def test_prompts_do_not_see_other_slots_of_a_page(hd, page, window, rows, form):
    """What a page's former owner left behind the last token."""
    if form == "kept" and not window:
        return
    extra = {"softmax": {}, "cap": {"softcap": 20.0}, "kept": {"keep_first": 5},
             "sigmoid": {"score_bias": torch.zeros(8, device=DEV)}}[form]
    _other_slots(hd, page, window, rows, None, **extra)


def _other_slots(hd, page, window, rows, held, **extra):
    """held: the last keys of a request that hold numbers (None: all)."""
    nq, nkv, kvs = 8, 2, [n + s for n, s in rows]
    cm = CacheManager([CacheNeed(nkv, hd, window, keep_first=extra.get("keep_first", 0))], [], page, sum(-(-k // page) for k in kvs) + 2, len(rows), max(kvs),
                      BF, DEV)
    for i, (n, s) in enumerate(rows):
        cm.add_request(i)
        if s:
            cm.append([(i, s)])
    cm.append([(i, n) for i, (n, _) in enumerate(rows)])
    ctx = StepContext(cm, Workspace(DEV)).build([StepEntry(i, [0] * n) for i, (n, _) in enumerate(rows)], [s for _, s in rows])
    T = sum(n for n, _ in rows)
    view, g = ctx.cache_view(0), torch.Generator(device=DEV).manual_seed(2)
    q = torch.empty(T, nq * hd, device=DEV, dtype=BF).normal_(generator=g)
    new = [[torch.empty(k, nkv, hd, device=DEV, dtype=BF).normal_(generator=g) for _ in range(2)] for k in kvs]
    outs = []
    for fill in (0.0, INF, math.nan):
        for a, which in ((view.k, 0), (view.v, 1)):
            a.fill_(fill)
            for i, k in enumerate(kvs):
                first = max(0, k - held) if held else 0
                s = torch.from_numpy(cm.slot_mapping(0, i, 0, k)).long().to(DEV)[first:]
                a.permute(0, 2, 1, 3)[s // page, s % page] = new[i][which][first:]
        outs.append(torch.empty(T, nq * hd, device=DEV, dtype=BF))
        ops.paged_attention(q, outs[-1], view.k, view.v, ctx.positions, ctx.row_of_token, view.block_table, nq, nkv, hd, page, hd ** -0.5, window,
                            batch=ctx, **extra)
    assert outs[0].isfinite().all() and torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    ops.check_errors(DEV)
