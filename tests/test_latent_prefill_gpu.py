"""Latent attention with built keys and values (``ops.latent_prefill``) against float64, at the sizes where it can go wrong: rows just below
and at the least length, portions behind a context, windows shorter and longer than a key tile, every combination of slices, all heads at a
time and some, and rows that it leaves alone."""
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
BF = torch.bfloat16


def _reference(q, rec, w_uk, w_uv, lens, kvs, rank, scale, window, gate):
    """q [T, H, dn + dr], rec: one [kv, rank + dr] per row; float64, keys and values in full precision."""
    H, dn = w_uk.shape[:2]
    outs, at = [], 0
    for n, kv, r in zip(lens, kvs, rec):
        c = r[:, :rank].double()
        k = torch.einsum("jr,hdr->jhd", c, w_uk.double())
        v = torch.einsum("jr,hdr->jhd", c, w_uv.double())
        k = torch.cat([k, r[:, None, rank:].double().expand(kv, H, r.shape[1] - rank)], -1)
        s = torch.einsum("thd,jhd->htj", q[at: at + n].double(), k) * scale
        p = torch.arange(kv - n, kv, device=DEV)[:, None]
        j = torch.arange(kv, device=DEV)[None]
        seen = (j <= p) & ((j > p - window) if window else True)
        o = torch.einsum("htj,jhd->thd", s.masked_fill(~seen, -math.inf).softmax(-1), v).reshape(n, H * dn)
        outs.append(o * torch.sigmoid(gate[at: at + n].double()) if gate is not None else o)
        at += n
    return torch.cat(outs)


@pytest.mark.parametrize("dn,dr,rank,heads", [(128, 64, 512, 3), (64, 32, 256, 2), (128, 0, 128, 2), (64, 0, 64, 5), (128, 8, 96, 1)])
@pytest.mark.parametrize("rows,window", [([(64, 0)], None), ([(300, 0), (1, 40), (63, 9), (129, 77)], None), ([(257, 300), (513, 0)], 100),
                                          ([(200, 60), (64, 16)], 1), ([(640, 0), (3, 500)], 256)],
                         ids=["least", "mixed", "portions", "window1", "window256"])
def test_against_float64(dn, dr, rank, heads, rows, window, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(dn + dr + rank + len(rows))
    kd, lens, starts = rank + dr, [n for n, _ in rows], [s for _, s in rows]
    kvs = [n + s for n, s in rows]
    T = sum(lens)

    def rand(*shape, std=1.0):
        return torch.empty(shape, device=DEV, dtype=BF).normal_(0.0, std, generator=g)

    cm = CacheManager([CacheNeed(streams=((1, kd),), window=window)], [], 16, sum(-(-k // 16) for k in kvs) + 3, len(rows), max(kvs), BF, DEV)
    for i in range(len(rows)):
        cm.add_request(i)
    for i, s in enumerate(starts):                                 # the requests' pages alternate
        if s > 32:
            cm.append([(i, 17)])
    for i, s in enumerate(starts):
        if s - (17 if s > 32 else 0):
            cm.append([(i, s - (17 if s > 32 else 0))])
    cm.append([(i, n) for i, n in enumerate(lens)])
    cm.groups[0].arrays[0].normal_(generator=g)
    ctx = StepContext(cm, Workspace(DEV)).build([StepEntry(i, [0] * n) for i, n in enumerate(lens)], starts)
    view = ctx.cache_view(0)
    flat = view.streams[0].reshape(-1, kd)
    rec = [flat[torch.from_numpy(cm.slot_mapping(0, i, 0, k)).long().to(DEV)] for i, k in enumerate(kvs)]
    wide = rand(T, heads * (dn + dr) + 24)
    q = wide[:, : heads * (dn + dr)]
    w_uk, w_uv = rand(heads, dn, rank, std=rank ** -0.5), rand(heads, dn, rank, std=rank ** -0.5)
    w_ukv = torch.cat([w_uk.reshape(heads * dn, rank), w_uv.reshape(heads * dn, rank)])
    scale = (dn + dr) ** -0.5
    places = ops.latent_built_places(ctx, q, dn, dr, dn, rank, 16, window)
    assert places > 0
    for gate, numbers in ((None, 1 << 25), (rand(T, heads * dn), 1)):         # all heads at a time, and as few as the tokens give room for
        monkeypatch.setattr(ops, "LATENT_BUILT_NUMBERS", numbers)
        want = _reference(q.unflatten(1, (heads, dn + dr)), rec, w_uk, w_uv, lens, kvs, rank, scale, window, gate)
        out = torch.full((T, heads * dn), 7.0, device=DEV, dtype=BF)
        ctx.memo.clear()
        ops.latent_prefill(q, out, view.streams[0], ctx, view.block_table, w_ukv, heads, places, dr, rank, 16, scale, window, gate=gate)
        at = 0
        for n in lens:
            got, ref = out[at: at + n].double(), want[at: at + n]
            if n < ops.LATENT_BUILT_LEAST:
                assert (got == 7.0).all()
            else:
                # keys, values, probabilities and the result are rounded to 8 bits: errors of 2^-9 each, relative to unit scores' weights
                # and to the values (of size about 1); a wrong key or page is an error of order 1
                assert ((got - ref).norm() / ref.norm()) < 4 * 2.0 ** -8
                assert (got - ref).abs().max() < 0.1
            at += n
    ops.check_errors(DEV)


@pytest.mark.parametrize("rank,dr", [(96, 16), (128, 8), (128, 32)])
def test_the_folded_form_leaves_long_rows_alone(rank, dr):
    """On the general kernel (a rank of 96, eight rotated numbers) as on the tensor cores."""
    heads, kd, lens = 4, rank + dr, [70, 5, 64, 63]
    cm = CacheManager([CacheNeed(streams=((1, kd),))], [], 16, 20, len(lens), 80, BF, DEV)
    for i in range(len(lens)):
        cm.add_request(i)
    cm.append([(i, n) for i, n in enumerate(lens)])
    ctx = StepContext(cm, Workspace(DEV)).build([StepEntry(i, [0] * n) for i, n in enumerate(lens)], [0] * len(lens))
    view, T = ctx.cache_view(0), sum(lens)
    view.streams[0].normal_()
    q = torch.randn(T, heads, kd, device=DEV).to(BF)
    want, out = torch.empty(T, heads, rank, device=DEV, dtype=BF), torch.full((T, heads, rank), 7.0, device=DEV, dtype=BF)
    args = (view.streams[0], ctx.positions, ctx.row_of_token, view.block_table, rank, 16, kd ** -0.5, None)
    ops.latent_attention(q, want, *args, batch=ctx)
    ops.latent_attention(q, out, *args, batch=ctx, but_built=True)
    at = 0
    for n in lens:
        assert n >= 64 or torch.equal(out[at: at + n], want[at: at + n])
        if n >= 64 and not ops.latent_mma_supported(q, rank):
            assert (out[at: at + n] == 7.0).all()
        at += n


def test_a_row_is_built_by_its_own_lengths(monkeypatch):
    """Rows whose records do not fit beside one another are built in groups, a row whose context is long beside its queries stays folded, and
    neither shows in the other rows' numbers."""
    monkeypatch.setattr(ops, "LATENT_BUILT_PLACES", 400)
    monkeypatch.setattr(ops, "LATENT_BUILT_MOST", 1)
    dn, dr, rank, heads = 64, 32, 128, 3
    kd, rows = rank + dr, [(64, 300), (70, 340), (5, 20), (64, 420), (130, 0), (64, 16), (200, 0), (64, 330)]
    lens, kvs = [n for n, _ in rows], [n + s for n, s in rows]
    g = torch.Generator(device=DEV).manual_seed(2)
    cm = CacheManager([CacheNeed(streams=((1, kd),))], [], 16, sum(-(-k // 16) for k in kvs) + 3, len(rows), max(kvs), BF, DEV)
    for i, (_, s) in enumerate(rows):
        cm.add_request(i)
        if s:
            cm.append([(i, s)])
    cm.append([(i, n) for i, n in enumerate(lens)])
    cm.groups[0].arrays[0].normal_(generator=g)
    T = sum(lens)
    q = torch.empty(T, heads * (dn + dr), device=DEV, dtype=BF).normal_(generator=g)
    w = torch.empty(2 * heads * dn, rank, device=DEV, dtype=BF).normal_(0.0, rank ** -0.5, generator=g)

    def run(idx, lo, hi):
        ctx = StepContext(cm, Workspace(DEV)).build([StepEntry(i, [0] * lens[i]) for i in idx], [rows[i][1] for i in idx])
        view, out = ctx.cache_view(0), torch.full((hi - lo, heads * dn), 7.0, device=DEV, dtype=BF)
        places = ops.latent_built_places(ctx, q[lo:hi], dn, dr, dn, rank, 16, None)
        if places:
            ops.latent_prefill(q[lo:hi], out, view.streams[0], ctx, view.block_table, w, heads, places, dr, rank, 16, kd ** -0.5, None)
        return ctx, out

    ctx, whole = run(range(len(rows)), 0, T)
    groups, folded = ops._latent_groups(ctx, None)
    plan = ops._latent_plan(ctx, None).tolist()
    assert len(groups) >= 2 and folded == 3                          # 5 queries; contexts of 410 and 484 behind 70 and 64 queries
    at = 0
    for i, n in enumerate(lens):
        _, one = run([i], at, at + n)
        # the product that builds keys and values may take another order of sums for another number of records: bfloat16 roundings apart
        assert (one.double() - whole[at: at + n].double()).norm() <= 2.0 ** -7 * one.double().norm()
        assert (plan[i][1] < 0) == bool((one == 7.0).all()) == (i in (1, 2, 3))
        at += n
    ops.check_errors(DEV)
