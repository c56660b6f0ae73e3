"""Gated linear attention over rows cut into segments against float64: lengths around the first that is cut and around a segment's end, one
and several cut rows beside short ones, sizes that do not fill the lanes or a block's columns; no further off than the scan of whole rows;
a row's bits do not depend on what stands beside it, and an overflow stays with the tokens behind it."""
import pytest
import torch

from arle_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(lens, heads, dim, vdim, low=0.9):
    g = torch.Generator(device=DEV).manual_seed(dim + vdim + sum(lens))
    T = sum(lens)
    wide = torch.randn(T, heads * (2 * dim + vdim), generator=g, device=DEV).to(torch.bfloat16)
    alpha = torch.rand(T, heads * dim, generator=g, device=DEV) * (1 - low) + low
    return (*wide.split([heads * dim, heads * dim, heads * vdim], 1), alpha, torch.randn(len(lens) + 1, heads, vdim, dim, generator=g, device=DEV))


def _run(q, k, v, alpha, state, lens, heads, dim, vdim, cut=True, slots=None):
    at = torch.tensor([0] + lens, dtype=torch.int32, device=DEV).cumsum(0).to(torch.int32)
    out = torch.full((q.shape[0] + 1, heads * vdim), 7.0, device=DEV)
    state, n = state.clone(), ops.gla_scan_scratch(q, k, alpha, len(lens), heads, dim, vdim, max(lens)) if cut else 0
    assert not cut or n > 0
    scratch = torch.full((n + 4,), float("nan"), device=DEV) if n else None
    slots = torch.tensor(slots or list(range(len(lens))), dtype=torch.int32, device=DEV)
    ops.gla_scan(q, k, v, alpha, state, at, slots, out[:-1], heads, dim, vdim, 0.25, max(lens), scratch=scratch[:n] if n else None)
    assert (out[-1] == 7.0).all() and (scratch is None or scratch[n:].isnan().all())
    return out[:-1], state


def _exact(q, k, v, alpha, state, lens, heads, dim, vdim):
    S, outs, t = state.double().clone(), [], 0
    for r, n in enumerate(lens):
        for _ in range(n):
            kk, vv, aa, qq = (x[t].double().view(heads, -1) for x in (k, v, alpha, q))
            S[r] = S[r] * aa[:, None] + vv[..., None] * kk[:, None]
            outs.append(torch.einsum("hvd,hd->hv", S[r], qq * 0.25).reshape(-1))
            t += 1
    return torch.stack(outs), S


@pytest.mark.parametrize("lens", [[384], [511], [2049], [5, 400, 1, 900, 383, 640], [1] * 40 + [513]])
@pytest.mark.parametrize("heads,dim,vdim", [(2, 128, 128), (3, 100, 36), (1, 68, 200)])
def test_segments(lens, heads, dim, vdim):
    q, k, v, alpha, state = _inputs(lens, heads, dim, vdim)
    want, want_s = _exact(q, k, v, alpha, state, lens, heads, dim, vdim)
    got, got_s = _run(q, k, v, alpha, state, lens, heads, dim, vdim)
    whole, whole_s = _run(q, k, v, alpha, state, lens, heads, dim, vdim, cut=False)
    for a, b, w in ((got, whole, want), (got_s, whole_s, want_s)):
        off, ref = ((x.double() - w).norm() / w.norm() for x in (a, b))
        assert off < 3e-7 and off < 1.2 * ref + 2e-8           # the float32 sums of both come in different orders
    t = 0
    for r, n in enumerate(lens):                                # a row by itself: the same bits
        if n < 384:
            assert torch.equal(got[t: t + n], whole[t: t + n])
        else:
            alone, s = _run(q[t: t + n], k[t: t + n], v[t: t + n], alpha[t: t + n], state, [n], heads, dim, vdim, slots=[r])
            assert torch.equal(alone, got[t: t + n]) and torch.equal(s[r], got_s[r])
        t += n


def test_strong_decays_and_overflow():
    lens, heads, dim, vdim = [600], 2, 128, 64
    q, k, v, alpha, state = _inputs(lens, heads, dim, vdim)
    alpha[::7] = 0.0
    alpha[3::11, 5] = 1e-30
    want, want_s = _exact(q, k, v, alpha, state, lens, heads, dim, vdim)
    got, got_s = _run(q, k, v, alpha, state, lens, heads, dim, vdim)
    assert (got.double() - want).norm() < 3e-7 * want.norm() and (got_s[0].double() - want_s[0]).norm() < 3e-7 * want_s[0].norm()
    v[200] = float("inf")
    odd, _ = _run(q, k, v, alpha, state, lens, heads, dim, vdim)
    assert torch.equal(odd[:200], got[:200]) and not odd[200:].isfinite().all()
