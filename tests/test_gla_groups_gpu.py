"""The gated linear attention's scan in groups of eight tokens: a token's bits do not depend on whether it runs in a group or by itself, at row
lengths around a group and a chunk; against float64 for sizes that do and do not fill the lanes, with and without a bonus."""
import pytest
import torch

from arle_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _run(q, k, v, alpha, state, lens, heads, dim, vdim, bonus):
    at = torch.tensor([0] + lens, dtype=torch.int32, device=DEV).cumsum(0).to(torch.int32)
    out = torch.full((q.shape[0], heads * vdim), 7.0, device=DEV)
    ops.gla_scan(q, k, v, alpha, state, at, torch.arange(len(lens), dtype=torch.int32, device=DEV), out, heads, dim, vdim, 0.25, max(lens), bonus=bonus)
    return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dim,vdim", [(128, 128), (100, 36), (256, 20), (68, 64), (16, 24), (4, 520)])
@pytest.mark.parametrize("bonus", [False, True])
def test_groups_of_tokens(dtype, dim, vdim, bonus):
    g = torch.Generator(device=DEV).manual_seed(dim + vdim)
    heads, lens = 2, [7, 8, 9, 16, 17, 40, 1]
    T = sum(lens)
    wide = torch.randn(T, heads * (2 * dim + vdim), generator=g, device=DEV).to(dtype)
    q, k, v = wide.split([heads * dim, heads * dim, heads * vdim], 1)
    alpha = torch.rand(T, heads * dim, generator=g, device=DEV) * 0.2 + 0.8
    u = torch.rand(heads * dim, generator=g, device=DEV) if bonus else None
    state0 = torch.randn(len(lens), heads, vdim, dim, generator=g, device=DEV)
    state = state0.clone()
    out = _run(q, k, v, alpha, state, lens, heads, dim, vdim, u)
    one, t = state0.clone(), 0
    for r, n in enumerate(lens):                                # the same, one token a call
        for _ in range(n):
            s = one[r: r + 1].contiguous()
            o = _run(q[t: t + 1], k[t: t + 1], v[t: t + 1], alpha[t: t + 1], s, [1], heads, dim, vdim, u)
            one[r] = s[0]
            assert torch.equal(o[0], out[t])
            t += 1
    assert torch.equal(one, state)
    S, t = state0.double(), 0
    for r, n in enumerate(lens):
        for _ in range(n):
            kk, vv, aa, qq = (x[t].double().view(heads, -1) for x in (k, v, alpha, q))
            kv = vv[..., None] * kk[:, None]
            read = S[r] + u.double().view(heads, 1, dim) * kv if bonus else S[r] * aa[:, None] + kv
            S[r] = S[r] * aa[:, None] + kv
            want = torch.einsum("hvd,hd->hv", read, qq * 0.25).reshape(-1)
            # dim products of sums of a few dozen terms: float32 roundings of numbers of size 10
            assert (out[t].double() - want).abs().max() < 1e-5 * max(1.0, want.abs().max().item()) * dim ** 0.5
            t += 1
