"""The gated linear attention's scan with warps that bring the chunks (few blocks) and without (many): a row has the same bits by itself and among so
many others that the other form runs, at the edges of chunks of eight tokens and of the ring, for widths that do not fill a block; against a
chain of float64 steps."""
import pytest
import torch

from arle_b200 import ops
from launched import launched

pytestmark = pytest.mark.gpu
DEV = "cuda"


def prepared(q, k, v, alpha, state, lens, dims, bonus):
    H, d, dv = dims
    out = torch.full((sum(lens) + 1, H * dv), 7.0, device=DEV)
    cuts = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    slots = torch.arange(len(lens), dtype=torch.int32, device=DEV)
    return lambda: ops.gla_scan(q, k, v, alpha, state, cuts, slots, out[:-1], H, d, dv, d ** -0.5, max(lens), bonus), out


def scan(*args):
    run, out = prepared(*args)
    run()
    assert (out[-1] == 7.0).all()
    return out[:-1]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("with_bonus", [False, True])
@pytest.mark.parametrize("H,d,dv,n", [(2, 128, 128, 8), (1, 128, 40, 9), (2, 68, 16, 23), (2, 66, 5, 24), (1, 128, 128, 25), (2, 100, 33, 31), (2, 128, 20, 64), (1, 128, 16, 200)])
def test_with_and_without_loaders(dtype, with_bonus, H, d, dv, n):
    g = torch.Generator(device=DEV).manual_seed(n + d)
    blocks = H * -(-dv // 16)
    rows = 296 // blocks + 1
    lens = [n] + [8] * (rows - 1)
    T = sum(lens)
    wide = torch.randn(T, H * (2 * d + dv), generator=g, device=DEV).to(dtype)
    q, k, v = wide[:, : H * d], wide[:, H * d: 2 * H * d], wide[:, 2 * H * d:]
    alpha = torch.sigmoid(torch.randn(T, H * d, generator=g, device=DEV)).pow(1 / 16).contiguous()
    bonus = torch.randn(H * d, generator=g, device=DEV) if with_bonus else None
    state = torch.randn(rows, H, dv, d, generator=g, device=DEV)
    many, one = state.clone(), state[:1].clone()
    a = scan(q, k, v, alpha, many, lens, (H, d, dv), bonus)[:n]
    ran = launched(prepared(q[:n], k[:n], v[:n], alpha[:n], one.clone(), [n], (H, d, dv), bonus)[0], r"gla_scan_kernel<.*?>(?=\()")
    assert len(ran) == 1 and ran.pop().endswith("true, true>")
    b = scan(q[:n], k[:n], v[:n], alpha[:n], one, [n], (H, d, dv), bonus)
    assert torch.equal(a, b) and torch.equal(many[:1], one)
    S = state[0].double()
    for t in range(n):
        kt, vt, qt, at = (x[t].double().view(H, -1) for x in (k, v, q, alpha))
        new = S * at[:, None] + vt[..., None] * kt[:, None]
        seen = S + vt[..., None] * (kt * bonus.double().view(H, d))[:, None] if with_bonus else new
        want, size = torch.einsum("hvd,hd->hv", seen, qt) * d ** -0.5, torch.einsum("hvd,hd->hv", seen.abs(), qt.abs()) * d ** -0.5
        # a number of the memory has been rounded t times at most, twice a step; the sum over d
        assert ((b[t].double().view(H, dv) - want).abs() <= (2 * t + d + 8) * 2.0 ** -24 * size + 1e-6).all()
        S = new
    assert (one[0].double() - S).abs().max() <= 1e-4


def test_no_tokens_and_few():
    g = torch.Generator(device=DEV).manual_seed(1)
    H, d, lens = 2, 128, [0, 12, 0, 3]
    wide, alpha = torch.randn(15, 3 * H * d, generator=g, device=DEV), torch.rand(15, H * d, generator=g, device=DEV)
    state = torch.randn(4, H, d, d, generator=g, device=DEV)
    got, parts = state.clone(), state.clone()
    out = scan(wide[:, : H * d], wide[:, H * d: 2 * H * d], wide[:, 2 * H * d:], alpha, got, lens, (H, d, d), None)
    assert torch.equal(got[0], state[0]) and torch.equal(got[2], state[2])
    for r, at, n in ((1, 0, 12), (3, 12, 3)):
        x, one = wide[at: at + n], parts[r: r + 1].clone()
        alone = scan(x[:, : H * d], x[:, H * d: 2 * H * d], x[:, 2 * H * d:], alpha[at: at + n].contiguous(), one, [n], (H, d, d), None)
        assert torch.equal(alone, out[at: at + n]) and torch.equal(one[0], got[r])
