"""Memories with a scalar decay in chunks on the tensor cores against the recurrence in float64, beside the scan's own error: row lengths
around a chunk, short rows beside long ones, groups of heads, the column of ones, column tiles that vdim does not fill, states carried in,
decays of one, nearly zero and zero in front of slow ones."""
import pytest
import torch

from arle_b200 import ops
from arle_b200.cache import CacheManager
from arle_b200.engine import StepEntry
from arle_b200.engine.batch import StepContext, Workspace
from arle_b200.parts.base import StateNeed

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _ctx(lens, width, starts=None):
    cm = CacheManager([], [StateNeed((width,), torch.float32)], 16, 4, len(lens) + 1, 4096, torch.bfloat16, DEV)
    for i in range(len(lens)):
        cm.add_request(i)
    cm.append([(i, n) for i, n in enumerate(lens)])
    return StepContext(cm, Workspace(DEV)).build([StepEntry(i, [0] * n) for i, n in enumerate(lens)], starts or [0] * len(lens))


@pytest.mark.parametrize("dim,vdim,ones,H,G", [(64, 64, True, 4, 2), (64, 40, False, 3, 3), (128, 64, False, 8, 2), (128, 200, False, 2, 1),
                                               (128, 128, True, 2, 2), (256, 64, True, 2, 1), (256, 32, False, 3, 3), (128, 64, False, 80, 8),
                                               # tiles of 64 columns: more than 74 blocks of them
                                               (64, 64, True, 40, 8), (64, 200, False, 20, 4), (128, 128, True, 32, 32)])
@pytest.mark.parametrize("lens", [[33], [64, 5, 65], [200, 1, 32, 128]], ids=["33", "64-5-65", "200-1-32-128"])
@pytest.mark.parametrize("kind", ["slow", "wild"])
def test_against_float64(dim, vdim, ones, H, G, lens, kind):
    g = torch.Generator(device=DEV).manual_seed(dim + vdim + H + len(lens))
    T, vcols = sum(lens), vdim + int(ones)

    def rand(*s):
        return torch.randn(*s, generator=g, device=DEV)

    wide = rand(T, 2 * G * dim + H * vdim + 8).to(torch.bfloat16)
    q, k, v = wide[:, : G * dim], wide[:, G * dim: 2 * G * dim], wide[:, 2 * G * dim: 2 * G * dim + H * vdim]
    u = torch.rand(T, H, generator=g, device=DEV)
    a = (1.0 - 0.02 * u) if kind == "slow" else torch.where(u < 0.1, torch.zeros_like(u), torch.where(u < 0.3, u * 1e-30, torch.where(u < 0.5, torch.ones_like(u), 1 - 1e-4 * u)))
    b = torch.rand(T, H, generator=g, device=DEV) * 2
    ctx = _ctx(lens, H * vcols * dim + 4)
    state0 = rand(len(lens) + 1, H * vcols * dim + 4)
    state, out = state0.clone(), torch.full((T, H, vcols), 7.0, device=DEV)
    assert ops.decay_tc_takes(q, k, v, dim, vdim, ones, ctx.max_q_len)
    ops.decay_memories(q, k, v, a, b, state, ctx, out, H, G, dim, vdim, ones, 0.3)
    state1, out1 = state0.clone(), torch.empty_like(out)
    ops.decay_scan(q, k, v, a, b, state1, ctx.q_indptr, ctx.state_slots, out1, H, G, dim, vdim, ones, 0.3)
    qd, kd = (x.double().view(T, G, dim).repeat_interleave(H // G, 1) for x in (q, k))
    vd = v.double().view(T, H, vdim)
    if ones:
        vd = torch.cat([vd, vd.new_ones(T, H, 1)], -1)
    want, last, t = torch.empty(T, H, vcols, dtype=torch.float64, device=DEV), state0.double(), 0
    for r, n in enumerate(lens):
        slot = int(ctx.state_slots[r])
        S = state0[slot, : H * vcols * dim].double().view(H, vcols, dim)
        for _ in range(n):
            S = a[t].double()[:, None, None] * S + (b[t].double()[:, None] * vd[t])[..., None] * kd[t][:, None]
            want[t] = torch.einsum("hcd,hd->hc", S, qd[t] * 0.3)
            t += 1
        last[slot, : H * vcols * dim] = S.reshape(-1)
    for got, scan, ref in ((out, out1, want), (state, state1, last)):
        mine, theirs = (x.double() - ref for x in (got, scan))
        # no further from float64 than the scan by more than the order of the sums explains (both 24-bit sums of the same terms)
        assert mine.norm() <= 1.5 * theirs.norm() + 2.0 ** -22 * ref.norm()
        assert mine.abs().max() <= 4 * theirs.abs().max() + 2.0 ** -20 * ref.abs().max()


@pytest.mark.parametrize("dim,vdim,ones,H,G", [(64, 64, True, 8, 8), (128, 64, False, 40, 8), (256, 64, True, 8, 2)])
def test_a_row_does_not_depend_on_the_others(dim, vdim, ones, H, G):
    """One row alone runs tiles of 32 columns, several together tiles of 64; a short row takes the scan either way."""
    g = torch.Generator(device=DEV).manual_seed(dim)
    lens, vcols = [33, 7, 200, 1, 32, 64, 90], vdim + int(ones)
    T, width = sum(lens), H * vcols * dim
    wide = torch.randn(T, 2 * G * dim + H * vdim, generator=g, device=DEV).to(torch.bfloat16)
    a, b = 1 - 0.02 * torch.rand(T, H, generator=g, device=DEV), torch.rand(T, H, generator=g, device=DEV)
    state0 = torch.randn(len(lens) + 1, width, generator=g, device=DEV)

    def run(ctx, lo, hi, state):
        q, k, v = wide[lo:hi].split([G * dim, G * dim, H * vdim], 1)
        out = torch.empty(hi - lo, H, vcols, device=DEV)
        ops.decay_memories(q, k, v, a[lo:hi].contiguous(), b[lo:hi].contiguous(), state, ctx, out, H, G, dim, vdim, ones, 0.3)
        return out

    ctx, state = _ctx(lens, width), state0.clone()
    whole, at = run(ctx, 0, T, state), 0
    for r, n in enumerate(lens):
        one, slot = _ctx([n], width), int(ctx.state_slots[r])
        st = torch.zeros(2, width, device=DEV)
        st[int(one.state_slots[0])] = state0[slot]
        assert torch.equal(run(one, at, at + n, st), whole[at: at + n])
        assert torch.equal(st[int(one.state_slots[0])], state[slot])
        at += n
