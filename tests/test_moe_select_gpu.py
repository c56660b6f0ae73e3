"""The choice of experts where a warp has a token: ids in the order chosen, ties to the lower group and expert, one and eight experts a lane, up to 32
groups, one token a block and four; scores that are NaN."""
import numpy as np
import pytest
import torch

from arle_b200 import ops
from launched import launched

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _select(z, corr, top, groups, keep, **kw):
    T, E = z.shape
    wide = torch.full((T, E + 3), 9.0)
    wide[:, :E] = z
    ids, wts = torch.full((T + 1, top), -7, dtype=torch.int32, device=DEV), torch.full((T + 1, top), 7.0, device=DEV)
    args = (wide.to(DEV)[:, :E], None if corr is None else corr.to(DEV), torch.zeros(T, E + groups, device=DEV), E, top, groups, keep, 1.7, ids[:T], wts[:T])
    assert launched(lambda: ops.moe_select(*args, **kw), r"moe_select_\w*kernel") == {"moe_select_warp_kernel"}
    assert (ids[T] == -7).all() and (wts[T] == 7.0).all()
    return ids[:T].cpu(), wts[:T].cpu()


def _chosen(ch, top, groups, keep, two):
    """ch float32 [T, E]: the rules in float32, with sorts that keep the order of equals."""
    T, E = ch.shape
    g = -np.sort(-ch.reshape(T, groups, -1), axis=-1)
    score = g[..., 0] + g[..., 1] if two and g.shape[-1] > 1 else g[..., 0]
    kept = np.argsort(-score, axis=-1, kind="stable")[:, :keep]
    open_ = np.zeros((T, groups), dtype=bool)
    np.put_along_axis(open_, kept, True, axis=1)
    masked = np.where(np.repeat(open_, E // groups, axis=1), ch, -np.inf)
    return np.argsort(-masked, axis=-1, kind="stable")[:, :top]


@pytest.mark.parametrize("T", [1, 592, 593, 1501])
@pytest.mark.parametrize("E,top,groups,keep", [(8, 2, 8, 3), (32, 4, 4, 2), (64, 6, 32, 5), (96, 6, 8, 4), (160, 6, 8, 3), (256, 8, 8, 4), (256, 8, 32, 4), (256, 200, 32, 31),
                                               (200, 8, 1, 1)])
@pytest.mark.parametrize("group_score", ["top2_sum", "max"])
def test_order_and_ties(T, E, top, groups, keep, group_score):
    """Sums that are whole numbers decide by themselves, many of them equal: every choice and its place are the rule's."""
    g = torch.Generator().manual_seed(E + T + groups)
    z = torch.randint(-3, 4, (T, E), generator=g).float()
    ids, wts = _select(z, None, top, groups, keep, scores="softmax_chosen", group_score=group_score)
    want = torch.from_numpy(_chosen(z.numpy(), top, groups, keep, group_score == "top2_sum"))
    assert torch.equal(ids.long(), want)
    torch.testing.assert_close(wts, 1.7 * torch.softmax(z.gather(1, want), 1), rtol=1e-5, atol=0)


@pytest.mark.parametrize("T,E,top,groups,keep", [(593, 256, 8, 8, 4), (2048, 256, 8, 32, 3), (70, 160, 6, 8, 3)])
def test_scores_with_corrections(T, E, top, groups, keep):
    g = torch.Generator().manual_seed(E + T)
    z, corr = torch.randn(T, E, generator=g) * 2, torch.randn(E, generator=g) * 0.3 - 2.0
    ids, wts = _select(z, corr, top, groups, keep)
    s = torch.sigmoid(z.double())
    ch = (s + corr.double()).numpy()
    want = _chosen(ch, top, groups, keep, True)
    clear = torch.from_numpy(np.sort(want, axis=1) == np.sort(ids.numpy(), axis=1)).all(1)
    assert clear.double().mean() > 0.995                           # float32 scores may tie where float64 ones differ
    torch.testing.assert_close(wts.double(), s.gather(1, ids.long()) * 1.7, rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("E,groups,keep", [(32, 1, 1), (256, 8, 4), (64, 32, 8)])
def test_scores_that_are_nan(E, groups, keep):
    g = torch.Generator().manual_seed(E)
    z = torch.randn(9, E, generator=g)
    z[0], z[1, :3], z[2, 5::2], z[3, E - 1], z[4, ::7] = (float("nan"),) * 5
    ids, _ = _select(z, None, 6, groups, keep)
    assert ((ids >= 0) & (ids < E)).all() and all(len(set(r)) == 6 for r in ids.tolist())
    free = torch.isfinite(z).all(1)
    assert torch.equal(ids[free].long(), torch.from_numpy(_chosen(torch.sigmoid(z[free]).numpy(), 6, groups, keep, True)))
    if groups == 1:                                                # chosen last
        assert torch.isfinite(z.gather(1, ids.long()))[1:].all()
