"""Memories with a scalar decay and 128 keys: the scores of all chunks formed side by side and the chain behind them give the bits of the one launch
that does both, for rows around a chunk's end, short rows beside long ones, heads in fours and by themselves, columns that do not fill a block, one
group of columns a block and four, and decays of zero; with values that overflow the same to the last bits."""
import pytest
import torch

from arle_b200 import ops
from launched import launched
from test_decay_tc_gpu import DEV, _ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,vdim", [(8, 2, 64), (3, 3, 40), (2, 1, 200), (80, 8, 64)])
@pytest.mark.parametrize("lens", [[192], [257], [300, 1, 33, 128, 20]], ids=["192", "257", "300-1-33-128-20"])
@pytest.mark.parametrize("kind", ["slow", "wild", "odd"])
def test_the_bits_of_the_one_launch(monkeypatch, H, G, vdim, lens, kind):
    g = torch.Generator(device=DEV).manual_seed(H + vdim + len(lens))
    T, dim = sum(lens), 128
    wide = torch.randn(T, 2 * G * dim + H * vdim + 8, generator=g, device=DEV).to(torch.bfloat16)
    q, k, v = wide[:, : G * dim], wide[:, G * dim: 2 * G * dim], wide[:, 2 * G * dim: 2 * G * dim + H * vdim]
    u, b = (torch.rand(T, H, generator=g, device=DEV) for _ in range(2))
    a = 1.0 - 0.05 * u if kind == "slow" else torch.where(u < 0.1, torch.zeros_like(u), torch.where(u < 0.3, u * 1e-30, 1 - 1e-3 * u))
    if kind == "odd":
        v[T // 2, 1], v[T // 3, vdim // 2] = float("inf"), float("nan")
    ctx, width = _ctx(lens, H * vdim * dim + 4), H * vdim * dim + 4
    state0 = torch.randn(len(lens) + 1, width, generator=g, device=DEV)
    assert ops.decay_rows_chunks(ctx, dim, False) > 0 and ops.decay_rows_chunks(ctx, dim, True) == 0
    got = []
    for split in (True, False):
        if not split:
            monkeypatch.setattr(ops, "decay_rows_chunks", lambda *_: 0)
        state, out = state0.clone(), torch.full((T + 1, H, vdim), 7.0, device=DEV)
        ops.decay_memories(q, k, v, a, b, state, ctx, out[:T], H, G, dim, vdim, False, 0.3)
        got.append((out, state))
    for x, y in zip(*got):
        if kind == "odd":                               # a warp that meets such a value adds a tile up one by one, for 16 columns here and 32 there
            torch.testing.assert_close(x, y, rtol=1e-5, atol=1e-5, equal_nan=True)
        else:
            assert torch.equal(x, y)
    assert (got[0][0][T] == 7.0).all()


@pytest.mark.parametrize("H,n", [(32, 2048), (8, 192)])
def test_the_chain_goes_by_the_rows_that_it_runs(H, n):
    """A long row beside decoded tokens takes the chain's kernel that it takes by itself (as many groups of columns a block)."""
    dim, vdim, names = 128, 64, []
    for lens in ([n], [n] + [1] * 40):
        T = sum(lens)
        q, k, v = (torch.zeros(T, w, device=DEV, dtype=torch.bfloat16) for w in (dim, dim, H * vdim))
        a, b = (torch.ones(T, H, device=DEV) for _ in range(2))
        ctx, state, out = _ctx(lens, H * vdim * dim), torch.zeros(len(lens) + 1, H * vdim * dim, device=DEV), torch.empty(T, H, vdim, device=DEV)
        names.append(launched(lambda: ops.decay_memories(q, k, v, a, b, state, ctx, out, H, 1, dim, vdim, False, 1.0), r"decay_rows_tc_kernel<\d+>"))
    assert len(names[0]) == 1 and names[0] == names[1]


@pytest.mark.parametrize("H,G,vdim", [(128, 8, 40), (24, 6, 200)])      # four groups of columns a block: one block part full, and a last one with one group
@pytest.mark.parametrize("lens", [[256], [300, 1, 33, 128, 20]], ids=["256", "300-1-33-128-20"])
def test_four_groups_with_columns_left_over(monkeypatch, H, G, vdim, lens):
    test_the_bits_of_the_one_launch(monkeypatch, H, G, vdim, lens, "wild")


@pytest.mark.parametrize("H,lens,split", [(32, [192], True), (64, [192], False), (64, [256], True), (32, [192] * 3, False), (32, [200] * 12, True),
                                          (8, [192] + [1] * 60, True), (128, [191, 257], True)])
def test_which_steps_are_split(H, lens, split):
    """Four chunks and more always; three while every group of columns of the rows that run finds an SM, and once blocks of four groups don't."""
    dim, vdim, T = 128, 64, sum(lens)
    q, k, v = (torch.zeros(T, w, device=DEV, dtype=torch.bfloat16) for w in (dim, dim, H * vdim))
    a, b = (torch.ones(T, H, device=DEV) for _ in range(2))
    ctx, state, out = _ctx(lens, H * vdim * dim), torch.zeros(len(lens) + 1, H * vdim * dim, device=DEV), torch.empty(T, H, vdim, device=DEV)
    ran = launched(lambda: ops.decay_memories(q, k, v, a, b, state, ctx, out, H, 1, dim, vdim, False, 1.0), r"decay\w*_tc_kernel")
    assert ran == {"decay_rows_tc_kernel" if split else "decay_tc_kernel"}
