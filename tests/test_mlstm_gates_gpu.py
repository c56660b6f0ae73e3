"""The matrix LSTM's gates at the edges of their chunks of 128 tokens and groups of four: against a chain of maxima in float64, the rows beside one
another and cut into portions with the same bits; an infinite gate stays with the tokens behind it."""
import pytest
import torch

from arle_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def gates(pre, lens, state, H):
    T, R = pre.shape[0], len(lens)
    outs = [torch.full((T + 1, H), 7.0, device=DEV) for _ in range(3)]
    ops.mlstm_gates(pre, BI[:H], BF[:H], 10.0, torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV),
                    torch.arange(R, dtype=torch.int32, device=DEV), state, 4, *(o[:T] for o in outs))
    assert all((o[T] == 7.0).all() for o in outs)
    return torch.stack([o[:T] for o in outs])


BI, BF = torch.linspace(-1, 1, 8, device="cpu"), torch.linspace(0, 6, 8, device="cpu")


@pytest.fixture(autouse=True)
def biases():
    global BI, BF
    BI, BF = BI.to(DEV), BF.to(DEV)


@pytest.mark.parametrize("lens", [[1], [2, 3, 4, 5], [127, 128, 129], [255, 256, 257], [131, 1, 4, 700]])
def test_chunks_rows_and_cuts(lens):
    H, T = 5, sum(lens)
    g = torch.Generator(device=DEV).manual_seed(T)
    pre = torch.randn(T, 2 * H, generator=g, device=DEV) * 6
    state = torch.randn(len(lens), 16, generator=g, device=DEV)
    whole, after = state.clone(), []
    got = gates(pre, lens, whole, H)
    at = 0
    for r, n in enumerate(lens):
        m = state[r, 4: 4 + H].double()
        for t in range(at, at + n):
            i = 10 * torch.tanh((pre[t, :H].double() + BI[:H]) / 10)
            f = torch.nn.functional.logsigmoid(10 * torch.tanh((pre[t, H:].double() + BF[:H]) / 10))
            new = torch.maximum(f + m, i)
            want = torch.stack([torch.exp(f + m - new), torch.exp(i - new), torch.exp(-new)])
            # n sums of numbers up to 20 in front of an exponential
            assert ((got[:, t].double() - want).abs() <= (n + 8) * 2.0 ** -24 * 20 * want + 1e-30).all()
            m = new
        assert ((whole[r, 4: 4 + H].double() - m).abs() <= (n + 8) * 2.0 ** -24 * 20).all()
        one = state[r: r + 1].clone()                                   # the row by itself, in portions
        cuts = [0, n // 3, n // 3 + (n > 4), n]
        parts = [gates(pre[at + a: at + b], [b - a], one, H) for a, b in zip(cuts, cuts[1:]) if b > a]
        assert torch.equal(torch.cat(parts, 1), got[:, at: at + n]) and torch.equal(one[0], whole[r])
        at += n


def test_an_infinite_gate():
    pre = torch.zeros(200, 2, device=DEV)
    clean = gates(pre, [200], torch.zeros(1, 16, device=DEV), 1)
    pre[130, 1] = float("nan")
    odd = gates(pre, [200], torch.zeros(1, 16, device=DEV), 1)
    assert torch.equal(odd[:, :130], clean[:, :130]) and odd[0, 130].isnan().all()
