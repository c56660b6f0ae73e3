"""silu in front of a bfloat16 rounding (fast exponential and division): every bfloat16 number through the short convolution whose only tap is
the present token's, in the windowed kernel and in the one that takes a token a thread."""
import pytest
import torch

from arle_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows", [1, 64])                  # 64 rows of one token: not the windowed kernel
def test_silu_of_every_bfloat16_number(rows):
    C, T = 1024, 64
    x = torch.arange(65536, dtype=torch.int32, device=DEV).to(torch.int16).view(torch.bfloat16).view(T, C)
    w = torch.zeros(C, 4, device=DEV)
    w[:, 3] = 1
    cuts = torch.arange(0, T + 1, T // rows, dtype=torch.int32, device=DEV)
    row_of = torch.arange(T, device=DEV).div(T // rows, rounding_mode="floor").int()
    state = torch.zeros(rows, C * 3, device=DEV)
    out = torch.empty_like(x)
    ok = x.isfinite()
    ops.conv_silu(x.masked_fill(~ok, 0), w, None, state, 0, cuts, row_of, torch.arange(rows, dtype=torch.int32, device=DEV), out)
    v = x.double()[ok]
    exact = v * torch.sigmoid(v)
    got = out.double()[ok]
    # float32's exponential, sum and quotient: 2^-21 at most with what |x| does to the exponent (2^-24 |x|), then bfloat16's half unit, 2^-8;
    # behind an exponential beyond 2^126 the quotient is zero, 1e-36 off
    assert ((got - exact).abs() <= exact.abs() * (2.0 ** -8 + 2.0 ** -21 + 2.0 ** -23 * v.abs()) + 1.1e-36).all()
    rounded = exact.to(torch.bfloat16).double()
    assert (got != rounded)[exact.abs() > 1e-30].double().mean() < 1e-3


def test_infinities_and_nans():
    C, T = 8, 40
    x = torch.ones(T, C, device=DEV, dtype=torch.bfloat16)
    x[7, 0], x[7, 1], x[7, 2] = float("inf"), float("nan"), -float("inf")
    w = torch.zeros(C, 4, device=DEV)
    w[:, 3] = 1
    out = torch.empty_like(x)
    ops.conv_silu(x, w, None, torch.zeros(1, C * 3, device=DEV), 0, torch.tensor([0, T], dtype=torch.int32, device=DEV),
                  torch.zeros(T, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV), out)
    assert out[7, 0] == float("inf") and out[7, 1].isnan() and out[7, 2].isnan() and out[7, 3:].isfinite().all()
    assert out[:7].isfinite().all()
