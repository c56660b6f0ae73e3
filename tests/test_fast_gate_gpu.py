"""Gates in bfloat16 have the bits of the full exponential and division, rounded once: every bfloat16 number through the short convolution whose
only tap is the present token's (in the windowed kernel and in the one that takes a token a thread), and the norms with a gate, against the same
kernels on float32 arrays."""
import math

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
    # float32's exponential, sum and quotient: 2^-21 at most with what |x| does to the exponent (2^-24 |x|), then bfloat16's half unit, 2^-8,
    # and results that small end at 1e-36
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


def _every_bfloat16(T=64, C=1024):
    return torch.arange(65536, dtype=torch.int32, device=DEV).to(torch.int16).view(torch.bfloat16).view(T, C)


def _same(got, full):
    """Equal bits but for what a NaN holds."""
    want = full.to(torch.bfloat16)
    return bool(((got.view(torch.int16) == want.view(torch.int16)) | (got.isnan() & want.isnan())).all())


@pytest.mark.parametrize("kind", ["causal_conv", "conv_silu"])
@pytest.mark.parametrize("rows", [1, 64])                  # 64 rows of one token: not the windowed kernel
def test_silu_is_the_full_form(kind, rows):
    x = _every_bfloat16()
    T, C = x.shape
    x = x.masked_fill(~x.isfinite(), 0)                    # in the window they would reach their neighbours
    w = torch.zeros(C, 4, device=DEV)
    w[:, 3] = 1
    cuts = torch.arange(0, T + 1, T // rows, dtype=torch.int32, device=DEV)
    row_of = torch.arange(T, device=DEV).div(T // rows, rounding_mode="floor").int()
    slots = torch.arange(rows, dtype=torch.int32, device=DEV)

    def run(a, out):
        state = torch.zeros(rows, C * 3, device=DEV)
        if kind == "conv_silu":
            ops.conv_silu(a, w, None, state, 0, cuts, row_of, slots, out)
        else:
            ops.causal_conv(a, None, w, None, "silu", state, 0, cuts, row_of, slots, out)
        return out

    assert _same(run(x, torch.empty_like(x)), run(x.float(), torch.empty(T, C, device=DEV)))


@pytest.mark.parametrize("op,vdim", [("gla_silu", 128), ("gla_silu", 256), ("gla_silu", 63), ("gla_sigmoid", 128), ("gla_sigmoid", 63),
                                     ("mlstm", 128), ("group_norm", 128), ("group_norm", 63)])
def test_gated_norms_are_the_full_form(op, vdim):
    g = torch.Generator(device=DEV).manual_seed(vdim)
    T, heads = 300, 4
    n = heads * vdim
    gate = _every_bfloat16(1, 65536).view(-1)[torch.randint(0, 65536, (T, n), generator=g, device=DEV)]
    gate = torch.where(gate.isfinite() & (gate.abs() < 200), gate, torch.randn(T, n, generator=g, device=DEV).to(torch.bfloat16) * 4)
    y = torch.randn(T, n, generator=g, device=DEV)
    w = torch.rand(n, generator=g, device=DEV) + 0.5

    def run(z):
        out = torch.empty(T, n, device=DEV, dtype=z.dtype)
        if op == "mlstm":
            num = torch.cat([y.view(T, heads, vdim), torch.ones(T, heads, 1, device=DEV)], 2).contiguous()
            ops.mlstm_out(num, torch.full((T, heads), 0.5, device=DEV), z, w, 1e-6, out, heads, vdim)
        elif op == "group_norm":
            ops.gated_group_norm(y, z, None, vdim, z, w, 1e-6, out, heads)
        else:
            ops.gla_out(y, z, w, 1e-6, 0.7, out, heads, vdim, gate_act=op[4:])
        return out

    assert _same(run(gate), run(gate.float()))


def test_gated_product_divides_in_full():
    """A gate of -88: 1 + exp(88) is beyond 2^126, where the fast division gives zero, and NaN times an infinite up."""
    M, K = 1024, 64
    x = torch.zeros(M, K, device=DEV, dtype=torch.bfloat16)
    x[:, 0] = 1
    w = torch.zeros(256, K, device=DEV, dtype=torch.bfloat16)
    w[0::2, 0] = -88
    w[1::2, 0] = torch.tensor(1e30)
    w[3, 0] = float("inf")
    w[3, 1:] = 1
    out = torch.empty(M, 128, device=DEV, dtype=torch.bfloat16)
    ops.gemm_tcgen05_pair(x, w, out, gated=True)
    want = -88 / (1 + math.exp(88)) * 1e30
    assert (out[:, 1] == -float("inf")).all()
    rest = out[:, [0, 2, 127]].double()
    # exp in float32 with a relative error below 2^-16 (88 x 1.173 units), the gate's factors and the result in bfloat16: 3 x 2^-9
    assert ((rest - want).abs() <= abs(want) * 2.0 ** -7).all()
