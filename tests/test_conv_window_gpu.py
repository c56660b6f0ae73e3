"""The convolution's sliding window against the kernel that takes a token a thread (the same bits): rows that begin and end inside a
thread's tokens, few and many channels; and the gated norm in parts against float64."""
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


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens", [[40], [37, 1, 2, 80, 3], [16, 16, 17]])
@pytest.mark.parametrize("C", [8, 264, 1032])
def test_convolution_window_gives_the_same_bits(dtype, lens, C):
    g = torch.Generator(device=DEV).manual_seed(C + len(lens))
    T = sum(lens)
    ctx = _ctx(lens, 3 * C + 8)
    x = torch.randn(T, C + 8, generator=g, device=DEV).to(dtype)
    odd = torch.empty(T, C + 1, device=DEV, dtype=dtype)
    odd[:, 1:] = x[:, :C]
    w, bias, extra = (torch.randn(*s, generator=g, device=DEV) for s in ((C, 4), (C,), (C,)))
    state0 = torch.randn(len(lens) + 1, 3 * C + 8, generator=g, device=DEV)
    got = []
    for src in (x[:, :C], odd[:, 1:]):
        for fn in (lambda st, o: ops.conv_silu(src, w, bias, st, 5, ctx.q_indptr, ctx.row_of_token, ctx.state_slots, o),
                   lambda st, o: ops.causal_conv(src, extra, w, None, "none", st, 5, ctx.q_indptr, ctx.row_of_token, ctx.state_slots, o)):
            st, o = state0.clone(), torch.empty(T, C, device=DEV, dtype=dtype)
            fn(st, o)
            got.append((o, st))
    for (o1, s1), (o2, s2) in ((got[0], got[2]), (got[1], got[3])):
        assert torch.equal(o1, o2) and torch.equal(s1, s2)


@pytest.mark.parametrize("C", [4, 260])                          # groups of four channels, of which eight do not make whole ones
def test_convolution_window_of_channels_in_fours(C):
    test_convolution_window_gives_the_same_bits(torch.bfloat16, [37, 1, 2, 80, 3], C)


@pytest.mark.parametrize("inner,parts,skip", [(1024, 1, True), (8192, 1, True), (8192, 2, False), (4160, 1, True), (2048 * 3, 3, True)])
def test_gated_group_norm(inner, parts, skip):
    g = torch.Generator(device=DEV).manual_seed(inner)
    T, vdim = 5, 64 if inner % 64 == 0 else 8
    y = torch.randn(T, inner, generator=g, device=DEV)
    x, z = (torch.randn(T, inner + 8, generator=g, device=DEV).to(torch.bfloat16)[:, :inner] for _ in range(2))
    d, w = torch.rand(inner // vdim, generator=g, device=DEV), torch.rand(inner, generator=g, device=DEV)
    out = torch.full((T + 1, inner), 7.0, device=DEV, dtype=torch.bfloat16)
    ops.gated_group_norm(y, x, d if skip else None, vdim, z, w, 1e-5, out[:T], parts)
    val = (y.double() + (d.double().repeat_interleave(vdim) * x.double() if skip else 0)) * z.double() * torch.sigmoid(z.double())
    val = val.view(T, parts, -1)
    want = (val * torch.rsqrt(val.square().mean(-1, keepdim=True) + 1e-5)).reshape(T, inner) * w.double()
    assert ((out[:T].double() - want).abs() <= (2.0 ** -8 + 1e-5) * want.abs() + 1e-6).all() and (out[T] == 7.0).all()


@pytest.mark.parametrize("inner,parts", [(4104, 1), (6144, 1), (6152, 1), (12288, 2)])
def test_gated_group_norm_of_six_thousand(inner, parts):         # parts of 4,097 to 6,144 numbers have threads of their own number
    test_gated_group_norm(inner, parts, True)
