"""The delta rule's scan with the next chunk's numbers loaded ahead and without: the same bits (rows off a 16-byte boundary run without), at
row lengths around a chunk of 16, with few blocks and with more than are resident at a time."""
import pytest
import torch

from arle_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,dim,vdim", [(2, 8, 12), (2, 64, 40), (3, 128, 128), (2, 256, 64), (8, 256, 256), (1, 512, 96)])
@pytest.mark.parametrize("lens", [[40, 16, 1, 33, 17], [15, 128], [4] * 16], ids=["mixed", "two", "short"])
def test_same_bits(dtype, heads, dim, vdim, lens):
    g = torch.Generator(device=DEV).manual_seed(dim + len(lens))
    T, R, width = sum(lens), len(lens), heads * (2 * dim + vdim)
    at = torch.tensor([0] + lens, device=DEV).cumsum(0).to(torch.int32)
    slots = torch.arange(R, dtype=torch.int32, device=DEV)
    x = torch.randn(T, width, generator=g, device=DEV).to(dtype)
    beta, decay = torch.rand(T, heads, generator=g, device=DEV), 1 - 0.2 * torch.rand(T, heads, generator=g, device=DEV)
    state0 = torch.randn(R, heads * vdim * dim, generator=g, device=DEV)
    got = []
    for off in (0, 1):
        rows = torch.empty(T, width + 8, dtype=dtype, device=DEV)[:, off: off + width].copy_(x)
        q, k, v = rows.split([heads * dim, heads * dim, heads * vdim], 1)
        state, out = state0.clone(), torch.full((T, heads, vdim), 7.0, device=DEV)
        ops.delta_scan(q, k, v, beta, decay, state, at, slots, out, heads, heads, dim, vdim, dim ** -0.5, 1e-6)
        got.append((out, state))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert not (got[0][0] == 7.0).all(-1).any()
