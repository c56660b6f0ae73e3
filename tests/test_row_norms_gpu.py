"""Norms of plain rows at the widths where a row is kept in registers in part, and where many wide rows go to a kernel of their own: against float64,
and the same bits of a row whichever kernel runs it."""
import pytest
import torch

from arle_b200 import ops
from launched import launched

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("src,dst", [(torch.bfloat16, torch.bfloat16), (torch.float32, torch.bfloat16), (torch.float32, torch.float32)])
@pytest.mark.parametrize("n", [1025, 2048, 2049, 4096, 4097, 8200])
def test_rows_of_every_width(n, src, dst):
    g = torch.Generator(device=DEV).manual_seed(n)
    x = torch.randn(513, n + 3, generator=g, device=DEV).to(src)[:, :n]
    w = torch.rand(n, generator=g, device=DEV) + 0.5

    def run(rows):
        out = torch.full((rows + 1, n + 5), 7.0, device=DEV, dtype=dst)
        kernel, = launched(lambda: ops.rms_rows(x[:rows], w, 1e-6, out[:rows, :n]), r"rms_rows_\w+_kernel")
        assert kernel == ("rms_rows_wide_kernel" if n > 4096 and rows > 512 else "rms_rows_block_kernel")
        assert (out[rows] == 7).all() and (out[:, n:] == 7).all()
        return out[:rows, :n]

    many = run(513)
    exact = x.double() / (x.double().square().mean(1, keepdim=True) + 1e-6).sqrt() * w.double()
    # a float32 sum of squares in strands of n / 256 and a tree, a square root, a division and two products: under 2^-18; then dst's half unit
    assert ((many.double() - exact).abs() <= exact.abs() * ((2.0 ** -8 if dst == torch.bfloat16 else 0) + 2.0 ** -18)).all()
    for rows in (512, 1):
        assert torch.equal(run(rows), many[:rows])
