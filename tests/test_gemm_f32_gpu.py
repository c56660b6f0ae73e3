"""The float32 products: every kernel sums k in ascending order, so the tiles and the row kernel give the bits of the general kernel (which
runs when rows are not on 16-byte boundaries), at the edges of their tiles; and float64 stays within a K-term sum's error."""
import pytest
import torch

from arle_b200 import ops
from launched import launched

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("wdtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M", [1, 2, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 130, 301, 700])
@pytest.mark.parametrize("N,K", [(31, 8), (32, 64), (129, 72), (1000, 136), (2049, 16), (20000, 24)])
def test_same_bits_as_the_general_kernel(wdtype, M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g, device=DEV)
    w = torch.randn(N, K, generator=g, device=DEV).to(wdtype)
    odd = torch.empty(M, K + 1, device=DEV)[:, :K].copy_(x)            # rows off the boundaries: the general kernel
    got, want = torch.full((M + 1, N), 7.0, device=DEV), torch.empty(M, N, device=DEV)
    ops.gemm(x, w, got[:M])
    ops.gemm(odd, w, want)
    assert torch.equal(got[:M], want) and (got[M] == 7.0).all()
    exact = x.double() @ w.double().t()
    assert ((got[:M].double() - exact).abs() <= K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().t())).all()


def test_as_many_rows_as_the_general_kernel_takes():
    M, N, K = 65535 * 32 + 1, 3, 8                                     # one more than a grid of tiles of 32 rows holds
    g = torch.Generator(device=DEV).manual_seed(1)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV)
    got = torch.empty(M, N, device=DEV)
    ops.gemm(x, w, got)
    exact = x.double() @ w.double().t()
    assert ((got.double() - exact).abs() <= K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().t())).all()


F32, BF16 = torch.float32, torch.bfloat16


@pytest.mark.parametrize("wdtype,M,N,K,kernel", [
    (w, M, N, K, f"stages_kernel<{t}, {tile}") for w, t in ((F32, "float"), (BF16, "__nv_bfloat16"))
    for M, N, K, tile in ((33, 1000, 1032, "32, 32"), (301, 2050, 264, "32, 32"), (301, 3072, 128, "64, 64"), (301, 3072, 136, "64, 64"), (333, 3077, 1032, "64, 64"))
] + [(w, 301, 6145, 264, f"tiles_kernel<{t}, 64, 128") for w, t in ((F32, "float"), (BF16, "__nv_bfloat16"))]
  + [(BF16, 700, 4100, 264, "tiles_kernel<__nv_bfloat16, 64, 64"), (F32, 700, 4100, 264, "stages_kernel<float, 64, 64")])
def test_every_tile_goes_round_its_stages(wdtype, M, N, K, kernel):
    """Each kernel at a K of several rounds of its stages and a part of one, and the size that has the launcher choose it."""
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    x, w = torch.randn(M, K, generator=g, device=DEV), torch.randn(N, K, generator=g, device=DEV).to(wdtype)
    odd = torch.empty(M, K + 1, device=DEV)[:, :K].copy_(x)
    got, want = torch.full((M + 1, N), 7.0, device=DEV), torch.empty(M, N, device=DEV)
    ran = launched(lambda: ops.gemm(x, w, got[:M]), r"gemm_f32_.*?>(?=\()")
    assert len(ran) == 1 and kernel in ran.pop()
    ops.gemm(odd, w, want)
    assert torch.equal(got[:M], want) and (got[M] == 7.0).all()
