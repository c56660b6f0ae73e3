"""Which kernel a float32 product takes goes by sizes and by how the arrays lie in memory; asked here of arrays without memory (meta tensors), some
larger than any GPU's."""
import pytest
import torch

from arle_b200 import ops


def _rows(n, k):
    return torch.empty(n, k, dtype=torch.float32, device="meta")


def _matrix(n, k):
    return torch.empty(n, k, dtype=torch.bfloat16, device="meta")


@pytest.mark.parametrize("M,N,K,pieces", [(1, 256, 512, True), (301, 6144, 1024, True), (900_000, 24_576, 12_288, True), (932_064, 24_576, 12_288, True),
                                          (932_065, 24_576, 12_288, False), (1 << 20, 24_576, 12_288, False), (5, 255, 512, False), (5, 256, 448, False)])
def test_products_beyond_its_counters_stay_with_the_general_kernels(M, N, K, pieces):
    assert ops.f32_pieces_supported(_rows(M, K), _matrix(N, K)) is pieces


def test_rows_that_overlap_stay_with_the_general_kernels():
    x, w = _rows(64, 1024), _matrix(256, 1024)
    assert ops.f32_pieces_supported(x, w)
    assert not ops.f32_pieces_supported(x[:1].expand(64, 1024), w)                       # one row 64 times
    assert not ops.f32_pieces_supported(_rows(1, 4096).as_strided((64, 1024), (4, 1)), w)  # windows of one row
    assert not ops.f32_pieces_supported(x, w[:1].expand(256, 1024))
