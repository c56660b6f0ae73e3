"""float32 rows times a bfloat16 W in three pieces on the tensor cores: against float64 at the edges of the tiles (16, 32, 64 and 80 rows by
128 columns), rows of other tensors untouched; no further off than the FFMA kernels; a row's bits whatever stands beside it; infinities,
NaNs and the ends of float32's range."""
import pytest
import torch

from arle_b200 import ops
from launched import launched

pytestmark = pytest.mark.gpu
DEV = "cuda"


def inputs(M, N, K, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed + M + N + K)
    x = torch.randn(M, K, generator=g, device=DEV) * torch.exp(torch.randn(M, K, generator=g, device=DEV))
    return x, torch.randn(N, K, generator=g, device=DEV).bfloat16()


def ffma(x, w):
    out = torch.empty(x.shape[0], w.shape[0], device=DEV)
    with ops.use_kernel_set("plain"):
        ops.gemm(x, w, out)
    return out


@pytest.mark.parametrize("M,N,K,kernel", [
    (1, 256, 512, "<16, 1>"), (16, 300, 576, "<16, 1>"), (17, 4097, 1024, "<16, 1>"), (1, 20000, 512, "<16, 2>"), (16, 37900, 1024, "<16, 2>"),
    (200, 2050, 640, "<32, 1>"), (129, 3000, 1024, "<32, 1>"), (301, 1024, 3072, "<32, 1>"), (301, 6145, 512, "<64, 1>"), (640, 2304, 4096, "<80, 1>"), (80, 15000, 640, "<80, 1>"), (301, 4096, 512, "<80, 1>"),
    (64, 20000, 512, "<64, 1>")])
def test_against_float64(M, N, K, kernel):
    x, w = inputs(M, N, K)
    out = torch.full((M + 1, N + 4), 7.0, device=DEV)
    ran = launched(lambda: ops.gemm(x, w, out[:M, :N]), r"gemm_f32_.*?>(?=\()")
    assert len(ran) == 1 and "tc_kernel" + kernel in ran.pop()
    assert (out[M] == 7.0).all() and (out[:, N:] == 7.0).all()
    exact, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    err, plain = (out[:M, :N].double() - exact).abs(), (ffma(x, w).double() - exact).abs()
    # a block of 64: four sums of 16 in the accumulator, cut off (2^-23 each, the later ones of the first pieces alone count), then one
    # rounding (2^-24) for each of the K / 64 blocks: no element's error is beyond (4 * 2 + K / 64) * 2^-24 of its numbers' sum
    assert (err <= (8 + K / 64) * 2.0 ** -24 * size).all()
    assert err.square().mean() <= plain.square().mean()
    ops.check_errors(DEV)


def test_a_row_has_the_same_bits_whatever_stands_beside_it():
    x, w = inputs(301, 4096, 1024)
    want = torch.empty(301, 4096, device=DEV)
    ops.gemm(x, w, want)
    for rows in (slice(0, 1), slice(300, 301), slice(7, 23), slice(7, 24), slice(40, 140), slice(40, 200), slice(0, 257)):
        got = torch.empty(x[rows].shape[0], 4096, device=DEV)
        ops.gemm(x[rows], w, got)
        assert torch.equal(got, want[rows])
    wide = torch.empty(301, 4096 + 12, device=DEV)[:, 8:-4]
    ops.gemm(torch.empty(301, 1028, device=DEV)[:, :1024].copy_(x), w, wide)
    assert torch.equal(wide, want)


def test_not_for_short_sums_few_columns_or_rows_off_the_boundaries():
    for M, N, K, off in ((5, 256, 448, 0), (5, 255, 512, 0), (5, 256, 520, 0), (5, 256, 512, 1)):
        x, w = inputs(M, N, K)
        x = torch.empty(M, K + off, device=DEV)[:, :K].copy_(x)
        out = torch.empty(M, N, device=DEV)
        assert not any("_tc_" in k for k in launched(lambda: ops.gemm(x, w, out), r"gemm_f32_.*?>(?=\()"))
        assert torch.equal(out, ffma(x, w))


def test_infinities_nans_and_the_ends_of_the_range():
    M, N, K = 70, 300, 512
    x, w = inputs(M, N, K)
    inf, nan, big = float("inf"), float("nan"), torch.finfo(torch.float32).max
    x[3, 5], x[4, 9], x[5, 0], x[6, 1], x[6, 2] = inf, nan, -inf, inf, -inf
    x[7] *= 2.0 ** -120                                   # pieces below bfloat16's smallest normal number
    x[8] = 0
    x[8, 17] = big                                        # would round to an infinity as a bfloat16
    x[9, 40] = torch.tensor(0x7f800001, dtype=torch.int32).view(torch.float32)      # a NaN whose upper half is an infinity's
    w[20, 11], w[21, 11], w[22, 3], w[23, 30] = inf, -inf, nan, 0.0
    w[:, 17] = w[:, 17].sign() * 0.5
    out = torch.empty(M, N, device=DEV)
    ops.gemm(x, w, out)
    want = ffma(x, w)
    assert torch.equal(out.isnan(), want.isnan()) and torch.equal(out.isinf(), want.isinf())
    assert torch.equal(out[out.isinf()], want[want.isinf()])
    ok = want.isfinite()
    size = x.double().abs() @ w.double().abs().t()
    assert ((out.double() - want.double()).abs()[ok] <= 2 * K * 2.0 ** -24 * size[ok] + K * 2.0 ** -133).all()
    ops.check_errors(DEV)
