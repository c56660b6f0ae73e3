"""Products of up to 8 rows that read their weights straight from memory, against float64: each way of cutting them (8 and 16 rows a block, 8 to
32 warps), sizes at which a block's rows and a warp's share of K do not come out whole, and the sizes on both sides of the rule; with and without
the rows' norm factors, as a gated pair and into a residual."""
import pytest
import torch

from arle_b200 import ops
from launched import launched

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,N,K", [(1, 1, 32), (8, 9, 96), (3, 1152, 1056), (5, 1147, 1600), (2, 1151, 2080), (7, 1153, 2048), (1, 2303, 1568), (8, 4608, 1056),
                                   (4, 9215, 64), (6, 9217, 64), (8, 4096, 4096), (2, 4097, 4096)])
def test_direct_products(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(N + K)
    wide = torch.randn(M, K + 8, generator=g, device=DEV).to(torch.bfloat16)
    x, w = wide[:, :K], (torch.randn(N, K + 8, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)[:, :K]
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    room = K * 2.0 ** -24 * size                                # float32 sums of exact products, whatever their order
    for dtype, unit in ((torch.float32, 2.0 ** -24), (torch.bfloat16, 2.0 ** -8)):
        out = torch.full((M + 1, N + 8), 7.0, device=DEV, dtype=dtype)
        ops.gemm(x, w, out[:M, :N])
        assert ((out[:M, :N].double() - want).abs() <= room + unit * want.abs()).all() and (out[M] == 7.0).all() and (out[:, N:] == 7.0).all()
    rows = ops.ScaledRows(x, torch.rand(ops.SS_TABLE_SHAPE, generator=g, device=DEV), 1e-6)
    f = torch.rsqrt(rows.ss[:M].double().sum(1, keepdim=True) / K + 1e-6)
    out = torch.empty(M, N, device=DEV)
    ops.gemm(rows, w, out)
    assert ((out.double() - want * f).abs() <= (room + 1e-6 * want.abs()) * f).all()
    if N % 2 == 0:
        out = torch.empty(M, N // 2, device=DEV, dtype=torch.float32)
        ops.gemm_silu_mul(rows, w, torch.empty(M, N, device=DEV, dtype=torch.bfloat16), out)
        gate, up = (want * f)[:, 0::2], (want * f)[:, 1::2]
        near = (room * f)[:, 0::2] * 1.1 * up.abs() + (room * f)[:, 1::2] * gate.abs() + 2e-6 * (gate * up).abs() + 1e-12
        assert ((out.double() - gate * torch.sigmoid(gate) * up).abs() <= near).all()
    resid0, gain = torch.randn(M, N, generator=g, device=DEV), torch.rand(N, generator=g, device=DEV)
    got = []
    for _ in range(2):
        sink = ops.ResidualSink(resid0.clone(), gain, 1e-6, torch.empty(M, N, device=DEV, dtype=torch.bfloat16), torch.full(ops.SS_TABLE_SHAPE, 7.0, device=DEV), 0.5)
        assert ops.gemm(x, w, None, sink=sink)
        got.append(sink)
    r = got[0].resid.double()
    assert ((r - resid0.double() - 0.5 * want).abs() <= room + 2.0 ** -23 * (resid0.double().abs() + want.abs())).all()
    assert ((got[0].xs.double() - r * gain.double()).abs() <= 2.0 ** -8 * (r * gain.double()).abs()).all()
    ss = got[0].ss.double()
    assert (ss[M:] == 0).all() and ((ss[:M].sum(1) - r.square().sum(1)).abs() <= 1e-5 * r.square().sum(1)).all()
    assert torch.equal(got[0].resid, got[1].resid) and torch.equal(got[0].ss, got[1].ss)
    ops.check_errors(DEV)


@pytest.mark.parametrize("M,N,K,direct", [(8, 512, 12288, True), (1, 40, 12320, False), (8, 512, 16384, False), (3, 700, 16384, True), (1, 700, 16416, False),
                                          (8, 128, 32768, False), (1, 200, 65536, True)])
def test_long_shares_go_to_the_ring(M, N, K, direct):
    """Few rows of a long K would leave a warp one block of K after the other; the ring takes K apart over a cluster (up to what it holds)."""
    x, w = (torch.randn(m, K, device=DEV).to(torch.bfloat16) for m in (M, N))
    out = torch.empty(M, N, device=DEV)
    assert launched(lambda: ops.gemm(x, w, out), r"\w+_gemm_kernel") == {"direct_gemm_kernel" if direct else "skinny_gemm_kernel"}
    want, size = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    assert ((out.double() - want).abs() <= K * 2.0 ** -24 * size).all()
    ops.check_errors(DEV)


# (rows, warps, blocks of K under way): (16, 8, 4), (16, 16, 2), (16, 24, 2), (8, 8, 4), (8, 16, 2), (8, 24, 2); shares of 5 and 6 blocks, of which a second
# round has one and two, and one whose last warp has fewer
@pytest.mark.parametrize("M,N,K", [(2, 6144, 1024), (3, 4096, 1024), (1, 3000, 1536), (8, 1152, 544), (4, 1000, 1024), (5, 1000, 1536), (2, 6144, 1344), (8, 1000, 5088)])
def test_further_cuts(M, N, K):
    test_direct_products(M, N, K)


@pytest.mark.parametrize("M,H,F", [(1, 1024, 3072), (5, 1024, 3072), (8, 256, 4608)])
def test_products_behind_one_another(M, H, F):
    """Products that start beside the one in front of them read what it wrote: into a residual, out of its norm factors, a gated pair and into the residual
    again, with weights that the kernel in front has just written; in stream order, with a wait behind each, and in a graph, over and over."""
    g = torch.Generator(device=DEV).manual_seed(M + H)
    x0 = torch.randn(M, F, generator=g, device=DEV).to(torch.bfloat16)
    w_new = [(torch.randn(*s, generator=g, device=DEV) * s[1] ** -0.5).to(torch.bfloat16) for s in ((H, F), (2 * F, H), (H, F))]
    gain, r0 = torch.rand(H, generator=g, device=DEV), torch.randn(M, H, generator=g, device=DEV)
    bf = dict(device=DEV, dtype=torch.bfloat16)
    ws, gains = [torch.empty_like(w) for w in w_new], torch.empty_like(gain)
    resid, mid, pair = torch.empty(M, H, device=DEV), torch.empty(M, F, **bf), torch.empty(M, 2 * F, **bf)
    sinks = [ops.ResidualSink(resid, gains, 1e-6, torch.empty(M, H, **bf), torch.empty(ops.SS_TABLE_SHAPE, device=DEV), 1.0) for _ in range(2)]

    def chain(wait):
        for t in ws:
            t.fill_(float("nan"))
        gains.fill_(float("nan"))
        resid.copy_(r0)
        x = x0
        for i in range(3):
            gains.copy_(gain)
            ws[0].copy_(w_new[0])                                # by a kernel that the product stands right behind
            assert ops.gemm(x, ws[0], None, sink=sinks[0])
            wait()
            ws[1].copy_(w_new[1])
            ops.gemm_silu_mul(ops.ScaledRows(sinks[0].xs, sinks[0].ss, 1e-6), ws[1], pair, mid)
            wait()
            ws[2].copy_(w_new[2])
            assert ops.gemm(mid, ws[2], None, sink=sinks[1])
            wait()
            x = mid
        return [t.clone() for t in (resid, sinks[1].xs, sinks[1].ss, mid)]

    want = chain(torch.cuda.synchronize)
    assert torch.isfinite(want[0]).all()
    for _ in range(20):
        assert all(torch.equal(a, b) for a, b in zip(want, chain(lambda: None)))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        chain(lambda: None)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(lambda: None)
    for _ in range(20):
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(want, got))
    ops.check_errors(DEV)
