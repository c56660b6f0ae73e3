"""The experts' products on tcgen05 tiles (weights in the tile's rows, 32 to 256 tokens beside them) against float64, at the edges of
the tiles: experts with no token, one, around 32, 256 and 512 tokens and more than eight parts of 256; weight rows that do and do not
fill a tile of 256; K below, at and past a block of 64; gathered and place-ordered rows; every finish."""
import pytest
import torch

from arle_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"

COUNTS = [[129], [0, 31, 32, 33, 0, 64, 1], [255, 0, 256, 257], [511, 512, 513], [2305, 3], [8] * 32]


def _gate(z, act, limit, alpha):
    g, u = z[:, 0::2], z[:, 1::2]
    if act == "silu":
        return g * torch.sigmoid(g) * u
    if act == "gelu_tanh":
        return torch.nn.functional.gelu(g, approximate="tanh") * u
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(alpha * g) * (u + 1)


def _setup(counts, N, K, gathered, seed=0):
    g = torch.Generator().manual_seed(seed + sum(counts) + N)
    E, pairs = len(counts), sum(counts)
    ids = torch.cat([torch.full((c,), e, dtype=torch.int32) for e, c in enumerate(counts)])[torch.randperm(pairs, generator=g)]
    plan = torch.zeros(ops.moe_plan_size(E, pairs), dtype=torch.int32, device=DEV)
    place, row = (torch.zeros(pairs, dtype=torch.int32, device=DEV) for _ in range(2))
    ops.moe_plan(ids[:, None].contiguous().to(DEV), E, plan, place, row)
    wide = torch.randn(pairs, K + 8, generator=g).to(torch.bfloat16).to(DEV)
    x = wide[:, :K]                                            # rows of a wider buffer
    w = (torch.randn(E, N, K, generator=g) * K ** -0.5).to(torch.bfloat16).to(DEV)
    at = row.long() if gathered else torch.arange(pairs, device=DEV)
    expert = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).to(DEV)
    z = torch.empty(pairs, N, dtype=torch.float64, device=DEV)
    mag = torch.empty_like(z)
    for e in range(E):
        s = expert == e
        z[s] = x[at[s]].double() @ w[e].double().t()
        mag[s] = x[at[s]].double().abs() @ w[e].double().abs().t()
    return x, row if gathered else None, w, plan, z, mag


@pytest.mark.parametrize("counts", COUNTS, ids=lambda c: "-".join(map(str, c))[:24])
@pytest.mark.parametrize("N,K,gathered", [(256, 64, True), (130, 200, True), (515, 8, False), (96, 320, False)])
def test_products_at_tile_edges(counts, N, K, gathered):
    x, rows, w, plan, z, mag = _setup(counts, N, K, gathered)
    pairs, E = z.shape[0], w.shape[0]
    scale = torch.rand(pairs, device=DEV) + 0.5
    for act in ("none", "square_relu"):
        out = torch.full((pairs + 1, N), 7.0, dtype=torch.bfloat16, device=DEV)
        ops.moe_gemm(x, rows, w, out[:pairs], plan, E, place_scale=scale, act=act)
        s = scale.double()[:, None]
        want = z * s if act == "none" else (z * s).clamp(min=0).square()
        # float32 sums in any order: K roundings of the summed magnitudes; then one rounding to 8 bits
        err = K * 2.0 ** -23 * mag * s
        bound = (err if act == "none" else 2 * (z * s).abs() * err + err.square()) + 2.0 ** -8 * want.abs() + 1e-30
        assert ((out[:pairs].double() - want).abs() <= bound).all()
        assert (out[pairs] == 7.0).all()
    ops.check_errors(DEV)


def test_every_set_of_boxes():
    """Half a tile's tokens are 16 to 128: boxes of 128, 64, 32 and 16 rows, one of each at most; the last expert's end where x does."""
    x, rows, w, plan, z, mag = _setup([32 * i - i % 2 for i in range(1, 9)] + [480, 31 + 256], 300, 136, False, seed=5)
    out = torch.full((z.shape[0] + 1, 300), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.moe_gemm(x, None, w, out[:-1], plan, w.shape[0])
    assert ((out[:-1].double() - z).abs() <= 136 * 2.0 ** -23 * mag + 2.0 ** -8 * z.abs() + 1e-30).all()
    assert (out[-1] == 7.0).all()
    ops.check_errors(DEV)


@pytest.mark.parametrize("counts", [COUNTS[1], COUNTS[2], [300]], ids=["small", "mid", "one"])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh", "clamped_glu"])
def test_gated_products(counts, act):
    N, K = 318, 136
    x, rows, w, plan, z, mag = _setup(counts, N, K, True, seed=3)
    pairs, E = z.shape[0], w.shape[0]
    side = torch.empty(pairs, K, dtype=torch.bfloat16, device=DEV)
    ops.moe_rows(x, rows, side)
    assert torch.equal(side, x[rows.long()])
    want = _gate(z, act, 1.5, 1.702)
    # the gates' slopes are below 1.2 times the other factor; __expf and __fdividef are good to a few units of 2^-22
    both = mag[:, 0::2] + mag[:, 1::2]
    bound = 2.0 ** -8 * want.abs() + (1.2 * K * 2.0 ** -23 + 2.0 ** -20) * both * (1 + z[:, 0::2].abs() + z[:, 1::2].abs()) + 1e-30
    for src, at in ((x, rows), (side, None)):
        out = torch.full((pairs + 1, N // 2), 7.0, dtype=torch.bfloat16, device=DEV)
        ops.moe_gemm_gated(src, at, w, out[:pairs], plan, E, act, None, 1.5, 1.702)
        assert ((out[:pairs].double() - want).abs() <= bound).all()
        assert (out[pairs] == 7.0).all()
    ops.check_errors(DEV)
