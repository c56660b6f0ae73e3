"""Norms and gates that are launched programmatically (up to 256 rows) between products: a chain of them in a graph and launched one after another
has the bits of the chain that is waited for at every step; more rows and the largest width go the ordinary way with the same bits a row."""
import pytest
import torch

from arle_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows,hidden", [(9, 1024), (64, 4096), (256, 1024), (257, 1024)])
def test_a_chain_of_products_norms_and_gates(rows, hidden):
    g = torch.Generator(device=DEV).manual_seed(rows)
    ff, layers = 2 * hidden, 6
    w1 = (torch.randn(2 * ff, hidden, generator=g, device=DEV) * 0.02).bfloat16()
    w2 = (torch.randn(hidden, ff, generator=g, device=DEV) * 0.02).bfloat16()
    gain = torch.rand(hidden, generator=g, device=DEV) + 0.5
    resid0 = torch.randn(rows, hidden, generator=g, device=DEV)
    resid, delta0 = resid0.clone(), torch.randn(rows, hidden, generator=g, device=DEV).bfloat16()
    delta, x = delta0.clone(), torch.empty_like(delta0)
    gu, act = torch.empty(rows, 2 * ff, dtype=torch.bfloat16, device=DEV), torch.empty(rows, ff, dtype=torch.bfloat16, device=DEV)

    def chain(wait):
        for _ in range(layers):
            for step in (lambda: ops.rmsnorm(resid, delta, None, gain, 1e-6, x, True), lambda: torch.mm(x, w1.t(), out=gu),
                         lambda: ops.silu_mul(gu, act), lambda: torch.mm(act, w2.t(), out=delta)):
                step()
                if wait:
                    torch.cuda.synchronize()

    def run(go):
        resid.copy_(resid0)
        delta.copy_(delta0)
        go()
        torch.cuda.synchronize()
        return resid.clone(), delta.clone()

    want = run(lambda: chain(True))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(False)
    assert want[0].isfinite().all() and not torch.equal(want[0], resid0)
    for _ in range(5):
        for go in (lambda: chain(False), graph.replay):
            got = run(go)
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hidden", [64, 4096, 16384])
def test_a_row_s_bits_do_not_depend_on_the_launch(dtype, hidden):
    g = torch.Generator(device=DEV).manual_seed(hidden)
    resid, delta = torch.randn(300, hidden, generator=g, device=DEV), torch.randn(300, hidden, generator=g, device=DEV).to(dtype)
    extra, gain = torch.randn(300, hidden, generator=g, device=DEV), torch.rand(hidden, generator=g, device=DEV)
    for add in (None, extra):
        a, out = resid.clone(), torch.empty_like(delta)
        ops.rmsnorm(a, delta, None, gain, 1e-6, out, True, 0.5, add)
        b, few = resid[:77].clone(), torch.empty_like(delta[:77])
        ops.rmsnorm(b, delta[:77].contiguous(), None, gain, 1e-6, few, True, 0.5, add if add is None else add[:77].contiguous())
        assert torch.equal(a[:77], b) and torch.equal(out[:77], few)
        x = resid.double() + 0.5 * delta.double() + (0 if add is None else add.double())
        want = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * gain.double()
        assert (out.double() - want).abs().max() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -19) * want.abs().max()
