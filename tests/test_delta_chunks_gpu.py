"""The gated delta rule in chunks on the tensor cores against float64: lengths around the first row that runs in chunks and around a chunk's
end, long rows beside short ones, columns that do not fill a block, shared q/k heads; no further off than the scan of whole rows; a row's
bits do not depend on what stands beside it; decays of zero, and an overflow that stays with the tokens behind it."""
import pytest
import torch

from arle_b200 import ops
from launched import launched

pytestmark = pytest.mark.gpu
DEV, DIM = "cuda", 128


def _inputs(lens, H, kq, vdim):
    g = torch.Generator(device=DEV).manual_seed(vdim + sum(lens))
    T = sum(lens)
    wide = torch.nn.functional.silu(torch.randn(T, 2 * kq * DIM + H * vdim, generator=g, device=DEV) * 0.7).to(torch.bfloat16)
    q, k, v = wide.split([kq * DIM, kq * DIM, H * vdim], 1)
    beta = torch.sigmoid(torch.randn(T, H, generator=g, device=DEV))
    decay = torch.exp(-torch.rand(T, H, generator=g, device=DEV) * 0.3)
    return q, k, v, beta, decay, torch.randn(len(lens) + 1, H * vdim * DIM + 8, generator=g, device=DEV)


def _run(q, k, v, beta, decay, state, lens, H, kq, vdim, chunks=True, slots=None, eps=1e-6):
    at = torch.tensor([0] + lens, dtype=torch.int32, device=DEV).cumsum(0).to(torch.int32)
    out = torch.full((q.shape[0] + 1, H, vdim), 7.0, device=DEV)
    state, n = state.clone(), ops.delta_scan_scratch(q.shape[0], len(lens), H)
    assert n > 0 and ops.delta_scan_takes_chunks(q, vdim, DIM, max(lens))
    scratch = torch.full((n + 4,), float("nan"), device=DEV)
    slots = torch.tensor(slots or list(range(len(lens))), dtype=torch.int32, device=DEV)
    ops.delta_scan(q, k, v, beta, decay, state, at, slots, out[:-1], H, kq, DIM, vdim, DIM ** -0.5, eps,
                   **(dict(max_q_len=max(lens), scratch=scratch[:n]) if chunks else {}))
    assert (out[-1] == 7.0).all() and scratch[n:].isnan().all()
    return out[:-1], state


def _exact(q, k, v, beta, decay, state, lens, H, kq, vdim, eps=1e-6):
    def unit(x):
        x = x.double().view(-1, kq, DIM)
        return (x * torch.rsqrt(x.square().sum(-1, keepdim=True) + eps)).repeat_interleave(H // kq, 1)

    qq, kk, vv = unit(q) * DIM ** -0.5, unit(k), v.double().view(-1, H, vdim)
    S, outs, t = state[:, : H * vdim * DIM].double().view(-1, H, vdim, DIM).clone(), [], 0
    for r, n in enumerate(lens):
        for _ in range(n):
            S[r] *= decay[t].double()[:, None, None]
            u = beta[t].double()[:, None] * (vv[t] - torch.einsum("hvd,hd->hv", S[r], kk[t]))
            S[r] += u[..., None] * kk[t][:, None]
            outs.append(torch.einsum("hvd,hd->hv", S[r], qq[t]))
            t += 1
    return torch.stack(outs), S.reshape(S.shape[0], -1)


@pytest.mark.parametrize("lens", [[80], [127], [128], [129], [1000], [5, 200, 1, 79, 80, 333], [1] * 40 + [190]])
@pytest.mark.parametrize("H,kq,vdim", [(2, 2, 128), (4, 2, 40), (1, 1, 8)])
def test_chunks(lens, H, kq, vdim):
    x = _inputs(lens, H, kq, vdim)
    want, want_s = _exact(*x, lens, H, kq, vdim)
    got, got_s = _run(*x, lens, H, kq, vdim)
    whole, whole_s = _run(*x, lens, H, kq, vdim, chunks=False)
    used = H * vdim * DIM
    for a, b, w in ((got, whole, want), (got_s[:, :used], whole_s[:, :used], want_s)):
        off, ref = ((y.double() - w).norm() / w.norm() for y in (a, b))
        assert off < 4e-7 and off < 1.3 * ref + 2e-8           # the float32 sums of both come in different orders
    assert torch.equal(got_s[:, used:], x[-1][:, used:])
    t = 0
    for r, n in enumerate(lens):                                # a row by itself: the same bits
        if n < 80:
            assert torch.equal(got[t: t + n], whole[t: t + n])
        else:
            alone, s = _run(*(y[t: t + n] for y in x[:-1]), x[-1], [n], H, kq, vdim, slots=[r])
            assert torch.equal(alone, got[t: t + n]) and torch.equal(s[r], got_s[r])
        t += n


def test_decays_of_zero_and_overflow():
    lens, H, kq, vdim = [150], 2, 1, 48
    q, k, v, beta, decay, state = _inputs(lens, H, kq, vdim)
    decay[::13] = 0.0
    decay[5::17, 0] = 1e-30
    want, want_s = _exact(q, k, v, beta, decay, state, lens, H, kq, vdim)
    got, got_s = _run(q, k, v, beta, decay, state, lens, H, kq, vdim)
    assert (got.double() - want).norm() < 4e-7 * want.norm()
    assert (got_s[0, : want_s.shape[1]].double() - want_s[0]).norm() < 4e-7 * want_s[0].norm()
    decay[:] = 0.97
    clean, _ = _run(q, k, v, beta, decay, state, lens, H, kq, vdim)
    bad = v.clone()
    bad[75, 3] = float("inf")                                   # one head's column, in the middle of a tile
    odd, _ = _run(q, k, bad, beta, decay, state, lens, H, kq, vdim)
    close = dict(rtol=1e-5, atol=1e-6)
    assert torch.allclose(odd[:75], clean[:75], **close) and not odd[75:, 0, 3].isfinite().any()
    assert torch.equal(odd[:, 1], clean[:, 1])
    odd[:, 0, 3] = clean[:, 0, 3]
    assert torch.allclose(odd, clean, **close)                  # the other columns as they were
    worse = k.clone()
    worse[75, 4] = float("nan")
    odd, _ = _run(q, worse, v, beta, decay, state, lens, H, kq, vdim)
    assert torch.allclose(odd[:75], clean[:75], **close) and not odd[75:].isfinite().any()


@pytest.mark.parametrize("lens", [[81], [128], [100, 5, 229]])
def test_lengths_without_an_epsilon(lens):
    """The places behind a row's end have q and k of zeros, whose length has no inverse: they stay out of the memory all the same."""
    H, kq, vdim = 3, 1, 40
    x = _inputs(lens, H, kq, vdim)
    want, want_s = _exact(*x, lens, H, kq, vdim, eps=0.0)
    got, got_s = _run(*x, lens, H, kq, vdim, eps=0.0)
    whole, whole_s = _run(*x, lens, H, kq, vdim, chunks=False, eps=0.0)
    used = H * vdim * DIM
    for a, b, w in ((got, whole, want), (got_s[:-1, :used], whole_s[:-1, :used], want_s[:-1])):
        off, ref = ((y.double() - w).norm() / w.norm() for y in (a, b))
        assert off < 4e-7 and off < 1.3 * ref + 2e-8


@pytest.mark.parametrize("lens,spare", [([100, 5], 0), ([300, 5], 1), ([81], 3), ([2, 79, 64], 0), ([100, 90, 229], 0)])
@pytest.mark.parametrize("say", [dict(), dict(max_q_len=200), dict(max_q_len=40), "q_lens"], ids=str)
def test_every_row_runs(lens, spare, say):
    """Whatever is said about the rows' lengths, short rows beside long ones run, also where the arrays have more rows than q_indptr ends at."""
    H, kq, vdim = 2, 1, 64
    *x, state = _inputs(lens + [spare] if spare else lens, H, kq, vdim)
    T, n = sum(lens), ops.delta_scan_scratch(sum(lens) + spare, len(lens), H)
    at = torch.tensor([0] + lens, dtype=torch.int32, device=DEV).cumsum(0).to(torch.int32)
    slots = torch.arange(len(lens), dtype=torch.int32, device=DEV)
    got = []
    for kw in (dict(scratch=torch.empty(n, device=DEV), **(dict(q_lens=lens) if say == "q_lens" else say)), {}):
        s, out = state.clone(), torch.full((T + spare, H, vdim), 7.0, device=DEV)
        ops.delta_scan(*x, s, at, slots, out, H, kq, DIM, vdim, DIM ** -0.5, 1e-6, **kw)
        got.append((out, s))
    (a, sa), (b, sb) = got
    assert (a[T:] == 7.0).all() and not (a[:T] == 7.0).any()
    assert (a - b).norm() < 1e-6 * b.norm() and (sa - sb).norm() < 1e-6 * sb.norm()


def test_lengths_that_are_not_the_rows():
    *x, state = _inputs([100, 5], 1, 1, 8)
    at, slots = (torch.tensor(v, dtype=torch.int32, device=DEV) for v in ([0, 100, 105], [0, 1]))
    for lens in ([105], [100, 6]):
        with pytest.raises(ops.KernelError):
            ops.delta_scan(*x, state, at, slots, torch.empty(105, 1, 8, device=DEV), 1, 1, DIM, 8, DIM ** -0.5, 1e-6,
                           scratch=torch.empty(ops.delta_scan_scratch(105, 2, 1), device=DEV), q_lens=lens)


@pytest.mark.parametrize("H,vdim,n", [(8, 128, 2048), (32, 128, 300), (1, 16, 80)])
def test_launches_go_by_the_rows_that_they_run(H, vdim, n):
    """A long row beside decoded tokens takes the chunks' kernel that it takes by itself, and the decoded tokens the scan that they take by
    themselves, with the bits that rows among their like have."""
    def step(lens):
        *x, state = _inputs(lens, H, H, vdim)
        at = torch.tensor([0] + lens, dtype=torch.int32, device=DEV).cumsum(0).to(torch.int32)
        slots, out = torch.arange(len(lens), dtype=torch.int32, device=DEV), torch.empty(sum(lens), H, vdim, device=DEV)
        kw = dict(scratch=torch.empty(ops.delta_scan_scratch(sum(lens), len(lens), H), device=DEV), q_lens=lens) if max(lens) >= 80 else {}
        return launched(lambda: ops.delta_scan(*x, state, at, slots, out, H, H, DIM, vdim, DIM ** -0.5, 1e-6, **kw), r"delta_\w+_kernel(<.*?>(?=\())?")

    alone, decoded, both = step([n]), step([1] * 12), step([n] + [1] * 12)
    assert len(alone) == 2 and len(decoded) == 1 and both == alone | decoded
