"""The delta rule over portions and single tokens against the same recurrence in float64, at the edges of the chunks in which tokens come
into shared memory, heads that are no multiple of 4, several requests, strided rows.  Everything is float32; a position's output is a sum of D
products whose factors carry some tens of roundings, so 1e-5 of the outputs' root mean square is far above float32 and far below any
error of indexing.  How a request is cut and what shares its steps changes no bit."""
from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def run(proj, wpre, ab, wb, S, lens, H, D, scale):
    from quanta_b200 import kernels
    starts = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device=DEV)
    slots = torch.arange(len(lens), dtype=torch.int32, device=DEV)
    out = torch.full((sum(lens), H, D), float("nan"), device=DEV)
    HD = H * D
    kernels.delta_rule(proj, (0, HD, 2 * HD, 3 * HD), wpre, ab, wb, S, out, starts, slots, H, D, scale, 1e-6)
    return out


def exact(proj, wpre, ab, wb, S, H, D, scale):
    T, HD, p = proj.shape[0], H * D, proj.double()
    r, k, v, a = (p[:, i * HD:(i + 1) * HD].view(T, H, D) for i in range(4))
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    a = torch.sigmoid(a + ab.double().view(H, D))
    w = torch.exp(-scale * torch.sigmoid(wpre.double().view(T, H, D) + wb.double().view(H, D)))
    S, out = S.double(), []
    for t in range(T):
        uS = torch.matmul(u[t][:, None, :], S)
        S = w[t][:, :, None] * S - (a[t] * u[t])[:, :, None] * uS + k[t][:, :, None] * v[t][:, None, :]
        out.append(torch.matmul(r[t][:, None, :], S)[:, 0])
    return torch.stack(out), S


@pytest.mark.parametrize("H,D,lens,extra", [(1, 1, [40], 0), (3, 5, [33, 40], 3), (2, 32, [32], 0), (5, 33, [47, 1, 64], 0), (2, 64, [200, 15, 16, 17], 4),
                                            (4, 100, [90], 0), (2, 128, [65, 31], 8), (3, 64, [1] * 40 + [400], 0), (2, 64, [32], 0)])
@pytest.mark.parametrize("scale", [math.exp(-0.5), 2.5])
def test_chunks(H, D, lens, extra, scale):
    g = torch.Generator(device=DEV).manual_seed(H * 100 + D)
    T, HD = sum(lens), H * D
    proj = torch.randn(T, 4 * HD + extra, device=DEV, generator=g)
    wpre, ab, wb = (torch.randn(n, device=DEV, generator=g) for n in ((T, HD), (HD,), (HD,)))
    wpre[::7] = -40.0                                   # hardly any decay, and the strongest one
    wpre[3::11] = 40.0
    S0 = torch.randn(len(lens), H, D, D, device=DEV, generator=g) * 0.3
    S = S0.clone()
    out = run(proj, wpre, ab, wb, S, lens, H, D, scale)
    at = 0
    for i, n in enumerate(lens):
        want, end = exact(proj[at: at + n], wpre[at: at + n], ab, wb, S0[i], H, D, scale)
        for got, ref in ((out[at: at + n], want), (S[i], end)):
            assert float((got.double() - ref).abs().max()) <= 1e-5 * float(ref.pow(2).mean().sqrt())
        at += n
    # the same tokens a few at a time
    if lens == [200, 15, 16, 17]:
        S1, parts = S0[:1].clone(), []
        for lo in range(0, 200, 16):
            hi = min(200, lo + 16)
            parts.append(run(proj[lo:hi].contiguous(), wpre[lo:hi].contiguous(), ab, wb, S1, [hi - lo], H, D, scale))
        chain = torch.cat(parts)
        assert float((chain - out[:200]).abs().max()) <= 1e-5 * float(chain.pow(2).mean().sqrt())


@pytest.mark.parametrize("R,H,D", [(1, 1, 4), (1, 3, 64), (5, 2, 20), (9, 32, 64), (2, 1, 128), (40, 4, 100), (3, 2, 33)])
def test_single_tokens(R, H, D):
    """One launch for steps of single tokens (heads that are multiples of 4), the state carried over three steps."""
    g = torch.Generator(device=DEV).manual_seed(R + D)
    S0 = torch.randn(R, H, D, D, device=DEV, generator=g) * 0.3
    S, HD = S0.clone(), H * D
    ab, wb = (torch.randn(HD, device=DEV, generator=g) for _ in range(2))
    steps = [(torch.randn(R, 4 * HD + 3, device=DEV, generator=g), torch.randn(R, HD, device=DEV, generator=g)) for _ in range(3)]
    outs = [run(proj, wpre, ab, wb, S, [1] * R, H, D, 0.6) for proj, wpre in steps]
    for r in range(R):
        want, end = exact(torch.stack([p[r] for p, _ in steps]), torch.stack([w[r] for _, w in steps]), ab, wb, S0[r], H, D, 0.6)
        got = torch.stack([o[r] for o in outs])
        for a, b in ((got, want), (S[r], end)):
            assert float((a.double() - b).abs().max()) <= 1e-5 * float(b.pow(2).mean().sqrt())


@pytest.mark.parametrize("H,D,T", [(32, 64, 100), (3, 33, 70), (2, 128, 50), (1, 256, 20), (4, 20, 40), (2, 3, 35)])
def test_cut_and_batch_change_no_bit(H, D, T):
    """One request whole, in portions, one token at a time, as the last of many requests (so that a block has other columns) and beside
    single tokens: the same outputs and the same state, bit by bit."""
    g = torch.Generator(device=DEV).manual_seed(D)
    HD, others = H * D, 7
    proj, wpre = torch.randn(T, 4 * HD, device=DEV, generator=g), torch.randn(T, HD, device=DEV, generator=g)
    ab, wb = (torch.randn(HD, device=DEV, generator=g) for _ in range(2))
    S0 = torch.randn(1, H, D, D, device=DEV, generator=g) * 0.3
    whole = S0.clone()
    out = run(proj, wpre, ab, wb, whole, [T], H, D, 0.6)
    for sizes in ([1] * T, [5, 1, 17] * T, [33] * T):
        S, at, parts = S0.clone(), 0, []
        for n in sizes:
            if at < T:
                parts.append(run(proj[at: at + n].contiguous(), wpre[at: at + n].contiguous(), ab, wb, S, [min(n, T - at)], H, D, 0.6))
                at += n
        assert torch.equal(torch.cat(parts), out) and torch.equal(S, whole)
    for beside in ([1] * others, [T] * 40):
        n = sum(beside)
        more = torch.randn(n, 4 * HD, device=DEV, generator=g), torch.randn(n, HD, device=DEV, generator=g)
        S = torch.cat([torch.randn(len(beside), H, D, D, device=DEV, generator=g), S0])
        got = run(torch.cat([more[0], proj]), torch.cat([more[1], wpre]), ab, wb, S, [*beside, T], H, D, 0.6)
        assert torch.equal(got[n:], out) and torch.equal(S[-1:], whole)
        if beside[0] == 1:      # a step of single tokens in its own kernel
            S, S1 = torch.cat([S[:-1], S0]), S0.clone()
            got = run(torch.cat([more[0], proj[:1]]), torch.cat([more[1], wpre[:1]]), ab, wb, S, [1] * (others + 1), H, D, 0.6)
            alone = run(torch.cat([proj[:1]]), wpre[:1].contiguous(), ab, wb, S1, [1], H, D, 0.6)
            assert torch.equal(got[-1:], out[:1]) and torch.equal(alone, out[:1]) and torch.equal(S[-1:], S1)


def test_a_later_infinity_reaches_no_earlier_token():
    H, D, T = 2, 64, 64
    g = torch.Generator(device=DEV).manual_seed(5)
    proj = torch.randn(T, 4 * H * D, device=DEV, generator=g)
    wpre, ab, wb = torch.randn(T, H * D, device=DEV, generator=g), torch.zeros(H * D, device=DEV), torch.zeros(H * D, device=DEV)
    S0 = torch.randn(1, H, D, D, device=DEV, generator=g)
    clean = run(proj, wpre, ab, wb, S0.clone(), [T], H, D, 0.6)
    for col in (0, H * D, 2 * H * D):                   # r, k, v of token 37
        bad = proj.clone()
        bad[37, col + 3] = float("inf")
        out = run(bad, wpre, ab, wb, S0.clone(), [T], H, D, 0.6)
        assert torch.equal(out[:37], clean[:37]) and not torch.isfinite(out[37:, 0]).all()
