"""The float32 kernels for few rows (products bound by the weights' bytes), their tile form and the attention of head sizes that are
multiples of 4, each against float64.  Tolerances: a float32 sum of K products in any order is within 2 K 2^-24 sum |x_i w_i| of the
exact one (Higham, Accuracy and Stability of Numerical Algorithms, section 3.1: gamma_K <= 2 K u here)."""
from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = 2.0 ** -24


def K():
    from quanta_b200 import kernels
    return kernels


@pytest.mark.parametrize("n,k,m", [(1, 4, 1), (1, 2048, 33), (2, 132, 7), (3, 516, 130), (4, 4096, 65), (4, 8192, 9), (5, 128, 31),
                                   (8, 2816, 64), (9, 260, 17), (16, 1536, 100), (16, 4096, 5)])
def test_linear_rows(n, k, m):
    g = torch.Generator(device=DEV).manual_seed(n * 1000 + m)
    x, w = torch.randn(n, k, device=DEV, generator=g), torch.randn(m, k, device=DEV, generator=g)
    out = torch.full((n, m), float("nan"), device=DEV)
    K().linear_rows(x, w, out)
    bound = 2 * k * U * (x.double().abs() @ w.double().abs().T)
    assert torch.all((out.double() - x.double() @ w.double().T).abs() <= bound)
    if n > 1:          # a row's sums do not depend on the others, nor on how many there are
        one = torch.empty(1, m, device=DEV)
        K().linear_rows(x[1:2].contiguous(), w, one)
        assert torch.equal(one[0], out[1])


def test_linear_takes_the_library_where_rows_do_not_fit():
    """Inputs that are no whole 16-byte rows, strided or unaligned run as before."""
    from quanta_b200.matmul import linear
    wide = torch.randn(4, 300, device=DEV)
    w = torch.randn(9, 150, device=DEV)
    flat = torch.randn(4 * 128 + 1, device=DEV)
    for x, ww in ((wide[:, :150], w), (wide[:, :148], w[:, :148]), (flat[1:].view(4, 128), torch.randn(5, 128, device=DEV)),
                  (torch.randn(17, 64, device=DEV), torch.randn(5, 64, device=DEV)), (torch.randn(9, 8196, device=DEV), torch.randn(5, 8196, device=DEV))):
        want = x.double() @ ww.double().T
        assert torch.all((linear(x, ww).double() - want).abs() <= 2 * x.shape[1] * U * (x.double().abs() @ ww.double().abs().T))


def test_linear_leaves_to_torch_what_is_torchs():
    """Gradients, forward mode, vmap, autocast, another result type, an empty inner dimension and operands that do not fit: as torch.mm."""
    import torch.autograd.forward_ad as forward_ad
    from torch.func import vmap
    from quanta_b200.matmul import linear
    g = torch.Generator(device=DEV).manual_seed(2)
    x, w = torch.randn(3, 64, device=DEV, generator=g), torch.randn(8, 64, device=DEV, generator=g)
    xg, wg = x.clone().requires_grad_(), torch.nn.Parameter(w.clone())
    linear(xg, wg).sum().backward()
    assert torch.allclose(xg.grad, w.sum(0).expand(3, 64), rtol=1e-4, atol=1e-4) and torch.allclose(wg.grad, x.sum(0).expand(8, 64), rtol=1e-4, atol=1e-4)
    with torch.no_grad():
        assert torch.allclose(linear(xg, wg), x @ w.T, rtol=1e-4, atol=1e-4)
    with forward_ad.dual_level():
        out = linear(forward_ad.make_dual(x, torch.ones_like(x)), w)
        assert torch.allclose(forward_ad.unpack_dual(out).tangent, w.sum(1).expand(3, 8), rtol=1e-4, atol=1e-4)
    many = torch.randn(5, 40, 64, device=DEV, generator=g)
    assert torch.allclose(vmap(lambda t: linear(t, w))(many), many @ w.T, rtol=1e-4, atol=1e-4)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert linear(x, w).dtype == torch.mm(x, w.T).dtype
    for op in (lambda f: f(x, w, torch.bfloat16), lambda f: f(x, w[:, :60].contiguous()), lambda f: f(x, w[0]), lambda f: f(x, w.cpu()),
               lambda f: f(x, w.bfloat16())):
        got = []
        for f in (linear, lambda a, b, dt=None: torch.mm(a, b.t(), out_dtype=dt) if dt else torch.mm(a, b.t())):
            try:
                got.append(op(f).dtype)
            except Exception as e:
                got.append(type(e))
        assert got[0] == got[1], got
    assert torch.equal(linear(x[:, :0], w[:, :0]), torch.zeros(3, 8, device=DEV))


@pytest.mark.parametrize("T,H,I,E,k,mode,kind", [
    (1, 8, 4, 4, 2, 1, 0), (3, 132, 36, 5, 2, 1, 1), (4, 2048, 68, 3, 3, 3, 0), (4, 8192, 20, 4, 1, 1, 0), (7, 64, 100, 6, 4, 1, 0),
    (16, 260, 130, 2, 1, 3, 0), (40, 64, 36, 16, 2, 1, 1), (60, 132, 70, 4, 1, 1, 0), (100, 36, 260, 2, 2, 3, 0)])
def test_expert_products_float32(T, H, I, E, k, mode, kind):
    kern = K()
    g = torch.Generator(device=DEV).manual_seed(T + H)
    x = torch.randn(T, H, device=DEV, generator=g)
    w1 = torch.randn(E, (2 if mode == 1 else 1) * I, H, device=DEV, generator=g) / math.sqrt(H)
    w2 = torch.randn(E, H, I, device=DEV, generator=g) / math.sqrt(I)
    idx = torch.stack([torch.randperm(E, device=DEV, generator=g)[:k] for _ in range(T)]).int()
    if T == 7:
        idx[:, :] = 5                                   # more rows an expert than the step has tokens
    pw = torch.rand(T, k, device=DEV, generator=g) + 0.2
    n = T * k
    words, tiles = kern.moe_plan_sizes(n, E, kern.MOE_SIMT_BM)
    plan, sp = torch.empty(words, device=DEV, dtype=torch.int32), torch.empty(n, device=DEV, dtype=torch.int32)
    te, tr = torch.empty(tiles, device=DEV, dtype=torch.int32), torch.empty(tiles, device=DEV, dtype=torch.int32)
    st = kern.new_status(DEV)
    kern.moe_plan(idx, E, kern.MOE_SIMT_BM, plan, sp, te, tr, st)
    act, y = torch.full((n, I), float("nan"), device=DEV), torch.full((n, H), float("nan"), device=DEV)
    limit, alpha = 1.5, 1.7
    kern.moe_grouped_simt(mode, x, w1, act, sp, pw, plan, te, tr, E, k, act=(kind, limit, alpha))
    kern.moe_grouped_simt(2, act, w2, y, sp, None if kind else pw.view(-1), plan, te, tr, E, k)
    order = sp.long()
    tok, e = order // k, idx.flatten().long()[order]
    xd, scale = x.double()[tok], pw.double().flatten()[order]
    p = torch.einsum("ph,pjh->pj", xd, w1.double()[e])
    size = torch.einsum("ph,pjh->pj", xd.abs(), w1.double().abs()[e]) * 2 * H * U
    if mode == 3:
        want, slope = torch.relu(p) ** 2, 2 * torch.relu(p) + size
    else:
        a, u = p[:, :I], p[:, I:]
        size = size[:, :I] + size[:, I:]
        if kind:
            a, u, size = torch.clamp(a * scale[:, None], max=limit), torch.clamp(u * scale[:, None], -limit, limit), size * 1.2
            want = a * torch.sigmoid(alpha * a) * (u + 1)
        else:
            want = a * torch.sigmoid(a) * u
        slope = 2.0 * (1 + a.abs() + u.abs())            # |d act| <= 1.1 |u + 1| + |a|, and expf is within 2 units
    assert torch.all((act.double() - want).abs() <= slope * size + 16 * U * (want.abs() + 1e-6))
    yw = torch.einsum("pi,pji->pj", act.double(), w2.double()[e])
    ys = torch.einsum("pi,pji->pj", act.double().abs(), w2.double().abs()[e]) * 2 * (I + 2) * U
    if not kind:
        yw, ys = yw * scale[:, None], ys * scale[:, None]
    assert torch.all((y.double()[order] - yw).abs() <= ys + 1e-12)
    assert st.tolist()[0] == 0


@pytest.mark.parametrize("H,I,E,k,mode,kind", [(132, 36, 4, 2, 1, 0), (64, 100, 6, 4, 1, 1), (260, 70, 3, 1, 3, 0), (2048, 68, 8, 2, 1, 0), (36, 260, 2, 2, 3, 0)])
def test_expert_products_do_not_depend_on_the_step(H, I, E, k, mode, kind):
    """A token alone, in a step of few rows an expert (in turns of 16 too), of many, and through the kernel that reads number by number
    (rows that do not start on 16 bytes): the same bits."""
    kern = K()
    T = 130
    g = torch.Generator(device=DEV).manual_seed(H)
    x = torch.randn(T, H, device=DEV, generator=g)
    w1 = torch.randn(E, (2 if mode == 1 else 1) * I, H, device=DEV, generator=g) / math.sqrt(H)
    w2 = torch.randn(E, H, I, device=DEV, generator=g) / math.sqrt(I)
    idx = torch.stack([torch.randperm(E, device=DEV, generator=g)[:k] for _ in range(T)]).int()
    pw = torch.rand(T, k, device=DEV, generator=g) + 0.2

    def run(lo, hi, by=1):
        n, m = (hi - lo) * k, hi - lo
        words, tiles = kern.moe_plan_sizes(n, E, kern.MOE_SIMT_BM)
        plan, sp, te, tr = (torch.empty(c, device=DEV, dtype=torch.int32) for c in (words, n, tiles, tiles))
        st = kern.new_status(DEV)
        kern.moe_plan(idx[lo:hi].contiguous(), E, kern.MOE_SIMT_BM, plan, sp, te, tr, st)
        at = lambda t: t.contiguous() if by else torch.cat([t.new_zeros(1), t.flatten()])[1:].view(t.shape)      # off 16 bytes
        act, y = torch.empty(n * I + 1, device=DEV)[1 - by: n * I + 1 - by].view(n, I), torch.empty(n, H, device=DEV)
        kern.moe_grouped_simt(mode, at(x[lo:hi]), w1, act, sp, pw[lo:hi].contiguous(), plan, te, tr, E, k, act=(kind, 1.5, 1.7))
        kern.moe_grouped_simt(2, act, w2, y, sp, None if kind else pw[lo:hi].contiguous().view(-1), plan, te, tr, E, k)
        assert st.tolist()[0] == 0
        return y.view(m, k, H)

    whole = run(0, T)
    assert torch.equal(run(0, T, by=0), whole)
    for lo, hi in ((0, 1), (5, 7), (9, 12), (20, 27), (40, 53), (60, 90), (0, 64)):
        assert torch.equal(run(lo, hi), whole[lo:hi]), (lo, hi)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq,nkv,hd,vd,page,window,lens", [
    (4, 1, 4, 4, 4, 0, [1, 9]), (6, 3, 64, 64, 8, 0, [70, 3]), (5, 5, 132, 20, 16, 0, [33]), (8, 1, 128, 128, 16, 40, [130, 7, 8]),
    (16, 4, 256, 256, 16, 0, [65]), (3, 1, 60, 256, 5, 11, [40])])
def test_attention_by_rows(dtype, nq, nkv, hd, vd, page, window, lens):
    kern = K()
    g = torch.Generator(device=DEV).manual_seed(hd + nq)
    per = [-(-n // page) for n in lens]
    pages = sum(per) + 2
    kc = torch.randn(pages, nkv, page, hd, device=DEV, generator=g).to(dtype)
    vc = torch.randn(pages, nkv, page, vd, device=DEV, generator=g).to(dtype)
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(1)).int()
    table = torch.full((len(lens), max(per)), -1, dtype=torch.int32)
    at, toks, reqs = 0, [], []
    for r, n in enumerate(lens):
        table[r, : per[r]] = order[at: at + per[r]]
        at += per[r]
        some = sorted({0, n // 2, n - 1})
        toks += some
        reqs += [r] * len(some)
    table = table.to(DEV)
    T = len(toks)
    q = (torch.randn(T, nq, hd, device=DEV, generator=g) * 2).to(dtype)
    pos, req = torch.tensor(toks, dtype=torch.int32, device=DEV), torch.tensor(reqs, dtype=torch.int32, device=DEV)
    out = torch.full((T, nq, vd), float("nan"), device=DEV, dtype=dtype)
    st = kern.new_status(DEV)
    kern.paged_attention_simt(q, kc, vc, out, pos, req, table, hd ** -0.5, window, st)
    for t in range(T):
        lo = max(0, toks[t] - window + 1) if window else 0
        keys = torch.arange(lo, toks[t] + 1, device=DEV)
        rows = table[reqs[t]].long()[keys // page]
        k, v = kc[rows, :, keys % page].double(), vc[rows, :, keys % page].double()
        for h in range(nq):
            s = (k[:, h // (nq // nkv)] @ q[t, h].double()) * hd ** -0.5
            want = torch.softmax(s, 0) @ v[:, h // (nq // nkv)]
            # scores within 2 hd U sum |q k| scale of the exact ones move the weights by as much relatively; then one rounding
            off = 2 * (2 * hd * U * float((k[:, h // (nq // nkv)].abs() @ q[t, h].double().abs()).max()) * hd ** -0.5 + (len(keys) + 16) * U)
            tol = off * float(v.abs().max()) + (2.0 ** -8 * float(want.abs().max()) if dtype == torch.bfloat16 else 0.0)
            assert float((out[t, h].double() - want).abs().max()) <= tol
    assert st.tolist()[0] == 0
    table[0, 0] = pages + 3                            # a page outside the pool is recorded, its keys are passed over
    kern.paged_attention_simt(q, kc, vc, out, pos, req, table, hd ** -0.5, 0, st)
    assert st.tolist()[0] == 2 and torch.isfinite(out.float()).all()
