"""q/k norm, rotation and the write into the pages for heads of 128 (kept in registers, two, four or eight heads a warp) against float64, on
both sides of every line of its launch rule, with every option.  Tolerance: a dozen float32 roundings of numbers up to some ten (an
angle, its sine and a sum of 128 squares among them), 2^-8 where the result is bfloat16."""
from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
HD = 128


def _case(T, nq, nkv, rd=128, norm="layer", interleaved=False, tied=False, bias=False, blend=False, scale=False, temp=0, page=16, wide=0,
          dtype=torch.bfloat16, rows=torch.bfloat16, has_kv=True):
    return dict(T=T, nq=nq, nkv=nkv, rd=rd, norm=norm, interleaved=interleaved, tied=tied, bias=bias, blend=blend, scale=scale, temp=temp,
                page=page, wide=wide, dtype=dtype, rows=rows, has_kv=has_kv)


F32 = torch.float32
CASES = [
    # tokens on both sides of 64 (two heads a warp, or four and eight), heads on both sides of 32, 64 and 128
    *[_case(T, nq, nkv) for T in (1, 64, 65) for nq, nkv in ((1, 1), (28, 2), (29, 2), (48, 8), (61, 2), (120, 4))],
    _case(2, 121, 4), _case(66, 125, 2, rd=64), _case(70, 48, 8, norm="head"), _case(3, 16, 4, norm="none", rd=0),
    # both layouts of the pairs, whole, in part and not at all
    *[_case(T, 6, 3, rd=rd, interleaved=i) for T in (5, 67) for rd, i in ((0, False), (64, False), (8, False), (120, False), (128, True), (4, True), (64, True))],
    _case(9, 4, 2, rd=12), _case(70, 4, 2, rd=6, interleaved=True),                       # pairs that fall into a lane's piece: element by element
    *[_case(T, 8, 2, norm=n) for T in (7, 80) for n in ("head", "head without gains", "none")],
    *[_case(T, 8, 2, tied=True, bias=True, norm="head", rd=64) for T in (4, 65)],
    *[_case(T, 12, 4, bias=True, blend=True, scale=True, temp=16, rows=F32) for T in (6, 130)],
    *[_case(T, 12, 4, blend=True, dtype=F32, rows=F32, wide=8, page=5) for T in (33, 66)],
    _case(12, 8, 8, page=7, wide=3), _case(75, 8, 8, page=7, wide=16), _case(20, 16, 4, has_kv=False, norm="head"), _case(90, 40, 4, has_kv=False),
]


@pytest.mark.parametrize("c", CASES, ids=lambda c: "-".join(str(v).replace("torch.", "") for v in c.values()))
def test_heads_of_128(c):
    from quanta_b200 import kernels as k
    T, nq, nkv, rd, page = c["T"], c["nq"], c["nkv"], c["rd"], c["page"]
    nk = nkv if c["has_kv"] else 0
    g = torch.Generator(device=DEV).manual_seed(T * 1000 + nq)
    randn = lambda *s: torch.randn(*s, device=DEV, generator=g)
    n_row = (nq + nk * (1 if c["tied"] else 2)) * HD
    whole = (randn(T, n_row + c["wide"]) * 2).to(c["rows"])
    layer, gained = c["norm"] == "layer", c["norm"] in ("layer", "head")
    qw = 1 + 0.2 * randn(nq * HD if layer else HD) if gained else None
    kw = 1 + 0.2 * randn(nkv * HD if layer else HD) if gained and nk else None
    kind = {"layer": k.NORM_PER_LAYER, "none": k.NORM_NONE}.get(c["norm"], k.NORM_PER_HEAD)
    inv = (1e4 ** (-torch.arange(rd // 2, device=DEV) * 2 / max(rd, 1))).float()
    bias = randn(n_row) if c["bias"] else None
    first, lam = (randn(T, nkv * HD), torch.full((1,), 0.3, device=DEV)) if c["blend"] else (None, None)
    export = torch.full((T, nkv * HD), 7.0, device=DEV) if c["blend"] else None
    scale = 0.5 + torch.rand(nq, device=DEV, generator=g) if c["scale"] else None
    starts = {0: 0, 1: 37}                                            # two requests, the second from position 37 on
    req = torch.tensor([0 if t < (T + 1) // 2 else 1 for t in range(T)], dtype=torch.int32)
    pos = torch.tensor([t if r == 0 else starts[1] + t - (T + 1) // 2 for t, r in enumerate(req.tolist())], dtype=torch.int32)
    per = -(-(T + 40) // page)
    table = torch.randperm(2 * per, generator=torch.Generator().manual_seed(1)).int().view(2, per)
    kc, vc = (torch.full((2 * per, nkv, page, HD), 5.0, device=DEV, dtype=c["dtype"]) for _ in range(2)) if nk else (None, None)
    q, st = torch.empty(T, nq, HD, device=DEV, dtype=c["dtype"]), k.new_status(DEV)
    dev = lambda t: t.to(DEV)

    def run(tbl):
        k.qknorm_rope_write(whole, q, kc, vc, qw, kw, kind, 1e-5, inv, None, dev(pos), dev(pos), dev(req), dev(tbl), nq, nkv, HD, rd, page, st,
                            has_kv=c["has_kv"], q_temp_coef=0.1, q_temp_every=c["temp"], bias=bias, v_first=first, v_lambda=lam,
                            v_export=export, head_scale=scale, interleaved=c["interleaved"], tied_values=c["tied"])

    run(table)
    assert st.tolist()[0] == 0
    x = whole[:, :n_row].double() + (bias.double() if c["bias"] else 0)
    heads = x.view(T, -1, HD)
    qk, v = heads[:, : nq + nk], heads[:, nq: nq + nk] if c["tied"] else heads[:, nq + nk:]
    if layer:
        parts = [t.reshape(T, -1) for t in (qk[:, :nq], qk[:, nq:])]
        qk = torch.cat([(t * torch.rsqrt((t * t).mean(-1, keepdim=True) + 1e-5) * w.double()).view(T, -1, HD) for t, w in zip(parts, (qw, kw)) if t.numel()], 1)
    elif kind == k.NORM_PER_HEAD:
        qk = qk * torch.rsqrt((qk * qk).mean(-1, keepdim=True) + 1e-5)
        if gained:
            qk = torch.cat([qk[:, :nq] * qw.double(), *([qk[:, nq:] * kw.double()] if nk else [])], 1)
    ang = (dev(pos).float()[:, None] * inv).double()                  # the angle is a float32 product
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]
    a, b = (qk[..., 0:rd:2], qk[..., 1:rd:2]) if c["interleaved"] else (qk[..., : rd // 2], qk[..., rd // 2: rd])
    ra, rb = a * cos - b * sin, b * cos + a * sin
    turned = torch.stack([ra, rb], -1).flatten(-2) if c["interleaved"] else torch.cat([ra, rb], -1)
    qk = torch.cat([turned, qk[..., rd:]], -1)
    want_q = qk[:, :nq]
    if c["temp"]:
        want_q = want_q * (1 + 0.1 * torch.log(((dev(pos) + 1) // c["temp"]).double() + 1))[:, None, None]
    if c["scale"]:
        want_q = want_q * scale.double()[None, :, None]

    def near(got, want):
        tol = 2.0 ** -8 if got.dtype == torch.bfloat16 else 2.0 ** -18
        assert torch.all((got.double() - want).abs() <= tol * want.abs() + 2.0 ** -18 * float(want.abs().max()))

    near(q, want_q)
    if not nk:
        return
    rows = dev(table)[dev(req).long(), (dev(pos) // page).long()].long()
    at = (dev(pos) % page).long()
    near(kc[rows, :, at], qk[:, nq:])
    near(vc[rows, :, at], 0.7 * v + 0.3 * first.double().view(T, nkv, HD) if c["blend"] else v)
    if c["blend"]:
        near(export.view(T, nkv, HD), v)
    written = torch.zeros(2 * per, page, dtype=torch.bool, device=DEV)
    written[rows, at] = True
    for cache in (kc, vc):                                            # no other slot is touched
        assert torch.all(cache.transpose(1, 2)[~written] == 5.0)
    # a page outside the pool is recorded, its token's queries are still there and nothing is written
    before = kc.clone()
    bad = table.clone()
    bad[0, 0] = 2 * per
    kept = q.clone()
    run(bad)
    assert st.tolist()[0] == 2 and torch.equal(q, kept) and torch.equal(kc, before)


@pytest.mark.parametrize("c", [c for c in CASES if c["T"] > 64], ids=lambda c: "-".join(str(v).replace("torch.", "") for v in c.values()))
def test_a_tokens_numbers_do_not_depend_on_the_step(c):
    """Steps on both sides of 64 tokens (a warp a head, half a warp a head): the same bits."""
    from quanta_b200 import kernels as k
    T, nq, nkv, rd, page = c["T"], c["nq"], c["nkv"], c["rd"], c["page"]
    nk = nkv if c["has_kv"] else 0
    g = torch.Generator(device=DEV).manual_seed(T + nq)
    randn = lambda *s: torch.randn(*s, device=DEV, generator=g)
    n_row = (nq + nk * (1 if c["tied"] else 2)) * HD
    rows = (randn(T, n_row) * 2).to(c["rows"])
    layer, gained = c["norm"] == "layer", c["norm"] in ("layer", "head")
    qw = 1 + 0.2 * randn(nq * HD if layer else HD) if gained else None
    kw = 1 + 0.2 * randn(nkv * HD if layer else HD) if gained and nk else None
    kind = {"layer": k.NORM_PER_LAYER, "none": k.NORM_NONE}.get(c["norm"], k.NORM_PER_HEAD)
    inv = (1e4 ** (-torch.arange(rd // 2, device=DEV) * 2 / max(rd, 1))).float()
    bias = randn(n_row) if c["bias"] else None
    pos, req = torch.arange(T, dtype=torch.int32, device=DEV), torch.zeros(T, dtype=torch.int32, device=DEV)
    pages = -(-T // page)
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(1)).int().view(1, pages).to(DEV)

    def run(step):
        q, st = torch.empty(T, nq, HD, device=DEV, dtype=c["dtype"]), k.new_status(DEV)
        kc, vc = (torch.zeros((pages, nkv, page, HD), device=DEV, dtype=c["dtype"]) for _ in range(2)) if nk else (None, None)
        for t in range(0, T, step):
            s = slice(t, min(T, t + step))
            k.qknorm_rope_write(rows[s], q[s], kc, vc, qw, kw, kind, 1e-5, inv, None, pos[s], pos[s], req[s], table, nq, nkv, HD, rd, page, st,
                                has_kv=c["has_kv"], bias=bias, interleaved=c["interleaved"], tied_values=c["tied"])
        assert st.tolist()[0] == 0
        return [t for t in (q, kc, vc) if t is not None]

    for many, few in zip(run(T), run(33)):
        assert torch.equal(many, few)
