"""The attention of single tokens whose operands come straight from the cache rows, against float64: one to eight q heads a kv head, pages of
any size, contexts at the edges of its rounds of 16 keys, of a block's warps and of the blocks of a cluster, windows.  Tolerance: weights and
output are rounded to bfloat16 (2^-9 each, relative to the largest value), scores are float32."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def K():
    from quanta_b200 import kernels
    return kernels


@pytest.mark.parametrize("nq,nkv,page,lens,window", [
    (48, 8, 16, [1], 0), (48, 8, 16, [2100], 0), (6, 1, 16, [16, 17, 15, 128, 129, 1024, 1025], 0), (8, 1, 5, [333], 0), (2, 2, 64, [40] * 9, 0),
    (16, 4, 16, [700, 3, 5000], 300), (7, 1, 128, [257], 16), (12, 4, 8, [600 + 7 * i for i in range(40)], 0), (4, 4, 16, [90] * 160, 33),
    (5, 5, 16, [2000] * 30, 0)])
def test_decode_direct(nq, nkv, page, lens, window):
    kern, hd, G = K(), 128, nq // nkv
    assert kern.attn_decode_direct_supported(nq, nkv, hd)
    g = torch.Generator(device=DEV).manual_seed(len(lens) + nq)
    per = [-(-n // page) for n in lens]
    pages = sum(per) + 1
    kc = torch.randn(pages, nkv, page, hd, device=DEV, generator=g).bfloat16()
    vc = torch.randn(pages, nkv, page, hd, device=DEV, generator=g).bfloat16()
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(2)).int()
    table = torch.full((len(lens), max(per)), -1, dtype=torch.int32)
    at = 0
    for r, n in enumerate(lens):
        table[r, : per[r]] = order[at: at + per[r]]
        at += per[r]
        if window:
            table[r, : max(0, n - window) // page] = -1            # given back
    table = table.to(DEV)
    R = len(lens)
    q = (torch.randn(R + 2, nq, hd, device=DEV, generator=g) * 1.5).bfloat16()
    rows = torch.randperm(R + 2, generator=torch.Generator().manual_seed(5))[:R].int()      # single tokens beside others of the step
    pos, req = torch.zeros(R + 2, dtype=torch.int32), torch.zeros(R + 2, dtype=torch.int32)
    for r, t in enumerate(rows.tolist()):
        pos[t], req[t] = lens[r] - 1, r
    out = torch.full((R + 2, nq, hd), 7.0, device=DEV, dtype=torch.bfloat16)
    st = kern.new_status(DEV)
    kern.attn_decode_direct(q, kc, vc, out, rows.to(DEV), R, pos.to(DEV), req.to(DEV), table, hd ** -0.5, window, max(lens) + 100, st)
    assert st.tolist()[0] == 0
    for r, t in enumerate(rows.tolist()):
        j = torch.arange(max(0, lens[r] - window) if window else 0, lens[r], device=DEV)
        row = table[r].long()[j // page]
        k, v = kc[row, :, j % page].double(), vc[row, :, j % page].double()
        s = torch.einsum("hgd,jhd->hgj", q[t].double().view(nkv, G, hd), k) * hd ** -0.5
        want = torch.einsum("hgj,jhd->hgd", torch.softmax(s, -1), v).reshape(nq, hd)
        assert float((out[t].double() - want).abs().max()) <= 2.0 ** -8 * float(v.abs().max())
    others = [t for t in range(R + 2) if t not in rows.tolist()]
    assert torch.all(out[others] == 7.0)
    table[0, (lens[0] - 1) // page] = pages                        # a page outside the pool is recorded
    kern.attn_decode_direct(q, kc, vc, out, rows.to(DEV), R, pos.to(DEV), req.to(DEV), table, hd ** -0.5, window, max(lens), st)
    assert st.tolist()[0] == 2 and torch.isfinite(out.float()).all()


@pytest.mark.parametrize("lens,window,chunk,cap", [([700, 1, 31], 300, 0, 30.0), ([1500] * 16, 1024, 0, 5.0), ([2100], 0, 128, 0.0),
                                                   ([128, 129, 127, 256], 0, 128, 0.0), ([5000], 0, 0, 0.0), ([90] * 50, 17, 0, 0.0)])
def test_weights_of_two_parts(lens, window, chunk, cap):
    """As above with weights that hold 16 bits: 2^-12 of the largest value for them and their scores, and the output's rounding."""
    kern, hd, nq, nkv, page = K(), 128, 16, 4, 16
    g = torch.Generator(device=DEV).manual_seed(len(lens))
    per = [-(-n // page) for n in lens]
    kc = torch.randn(sum(per), nkv, page, hd, device=DEV, generator=g).bfloat16()
    vc = torch.randn(sum(per), nkv, page, hd, device=DEV, generator=g).bfloat16()
    table, at = torch.full((len(lens), max(per)), -1, dtype=torch.int32), 0
    for r, n in enumerate(lens):
        table[r, : per[r]] = torch.arange(at, at + per[r], dtype=torch.int32)
        at += per[r]
    table = table.to(DEV)
    R = len(lens)
    q = (torch.randn(R, nq, hd, device=DEV, generator=g) * 1.5).bfloat16()
    pos, req = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV), torch.arange(R, dtype=torch.int32, device=DEV)
    out, st = torch.empty_like(q), kern.new_status(DEV)
    kern.attn_decode_direct(q, kc, vc, out, req, R, pos, req, table, hd ** -0.5, window, max(lens), st, two_part=True, softcap=cap, chunk=chunk)
    assert st.tolist()[0] == 0
    for r, n in enumerate(lens):
        lo = (n - 1) // chunk * chunk if chunk else max(0, n - window) if window else 0
        j = torch.arange(lo, n, device=DEV)
        row = table[r].long()[j // page]
        k, v = kc[row, :, j % page].double(), vc[row, :, j % page].double()
        s = torch.einsum("hgd,jhd->hgj", q[r].double().view(nkv, nq // nkv, hd), k) * hd ** -0.5
        s = cap * torch.tanh(s / cap) if cap else s
        want = torch.einsum("hgj,jhd->hgd", torch.softmax(s, -1), v).reshape(nq, hd)
        assert torch.all((out[r].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -12 * float(v.abs().max()))


@pytest.mark.parametrize("two_part", [False, True])
@pytest.mark.parametrize("lens", [[40, 2100], [300] * 40])
def test_what_is_no_number_stays_none(two_part, lens):
    """A query, a key or a value that holds NaN gives NaN to the heads (and dims) that meet it and to no other."""
    kern, hd, nq, nkv, page = K(), 128, 8, 2, 16
    g = torch.Generator(device=DEV).manual_seed(1)
    per = [-(-n // page) for n in lens]
    kc = torch.randn(sum(per), nkv, page, hd, device=DEV, generator=g).bfloat16()
    vc = torch.randn(sum(per), nkv, page, hd, device=DEV, generator=g).bfloat16()
    table, at = torch.full((len(lens), max(per)), -1, dtype=torch.int32), 0
    for r, n in enumerate(per):
        table[r, :n] = torch.arange(at, at + n, dtype=torch.int32)
        at += n
    R = len(lens)
    q = torch.randn(R, nq, hd, device=DEV, generator=g).bfloat16()
    pos, req = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV), torch.arange(R, dtype=torch.int32, device=DEV)

    def run(q_, k_, v_):
        out, st = torch.empty_like(q), kern.new_status(DEV)
        kern.attn_decode_direct(q_, k_, v_, out, req, R, pos, req, table.to(DEV), hd ** -0.5, 0, max(lens), st, two_part=two_part)
        assert st.tolist()[0] == 0
        return out

    clean = run(q, kc, vc)
    where = (torch.tensor(per[:1]).sum().item(), 1, 5)                # token 1's key 5, kv head 1: its q heads 4 .. 7
    for name in ("q", "k", "v"):
        qq, kk, vv = q.clone(), kc.clone(), vc.clone()
        hit = torch.zeros(R, nq, hd, dtype=torch.bool, device=DEV)
        if name == "q":
            qq[1, 6, 17] = float("nan")
            hit[1, 6] = True
        elif name == "k":
            kk[where][3] = float("nan")
            hit[1, 4:] = True
        else:
            vv[where][100] = float("nan")
            hit[1, 4:, 100] = True
        out = run(qq, kk, vv)
        assert torch.isnan(out[hit].float()).all() and torch.equal(out[~hit], clean[~hit])


@pytest.mark.parametrize("R,n,window,cap", [(16, 1500, 1024, 30.0), (32, 700, 0, 0.0), (4, 9000, 0, 5.0)])
def test_weights_hold_24_bits(R, n, window, cap):
    """The share of outputs that are not the bfloat16 nearest to the exact value.  Queries are short, so that the weights are near one
    another and all of them count: an error of e in each weight, independent of the others, moves an output by some e / 2 of its
    size, and a bfloat16 boundary lies within that of it for e / 2^-8 of the outputs.  Weights of 16 bits (e = 2^-17) put 2e-3 of them
    on the wrong side (measured 1.4e-3 to 3.1e-3), float32 arithmetic throughout 1e-4 to 7e-4 (scores of 128 products)."""
    kern, hd, nq, nkv, page = K(), 128, 16, 4, 16
    g = torch.Generator(device=DEV).manual_seed(n)
    per = -(-n // page)
    kc = torch.randn(R * per, nkv, page, hd, device=DEV, generator=g).bfloat16()
    vc = torch.randn(R * per, nkv, page, hd, device=DEV, generator=g).bfloat16()
    table = torch.arange(R * per, dtype=torch.int32, device=DEV).view(R, per)
    q = (torch.randn(R, nq, hd, device=DEV, generator=g) * 0.3).bfloat16()
    pos, req = torch.full((R,), n - 1, dtype=torch.int32, device=DEV), torch.arange(R, dtype=torch.int32, device=DEV)
    lo = max(0, n - window) if window else 0
    k, v = (c.view(R, per, nkv, page, hd).transpose(1, 2).reshape(R, nkv, per * page, hd)[:, :, lo:n].double() for c in (kc, vc))
    s = torch.einsum("rmgd,rmjd->rmgj", q.double().view(R, nkv, nq // nkv, hd), k) * hd ** -0.5
    s = cap * torch.tanh(s / cap) if cap else s
    want = torch.einsum("rmgj,rmjd->rmgd", torch.softmax(s, -1), v).reshape(R, nq, hd).bfloat16()
    out, st = torch.empty_like(q), kern.new_status(DEV)
    kern.attn_decode_direct(q, kc, vc, out, req, R, pos, req, table, hd ** -0.5, window, n, st, two_part=True, softcap=cap)
    assert st.tolist()[0] == 0 and float((out != want).float().mean()) <= 9e-4


@pytest.mark.parametrize("two_part", [False, True])
@pytest.mark.parametrize("batch,length,page,nq,nkv,window", [(1, 131072, 16, 6, 1, 0), (4, 131072, 16, 6, 1, 0), (2, 9100, 4, 4, 2, 0), (40, 20000, 64, 16, 4, 0),
                                                           (3, 131072, 16, 8, 1, 70000)])
def test_long_contexts(batch, length, page, nq, nkv, window, two_part):
    """Many rounds of the ring, clusters of eight blocks at full length, tables of more than 2,048 pages; one far key carries a row."""
    kern, hd = K(), 128
    g = torch.Generator(device=DEV).manual_seed(batch + page)
    per = -(-length // page)
    kc = torch.empty(batch * per, nkv, page, hd, device=DEV, dtype=torch.bfloat16).normal_(generator=g)
    vc = torch.empty(batch * per, nkv, page, hd, device=DEV, dtype=torch.bfloat16).normal_(generator=g)
    table = torch.randperm(batch * per, generator=torch.Generator().manual_seed(4)).int().view(batch, per)
    lens = [max(1, length - 37 * r * r) for r in range(batch)]
    q = torch.randn(batch, nq, hd, device=DEV, generator=g).bfloat16()
    far = max(0, lens[0] - window) if window else 1
    page_of, slot = int(table[0, far // page]), far % page
    kc[page_of, :, slot] = 0
    kc[page_of, :, slot, 0] = 30.0
    q[0, : nq // 2, 0] = 8.0
    pos, req = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV), torch.arange(batch, dtype=torch.int32, device=DEV)
    table = table.to(DEV)
    out, st = torch.full_like(q, float("nan")), kern.new_status(DEV)
    kern.attn_decode_direct(q, kc, vc, out, req, batch, pos, req, table, hd ** -0.5, window, length, st, two_part=two_part)
    assert st.tolist()[0] == 0
    for r in {0, batch // 2, batch - 1}:
        j = torch.arange(max(0, lens[r] - window) if window else 0, lens[r], device=DEV)
        rows = table[r].long()[j // page]
        for m in range(nkv):
            k, v = kc[rows, m, j % page].double(), vc[rows, m, j % page].double()
            G = nq // nkv
            w = torch.softmax(q[r, m * G: (m + 1) * G].double() @ k.T * hd ** -0.5, -1)
            # rounded weights: 2^-9 each, of random sign; their sum in float32
            tol = 2.0 ** -8 * (w @ v).abs() + (2.0 ** -20 if two_part else 2.0 ** -8 * float(w.pow(2).sum(-1).max().sqrt())) * float(v.abs().max())
            assert torch.all((out[r, m * G: (m + 1) * G].double() - w @ v).abs() <= tol)
    assert torch.allclose(out[0, 0].float(), vc[page_of, 0, slot].float(), atol=0.05)


def test_sizes_that_are_not_taken():
    assert not K().attn_decode_direct_supported(9, 1, 128) and not K().attn_decode_direct_supported(8, 8, 64)
