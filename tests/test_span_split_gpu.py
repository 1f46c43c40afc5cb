"""The tcgen05 attention of prompt portions with softmax weights in two bfloat16 parts, against float64, at the edges of its tiles of
128 rows and 128 keys, with windows, chunks and capped scores, single tokens as portions of one.  Tolerance: the weights hold 16 bits, their
exponents come from float32 scores (within 128 2^-24 sum |q k| scale, the cap adds a float32 next to the cap) through a 2^x of two units: 2^-12 of the
largest value covers them at these sizes, and the output is rounded to bfloat16 once."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nq,nkv,page,lens,cached", [
    (16, 4, 16, [128, 1, 33], [0, 200, 95]), (6, 2, 8, [127, 44], [1, 300]), (8, 8, 32, [129, 256], [127, 0]), (2, 1, 128, [70], [500]),
    (32, 1, 4, [5, 9], [130, 0])])
@pytest.mark.parametrize("window,chunk,cap", [(0, 0, 0.0), (100, 0, 30.0), (129, 0, 0.0), (0, 96, 0.0), (0, 128, 5.0), (1, 0, 0.0)])
def test_split_spans(nq, nkv, page, lens, cached, window, chunk, cap):
    from quanta_b200 import kernels
    hd, G, scale = 128, nq // nkv, 128 ** -0.5
    g = torch.Generator(device=DEV).manual_seed(nq + window + chunk)
    per = [-(-(n + c) // page) for n, c in zip(lens, cached)]
    pages = sum(per) + 1
    kc = torch.randn(pages, nkv, page, hd, device=DEV, generator=g).bfloat16()
    vc = torch.randn(pages, nkv, page, hd, device=DEV, generator=g).bfloat16()
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(3)).int()
    table = torch.full((len(lens), max(per)), -1, dtype=torch.int32)
    at, tiles, t0 = 0, [], 0
    for r, n in enumerate(lens):
        table[r, : per[r]] = order[at: at + per[r]]
        at += per[r]
        tiles += [[r, t0, n, r0] for r0 in range(0, n * G, kernels.attn_span_tc_rows())]
        t0 += n
    T = sum(lens)
    q = (torch.randn(T, nq, hd, device=DEV, generator=g) * 1.5).bfloat16()
    pos = torch.cat([torch.arange(c, c + n) for n, c in zip(lens, cached)]).int().to(DEV)
    out = torch.full((T, nq, hd), float("nan"), device=DEV, dtype=torch.bfloat16)
    st = kernels.new_status(DEV)
    table = table.to(DEV)
    # pages that no query of the request reads any more have been given back
    for r, c in enumerate(cached):
        lo = c // chunk * chunk if chunk else max(0, c - window + 1) if window else 0
        table[r, : lo // page] = -1
    kernels.attn_span_split(q, kc, vc, out, pos, table, torch.tensor(tiles, dtype=torch.int32, device=DEV), scale, window, st,
                            softcap=cap, chunk=chunk)
    assert st.tolist()[0] == 0
    t0 = 0
    for r, (n, c) in enumerate(zip(lens, cached)):
        j = torch.arange(c + n, device=DEV)
        i = torch.arange(c, c + n, device=DEV)[:, None]
        lo = i // chunk * chunk if chunk else (i - window + 1 if window else 0 * i)
        seen = (j[None] <= i) & (j[None] >= lo)
        rows = table[r].long()[j // page].clamp(min=0)
        k, v = kc[rows, :, j % page].double(), vc[rows, :, j % page].double()
        for h in range(nq):
            s = (q[t0: t0 + n, h].double() @ k[:, h // G].T) * scale
            s = cap * torch.tanh(s / cap) if cap else s
            want = torch.softmax(s.masked_fill(~seen, float("-inf")), -1) @ v[:, h // G]
            tol = 2.0 ** -8 * want.abs() + 2.0 ** -12 * float(v.abs().max())
            assert torch.all((out[t0: t0 + n, h].double() - want).abs() <= tol)
        t0 += n


@pytest.mark.parametrize("cap", [5.0, 50.0, 1000.0])
def test_capped_scores_keep_their_accuracy(cap):
    """A cap of any size costs the weights nothing: an output (of unit values' averages) is off by less than the bits of its weights, so few
    come out as another bfloat16 than the one nearest the exact value.  A relative error e of an output moves a share of about e / 2^-8 of
    roundings: 2^-16 of weights and scores together 0.4 %, scores off by some 2e-4 (a difference that cancels, at a cap of 1,000) 3 %."""
    from quanta_b200 import kernels
    T, nq, nkv, hd, page, scale = 256, 4, 2, 128, 16, 128 ** -0.5
    g = torch.Generator(device=DEV).manual_seed(11)
    q = torch.randn(T, nq, hd, device=DEV, generator=g).bfloat16()
    kc, vc = (torch.randn(T // page, nkv, page, hd, device=DEV, generator=g).bfloat16() for _ in range(2))
    table = torch.arange(T // page, device=DEV, dtype=torch.int32)[None]
    tiles = torch.tensor([[0, 0, T, r] for r in range(0, T * nq // nkv, kernels.attn_span_tc_rows())], dtype=torch.int32, device=DEV)
    out, st = torch.empty_like(q), kernels.new_status(DEV)
    kernels.attn_span_split(q, kc, vc, out, torch.arange(T, device=DEV, dtype=torch.int32), table, tiles, scale, 0, st, softcap=cap)
    assert st.tolist()[0] == 0
    k, v = (t.transpose(1, 2).reshape(T, nkv, hd).repeat_interleave(nq // nkv, 1).double() for t in (kc, vc))
    s = cap * torch.tanh(torch.einsum("thd,jhd->htj", q.double(), k) * scale / cap)
    s = s.masked_fill(torch.ones(T, T, device=DEV, dtype=torch.bool).triu(1), float("-inf"))
    want = torch.einsum("htj,jhd->thd", torch.softmax(s, -1), v).bfloat16()
    assert float((out != want).float().mean()) < 0.008


def test_which_steps_have_weights_of_16_bits():
    """The steps that kernels.window_attention gives to the tensor cores: at least 32 tokens and eight a request; no others."""
    from types import SimpleNamespace
    from quanta_b200.parts.attention import split_span_tiles
    cache = torch.zeros(4, 2, 16, 128, device=DEV, dtype=torch.bfloat16)
    for lens, taken in (([32], True), ([31], False), ([1, 40], True), ([1] * 24 + [32], False), ([1] * 24 + [176], True), ([1] * 24 + [175], False),
                        ([1] * 64, False), ([8] * 9, True), ([7] * 9, False)):
        T, starts = sum(lens), [0, *torch.tensor(lens).cumsum(0).tolist()]
        ctx = SimpleNamespace(host={"req_start": starts}, work={})
        tiles = split_span_tiles(ctx, torch.zeros(T, 8, 128, device=DEV, dtype=torch.bfloat16), cache, cache)
        assert (tiles is not None) == taken, lens


@pytest.mark.parametrize("page", [4, 16])
def test_single_tokens_of_long_requests_beside_a_portion(page):
    """Every single token of a mixed step is a portion of one: contexts of up to 9,300 keys (more than 2,048 pages of 4)."""
    test_split_spans(16, 4, page, [1, 40, 1, 1, 1], [9299, 3, 127, 4096, 8191], 0, 0, 0.0)
    test_split_spans(16, 4, page, [1, 40, 1], [9299, 3, 5000], 1000, 0, 30.0)
