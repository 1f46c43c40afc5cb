"""What cache slots hold that no query reads (the rest of a page behind a request's last key, keys before the window in a page that is
still held, pages of other requests) reaches no result, not as a number that is not finite either: a page is handed on as its last holder
left it.  Every attention kernel over pages: the same bits with zeros, NaN and infinities there; whole models too."""
from __future__ import annotations

import pytest
import torch

from tests import helpers as H
from tests import test_gedelorn_gpu as gedelorn
from tests import test_puvolix_gpu as puvolix

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BAD = [float("nan"), float("inf"), -float("inf")]


def K():
    from quanta_b200 import kernels
    return kernels


def _lo(p, window, chunk):
    return p // chunk * chunk if chunk else max(0, p - window + 1) if window else 0


def _case(nq, nkv, page, lens, cached, window, chunk, hd=128):
    """q, caches, places, block table, and the mask of the slots that the step reads."""
    g = torch.Generator(device=DEV).manual_seed(len(lens) * 100 + window + chunk + page)
    per = [-(-(n + c) // page) for n, c in zip(lens, cached)]
    pages = sum(per) + 2
    kc = torch.randn(pages, nkv, page, hd, device=DEV, generator=g).bfloat16()
    vc = torch.randn(pages, nkv, page, hd, device=DEV, generator=g).bfloat16()
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(7)).int()
    table, at = torch.full((len(lens), max(per)), -1, dtype=torch.int32), 0
    read = torch.zeros(pages, page, dtype=torch.bool)
    for r, (n, c) in enumerate(zip(lens, cached)):
        table[r, : per[r]] = order[at: at + per[r]]
        at += per[r]
        for p in range(c, c + n):
            j = torch.arange(_lo(p, window, chunk), p + 1)
            read[table[r][j // page].long(), j % page] = True
    T = sum(lens)
    q = (torch.randn(T, nq, hd, device=DEV, generator=g) * 1.5).bfloat16()
    pos = torch.cat([torch.arange(c, c + n) for n, c in zip(lens, cached)]).int().to(DEV)
    req = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).int().to(DEV)
    return q, kc, vc, pos, req, table.to(DEV), read.to(DEV)[:, None, :, None]


def _tiles(lens, G, rows):
    out, t0 = [], 0
    for r, n in enumerate(lens):
        out += [[r, t0, n, x] for x in range(0, n * G, rows)]
        t0 += n
    return torch.tensor(out, dtype=torch.int32, device=DEV)


def _same_with_anything_unread(run, q, kc, vc, read):
    k = K()
    results = []
    for bad in [0.0, *BAD]:
        kk, vv = (torch.where(read, t, torch.full_like(t, bad)) for t in (kc, vc))
        out, st = torch.full_like(q, 3.0), k.new_status(DEV)
        run(kk, vv, out, st)
        assert st.tolist()[0] == 0
        results.append(out)
    assert torch.isfinite(results[0].float()).all()
    assert all(torch.equal(results[0], r) for r in results[1:])


@pytest.mark.parametrize("page,lens,cached", [(16, [128, 1, 33, 5], [0, 200, 95, 260]), (8, [61], [300]), (128, [70, 40], [500, 0]), (4, [9], [130])])
@pytest.mark.parametrize("window,chunk", [(0, 0), (100, 0), (129, 0), (0, 96)])
def test_portions(page, lens, cached, window, chunk, monkeypatch):
    k = K()
    nq, nkv = 8, 2
    q, kc, vc, pos, req, table, read = _case(nq, nkv, page, lens, cached, window, chunk)
    _same_with_anything_unread(lambda kk, vv, out, st: k.attn_span_split(
        q, kk, vv, out, pos, table, _tiles(lens, nq // nkv, k.attn_span_tc_rows()), 128 ** -0.5, window, st, chunk=chunk), q, kc, vc, read)
    for tensor_cores in (True, False):
        _same_with_anything_unread(lambda kk, vv, out, st: k.window_attention(
            q, kk, vv, out, pos, req, table, 128 ** -0.5, window, st, chunk=chunk, tensor_cores=tensor_cores, n_requests=len(lens)), q, kc, vc, read)
    if not chunk:
        for which in ("", "mma"):
            monkeypatch.setenv("QUANTA_B200_SPAN_KERNEL", which)
            _same_with_anything_unread(lambda kk, vv, out, st: k.attn_span(
                q, kk, vv, out, pos, table, _tiles(lens, nq // nkv, k.attn_span_rows(128, nq, nkv, page)), 128 ** -0.5, window, st), q, kc, vc, read)


@pytest.mark.parametrize("page,cached", [(16, [0, 30, 1500, 127]), (64, [2100]), (5, [333, 4])])
@pytest.mark.parametrize("window", [0, 100])
def test_single_tokens(page, cached, window):
    k = K()
    nq, nkv, lens = 8, 2, [1] * len(cached)
    q, kc, vc, pos, req, table, read = _case(nq, nkv, page, lens, cached, window, 0)
    n, longest = len(lens), max(cached) + 1
    for two_part in (False, True):
        _same_with_anything_unread(lambda kk, vv, out, st: k.attn_decode_direct(
            q, kk, vv, out, req, n, pos, req, table, 128 ** -0.5, window, longest, st, two_part=two_part), q, kc, vc, read)
    parts = k.attn_decode_parts(nkv, longest)
    po = torch.empty(n * nq * parts * 128, dtype=torch.float32, device=DEV)
    ml = torch.empty(n * nq * parts * 2, dtype=torch.float32, device=DEV)
    _same_with_anything_unread(lambda kk, vv, out, st: k.attn_decode(
        q, kk, vv, out, po, ml, req, n, pos, req, table, 128 ** -0.5, window, parts, st), q, kc, vc, read)


def _gedelorn():
    par, dense = gedelorn._par, gedelorn._dense
    return gedelorn, gedelorn._config(90, 64, [par(4, 2, 128, 48, 9.0, 32, 1e4, 0.09, 1.0, 2, 16, 16, [0.9, 0.5], 0.5, dense(48)),
                                               par(4, 1, 128, 20, 5.0, 64, 1e3, 0.09, 1.0, 1, 8, 8, [0.7], 0.5, dense(40))])


def _puvolix():
    left, right, layer = puvolix._left, puvolix._right, puvolix._layer
    return puvolix, puvolix._config(90, 64, [layer(left(4, 2, 128, 128, 2, (32, 1e4, None)), right(2, 1, 16, 16, 2), puvolix._dense(48)),
                                             layer(left(2, 2, 128, 128, 2, (64, 500.0, None)), right(2, 2, 16, 16, 3), None)])


@pytest.mark.parametrize("which", [_gedelorn, _puvolix])
def test_pages_that_others_left(which, tmp_path_factory):
    """Every page of the pool holds numbers that are not finite before the first request comes: prompts in portions, single tokens, both
    beside one another; the logits' bits are those of an engine with a clean pool."""
    module, cfg = which()
    folder, _, _ = module._folder(tmp_path_factory, "left", cfg=cfg, seed=5)
    reqs = {f"r{i}": H.random_tokens(n, cfg["vocab"], 40 + i) for i, n in enumerate([70, 41, 133])}
    for steps in (H.cut_tail_decode(reqs, tail=30), H.cut_mixed(reqs, seed=3, portion_sizes=(35, 50))):
        got = []
        for bad in [0.0, *BAD[:2]]:
            eng = module._engine(folder, "bfloat16", steps)
            for streams in eng.kv.values():
                for pages in streams.values():
                    pages.fill_(bad)
            got.append(H.replay(eng, steps))
        assert all(torch.isfinite(v).all() for v in got[0].values())
        for other in got[1:]:
            assert all(torch.equal(other[key], got[0][key]) for key in got[0])
