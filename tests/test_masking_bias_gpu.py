"""Biases by distance that mask keys (minus infinity, or the lowest float32) in the attention of few tokens: the masked keys have no
weight, wherever they lie among the turns and ranges that the kernel takes the keys in; a token whose keys are all masked reads nothing.
Tolerance: float32 scores and weights (tests/test_float32_rows_gpu.py), one rounding to bfloat16 where the result is."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n_split", [1, 3, None])
@pytest.mark.parametrize("masked", ["nearest", "farthest", "turns", "all"])
@pytest.mark.parametrize("low", [-float("inf"), torch.finfo(torch.float32).min])
@pytest.mark.parametrize("with_sink", [False, True])
def test_masked_distances(dtype, n_split, masked, low, with_sink):
    from quanta_b200 import kernels as k
    nq, nkv, hd, page, window, lens = 6, 2, 64, 16, 300, [1, 9, 70, 500]
    g = torch.Generator(device=DEV).manual_seed(3)
    per = [-(-n // page) for n in lens]
    kc = torch.randn(sum(per), nkv, page, hd, device=DEV, generator=g).to(dtype)
    vc = torch.randn(sum(per), nkv, page, hd, device=DEV, generator=g).to(dtype)
    table, at = torch.zeros((len(lens), max(per)), dtype=torch.int32), 0
    for r, n in enumerate(per):
        table[r, :n] = torch.arange(at, at + n, dtype=torch.int32)
        at += n
    table = table.to(DEV)
    T = len(lens)
    q = torch.randn(T, nq, hd, device=DEV, generator=g).to(dtype)
    pos, req = torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV), torch.arange(T, dtype=torch.int32, device=DEV)
    bias = torch.randn(window, nq, device=DEV, generator=g)
    d = torch.arange(window, device=DEV)
    gone = {"nearest": d < 130, "farthest": d > 3, "turns": (d // 8) % 2 == 0, "all": d >= 0}[masked]
    bias[gone, : nq - 1] = low                                      # the last head keeps its keys
    sink = torch.randn(nq, device=DEV, generator=g) if with_sink else None
    out, st = torch.full_like(q, 9.0), k.new_status(DEV)
    k.window_attention(q, kc, vc, out, pos, req, table, hd ** -0.5, window, st, dist_bias=bias, sink=sink, n_split=n_split)
    assert st.tolist()[0] == 0
    for t, n in enumerate(lens):
        j = torch.arange(max(0, n - window), n, device=DEV)
        row = table[t].long()[j // page]
        kk, vv = kc[row, :, j % page].double(), vc[row, :, j % page].double()
        for h in range(nq):
            b = bias[n - 1 - j, h].double()
            s = kk[:, h // 3] @ q[t, h].double() * hd ** -0.5 + b
            if low > -float("inf") and bool((b == low).all()):      # every score is the lowest number, as float32 adds it
                s = torch.zeros_like(s)
            if with_sink:
                s = torch.cat([s, sink[h].double()[None]])
            w = torch.softmax(s, 0) if bool((s > -float("inf")).any()) else torch.zeros_like(s)
            want = w[: len(j)] @ vv[:, h // 3]
            if with_sink and low > -float("inf") and bool((b == low).all()):
                want = torch.zeros_like(want)
            off = 1e-5 * float(vv.abs().max()) + (2.0 ** -8 * float(want.abs().max()) if dtype == torch.bfloat16 else 0.0)
            assert float((out[t, h].double() - want).abs().max()) <= off, (t, h)
