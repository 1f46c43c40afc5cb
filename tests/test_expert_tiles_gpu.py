"""Experts of steps of few tokens on tcgen05: both products one behind the other, at the sizes where blocks of 64 features, two slabs of k a
stage, odd slabs, partial slabs and partial feature tiles meet, against float64 of the same bfloat16 operands.  Tolerance: an
activation is rounded to bfloat16 (2^-9 of it) and enters sums of float32; 2^-7 of the largest value bounds both."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T,E,top,H,I,gated,clamped,with_weights", [
    (1, 16, 8, 512, 192, True, False, 16), (1, 8, 2, 448, 200, True, True, 8), (3, 4, 2, 456, 136, True, False, 4), (2, 8, 3, 64, 64, True, False, 6),
    (16, 8, 2, 576, 320, False, False, 8), (1, 8, 2, 128, 72, False, False, 8), (5, 64, 8, 320, 256, True, False, 64), (30, 2, 1, 192, 136, False, False, 2),
    (24, 200, 8, 256, 2048, True, False, 200)])
def test_two_products(T, E, top, H, I, gated, clamped, with_weights):
    from quanta_b200 import kernels as k
    g = torch.Generator(device=DEV).manual_seed(T * H + I)
    rand = lambda *s, by=1.0: (torch.randn(*s, device=DEV, generator=g) * by).bfloat16()
    x, w13, w2 = rand(T, H), rand(with_weights, (2 if gated else 1) * I, H, by=H ** -0.5), rand(with_weights, H, I, by=I ** -0.5)
    cg = torch.Generator().manual_seed(T)
    idx = torch.stack([torch.randperm(E, generator=cg)[:top] for _ in range(T)]).int().to(DEV)
    w, n = torch.rand(T * top, device=DEV, generator=g) + 0.5, T * top
    bm = k.expert_tile_rows(T, n / E)
    words, tiles = k.moe_plan_sizes(n, E, bm)
    st = k.new_status(DEV)
    plan, pairs, te, tr = (torch.zeros(m, dtype=torch.int32, device=DEV) for m in (words, n, tiles, tiles))
    k.moe_plan(idx, E, bm, plan, pairs, te, tr, st, tiled_experts=with_weights)
    act, limits = torch.zeros(n, I, dtype=torch.bfloat16, device=DEV), (k.EXPERT_ACT_CLAMPED, 1.5, 1.7) if clamped else (0, 0.0, 1.0)
    mode, w_down = 1 if gated else 3, None if clamped else w
    results = []
    for gather, behind in ((top, True), (0, False)):
        rows = x if gather else x[(pairs.long() // top)].contiguous()
        y = torch.zeros(n, H, device=DEV)
        k.expert_gemm_tc(mode, rows, w13, act, pairs, w, plan, te, tr, E, bm, st, gather_top_k=gather, weight_experts=with_weights, act=limits)
        k.expert_gemm_tc(2, act, w2, y, pairs, w_down, plan, te, tr, E, bm, st, weight_experts=with_weights, after_first=behind)
        results.append(y)
    assert st.tolist()[0] == 0 and torch.equal(*results)
    for p, e in enumerate(idx.view(-1).tolist()):
        if e >= with_weights:
            assert float(results[0][p].abs().max()) == 0.0
            continue
        h = w13[e].double() @ x[p // top].double()
        if not gated:
            a = torch.relu(h) ** 2
        elif clamped:
            gate, up = (h[:I] * w[p]).clamp(max=limits[1]), (h[I:] * w[p]).clamp(-limits[1], limits[1])
            a = gate * torch.sigmoid(limits[2] * gate) * (up + 1)
        else:
            a = torch.nn.functional.silu(h[:I]) * h[I:]
        want = (w2[e].double() @ a) * (1.0 if clamped else float(w[p]))
        assert float((results[0][p].double() - want).abs().max()) <= 2.0 ** -7 * float(want.abs().max())
