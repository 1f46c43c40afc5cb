"""Launches of a step of few rows that do the work of two: each against the two launches (bit by bit where the operations are the same ones) or
against float64."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


@pytest.mark.parametrize("n,k,inner", [(1, 64, 8), (3, 2048, 5632), (8, 528, 20), (9, 256, 9), (16, 1024, 96), (20, 512, 40), (32, 2048, 1100)])
def test_gate_up_and_silu(n, k, inner):
    from quanta_b200 import kernels
    g = _gen(n + inner)
    x, w = (torch.randn(*s, device=DEV, generator=g).to(torch.bfloat16) for s in ((n, k), (2 * inner, k)))
    both, want, out = (torch.empty((n, m), device=DEV, dtype=torch.bfloat16) for m in (2 * inner, inner, inner))
    kernels.linear_few(x, w, both)
    kernels.silu_mul(both, want)
    kernels.linear_few_silu(x, w, out)
    assert torch.equal(out, want)


@pytest.mark.parametrize("T,n,N,off,wide", [(1, 1, 5, 0, 4), (2, 16, 300, 3, 20), (32, 16, 128, 0, 16), (7, 17, 129, 2, 64), (9, 64, 2048, 8, 80)])
def test_tanh_product(T, n, N, off, wide):
    """One rounding of the result; tanhf may be two units off where its rounding to bfloat16 turns, half a unit of that being 2^-9."""
    from quanta_b200 import kernels
    g = _gen(T * n)
    x, w = torch.randn(T, wide, device=DEV, generator=g), torch.randn(N, n, device=DEV, generator=g).to(torch.bfloat16)
    out = torch.empty(T, N, device=DEV)
    kernels.tanh_product(x, off, w, out)
    inner = torch.empty((T, n), device=DEV, dtype=torch.bfloat16)
    kernels.tanh_cols(x, off, n, inner)
    want = inner.double() @ w.double().T
    assert torch.all((out.double() - want).abs() <= 2.0 ** -24 * want.abs())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,H,taps,slots", [(1, 8, 3, 0), (3, 256, 4, 2), (8, 2048, 3, 0), (5, 4096, 4, 0)])
def test_norm_and_convolution(T, H, taps, slots, dtype):
    """Norm, stream, outputs and state as the norm into float32 rows and the convolution's own launch leave them."""
    from quanta_b200 import kernels
    g = _gen(T * H)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    h, gy, w, cw = r(T, H), r(H), r(H), r(H, taps)
    y = r(T, slots, H) if slots else r(T, H)
    extra = r(T, H) if slots else None
    state = r(T + 3, taps - 1, H)
    order = torch.randperm(T + 3, device=DEV, generator=g)[:T].int()
    h2, state2, normed = h.clone(), state.clone(), torch.empty(T, H, device=DEV)
    out, want = (torch.empty(T, H, device=DEV, dtype=dtype) for _ in range(2))
    starts = torch.arange(T + 1, dtype=torch.int32, device=DEV)
    kernels.normed_add_rmsnorm(h2, y, gy, 1e-6, w, 1e-5, normed, extra=extra, extra_scale=0.5)
    kernels.short_conv(normed, cw, state2, want, starts[:-1], starts, order)
    kernels.normed_add_rmsnorm(h, y, gy, 1e-6, w, 1e-5, out, extra=extra, extra_scale=0.5, conv=(cw, state, order))
    assert torch.equal(h, h2) and torch.equal(state, state2) and torch.equal(out, want)
    with pytest.raises(ValueError):
        kernels.normed_add_rmsnorm(h, y, gy, 1e-6, w, 1e-5, out, conv=(cw, state, order[:-1].contiguous()))


@pytest.mark.parametrize("lens,ranges", [([1] * 70, 3), ([1] * 31 + [5] + [1] * 40, 1), ([40, 1, 1, 3] * 12, 2), ([1] * 33, 40)])
def test_latent_attention_of_many_requests(lens, ranges):
    """Every request's rows are found whatever their number: the same numbers as a request alone."""
    from quanta_b200 import kernels
    g, H, C, R, page = _gen(len(lens)), 4, 64, 16, 16
    T, before = sum(lens), [int(x) for x in torch.randint(0, 150, (len(lens),), generator=torch.Generator().manual_seed(3))]
    mp = max(b + n for b, n in zip(before, lens)) // page + 1
    cache = torch.randn(len(lens) * mp, 1, page, C + R, device=DEV, generator=g).to(torch.bfloat16)
    table = torch.randperm(len(lens) * mp, generator=torch.Generator().manual_seed(1)).int().view(len(lens), mp).to(DEV)
    q_lat, q_rot = torch.randn(H, T, C, device=DEV, generator=g), torch.randn(T, H, R, device=DEV, generator=g)
    sink = torch.randn(H, device=DEV, generator=g)

    def run(rows):
        at = [sum(lens[:r]) for r in rows]
        pick = torch.tensor([a + i for a, r in zip(at, rows) for i in range(lens[r])], device=DEV)
        pos = torch.tensor([before[r] + i for r in rows for i in range(lens[r])], dtype=torch.int32, device=DEV)
        req = torch.tensor([k for k, r in enumerate(rows) for _ in range(lens[r])], dtype=torch.int32, device=DEV)
        starts = torch.tensor([0, *torch.tensor([lens[r] for r in rows]).cumsum(0).tolist()], dtype=torch.int32, device=DEV)
        out, st = torch.empty(H, len(pick), C, device=DEV, dtype=torch.bfloat16), kernels.new_status(DEV)
        kernels.latent_attend(q_lat[:, pick].contiguous(), q_rot[pick].contiguous(), cache, sink, out, pos, req, table[rows].contiguous(),
                              0.1, ranges, st, req_start=starts)
        assert st.tolist()[0] == 0
        return out

    whole, at = run(list(range(len(lens)))), 0
    assert torch.isfinite(whole.float()).all()
    for r, n in enumerate(lens):
        assert torch.equal(run([r]), whole[:, at: at + n]), r
        at += n


def test_state_rows_are_zeroed_together():
    """Rows of whole 16-byte pieces, of odd numbers of bytes and of none, more of them than one launch takes; the neighbours stay."""
    from quanta_b200 import kernels
    state = [torch.ones(shape, dtype=dt, device=DEV) for shape, dt in (((5, 3, 128), torch.float32), ((5, 7), torch.float32), ((5, 3), torch.bfloat16),
                                                                       ((5,), torch.int64), ((5, 0), torch.float32), ((5, 64, 64, 64), torch.float32))]
    state += [torch.ones((5, 1 + i), dtype=torch.uint8, device=DEV) for i in range(130)]
    state.append(torch.ones((6, 5), device=DEV).t())               # not contiguous
    kernels.zero_state_rows(state, 3)
    for t in state:
        assert not t[3].any() and all(bool((t[i] == 1).all()) for i in (0, 1, 2, 4))
    for slot in (-1, 5):
        with pytest.raises(IndexError):
            kernels.zero_state_rows(state, slot)
    assert all(bool((t[4] == 1).all()) for t in state)
    kernels.zero_state_rows([], 0)


def test_admission_zeroes_the_state_that_the_engine_has_now(tmp_path_factory):
    """A state tensor that was put in the place of another one is zeroed in its stead."""
    from quanta_b200.engine.model import load_model
    from quanta_b200.engine.step import Engine
    from tests import test_guravik_gpu as guravik
    model, _ = load_model(guravik._folder(tmp_path_factory, "D")[0], dtype="float32")
    eng = Engine(model, num_pages=8, page_size=16, max_requests=3)
    old = [dict(per_pos) for per_pos in eng.state]
    assert any(old)
    for per_pos in eng.state:
        for name, t in per_pos.items():
            t.fill_(2)
            per_pos[name] = torch.ones_like(t)
    slot = eng.admit("a")
    for before, now in zip(old, eng.state):
        for name, t in now.items():
            assert not t[slot].any() and t.sum() == t.numel() - t[slot].numel() and bool((before[name] == 2).all())


@pytest.mark.parametrize("T,H,I,E,k,mode", [(3, 64, 40, 8, 2, 1), (40, 72, 72, 4, 2, 1), (100, 200, 136, 8, 2, 3), (300, 136, 264, 4, 1, 1), (700, 64, 72, 8, 2, 1)])
def test_expert_rows_fetched_inside(T, H, I, E, k, mode):
    """Token rows fetched inside the first product, one or four at a time, in tiles of every size: the same bits as from a gathered copy."""
    from quanta_b200 import kernels
    g = _gen(T + I)
    x = torch.randn(T, H, device=DEV, generator=g).to(torch.bfloat16)
    w = (torch.randn(E, (2 if mode == 1 else 1) * I, H, device=DEV, generator=g) / H ** 0.5).to(torch.bfloat16)
    idx = torch.stack([torch.randperm(E, device=DEV, generator=g)[:k] for _ in range(T)]).int()
    idx[: T // 2] = torch.arange(k, device=DEV, dtype=torch.int32)          # some experts have many rows, some few
    pw, n = torch.rand(T, k, device=DEV, generator=g), T * k
    for bm in (16, 32, 64, 128, 256):
        words, tiles = kernels.moe_plan_sizes(n, E, bm)
        plan, sp, te, tr = (torch.empty(c, device=DEV, dtype=torch.int32) for c in (words, n, tiles, tiles))
        st = kernels.new_status(DEV)
        kernels.moe_plan(idx, E, bm, plan, sp, te, tr, st)
        rows = torch.empty((n, H), device=DEV, dtype=torch.bfloat16)
        kernels.gather_rows(x, rows, sp, k)
        a, b = (torch.full((n, I), float("nan"), device=DEV, dtype=torch.bfloat16) for _ in range(2))
        kernels.expert_gemm_tc(mode, rows, w, a, sp, pw.view(-1), plan, te, tr, E, bm, st)
        kernels.expert_gemm_tc(mode, x, w, b, sp, pw.view(-1), plan, te, tr, E, bm, st, gather_top_k=k)
        assert st.tolist()[0] == 0 and torch.isfinite(a.float()).all() and torch.equal(a, b), bm


@pytest.mark.parametrize("T,E,H,tensor_cores", [(64, 40, 264, False), (65, 40, 264, True), (16, 512, 8192, False), (17, 512, 8192, True), (17, 16, 200, False)])
def test_router_logits_on_both_sides_of_the_line(T, E, H, tensor_cores):
    """Few products on the CUDA cores, many on the tensor cores: the float64 product to float32 rounding."""
    from quanta_b200 import kernels
    from quanta_b200.parts.moe import SigmoidTopKExperts
    g = _gen(T + E)
    part = SigmoidTopKExperts.__new__(SigmoidTopKExperts)
    part.E, part.H, part.bias = E, H, torch.zeros(E, device=DEV)
    part.gate_w = torch.randn(E, H, device=DEV, generator=g) / H ** 0.5
    part.gate_pieces = kernels.split3_bf16(part.gate_w)
    x = torch.randn(T, H, device=DEV, generator=g).to(torch.bfloat16)
    status = kernels.new_status(DEV)
    logits = part.router_logits(x, status)
    assert part._on_tensor_cores(x) == tensor_cores == (logits.dim() == 3) and status.tolist()[0] == 0
    got = logits.sum(0) if tensor_cores else logits
    # sums of H products of size 1 / sqrt(H) in float32: no more than a few units of 2^-24 of sqrt(H) such products' absolute sum
    assert torch.allclose(got.double(), x.double() @ part.gate_w.double().T, atol=2e-5, rtol=1e-5)


@pytest.mark.parametrize("T,E,H", [(64, 8, 72), (129, 130, 776), (500, 256, 1536), (4100, 300, 800), (12800, 256, 776), (9000, 129, 1600)])
def test_router_logits_in_every_token_tile(T, E, H):
    """Prompts whose router logits take tiles of 64, 128 and 192 tokens, several items a block: a token's logits are the bits it has alone."""
    from quanta_b200 import kernels
    g = _gen(T)
    x = torch.randn(T, H, device=DEV, generator=g).to(torch.bfloat16)
    gate = torch.randn(E, H, device=DEV, generator=g) / H ** 0.5
    pieces, parts, status = kernels.split3_bf16(gate), kernels.router_gemm_mma_parts(H), kernels.new_status(DEV)
    logits = torch.full((parts, T, E), float("nan"), device=DEV)
    kernels.router_gemm_mma(x, pieces, logits, status)
    assert status.tolist()[0] == 0
    assert torch.allclose(logits.double().sum(0), x.double() @ gate.double().T, atol=2e-5, rtol=1e-5)
    for t in (0, T // 3, T - 1):
        alone = torch.empty((parts, 1, E), device=DEV)
        kernels.router_gemm_mma(x[t: t + 1], pieces, alone, status)
        assert torch.equal(alone[:, 0], logits[:, t])


@pytest.mark.parametrize("mode", range(5))
@pytest.mark.parametrize("T,E,k", [(3, 40, 4), (300, 256, 8)])
def test_logits_that_are_no_numbers_choose_experts_of_the_table(T, E, k, mode):
    """A token whose logits a wait kept back (NaN): its experts are inside the table and its weights are no numbers."""
    from quanta_b200 import kernels
    logits = torch.randn(2, T, E, device=DEV, generator=_gen(T))
    logits[0, 1] = torch.full((E,), 0x7FFFFFFF, dtype=torch.int32, device=DEV).view(torch.float32)
    idx, w = torch.empty((T, k), dtype=torch.int32, device=DEV), torch.empty((T, k), device=DEV)
    kernels.router_topk(logits, torch.zeros(E, device=DEV), idx, w, mode, 1.0)
    assert bool(((idx >= 0) & (idx < E)).all()) and bool(torch.isnan(w[1]).all())
    others = torch.arange(T, device=DEV) != 1
    assert bool(torch.isfinite(w[others]).all())
