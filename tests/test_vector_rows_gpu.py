"""Kernels that read rows in 16-byte pieces, at the sizes where they hand over to those that read a number at a time, against float64.
Tolerance: a few float32 roundings (2^-24) of the terms, 2^-8 where the result is bfloat16."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def K():
    from quanta_b200 import kernels
    return kernels


def randn(*shape, seed):
    return torch.randn(*shape, device=DEV, generator=torch.Generator(device=DEV).manual_seed(seed))


def rms(x, gain, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * gain


def near(got, want, dtype):
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
    assert float((got.double() - want).abs().max()) <= tol * max(1.0, float(want.abs().max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H", [8, 70, 264, 8192, 8200])
def test_norm_rows(H, dtype):
    h, delta, w = randn(5, H, seed=1), randn(5, 2, H, seed=2), 1 + 0.1 * randn(H, seed=3)
    y, y2, g, b = randn(5, H, seed=4), randn(5, H, seed=5), 1 + 0.1 * randn(H, seed=6), randn(H, seed=7)
    stream, out = h.clone(), torch.empty(5, H, device=DEV, dtype=dtype)
    K().add_rmsnorm(stream, delta, w, 1e-5, out)
    want = h.double() + delta.double().sum(1)
    near(stream, want, torch.float32)
    near(out, rms(want, w.double(), 1e-5), dtype)
    stream = h.clone()
    K().normed_add_rmsnorm(stream, y, g, 1e-6, w, 1e-5, out, y_scale=0.5, y_bias=b, extra=y2, extra_scale=2.0)
    want = h.double() + rms(0.5 * (y.double() + b.double()) + 2.0 * y2.double(), g.double(), 1e-6)
    near(stream, want, torch.float32)
    near(out, rms(want, w.double(), 1e-5), dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H", [6136, 6144, 6152, 7176, 8184])
def test_normed_rows_at_the_end_of_their_registers(H, dtype):
    """768 threads hold rows of up to 6,144 numbers; longer ones pass through shared memory.  Every summand alone and all together."""
    h, y, y2 = randn(3, H, seed=1), randn(3, 2, H, seed=2), randn(3, H, seed=3)
    g, w, b, b2 = 1 + 0.1 * randn(H, seed=4), 1 + 0.1 * randn(H, seed=5), randn(H, seed=6), randn(H, seed=7)
    for bias, extra, extra_bias in ((None, None, None), (b, None, None), (None, y2, None), (b, y2, b2)):
        stream, out = h.clone(), torch.empty(3, H, device=DEV, dtype=dtype)
        K().normed_add_rmsnorm(stream, y, g, 1e-6, w, 1e-5, out, y_scale=0.5, y_bias=bias, extra=extra, extra_scale=2.0, extra_bias=extra_bias)
        v = y.double().sum(1) + (bias.double() if bias is not None else 0)
        v = 0.5 * v + (2.0 * (extra.double() + (extra_bias.double() if extra_bias is not None else 0)) if extra is not None else 0)
        want = h.double() + rms(v, g.double(), 1e-6)
        near(stream, want, torch.float32)
        near(out, rms(want, w.double(), 1e-5), dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("E,width", [(8, 64), (33, 516), (256, 3072), (5, 4100), (7, 6144), (9, 130)])
def test_router_logits_depend_on_the_width_alone(E, width, dtype):
    """Steps of up to 16 tokens and of more run in two kernels with the same additions: a token's logits have the same bits in both."""
    x, gate = randn(40, width, seed=E).to(dtype), randn(E, width, seed=width)
    whole = torch.empty(40, E, device=DEV)
    K().router_small(x, gate, None, whole)
    want = x.double() @ gate.double().T
    assert float((whole.double() - want).abs().max()) <= 2.0 ** -20 * float((x.double().abs() @ gate.double().abs().T).max())
    for lo, hi in ((0, 1), (3, 5), (7, 16), (9, 25), (20, 37)):
        some = torch.empty(hi - lo, E, device=DEV)      # (a copy: rows that start on 16 bytes, as the whole does)
        K().router_small(x[lo:hi].clone(), gate, None, some)
        assert torch.equal(some, whole[lo:hi])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("inner", [7, 8, 12, 2056])
def test_silu_mul(inner, dtype):
    gu = randn(9, 2 * inner, seed=inner).to(dtype)
    out = torch.empty(9, inner, device=DEV, dtype=dtype)
    K().silu_mul(gu, out)
    near(out, torch.nn.functional.silu(gu[:, :inner].double()) * gu[:, inner:].double(), dtype)


@pytest.mark.parametrize("rows,inner", [(1, 8), (65, 8), (70000, 16), (8193, 64), (300, 504), (2100, 512), (513, 2048), (3, 2064)])
def test_silu_mul_of_many_short_rows(rows, inner):
    """Short rows lie several to a block, on both sides of a million numbers and past the grid's 32,768 rows of blocks."""
    gu = randn(rows, 2 * inner, seed=inner)
    out = torch.full((rows, inner), float("nan"), device=DEV)
    K().silu_mul(gu, out)
    near(out, torch.nn.functional.silu(gu[:, :inner].double()) * gu[:, inner:].double(), torch.float32)


@pytest.mark.parametrize("gate", ["sigmoid", "silu"])
@pytest.mark.parametrize("heads,dim,off,shared", [(3, 4, 0, False), (5, 64, 8, True), (33, 8, 4, False), (2, 128, 0, True), (3, 12, 0, False),
                                                  (3, 64, 3, True), (2, 256, 0, False)])
def test_head_norm_gate(heads, dim, off, shared, gate):
    T, P = 7, off + heads * dim + (-(off + heads * dim)) % 4
    o, proj, gain = randn(T, heads * dim, seed=1), randn(T, P, seed=2), 1 + 0.1 * randn(dim if shared else heads * dim, seed=3)
    x = o.double().view(T, heads, dim)
    want = rms(x, gain.double().view(-1, dim), 1e-5)
    z = proj.double()[:, off:off + heads * dim].view(T, heads, dim)
    want = want * (torch.sigmoid(z) if gate == "sigmoid" else torch.nn.functional.silu(z))
    for dtype in (torch.float32, torch.bfloat16):
        out = torch.empty(T, heads * dim, device=DEV, dtype=dtype)
        K().head_norm_gate(o, proj, off, gain, out, heads, dim, 1e-5, gate)
        near(out, want.reshape(T, -1), dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq,nkv,hd,vd,window,n_split", [(4, 1, 64, 64, 0, None), (6, 3, 36, 20, 17, 3), (5, 5, 128, 132, 300, None), (8, 1, 256, 4, 0, 5),
                                                         (4, 2, 50, 64, 90, 2), (4, 2, 64, 66, 0, 1)])
def test_attention_of_few_tokens(nq, nkv, hd, vd, window, n_split, dtype):
    """One to several tokens a request, ranges of keys, a bias by distance, a sink, a cap, given-back pages."""
    kern, page, lens, G = K(), 8, [700, 3, 65], nq // nkv
    per = -(-max(lens) // page)
    kc, vc = randn(3 * per, nkv, page, hd, seed=1).to(dtype), randn(3 * per, nkv, page, vd, seed=2).to(dtype)
    table = torch.randperm(3 * per, generator=torch.Generator().manual_seed(3)).int().view(3, per)
    req, pos = [0, 0, 1, 2, 2, 2], [698, 699, 2, 62, 63, 64]
    if window:
        table[0, : max(0, 699 - window) // page] = -1
    bias = randn(window, nq, seed=4) if window else None
    sink, cap, scale = randn(nq, seed=5), 5.0, hd ** -0.5
    q, st = randn(6, nq, hd, seed=6).to(dtype), kern.new_status(DEV)
    out = torch.empty(6, nq, vd, device=DEV, dtype=dtype)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    kern.window_attention(q, kc, vc, out, i32(pos), i32(req), table.to(DEV), scale, window, st, dist_bias=bias, sink=sink, softcap=cap,
                          n_split=n_split, tensor_cores=False)
    assert st.tolist()[0] == 0
    for t in range(6):
        j = torch.arange(max(0, pos[t] - window + 1) if window else 0, pos[t] + 1)
        rows = table[req[t]].long()[j // page].to(DEV)
        k, v = kc[rows, :, (j % page).to(DEV)].double(), vc[rows, :, (j % page).to(DEV)].double()
        s = torch.einsum("hgd,jhd->hgj", q[t].double().view(nkv, G, hd), k).reshape(nq, -1) * scale
        s = cap * torch.tanh(s / cap)
        if window:
            s = s + bias.double()[(pos[t] - j).to(DEV)].T
        w = torch.softmax(torch.cat([s, sink.double()[:, None]], 1), 1)[:, :-1]
        want = torch.einsum("hgj,jhd->hgd", w.view(nkv, G, -1), v).reshape(nq, vd)
        # float32: some 700 terms; the exponents carry a few roundings of scores up to 10
        tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -17
        assert float((out[t].double() - want).abs().max()) <= tol * float(v.abs().max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq,nkv,hd,T,window,chunk", [(8, 8, 64, 40, 100, 0), (6, 2, 128, 70, 0, 96), (16, 4, 16, 33, 50, 0), (12, 2, 256, 24, 300, 0)])
def test_a_block_or_a_warp_a_range(nq, nkv, hd, T, window, chunk, dtype):
    """Steps that either kernel may take (the choice is by speed): both within float32 sums of one another, each range cut or not."""
    kern, page = K(), 16
    per = -(-400 // page)
    kc, vc = randn(T * per, nkv, page, hd, seed=1).to(dtype), randn(T * per, nkv, page, hd, seed=2).to(dtype)
    table = torch.arange(T * per, dtype=torch.int32, device=DEV).view(T, per)
    pos = torch.arange(400 - T, 400, dtype=torch.int32, device=DEV)
    req = torch.arange(T, dtype=torch.int32, device=DEV)
    q, outs = randn(T, nq, hd, seed=3).to(dtype), []
    for by_rows, n_split in ((True, None), (True, 3), (False, None), (False, 5)):
        out, st = torch.full_like(q, float("nan")), kern.new_status(DEV)
        kern.window_attention(q, kc, vc, out, pos, req, table, hd ** -0.5, window, st, chunk=chunk, n_split=n_split, by_rows=by_rows,
                              tensor_cores=False)
        assert st.tolist()[0] == 0
        outs.append(out.double())
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -18
    for out in outs[1:]:
        assert float((out - outs[0]).abs().max()) <= tol * float(vc.double().abs().max())
