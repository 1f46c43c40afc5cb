"""Kernels that start to read weights, state or old cache rows before the launch before them has ended (``early``): what that launch writes is
read behind it.  In each test a launch whose blocks the early one overlaps writes the kernel's inputs, as the last rows of a long result, over
NaN, while the stream is kept busy so that the launches queue up; the outputs have the bits of the same call on inputs that lie ready."""
from __future__ import annotations

import pytest
import torch

from tests import helpers as H
from tests import test_gedelorn_gpu as gedelorn
from tests import test_guravik_gpu as guravik
from tests.conftest import TINY

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
REPEATS, BUSY, ROWS = 6, 400_000, 4000        # clock cycles that the stream is kept busy; rows that the launch before writes


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


class Late:
    """A tensor ``[n, width]`` that ``write`` puts in place as the last rows of a launch over many."""

    def __init__(self, n, width, dtype, seed):
        from quanta_b200 import kernels
        self.source, self.all = torch.randn(ROWS, width, device=DEV, generator=_gen(seed)), torch.empty((ROWS, width), dtype=dtype, device=DEV)
        self.rows, self._act = self.all[ROWS - n:], kernels.rows_act

    def poison(self):
        self.all.fill_(float("nan"))

    def write(self):
        self._act(self.source, self.all)


def _same_behind_a_launch(late: list, run, restore=lambda: None):
    """``run(early)`` returns its outputs (new ones); each of ``late`` is once what the launch before writes, the others the launch before that."""
    for t in late:
        t.write()
    restore()
    torch.cuda.synchronize()
    want = [t.clone() for t in run(False)]
    assert all(torch.isfinite(t.float()).all() for t in want)
    for again in range(REPEATS):
        for t in late:
            t.poison()
        restore()
        torch.cuda.synchronize()
        torch.cuda._sleep(BUSY)
        for t in late[again % len(late):] + late[: again % len(late)]:
            t.write()
        got = run(True)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want)), again


@pytest.mark.parametrize("n,k,m", [(1, 3072, 4096), (8, 2048, 4000), (16, 1024, 96), (24, 2048, 1024)])
@pytest.mark.parametrize("silu", [False, True])
def test_products_of_few_rows(n, k, m, silu):
    from quanta_b200 import kernels
    x, w = Late(n, k, torch.bfloat16, n), torch.randn(m, k, device=DEV, generator=_gen(m)).to(torch.bfloat16)

    def run(early):
        out = torch.empty((n, m // 2 if silu else m), dtype=torch.bfloat16 if silu else torch.float32, device=DEV)
        (kernels.linear_few_silu if silu else kernels.linear_few)(x.rows, w, out, early=early)
        return [out]

    _same_behind_a_launch([x], run)


@pytest.mark.parametrize("R,heads,dim", [(1, 32, 64), (8, 32, 64), (5, 6, 128), (40, 16, 32)])
def test_delta_rule(R, heads, dim):
    from quanta_b200 import kernels
    HD, g = heads * dim, _gen(R)
    proj, wpre = Late(R, 4 * HD, torch.float32, 1), Late(R, HD, torch.float32, 2)
    ab, wb = (torch.randn(HD, device=DEV, generator=g) for _ in range(2))
    before = torch.randn(R + 2, heads, dim, dim, device=DEV, generator=g) * 0.3
    state = before.clone()
    starts = torch.arange(R + 1, dtype=torch.int32, device=DEV)
    slots = torch.randperm(R + 2, device=DEV, generator=g)[:R].int()

    def run(early):
        out = torch.empty(R, heads, dim, device=DEV)
        kernels.delta_rule(proj.rows, (0, HD, 2 * HD, 3 * HD), wpre.rows, ab, wb, state, out, starts, slots, heads, dim, 0.6, 1e-6, early=early)
        return [out, state]

    _same_behind_a_launch([proj, wpre], run, lambda: state.copy_(before))


@pytest.mark.parametrize("R,heads,groups,dim,vdim,kind", [(1, 16, 4, 64, 128, "given"), (16, 64, 1, 64, 128, "step"), (7, 4, 4, 128, 64, "constant"),
                                                          (3, 3, 3, 33, 13, "given")])
def test_decaying_state(R, heads, groups, dim, vdim, kind):
    from quanta_b200 import kernels
    g, G, HE = _gen(R + heads), groups * dim, heads * vdim
    proj, gate = Late(R, 2 * G + HE, torch.float32, 3), Late(R, 3 * heads, torch.float32, 4)
    before, n_before = torch.randn(R + 2, heads, dim, vdim, device=DEV, generator=g), torch.randn(R + 2, heads, dim, device=DEV, generator=g)
    state, n_state, decay = before.clone(), n_before.clone(), torch.rand(heads, device=DEV, generator=g)
    bias, A_log = (torch.randn(heads, device=DEV, generator=g) for _ in range(2))
    den = torch.zeros(R, heads, device=DEV)
    late = [proj] if kind == "constant" else [proj, gate]
    starts = torch.arange(R + 1, dtype=torch.int32, device=DEV)
    slots = torch.randperm(R + 2, device=DEV, generator=g)[:R].int()
    parts = gate.rows.view(3, R, heads)                     # given gates are whole tensors
    constant = kernels.DecayGates.constant(decay)           # (made here: its launches would come between)

    def restore():
        state.copy_(before)
        n_state.copy_(n_before)
        den.zero_()

    def run(early):
        out, extra = torch.empty(R, heads, vdim, device=DEV), {}
        if kind == "given":
            gates, extra = kernels.DecayGates.given(parts[0], parts[1]), dict(n_state=n_state, floor=parts[2], den=den)
        else:
            gates = constant if kind == "constant" else kernels.DecayGates.step(gate.rows[:, :heads], bias, A_log)
        p = proj.rows
        kernels.decay_state(p[:, :G], p[:, G: 2 * G], p[:, 2 * G:], gates, state, out, starts, slots, heads, groups, dim, vdim, early=early, **extra)
        return [out, state, n_state, den]

    _same_behind_a_launch(late, run, restore)


@pytest.mark.parametrize("T,E,width,k", [(1, 256, 3072, 8), (8, 256, 3072, 8), (16, 40, 264, 4), (5, 16, 6144, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_router(T, E, width, k, dtype):
    from quanta_b200 import kernels
    g = _gen(T + E)
    x, gate = Late(T, width, dtype, 5), torch.randn(E, width, device=DEV, generator=g) / width ** 0.5
    bias, counters, status = torch.randn(E, device=DEV, generator=g), torch.zeros(64, dtype=torch.int32, device=DEV), kernels.new_status(DEV)
    words, tiles = kernels.moe_plan_sizes(T * k, E, 16)

    def run(early):
        logits, w, idx = torch.empty(T, E, device=DEV), torch.empty(T, k, device=DEV), torch.empty((T, k), dtype=torch.int32, device=DEV)
        plan, pair, expert, row0 = (torch.empty(n, dtype=torch.int32, device=DEV) for n in (words, T * k, tiles, tiles))
        kernels.router_small(x.rows, gate, bias, logits, idx, w, True, 1.0, counters=counters, bm=16, plan=plan, sorted_pair=pair, tile_expert=expert,
                             tile_row0=row0, status=status, early=early)
        return [logits, w, idx]

    _same_behind_a_launch([x], run)
    assert status.tolist()[0] == 0


@pytest.mark.parametrize("two_part", [False, True])
@pytest.mark.parametrize("lens,window", [([700], 0), ([16, 17, 15, 128, 129, 1024, 1025, 1], 0), ([2100] * 16, 0), ([600 + 7 * i for i in range(40)], 300)])
def test_attention_of_single_tokens(lens, window, two_part):
    """The queries and the tokens' own keys and values come from the rotation's launch, which writes a long prompt's as well."""
    from quanta_b200 import kernels
    nq, nkv, hd, page, other, g = 16, 4, 128, 16, 3000, _gen(len(lens))
    lens = [other] + lens                                  # request 0: the prompt, in pages of its own
    per, R = [-(-n // page) for n in lens], len(lens)
    table, at = torch.zeros((R, max(per)), dtype=torch.int32), 0
    for r, n in enumerate(per):
        table[r, :n] = torch.arange(at, at + n, dtype=torch.int32)
        at += n
    table = table.to(DEV)
    old = [torch.randn(at, nkv, page, hd, device=DEV, generator=g).bfloat16() for _ in range(2)]
    kc, vc = (t.clone() for t in old)
    T = other + R - 1
    pos = torch.tensor(list(range(other)) + [n - 1 for n in lens[1:]], dtype=torch.int32, device=DEV)
    req = torch.tensor([0] * other + list(range(1, R)), dtype=torch.int32, device=DEV)
    rows, q = torch.randn(T, (nq + 2 * nkv) * hd, device=DEV, generator=g), torch.empty(T, nq, hd, device=DEV, dtype=torch.bfloat16)
    single, status = torch.arange(other, T, dtype=torch.int32, device=DEV), kernels.new_status(DEV)
    inv = torch.empty(0, device=DEV)

    class Written:
        def poison(self):
            q.fill_(float("nan"))
            for mine, was in ((kc, old[0]), (vc, old[1])):
                mine.copy_(was)
                mine[table[req.long(), (pos // page).long()].long(), :, (pos % page).long()] = float("nan")      # the tokens' own rows

        def write(self):
            kernels.qknorm_rope_write(rows, q, kc, vc, None, None, kernels.NORM_NONE, 1e-5, inv, None, pos, pos, req, table, nq, nkv, hd, 0, page,
                                      status)

    def run(early):
        out = torch.empty_like(q)
        kernels.attn_decode_direct(q, kc, vc, out, single, R - 1, pos, req, table, hd ** -0.5, window, max(lens[1:]), status, two_part=two_part,
                                   early=early)
        return [out[other:]]

    _same_behind_a_launch([Written()], run)
    assert status.tolist()[0] == 0


@pytest.mark.parametrize("graphs", [False, True])
@pytest.mark.parametrize("which", ["minimax", "guravik", "gedelorn"])
def test_steps_read_early_and_not(which, graphs, model_dirs, tmp_path_factory, monkeypatch):
    """Prompts, single tokens beside portions and decode steps: the bits of an engine whose kernels wait before they read."""
    from quanta_b200.engine import step as engine_step
    from quanta_b200.engine.model import load_model
    if which == "minimax":
        folder, vocab = model_dirs["D"], TINY["D"]["vocab_size"]
    else:
        module = {"guravik": guravik, "gedelorn": gedelorn}[which]
        folder, _, cfg = module._folder(tmp_path_factory, "D")
        vocab = cfg["vocab"]
    model, _ = load_model(folder, dtype="bfloat16")
    known, seen = engine_step.StepContext, set()
    results = []
    for settled in (True, False):
        def context(*args, settled_here=settled, **kw):
            seen.add(kw["settled"])
            return known(*args, **{**kw, "settled": settled_here})
        monkeypatch.setattr(engine_step, "StepContext", context)
        eng = engine_step.Engine(model, num_pages=400, page_size=16, max_requests=8, use_graphs=graphs)
        toks = {f"r{i}": H.random_tokens(300 - 31 * i, vocab, 70 + i) for i in range(4)}
        got = [eng.step([engine_step.StepEntry(r, t[:200], (199,)) for r, t in toks.items() if r != "r3"]).clone()]
        for n in range(4):      # single tokens of three requests beside portions of the fourth, then of all
            entries = [engine_step.StepEntry(r, t[200 + n: 201 + n], (0,)) for r, t in toks.items() if r != "r3"]
            got.append(eng.step([engine_step.StepEntry("r3", toks["r3"][40 * n: 40 * n + 40], (39,))] + entries).clone())
        for n in range(4):
            got.append(eng.step([engine_step.StepEntry(r, t[n: n + 1], (0,)) for r, t in toks.items()]).clone())
        eng.check()
        results.append(got)
    assert seen == {True}
    for n, (a, b) in enumerate(zip(*results)):
        assert torch.isfinite(a).all() and torch.equal(a, b), n
