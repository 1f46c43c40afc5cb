"""The engine's work, case by case, for measurements: inputs, one pass through the public entry points, what a pass cannot
do without, and what it should return (in 64 bits, written out in plain torch without the engine).

Three models, with the widths that ``bench.py`` and ``bench_designs.py`` run: the MiniMax-M3 decoder at the M2-family layer sizes (4 of
its 62 layers; the vocabulary is cut in the same proportion, so that the output matrix keeps its share of a step), Guravik (latent
attention and a delta rule) and Gedelorn (a matrix memory, a state-space recurrence, windowed attention beside linear attention) of
width 2,048.  Weights are random: gains, decays and biases at the scale where every mechanism matters, the matrices that write to
the residual stream small, as in a deep model.  Routers are decisive, as trained ones are: a token's embedding leans towards the
directions of the experts that take it, a draw of its own, so that near ties, which rounding turns, are rare.

A case is one of

* ``prompt``: new prompts as one step, the logits of their last places (``Engine.step``);
* ``chat``: requests that have read their prompts and decode: ``steps`` tokens each per pass, the ids given (``Engine.step``; the
  captured decode step).  The requests grow from pass to pass; after ``GROWTH`` tokens they end and their like come in;
* ``mixed``: a portion of a new prompt beside decoding requests, as one step: continuous batching;
* ``generate``: prompts in, greedily chosen tokens out (``generate``), then the logits of every chosen token from one step over
  the whole texts; in float32.
"""

from __future__ import annotations

import hashlib
import math
import random

import torch
import torch.nn.functional as F

from quanta_b200 import generate as generate_tokens
from quanta_b200.config import GedelornConfig, GuravikConfig, MiniMaxM3Config
from quanta_b200.config.registry import resolve
from quanta_b200.engine.generate import LLM
from quanta_b200.engine.model import Model
from quanta_b200.engine.step import Engine, StepEntry
from quanta_b200.matmul import configure

DEVICE = "cuda:0"
PAGE = 16
GROWTH = 1800           # tokens a decoding request grows by before it ends
WARM = 2                # decoded tokens before the first pass: the step's graph is captured at its second use
PORTION = 8192          # tokens of prompts a step takes while requests come in

M3 = dict(vocab_size=12928, hidden_size=3072, intermediate_size=1536, num_hidden_layers=4, num_attention_heads=48,
          num_key_value_heads=8, head_dim=128, rotary_dim=64, rope_theta=5e6, use_qk_norm=True, qk_norm_type="per_layer",
          num_local_experts=256, num_experts_per_tok=8, use_routing_bias=True, rms_norm_eps=1e-6, tie_word_embeddings=False,
          architectures=["MiniMaxM3ForCausalLM"], model_type="minimax_m3")
M3_SMALL = dict(M3, vocab_size=32000, hidden_size=2048, intermediate_size=2816, num_hidden_layers=6, num_attention_heads=16,
                num_key_value_heads=4, rope_theta=1e6, num_local_experts=8, num_experts_per_tok=2, rms_norm_eps=1e-5)
M3_DEPTH = 62           # layers of the whole decoder: its output matrices are drawn smaller by sqrt(2 * depth)


def _guravik() -> dict:
    latent = {"type": "latent_attention", "mlp": {"kind": "dense", "ff": 5632},
              "mixer": {"heads": 16, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 768, "kv_rank": 256,
                        "scale": 1.0 / math.sqrt(192), "rot": {"base": 1e6, "dims": 64}}}
    delta = {"type": "general_delta", "mixer": {"heads": 32, "dim": 64}, "mlp": None}
    return {"architecture": "Guravik", "vocab": 32000, "width": 2048, "layers": [latent, delta, delta] * 2, "canon": {"taps": 3},
            "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5}, "loop": {"start": 0, "stop": 0, "times": 1}}


def _gedelorn() -> dict:
    moe = {"kind": "moe", "expert": {"ff": 2112}, "router": {"experts": 8, "top": 2, "scale": 1.5}, "shared": {"ff": 1408}}
    ssm = {"heads": 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}
    left = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 1.0 / math.sqrt(128), "softcap": 30.0,
            "mask": {"size": 1024}, "rot": {"dims": 128, "base": 1e6}}
    right = {"heads": 16, "dim": 128, "vdim": 128, "decay": [math.exp(-(2.0 ** (-8.0 * (h + 1) / 16))) for h in range(16)]}
    par = {"left": left, "right": right, "left_scale": 0.8, "right_scale": 1.1}
    mem = {"heads": 8, "dim": 128, "vdim": 256, "gate_cap": 15.0}
    layers = [{"type": "mamba2", "mixer": ssm, "mlp": {"kind": "dense", "ff": 5632}}, {"type": "parallel", "mixer": par, "mlp": moe},
              {"type": "mlstm", "mixer": mem, "mlp": moe}] * 2
    return {"architecture": "Gedelorn", "vocab": 32000, "width": 2048, "layers": layers, "norm": {"eps": 1e-5}}


RAW = {"m3": M3, "m3_small": M3_SMALL, "guravik": _guravik(), "gedelorn": _gedelorn()}
CONFIG = {"m3": MiniMaxM3Config, "m3_small": MiniMaxM3Config, "guravik": GuravikConfig, "gedelorn": GedelornConfig}


# ---- the cases -----------------------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # one user at a terminal: every token is a step of its own, nothing shares its launches
        dict(name="m3_chat_1", model="m3", kind="chat", requests=1, context=2100, steps=4),
        # a small server: the batch and the contexts that bench.py's headline has
        dict(name="m3_chat_8", model="m3", kind="chat", requests=8, context=2100, steps=2),
        # a busy server: most experts are read in every step
        dict(name="m3_chat_64", model="m3", kind="chat", requests=64, context=2100, steps=1),
        # a question of a line or two, of an odd length
        dict(name="m3_prompt_93", model="m3", kind="prompt", requests=1, longest=93, want=1),
        # several documents at once, no two of one length: the largest step a server takes
        dict(name="m3_prompts_8", model="m3", kind="prompt", requests=8, longest=2048, want=8),
        # continuous batching: a portion of one request's prompt goes beside the others' next tokens
        dict(name="m3_mixed_24", model="m3", kind="mixed", requests=24, context=1500, portion=512),
        # two requests over long documents: the step reads more keys and values than weights of its attention
        dict(name="m3_long_2", model="m3", kind="chat", requests=2, context=24000, steps=2),
        # the float32 mode: short prompts to tokens through generate(), and their scores
        dict(name="m3_float32_generate", model="m3_small", kind="generate", requests=4, longest=120, steps=16),
        # Guravik: a document in, and a batch that decodes
        dict(name="guravik_prompt_2048", model="guravik", kind="prompt", requests=1, longest=2048, want=8),
        dict(name="guravik_chat_8", model="guravik", kind="chat", requests=8, context=2100, steps=2),
        # Gedelorn: several prompts of different lengths in one step, and a batch that decodes behind its window
        dict(name="gedelorn_prompts_4", model="gedelorn", kind="prompt", requests=4, longest=1500, want=4),
        dict(name="gedelorn_chat_16", model="gedelorn", kind="chat", requests=16, context=2100, steps=2),
    ]


def draw(rng: random.Random) -> dict:
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model = rng.choice(["m3", "m3", "m3", "guravik", "gedelorn", "m3", "guravik", "gedelorn", "m3", "m3_small"])
    if model == "m3_small":
        return dict(model=model, kind="generate", requests=rng.randint(1, 5), longest=spread(8, 150), steps=rng.randint(4, 20))
    kind = rng.choice(["chat", "chat", "prompt", "prompt", "mixed", "long" if model == "m3" else "chat"])
    if kind == "long":
        return dict(model=model, kind="chat", requests=rng.randint(1, 3), context=spread(4000, 20000), steps=rng.randint(1, 4))
    if kind == "chat":
        return dict(model=model, kind="chat", requests=spread(1, 64), context=spread(60, 2100), steps=rng.randint(1, 3))
    if kind == "prompt":
        longest = spread(17, 4000)
        most = min(8, max(1, 9000 // longest))
        return dict(model=model, kind="prompt", requests=rng.randint(1, most), longest=longest, want=rng.randint(1, 8))
    return dict(model=model, kind="mixed", requests=spread(2, 48), context=spread(100, 2000), portion=spread(40, 1500))


def _lengths(case: dict) -> list[int]:
    """The requests' lengths: from the longest down to half of it."""
    n, top = case["requests"], case.get("longest") or case["context"]
    return [top - (top // 2) * i // max(1, n) for i in range(n)]


# ---- inputs ----------------------------------------------------------------------------------------------
def _seed_of(seed: int, name: str) -> int:
    return int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:7], "little")


def _experts(model: str) -> tuple[int, int, int]:
    """Experts, chosen experts and width of the model's routers."""
    raw = RAW[model]
    if model.startswith("m3"):
        return raw["num_local_experts"], raw["num_experts_per_tok"], raw["hidden_size"]
    router = raw["layers"][1]["mlp"]["router"]
    return router["experts"], router["top"], raw["width"]


def _directions(model: str, seed: int) -> torch.Tensor:
    """A direction of length one for each expert; the routers' rows are these, in an order of each layer's own."""
    experts, _, width = _experts(model)
    g = torch.Generator(device=DEVICE)
    g.manual_seed(_seed_of(seed, "directions"))
    return torch.empty((experts, width), device=DEVICE).normal_(0.0, width ** -0.5, generator=g)


def _router(model: str, seed: int, name: str) -> torch.Tensor:
    layer = int(next(part for part in name.replace("l", "").split(".") if part.isdigit()))
    return 0.4 * torch.roll(_directions(model, seed), 3 * layer + 1, 0)


def _embedding(model: str, seed: int, g, shape, std: float, dtype) -> torch.Tensor:
    experts, top, _ = _experts(model)
    t = torch.empty(shape, device=DEVICE).normal_(0.0, std, generator=g)
    mine = torch.empty((shape[0], experts), device=DEVICE).uniform_(0.0, 1.0, generator=g).topk(top, dim=1).indices
    lean = torch.zeros((shape[0], experts), device=DEVICE)
    lean.scatter_(1, mine, torch.empty(mine.shape, device=DEVICE).uniform_(7.0, 9.0, generator=g))
    return t.add_(lean @ _directions(model, seed), alpha=std).to(dtype)


def _tensor(model: str, seed: int, name: str, shape, float32: bool = False) -> torch.Tensor:
    """A tensor of the model by name: it depends on the seed, its name and shape alone.  Matrices are bfloat16."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(_seed_of(seed, name))
    leaf = name.rsplit(".", 1)[-1]

    def uniform(lo, hi):
        return torch.empty(shape, device=DEVICE).uniform_(lo, hi, generator=g)

    def matrix(std):
        return torch.empty(shape, dtype=torch.float32 if float32 else torch.bfloat16, device=DEVICE).normal_(0.0, std, generator=g)

    if model.startswith("m3"):
        if name.endswith("embed_tokens.weight"):
            return _embedding(model, seed, g, shape, 0.5, torch.float32 if float32 else torch.bfloat16)
        if name.endswith(("q_norm.weight", "k_norm.weight")):
            return uniform(1.3, 1.5)            # scores of a spread of two: a softmax that picks some keys out
        if name.endswith("norm.weight"):
            return uniform(0.9, 1.1)
        if name.endswith("e_score_correction_bias"):
            return uniform(-0.05, 0.05)
        if name.endswith("gate.weight"):
            return _router(model, seed, name)
        return matrix(0.02 / math.sqrt(2 * M3_DEPTH) if name.endswith(("o_proj.weight", "w2.weight")) else 0.02)
    around_zero = model == "gedelorn" and not name.endswith("mix.norm") and not name.endswith("right.norm")
    if leaf in ("norm1b", "norm2b"):            # what a sublayer adds to the stream: a tenth of it
        return uniform(0.05, 0.15) - (1.0 if around_zero else 0.0)
    if leaf in ("norm1", "norm2", "norm"):
        return uniform(0.7, 1.3) - (1.0 if around_zero else 0.0)
    if leaf in ("conv", "canon1"):
        t = uniform(-0.5, 0.5)
        if leaf == "conv":
            t[:, -1] += 1.0
        return t
    if leaf in ("sink", "w0") or name.endswith("a.b"):
        return torch.empty(shape, device=DEVICE).normal_(0.0, 1.0, generator=g)
    if leaf == "A_log":
        return uniform(-2.5, 0.5)
    if leaf == "dt_bias":
        return uniform(-3.0, 1.0)
    if leaf == "D":
        return uniform(-1.0, 1.0)
    if name.endswith(".f.b"):
        return uniform(0.0, 4.0)
    if name.endswith(".i.b"):
        return uniform(-2.0, 1.0)
    if leaf == "b":
        return uniform(-0.5, 0.5)
    if leaf == "router":
        return _router(model, seed, name)
    if name == "embed":
        return _embedding(model, seed, g, shape, 1.0, torch.bfloat16) if model == "gedelorn" else matrix(1.0)
    return matrix((2.0 if leaf == "uq" else 1.0) / math.sqrt(shape[-1]))


class _Weights:
    """A source of weights, drawn when the model asks for them."""

    def __init__(self, model: str, seed: int, specs, float32: bool):
        self.model, self.seed, self.float32 = model, seed, float32
        self.specs = {s.name: s for s in specs}

    def names(self):
        return list(self.specs)

    def meta(self, name):
        s = self.specs[name]
        return ("BF16" if s.kind == "matrix" and not self.float32 else "F32"), tuple(s.shape)

    def read(self, name, device):
        return _tensor(self.model, self.seed, name, tuple(self.specs[name].shape), self.float32)

    def close(self):
        pass


def _tokens(case: dict, seed: int):
    """The requests' prompts, the tokens they are fed afterwards (a step's tokens at a time, over and over), and the portion."""
    rng = random.Random(seed)
    vocab = RAW[case["model"]].get("vocab_size") or RAW[case["model"]]["vocab"]
    prompts = [rng.choices(range(vocab), k=n) for n in _lengths(case)]
    fed = [rng.choices(range(vocab), k=case["requests"]) for _ in range(61)]
    portion = rng.choices(range(vocab), k=case.get("portion", 0))
    return prompts, fed, portion


class _State:
    pass


def prepare(case: dict, seed: int):
    configure()
    raw, float32 = RAW[case["model"]], case["kind"] == "generate"
    cfg = CONFIG[case["model"]].from_dict(raw)
    model = Model(resolve(raw).build_spec(cfg), dtype="float32" if float32 else "bfloat16", device=DEVICE)
    model.load(_Weights(case["model"], seed, model.tensor_specs(), float32))
    s = _State()
    s.case = case
    s.prompts, s.fed, s.portion = _tokens(case, seed)
    grown = {"chat": GROWTH + WARM + 8, "mixed": GROWTH + WARM + 8, "prompt": 0, "generate": case.get("steps", 0)}[case["kind"]]
    pages = sum(-(-(n + grown) // PAGE) for n in _lengths(case)) + -(-len(s.portion) // PAGE) + 1
    if float32:
        s.llm = LLM(model, page_size=PAGE, num_pages=pages, max_requests=case["requests"])
        return s
    s.engine = Engine(model, page_size=PAGE, num_pages=pages, max_requests=case["requests"] + 1)
    if case["kind"] != "prompt":
        _come_in(s)
    return s


def _come_in(s) -> None:
    """Requests come in and read their prompts, several of them or a portion of one in a step; then they decode."""
    for i in range(len(s.prompts)):
        s.engine.release(i)
    step, room = [], PORTION
    for i, prompt in enumerate(s.prompts):
        at = 0
        while at < len(prompt):
            n = min(room, len(prompt) - at)
            step.append(StepEntry(i, prompt[at: at + n], ()))
            at, room = at + n, room - n
            if room == 0:
                s.engine.step(step)
                step, room = [], PORTION
    if step:
        s.engine.step(step)
    s.grown = 0
    for _ in range(WARM):
        s.engine.step(_next(s))


def _next(s) -> list:
    ids = s.fed[s.grown % len(s.fed)]
    s.grown += 1
    return [StepEntry(i, [t], (0,)) for i, t in enumerate(ids)]


# ---- one pass ------------------------------------------------------------------------------------------------
def run(s):
    case = s.case
    if case["kind"] == "generate":
        tokens = generate_tokens(s.llm, s.prompts, max_new_tokens=case["steps"])
        entries, n = [], case["steps"]
        for i, (prompt, new) in enumerate(zip(s.prompts, tokens)):
            text = prompt + new[:-1]
            entries.append(StepEntry(("score", i), text, tuple(range(len(text) - n, len(text)))))
        return {"tokens": torch.tensor(tokens), "logits": s.llm.engine.step(entries, end=[e.rid for e in entries])}
    if case["kind"] == "prompt":
        entries = [StepEntry(i, p, tuple(range(max(0, len(p) - case["want"]), len(p)))) for i, p in enumerate(s.prompts)]
        return s.engine.step(entries, end=[e.rid for e in entries])
    if s.grown > GROWTH:
        _come_in(s)
    if case["kind"] == "mixed":
        return s.engine.step(_next(s) + [StepEntry("new", s.portion, (len(s.portion) - 1,))], end=["new"])
    return [s.engine.step(_next(s)).clone() for _ in range(case["steps"])]


# ---- what a pass cannot do without --------------------------------------------------------------------------------
def _distinct(experts: int, top: int, tokens: int) -> float:
    """Experts that a step of so many tokens reads, each token choosing evenly."""
    return experts * (1.0 - (1.0 - top / experts) ** tokens)


def _step_work(model: str, new: list[int], before: list[int], rows: int) -> tuple[float, float]:
    """Bytes and operations of one step: ``new[i]`` tokens of a request after ``before[i]`` cached ones, logits at ``rows`` places."""
    raw, T, R = RAW[model], sum(new), len(new)
    size = 4 if model == "m3_small" else 2
    pairs = sum(n * b + n * (n + 1) / 2 for n, b in zip(new, before))
    by = fl = 0.0
    if model.startswith("m3"):
        H, I, nq, nkv, hd = (raw[k] for k in ("hidden_size", "intermediate_size", "num_attention_heads", "num_key_value_heads", "head_dim"))
        E, k, L, V = raw["num_local_experts"], raw["num_experts_per_tok"], raw["num_hidden_layers"], raw["vocab_size"]
        attn = H * (2 * nq + 2 * nkv) * hd
        by = L * (size * (attn + 3 * H * I * _distinct(E, k, T) + (sum(before) + T) * 2 * nkv * hd) + 4 * E * H)
        fl = L * (2 * T * (attn + E * H + 3 * H * I * k) + 4 * nq * hd * pairs)
    elif model == "guravik":
        H, V = raw["width"], raw["vocab"]
        for layer in raw["layers"]:
            m = layer["mixer"]
            if layer["type"] == "general_delta":
                inner = m["heads"] * m["dim"]
                w, more = 6 * H * inner + 16 * (H + inner), 7 * inner * m["dim"] * T
                by += 2 * 4 * R * inner * m["dim"]
            else:
                h, D, r, vd, q, c = (m[k] for k in ("heads", "dim", "rot_dim", "vdim", "q_rank", "kv_rank"))
                w = H * (q + c + r + h * vd) + h * (D + r) * q + h * (D + vd) * c
                more = 2 * h * (D + r + vd) * pairs
                by += size * (sum(before) + T) * (c + r)
            w += 3 * H * layer["mlp"]["ff"] if layer["mlp"] else 0
            by, fl = by + size * w, fl + 2 * T * w + more
    else:
        H, V = raw["width"], raw["vocab"]
        for layer in raw["layers"]:
            m = layer["mixer"]
            if layer["type"] == "mamba2":
                inner, cells = m["heads"] * m["vdim"], m["heads"] * m["vdim"] * m["state"]
                w = H * (3 * inner + 2 * m["groups"] * m["state"] + m["heads"])
            elif layer["type"] == "mlstm":
                cells = m["heads"] * m["dim"] * (m["vdim"] + 1)
                w = m["heads"] * H * (2 * m["dim"] + 3 * m["vdim"] + 2)
            else:
                a, m = m["left"], m["right"]
                cells = m["heads"] * m["dim"] * m["vdim"]
                w = m["heads"] * H * (2 * m["dim"] + 3 * m["vdim"]) + H * a["dim"] * (2 * a["heads"] + a["kv_heads"])
                win = a["mask"]["size"]
                seen = sum(min(win, b + j + 1) for n, b in zip(new, before) for j in range(n))
                by += size * 2 * a["kv_heads"] * a["dim"] * sum(min(b, win) + n for n, b in zip(new, before))
                fl += 4 * a["heads"] * a["dim"] * seen
            by, fl = by + 8 * R * cells + size * w, fl + 2 * T * w + 4 * T * cells
            mlp = layer["mlp"]
            if mlp["kind"] == "dense":
                by, fl = by + 3 * size * H * mlp["ff"], fl + 6 * T * H * mlp["ff"]
            else:
                E, k, f, sh = mlp["router"]["experts"], mlp["router"]["top"], mlp["expert"]["ff"], mlp["shared"]["ff"]
                by += 2 * size * H * (f * _distinct(E, k, T) + sh) + 4 * E * H
                fl += 2 * T * H * (E + 2 * f * k + 2 * sh)
    by += size * (T * H + H * V) + 4 * rows * V
    return by, fl + 2 * rows * H * V


def work(case: dict) -> dict:
    lens, kind, model, n = _lengths(case), case["kind"], case["model"], case["requests"]
    if kind == "prompt":
        steps = [(lens, [0] * n, sum(min(case["want"], t) for t in lens))]
    elif kind == "mixed":
        steps = [([1] * n + [case["portion"]], [t + WARM for t in lens] + [0], n + 1)]
    elif kind == "chat":
        steps = [([1] * n, [t + WARM + j for t in lens], n) for j in range(case["steps"])]
    else:
        steps = [(lens, [0] * n, n)] + [([1] * n, [t + j for t in lens], n) for j in range(case["steps"] - 1)]
        steps.append(([t + case["steps"] - 1 for t in lens], [0] * n, n * case["steps"]))
    total = [_step_work(model, *s) for s in steps]
    return {"bytes": sum(b for b, _ in total), "flops": sum(f for _, f in total)}


def tolerance(case: dict):
    if case["kind"] == "generate":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    # bfloat16 logits are 0.002 off 64 bits; 0.01 where a token's expert is chosen differently on a near tie after all
    return {"rel": 0.02, "max": 0.4}


# ---- the same in 64 bits, without the engine ------------------------------------------------------------------------
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, cap=0.0, window=0, sink=None):
    """Causal softmax attention of one sequence: ``q`` [T, H, D], ``k`` [T, G, D], ``v`` [T, G, V] -> [T, H, V]."""
    T, H, _ = q.shape
    G = k.shape[1]
    kt, vt, out = k.permute(1, 2, 0), v.transpose(0, 1), q.new_empty(T, H, v.shape[2])
    for lo in range(0, T, 1024):
        hi = min(T, lo + 1024)
        qs = q[lo:hi].reshape(hi - lo, G, H // G, -1).permute(1, 2, 0, 3).reshape(G, -1, q.shape[2])
        s = torch.matmul(qs, kt[:, :, :hi]).mul_(scale).view(G, H // G, hi - lo, hi)
        if cap:
            s = cap * torch.tanh(s / cap)
        i, j = torch.arange(lo, hi, device=q.device)[:, None], torch.arange(hi, device=q.device)[None, :]
        s.masked_fill_((j > i) | ((i - j >= window) if window else (j > i)), float("-inf"))
        if sink is not None:                    # one more score a head, whose value is zero
            s = torch.cat([s, sink.view(G, H // G, 1, 1).expand(-1, -1, hi - lo, 1)], -1)
        p = torch.softmax(s, -1)[..., :hi]
        out[lo:hi] = torch.matmul(p.view(G, -1, hi), vt[:, :hi]).view(G, H // G, hi - lo, -1).permute(2, 0, 1, 3).reshape(hi - lo, H, -1)
    return out


def _turn(x, base, dims, neighbours=False):
    """Rotary positions 0, 1, ... on the first ``dims`` of ``x`` [T, heads, D]: pairs (i, i + dims/2), or neighbours."""
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=x.device) / dims)
    a = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None, None] * f
    c, s = torch.cos(a), torch.sin(a)
    if neighbours:
        u, v = x[..., 0:dims:2], x[..., 1:dims:2]
        return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), x[..., dims:]], -1)
    u, v = x[..., : dims // 2], x[..., dims // 2: dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], -1)


def _by_sequence(fn, lens, *flat):
    """``fn`` on each sequence's rows of the flat tensors, the results as flat rows."""
    return torch.cat([fn(*parts) for parts in zip(*(t.split(lens) for t in flat))])


def _padded(x, lens):
    return torch.nn.utils.rnn.pad_sequence(x.split(lens), batch_first=True)


def _flat(x, lens):
    return torch.cat([x[i, :n] for i, n in enumerate(lens)])


def _routed(x, scores, choice, top, scale, expert):
    """Sum of the chosen experts' outputs by the chosen scores' shares of their sum."""
    idx = torch.topk(choice, top, dim=-1).indices
    w = torch.gather(scores, 1, idx)
    w = w / (w.sum(-1, keepdim=True) + 1e-20) * scale
    out = torch.zeros_like(x)
    for e in torch.unique(idx).tolist():
        row, slot = torch.nonzero(idx == e, as_tuple=True)
        out.index_add_(0, row, expert(e, x[row]) * w[row, slot][:, None])
    return out


def _exact_m3(raw, W, ids, lens, rows):
    H, I, nq, nkv, hd = (raw[k] for k in ("hidden_size", "intermediate_size", "num_attention_heads", "num_key_value_heads", "head_dim"))
    eps, E = raw["rms_norm_eps"], raw["num_local_experts"]
    x = W("model.embed_tokens.weight", (raw["vocab_size"], H))[ids]
    for i in range(raw["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, eps) * W(p + "input_layernorm.weight", (H,))
        q = _rms(h @ W(p + "self_attn.q_proj.weight", (nq * hd, H)).T, eps) * W(p + "self_attn.q_norm.weight", (nq * hd,))
        k = _rms(h @ W(p + "self_attn.k_proj.weight", (nkv * hd, H)).T, eps) * W(p + "self_attn.k_norm.weight", (nkv * hd,))
        v = (h @ W(p + "self_attn.v_proj.weight", (nkv * hd, H)).T).view(-1, nkv, hd)

        def attend(q, k, v):
            turn = lambda t: _turn(t, raw["rope_theta"], raw["rotary_dim"])  # noqa: E731
            return _attend(turn(q), turn(k), v, hd ** -0.5)

        a = _by_sequence(attend, lens, q.view(-1, nq, hd), k.view(-1, nkv, hd), v)
        x = x + a.flatten(1) @ W(p + "self_attn.o_proj.weight", (H, nq * hd)).T
        h = _rms(x, eps) * W(p + "post_attention_layernorm.weight", (H,))
        m = p + "block_sparse_moe."
        scores = torch.sigmoid(h @ W(m + "gate.weight", (E, H)).T)

        def expert(e, y):
            g, u = y @ W(f"{m}experts.{e}.w1.weight", (I, H)).T, y @ W(f"{m}experts.{e}.w3.weight", (I, H)).T
            return (F.silu(g) * u) @ W(f"{m}experts.{e}.w2.weight", (H, I)).T

        x = x + _routed(h, scores, scores + W(m + "e_score_correction_bias", (E,)), raw["num_experts_per_tok"], 1.0, expert)
    return (_rms(x[rows], eps) * W("model.norm.weight", (H,))) @ W("lm_head.weight", (raw["vocab_size"], H)).T


def _causal_conv(u, w):
    """``u`` [B, T, C], ``w`` [C, taps], zeros before the start."""
    taps = w.shape[1]
    padded = F.pad(u, (0, 0, taps - 1, 0))
    return sum(w[:, j] * padded[:, j: j + u.shape[1]] for j in range(taps))


def _delta(W, p, m, width, h, lens, eps):
    H, D = m["heads"], m["dim"]
    lin = lambda n, a=H * D, b=width: W(p + n, (a, b)).T  # noqa: E731
    B, T = len(lens), max(lens)
    heads = lambda t: _padded(t, lens).view(B, T, H, D)  # noqa: E731
    r, k, v = (heads(h @ lin(n)) for n in "rkv")
    a = heads(torch.sigmoid(h @ lin("a") + W(p + "a.b", (H * D,))))
    low = torch.tanh(h @ lin("w1", 16)) @ lin("w2", H * D, 16) + W(p + "w0", (H * D,))
    decay = heads(torch.exp(-math.exp(-0.5) * torch.sigmoid(low)))
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    au = a * u
    S, out = h.new_zeros(B, H, D, D), h.new_empty(B, T, H, D)
    for t in range(T):
        uS = torch.matmul(u[:, t, :, None, :], S)
        S = decay[:, t, :, :, None] * S - au[:, t, :, :, None] * uS + k[:, t, :, :, None] * v[:, t, :, None, :]
        out[:, t] = torch.matmul(r[:, t, :, None, :], S).squeeze(2)
    out = _flat(_rms(out, eps), lens).flatten(1) * W(p + "norm", (H * D,)) * torch.sigmoid(h @ lin("g"))
    return out @ W(p + "o", (width, H * D)).T


def _latent(W, p, m, width, h, lens, eps):
    H, D, R, V, Q, C = (m[k] for k in ("heads", "dim", "rot_dim", "vdim", "q_rank", "kv_rank"))
    cq = _rms(h @ W(p + "dq", (Q, width)).T, eps) * W(p + "dq.norm", (Q,))
    q = (cq @ W(p + "uq", (H * (D + R), Q)).T).view(-1, H, D + R)
    down = h @ W(p + "dkv", (C + R, width)).T
    c = _rms(down[:, :C], eps) * W(p + "dkv.norm", (C,))
    k = (c @ W(p + "uk", (H * D, C)).T).view(-1, H, D)
    v = (c @ W(p + "uv", (H * V, C)).T).view(-1, H, V)
    sink = W(p + "sink", (H,))

    def attend(q, k, k_rot, v):
        turn = lambda t: _turn(t, m["rot"]["base"], m["rot"]["dims"])  # noqa: E731
        q = torch.cat([q[..., :D], turn(q[..., D:])], -1)
        k = torch.cat([k, turn(k_rot[:, None]).expand(-1, H, -1)], -1)
        return _attend(q, k, v, m["scale"], sink=sink)

    return _by_sequence(attend, lens, q, k, down[:, C:], v).flatten(1) @ W(p + "o", (width, H * V)).T


def _exact_guravik(raw, W, ids, lens, rows):
    width, eps = raw["width"], raw["norm"]["eps"]
    x = W("embed", (raw["vocab"], width))[ids]
    for i, layer in enumerate(raw["layers"]):
        p = f"l{i}."
        h = _rms(x, eps) * W(p + "norm1", (width,))
        h = h + _flat(_causal_conv(_padded(h, lens), W(p + "canon1", (width, raw["canon"]["taps"]))), lens)
        mixer = _delta if layer["type"] == "general_delta" else _latent
        y = mixer(W, p + "mix.", layer["mixer"], width, h, lens, eps)
        x = x + _rms(y, eps) * W(p + "norm1b", (width,))
        if layer["mlp"]:
            ff = layer["mlp"]["ff"]
            h = _rms(x, eps) * W(p + "norm2", (width,))
            y = F.silu(h @ W(p + "mlp.gate", (ff, width)).T) * (h @ W(p + "mlp.up", (ff, width)).T)
            x = x + _rms(y @ W(p + "mlp.down", (width, ff)).T, eps) * W(p + "norm2b", (width,))
    return (_rms(x[rows], eps) * W("final.norm", (width,))) @ W("head", (raw["vocab"], width)).T


def _decayed(q, k, v, decay, put):
    """``S <- decay S + put k v^T``, ``o = S^T q`` for ``q``, ``k`` [B, T, H, D], ``v`` [B, T, H, V], gates [B, T, H]."""
    B, T, H, D = k.shape
    S, out = q.new_zeros(B, H, D, v.shape[3]), q.new_empty(B, T, H, v.shape[3])
    pk = put[..., None] * k
    for t in range(T):
        S = torch.baddbmm((decay[:, t, :, None, None] * S).flatten(0, 1), pk[:, t].reshape(B * H, D, 1), v[:, t].reshape(B * H, 1, -1)).view_as(S)
        out[:, t] = torch.matmul(q[:, t, :, None, :], S).squeeze(2)
    return out


def _memory(W, p, m, width, h, lens, eps):
    H, D, V, cap = m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    B, T = len(lens), max(lens)
    lin = lambda n, a: h @ W(p + n, (a, width)).T  # noqa: E731
    q, k, v = (_padded(lin(n, H * d), lens).view(B, T, H, d) for n, d in (("q", D), ("k", D), ("v", V)))
    i = _padded(cap * torch.tanh((lin("i", H) + W(p + "i.b", (H,))) / cap), lens)
    f = _padded(F.logsigmoid(cap * torch.tanh((lin("f", H) + W(p + "f.b", (H,))) / cap)), lens)
    top, now = torch.empty_like(i), h.new_zeros(B, H)
    before = torch.empty_like(i)
    for t in range(T):
        before[:, t] = now
        now = top[:, t] = torch.maximum(f[:, t] + now, i[:, t])
    keep, put = torch.exp(f + before - top), torch.exp(i - top)
    o = _decayed(q * D ** -0.5, k, torch.cat([v, torch.ones_like(v[..., :1])], -1), keep, put)      # the last column: n . q
    o = o[..., :V] / (torch.maximum(o[..., V:].abs(), torch.exp(-top)[..., None]) + 1e-6)
    o = _flat(_rms(o, eps), lens).flatten(1) * W(p + "norm", (H * V,)) * torch.sigmoid(lin("g", H * V))
    return o @ W(p + "o", (width, H * V)).T


def _state_space(W, p, m, width, h, lens, eps):
    H, V, N, G, parts, taps = (m[k] for k in ("heads", "vdim", "state", "groups", "norm_groups", "conv"))
    inner, C, B, T = H * V, H * V + 2 * G * N, len(lens), max(lens)
    z, u, dt = (h @ W(p + "in", (inner + C + H, width)).T).split([inner, C, H], 1)
    u = F.silu(_causal_conv(_padded(u, lens), W(p + "conv", (C, taps))) + W(p + "conv.b", (C,)))
    x, b, c = u.split([inner, G * N, G * N], 2)
    x = x.reshape(B, T, H, V)
    b, c = (t.reshape(B, T, G, 1, N).expand(-1, -1, -1, H // G, -1).reshape(B, T, H, N) for t in (b, c))
    dt = _padded(F.softplus(dt + W(p + "dt_bias", (H,))), lens)
    y = _decayed(c, b, x, torch.exp(-torch.exp(W(p + "A_log", (H,))) * dt), dt) + W(p + "D", (H,))[:, None] * x
    y = _flat(y, lens).flatten(1) * F.silu(z)
    y = _rms(y.view(-1, parts, inner // parts), eps).flatten(1) * W(p + "norm", (inner,))
    return y @ W(p + "o", (width, inner)).T


def _side_by_side(W, p, m, width, h, lens, eps):
    a, r = m["left"], m["right"]
    H, G, D = a["heads"], a["kv_heads"], a["dim"]
    q = (h @ W(p + "left.q", (H * D, width)).T + W(p + "left.q.b", (H * D,))).view(-1, H, D)
    v = (h @ W(p + "left.k", (G * D, width)).T + W(p + "left.k.b", (G * D,))).view(-1, G, D)

    def attend(q, v):
        turn = lambda t: _turn(t, a["rot"]["base"], a["rot"]["dims"], neighbours=True)  # noqa: E731
        return _attend(turn(q), turn(v), v, a["scale"], cap=a["softcap"], window=a["mask"]["size"])

    left = _by_sequence(attend, lens, q, v).flatten(1) @ W(p + "left.o", (width, H * D)).T
    H, D, V, B, T = r["heads"], r["dim"], r["vdim"], len(lens), max(lens)
    lin = lambda n, s: h @ W(p + "right." + n, (s, width)).T  # noqa: E731
    q, k, v = (_padded(F.silu(lin(n, H * d)), lens).view(B, T, H, d) for n, d in (("q", D), ("k", D), ("v", V)))
    decay = torch.tensor(r["decay"], dtype=torch.float64, device=h.device).expand(B, T, H)
    o = _flat(_decayed(q, k, v, decay, torch.ones_like(decay)), lens).flatten(1)
    o = _rms(o, eps) * W(p + "right.norm", (H * V,)) * torch.sigmoid(lin("g", H * V))
    return m["left_scale"] * left + m["right_scale"] * (o @ W(p + "right.o", (width, H * V)).T)


def _exact_gedelorn(raw, W, ids, lens, rows):
    width, eps = raw["width"], raw["norm"]["eps"]
    norm = lambda t, n: _rms(t, eps) * (1.0 + W(n, (width,)))  # noqa: E731
    x = W("embed", (raw["vocab"], width))[ids]
    for i, layer in enumerate(raw["layers"]):
        p, mlp = f"l{i}.", layer["mlp"]
        mixer = {"mlstm": _memory, "mamba2": _state_space, "parallel": _side_by_side}[layer["type"]]
        x = x + norm(mixer(W, p + "mix.", layer["mixer"], width, norm(x, p + "norm1"), lens, eps), p + "norm1b")
        h, m = norm(x, p + "norm2"), p + "mlp."
        if mlp["kind"] == "dense":
            y = F.silu(h @ W(m + "gate", (mlp["ff"], width)).T) * (h @ W(m + "up", (mlp["ff"], width)).T)
            y = y @ W(m + "down", (width, mlp["ff"])).T
        else:
            def squared(name, t, f):
                return F.relu(t @ W(name + "up", (f, width)).T) ** 2 @ W(name + "down", (width, f)).T

            scores = torch.sigmoid(h @ W(m + "router", (mlp["router"]["experts"], width)).T)
            y = _routed(h, scores, scores, mlp["router"]["top"], mlp["router"]["scale"],
                        lambda e, t: squared(f"{m}e{e}.", t, mlp["expert"]["ff"])) + squared(m + "shared.", h, mlp["shared"]["ff"])
        x = x + norm(y, p + "norm2b")
    return norm(x[rows], "final.norm") @ W("head", (raw["vocab"], width)).T


def _exact_logits(case, seed, texts, wants):
    """Logits of the wanted places of whole texts, in the order of the texts."""
    model, float32 = case["model"], case["kind"] == "generate"
    W = lambda name, shape: _tensor(model, seed, name, shape, float32).double()  # noqa: E731
    lens = [len(t) for t in texts]
    ids = torch.tensor([t for text in texts for t in text], device=DEVICE)
    at, rows = 0, []
    for n, want in zip(lens, wants):
        rows += [at + w for w in want]
        at += n
    fn = {"m3": _exact_m3, "m3_small": _exact_m3, "guravik": _exact_guravik, "gedelorn": _exact_gedelorn}[model]
    return fn(RAW[model], W, ids, lens, torch.tensor(rows, device=DEVICE))


def exact(case: dict, seed: int):
    prompts, fed, portion = _tokens(case, seed)
    kind, n = case["kind"], case["requests"]
    if kind == "prompt":
        return _exact_logits(case, seed, prompts, [range(max(0, len(p) - case["want"]), len(p)) for p in prompts])
    if kind == "generate":
        texts = [list(p) for p in prompts]
        for _ in range(case["steps"]):
            best = _exact_logits(case, seed, texts, [[len(t) - 1] for t in texts]).argmax(-1).tolist()
            texts = [t + [b] for t, b in zip(texts, best)]
        steps = case["steps"]
        return {"tokens": torch.tensor([t[-steps:] for t in texts]),
                "logits": _exact_logits(case, seed, [t[:-1] for t in texts], [range(len(t) - 1 - steps, len(t) - 1) for t in texts])}
    steps = case.get("steps", 1)
    texts = [p + [fed[j][i] for j in range(WARM + steps)] for i, p in enumerate(prompts)]
    wants = [range(len(t) - steps, len(t)) for t in texts]
    if kind == "mixed":
        texts, wants = texts + [portion], wants + [[len(portion) - 1]]
        return _exact_logits(case, seed, texts, wants)
    lg = _exact_logits(case, seed, texts, wants).view(n, steps, -1)
    return [lg[:, j].contiguous() for j in range(steps)]
