"""Launches that follow one another without a gap (their blocks are placed while the launch before ends): a captured decode step, whose
launches are edges of a graph, gives the bits of the same step launched one by one, step after step and with several batch sizes."""
from __future__ import annotations

import pytest
import torch

from tests import helpers as H
from tests import test_gedelorn_gpu as gedelorn
from tests import test_guravik_gpu as guravik
from tests.conftest import TINY

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("which", ["minimax", "guravik", "gedelorn"])
def test_captured_and_eager_steps_agree(which, dtype, model_dirs, tmp_path_factory):
    from quanta_b200.engine.model import load_model
    from quanta_b200.engine.step import Engine, StepEntry
    if which == "minimax":
        folder, vocab = model_dirs["D"], TINY["D"]["vocab_size"]
    else:
        module = {"guravik": guravik, "gedelorn": gedelorn}[which]
        folder, _, cfg = module._folder(tmp_path_factory, "D")
        vocab = cfg["vocab"]
    model, _ = load_model(folder, dtype=dtype)
    engines = [Engine(model, num_pages=400, page_size=16, max_requests=8, use_graphs=graphs) for graphs in (True, False)]
    replays = 0
    for turn in range(5):
        batch = (1, 3, 8)[turn % 3] if turn < 4 else 1
        # the longest request has 512 tokens after its last step, so that the captured step's bounds are those of the step itself
        reqs = {f"{turn}.{i}": H.random_tokens(512 - 31 * i, vocab, 900 + 10 * turn + i) for i in range(batch)}
        for again in range(3):
            got = []
            for eng in engines:
                for rid, toks in reqs.items():
                    eng.step([StepEntry(f"{rid}.{again}", toks[:-1], ())])
                out = eng.step([StepEntry(f"{rid}.{again}", toks[-1:], (0,)) for rid, toks in reqs.items()], end=[f"{r}.{again}" for r in reqs])
                eng.check()
                got.append(out.clone())
            assert torch.isfinite(got[0]).all() and torch.equal(*got), (turn, again)
    replays = engines[0].graph_replays
    assert replays >= 8 and engines[1].graph_replays == 0
