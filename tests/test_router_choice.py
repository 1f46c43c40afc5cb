"""Which way a routed step takes.  The router: the tensor cores' copies start on 16 bytes, the CUDA cores take rows that start anywhere."""
from __future__ import annotations

import pytest
import torch

from quanta_b200.parts.moe import SigmoidTopKExperts


@pytest.mark.parametrize("tokens", [65, 95, 300])
@pytest.mark.parametrize("off,tensor_cores", [(0, True), (8, True), (1, False), (4, False)])
def test_rows_that_start_anywhere(tokens, off, tensor_cores):
    part = SigmoidTopKExperts.__new__(SigmoidTopKExperts)
    part.E, part.H, part.gate_pieces = 8, 64, torch.empty(0)
    x = torch.zeros(tokens * 64 + 16, dtype=torch.bfloat16)[off: off + tokens * 64].view(tokens, 64)
    assert part._on_tensor_cores(x) == tensor_cores


@pytest.mark.parametrize("inner,rows", [(768, 32), (8192, 32), (8200, 10), (14336, 10)])
def test_token_rows_are_fetched_inside_where_that_is_no_slower(inner, rows):
    part = SigmoidTopKExperts.__new__(SigmoidTopKExperts)
    part.E, part.I = 8, inner
    assert part.gathers_inside(8 * rows) and not part.gathers_inside(8 * rows + 1)
