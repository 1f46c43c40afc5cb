"""Bounded waits between the warps of a block: whichever warp gives up, the block records it.  The status word is written behind a barrier that
every warp reaches after its last wait; a warp that left before it, or a record that only one role writes, could lose a failure."""
from __future__ import annotations

import re

import pytest

from quanta_b200.csrc import build
from tests.test_launch_order import _functions

WAIT = re.compile(r"\w+_wait\([^;]*\babort_flag\)")


def _without_lambdas(body: str) -> str:
    while m := re.search(r"\[[&=\w, ]*\]\s*\([^()]*\)\s*\{", body):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(body[at], 0)
            at += 1
        body = body[: m.start()] + "0" + body[at:]
    return body


def _waiting():
    for path in sorted(build.SRC_DIR.glob("*.cu")):
        for name, _, body in _functions(path.read_text()):
            if WAIT.search(body):
                yield pytest.param(body, id=f"{path.stem}-{name}")


@pytest.mark.parametrize("body", list(_waiting()))
def test_a_wait_that_ran_out_is_recorded_behind_the_last_barrier(body):
    body = _without_lambdas(body)
    first, last = WAIT.search(body).start(), [m.end() for m in WAIT.finditer(body)][-1]
    barrier = body.rindex("__syncthreads();")
    records = [m.start() for m in re.finditer("QB_STATUS_WAIT_TIMEOUT", body)]
    assert last < barrier and records and all(at > barrier for at in records)
    assert not re.search(r"\breturn;", body[first: barrier])


def test_the_waits_are_found():
    assert len(list(_waiting())) >= 6


def test_router_logits_that_a_wait_kept_back_are_no_numbers():
    """The router takes no status words from some callers: what it could not sum is NaN there, and the selection passes NaN on (its experts
    stay inside the table, see the GPU test of the selection)."""
    (body,) = [b for n, _, b in _functions((build.SRC_DIR / "router_gemm_mma.cu").read_text()) if n == "router_gemm_tc_kernel"]
    sums = body[body.index("float total[COLS]"):]
    assert re.search(r"if \(!ok\) \{[^}]*total\[i\] = __int_as_float\(0x7fffffff\);\s*\}", sums)
    assert "if (ok && e < E)" not in sums and "items && ok" not in body[body.index("const int quarter"):]
