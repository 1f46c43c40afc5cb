"""A kernel's limit of shared memory belongs to the device that is current when it is raised, so it is raised with every launch: kept in a
static variable it would hold for the first device of a process only."""
from __future__ import annotations

import re

from quanta_b200.csrc import build


def test_limits_are_raised_with_every_launch():
    kept = [(p.name, m.group(0)) for p in sorted(build.SRC_DIR.glob("*.cu*"))
            for m in re.finditer(r"\bstatic\s+(?:const\s+)?\w+\s+\w+\s*=\s*cudaFuncSetAttribute", p.read_text())]
    assert not kept
    assert any("cudaFuncSetAttribute" in p.read_text() for p in build.SRC_DIR.glob("*.cu"))
