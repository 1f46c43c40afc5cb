"""What belongs to the device that is current is asked for with every launch.  A kernel's limit of shared memory is raised on that device, and
the number of SMs is its own: kept in a static variable either would hold for the first device of a process only."""
from __future__ import annotations

import re

from quanta_b200.csrc import build


def test_limits_are_raised_with_every_launch():
    kept = [(p.name, m.group(0)) for p in sorted(build.SRC_DIR.glob("*.cu*"))
            for m in re.finditer(r"\bstatic\s+(?:const\s+)?\w+\s+\w+\s*=\s*cudaFuncSetAttribute", p.read_text())]
    assert not kept
    assert any("cudaFuncSetAttribute" in p.read_text() for p in build.SRC_DIR.glob("*.cu"))


def test_no_property_of_a_device_is_kept():
    kept = [(p.name, m.group(1)) for p in sorted(build.SRC_DIR.glob("*.cu*")) for m in re.finditer(r"\bstatic\s+int\s+(\w+)\b", p.read_text())
            if re.search(rf"cudaDeviceGetAttribute\(&{m.group(1)}\b", p.read_text())]
    assert not kept
