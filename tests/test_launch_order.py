"""Kernels that may be placed while the launch before them runs (``qb_follow`` in ``csrc/common.cuh``): what that launch may still be writing is
not read through a ``__restrict__`` pointer.  Such a pointer tells the compiler that nobody else writes there while the kernel runs, and the
read may be moved in front of the wait."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "quanta_b200" / "csrc"
# parameters that these kernels only ever write (reads of other pointers may then pass the stores)
WRITTEN_ONLY = {"out", "cq", "cache", "part", "q_plain", "q_rot", "q_out", "k_cache", "v_cache", "den", "log_decay", "weight", "floor_out", "h",
                "w_out", "plan", "sorted_pair", "tile_expert", "tile_row0"}
# of these names, the ones that a kernel reads as well
READ_TOO = {"attn_decode_direct_kernel": {"k_cache", "v_cache"}, "latent_attend_mma_kernel": {"cache"}, "latent_merge_kernel": {"part"},
            "add_rmsnorm_rows_kernel": {"h"}, "normed_add_rmsnorm_rows_kernel": {"h"}, "decay_out_kernel": {"den"},
            "expert_gemm_tc_body": {"plan", "sorted_pair", "tile_expert", "tile_row0"}}


def _functions(text: str):
    """(name, parameters, body) of the kernels and of the device functions."""
    text = re.sub(r"//[^\n]*", "", text)
    text = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)
    for m in re.finditer(r"(?:__global__|__device__)\s[^;{}]*?\b(\w+)\s*\(([^;{}]*)\)\s*(?:const\s*)?\{", text):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield m.group(1), m.group(2), text[m.end(): at]


def _followers():
    for path in sorted(CSRC.glob("*.cu*")):
        macros = dict(re.findall(r"#define (\w+_PARAMS)((?:.*\\\n)*.*)", path.read_text()))
        for name, params, body in _functions(path.read_text()):
            if "qb_follow()" in body or any(m in params for m in macros):
                yield pytest.param(path.name, name, macros.get(params.strip(), params), id=f"{path.stem}-{name}")


@pytest.mark.parametrize("source,name,params", list(_followers()))
def test_what_the_launch_before_writes_is_not_restricted(source, name, params):
    marked = {re.search(r"(\w+)\s*$", p).group(1): p for p in params.replace("\\", " ").split(",") if "__restrict__" in p}
    assert not [p for p in marked.values() if re.search(r"\bconst\b", p)]
    assert not (set(marked) - WRITTEN_ONLY) and not (set(marked) & READ_TOO.get(name, set()))


def test_the_kernels_are_found():
    assert len(list(_followers())) >= 26
