"""Which kernel takes a step's single tokens, and which captured step: a request's keys are walked by blocks of its own in one kernel and
shared by all blocks in the other, so the mix of lengths decides.  Rules of sizes alone; the times they stand on are beside the code."""
from __future__ import annotations

import pytest
import torch

from quanta_b200 import kernels as k
from quanta_b200.engine.step import Engine


@pytest.mark.parametrize("nq,nkv", [(48, 8), (16, 4), (6, 1), (8, 8)])
def test_like_lengths_unlike_lengths_and_few_units(nq, nkv):
    wins = lambda lens, **kw: k.attn_decode_direct_wins(len(lens), nq, nkv, 128, max(lens), sum(lens), kw.pop("window", 0), **kw)
    for n in (1, 17, 500, 2000, 8000):                                     # up to some thousand keys, alike
        for batch in (1, 2, 5, 8, 16, 64):
            assert wins([n] * batch) and wins([n] * batch, two_part=True)
    for batch in (64, 128):                                                # the SMs are full
        assert wins([60000] * batch)
    assert not wins([131072] + [500] * 31) and not wins([32000] + [500] * 31)
    if nq == 4 * nkv:
        assert not wins([131072] + [500] * 15, two_part=True)
    assert wins([131072] + [500] * 15, window=1024) and wins([131072] + [500] * 15, chunk=512)
    if nkv == 1:
        assert not wins([131072]) and wins([24000])                        # eight blocks on 148 SMs
    # more keys in the other requests never speak against the kernel, more in the longest never for it
    for two in (False, True):
        for longest in (4000, 30000, 100000):
            chosen = [wins([longest] + [n] * 15, two_part=two) for n in (1, longest // 8, longest // 4, longest // 2, longest)]
            assert chosen == sorted(chosen)
    assert not k.attn_decode_direct_wins(4, nkv * 9, nkv, 128, 500, 2000, 0) and not k.attn_decode_direct_wins(4, nq, nkv, 64, 500, 2000, 0)
    assert not k.attn_decode_direct_wins(0, nq, nkv, 128, 500, 0, 0)


def test_captured_steps():
    key = Engine._graph_key
    assert key([1]) == (1, 512) and key([513]) == (1, 1024) and key([100000]) == (1, 131072)
    assert key([40, 2000, 3]) == (3, 2048)                                 # short contexts: one class
    assert key([5000] * 4) == (4, 8192) and key([5000, 4000, 2000, 1500]) == (4, 8192)
    assert key([5000, 300, 300, 300]) == (4, 8192, "uneven") and key([9000, 100]) == (2, 16384, "uneven")
    assert key([9000], 4) == (4, 16384)                                    # lengths that are not known


def test_a_block_or_a_warp_a_range_of_keys():
    rows = lambda dtype, T, nq, nkv, hd, vd=None: k.window_attention_by_rows(dtype, T, nq, nkv, hd, vd or hd)
    for dtype in (torch.float32, torch.bfloat16):
        for nq, nkv, hd in ((16, 4, 128), (8, 8, 64), (6, 2, 128), (5, 5, 36), (12, 2, 256), (16, 4, 16)):
            assert rows(dtype, 1, nq, nkv, hd)                             # few blocks
        assert rows(dtype, 4096, 16, 4, 128) and rows(dtype, 64, 16, 4, 64)
        for nq, nkv, hd in ((5, 5, 36), (12, 2, 256), (16, 4, 16), (16, 4, 32), (6, 2, 128), (8, 8, 64), (6, 1, 64)):
            assert not rows(dtype, 1000, nq, nkv, hd)
        assert not rows(dtype, 1, 4, 2, 50) and not rows(dtype, 1, 4, 2, 64, 66) and not rows(dtype, 1, 5, 2, 64)
