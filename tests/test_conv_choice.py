"""When a step of single tokens takes norm and short convolution in one launch: for the very parts whose work that launch knows, and for operands
that it can move."""
from __future__ import annotations

import pytest
import torch

from quanta_b200.parts.base import NormedPending
from quanta_b200.parts.conv import ResidualShortConv
from quanta_b200.parts.norms import NoNorm, RMSNorm, takes_conv

H, T, TAPS = 64, 2, 3


class Doubled(RMSNorm):
    def forward(self, h, delta, out, rows=None, store_h=True):
        super().forward(h, delta, out, rows, store_h)
        out.mul_(2)


class Silent(ResidualShortConv):
    def forward(self, x, ctx, state, out):
        out.zero_()


def _place(*shape, off=0):
    n = torch.Size(shape).numel()
    return torch.zeros(n + 8)[off: off + n].view(shape)


def _choice(norm=RMSNorm, conv=ResidualShortConv, after=RMSNorm, pending=True, off=None, groups=1):
    at = lambda name, *shape: _place(*shape, off=1 if off == name else 0)  # noqa: E731
    n = norm(H, 1e-5, "w", groups=groups) if norm is not NoNorm else NoNorm(H)
    a = after(H, 1e-5, "w") if after is not NoNorm else NoNorm(H)
    n.weight, a.weight = at("weight", H), at("gain", H)
    c = conv(H, TAPS, "c")
    c.weight = at("taps", H, TAPS)
    delta = NormedPending(at("y", T, H), a) if pending else at("y", T, H)
    return takes_conv(n, delta, c, {c.state_name: at("state", 4, TAPS - 1, H)}, at("h", T, H), at("out", T, H))


def test_the_parts_it_knows():
    assert _choice()


@pytest.mark.parametrize("other", [dict(norm=Doubled), dict(norm=NoNorm), dict(conv=Silent), dict(after=NoNorm), dict(pending=False), dict(groups=2)])
def test_other_parts_keep_their_own_launches(other):
    assert not _choice(**other)


@pytest.mark.parametrize("off", ["weight", "gain", "taps", "y", "state", "h", "out"])
def test_operands_that_do_not_start_on_16_bytes_keep_the_two_launches(off):
    assert not _choice(off=off)
