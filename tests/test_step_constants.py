"""The search step's sentinel as the sources state it (search_step.cuh) against what the step needs of
it: bits for every step a parked lane may take between two refreshes (plain.cu, batched.cu), a row
that stays without candidates whatever bits have been placed, and no solution counted."""
import os
import re

import pytest

from conftest import PKG_DIR

M32 = 0xFFFFFFFF


def source(name):
    with open(os.path.join(PKG_DIR, "csrc", name)) as f:
        return f.read()


def constant(text, name):
    return int(re.search(rf"\b{name} = (0x[0-9A-Fa-f]+|\d+)u?[,;]", text).group(1), 0)


STEP = source("search_step.cuh")
AVAIL, NC, L = (constant(STEP, k) for k in ("kSentinelAvail", "kSentinelNc", "kSentinelL"))
PARKED = constant(STEP, "kMaxParkedSteps")


def test_the_entry_written_is_the_one_modelled():
    # {avail, nc, l, r}; an entry lies in memory as {nc, avail, r, l}, so the refresh writes its second word
    assert "make_uint4(kSentinelAvail, kSentinelNc, kSentinelL, 0u)" in STEP
    assert "[%0+4], %1" in STEP.split("void refresh_sentinel")[1][:200]
    assert bin(AVAIL).count("1") > PARKED


@pytest.mark.parametrize("kernel", ["plain.cu", "batched.cu"])
def test_parked_lane_between_refreshes(kernel):
    text = source(kernel)
    refresh = constant(text, "kRefresh")
    unroll = int(re.search(r"(?:kUnroll = |NQB_BATCHED_UNROLL )(\d+)", text).group(1))
    assert refresh <= PARKED and unroll % refresh == 0 and refresh % 2 == 0
    # whole rounds, refreshed as the kernel does it; the lane's row of a moment ago is arbitrary
    stack, a = (AVAIL, NC, L, 0), 0
    for step in range(3 * unroll):
        if step % unroll % refresh == 0:
            stack = (AVAIL,) + stack[1:]
        assert a == 0  # the row entered before had no candidate: pop
        a, nc, l, r = stack
        b, a = a & -a, a & (a - 1)
        assert b and a  # something to place, and something left to push back into the same slot
        stack = (a, nc, l, r)
        nc &= ~b
        x = (2 * b + l) & M32
        l, r = (x << 1) & M32, ((r + b) & M32) >> 1
        a = nc & ~(x | r)
        assert a == 0 and nc & (nc - 1)  # no node, and not a last row
