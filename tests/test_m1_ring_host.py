"""The rings of the one-row kernels.  Four warp groups take the fills in turn (group f % 4 takes fill f, which lies in slot f % depth) and
wait for a slot by the parity of its phase.  A parity cannot tell phase k from phase k - 2, so a group has to see every phase of the
slots that it waits for: the depth is a multiple of four."""
import ctypes
import random

import pytest

from boostr_b200 import _cabi
from boostr_b200.format import QuantFormat as F


def _early(depth, nfill, rng):
    """Runs the groups in a random order; True if a wait passed before its fill had landed."""
    phase = [0] * depth                     # fills that have landed in a slot
    issued, landed = set(range(min(depth, nfill))), set()
    nxt = [0, 1, 2, 3]
    while min(nxt) < nfill:
        pending = sorted(issued - landed)
        if pending and rng.random() < 0.6:  # copies land in the order in which they were issued
            f = pending[0]
            landed.add(f)
            phase[f % depth] += 1
        g = rng.choice((0, 0, 0, 1, 1, 2, 3))  # groups of different speed
        f = nxt[g]
        if f < nfill and phase[f % depth] & 1 != f // depth & 1:  # mbarrier.try_wait.parity
            if f not in landed:
                return True
            nxt[g] += 4
            if f + depth < nfill:
                issued.add(f + depth)
    return False


def test_a_parity_passes_early_in_a_ring_that_groups_share():
    rng = random.Random(1)
    assert any(_early(13, 400, rng) for _ in range(50))
    assert not any(_early(12, 400, rng) for _ in range(50))


@pytest.mark.parametrize("fmt", ["Q4_0", "Q8_0", "Q4_K", "Q6_K"])
def test_ring_depths(fmt):
    depth = _cabi.lib().b200q_m1_ring_depth
    depth.restype, depth.argtypes = ctypes.c_int, [ctypes.c_int, ctypes.c_size_t, ctypes.c_int]
    got = [depth(F[fmt].format_id, k, sw) for k in range(32, 16385, 32) for sw in (0, 1)]
    assert max(got) >= 8 and all(d == 0 or (d >= 4 and d % 4 == 0) for d in got), sorted(set(got))
