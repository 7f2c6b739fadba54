"""The packed pair kernel's order over a record, restated in Python: eight lanes, lane l with
the i atoms l and l + 8, meets at step k of group g entry 8 g + ((l + k) & 7); a record's
stored mask words (entry halves rotated right by the i atom) become that order's bits by
step_mask (j_presto_b200/csrc/jp_pair.cu).  Every listed (i atom, entry) pair is met once and no
other, the j-force accumulator a lane ends a group with is that of entry (l + 7) & 7, and the
staged copies a lane reads are the entries it meets.
"""
import random

import pytest

M32 = 0xFFFFFFFF


def stored_word(row, r):
    """k_ct_emit's word of i atom r: each 16-bit half of the entry bits rotated right by r"""
    lo, hi = row & 0xFFFF, row >> 16
    rot = lambda v: ((v >> r) | (v << (16 - r))) & 0xFFFF  # noqa: E731
    return rot(lo) | (rot(hi) << 16)


def byte_rotr(row, l):
    m = ((0xFF >> l) * 0x01010101) & M32
    return ((row >> l) & m) | ((row << (8 - l)) & ~m & M32)


def step_mask(w, r):
    lo, hi = (w & 0xFFFF) * 0x10001, (w >> 16) * 0x10001
    row = (((lo << r) & M32) >> 16) | ((hi << r) & 0xFFFF0000)
    return byte_rotr(row, r & 7)


@pytest.mark.parametrize("seed", range(4))
def test_every_listed_pair_is_met_once(seed):
    rng = random.Random(seed)
    rows = [rng.getrandbits(32) if seed else M32 for _ in range(16)]
    met = []
    for l in range(8):
        for half in (0, 8):
            r = l + half
            m = step_mask(stored_word(rows[r], r), r)
            met += [(r, 8 * g + ((l + k) & 7)) for g in range(4) for k in range(8) if (m >> (8 * g + k)) & 1]
    want = [(r, e) for r in range(16) for e in range(32) if (rows[r] >> e) & 1]
    assert sorted(met) == want


def test_rotation_brings_each_entry_home():
    acc = [[] for _ in range(8)]                 # per lane: the entries its accumulator holds
    typ = list(range(8))                         # per lane: the type word it carries
    for k in range(8):
        for l in range(8):
            acc[l].append((l + k) & 7)
            assert typ[l] == (l + k) & 7
            assert (l + k) % 8 == (l + k) - (8 if l + k >= 8 else 0)   # slot l + k of the doubled stage
        if k < 7:                                # every lane takes its neighbour's
            acc = [acc[(l + 1) & 7] for l in range(8)]
            typ = [typ[(l + 1) & 7] for l in range(8)]
    for l in range(8):
        assert acc[l] == [(l + 7) & 7] * 8
