"""The fused triplet kernel's index arithmetic on the CPU: the room for a
warp's list (the library's own bound) against the walk of stripes of 8 rows
and groups of 4 columns over every split of the neighbours into species, each
pair visited once, the column numbering of the reverse pass, its tile reads,
and that one warp an atom always fits in shared memory."""
from __future__ import annotations

import itertools

import numpy as np
import pytest

MAX_CAP = 128


def _walk(counts, warps):
    """Per warp, per species block, the pairs (a, b) in reach (all of them)."""
    off = np.concatenate([[0], np.cumsum(counts)])
    ns = len(counts)
    out = [[] for _ in range(warps)]
    for al in range(ns):
        for be in range(al, ns):
            oa, ea, ob, eb = off[al], off[al + 1], off[be], off[be + 1]
            for w in range(warps):
                pairs = []
                st = oa >> 3
                while 8 * st < ea and ea > oa:
                    g = max(ob, max(oa, 8 * st) + 1) >> 2
                    g += (w - g) & (warps - 1)
                    while 4 * g < eb:
                        for lane in range(32):
                            a, b = 8 * st + (lane & 7), 4 * g + (lane >> 3)
                            if oa <= a < ea and max(ob, a + 1) <= b < eb:
                                pairs.append((a, b))
                        g += warps
                    st += 1
                out[w].append(pairs)
    return out


def _splits(n):
    yield (n,)
    for a in {0, 1, n // 3, n // 2, n - 1, n}:
        yield (a, n - a)
    for a, b in itertools.product({0, 1, n // 4, n // 2}, repeat=2):
        if a + b <= n:
            yield (a, b, n - a - b)


@pytest.mark.parametrize("warps", [1, 2, 4, 8])
@pytest.mark.parametrize("n", [2, 3, 8, 9, 31, 40, 72, MAX_CAP])
def test_lists_fit_and_hold_every_pair_once(n, warps):
    import maise_b200

    lib = maise_b200.load_library()
    cap = (n + 7) & ~7
    room = lib.mbk_tri_list(cap, warps)
    for counts in _splits(n):
        lists = _walk(counts, warps)
        seen = [p for w in lists for block in w for p in block]
        assert len(seen) == n * (n - 1) // 2 and len(set(seen)) == len(seen)
        for w, blocks in enumerate(lists):
            assert sum((len(p) + 3) & ~3 for p in blocks) <= room  # blocks padded to 4 entries
            for a, b in (p for block in blocks for p in block):
                col = ((b >> 2) // warps << 2) | (b & 3)  # number among the warp's columns
                assert (((col >> 2) * warps + w) << 2 | (col & 3)) == b


def test_tile_reads_are_conflict_free():
    """FP64 operand reads of a half-warp: a tile row of 20 doubles, its
    transpose, and the staging rows of 36, touch 16 distinct 8-byte banks."""
    lanes = np.arange(32).reshape(2, 16)
    for half in lanes:
        for addr in (20 * (half >> 2) + (half & 3), 20 * (half & 3) + (half >> 2), 36 * (half >> 2) + (half & 3)):
            assert len(set(addr % 16)) == 16


def test_one_warp_an_atom_always_fits():
    import ctypes

    import maise_b200

    lib = maise_b200.load_library()
    lib.mbk_tri_smem.restype = ctypes.c_size_t
    # the most the parser takes: 1024 inputs, 3 species, 32 pair functions
    assert 4 * lib.mbk_tri_smem(MAX_CAP, 1024, 3, 32, 1) <= 226 * 1024  # four atoms a CTA
