"""Warp-private regions of the 256 x 256 cluster FFT (csrc/fft256_cluster.cuh), restated here:
every layout is injective, a warp's four lines stay inside its own region (so the line-local
exchanges need no CTA barrier), every local warp access touches each of the 16 float2 bank pairs
at most twice (two 128-byte wavefronts), and remote stores fill whole sectors."""
from collections import Counter

import pytest

GS, LP, BP, AP = 1056, 264, 260, 256


def lx(ln, k1, t):
    return (ln >> 2) * GS + (ln & 3) * LP + 33 * (k1 >> 2) + 8 * (k1 & 3) + t


def bx(kcl, r):
    return (kcl >> 2) * GS + (kcl & 3) * BP + r


def ax(rl, kc):
    return (rl >> 2) * GS + (rl & 3) * AP + (kc & ~3) + ((kc + 2 * (kc >> 4 & 1) + (rl & 1)) & 3)


LAYOUTS = [lambda a, b: lx(a, b >> 3, b & 7), bx, ax]


def _worst(addrs):
    return max(Counter(a % 16 for a in addrs).values())


@pytest.mark.parametrize("fn", LAYOUTS)
def test_injective_and_inside_the_warps_region(fn):
    idx = {}
    for ln in range(64):
        for j in range(256):
            a = fn(ln, j)
            assert a not in idx
            idx[a] = ln
            assert (ln >> 2) * GS <= a < ((ln >> 2) + 1) * GS


def test_two_wavefronts_per_access():
    for w in range(16):
        lanes = range(32 * w, 32 * w + 32)
        for k1 in range(32):
            assert _worst([lx(t >> 3, k1, t & 7) for t in lanes]) <= 2
        for a in range(4):
            for tt in range(8):
                assert _worst([lx(t >> 3, 4 * (t & 7) + a, tt) for t in lanes]) <= 2
            for kB in range(8):
                assert _worst([ax(t >> 3, 4 * (t & 7) + a + 32 * kB) for t in lanes]) <= 2  # A reads
        for e in range(32):
            assert _worst([bx(t >> 3, (t & 7) + 8 * e) for t in lanes]) <= 2  # B reads


def test_remote_stores_fill_whole_sectors():
    """Each remote store of a warp writes 8 aligned 32-byte sectors (4 float2 each)."""
    for w in range(16):
        lanes = range(32 * w, 32 * w + 32)
        for q in range(4):
            for a in range(4):
                for x in range(2):  # A -> B
                    assert len({bx(4 * (t & 7) + a + 32 * x, 64 * q + (t >> 3)) // 4 for t in lanes}) == 8
            for j in range(8):  # B -> A
                assert len({ax((t & 7) + 8 * j, 64 * q + (t >> 3)) // 4 for t in lanes}) == 8


def test_store_addresses_are_a_base_plus_constants():
    """The kernel's per-thread bases and compile-time offsets reproduce the layouts."""
    for tl in range(8):
        for a in range(4):
            for x in range(2):
                assert bx(4 * tl + a + 32 * x, 5) == GS * tl + 5 + BP * a + 8 * GS * x
        for line in range(64):
            for j in range(8):
                for q in range(4):
                    pos = ((line & 3) + 2 * ((line >> 4) & 1) + (tl & 1)) & 3
                    base = GS * (tl >> 2) + AP * (tl & 3) + 64 * q + (line & ~3) + pos
                    assert ax(tl + 8 * j, 64 * q + line) == base + 2 * GS * j
            for a in range(4):
                for kB in range(8):
                    base = (line >> 2) * GS + (line & 3) * AP + 4 * tl
                    assert ax(line, 4 * tl + a + 32 * kB) == base + ((a + 2 * (tl >> 2) + (line & 1)) & 3) + 32 * kB
