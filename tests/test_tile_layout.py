"""Shared memory of the generic stage tile (bb_stage_tile_bytes, host arithmetic only), byte for
byte: whole lift stacks wherever they fit in 224 KB, in both precisions, else one row per chain and
a volume block; and the degree tables that a tile reads, nothing more."""
import ctypes

import pytest


def np3(n):
    return (n + 1) * (n + 2) * (n + 3) // 6


def np2(n):
    return (n + 1) * (n + 2) // 2


def align16(x):
    return (x + 15) // 16 * 16


def table_words(N):
    """node3, node3m1 (32 bits an entry); node2 of degrees 0..N+1, fvol, fperm (16 bits)."""
    return (np3(N) + np3(N - 1) + (np3(N + 1) + 1) // 2 + (4 * np2(N) + 1) // 2
            + (6 * np2(N) + 1) // 2)


def tile(phys, N, f64, epb):
    nf, nw, nch = {0: (4, 4, 2), 1: (6, 6, 6), 2: (1, 1, 1), 3: (3, 1, 3)}[phys]
    size = 8 if f64 else 4
    per_element = 24 + 8 + 9   # geometry, penalty weights, half weights

    def total(scalars):
        b = align16(scalars * size) + align16(epb * 16) + 4 * table_words(N)
        return align16(b)

    stacks = total(epb * (nf * np3(N) + 4 * nch * np2(N) + nw * np3(N - 1)
                          + 4 * nch * (np3(N) | 1) + per_element)
                   + ((N + 1) * (N + 2) if f64 else 0))
    rows = total(epb * (2 * nf * np3(N) + 4 * nf * np2(N)
                        + max(nw * np3(N - 1), 2 * nch * np2(N + 1)) + per_element))
    return stacks if stacks <= 224 * 1024 else rows


@pytest.mark.parametrize("phys", [0, 1, 2, 3])
def test_bytes_of_every_tile(phys):
    from bbdg import _lib
    lib = _lib.load()
    b, c = ctypes.c_int64(), ctypes.c_int()
    for N in range(1, 21):
        for f64 in (0, 1):
            for epb in (1, 2, 3, 4, 6, 8, 16, 24):
                assert lib.bb_stage_tile_bytes(phys, N, f64, epb, ctypes.byref(b),
                                               ctypes.byref(c)) == 0
                assert b.value == tile(phys, N, f64, epb), (N, f64, epb)
