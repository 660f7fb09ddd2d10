"""The window list of a layered job never outgrows its arena (CPU restatement of the cutting rule).

A window of the list ends after a whole z bin, chosen by how full it leaves the last round of tiles,
or inside a bin larger than the window's span. The list's arena holds 3 * (n / window deposits) + 8
entries (window_cap in st_device.cuh); the restatement cuts bins of every kind that the rule treats
differently, random ones and ones whose bins make the rule prefer short windows, and counts.
"""
import numpy as np
import pytest

TILE, WARPS = 128, 32


def cut(sizes, m, win_tiles):
    """Windows of a job whose z bins hold `sizes` deposits, with m deposits per occupied cell."""
    ends = np.cumsum(sizes)
    kept, k0, n, b = int(ends[-1]), 0, 0, 0
    tiles = (1 if m < 2 else 2 if m < 4 else min(m, 8)) * win_tiles
    covered = []
    while k0 < kept:
        n += 1
        limit = (k0 // TILE + tiles) * TILE
        last = int(np.searchsorted(ends, limit, side="right"))
        e = ends[b:last]
        e = e[e > k0]
        if len(e):
            t = (e + TILE - 1) // TILE - k0 // TILE
            rounds = (t + WARPS - 1) // WARPS
            score = t if m < 4 else ((t * 4096 // (4 * rounds + 3)) << 12) | (t & 0xFFF)
            w = int(np.flatnonzero(score == score.max())[-1])
            end = int(e[w])
            b = int(np.searchsorted(ends, end, side="right"))
        else:
            end = limit
        covered.append((k0, end))
        k0 = end
    assert covered[0][0] == 0 and covered[-1][1] >= kept
    assert all(a[1] == c[0] and a[1] > a[0] for a, c in zip(covered, covered[1:]))
    return n


@pytest.mark.parametrize("win_tiles", [WARPS, 2 * WARPS])
@pytest.mark.parametrize("m", [1, 3, 4, 5, 8, 100])
def test_window_list_fits_its_arena(win_tiles, m):
    rng = np.random.default_rng(win_tiles * 1000 + m)
    span = win_tiles * TILE
    lists = [np.full(4096, s) for s in (1, 5, 127, 128, 129, 1000)]
    # bins just over a round of tiles, just over a window, and small ones in front of large ones
    for a in (1, 21, 22, 31, 32, 33, win_tiles):
        for big in (12, 34, 64, win_tiles + 1, 4 * win_tiles, 8 * win_tiles + 1):
            lists.append(np.tile([a * TILE, big * TILE], 40))
            lists.append(np.tile([a * TILE + 1, big * TILE - 1, 3], 40))
    for _ in range(40):
        lists.append(rng.integers(0, 2 ** rng.integers(1, 18), size=rng.integers(1, 600)))
        lists.append((rng.pareto(0.8, size=300) * 200).astype(np.int64) % 300_000)
    for sizes in lists:
        n = int(sizes.sum())
        if n == 0:
            continue
        assert cut(sizes, m, win_tiles) + 1 <= 3 * (n // span) + 8
