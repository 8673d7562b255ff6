"""The duplicate remover's rule on the CPU: the rounds over all cells at once (k_dup_resolve) end in
what the reference's ordered walk over the cells leaves, for overlapping lists, ties and long chains."""
import random

import pytest

NONE = 1 << 32


def ordered_walk(cells, tip, loose):
    """kernel_fast_duplicate_remover: cell by cell, the loose track of smallest |tip| (first on ties) stays."""
    loose = set(loose)
    for tracks in cells:
        best, keep = 10000.0, None
        for t in tracks:
            if t in loose and tip[t] < best:
                best, keep = tip[t], t
        loose -= {t for t in tracks if t != keep}
    return loose


def rounds(cells, tip, loose):
    lists = [(c, [t for t in tracks if t in loose]) for c, tracks in enumerate(cells)]
    lists = [(c, l) for c, l in lists if len(l) > 1]
    random.Random(1).shuffle(lists)  # the cells are taken in any order
    death, n = {t: NONE for t in loose}, 0
    while True:
        new, n = {t: NONE for t in loose}, n + 1
        for c, l in lists:
            ahead = [(tip[t], j) for j, t in enumerate(l) if death[t] >= c]
            if ahead:
                for j, t in enumerate(l):
                    if (tip[t], j) > min(ahead):
                        new[t] = min(new[t], c)
        if new == death:
            return {t for t in loose if death[t] == NONE}, n
        death = new
        assert n <= len(loose) + 1


@pytest.mark.parametrize("tracks,cells,rows,values", [(6, 8, 3, 3), (40, 60, 5, 1000), (60, 200, 8, 6), (200, 150, 64, 50)])
def test_rounds_equal_ordered_walk(tracks, cells, rows, values):
    rng = random.Random(tracks * cells)
    for _ in range(60):
        tip = [rng.randrange(values) / 100 for _ in range(tracks)]
        loose = {t for t in range(tracks) if rng.random() < 0.7}
        lists = [sorted(rng.sample(range(tracks), rng.randint(1, min(rows, tracks)))) for _ in range(cells)]
        assert rounds(lists, tip, loose)[0] == ordered_walk(lists, tip, loose)


def test_longest_chain():
    n = 50  # cell c holds tracks c and c + 1: each track's fate hangs on the one before it
    for order in (range(n), reversed(range(n))):
        lists = [[c, c + 1] for c in order]
        tip = [t / 100 for t in range(n + 1)]
        got, k = rounds(lists, tip, set(range(n + 1)))
        assert got == ordered_walk(lists, tip, set(range(n + 1)))
        assert k <= n + 2
