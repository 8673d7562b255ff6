"""Doublets of built hits at the counts where a 32-item group of the doublet count changes hands: one inner hit with
about as many doublets as the group's staging holds, and others behind it; cells equal the oracle's one by one."""
import numpy as np
import pytest

import built_events as B
from oracle import oracle
from parity import compare_ca, compare_digis_clusters, compare_hits

pytestmark = pytest.mark.gpu

INNER, OUTER, C = B.INNER, B.OUTER, B.CENTRE
COLS = range(0, 416, 2)


def event(doublets, cut, before, rng):
    """An inner hit with `doublets` outer hits and `cut` more in its phi window that the pt cut takes, three inner
    hits that share some of them, and `before` inner hits elsewhere in front of it."""
    outer = np.array(B.grid(range(C - 56, C + 41, 2), COLS))
    outer = outer[rng.choice(len(outer), doublets, replace=False)]
    edge = np.array(B.grid((C - 62, C - 60), COLS))
    edge = edge[rng.choice(len(edge), cut, replace=False)]
    outer = np.concatenate([outer, edge])[rng.permutation(doublets + cut)]
    far = B.grid(range(2, 158, 2), range(0, 416, 2))[:before]
    px = [(B.module(2, 0, 4), r, c) for r, c in far]
    px += [(INNER, r, c) for r, c in ((C, 100), (C + 30, 104), (C + 22, 60), (C + 14, 140))]
    return B.event(px + [(OUTER, r, c) for r, c in outer])


@pytest.mark.parametrize("before", [0, 20, 224])
def test_items_near_the_staging_size(conditions, before):
    from pixeltrack import PixelChain, batch_params, default_params
    rng = np.random.default_rng(before)
    sizes = [(700, 20), (736, 31), (737, 31), (750, 20), (767, 20), (768, 0), (768, 20), (769, 7), (800, 20), (20, 3)]
    events = [event(n, cut, before, rng) for n, cut in sizes]
    orc = oracle.Oracle(conditions)
    blob, offs = B.batch(events)
    with PixelChain(conditions, batch_params(len(events))) as batch, PixelChain(conditions, default_params()) as chain:
        batch.run_batch(blob, offs, stages=7)
        assert batch.sync() == 0
        for e, (n, _) in enumerate(sizes):
            orc.run_event(events[e], 7)
            inner = np.bincount(orc.get("cells").reshape(-1, 5)[:, 0], minlength=before + 5)
            assert inner[before + 1] == n and (n < 700 or (inner[before + 2:before + 5] > 30).all())
            chain.run_event(events[e], 7)
            for c, k in ((batch, e), (chain, 0)):
                errs = compare_digis_clusters(c, orc, k) + compare_hits(c, orc, k) + compare_ca(c, orc, k)
                assert not errs, (sizes[e], before, errs)
