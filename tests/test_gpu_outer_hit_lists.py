"""Lists of the cells that end on a hit, at the lengths where the list sort changes hands: a warp's staging holds
512 entries, and a longer list is sorted by one lane. Lists and neighbours equal the oracle's."""
import numpy as np
import pytest

import built_events as B
from oracle import oracle
from parity import compare_ca, compare_hits

pytestmark = pytest.mark.gpu

C = B.CENTRE


@pytest.mark.parametrize("n", [511, 512, 513, 700])
def test_long_outer_hit_lists(conditions, n):
    from pixeltrack import PixelChain, batch_params, default_params
    rng = np.random.default_rng(n)
    inner = np.array(B.grid(range(C - 20, C + 27, 2), range(0, 280, 2)))
    inner = inner[rng.choice(len(inner), n, replace=False)]
    # the rows from C + 54 on look back at a part of the inner hits only
    outer = [(C, 60), (C + 4, 100), (C + 54, 70), (C + 56, 90), (C + 2, 140), (C + 58, 110)]
    ev = B.event([(B.INNER, r, c) for r, c in inner] + [(B.OUTER, r, c) for r, c in outer])
    orc = oracle.Oracle(conditions)
    orc.run_event(ev, 7)
    lists = np.bincount(orc.get("cells").reshape(-1, 5)[:, 1])
    assert lists.max() == n and ((lists > 0) & (lists < 400)).any()
    blob, offs = B.batch([ev] * 9)
    with PixelChain(conditions, batch_params(9)) as batch, PixelChain(conditions, default_params()) as chain:
        batch.run_batch(blob, offs, stages=7)
        chain.run_event(ev, 7)
        assert batch.sync() == chain.sync() == 0x400  # lists above the reference's 128 rows are flagged
        for c, k in ((batch, 0), (batch, 8), (chain, 0)):
            assert not (compare_hits(c, orc, k) + compare_ca(c, orc, k))
