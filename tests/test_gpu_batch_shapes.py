"""Batches of small events at the sizes where the blocks per event reach their floor: products equal the oracle's, and
those of the same events run on the device's own copy of the input, whose sizes the host does not know."""
import numpy as np
import pytest

from oracle import oracle
from parity import compare_event

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [296, 297, 2369])
def test_small_events(conditions, n):
    import torch
    from pixeltrack import PixelChain, batch_params, gen
    blob, offs = gen.events(n, gen.MODE_SINGLE, ntracks=8, seed=n)
    params = batch_params(n, words_per_event=1600, hits_per_event_avg=300, doublets_per_event_avg=2000,
                          tuples_per_event_avg=400)
    orc = oracle.Oracle(conditions)
    with PixelChain(conditions, params) as chain:
        counts = []
        db, do = torch.as_tensor(blob).cuda(), torch.as_tensor(offs.astype(np.int64)).cuda()
        for run in (lambda: chain.run_batch(blob, offs), lambda: chain.run_batch_device(db.data_ptr(), do.data_ptr(), n)):
            run()
            assert chain.sync() == 0
            for e in (0, n // 2, n - 1):
                orc.run_event(blob[offs[e]:offs[e + 1]], 63)
                assert not compare_event(chain, orc, e), e
            counts.append([chain.counts(e) for e in range(n)])
        assert counts[0] == counts[1]
