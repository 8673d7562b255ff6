"""Qualities after the duplicate removers where the fast remover's rarer paths run: cells with more than four loose
tracks, and equal impact parameters among them, in one event (a cell per thread) and in a batch (a word of cells)."""
import numpy as np
import pytest

from oracle import oracle
from parity import compare_quality

pytestmark = pytest.mark.gpu

E = 9
CHI2_COEFF = np.float32([0.68177776, 0.74609577, -0.08035491, 0.00315399])


def crowded_cells(orc):
    """Cells with more than four loose tracks after the fits, and those of them with equal |tip|."""
    nt, nc = orc.counts()["n_tuples"], orc.counts()["n_cells"]
    quality, pt, chi2 = orc.get("quality")[:nt], orc.get("pt")[:nt], orc.get("chi2")[:nt]
    state, n = orc.get("state").reshape(-1, 5)[:nt], np.diff(orc.get("tuple_off").astype(np.int64))[:nt]
    p, c = np.minimum(pt, np.float32(10)), CHI2_COEFF
    quad = n > 3
    loose = ((quality != 1) & (n >= 3) & np.isfinite(state).all(1) & (np.abs(state[:, 4]) < 12)
             & (3 * chi2 < 30 * (c[0] + p * (c[1] + p * (c[2] + p * c[3]))))
             & (np.abs(state[:, 1]) < np.where(quad, 0.5, 0.3)) & (pt > np.where(quad, 0.3, 0.5)))
    lists = orc.get("cell_tracks")
    off, tracks = lists[:nc + 1].astype(np.int64), lists[nc + 1:].astype(np.int64) - 1
    crowded = ties = 0
    for k in np.flatnonzero(np.diff(off) > 4):
        t = tracks[off[k]:off[k + 1]]
        tip = np.abs(state[t[loose[t]], 1])
        crowded += len(tip) > 4
        ties += len(tip) > 4 and len(np.unique(tip)) < len(tip)
    return crowded, ties


def test_crowded_cells(conditions):
    from pixeltrack import PixelChain, batch_params, default_params, gen
    blob, offs = gen.events(E, gen.MODE_PU, pu=100, seed=31)
    orc, found = oracle.Oracle(conditions), np.zeros(2, int)
    params = batch_params(E, words_per_event=100_000, hits_per_event_avg=24_000, doublets_per_event_avg=400_000,
                          tuples_per_event_avg=32_000)
    with PixelChain(conditions, params) as batch, PixelChain(conditions, default_params()) as chain:
        batch.run_batch(blob, offs)
        assert batch.sync() == 0
        for e in range(E):
            event = blob[offs[e]:offs[e + 1]]
            orc.run_event(event, 15)
            found += crowded_cells(orc)
            orc.run_event(event, 63)
            assert not compare_quality(batch, orc, e), e
            if e < 3:
                chain.run_event(event)
                assert not compare_quality(chain, orc, 0), e
    assert found[0] >= 20 and found[1] >= 1, found
