"""The vertex finder's three forms against the oracle: one wide CTA per event for small batches,
the narrow form with the wide one behind it for the events above 2048 selected tracks, and global
memory above the wide form's tracks. Integer products and ordered FP32 sums are compared exactly."""
import numpy as np
import pytest

from oracle import oracle
from parity import compare_event, compare_vertices

pytestmark = pytest.mark.gpu


def test_large_batch_takes_both_forms(conditions):
    from pixeltrack import PixelChain, batch_params, gen
    small, so = gen.events(149, gen.MODE_UNIFORM, pu=3, seed=31)
    large, lo = gen.events(1, gen.MODE_PU, pu=130, seed=32)
    blob = np.concatenate([small, large])
    offs = np.concatenate([so, [so[-1] + lo[1]]]).astype(np.uint64)
    n = len(offs) - 1
    orc = oracle.Oracle(conditions, oracle.EXTENDED_CAPS)
    params = batch_params(n, words_per_event=20_000, hits_per_event_avg=8_000, doublets_per_event_avg=60_000,
                          tuples_per_event_avg=6_000, extended=True)
    with PixelChain(conditions, params) as chain:
        assert chain.run_batch(blob, offs) == 0
        assert chain.counts(n - 1).n_vertices > 0
        for e in list(range(0, n, 12)) + [n - 1]:
            orc.run_event(blob[offs[e]:offs[e + 1]], 63)
            errs = compare_vertices(chain, orc, e)
            assert not errs, (e, errs)
    assert orc.counts()["n_vtx_tracks"] > 2048


def test_event_above_shared_memory(conditions):
    from pixeltrack import PixelChain, extended_params, gen
    blob, offs = gen.events(1, gen.MODE_PU, pu=480, seed=5)
    big = dict(oracle.EXTENDED_CAPS, tuples=1 << 20, fits_per_mult=1 << 20)
    orc = oracle.Oracle(conditions, big)
    orc.run_event(blob, 63)
    assert orc.counts()["n_vtx_tracks"] > 12288 and orc.counts()["flags"] == 0
    params = extended_params(max_words=400_000, max_hits=80_000, max_doublets=4_194_304, max_tuples=1 << 20,
                             tuples_per_event=1 << 20, fits_per_multiplicity=1 << 20)
    with PixelChain(conditions, params) as chain:
        assert chain.run_event(blob) & ~0x400 == 0  # hits with more than 128 cells: both cut the list
        errs = compare_event(chain, orc, 0)
        assert not errs, errs
