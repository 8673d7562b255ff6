"""Riemann fits of tracks across the beam (first and last hit at the same z) on the GPU, against the oracle."""
import numpy as np
import pytest

from edge_tracks import B_FIELD, flat_tracks
from oracle import oracle
from test_riemann_flat import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_flat_tracks(precision):
    import torch
    from pixeltrack.fits import riemann_fit
    tracks = flat_tracks()
    offs = np.concatenate([[0], np.cumsum([len(h) for h, _ in tracks])]).astype(np.int32)
    out = riemann_fit(torch.as_tensor(np.concatenate([h for h, _ in tracks])).cuda(),
                      torch.as_tensor(np.concatenate([g for _, g in tracks])).cuda(), torch.as_tensor(offs).cuda(),
                      B_FIELD, precision=precision)
    out = {k: v.cpu().numpy() for k, v in out.items()}
    for t, (hits, ge) in enumerate(tracks):
        o = oracle.riemann_fit(hits, ge, B_FIELD)
        assert out["status"][t] == o["rc"] == 0
        check(out["state"][t], out["chi2"][t], out["pt"][t], o, precision)
