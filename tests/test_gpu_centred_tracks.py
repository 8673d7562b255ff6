"""Broken-line fits of hits on a circle about the beam line on the GPU: the impact parameter is the radius."""
import numpy as np
import pytest

from edge_tracks import B_FIELD, centred_tracks
from test_centred_tracks import D0_ATOL

pytestmark = pytest.mark.gpu


def test_centred_tracks():
    import torch
    from pixeltrack.fits import bl_fit
    tracks = centred_tracks()
    offs = np.concatenate([[0], np.cumsum([len(t[0]) for t in tracks])]).astype(np.int32)
    out = bl_fit(torch.as_tensor(np.concatenate([t[0] for t in tracks])).cuda(),
                 torch.as_tensor(np.concatenate([t[1] for t in tracks])).cuda(), torch.as_tensor(offs).cuda(), B_FIELD)
    assert (out["status"] == 0).all()
    d0 = out["state"][:, 1].abs().cpu().numpy().astype(np.float64)
    assert np.abs(d0 - [t[2] for t in tracks]).max() < D0_ATOL
