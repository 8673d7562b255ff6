"""Fits of collinear hits on the GPU: refused, as the oracle refuses them."""
import numpy as np
import pytest

from edge_tracks import B_FIELD, rounded_straight_tracks, straight_tracks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("which", ["bl", "rm"])
def test_straight_tracks(which, precision):
    import torch
    from pixeltrack import fits
    tracks = straight_tracks()
    offs = np.concatenate([[0], np.cumsum([len(h) for h, _ in tracks])]).astype(np.int32)
    fit = fits.bl_fit if which == "bl" else fits.riemann_fit
    out = fit(torch.as_tensor(np.concatenate([h for h, _ in tracks])).cuda(),
              torch.as_tensor(np.concatenate([g for _, g in tracks])).cuda(), torch.as_tensor(offs).cuda(), B_FIELD,
              precision=precision)
    assert (out["status"] == 1).all() and torch.isnan(out["state"][:, :3]).all()


def test_rounded_straight_tracks():
    """Nearly all that the oracle's Riemann fit refuses are refused; rounding decides about the rest."""
    import torch
    from oracle import oracle
    from pixeltrack.fits import riemann_fit
    tracks = [t for t in rounded_straight_tracks() if oracle.riemann_fit(*t, B_FIELD)["rc"]]
    offs = np.concatenate([[0], np.cumsum([len(h) for h, _ in tracks])]).astype(np.int32)
    out = riemann_fit(torch.as_tensor(np.concatenate([h for h, _ in tracks])).cuda(),
                      torch.as_tensor(np.concatenate([g for _, g in tracks])).cuda(), torch.as_tensor(offs).cuda(), B_FIELD)
    assert out["status"].float().mean() > 0.8
