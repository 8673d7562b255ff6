"""Fits of collinear hits on the host build of the kernels' headers: refused, as the oracle refuses them."""
import numpy as np
import pytest

import host_fits
from edge_tracks import B_FIELD, rounded_straight_tracks, straight_tracks
from oracle import oracle


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("which", ["bl", "rm"])
def test_straight_tracks(tmp_path_factory, which, precision):
    lib = host_fits.load(tmp_path_factory.mktemp("host_fits"))
    for hits, ge in straight_tracks():
        o = oracle.bl_fit(hits.T, ge.T, B_FIELD) if which == "bl" else oracle.riemann_fit(hits, ge, B_FIELD)
        f = host_fits.fit(lib, which, precision, hits, ge, B_FIELD)
        assert o["rc"] != 0 and f["status"] == 1 and np.isnan(f["state"][:3]).all()


def test_rounded_straight_tracks(tmp_path_factory):
    """Nearly all that the oracle's Riemann fit refuses are refused; which of the rest are is decided by the order of
    the roundings (without the rounding of each product, half of them were fitted, with a chi2 of 1e5)."""
    lib = host_fits.load(tmp_path_factory.mktemp("host_fits"))
    refused = [t for t in rounded_straight_tracks() if oracle.riemann_fit(*t, B_FIELD)["rc"]]
    assert len(refused) > 200
    assert np.mean([host_fits.fit(lib, "rm", 0, *t, B_FIELD)["status"] for t in refused]) > 0.8
