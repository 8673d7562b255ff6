"""Fits of collinear hits on the host build of the kernels' headers: refused, as the oracle refuses them."""
import numpy as np
import pytest

import host_fits
from edge_tracks import B_FIELD, straight_tracks
from oracle import oracle


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("which", ["bl", "rm"])
def test_straight_tracks(tmp_path_factory, which, precision):
    lib = host_fits.load(tmp_path_factory.mktemp("host_fits"))
    for hits, ge in straight_tracks():
        o = oracle.bl_fit(hits.T, ge.T, B_FIELD) if which == "bl" else oracle.riemann_fit(hits, ge, B_FIELD)
        f = host_fits.fit(lib, which, precision, hits, ge, B_FIELD)
        assert o["rc"] != 0 and f["status"] == 1 and np.isnan(f["state"][:3]).all()
