"""Broken-line fits of hits on a circle about the beam line on the host build of the kernel's headers: the impact
parameter is the radius, as the oracle finds it where its own root does not round below 0 (the direction is any)."""
import numpy as np

import host_fits
from edge_tracks import B_FIELD, centred_tracks
from oracle import oracle

# 1 + rho A is all rounding there: its root is known to sqrt(2^-53) = 1e-8, the impact parameter to 1e-7 cm, which is
# less than half the spacing of FP32 numbers at 10 cm (5e-7)
D0_ATOL = 6e-7


def test_centred_tracks(tmp_path_factory):
    lib = host_fits.load(tmp_path_factory.mktemp("host_fits"))
    for hits, ge, r in centred_tracks():
        o, f = oracle.bl_fit(hits.T, ge.T, B_FIELD), host_fits.fit(lib, "bl", 0, hits, ge, B_FIELD)
        assert f["status"] == 0 and abs(abs(f["state"][1]) - r) < D0_ATOL
        if o["rc"] == 0 and np.isfinite(o["state"][1]):
            np.testing.assert_allclose(f["state"][1:3], o["state"][1:3], rtol=2e-6, atol=1e-6)
