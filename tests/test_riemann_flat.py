"""Riemann fits of tracks across the beam (first and last hit at the same z) on the host build of the kernel's
headers, against the oracle, with the bounds that the device fits are held to."""
import numpy as np
import pytest

import host_fits
from edge_tracks import B_FIELD, flat_tracks
from oracle import oracle


@pytest.mark.parametrize("precision", [0, 1])
def test_flat_tracks(tmp_path_factory, precision):
    lib = host_fits.load(tmp_path_factory.mktemp("host_fits"))
    for hits, ge in flat_tracks():
        f, o = host_fits.fit(lib, "rm", precision, hits, ge, B_FIELD), oracle.riemann_fit(hits, ge, B_FIELD)
        assert f["status"] == o["rc"] == 0
        check(f["state"], f["chi2"], f["pt"], o, precision)


def check(state, chi2, pt, o, precision):
    if precision == 0:
        np.testing.assert_allclose(state, o["state"], rtol=2e-6, atol=1e-7)
        np.testing.assert_allclose(pt, o["pt"], rtol=2e-6)
        np.testing.assert_allclose(chi2, [o["chi2_circle"], o["chi2_line"]], rtol=1e-4, atol=1e-6)
        return
    d = np.abs(np.asarray(state, np.float64) - o["state"])
    assert d[2] < 1e-5 * abs(o["state"][2]) and d[3] < 1e-5 * max(abs(o["state"][3]), 1e-3)
    assert d[0] < 1e-6 and d[1] < 1e-6 and d[4] < 1e-5
