"""Clustering at the module sizes where the kernels change hands (a thread, a warp with one digi per lane, a
warp with a column histogram, a block): clusters, charge cut and module records equal the oracle's."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 16, 17, 31, 32, 33), (63, 64, 65, 127, 128, 129), (254, 255, 256, 257, 300)])
@pytest.mark.parametrize("cut", [False, True])
def test_module_sizes(conditions, sizes, cut):
    from pixeltrack import PixelChain, default_params
    rng = np.random.default_rng(sum(sizes))
    ids, xs, ys = [], [], []
    for m, n in enumerate(sizes):
        cells = rng.choice(24 * 40, n, replace=False)  # dense enough for clusters of all shapes
        mod = np.full(n, 40 * m + 7, np.uint16)
        mod[1:][rng.random(n - 1) < 0.05] = 9999  # digis outside the clustering
        ids.append(mod)
        xs.append(cells % 24)
        ys.append(cells // 24 + (0, 376)[m % 2])  # the first and the last columns
    id_, x, y = (np.concatenate(a).astype(np.uint16) for a in (ids, xs, ys))
    adc = rng.integers(200, 3000, len(id_)).astype(np.uint16)
    o = oracle.clusterize_digis(id_, x, y, adc, charge_cut=cut)
    with PixelChain(conditions, default_params()) as chain:
        g = chain.clusterize_digis(id_, x, y, adc, charge_cut=cut)
    nm = int(o["module_start"][0])
    assert nm == len(sizes)
    for name in ("clus_in_module", "clus", "id"):
        assert np.array_equal(g[name], o[name]), name
    assert np.array_equal(g["module_id"][:nm], o["module_id"][:nm])
