"""The export of small batches (one kernel writes the pinned host arrays, up to eight events) and of larger
ones and pageable arrays (a copy per array) give the same rows: those of the per-event products."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 8, 9])
@pytest.mark.parametrize("pinned", [True, False])
def test_export_rows(conditions, n, pinned):
    from pixeltrack import PixelChain, TrackExport, batch_params, gen
    from pixeltrack._native import check
    blob, offs = gen.events(n, gen.MODE_PU, pu=17, seed=90 + n)
    with PixelChain(conditions, batch_params(n)) as chain:
        chain.run_batch(blob, offs)
        for room in (40_000, 37):  # all tracks, and a collection that holds the first ones only
            out = TrackExport(n, max_tracks=room, max_vertices=n * 1024, cov=True)
            mine = out.arrays if pinned else {k: t.clone() for k, t in out.arrays.items()}
            for k, t in mine.items():
                t.zero_()
                setattr(out.desc, k, t.data_ptr())
            check(chain._lib.pxl_export_async(chain._h, ctypes.byref(out.desc), None, None), "pxl_export_async")
            chain.sync()
            index = mine["index"].numpy().view(np.uint32).reshape(-1, 4)
            assert index[n, 0] == index[:n, 1].sum() and index[n, 2] == index[:n, 3].sum()
            for e in range(n):
                ft, nt, fv, nv = (int(v) for v in index[e])
                loose = np.nonzero(chain.product("quality", e) == 2)[0]
                assert nt == len(loose) and nv == chain.counts(e).n_vertices
                got = max(0, min(nt, room - ft))
                for name, w in (("state", 5), ("cov", 15), ("pt", 1), ("eta", 1), ("chi2", 1)):
                    want = chain.product(name, e).reshape(-1, w)[loose[:got]]
                    assert np.array_equal(mine[name].numpy()[w * ft:w * (ft + got)].reshape(-1, w), want), (e, name)
                assert np.array_equal(mine["vertex"].numpy()[ft:ft + got], chain.product("idv", e)[loose[:got]])
                assert np.array_equal(mine["tuple"].numpy()[ft:ft + got], loose[:got] + 1)
                off = chain.product("tuple_off", e).astype(np.int64)
                assert np.array_equal(mine["n_hits"].numpy()[ft:ft + got], np.diff(off)[loose[:got]])
                for name in ("zv", "wv", "vchi2", "ptv2", "ndof"):
                    assert np.array_equal(mine[name].numpy()[fv:fv + nv], chain.product(name, e)[:nv]), (e, name)
