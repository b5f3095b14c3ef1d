"""The GPU build against the host build at triangle counts where its two phases meet
(256 triangles a warp, 2048 a block), and where a node's triangles cannot be told
apart by their centroids (the middle index splits them, in order)."""
import numpy as np
import pytest

from mambatracer_gb300 import api, scenes

pytestmark = pytest.mark.gpu


def _check(ctx, sc):
    hn, hb, _ = api.bvh_build_host(sc)
    S = api.Scene(ctx, sc)
    dn, db = S.build_bvh_device()
    assert np.array_equal(dn, hn) and np.array_equal(db, hb)
    dev = S.layout()
    S.build_bvh_device(want_arrays=False)
    again = S.layout()
    S.import_bvh(hn, hb)
    host = S.layout()
    for got in (dev, again):
        assert got[2] == host[2] and got[1].tobytes() == host[1].tobytes()
        assert np.array_equal(got[0][:, :12], host[0][:, :12])
        assert got[0][:, 12:].tobytes() == host[0][:, 12:].tobytes()
    S.close()


@pytest.mark.parametrize("n", [255, 256, 257, 511, 513, 2047, 2048, 2049, 4097, 66001])
def test_sizes(ctx, n):
    _check(ctx, scenes.soup(n, seed=n, edge_sigma=0.02))


@pytest.mark.parametrize("copies", [257, 2500])
def test_coinciding_triangles(ctx, copies):
    one = scenes.soup(2, seed=5, edge_sigma=0.4)
    k = np.arange(copies) % 2
    _check(ctx, scenes.Scene(points=one.points, faces=one.faces[k].copy(), materials=one.materials, name="copies"))
