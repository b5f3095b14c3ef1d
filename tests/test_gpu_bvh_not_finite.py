"""The tree builders over meshes with coordinates that are infinite, too large for their
centroids to be finite, or not numbers: they end, and closest distances and any-hit answers
equal the CPU oracle's over the host-built tree, in the formats that hold such boxes.
Triangles of 10^38 overflow in the hit test itself, so their hits depend on the tree:
there the hits are triangles of the mesh. Of the sizes, 300 are built by one warp and
5000 level by level first."""
import numpy as np
import pytest

from mambatracer_gb300 import api, layout, scenes
from tests.helpers import oracle_any, oracle_trace

pytestmark = pytest.mark.gpu

VALUES = {"inf": [np.inf], "both": [np.inf, -np.inf], "huge": [3e38, -3e38], "nan": [np.nan],
          "mixed": [np.nan, np.inf, -np.inf, 3e38, -0.0]}


@pytest.mark.parametrize("share", [0.02, 0.5, 1.0])
@pytest.mark.parametrize("kind", sorted(VALUES))
@pytest.mark.parametrize("n", [3, 300, 5000])
def test_not_finite(ctx, orc, n, kind, share):
    rng = np.random.default_rng(n)
    sc = scenes.soup(n, seed=n, extent=0.8, edge_sigma=0.1)
    o, d = scenes.random_rays(sc, 4000, seed=3)
    rays = layout.make_rays(o, d)
    # a random coordinate of a share of the triangles' vertices, and of a few all of them
    for k, name in enumerate(("vx", "vy", "vz")):
        tri = np.flatnonzero(rng.random(n) < share / (1 + k))
        v = sc.faces[name][tri]
        sc.points[v, rng.integers(0, 3, len(v))] = rng.choice(VALUES[kind], len(v))
    whole = sc.faces["vx"][:: 97], sc.faces["vy"][:: 97], sc.faces["vz"][:: 97]
    for v in whole:
        sc.points[v, :3] = VALUES[kind][0]
    nodes, bounds, _ = api.bvh_build_host(sc)
    t, _ = oracle_trace(orc, sc, nodes, bounds, rays)
    occ = oracle_any(orc, sc, nodes, bounds, rays)
    S = api.Scene(ctx, sc)
    S.build_bvh_device(want_arrays=False)
    for precision in (0, 1, 3):
        S.set_precision(precision)
        got, prim = S.trace_closest(rays)
        anyhit = S.trace_any(rays)
        assert ((prim >= -1) & (prim < n)).all()
        if kind not in ("huge", "mixed"):
            assert np.array_equal(got, t), precision
            assert np.array_equal(anyhit, occ), precision
    if kind == "inf":  # the centroids are numbers: the device's tree is the host's
        dn, db = S.build_bvh_device()
        assert np.array_equal(dn, nodes) and np.array_equal(db, bounds)
    S.close()
