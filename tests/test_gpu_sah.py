"""The surface-area tree under the 4-wide nodes: every triangle stays reachable, so
closest distances and any-hit answers equal those of the FP32 records, at triangle
counts around the builder's sizes (256 triangles a warp, 2048 a block), with
coinciding centroids (no split but the middle), and for triangles of very uneven
size; near ties fall as on the FP32 records' tree order, run after run."""
import numpy as np
import pytest

from mambatracer_gb300 import api, layout, scenes

pytestmark = pytest.mark.gpu


def _check(ctx, sc, nrays=20000, seed=3):
    S = api.Scene(ctx, sc)
    S.build_bvh_device(want_arrays=False)
    o, d = scenes.random_rays(sc, nrays, seed=seed)
    rays = layout.make_rays(o, d)
    t0, p0 = S.trace_closest(rays)
    a0 = S.trace_any(rays)
    S.set_precision(3)
    t3, p3 = S.trace_closest(rays)
    assert np.array_equal(t3, t0) and np.array_equal(p3 >= 0, p0 >= 0)
    assert np.array_equal(S.trace_any(rays), a0)
    t4, p4 = S.trace_closest(rays)
    assert np.array_equal(t4, t3) and np.array_equal(p4, p3)
    S.close()
    return p0, p3


@pytest.mark.parametrize("n", [2, 3, 4, 31, 33, 255, 256, 257, 2047, 2049, 4097, 70001])
def test_sizes(ctx, n):
    p0, p3 = _check(ctx, scenes.soup(n, seed=n, edge_sigma=0.005 * np.sqrt(1e6 / n)))
    assert np.array_equal(p0, p3) and (p0 >= 0).any()


@pytest.mark.parametrize("copies", [2, 300, 5000])
def test_coinciding_triangles(ctx, copies):
    one = scenes.soup(3, seed=5, edge_sigma=0.4)
    k = np.arange(copies) % 3
    sc = scenes.Scene(points=one.points, faces=one.faces[k].copy(), materials=one.materials, name="copies")
    _check(ctx, sc)


def test_uneven_sizes(ctx):
    """The stadium's large ground triangles around a sphere of small ones."""
    _check(ctx, scenes.stadium(quads=60, level=5), nrays=100000)
