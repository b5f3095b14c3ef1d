"""Ray queues too short to fill every warp of the traversal grid are spread over
all of them (one ray to a warp at the shortest): closest and any hits against the
oracle around the sizes where the rays per warp change."""
import numpy as np
import pytest

from mambatracer_gb300 import api, layout, scenes
from tests.helpers import bvh_build, oracle_any, oracle_trace

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def soup(ctx, orc):
    sc = scenes.soup(20000, seed=8, extent=0.8, edge_sigma=0.03)
    nodes, bounds, _, _ = bvh_build(orc, sc)
    S = api.Scene(ctx, sc)
    S.import_bvh(nodes, bounds)
    yield sc, nodes, bounds, S
    S.close()


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 4863, 4865, 9729, 50001])
def test_short_queues(orc, soup, n):
    sc, nodes, bounds, S = soup
    o, d = scenes.random_rays(sc, n, seed=n)
    rays = layout.make_rays(o, d)
    t_ref, p_ref = oracle_trace(orc, sc, nodes, bounds, rays)[:2]
    a_ref = oracle_any(orc, sc, nodes, bounds, rays)
    for precision in (0, 1, 2, 3):
        S.set_precision(precision)
        t, p = S.trace_closest(rays)
        assert np.array_equal(t, t_ref) and np.array_equal(p, p_ref), precision
        assert np.array_equal(S.trace_any(rays) != 0, a_ref != 0), precision
    S.set_precision(0)
