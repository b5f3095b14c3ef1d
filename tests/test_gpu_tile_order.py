"""Camera rays in tiles: at sizes around a tile's (smaller, equal, ragged to the right and at the
bottom) every pixel is rendered by its own path, as the oracle renders it. The preview's
groups are the oracle's; the film is within the tolerance of the other frame tests
(transcendental functions round differently on the two sides)."""
import numpy as np
import pytest

from mambatracer_gb300 import api, scenes
from tests.helpers import bvh_build, oracle_frames, ptr, rel_rmse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (3, 20), (20, 3), (4, 8), (4, 7), (5, 8), (7, 9), (8, 16), (33, 31), (61, 47)])
def test_every_pixel_once(ctx, orc, w, h):
    sc = scenes.box_room(w, h)
    nodes, bounds, _, _ = bvh_build(orc, sc)
    S = api.Scene(ctx, sc)
    S.import_bvh(nodes, bounds)
    argb, group = S.preview(sc.camera, w, h)
    ra, rg, none = np.zeros(w * h, np.int32), np.zeros(w * h, np.int32), np.zeros((1, 4), np.float32)
    orc.lib.or_preview(ptr(sc.camera), w, h, ptr(sc.points), ptr(sc.uvs), ptr(sc.normals), ptr(sc.faces), sc.ntri,
                       ptr(sc.materials), ptr(nodes), ptr(bounds), ptr(none), 1, 1, 0, ptr(ra), ptr(rg))
    assert group.tobytes() == rg.tobytes()
    assert np.abs(argb.view(np.uint8).astype(np.int32) - ra.view(np.uint8).astype(np.int32)).max() <= 1
    J = api.Job(ctx, S, w, h, max_depth=3, mode=1, rr_depth=0)
    J.set_camera(sc.camera)
    J.render(None, 1.0)
    acc, counts, rays = oracle_frames(orc, sc, nodes, bounds, w, h, 3, 1, 0, [None])
    assert np.array_equal(J.stats()[0], rays)
    assert rel_rmse(J.film(), acc) < 1e-5
    J.close()
    films, _ = api.batch_render(ctx, S, [(sc.camera, w, h, 1, 1.0), (sc.camera, h, w, 1, 1.0)], max_depth=3,
                                rr_depth=0)
    assert rel_rmse(films[0], acc) < 1e-5
    S.close()
