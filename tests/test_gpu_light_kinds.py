"""The shading instances for one kind of lighting (mesh lights, a whole map, a map
through the light grid) against the general instance, which the tuning's bounds of 3
blocks per SM select: the same films and ray counts, bit for bit, in both semantics
and at sizes that leave partial warps."""
import numpy as np
import pytest

from mambatracer_gb300 import api, scenes

pytestmark = pytest.mark.gpu


def _render(ctx, S, cam, w, h, mode, inflight):
    J = api.Job(ctx, S, w, h, max_depth=5, mode=mode, rr_depth=3 if mode else 0, film_kahan=mode, inflight=inflight,
                grid_updates=0)
    J.set_camera(cam)
    seeds = np.arange(1, 2 * (1 + 2 * 5) + 1, dtype=np.int32) * 1000003 if mode == 0 else None
    for f in range(3):
        J.render(seeds, float(f + 1))
    film, (rays, counts) = J.film(), J.stats()
    J.close()
    return film, rays, counts


@pytest.mark.parametrize("lights", ["mesh", "mesh+map", "map", "grid", "none"])
@pytest.mark.parametrize("w,h", [(1, 1), (33, 7), (100, 75)])
def test_kinds_equal_the_general_instance(ctx, lights, w, h):
    room = lights.startswith("mesh")
    sc = scenes.box_room(w, h) if room else scenes.soup(20000, seed=8, extent=0.8, edge_sigma=0.02, width=w, height=h)
    S = api.Scene(ctx, sc)
    S.build_bvh_device(want_arrays=False)
    if lights not in ("mesh", "none"):
        S.set_env(scenes.sky_env(256, 128), 256, 128)
    if lights == "grid":
        S.grid_config(320, 320, 16, 32, enable=2)
    before = api.get_tuning()
    try:
        for mode in ((1,) if lights == "grid" else (0, 1)):
            for inflight in (1, 2):
                api.set_tuning(before, shade_minb=4)
                film, rays, counts = _render(ctx, S, sc.camera, w, h, mode, inflight)
                api.set_tuning(before, shade_minb=3)
                gfilm, grays, gcounts = _render(ctx, S, sc.camera, w, h, mode, inflight)
                assert film.tobytes() == gfilm.tobytes()
                assert np.array_equal(rays, grays) and np.array_equal(counts, gcounts)
    finally:
        api.set_tuning(before)
        S.close()
