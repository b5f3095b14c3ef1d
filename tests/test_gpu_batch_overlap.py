"""Merged batches whose passes overlap: the films equal the frames rendered alone, bit
for bit, with fewer, as many and more passes than run at once, frames that end after
different passes, and plain as well as compensated sums."""
import numpy as np
import pytest

from mambatracer_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spps", [[1], [2, 1], [4, 1, 3], [9, 2, 5, 1], [6, 6]])
@pytest.mark.parametrize("kahan", [0, 1])
def test_overlapping_batch_passes(ctx, spps, kahan):
    sc = scenes.textured_room(64, 64)
    S = api.Scene(ctx, sc)
    S.build_bvh_device(want_arrays=False)
    frames = [(sc.camera, 13 + 20 * k, 41 - 9 * k, spp, float(3 + 10 * k)) for k, spp in enumerate(spps)]
    films, rays = api.batch_render(ctx, S, frames, max_depth=5, rr_depth=3, film_kahan=kahan)
    total = np.zeros(3, np.int64)
    for (cam, w, h, spp, fc), film in zip(frames, films):
        J = api.Job(ctx, S, w, h, max_depth=5, mode=1, rr_depth=3, film_kahan=kahan, profile=1)
        J.set_camera(cam)
        for p in range(spp):
            J.render(None, fc + p)
            ctx.finish()
        assert film.tobytes() == J.film().tobytes(), (w, h, spp)
        total += J.total_rays()
        J.close()
    assert np.array_equal(rays, total)
    S.close()
