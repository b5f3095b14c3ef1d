"""Resolved film reads divide on the device: equal, bit for bit, to the film divided
by the frame count on the host with w = 1 (averageAccum), through the waiting and
the enqueued read, before the first frame and with several frames in flight."""
import numpy as np
import pytest

from mambatracer_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (37, 19), (300, 200)])
@pytest.mark.parametrize("inflight", [1, 3])
def test_resolved_reads(ctx, w, h, inflight):
    sc = scenes.box_room(w, h)
    S = api.Scene(ctx, sc)
    S.build_bvh_device(want_arrays=False)
    J = api.Job(ctx, S, w, h, max_depth=3, mode=1, rr_depth=3, inflight=inflight)
    J.set_camera(sc.camera)
    assert not J.film(resolve=True).any()  # no frame yet: the film as it is
    ring = [np.empty((w * h, 4), np.float32) for _ in range(4)]
    films = []
    for f in range(4):
        J.render(None, float(f + 1))
        J.film_async(ring[f], resolve=True)
        films.append(J.film())
    J.wait()
    for f, (got, film) in enumerate(zip(ring, films)):
        want = film / np.float32(f + 1)
        want[:, 3] = 1.0
        assert got.tobytes() == want.astype(np.float32).tobytes(), f
    assert J.film(resolve=True).tobytes() == ring[3].tobytes()
    J.close()
    S.close()
