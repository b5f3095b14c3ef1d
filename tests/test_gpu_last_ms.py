"""mt_job_last_ms covers a frame until it is in the film: a frame whose own passes are short,
submitted right after long ones that run beside it, is in the film only after those."""
import numpy as np
import pytest

from mambatracer_gb300 import api, layout, scenes

pytestmark = pytest.mark.gpu


def test_last_ms_ends_with_the_film(ctx):
    w, h = 1280, 960
    sc = scenes.soup(200_000, seed=4, width=w, height=h, edge_sigma=0.011)
    S = api.Scene(ctx, sc)
    S.build_bvh_device(want_arrays=False)
    away = layout.make_camera((0.0, 0.0, 9.0), (0.0, 0.0, 19.0), (0.0, 1.0, 0.0), 40.0, w, h)  # sees nothing
    J = api.Job(ctx, S, w, h, max_depth=8, mode=1, rr_depth=0)

    def frames(*cams):
        """last_ms of the last frame, and the device time of them all."""
        ctx.record(0)
        for k, cam in enumerate(cams):
            J.set_camera(cam)
            J.render(None, 1.0 + k)
        ctx.record(1)
        ctx.finish()
        return J.last_ms(), ctx.elapsed_ms(0, 1)

    frames(sc.camera, away, sc.camera, away)  # the graphs of the slots, of frames alone and among others
    frames(*[sc.camera] * 4)
    alone, empty = frames(sc.camera)[0], frames(away)[0]
    assert empty < 0.3 * alone
    # The short frame is the last in the film, and all four start when they are submitted, a
    # small part of a long frame's time after the first: its span is nearly the whole.
    runs = [frames(sc.camera, sc.camera, sc.camera, away) for _ in range(5)]
    span, whole = (float(np.median(v)) for v in zip(*runs))
    assert 0.85 * whole < span <= whole
    J.close()
    S.close()
