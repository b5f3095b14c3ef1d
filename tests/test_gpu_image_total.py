"""The image's log-luminance total, summed by the block that ends last: sizes of one block, one
pixel more, more partial sums than are summed side by side, twice in a row, and after a clear
(opaque black image, empty totals). The average is the FP64 one of the film's luminances within the
rounding of FP32 logarithms, and the same on every call."""
import numpy as np
import pytest

from mambatracer_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (16, 16), (257, 1), (100, 41), (640, 451), (1031, 600)])
def test_log_average(ctx, w, h):
    sc = scenes.box_room(w, h)
    S = api.Scene(ctx, sc)
    S.build_bvh_device(want_arrays=False)
    J = api.Job(ctx, S, w, h, max_depth=3, mode=1, rr_depth=0)
    J.set_camera(sc.camera)
    for again in range(2):
        J.render(None, 1.0)
        argb, average = J.image()
        film = J.film(resolve=True).astype(np.float64)
        lum = film[:, 0] * 0.2989 + film[:, 1] * 0.5866 + film[:, 2] * 0.1145
        lum = lum[lum > 0]
        want = np.exp(np.mean(np.log(0.01 + lum))) if lum.size else 0.0
        assert abs(average - want) <= 1e-5 * max(want, 1e-30), (average, want)
        same, average2 = J.image()
        assert average2 == average and same.tobytes() == argb.tobytes()
        J.clear()
        black, average = J.image()
        assert average == 0.0 and np.all(black.view(np.uint32) == 0xFF000000)
        assert not J.film().any() and not J.total_rays().any()
    J.close()
    S.close()
