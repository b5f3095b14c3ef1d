"""The FP64 table of an environment map at sizes around the row and column kernels'
steps (256 columns, 16 rows), against a host sum, with its FP32 copy rounded once, and
maps replaced by maps of the same and of other shapes."""
import numpy as np
import pytest

from mambatracer_gb300 import api, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (31, 15), (33, 16), (256, 17), (257, 33), (64, 1025)])
def test_table_sizes(ctx, w, h):
    S = api.Scene(ctx, scenes.box_room(8, 8))
    for seed, (a, b) in enumerate([(w, h), (w, h), (h, w), (w, h)]):
        rng = np.random.default_rng(seed)
        env = rng.uniform(0.0, 2.0, (a * b, 4)).astype(np.float32)
        S.set_env(env, a, b)
        lum, sat64, sat32 = S.env_arrays(a, b)
        want = np.cumsum(np.cumsum(lum.reshape(b, a).astype(np.float64), axis=1), axis=0).reshape(-1)
        assert np.allclose(sat64, want, rtol=1e-12, atol=0.0)
        assert np.array_equal(sat32, sat64.astype(np.float32))
    S.close()
