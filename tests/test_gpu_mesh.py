"""Mesh arrays checked and mesh lights listed on the device: the first bad face is the
one reported, whatever else is wrong after it, and the light count and a lit frame
follow the materials, for face counts around a block's 256."""
import numpy as np
import pytest

from mambatracer_gb300 import api, scenes
from mambatracer_gb300._lib import MTError

pytestmark = pytest.mark.gpu


def _mesh(n, seed=1):
    sc = scenes.soup(n, seed=seed, edge_sigma=0.05)
    sc.uvs = np.zeros((5, 2), np.float32)
    sc.normals = np.zeros((7, 4), np.float32)
    return sc


@pytest.mark.parametrize("n", [1, 255, 256, 257, 40001])
def test_first_bad_face_is_reported(ctx, n):
    at = sorted({0, n // 2, n - 1})
    wrong = {"vy": (3 * n, "vertex"), "vx": (-1, "vertex"), "mat": (0xFFFF, "material"), "uvx": (5, "uv"),
             "nx": (7, "normal")}
    for field, (value, word) in wrong.items():
        for i in at:
            sc = _mesh(n)
            sc.faces[field][i] = value
            sc.faces["vz"][i + 1:] = -3
            with pytest.raises(MTError, match=f"face {i}: {word}"):
                api.Scene(ctx, sc)
    sc = _mesh(n)
    sc.faces["uvx"][0], sc.faces["uvy"][0], sc.faces["uvz"][0] = 0, 4, -1
    with pytest.raises(MTError, match="face 0: uv"):
        api.Scene(ctx, sc)


@pytest.mark.parametrize("n", [1, 256, 257, 70000])
@pytest.mark.parametrize("every", [1, 3, 1000])
def test_light_list(ctx, n, every):
    sc = _mesh(n)
    glow = np.zeros(2, sc.materials.dtype)
    glow[:] = sc.materials[:2]
    glow["emission_color"][1] = (1.0, 1.0, 1.0, 1.0)
    glow["emission_param"][1] = (1.0, 5.0, 0.0, 0.0)
    lit = (np.arange(n) % every == every - 1).astype(np.int32)
    sc.faces["mat"] = lit
    sc.materials = glow
    S = api.Scene(ctx, sc)
    assert S.light_count == lit.sum()
    S.close()


def test_material_table_too_small(ctx):
    from mambatracer_gb300._lib import check, lib
    import ctypes as C
    sc = _mesh(300)
    sc.faces["mat"] = 0
    sc.faces["mat"][299] = 40
    S = api.Scene(ctx, sc)
    m = np.ascontiguousarray(sc.materials[:40])
    with pytest.raises(MTError, match="face 299 needs material 40"):
        check(lib().mt_scene_set_materials(S.h, m.ctypes.data_as(C.c_void_p), 40))
    check(lib().mt_scene_set_materials(S.h, np.ascontiguousarray(sc.materials[:41]).ctypes.data_as(C.c_void_p), 41))
    S.close()
