"""Every instance of the shading kernels against the general one (MT_LIGHT_KINDS=0) in the same
number of launches, and two launches against one (MT_SHADE_SPLIT): the same films, ray
counts and queue lengths, bit for bit, in both semantics, with and without textures,
for frames and merged batches, at sizes that leave partial warps. The switches are read
once per process, so each pair of them has its own."""
import os
import subprocess
import sys

import numpy as np
import pytest

from mambatracer_gb300 import api, scenes

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIGHTS = ("mesh", "textured", "mesh+map", "textured+map", "map", "grid", "none")
SIZES = ((1, 1), (33, 7), (100, 75))


def _scene(ctx, lights, w, h):
    kind = lights.split("+")[0]
    sc = (scenes.box_room(w, h) if kind == "mesh" else scenes.textured_room(w, h) if kind == "textured" else
          scenes.soup(20000, seed=8, extent=0.8, edge_sigma=0.02, width=w, height=h))
    S = api.Scene(ctx, sc)
    S.build_bvh_device(want_arrays=False)
    if lights not in ("mesh", "textured", "none"):
        S.set_env(scenes.sky_env(256, 128), 256, 128)
    if lights == "grid":
        S.grid_config(320, 320, 16, 32, enable=2)
    return sc, S


def render(out):
    ctx, got = api.Context(0), {}
    for lights in LIGHTS:
        for w, h in SIZES:
            sc, S = _scene(ctx, lights, w, h)
            for mode, inflight in ((0, 1), (1, 1), (1, 2)):
                if mode == 0 and lights == "grid":
                    continue
                J = api.Job(ctx, S, w, h, max_depth=5, mode=mode, rr_depth=3 if mode else 0, film_kahan=mode,
                            inflight=inflight, grid_updates=0)
                J.set_camera(sc.camera)
                seeds = np.arange(1, 2 * (1 + 2 * 5) + 1, dtype=np.int32) * 1000003 if mode == 0 else None
                for f in range(3):
                    J.render(seeds, float(f + 1))
                key = f"{lights} {w}x{h} mode{mode} inflight{inflight}"
                got[key + " film"] = J.film()
                got[key + " rays"], got[key + " counts"] = J.stats()
                J.close()
            frames = [(sc.camera, w, h, 2, 1.0), (sc.camera, h, w, 3, 9.0)]
            films, rays = api.batch_render(ctx, S, frames, max_depth=5, rr_depth=3)
            key = f"{lights} {w}x{h} batch"
            got[key + " rays"] = rays
            for k, film in enumerate(films):
                got[f"{key} film{k}"] = film
            S.close()
    np.savez(out, **got)


def test_instances(tmp_path):
    got = {}
    for kinds in "01":
        for split in "01":
            out = str(tmp_path / f"k{kinds}s{split}.npz")
            code = f"import sys; sys.path.insert(0, {ROOT!r}); import tests.test_gpu_shade_instances as m; m.render({out!r})"
            r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=600,
                               env=dict(os.environ, MT_LIGHT_KINDS=kinds, MT_SHADE_SPLIT=split))
            assert r.returncode == 0, r.stderr[-2000:]
            got[kinds, split] = dict(np.load(out))
    want = got["0", "0"]
    assert sum(bool(v[:, :3].any()) for k, v in want.items() if "film" in k) > 0.7 * sum("film" in k for k in want)
    for pair, g in got.items():
        assert g.keys() == want.keys()
        for k in want:
            assert g[k].tobytes() == want[k].tobytes(), (pair, k)
