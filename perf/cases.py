"""What a program that uses the library has it do, case by case.

A case names one call pattern and its sizes:

  frame    a progressive render: the film is cleared (as after a camera move), `frames` frames of
           `spp` passes are rendered, and the displayed image or the resolved film is read
  preview  one frame of the preview device
  query    closest and any hits of host rays in the reference's layout
  load     a new mesh and environment up to their first preview: arrays uploaded, BVH and
           environment tables built
  batch    frames of uneven size of one scene in one call
  served   requests of two scenes submitted to a render server and waited for

Scenes are the generators of mambatracer_gb300.scenes, seeded by the case's seed. The light grid of a
case that samples through it stays as it is set up from the map (no updates): the updates add with
float atomics, whose order no two runs share.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from mambatracer_gb300 import api, layout, scenes
from mambatracer_gb300._lib import check, lib


def _stadium(quads, level):
    """The stadium's ground plane and sphere, and the triangles the two come to."""
    return dict(quads=quads, level=level, tri=2 * quads * quads + 20 * 4 ** level)


def listed():
    return [
        # an editor's viewport while the camera is dragged: one pass of a small room, shown at once
        dict(name="room_256_drag", kind="frame", scene="room", tri=36, width=256, height=256, depth=4, mode=1,
             rr=3, spp=1, frames=1, prec=0, env=0, grid=0, inflight=1, read="image"),
        # the reference's own set-up (500 x 500, 15 bounces, its seeds and plain film), a few frames shown
        dict(name="room_500_reference", kind="frame", scene="room", tri=36, width=500, height=500, depth=15, mode=0,
             rr=0, spp=1, frames=4, prec=0, env=0, grid=0, inflight=1, read="image"),
        # a textured room at an odd size, eight passes in one call, the film read
        dict(name="textured_641x359", kind="frame", scene="textured", tri=36, width=641, height=359, depth=6, mode=1,
             rr=3, spp=8, frames=1, prec=0, env=0, grid=0, inflight=1, read="film"),
        # the headline benchmark's frame: 1M triangles under the sky, grid-guided light, frames in flight
        dict(name="soup_1m_1080p", kind="frame", scene="soup", tri=1_000_000, width=1920, height=1080, depth=8,
             mode=1, rr=3, spp=1, frames=8, prec=3, env=2048, grid=2, inflight=6, read="async"),
        # an ordinary still with the default records (FP32), full-map light, one frame at a time
        dict(name="soup_200k_800x600", kind="frame", scene="soup", tri=200_000, width=800, height=600, depth=8,
             mode=1, rr=3, spp=4, frames=1, prec=0, env=1024, grid=0, inflight=1, read="film"),
        # a small object on a very large ground plane, 4 passes a frame
        dict(name="stadium_1080p", kind="frame", scene="stadium", **_stadium(400, 7), width=1920, height=1080,
             depth=8, mode=1, rr=3, spp=4, frames=1, prec=3, env=2048, grid=0, inflight=2, read="film"),
        # the preview device at the size of a laptop's window
        dict(name="preview_1280x720", kind="preview", scene="soup", tri=300_000, width=1280, height=720, prec=0,
             env=1024),
        # picking and probing: a few thousand rays from the host
        dict(name="query_4096", kind="query", scene="soup", tri=20_000, rays=4096, prec=0),
        # a baking tool's ray set
        dict(name="query_1m", kind="query", scene="soup", tri=1_000_000, rays=1_000_003, prec=1),
        # opening a file: mesh and sky to the first preview
        dict(name="load_500k", kind="load", scene="soup", tri=500_000, width=960, height=540, prec=0, env=2048),
        # thumbnails and a camera sweep of one scene, known at once
        dict(name="batch_24", kind="batch", scene="stadium", **_stadium(200, 5), frames=24, lo=64, hi=640, spp=4,
             depth=8, rr=3, prec=3, env=512),
        # a render service: 16 requests of two scenes
        dict(name="served_16", kind="served", scene="soup", tri=100_000, frames=16, lo=48, hi=400, spp=4, depth=8,
             rr=3, prec=3, env=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _scene_of(rng, hi):
    if rng.random() < 0.65:
        return dict(scene="soup", tri=_log(rng, 5_000, hi))
    return dict(scene="stadium", **_stadium(rng.randint(40, 300), rng.choice((4, 5, 6))))


def draw(rng):
    kind = rng.choice(("room", "room", "frame", "frame", "preview", "query", "load", "batch", "served"))
    if kind == "room":
        ref = rng.random() < 0.4
        w = _log(rng, 40, 900)
        return dict(kind="frame", scene=rng.choice(("room", "textured")), tri=36, width=w,
                    height=max(24, int(w * rng.uniform(0.4, 1.1))), depth=15 if ref else rng.randint(2, 8),
                    mode=0 if ref else 1, rr=0 if ref else 3, spp=1 if ref else rng.choice((1, 1, 2, 4)),
                    frames=rng.randint(1, 4), prec=0, env=0, grid=0, inflight=1, read=rng.choice(("image", "film")))
    prec = rng.choice((0, 1, 3, 3))
    if kind == "frame":
        sc = _scene_of(rng, 1_000_000)
        w = _log(rng, 200, 1920)
        grid = rng.choice((0, 1, 2))
        return dict(kind=kind, **sc, width=w, height=int(w * rng.uniform(0.4, 0.56)),
                    depth=rng.randint(3, 8), mode=1, rr=3, spp=rng.choice((1, 1, 2)), frames=rng.randint(1, 2),
                    prec=prec, env=rng.choice((512, 1024, 2048)), grid=grid, inflight=rng.choice((1, 2, 6)),
                    read=rng.choice(("image", "film", "async")))
    if kind == "preview":
        sc = _scene_of(rng, 1_000_000)
        w = _log(rng, 100, 1920)
        return dict(kind=kind, **sc, width=w, height=int(w * rng.uniform(0.5, 1.0)), prec=prec,
                    env=rng.choice((0, 512, 1024)))
    if kind == "query":
        sc = _scene_of(rng, 1_000_000)
        return dict(kind=kind, **sc, rays=_log(rng, 1, 1_000_000), prec=prec)
    if kind == "load":
        sc = _scene_of(rng, 800_000)
        w = _log(rng, 200, 1280)
        return dict(kind=kind, **sc, width=w, height=int(w * rng.uniform(0.5, 0.75)), prec=prec,
                    env=rng.choice((512, 1024, 2048)))
    sc = _scene_of(rng, 300_000)
    return dict(kind=kind, **sc, frames=rng.randint(2, 24), lo=rng.randint(32, 64),
                hi=_log(rng, 100, 640 if kind == "batch" else 400), spp=rng.choice((1, 2, 4)), depth=rng.randint(3, 8),
                rr=3, prec=prec, env=512)


# ------------------------------------------------------------------ states


def _make_scene(case, rng, width=64, height=64):
    kind, tri = case["scene"], case["tri"]
    if kind in ("room", "textured"):
        sc = scenes.box_room(width, height) if kind == "room" else scenes.textured_room(width, height)
        eye = (0.5 + rng.uniform(-0.2, 0.2), 0.5 + rng.uniform(-0.2, 0.2), 2.2 + rng.uniform(-0.2, 0.3))
        sc.camera = layout.make_camera(eye, (0.5, 0.5, 0.0), (0.0, 1.0, 0.0), 40.0, width, height)
        return sc
    seed = int(rng.integers(1, 1 << 20))
    if kind == "soup":
        # a fixed share of the view is covered whatever the number of triangles
        sc = scenes.soup(tri, seed=seed, width=width, height=height, edge_sigma=0.005 * math.sqrt(1e6 / tri))
    else:
        sc = scenes.stadium(seed=seed, quads=case["quads"], level=case["level"], width=width, height=height)
    sc.camera = _camera(kind, rng, width, height)
    return sc


def _camera(kind, rng, w, h):
    if kind == "soup":
        d = rng.normal(size=3)
        return layout.make_camera(tuple(3.2 * d / np.linalg.norm(d)), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 40.0, w, h)
    a, r = rng.uniform(0.0, 2.0 * math.pi), rng.uniform(0.22, 0.3)
    return layout.make_camera((r * math.cos(a), rng.uniform(0.07, 0.15), r * math.sin(a)), (0.0, 0.05, 0.0),
                              (0.0, 1.0, 0.0), 40.0, w, h)


def _env_map(case, rng):
    w = case["env"]
    return scenes.sky_env(w, w // 2, sun_azim_deg=float(rng.uniform(0.0, 360.0)),
                          sun_elev_deg=float(rng.uniform(20.0, 60.0)))


class _State:
    """What the program holds between calls; its device objects go when it goes."""

    def __init__(self, case, seed):
        self.case, self.seed = case, seed
        self.rng = np.random.default_rng([seed, 77])
        self.open = []  # closed last to first
        self.ctx = self.keep(api.Context(0))

    def keep(self, obj):
        self.open.append(obj)
        return obj

    def scene(self, src, case):
        S = self.keep(api.Scene(self.ctx, src))
        if case["prec"]:
            S.set_precision(case["prec"])
        S.build_bvh_device(want_arrays=False)
        if case.get("env"):
            w = case["env"]
            S.set_env(_env_map(case, self.rng), w, w // 2)
        return S

    def __del__(self):
        while self.open:
            self.open.pop().close()


def prepare(case, seed):
    st = _State(case, seed)
    rng, kind = st.rng, case["kind"]
    if kind == "frame":
        w, h = case["width"], case["height"]
        src = _make_scene(case, rng, w, h)
        S = st.scene(src, case)
        if case["grid"]:
            S.grid_config(1600, 1600, 16, 32, enable=case["grid"])
        st.job = st.keep(api.Job(st.ctx, S, w, h, max_depth=case["depth"], mode=case["mode"], rr_depth=case["rr"],
                                 film_kahan=case["mode"], spp=case["spp"], use_graph=1, inflight=case["inflight"],
                                 grid_updates=0))
        st.camera = src.camera
        st.first = float(1 + int(rng.integers(0, 1000)))
        st.seeds = None
        if case["mode"] == 0:  # allocateState's pairs of odd 30-bit numbers, frame by frame
            n = 2 * (1 + 2 * case["depth"]) * case["spp"]
            st.seeds = (rng.integers(2 ** 29, 2 ** 30, size=(case["frames"], n)) | 1).astype(np.int32)
        if case["read"] == "async":
            st.pinned = torch.empty((w * h, 4), dtype=torch.float32, pin_memory=True)
            st.film = st.pinned.numpy()
    elif kind == "preview":
        src = _make_scene(case, rng, case["width"], case["height"])
        st.S, st.camera = st.scene(src, case), src.camera
    elif kind == "query":
        src = _make_scene(case, rng)
        st.S = st.scene(src, case)
        st.rays = _rays(case, src, seed)
    elif kind == "load":
        st.src = _make_scene(case, rng, case["width"], case["height"])
        st.map = _env_map(case, rng)
    else:
        src = _make_scene(case, rng)
        st.S = st.scene(src, case)
        st.frames = []
        sizes = np.random.default_rng(case["frames"])  # the same frame sizes whatever the seed
        for _ in range(case["frames"]):
            w, h = (_between(sizes, case["lo"], case["hi"]) for _ in range(2))
            st.frames.append((_camera(case["scene"], rng, w, h), w, h, int(sizes.integers(1, case["spp"] + 1)),
                              float(1 + int(rng.integers(0, 1000)))))
        if kind == "served":
            room = scenes.box_room(64, 64)
            st.other = st.scene(room, dict(prec=0))
            st.frames = [(room.camera if k % 4 == 3 else c, w, h, spp, fc)
                         for k, (c, w, h, spp, fc) in enumerate(st.frames)]
            st.films = [np.zeros((f[1] * f[2], 4), np.float32) for f in st.frames]
            st.server = st.keep(api.Server(st.ctx, lanes=16, max_width=case["hi"], max_height=case["hi"],
                                           max_spp=case["spp"], max_depth=case["depth"], rr_depth=case["rr"],
                                           merged=4))
    return st


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rays(case, src, seed):
    o, d = scenes.random_rays(src, case["rays"], seed=seed)
    return layout.make_rays(o, d)


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "frame":
        J = state.job
        J.clear()
        J.set_camera(state.camera)
        for f in range(case["frames"]):
            J.render(None if state.seeds is None else state.seeds[f], state.first + f * case["spp"])
        if case["read"] == "image":
            argb, log_average = J.image()
            return {"argb": argb, "log_average": float(log_average)}
        if case["read"] == "film":
            return J.film(resolve=True)
        J.film_async(state.film, resolve=True)
        J.wait()
        return state.pinned
    if kind == "preview":
        return state.S.preview(state.camera, case["width"], case["height"])
    if kind == "query":
        t, prim = state.S.trace_closest(state.rays)
        return {"t": t, "prim": prim, "occluded": state.S.trace_any(state.rays)}
    if kind == "load":
        S = api.Scene(state.ctx, state.src)
        if case["prec"]:
            S.set_precision(case["prec"])
        S.build_bvh_device(want_arrays=False)
        S.set_env(state.map, case["env"], case["env"] // 2)
        out = S.preview(state.src.camera, case["width"], case["height"])
        S.close()
        return out
    if kind == "batch":
        films, rays = api.batch_render(state.ctx, state.S, state.frames, max_depth=case["depth"],
                                       rr_depth=case["rr"])
        return {"films": films, "rays": rays}
    ids = []
    for k, ((cam, w, h, spp, fc), film) in enumerate(zip(state.frames, state.films)):
        scene = state.other if k % 4 == 3 else state.S
        rid = C.c_int64()
        cam = np.ascontiguousarray(cam)
        check(lib().mt_job_submit(state.server.h, scene.h, _ptr(cam), w, h, spp, fc, _ptr(film), C.byref(rid)))
        ids.append(rid.value)
    for rid in ids:
        check(lib().mt_job_wait(state.server.h, rid, -1.0))
    return state.films


# ------------------------------------------------------------------- work

# rays a path sample traces (camera, extension and shadow rays), as counted by the device
_RAYS = {"room": 6.0, "textured": 6.0, "soup": 2.5, "stadium": 4.0}


def _trace_flops(tri):
    """One ray's box and triangle tests: two child boxes (24 operations) a level of a balanced tree,
    entered about four times over, and three triangle tests (50 operations)."""
    return 24 * 4 * max(1.0, math.log2(tri)) + 150


def _scene_bytes(case):
    """The geometry a traversal reads: a 64-byte record and a 48-byte triangle, once each (a view that
    covers the scene reads nearly all of it), and the environment's texels."""
    return 112 * case["tri"] + 16 * (case.get("env") or 0) ** 2 // 2


def work(case):
    kind = case["kind"]
    ray = _trace_flops(case["tri"])
    if kind == "frame":
        px = case["width"] * case["height"]
        rays = px * case["spp"] * case["frames"] * _RAYS[case["scene"]]
        if case["mode"] == 0:  # no Russian roulette: two rays a bounce
            rays = px * case["spp"] * case["frames"] * 1.2 * case["depth"]
        return {"bytes": _scene_bytes(case) + 16 * px, "flops": rays * (ray + 300)}
    if kind == "preview":
        px = case["width"] * case["height"]
        return {"bytes": _scene_bytes(case) + 8 * px, "flops": px * (ray + 60)}
    if kind == "query":
        n = case["rays"]
        return {"bytes": min(_scene_bytes(case), n * 4096) + n * (80 + 12), "flops": 2 * n * ray}
    if kind == "load":
        px = case["width"] * case["height"]
        # points, faces and materials in; the traversal layout out; texels in, their tables out
        return {"bytes": case["tri"] * (48 + 40 + 112) + case["env"] ** 2 // 2 * (16 + 20) + 8 * px,
                "flops": px * (ray + 60) + 20 * case["tri"] * math.log2(case["tri"])}
    side = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])  # the mean of the sizes drawn
    px = case["frames"] * side * side
    return {"bytes": _scene_bytes(case) + 16 * px,
            "flops": px * (1 + case["spp"]) / 2 * _RAYS[case["scene"]] * (ray + 300)}


# ------------------------------------------------------------------ exact


def exact(case, seed):
    """Closest distances of the smaller ray sets in 64 bits, every ray against every triangle. The films
    of whole renders have no such value here: a path tracer in plain torch would take minutes."""
    if case["kind"] != "query" or case["rays"] * case["tri"] > 2.5e8:
        return None
    src = _make_scene(case, np.random.default_rng([seed, 77]))
    r = _rays(case, src, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    f64 = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev, torch.float64)  # noqa: E731
    p = f64(src.points[:, :3])
    v = [p[torch.from_numpy(src.faces[k].astype(np.int64)).to(dev)] for k in ("vx", "vy", "vz")]
    e1, e2 = v[1] - v[0], v[2] - v[0]
    o, d = f64(r["o"][:, :3]), f64(r["d"][:, :3])
    t_min, t_max = f64(r["tMin"]), f64(r["tMax"])
    best = t_max.clone()
    for k in range(0, src.ntri, 1024):
        a1, a2, a0 = e1[k:k + 1024], e2[k:k + 1024], v[0][k:k + 1024]
        h = torch.linalg.cross(d[:, None, :], a2[None])
        a = (a1[None] * h).sum(-1)
        s = o[:, None, :] - a0[None]
        b1 = (s * h).sum(-1) / a
        q = torch.linalg.cross(s, a1[None].expand_as(s))
        b2 = (d[:, None, :] * q).sum(-1) / a
        t = (a2[None] * q).sum(-1) / a
        ok = (a.abs() >= 1e-7) & (b1 >= 0) & (b1 <= 1) & (b2 >= 0) & (b1 + b2 <= 1) & (t > t_min[:, None])
        best = torch.minimum(best, torch.where(ok, t, torch.full_like(t, math.inf)).amin(1))
    return {"t": best.cpu().numpy(), "prim": None, "occluded": None}
