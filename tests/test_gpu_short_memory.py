"""Calls on a device that is nearly full (MT_DEVICE_ROOM, which fails the library's own
allocations; each case in a process of its own): what fits the device is not refused
because of memory that an earlier call keeps, and gives the results it gives on an empty
one."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from mambatracer_gb300 import api, layout, scenes
from mambatracer_gb300._lib import MTError, check, lib

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CASES = {}


def case(f):
    CASES[f.__name__] = f
    return f


def _room(n):
    """The library's arrays may grow by n bytes from here on (None: by any number)."""
    _room.calls += 1
    os.environ["MT_DEVICE_ROOM"] = "" if n is None else f"{n}" + " " * _room.calls


_room.calls = 0


def _rays(sc, n):
    o, d = scenes.random_rays(sc, n, seed=n)
    return layout.make_rays(o, d)


def _soup(n=20000):
    sc = scenes.soup(n, seed=4, extent=0.8, edge_sigma=0.05, width=320, height=240)
    return sc


def _scene(ctx, sc):
    S = api.Scene(ctx, sc)
    S.build_bvh_device(want_arrays=False)
    return S


def _film(ctx, S, cam, **kw):
    J = api.Job(ctx, S, 320, 240, **{**dict(max_depth=4, mode=1, rr_depth=3), **kw})
    J.set_camera(cam)
    for f in range(3):
        J.render(None, float(1 + f * kw.get("spp", 1)))
    film = J.film()
    J.close()
    return film


# ---------------------------------------------------------------- the kept scratch
def _beside_scratch(op, keep=400_000):
    """op(ctx, S, sc) with no room but the scratch that a query of `keep` rays left (88 bytes
    a ray), against op with room."""
    ctx = api.Context(0)
    sc = _soup()
    S = _scene(ctx, sc)
    rays = _rays(sc, keep)
    want = op(ctx, S, sc)
    S.trace_closest(rays)
    _room(0)
    got = op(ctx, S, sc)
    _room(None)
    for a, b in zip(want, got):
        assert np.asarray(a).tobytes() == np.asarray(b).tobytes()
    S.close()
    ctx.close()


@case
def scene_beside_scratch():
    big = _soup(100_000)  # 8.8 MB of mesh

    def op(ctx, S, sc):
        T = api.Scene(ctx, big)
        n = T.light_count
        T.close()
        return [n]
    _beside_scratch(op)


@case
def tree_beside_scratch():
    big = _soup(100_000)  # 11.2 MB of tree, 7 MB while it is built
    keep = {}

    def op(ctx, S, sc):
        T = keep.setdefault("T", None) or api.Scene(ctx, big)
        keep["T"] = T
        T.build_bvh_device(want_arrays=False)
        return [T.trace_closest(_rays(sc, 1000))[0]]
    _beside_scratch(op)

@case
def environment_beside_scratch():
    maps = [(scenes.sky_env(w, w // 2), w, w // 2) for w in (256, 512)]  # 5 MB of map and tables the larger

    def op(ctx, S, sc):
        out = []
        for m in maps:
            S.set_env(*m)
            out += S.env_arrays(*m[1:])
        return out
    _beside_scratch(op)


@case
def texture_beside_scratch():
    img = np.arange(1 << 20, dtype=np.int32).reshape(1024, 1024)

    def op(ctx, S, sc):
        S.set_texture(0, 0, img)
        S.set_texture(0, 0, None)
        return []
    _beside_scratch(op)


@case
def formats_beside_scratch():
    def op(ctx, S, sc):
        out = []
        for p in (1, 2, 0):
            S.set_precision(p)
            out.append(S.trace_any(_rays(sc, 1000)))
        return out
    _beside_scratch(op)


@case
def image_beside_scratch():
    jobs = []

    def op(ctx, S, sc):
        J = jobs.pop() if jobs else None
        if J is None:
            jobs.append(api.Job(ctx, S, 320, 240, max_depth=3, mode=1))  # its image is allocated by the next call
            J = api.Job(ctx, S, 320, 240, max_depth=3, mode=1)
        J.set_camera(sc.camera)
        J.render(None, 1.0)
        argb, la = J.image()
        J.close()
        return [argb]
    _beside_scratch(op)


@case
def lanes_beside_scratch():
    def op(ctx, S, sc):
        srv = api.Server(ctx, lanes=1, max_width=320, max_height=240, max_spp=1, max_depth=4, merged=0)
        rid = srv.submit(S, sc.camera, 320, 240, 1)
        film = srv.wait(rid).copy()
        srv.close()
        return [film]
    _beside_scratch(op)


@case
def job_beside_scratch():
    # 22 MB a pass with its log and four of those side by side; one pass alone takes 15 MB
    _beside_scratch(lambda ctx, S, sc: [_film(ctx, S, sc.camera)])


@case
def own_allocation_beside_scratch():
    """A query above what is kept (2 GiB) beside a kept scratch of nearly that."""
    ctx = api.Context(0)
    sc = _soup(200)
    S = _scene(ctx, sc)
    rays = np.tile(_rays(sc, 1 << 16), 400)
    S.trace_any(rays[:24_000_000])
    _room(200 << 20)
    occ = S.trace_any(rays[:25_000_000])
    _room(None)
    assert np.array_equal(occ[:1 << 16], occ[1 << 16:1 << 17])
    S.close()
    ctx.close()


@case
def quad_nodes_without_the_surface_area_tree():
    """4-wide nodes where only those over the reference's tree fit (64 bytes a triangle): made, as
    they were before that tree was built for them, and the same answers."""
    ctx = api.Context(0)
    sc = _soup()
    S = _scene(ctx, sc)
    rays = _rays(sc, 20_000)
    t0, p0 = S.trace_closest(rays)
    a0 = S.trace_any(rays)
    for room in (1_300_000, 2_600_000, 4_000_000, None):
        S.set_precision(0)
        _room(0)
        with pytest.raises(MTError, match="NOMEM"):  # the scratch kept so far goes
            api.Scene(ctx, sc)
        _room(room)
        S.set_precision(3)
        _room(None)
        t, p = S.trace_closest(rays)
        assert np.array_equal(t, t0) and np.array_equal(p, p0) and np.array_equal(S.trace_any(rays), a0)
    S.close()
    ctx.close()


@case
def mesh_without_scratch():
    """A mesh with lights and an imported tree where just their own arrays fit (88 bytes a triangle
    and the light list; 112 bytes a triangle): made without scratch, with the same contents."""
    ctx = api.Context(0)
    sc = _soup()
    sc.materials = np.concatenate([sc.materials, sc.materials[:1]])
    sc.materials["emission_param"][-1] = 2.0
    sc.materials["emission_color"][-1] = 1.0
    rng = np.random.default_rng(1)
    lit = rng.random(sc.ntri) < 0.3
    sc.faces["mat"] = np.where(lit, len(sc.materials) - 1, 0)
    nodes, bounds, _ = api.bvh_build_host(sc)
    S = api.Scene(ctx, sc)
    S.import_bvh(nodes, bounds)
    assert S.light_count == lit.sum()
    film = _film(ctx, S, sc.camera)
    for extra in (0, 100_000):  # bytes beyond the arrays: none, and less than any scratch that is kept
        _room(0)
        with pytest.raises(MTError, match="NOMEM"):  # the scratch kept so far goes
            api.Scene(ctx, sc)
        mesh = -(-sc.points.nbytes // 256) * 256 + 512 + 40 * sc.ntri
        _room(mesh + sc.materials.nbytes + 4 * int(lit.sum()) + extra)
        T = api.Scene(ctx, sc)
        assert T.light_count == lit.sum()
        _room(0)
        with pytest.raises(MTError, match="NOMEM"):
            api.Scene(ctx, sc)
        _room(64 * (sc.ntri - 1) + 48 * sc.ntri + extra)
        T.import_bvh(nodes, bounds)
        _room(None)
        for a, b in zip(T.layout()[:2], S.layout()[:2]):
            assert a.tobytes() == b.tobytes()
        assert _film(ctx, T, sc.camera).tobytes() == film.tobytes()
        T.close()
    S.close()
    ctx.close()


@case
def resolved_read_without_room():
    """Resolved reads of a film, waited for and enqueued (the same buffer twice), where the divided
    film has no room on the device: the values of a job that has it."""
    ctx = api.Context(0)
    sc = _soup(2000)
    S = _scene(ctx, sc)
    got = []
    for room in (None, 3_000_000):  # the film is 4.9 MB, the scratch of the build less than 2
        J = api.Job(ctx, S, 640, 480, max_depth=3, mode=1)
        J.set_camera(sc.camera)
        out = [np.empty((640 * 480, 4), np.float32) for _ in range(3)]
        J.render(None, 1.0)
        _room(room)
        J.film_async(out[0], resolve=True)
        J.render(None, 2.0)
        J.film_async(out[1], resolve=True)
        J.render(None, 3.0)
        J.film_async(out[1], resolve=True)
        J.wait()
        out[2][:] = J.film(resolve=True)
        _room(None)
        got.append(out + [J.film()])
        J.close()
    for a, b in zip(*got):
        assert a.tobytes() == b.tobytes()
    assert np.array_equal(got[0][1][:, :3], got[0][3][:, :3] / np.float32(3))
    S.close()
    ctx.close()


# ------------------------------------------------ path state of overlapping passes
def _leaves_room(make, needs, total):
    """make(ctx, S, cam), which needs `needs` bytes of its own arrays, leaves room for the rest of
    `total`, and gives what it gives on an empty device."""
    ctx = api.Context(0)
    sc = _soup()
    S = _scene(ctx, sc)
    S.set_env(scenes.sky_env(256, 128), 256, 128)
    S.grid_config(160, 160, 16, 32, enable=2)
    want, close = make(ctx, S, sc.camera)
    close()
    _room(total)
    got, close = make(ctx, S, sc.camera)
    b = C.c_void_p()
    check(lib().mt_buf_alloc(ctx.h, total - needs, C.byref(b)))  # raises where the room is gone
    check(lib().mt_buf_free(b))
    _room(None)
    close()
    for a, b in zip(want, got):
        assert a.tobytes() == b.tobytes()
    S.close()
    ctx.close()


@case
def job_leaves_room():
    # 304 bytes a pixel and pass with its log (depth 4) would be 93 MB for four at once; 192 with
    # films alone, 15 MB
    def make(ctx, S, cam):
        J = api.Job(ctx, S, 320, 240, max_depth=4, mode=1, rr_depth=3, spp=4, grid_updates=0)
        J.set_camera(cam)
        J.render(None, 1.0)
        return [J.film()], J.close
    _leaves_room(make, 20_000_000, 100_000_000)


@case
def server_leaves_room():
    # two slots: 31 MB of queues and films; 2 x 24 MB of queues more and 3 x 20 MB of logs for three sets
    def make(ctx, S, cam):
        srv = api.Server(ctx, lanes=2, max_width=320, max_height=240, max_spp=3, max_depth=4, merged=1)
        films = [srv.wait(srv.submit(S, cam, 320, 240, 3)).copy() for _ in range(2)]
        return films, srv.close
    _leaves_room(make, 36_000_000, 150_000_000)


@case
def batch_with_room_for_one_pass():
    """A batch whose four passes do not fit side by side: one after the other, the same films."""
    ctx = api.Context(0)
    sc = _soup()
    S = _scene(ctx, sc)
    frames = [(sc.camera, 320, 240, 4, 1.0), (sc.camera, 200, 100, 2, 9.0)]
    want, rays = api.batch_render(ctx, S, frames, max_depth=4)  # 97k pixels: 44 MB a pass with its log
    _room(0)
    with pytest.raises(MTError, match="NOMEM"):  # the scratch of that batch goes
        api.Scene(ctx, scenes.soup(4_000_000, seed=1, width=64, height=64))
    for room in (22_000_000, 60_000_000):
        _room(room)
        got, r = api.batch_render(ctx, S, frames, max_depth=4)
        _room(0)
        with pytest.raises(MTError, match="NOMEM"):
            api.batch_render(ctx, S, [(sc.camera, 1920, 1080, 4, 1.0)], max_depth=4)
        assert np.array_equal(r, rays) and all(a.tobytes() == b.tobytes() for a, b in zip(got, want))
    S.close()
    ctx.close()


# ------------------------------------------------------- allocations that fail half-way
@case
def image_arrays_in_part():
    """An image whose first arrays fit and whose later ones do not: refused each time it is asked
    for, and there once it fits."""
    ctx = api.Context(0)
    sc = _soup()
    S = _scene(ctx, sc)
    jobs = [api.Job(ctx, S, 1280, 960, max_depth=3, mode=1) for _ in range(2)]
    for J in jobs:
        J.set_camera(sc.camera)
        J.render(None, 1.0)
    # the image takes 4.9 MB, the averaged film after it 19.7 MB; the scratch given back for them 2 MB
    for room in (0, 6_400_000, 6_400_000, 22_000_000):
        _room(room)
        for _ in range(2):
            with pytest.raises(MTError, match="NOMEM"):
                jobs[0].image()
    _room(None)
    assert np.array_equal(jobs[0].image()[0], jobs[1].image()[0])
    for o in (*jobs, S, ctx):
        o.close()


@case
def formats_in_part():
    """A format whose arrays do not all fit is refused, and the scene renders from its FP32
    records meanwhile, whatever has been made of the format."""
    ctx = api.Context(0)
    sc = _soup()
    S = _scene(ctx, sc)
    rays = _rays(sc, 5000)
    want = S.trace_any(rays)
    refused = 0
    for p in (2, 1):
        for room in range(0, 2_400_000, 300_000):
            S.set_precision(0)
            _room(0)
            with pytest.raises(MTError, match="NOMEM"):  # the scratch kept so far goes
                api.Scene(ctx, sc)
            _room(room)
            try:
                S.set_precision(p)
            except MTError as e:
                assert "NOMEM" in str(e)
                refused += 1
            _room(None)
            assert np.array_equal(S.trace_any(rays), want), (p, room)
    assert refused >= 4
    S.close()
    ctx.close()


@case
def import_in_part():
    """An import beside a tree: in its place where both do not fit. Where no tree fits, the scene
    stays without one: queries are refused, and an import works once there is room. A failed
    import of one that is not a tree leaves the old one."""
    ctx = api.Context(0)
    sc = _soup()
    nodes, bounds, _ = api.bvh_build_host(sc)
    rays = _rays(sc, 5000)
    S = api.Scene(ctx, sc)
    for room in (0, 1_000_000, 1_400_000, 2_200_000):  # records 1.28 MB, triangles 0.96 MB
        _room(0)
        with pytest.raises(MTError, match="NOMEM"):
            api.Scene(ctx, sc)
        _room(room)
        with pytest.raises(MTError, match="NOMEM"):
            S.import_bvh(nodes, bounds)
        _room(None)
        with pytest.raises(MTError, match="no BVH"):
            S.trace_any(rays)
    S.import_bvh(nodes, bounds)
    t, p = S.trace_closest(rays)
    film = _film(ctx, S, sc.camera)
    J = api.Job(ctx, S, 320, 240, max_depth=4, mode=1, rr_depth=3)
    J.set_camera(sc.camera)
    for room in (0, 1_000_000, 1_400_000, 2_200_000, 3_000_000):
        _room(0)
        with pytest.raises(MTError, match="NOMEM"):
            api.Scene(ctx, sc)
        _room(room)
        S.import_bvh(nodes, bounds)
        _room(None)
        t1, p1 = S.trace_closest(rays)
        assert np.array_equal(t1, t) and np.array_equal(p1, p)
        J.clear()
        for f in range(3):
            J.render(None, float(1 + f))
        assert J.film().tobytes() == film.tobytes()
    bad = nodes.copy()
    bad.reshape(-1, 7)[0, 2] = len(bad.reshape(-1, 7))
    with pytest.raises(MTError, match="child"):
        S.import_bvh(bad, bounds)
    assert np.array_equal(S.trace_closest(rays)[0], t)
    for o in (J, S, ctx):
        o.close()


@pytest.mark.parametrize("name", sorted(CASES))
def test_short_memory(name):
    code = f"import sys; sys.path.insert(0, {ROOT!r}); import tests.test_gpu_short_memory as m; m.CASES[{name!r}]()"
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, MT_DEVICE_ROOM=""), timeout=300, cwd=ROOT,
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
