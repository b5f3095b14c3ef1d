"""Passes and frames of a job that run side by side (each logs its contributions, which
are added to the film in pass order) against the same passes rendered one by one: the
same film, totals and queue lengths bit for bit, for passes fewer than, as many as
and more than run at once, with reads, clears and camera changes between frames, in
both semantics, with and without graphs, Kahan sums and frames in flight."""
import numpy as np
import pytest

from mambatracer_gb300 import api, layout, scenes

pytestmark = pytest.mark.gpu

DEPTH = 5


@pytest.fixture(scope="module")
def room(ctx):
    sc = scenes.textured_room(61, 47)
    S = api.Scene(ctx, sc)
    S.build_bvh_device(want_arrays=False)
    yield sc, S
    S.close()


def _seeds(f, spp):
    n = 2 * (1 + 2 * DEPTH) * spp
    return (np.random.default_rng(f).integers(2 ** 29, 2 ** 30, size=n) | 1).astype(np.int32)


def _one_by_one(ctx, S, cam, mode, kahan, first, npass, seeds):
    """One-pass frames, each waited for, on a job that times its kernels (one pass at a time)."""
    J = api.Job(ctx, S, 61, 47, max_depth=DEPTH, mode=mode, rr_depth=3 if mode else 0, film_kahan=kahan, profile=1)
    J.set_camera(cam)
    per = 2 * (1 + 2 * DEPTH)
    for p in range(npass):
        J.render(None if seeds is None else seeds[p * per:(p + 1) * per], first + p)
        ctx.finish()
    out = J.film(), J.total_rays(), J.stats()[1]
    J.close()
    return out


@pytest.mark.parametrize("spp", [1, 2, 3, 4, 5, 9])
@pytest.mark.parametrize("mode,kahan,graph", [(1, 1, 1), (1, 0, 0), (0, 0, 1)])
def test_overlapping_passes(ctx, room, spp, mode, kahan, graph):
    sc, S = room
    frames = 5
    seeds = None if mode else np.concatenate([_seeds(f, spp) for f in range(frames)])
    want = _one_by_one(ctx, S, sc.camera, mode, kahan, 1.0, frames * spp, seeds)
    J = api.Job(ctx, S, 61, 47, max_depth=DEPTH, mode=mode, rr_depth=3 if mode else 0, film_kahan=kahan, spp=spp,
                use_graph=graph)
    per = 2 * (1 + 2 * DEPTH) * spp
    for again in range(2):
        # a frame of another camera, cleared away while it may still run
        J.set_camera(layout.make_camera((0.4, 0.6, 2.2), (0.5, 0.5, 0.0), (0.0, 1.0, 0.0), 50.0, 61, 47))
        J.render(None if mode else _seeds(99, spp), 7.0)
        J.clear()
        J.set_camera(sc.camera)
        for f in range(frames):
            J.render(None if mode else seeds[f * per:(f + 1) * per], 1.0 + f * spp)
            if again and f in (0, 2):
                J.film()
        assert J.film().tobytes() == want[0].tobytes()
        assert np.array_equal(J.total_rays(), want[1])
        assert np.array_equal(J.stats()[1], want[2])
    J.close()


@pytest.mark.parametrize("spp", [1, 3, 6])
def test_overlap_within_frames_in_flight(ctx, room, spp):
    """Two of the caller's frames in flight, whose passes overlap too: each frame equals
    the frame rendered alone from a cleared film."""
    sc, S = room
    alone = []
    for f in range(3):
        film, _, _ = _one_by_one(ctx, S, sc.camera, 1, 0, 1.0 + f * spp, spp, None)
        alone.append(film)
    J = api.Job(ctx, S, 61, 47, max_depth=DEPTH, mode=1, rr_depth=3, film_kahan=0, spp=spp, inflight=2, use_graph=1)
    J.set_camera(sc.camera)
    for f in range(3):
        J.render(None, 1.0 + f * spp)
    want = (alone[0] + alone[1]) + alone[2]
    assert J.film().tobytes() == want.tobytes()
    J.close()
