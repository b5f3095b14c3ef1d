"""Merged rounds of a server that overlap: films equal the jobs rendered alone, bit for
bit, with requests that share streams, join while others run, end after different
passes, are cancelled while their passes are in flight, and take over their slots."""
import numpy as np
import pytest

from mambatracer_gb300 import api, scenes

pytestmark = pytest.mark.gpu

DEPTH, RR = 5, 3


def _alone(ctx, S, cam, w, h, spp, fc, kahan):
    J = api.Job(ctx, S, w, h, max_depth=DEPTH, mode=1, rr_depth=RR, film_kahan=kahan, spp=spp)
    J.set_camera(cam)
    J.render(None, fc)
    film = J.film()
    J.close()
    return film


@pytest.mark.parametrize("lanes,merged,kahan", [(1, 1, 1), (3, 1, 0), (4, 2, 1), (6, 6, 1)])
def test_overlapping_rounds(ctx, lanes, merged, kahan):
    room = scenes.textured_room(64, 64)
    soup = scenes.soup(5000, seed=8, extent=0.8, edge_sigma=0.03, width=64, height=64)
    S = []
    for sc in (room, soup):
        s = api.Scene(ctx, sc)
        s.build_bvh_device(want_arrays=False)
        S.append(s)
    S[1].set_env(scenes.sky_env(128, 64), 128, 64)
    S[1].set_precision(3)
    srv = api.Server(ctx, lanes=lanes, max_width=80, max_height=80, max_spp=9, max_depth=DEPTH, rr_depth=RR,
                     film_kahan=kahan, merged=merged)
    rng = np.random.default_rng(lanes)
    sent = []
    for k in range(24):
        which = int(rng.integers(0, 2))
        w, h = (int(x) for x in rng.integers(3, 80, 2))
        spp, fc = int(rng.integers(1, 10)), float(1 + 10 * k)
        cam = (room, soup)[which].camera
        sent.append((srv.submit(S[which], cam, w, h, spp, fc), S[which], cam, w, h, spp, fc))
        if k % 5 == 4:
            srv.cancel(sent[-2][0])
        if k % 8 == 7:
            srv.wait(sent[-1][0])
    srv.drain()
    done = 0
    for rid, s, cam, w, h, spp, fc in sent:
        if srv.poll(rid)[0] == api.Server.DONE:
            done += 1
            assert srv.film(rid).tobytes() == _alone(ctx, s, cam, w, h, spp, fc, kahan).tobytes(), (w, h, spp)
    assert done >= 19
    srv.close()
    for s in S:
        s.close()
