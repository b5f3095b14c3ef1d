"""Calls that share the context's scratch: results do not depend on what ran before on
it, as the sizes grow, shrink and alternate between queries, previews and batches,
from several threads of one context and from two contexts at once."""
import threading

import numpy as np
import pytest

from mambatracer_gb300 import api, layout, scenes

pytestmark = pytest.mark.gpu


def _calls(ctx, S, sc, n, w, h):
    o, d = scenes.random_rays(sc, n, seed=n)
    rays = layout.make_rays(o, d)
    t, p = S.trace_closest(rays)
    out = [t, p, S.trace_any(rays), S.trace_counts(rays)[2]]
    out += list(S.preview(sc.camera, w, h))
    films, r = api.batch_render(ctx, S, [(sc.camera, w, h, 2, 1.0), (sc.camera, h, w, 1, 5.0)], max_depth=3)
    return out + [r] + list(films)


SIZES = [(1, 3, 2), (70001, 200, 150), (33, 17, 5), (5000, 64, 64)]


def _scene(ctx):
    sc = scenes.soup(3000, seed=4, extent=0.8, edge_sigma=0.05, width=64, height=64)
    S = api.Scene(ctx, sc)
    S.build_bvh_device(want_arrays=False)
    return sc, S


def test_results_do_not_depend_on_the_scratch(ctx):
    want = []
    for size in SIZES:  # each on a context of its own
        c = api.Context(0)
        sc, S = _scene(c)
        want.append(_calls(c, S, sc, *size))
        S.close()
        c.close()
    sc, S = _scene(ctx)
    for k in (0, 1, 2, 3, 1, 0, 2):
        for a, b in zip(_calls(ctx, S, sc, *SIZES[k]), want[k]):
            assert a.tobytes() == b.tobytes()

    other = api.Context(0)
    sc2, S2 = _scene(other)
    bad = []

    def work(c, s, k):
        for _ in range(3):
            for a, b in zip(_calls(c, s, sc, *SIZES[k]), want[k]):
                if a.tobytes() != b.tobytes():
                    bad.append(k)

    threads = [threading.Thread(target=work, args=(c, s, k)) for c, s in ((ctx, S), (other, S2)) for k in (0, 1, 3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    S.close()
    S2.close()
    other.close()
