"""Launch counts against a trace of the device: what mt_job_launches adds for a job's frames is
the number of kernels that ran for them, with and without graphs, frames in flight and
passes side by side. In a process of its own: tracing stays with the process."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_TRACE = r"""
import sys
sys.path.insert(0, {root!r})
import torch
from torch.profiler import profile, ProfilerActivity
from mambatracer_gb300 import api, scenes

def kernels(f):
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    return sum(e.device_type == torch.autograd.DeviceType.CUDA and not e.name.startswith(("Memcpy", "Memset"))
               for e in p.events())

torch.zeros(1, device="cuda")
if kernels(lambda: torch.ones(1 << 20, device="cuda")) == 0 and kernels(lambda: torch.ones(8, device="cuda")) == 0:
    sys.exit(77)  # no tracing here
ctx = api.Context(0)
sc = scenes.box_room(96, 64)
S = api.Scene(ctx, sc)
S.build_bvh_device(want_arrays=False)
for inflight, spp in ((1, 1), (1, 2), (1, 4), (2, 1), (2, 3), (6, 2)):
    for graph in (0, 1):
        J = api.Job(ctx, S, 96, 64, max_depth=6, mode=1, rr_depth=3, inflight=inflight, spp=spp, use_graph=graph)
        J.set_camera(sc.camera)
        def frames():
            for f in range(4):
                J.render(None, 1.0 + f * spp)
            ctx.finish()
        frames()
        before = J.launches()
        n = kernels(frames)
        assert J.launches() - before == n, (inflight, spp, graph, J.launches() - before, n)
        J.close()
"""


def test_launches_equal_the_trace():
    r = subprocess.run([sys.executable, "-c", _TRACE.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    if r.returncode == 77:
        pytest.skip("kernels cannot be traced here")
    assert r.returncode == 0, r.stderr[-2000:]
