"""Calls from several threads at once whose kernels need different amounts of
shared memory: a launch's limit must not depend on what another thread's launch
of the same kernel asks for."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import bvhraytracer_gb300 as pkg  # noqa: E402
from bvhraytracer_gb300 import scenes as S  # noqa: E402
from tests.test_gpu_histograms import _chain  # noqa: E402
from tests.test_gpu_pool import _rays  # noqa: E402

pytestmark = pytest.mark.gpu


def _in_threads(calls, times):
    errors = []

    def loop(call):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(times):
                    call()
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=loop, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


@pytest.mark.parametrize("jobs", [False, True], ids=["trace", "trace_jobs"])
def test_direction_sorts_of_several_widths(jobs):
    """More than 48 KB of shared memory from 27 bins per face side on."""
    tris = S.clutter(20, 3)
    scene = pkg.Scene(pkg.Bvh(tris, 8, 8))
    rays = _rays(tris, 64, 1)
    want = scene.trace(rays, kind="any")["occluded"]
    outs = {k: torch.full_like(want, 9) for k in (27, 28, 30, 32)}

    def call(k):
        if jobs:
            pkg.trace_jobs([(scene, rays, "any", outs[k], k)])
        else:
            scene.trace(rays, kind="any", out=outs[k], reorder=k)

    _in_threads([lambda k=k: call(k) for k in outs], 1500)
    for k, o in outs.items():
        assert torch.equal(o, want), k


def test_traversal_stacks_of_several_depths():
    """General and packed kernels on trees whose stacks take 49 to 113 KB."""
    rng = np.random.default_rng(2)
    r = np.zeros((64, 8), np.float32)
    r[:, :3] = rng.uniform(0.2, 0.8, (64, 3))
    r[:, 3] = 100.0
    r[:, 4:7] = rng.uniform(0.1, 1.0, (64, 3))
    rays = torch.from_numpy(r).cuda()
    scenes = [pkg.Scene(_chain(16, levels, 2)) for levels in (7, 9, 12, 14)]
    want = [s.trace(rays, scheme="persistent", counters=True)["hits"] for s in scenes]
    outs = [torch.full_like(w, 9.0) for w in want]
    for opts in ({"save_distance": True}, {"counters": True, "depth_hist": True},
                 {"counters": True, "scheme": "persistent"}):
        _in_threads([lambda s=s, o=o: s.trace(rays, out=o, **opts) for s, o in zip(scenes, outs)],
                    300)
        for o, w in zip(outs, want):
            assert torch.equal(o.view(torch.int32), w.view(torch.int32)), opts
            o.fill_(9.0)
