"""bvhgpu_trace_batches_noalloc with batches of every size class: the packed
scene's kernel is chosen by the batch's size and rays, so a warm-up call loads
all of them, and the words that the choice is kept in are shared by all calls."""
import subprocess
import sys
from pathlib import Path

import pytest

torch = pytest.importorskip("torch")

import bvhraytracer_gb300 as pkg  # noqa: E402
from bvhraytracer_gb300 import scenes as S  # noqa: E402
from tests.test_gpu_pool import LINE, _rays  # noqa: E402

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

WARM_UP = """
import sys, torch
import bvhraytracer_gb300 as pkg
from bvhraytracer_gb300 import scenes as S
from tests.test_gpu_pool import LINE, _rays
n, l, fmt, profile = int(sys.argv[1]), int(sys.argv[2]), sys.argv[3], sys.argv[4]
tris = S.clutter(30, 2)
scene = pkg.Scene(pkg.Bvh(tris, n, l), node_format=fmt)
rays = _rays(tris, LINE + 1000, 1)
cam, target, _ = S.clutter_viewpoints(30, 2)
together = pkg.camera_rays(cam, target, 1024, 512)
out = {"closest": torch.empty((together.shape[0], 4), device="cuda"),
       "any": torch.empty(together.shape[0], dtype=torch.uint8, device="cuda")}
def run(batch, **kw):
    for kind in ("closest", "any"):
        scene.trace_batches_noalloc([(batch, kind, out[kind][:batch.shape[0]])], profile=profile, **kw)
    torch.cuda.synchronize()
run(rays[:100])
before = torch.cuda.mem_get_info()[0]
for batch in (rays[:40000], rays[:140000], rays, together):
    run(batch)
    run(batch, any_order=True)
print("taken", before - torch.cuda.mem_get_info()[0])
"""


@pytest.mark.parametrize("n,l,fmt,profile", [(8, 8, "fp32", "instrumented"), (4, 4, "q8", "fast"),
                                             (16, 4, "fp32", "fast"), (12, 9, "q8", "instrumented")])
def test_one_small_call_warms_every_size_up(n, l, fmt, profile):
    """In a process of its own, where no other call has loaded a kernel."""
    r = subprocess.run([sys.executable, "-c", WARM_UP, str(n), str(l), fmt, profile], cwd=ROOT,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split()[-2:] == ["taken", "0"], r.stdout


@pytest.mark.parametrize("n,l,fmt", [(8, 8, "fp32"), (16, 4, "q8"), (4, 2, "fp32")])
@pytest.mark.parametrize("profile,any_order", [("instrumented", False), ("instrumented", True),
                                               ("fast", False)])
def test_large_batches_of_one_call(n, l, fmt, profile, any_order):
    """Scattered batches above the pool's line, ones that stay together, and
    smaller ones in one call; the same call again, in the other order, finds
    the words as the first one left them."""
    tris = S.clutter(30, 2)
    scene = pkg.Scene(pkg.Bvh(tris, n, l), node_format=fmt)
    scattered = _rays(tris, LINE + 4097, n, extreme=True)
    cam, target, _ = S.clutter_viewpoints(30, 2)
    together = pkg.camera_rays(cam, target, 768, 512)
    batches, want = [], []
    for rays in (scattered, together, scattered[:40000], scattered[7:LINE + 8], together[:3000],
                 scattered[:140001]):
        for kind in ("closest", "any"):
            key = "hits" if kind == "closest" else "occluded"
            ref = scene.trace(rays, kind=kind, profile=profile, scheme="persistent", counters=True)[key]
            want.append(ref)
            batches.append((rays, kind, torch.full_like(ref, 5)))
    for order in (1, -1):
        for _, _, out in batches:
            out.fill_(5)
        scene.trace_batches_noalloc(batches[::order], profile=profile, any_order=any_order)
        torch.cuda.synchronize()
        for (_, kind, got), ref in zip(batches, want):
            if kind == "any":
                assert torch.equal(got, ref)
            else:  # a NaN of a degenerate ray matches any NaN
                assert torch.equal(got.view(torch.int32)[:, 0], ref.view(torch.int32)[:, 0])
                same = (got[:, 1:] == ref[:, 1:]) | (torch.isnan(got[:, 1:]) & torch.isnan(ref[:, 1:]))
                assert bool(same.all())
    scene.status()
