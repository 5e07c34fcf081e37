"""Paths of the kernels on the packed scene that ordinary batches seldom take.
Results equal the counting kernels' bit for bit (tests/test_gpu_pool.py)."""
import pytest

torch = pytest.importorskip("torch")

import bvhraytracer_gb300 as pkg  # noqa: E402
from bvhraytracer_gb300 import scenes as S  # noqa: E402
from tests.test_gpu_pool import LINE, _rays, _same  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("active", ["one_in_32", "one_in_9", "alternate", "all_but_lane_0",
                                    "last_warp_only"])
@pytest.mark.parametrize("n,l,fmt", [(8, 8, "fp32"), (16, 4, "q8")])
def test_pool_refills_among_inactive_rays(active, n, l, fmt):
    """A refill step reads free slots and, for rays that are inactive, gives
    slots back in the same step: every slot stays in exactly one list."""
    tris = S.clutter(30, 2)
    scene = pkg.Scene(pkg.Bvh(tris, n, l), node_format=fmt)
    rays = _rays(tris, LINE + 4097, 11)
    i = torch.arange(rays.shape[0], device="cuda")
    off = {"one_in_32": i % 32 != 7, "one_in_9": i % 9 != 0, "alternate": i % 2 == 0,
           "all_but_lane_0": i % 32 == 0, "last_warp_only": i < rays.shape[0] - 33}[active]
    rays[off, 0] = float("nan")
    _same(scene, rays)
    _same(scene, rays, reorder=3)


@pytest.mark.parametrize("n,l,fmt", [(2, 1, "fp32"), (4, 4, "q8"), (8, 8, "fp32"), (8, 4, "q8"),
                                     (12, 9, "fp32"), (16, 16, "q8"), (16, 2, "fp32")])
def test_solo_kernel_of_one_wave(n, l, fmt):
    """A launch whose rays all run at once takes the one-thread-per-ray kernel
    with more registers: its last size, the next one, and a remainder."""
    tris = S.clutter(30, 5)
    scene = pkg.Scene(pkg.Bvh(tris, n, l), node_format=fmt)
    wave = torch.cuda.get_device_properties(0).multi_processor_count * 128 * 4
    rays = _rays(tris, wave + 1, n + l, extreme=True)
    for k in (wave - 127, wave, wave + 1):
        _same(scene, rays[:k])


@pytest.mark.parametrize("n,l", [(2, 1), (3, 2), (4, 2), (4, 3), (4, 4), (4, 5), (8, 1), (8, 8),
                                 (8, 9), (12, 12), (12, 13), (16, 2), (16, 16)])
@pytest.mark.parametrize("fmt", ["fp32", "q8"])
def test_small_leaves_and_leaves_in_turn(n, l, fmt):
    """The one-thread-per-ray kernel at the leaf sizes where its loop and its
    cheap tests change, in launches of one wave, of more, and planned ones."""
    tris = S.clutter(25, 6)
    scene = pkg.Scene(pkg.Bvh(tris, n, l), node_format=fmt)
    rays = _rays(tris, LINE + 1, 3 * n + l, extreme=True)
    for k in (40000, 140001, LINE + 1):
        _same(scene, rays[:k])
    cam, target, _ = S.clutter_viewpoints(25, 6)
    _same(scene, pkg.camera_rays(cam, target, 768, 512))  # stay together: not the pool


@pytest.mark.parametrize("n,l,fmt,objects", [(12, 4, "fp32", 800), (16, 1, "fp32", 300),
                                             (12, 4, "fp32", 300), (16, 1, "q8", 300)])
def test_wide_trees_on_both_sides_of_the_pool_line(n, l, fmt, objects):
    """Trees of wide nodes with more records than the pool kernel is good for,
    with fewer, and on Q8 records, for large unordered and ordered batches and
    as jobs."""
    tris = S.clutter(objects, 4)
    bvh = pkg.Bvh(tris, n, l)
    wide_bytes = bvh.info["n_inner"] * (560 if n == 12 else 720)
    assert (wide_bytes > 5 << 20) == (objects == 800 or n == 16)
    scene = pkg.Scene(bvh, node_format=fmt)
    rays = _rays(tris, LINE + 1, n + l)
    _same(scene, rays)
    _same(scene, rays, reorder=3)
    for kind in ("closest", "any"):
        key = "hits" if kind == "closest" else "occluded"
        want = scene.trace(rays, kind=kind, scheme="persistent", counters=True)[key]
        jobs = [(scene, rays, kind, torch.full_like(want, 5)) for _ in range(2)]
        pkg.trace_jobs(jobs)
        torch.cuda.synchronize()
        assert all(torch.equal(j[3].view(torch.uint8), want.view(torch.uint8)) for j in jobs)


@pytest.mark.parametrize("n,l,fmt", [(2, 1, "fp32"), (4, 16, "q8"), (8, 8, "fp32"), (8, 5, "q8"),
                                     (12, 13, "fp32"), (12, 5, "q8"), (16, 16, "fp32"),
                                     (16, 4, "q8")])
def test_counting_traces_of_large_batches(n, l, fmt):
    """Counters, histograms and results on both sides of the size from which
    counting traces run on the packed scene, against the persistent kernel's."""
    tris = S.clutter(20, 4)
    scene = pkg.Scene(pkg.Bvh(tris, n, l), node_format=fmt)
    line = 3 << 16
    rays = _rays(tris, line + 1, n + l)
    for d in (rays[:line], rays):
        for kind in ("closest", "any"):
            key = "hits" if kind == "closest" else "occluded"
            want = scene.trace(d, kind=kind, scheme="persistent", counters=True, depth_hist=True)
            for opts in ({"depth_hist": True}, {"depth_hist": True, "reorder": 3}, {}):
                got = scene.trace(d, kind=kind, counters=True, **opts)
                for k in ("counters", "depth_hist", "fullness") if opts else ("counters",):
                    assert torch.equal(got[k], want[k]), (kind, opts, k)
                assert torch.equal(got[key].view(torch.uint8), want[key].view(torch.uint8)), (kind, opts)
    scene.status()


@pytest.mark.parametrize("n,l,fmt", [(4, 4, "fp32"), (4, 4, "q8"), (8, 8, "fp32"), (8, 4, "q8"),
                                     (12, 9, "fp32"), (16, 16, "q8"), (16, 2, "fp32")])
def test_lines_between_the_kernels_of_small_and_middle_batches(n, l, fmt):
    """Teams per ray up to 16,384 to 32,768 closest-hit rays by node width, the
    solo kernel of one wave up to four to six blocks' rays per SM."""
    tris = S.clutter(30, 5)
    scene = pkg.Scene(pkg.Bvh(tris, n, l), node_format=fmt)
    block = torch.cuda.get_device_properties(0).multi_processor_count * 128
    rays = _rays(tris, 6 * block + 1, n + l, extreme=True)
    for k in (16384, 28672, 32768, 4 * block, 5 * block, 6 * block):
        _same(scene, rays[:k])
        _same(scene, rays[:k + 1])


@pytest.mark.parametrize("n,l", [(2, 8), (4, 7), (4, 8), (4, 9), (3, 16)])
def test_leaves_in_turn_on_q8_nodes(n, l):
    """The leaf sizes where 4-wide Q8 nodes stop visiting leaves in turn."""
    tris = S.clutter(25, 6)
    scene = pkg.Scene(pkg.Bvh(tris, n, l), node_format="q8")
    rays = _rays(tris, 140001, n + l, extreme=True)
    for k in (40000, 140001):
        _same(scene, rays[:k])
    cam, target, _ = S.clutter_viewpoints(25, 6)
    _same(scene, pkg.camera_rays(cam, target, 768, 512))
