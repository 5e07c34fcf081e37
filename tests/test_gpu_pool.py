"""The ray-pool kernel and the choice between it and one thread per ray:
results equal, bit for bit, to the counting kernels' (which are checked
against the oracle elsewhere) at the sizes where the choice changes, for every
node width and format, both profiles and ray kinds, and for rays that take the
exact forms."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import bvhraytracer_gb300 as pkg  # noqa: E402
from bvhraytracer_gb300 import scenes as S  # noqa: E402
from tests import _scenes as TS  # noqa: E402
from tests.test_gpu_histograms import _chain  # noqa: E402

pytestmark = pytest.mark.gpu

LINE = 1 << 18  # more rays than this may run on the pool kernel


def _rays(tris, n, seed, extreme=False):
    """Incoherent rays between points of the scene's box; every fourth short,
    some inactive."""
    rng = np.random.default_rng(seed)
    p = tris.reshape(-1, 3)
    lo, hi = p.min(0), p.max(0)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = rng.uniform(lo, hi, (n, 3))
    r[:, 4:7] = rng.normal(size=(n, 3))
    r[:, 3] = np.where(np.arange(n) % 4 == 0, 0.05 * np.linalg.norm(hi - lo), 1e4)
    r[rng.integers(0, n, 50), 0] = np.nan
    if extreme:
        vals = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-40, 3e38, 1e-20], np.float32)
        at = rng.integers(0, n, 4000)
        r[at, rng.integers(3, 7, 4000)] = vals[rng.integers(0, 8, 4000)]
    return torch.from_numpy(r).cuda()


def _same(scene, rays, **kw):
    for kind in ("closest", "any"):
        key = "hits" if kind == "closest" else "occluded"
        for profile in ("instrumented", "fast"):
            want = scene.trace(rays, kind=kind, profile=profile, scheme="persistent",
                               counters=True)[key]
            for order in ({}, {"any_order": True}) if kind == "any" else ({},):
                got = scene.trace(rays, kind=kind, profile=profile, **kw, **order)[key]
                a, b = got.view(torch.uint8), want.view(torch.uint8)
                if kind == "closest":  # a NaN of a degenerate ray matches any NaN
                    a = torch.where(torch.isnan(got[:, 1:]), 0.0, got[:, 1:]).view(torch.int32)
                    b = torch.where(torch.isnan(want[:, 1:]), 0.0, want[:, 1:]).view(torch.int32)
                    assert torch.equal(got.view(torch.int32)[:, 0], want.view(torch.int32)[:, 0])
                assert torch.equal(a, b), (kind, profile, kw, order)
    scene.status()


@pytest.mark.parametrize("n,l,fmt", [(2, 1, "fp32"), (4, 4, "fp32"), (5, 7, "q8"), (8, 8, "fp32"),
                                     (8, 4, "q8"), (9, 13, "fp32"), (12, 16, "q8"),
                                     (16, 16, "fp32"), (16, 5, "q8")])
def test_pool_equals_counting_kernel(n, l, fmt):
    tris = S.clutter(30, 2)
    scene = pkg.Scene(pkg.Bvh(tris, n, l), node_format=fmt)
    rays = _rays(tris, LINE + 1, n * 16 + l, extreme=True)
    _same(scene, rays)               # the rays' own choice: the pool
    _same(scene, rays, reorder=3)    # direction order: the pool
    _same(scene, rays[:LINE])        # one thread per ray


@pytest.mark.parametrize("n,l,fmt", [(3, 2, "fp32"), (4, 16, "fp32"), (8, 8, "q8"), (8, 3, "fp32"),
                                     (12, 12, "fp32"), (16, 16, "q8")])
@pytest.mark.parametrize("rays", [1, 5, 4865, 16384, 16385, 32768, 32769])
def test_team_and_solo_sizes(n, l, fmt, rays):
    """Around the sizes where a team per ray gives way to a thread per ray
    (16,384 closest-hit rays, 32,768 any-hit rays) and where a warp takes
    another team."""
    tris = S.clutter(20, 3)
    scene = pkg.Scene(pkg.Bvh(tris, n, l), node_format=fmt)
    _same(scene, _rays(tris, rays, rays + n, extreme=rays > 50))


@pytest.mark.parametrize("n", [LINE + 1, LINE + 31, 1000003])
def test_rays_that_stay_together(n):
    tris = S.clutter(30, 2)
    scene = pkg.Scene(pkg.Bvh(tris, 8, 8))
    cam, target, _ = S.clutter_viewpoints(30, 2)
    rays = pkg.camera_rays(cam, target, 1024, 1024)[:n].contiguous()
    _same(scene, rays)
    _same(scene, rays, scheme="persistent", policy=4, refill=3)


def test_root_leaf_deep_tree_and_inactive_batch():
    one = np.array([[0, 0, 0, 1, 0, 0, 0, 1, 0]], np.float32)
    _same(pkg.Scene(pkg.Bvh(one, 8, 8)), _rays(np.array([[-1, -1, -1, 1, 1, 1, 0, 0, 0]]), LINE + 5, 1))
    deep = pkg.Scene(_chain(2, 60, 2))  # more levels than the pool's stacks
    _same(deep, _rays(np.array([[0, 0, 0, 1, 1, 1, 0, 0, 0]]), LINE + 5, 2))
    tris = S.clutter(30, 2)
    rays = _rays(tris, LINE + 64, 3)
    rays[:, 0] = float("nan")
    _same(pkg.Scene(pkg.Bvh(tris, 4, 4)), rays)


def test_unordered_boxes_take_the_general_kernels():
    tris, bvh, _ = TS.bvh("clutter120", 8, 4)
    arrays = bvh.export_compact()
    arrays["lo3"] = arrays["lo3"].copy()
    leaf = np.flatnonzero(arrays["child_count"] == 0)[:5]
    arrays["lo3"][leaf, 0] = np.inf
    scene = pkg.Scene(pkg.Bvh.from_compact(arrays, 8, 4))
    _same(scene, _rays(tris, LINE + 1, 4))


@pytest.mark.parametrize("fmt", ["fp32", "q8"])
def test_boxes_that_are_not_nested(fmt):
    """Imported trees whose inner boxes are smaller than what they hold: nothing
    is dropped behind tMax, and Q8 records stay with the general kernels."""
    tris, bvh, _ = TS.bvh("clutter120", 8, 4)
    arrays = bvh.export_compact()
    inner = np.flatnonzero(arrays["child_count"] > 0)[1::3]
    lo, hi = arrays["lo3"].copy(), arrays["hi3"].copy()
    hi[inner] = lo[inner] + 0.8 * (hi[inner] - lo[inner])
    arrays["lo3"], arrays["hi3"] = lo, hi
    scene = pkg.Scene(pkg.Bvh.from_compact(arrays, 8, 4), node_format=fmt)
    rays = _rays(tris, LINE + 1, 6)
    _same(scene, rays)
    _same(scene, rays[:40000])
    _same(scene, rays[:3000])


def test_captured_and_concurrent_traces():
    tris = S.clutter(60, 2)
    scene = pkg.Scene(pkg.Bvh(tris, 8, 8))
    rays = _rays(tris, LINE + 1000, 5)
    want = scene.trace(rays, kind="any", counters=True)["occluded"]
    out = torch.full_like(want, 7)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        scene.trace(rays, kind="any", out=out)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    # more launches in flight than any ring of slots could hold
    streams = [torch.cuda.Stream() for _ in range(4)]
    outs = []
    for k in range(160):
        with torch.cuda.stream(streams[k % 4]):
            outs.append(scene.trace(rays, kind="any")["occluded"])
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs)
    scene.status()


@pytest.mark.parametrize("profile", ["instrumented", "fast"])
@pytest.mark.parametrize("reorder,any_order", [(0, False), (4, True), (4, False)])
@pytest.mark.parametrize("each", [3, 40001, 140001])
def test_many_scenes_on_the_packed_kernels(profile, reorder, any_order, each):
    """Jobs of scenes of several widths and formats, small and large in all."""
    jobs, want = [], []
    for i, (n, l, fmt) in enumerate([(8, 8, "fp32"), (8, 4, "fp32"), (4, 4, "q8"), (16, 3, "fp32"),
                                     (12, 9, "q8"), (8, 8, "fp32")]):
        tris = S.clutter(10 + 7 * i, i)
        scene = pkg.Scene(pkg.Bvh(tris, n, l), node_format=fmt)
        rays = _rays(tris, each + i, i, extreme=each > 3)
        for kind in ("closest", "any"):
            ref = scene.trace(rays, kind=kind, profile=profile, counters=True)
            ref = ref["hits" if kind == "closest" else "occluded"]
            want.append(ref)
            jobs.append((scene, rays, kind, torch.zeros_like(ref), reorder, any_order))
    pkg.trace_jobs(jobs, profile=profile)
    torch.cuda.synchronize()
    for (scene, rays, kind, got, _, _), ref in zip(jobs, want):
        if kind == "closest":
            same = (got == ref) | (torch.isnan(got) & torch.isnan(ref))
            assert torch.equal(got.view(torch.int32)[:, 0], ref.view(torch.int32)[:, 0])
            assert bool(same[:, 1:].all())
        else:
            assert torch.equal(got, ref)
        scene.status()


@pytest.mark.parametrize("n", [2, 31, 4095, 4096, 4097, 12289])
@pytest.mark.parametrize("k", [1, 10, 32])
@pytest.mark.parametrize("offset", [0, 4])
def test_direction_order_chunks(n, k, offset):
    """The direction sort at its chunk size (4,096 rays), few and many bins,
    rays on 32-byte and on 16-byte boundaries, alone and as jobs."""
    tris = S.clutter(20, 3)
    scene = pkg.Scene(pkg.Bvh(tris, 8, 8))
    flat = torch.zeros(8 * n + 4, dtype=torch.float32, device="cuda")
    rays = flat[offset:offset + 8 * n].view(n, 8)
    rays.copy_(_rays(tris, n, n + k, extreme=n > 100))
    want = scene.trace(rays, kind="any", counters=True)["occluded"]
    assert torch.equal(scene.trace(rays, kind="any", reorder=k)["occluded"], want)
    out = [torch.full_like(want, 9) for _ in range(3)]
    pkg.trace_jobs([(scene, rays, "any", o, k) for o in out])
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in out)
    scene.status()


@pytest.mark.parametrize("n,l,fmt", [(2, 1, "fp32"), (4, 16, "fp32"), (5, 7, "q8"), (8, 8, "fp32"),
                                     (9, 13, "fp32"), (12, 5, "q8"), (16, 16, "fp32"),
                                     (16, 16, "q8")])
@pytest.mark.parametrize("rays", [1, 127, 129, 30001])
def test_counting_traces(n, l, fmt, rays):
    """Counters, histograms and results of the packed counting kernel against
    the persistent kernel's, which reads the general records: all equal, with
    and without histograms, in any ray order."""
    tris = S.clutter(20, 4)
    scene = pkg.Scene(pkg.Bvh(tris, n, l), node_format=fmt)
    d = _rays(tris, rays, rays + l, extreme=rays > 200)
    for kind in ("closest", "any"):
        key = "hits" if kind == "closest" else "occluded"
        want = scene.trace(d, kind=kind, scheme="persistent", counters=True, depth_hist=True)
        for opts in ({"depth_hist": True}, {"depth_hist": True, "reorder": 3}, {}):
            got = scene.trace(d, kind=kind, counters=True, **opts)
            for k in ("counters", "depth_hist", "fullness") if "depth_hist" in opts else ("counters",):
                assert torch.equal(got[k], want[k]), (kind, opts, k)
            a, b = got[key], want[key]
            if kind == "closest":  # a NaN of a degenerate ray matches any NaN
                assert torch.equal(a[:, 0].contiguous().view(torch.int32), b[:, 0].contiguous().view(torch.int32))
                a, b = a[:, 1:], b[:, 1:]
                assert torch.equal(torch.isnan(a), torch.isnan(b))
                a, b = (torch.where(torch.isnan(x), 0.0, x).view(torch.int32) for x in (a, b))
            assert torch.equal(a, b), (kind, opts)
    scene.status()


def test_captured_jobs():
    """Reordered and plain jobs of one captured call, enough rays for the pool."""
    tris = S.clutter(40, 2)
    scene = pkg.Scene(pkg.Bvh(tris, 8, 8))
    rays = _rays(tris, LINE + 77, 8)
    want = {k: scene.trace(rays, kind=k, scheme="persistent", counters=True) for k in ("closest", "any")}
    want = {"closest": want["closest"]["hits"], "any": want["any"]["occluded"]}
    jobs = [(scene, rays, kind, torch.full_like(want[kind], 5), k, k > 0)
            for kind in ("closest", "any") for k in (0, 4)]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        pkg.trace_jobs(jobs)
    for _ in range(2):
        for j in jobs:
            j[3].fill_(5)
        graph.replay()
        torch.cuda.synchronize()
        for _, _, kind, out, _, _ in jobs:
            assert torch.equal(out.view(torch.uint8), want[kind].view(torch.uint8)), kind
    scene.status()
