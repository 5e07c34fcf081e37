"""The schemes' own kernels without counters, against the oracle. Ordinary
scenes trace on the packed records whatever the scheme; a stack limit just
below the tree's worst case, which no ray here needs, sends a scene to the
kernels that the options name. (They also run trees with unordered or, for Q8,
non-nested boxes, very deep ones, and scenes without room for the packed
records.)"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import bvhraytracer_gb300 as pkg  # noqa: E402
from oracle import oracle as O  # noqa: E402
from tests import _scenes as TS  # noqa: E402
from tests.test_gpu_parity import LIGHT, SCHEMES, bits, dev  # noqa: E402
from tests.test_gpu_pool import _rays  # noqa: E402

pytestmark = pytest.mark.gpu


def _oracle(b, cv, rays, kind, profile):
    if profile == "fast":
        r = O.trace_fast(O.FastView(b.export_fast()), cv, rays, any_hit=kind == "any")
    else:
        r = O.trace_instrumented(cv, rays, shadow=kind == "any")
    return r["hits" if kind == "closest" else "occluded"]


def _case(n, l, fmt, profile, res=(96, 64), name="clutter120"):
    """A scene on the general kernels, and its batches with the oracle's results."""
    tris, b, cv = TS.bvh(name, n, l)
    scene = pkg.Scene(b, node_format=fmt)
    scene.set_stack_limit(b.info["max_stack"] - 1)
    rays = TS.clutter_rays(tris, res=res)
    ref = _oracle(b, cv, rays, "closest", profile)
    sh, ao = TS.secondary(tris, rays, pkg.hit_prims(ref), LIGHT, ao_samples=3)
    return scene, [(rays, "closest", ref)] + [(r, "any", _oracle(b, cv, r, "any", profile))
                                              for r in (sh, ao)]


def _equal(got, want):
    return np.array_equal(bits(got.cpu().numpy().reshape(-1)) if got.dtype == torch.float32
                          else got.cpu().numpy(), bits(want).reshape(-1)
                          if want.dtype == np.float32 else want)


@pytest.mark.parametrize("n,l,fmt", [(4, 4, "fp32"), (4, 16, "q8"), (8, 8, "fp32"), (8, 4, "q8"),
                                     (12, 12, "fp32"), (12, 4, "q8"), (16, 16, "fp32"),
                                     (16, 8, "q8"), (3, 2, "fp32")])
@pytest.mark.parametrize("profile", ["instrumented", "fast"])
def test_every_scheme_and_policy(n, l, fmt, profile):
    scene, batches = _case(n, l, fmt, profile)
    for scheme, kw in SCHEMES:
        if scheme == "stream" and fmt == "q8":
            continue
        for rays, kind, want in batches:
            key = "hits" if kind == "closest" else "occluded"
            for extra in ({}, {"reorder": 4}, {"any_order": True}):
                got = scene.trace(dev(rays), kind=kind, scheme=scheme, profile=profile, **kw,
                                  **extra)[key]
                assert _equal(got, want), (scheme, kw, kind, extra)
    scene.status()


@pytest.mark.parametrize("policy", [0, 2])
@pytest.mark.parametrize("one_launch", [False, True], ids=["per_group", "one_launch"])
@pytest.mark.parametrize("profile", ["instrumented", "fast"])
@pytest.mark.parametrize("general", ["all", "one"])
def test_jobs(policy, one_launch, profile, general):
    """Several scenes of one call, all of them on the general kernels or one
    among scenes with packed records; plain and reordered jobs."""
    jobs, want = [], []
    for i, (n, l, fmt) in enumerate([(8, 8, "fp32"), (4, 16, "q8"), (16, 16, "fp32"), (12, 4, "q8")]):
        scene, batches = _case(n, l, fmt, profile, res=(40 + 8 * i, 30))
        if general == "one" and i != 2:
            scene.set_stack_limit(0)
        for rays, kind, ref in batches:
            for reorder, any_order in ((0, False), (5, True)):
                out = torch.full((rays.shape[0], 4) if kind == "closest" else (rays.shape[0],), 7,
                                 dtype=torch.float32 if kind == "closest" else torch.uint8,
                                 device="cuda")
                jobs.append((scene, dev(rays), kind, out, reorder, any_order))
                want.append(ref)
    pkg.trace_jobs(jobs, profile=profile, policy=policy, one_launch=one_launch)
    torch.cuda.synchronize()
    for (scene, _, kind, out, *rest), ref in zip(jobs, want):
        assert _equal(out, ref), (kind, rest)
        scene.status()


@pytest.mark.parametrize("profile", ["instrumented", "fast"])
def test_host_buffers_and_no_alloc_calls(profile):
    scene, batches = _case(8, 8, "fp32", profile)
    outs = scene.trace_host_batches([(rays, kind, None, {"scheme": "persistent", "policy": 2})
                                     for rays, kind, _ in batches], profile=profile)
    for got, (_, _, want) in zip(outs, batches):
        assert np.array_equal(bits(got) if got.dtype == np.float32 else got,
                              bits(want) if want.dtype == np.float32 else want)
    calls = [(dev(rays), kind, torch.zeros(want.shape, dtype=torch.float32 if kind == "closest"
                                           else torch.uint8, device="cuda"))
             for rays, kind, want in batches]
    for policy in range(4):
        scene.trace_batches_noalloc(calls, profile=profile, policy=policy)
        torch.cuda.synchronize()
        assert all(_equal(c[2], b[2]) for c, b in zip(calls, batches)), policy
    scene.status()


@pytest.mark.parametrize("fmt", ["fp32", "q8"])
def test_imported_trees(fmt):
    """Boxes that are not ordered (FP32) or not nested (Q8), every scheme and
    policy and both job launches; FP32 against the oracle on the same tree, Q8,
    whose boxes are wider, against the counting kernel."""
    tris, bvh, _ = TS.bvh("clutter120", 8, 4)
    arrays = {k: (v.copy() if isinstance(v, np.ndarray) else v)
              for k, v in bvh.export_compact().items()}
    if fmt == "fp32":
        leaf = np.flatnonzero(arrays["child_count"] == 0)[:5]
        arrays["lo3"][leaf, 0] = np.inf
    else:
        inner = np.flatnonzero(arrays["child_count"] > 0)[1::3]
        arrays["hi3"][inner] = arrays["lo3"][inner] + 0.8 * (arrays["hi3"][inner] - arrays["lo3"][inner])
    b = pkg.Bvh.from_compact(arrays, 8, 4)
    scene = pkg.Scene(b, node_format=fmt)
    d = _rays(tris, 20011, 3)
    for profile in ("instrumented", "fast"):
        jobs, want = [], []
        for kind in ("closest", "any"):
            key = "hits" if kind == "closest" else "occluded"
            if fmt == "fp32":
                ref = _oracle(b, O.CompactView(b.export_compact()), d.cpu().numpy(), kind, profile)
            else:
                ref = scene.trace(d, kind=kind, profile=profile, scheme="persistent",
                                  counters=True)[key].cpu().numpy()
            for scheme, kw in SCHEMES:
                if scheme == "stream" and fmt == "q8":
                    continue
                got = scene.trace(d, kind=kind, scheme=scheme, profile=profile, **kw)[key]
                assert _equal(got, ref), (scheme, kw, kind)
            want.append(ref)
            jobs.append((scene, d, kind, torch.full_like(got, 5)))
        for one_launch in (False, True):
            for policy in (0, 2):
                pkg.trace_jobs(jobs, profile=profile, policy=policy, one_launch=one_launch)
                torch.cuda.synchronize()
                assert all(_equal(j[3], w) for j, w in zip(jobs, want)), (one_launch, policy)
    scene.status()
