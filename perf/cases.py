"""Workloads of the traversal library as a program that uses it runs them.

Each case is one call, or one frame's calls, through the package's public
entry points: the reference's trace calls in batch form (FastNodeManager,
CompactNodeManager), Scene.trace with the options of the benchmark's plan,
whole frames from device and from host buffers, many scenes at once, and the
differentiable closest hit. Sizes are those of the benchmark's workloads and
of its smaller profiling cases.

A scene is built once and kept, as a renderer keeps it between frames; the
rays of a state (camera, light samples, hemisphere samples) come from the
seed. Primary rays are made here; secondary rays are made from the hits of
the state's primary rays, as a renderer has them in hand.
"""
import math
from functools import lru_cache

import numpy as np
import torch

import bvhraytracer_gb300 as bg
from bvhraytracer_gb300 import diff
from bvhraytracer_gb300 import scenes as gen

FOCAL = 0.866
TMAX = 222222.0
# The benchmark's plan for a frame: primary rays per ray with local stacks,
# shadow rays on the persistent kernel, ambient-occlusion rays on the
# persistent kernel grouped by direction with child-index push order.
PRIMARY = {"scheme": "per_ray", "stack": "local"}
SHADOW = {"scheme": "persistent", "policy": 2, "refill": 16}
AO = {"scheme": "persistent", "policy": 2, "refill": 24, "reorder": 10, "any_order": True}


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # One 16 x 16 workgroup of primary rays: the unit in which the
        # reference's renderer calls its traversal, so latency counts.
        {"name": "workgroup", "kind": "closest_fast", "scene": "terrain", "size": 128,
         "n": 4, "l": 4, "width": 16, "height": 16},
        # Line-of-sight queries between points of a room, an odd number of
        # them, on a wide tree: a game's or a sensor model's visibility call.
        {"name": "visibility", "kind": "visibility", "scene": "clutter", "size": 250,
         "n": 12, "l": 12, "rays": 4099},
        # The terrain workload: 512 x 512 primary rays and a shadow ray per hit.
        {"name": "terrain_frame", "kind": "frame", "scene": "terrain", "size": 128,
         "n": 4, "l": 4, "width": 512, "height": 512, "ao": 0, "plan": "per_ray",
         "format": "fp32"},
        # The instrumented renderer: per-ray counters and per-depth histograms
        # of primary and shadow rays, on the widest tree of the sweep.
        {"name": "statistics", "kind": "statistics", "scene": "clutter", "size": 1000,
         "n": 16, "l": 16, "width": 640, "height": 360},
        # The ray-stream calls of the fast renderer: packets of 256 rays,
        # primary rays and 4 ambient-occlusion rays per hit.
        {"name": "stream_frame", "kind": "manager_frame", "scene": "clutter", "size": 1000,
         "n": 8, "l": 8, "width": 960, "height": 540, "ao": 4, "wide": True},
        # The per-ray calls of the fast renderer at an odd image size.
        {"name": "per_ray_frame", "kind": "manager_frame", "scene": "clutter", "size": 1000,
         "n": 4, "l": 8, "width": 1001, "height": 563, "ao": 8, "wide": False},
        # The benchmark's frame: 1M triangles, full HD, primary, shadow and 8
        # ambient-occlusion rays per hit, rays and results on the device.
        {"name": "tuned_frame", "kind": "frame", "scene": "clutter", "size": 4000,
         "n": 8, "l": 8, "width": 1920, "height": 1080, "ao": 8, "plan": "tuned",
         "format": "fp32"},
        # The same kind of frame on quantised nodes and small leaves, as for
        # scenes whose nodes have to stay small.
        {"name": "quantised_frame", "kind": "frame", "scene": "clutter", "size": 2000,
         "n": 8, "l": 4, "width": 1280, "height": 720, "ao": 8, "plan": "tuned",
         "format": "q8"},
        # A frame rendered on the GPU from the camera to the ambient-occlusion
        # image: ray generation, traces and the per-pixel factor.
        {"name": "rendered_frame", "kind": "rendered", "scene": "clutter", "size": 1000,
         "n": 8, "l": 8, "width": 1280, "height": 720, "ao": 16},
        # A frame from pinned host buffers, results back on the host.
        {"name": "host_frame", "kind": "host", "scene": "clutter", "size": 1000,
         "n": 8, "l": 8, "width": 640, "height": 360, "ao": 8},
        # Twelve scenes of uneven size and ray count in one call.
        {"name": "many_scenes", "kind": "jobs", "scenes": 12, "n": 8, "l": 8, "tris": 200000,
         "rays": 1000000, "spec": 5},
        # Inverse rendering: loss of hit distances, gradients of all vertices
        # and rays.
        {"name": "gradient", "kind": "gradient", "scene": "terrain", "size": 256,
         "n": 8, "l": 8, "width": 1024, "height": 1024},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _any_scene(rng, most=1500):
    if rng.random() < 0.3:
        return {"scene": "terrain", "size": _spread(rng, 24, 256)}
    return {"scene": "clutter", "size": _spread(rng, 60, most)}


def draw(rng):
    kind = rng.choice(["closest_fast", "visibility", "frame", "frame", "statistics",
                       "manager_frame", "manager_frame", "rendered", "host", "jobs", "gradient"])
    c = {"kind": kind}
    width = rng.choice([4, 8, 8, 12, 16])
    leaf = rng.choice([4, 8, 8, 12, 16])
    if kind == "jobs":
        c.update(scenes=rng.randint(2, 12), n=rng.choice([4, 8, 16]), l=rng.choice([4, 8, 16]),
                 tris=_spread(rng, 20000, 150000), rays=_spread(rng, 60000, 800000),
                 spec=rng.randrange(1000))
        return c
    c.update(_any_scene(rng), n=width, l=leaf)
    if kind == "closest_fast":
        side = _spread(rng, 8, 128)
        c.update(width=side, height=_spread(rng, 8, 128))
    elif kind == "visibility":
        c.update(rays=_spread(rng, 200, 400000) | 1)
    elif kind == "gradient":
        c.update(scene="terrain", size=_spread(rng, 32, 256), n=8, l=8,
                 width=_spread(rng, 128, 1000), height=_spread(rng, 128, 1000))
    else:
        w = _spread(rng, 160, 1400)
        c.update(width=w, height=max(90, int(w * rng.uniform(0.5, 0.7))))
        if kind == "statistics":
            c.update(width=min(w, 640), height=min(c["height"], 400))
        elif kind == "manager_frame":
            c.update(ao=rng.randint(1, 8), wide=rng.random() < 0.5)
        elif kind == "frame":
            c.update(ao=rng.choice([0, 1, 4, 8]), plan=rng.choice(["per_ray", "tuned", "tuned"]),
                     format=rng.choice(["fp32", "fp32", "q8"]))
        elif kind == "rendered":
            c.update(ao=rng.randint(2, 16))
        elif kind == "host":
            c.update(width=min(w, 800), height=min(c["height"], 500), ao=rng.randint(1, 8))
    return c


# ------------------------------------------------------- scenes and inputs --
@lru_cache(maxsize=64)
def _tris(scene, size, seed=1):
    return gen.terrain(size, seed) if scene == "terrain" else gen.clutter(size, seed)


@lru_cache(maxsize=64)
def _view(scene, size, seed=1):
    """Camera, target, light and scene diagonal."""
    if scene == "terrain":
        cam, target = np.array([0.5, 0.95, 1.3]), np.array([0.5, 0.0, 0.5])
        light = np.array([2.0, 3.0, 2.0], np.float32)
    else:
        cam, target, light = gen.clutter_viewpoints(size, seed)
    return cam, target, light, gen.scene_diagonal(_tris(scene, size, seed))


@lru_cache(maxsize=64)
def _bvh(scene, size, n, l, seed=1):
    return bg.Bvh(_tris(scene, size, seed), n, l)


@lru_cache(maxsize=64)
def _scene(scene, size, n, l, fmt="fp32", seed=1):
    return bg.Scene(_bvh(scene, size, n, l, seed), node_format=fmt)


@lru_cache(maxsize=64)
def _fast_manager(scene, size, n, l):
    return bg.FastNodeManager(_bvh(scene, size, n, l))


@lru_cache(maxsize=64)
def _compact_manager(scene, size, n, l):
    return bg.CompactNodeManager(_bvh(scene, size, n, l))


def _camera(case, seed):
    """Camera position and target of a state: the scene's view point, moved
    a little and turned."""
    cam, target, light, diag = _view(case["scene"], case["size"])
    rng = np.random.default_rng([seed, 17])
    cam = cam + rng.uniform(-0.004, 0.004, 3) * diag
    target = target + rng.uniform(-0.06, 0.06, 3) * diag
    light = (light + rng.uniform(-0.01, 0.01, 3) * diag).astype(np.float32)
    return cam, target, light, 0.1 * diag


def _pinhole(cam, target, width, height, tile=16):
    """Pinhole primary rays, tile by tile (workgroups of 16 x 16 pixels):
    [width * height, 8] float32 on the GPU; direction not normalised."""
    f = np.asarray(target, np.float64) - cam
    f /= np.linalg.norm(f)
    r = np.cross(f, [0.0, 1.0, 0.0])
    r /= np.linalg.norm(r)
    u = np.cross(r, f)
    dev = torch.device("cuda")
    rows = torch.arange(height, device=dev)[:, None].expand(height, width)
    cols = torch.arange(width, device=dev)[None, :].expand(height, width)
    tiles = -(-width // tile)
    key = ((rows // tile) * tiles + cols // tile) * tile * tile + (rows % tile) * tile + cols % tile
    order = torch.argsort(key.reshape(-1))
    w = (cols - width // 2).reshape(-1)[order].double() / width
    h = -(rows - height // 2).reshape(-1)[order].double() / width
    d = (torch.from_numpy(r).to(dev) * w[:, None] + torch.from_numpy(u).to(dev) * h[:, None]
         + torch.from_numpy(f * FOCAL).to(dev))
    rays = torch.zeros((width * height, 8), dtype=torch.float32, device=dev)
    rays[:, 0:3] = torch.from_numpy(np.asarray(cam, np.float32)).to(dev)
    rays[:, 3] = TMAX
    rays[:, 4:7] = d.float()
    return rays


def _primary(case, seed):
    cam, target, _, _ = _camera(case, seed)
    return _pinhole(cam, target, case["width"], case["height"])


def _secondaries(case, seed, scene, rays):
    """Shadow and ambient-occlusion rays of a state's primary hits, on the
    device (pixels that hit nothing have inactive rays: NaN origin)."""
    _, _, light, length = _camera(case, seed)
    hits = scene.trace(rays, **PRIMARY)["hits"]
    return scene.secondary_rays(rays, hits, light=light, ao_samples=case.get("ao", 0),
                                ao_length=length, seed=seed)


def _segments(case, seed):
    """Rays between random points of the scene's box; tMax ends them at the
    second point (direction not normalised, tMax 1)."""
    tris = _tris(case["scene"], case["size"]).reshape(-1, 3)
    lo, hi = tris.min(0), tris.max(0)
    rng = np.random.default_rng([seed, 23])
    a = rng.uniform(lo, hi, (case["rays"], 3))
    b = rng.uniform(lo, hi, (case["rays"], 3))
    rays = np.zeros((case["rays"], 8), np.float32)
    rays[:, 0:3], rays[:, 4:7] = a, b - a
    rays[:, 3] = 1.0
    return torch.from_numpy(rays).cuda()


def _job_specs(case):
    """(scene, size, width, height) of each scene of a batch: triangles and
    rays log-uniform, terrain and clutter in turn."""
    rng = np.random.default_rng(case["spec"])
    specs = []
    for i in range(case["scenes"]):
        tris = math.exp(rng.uniform(math.log(1000), math.log(case["tris"])))
        pixels = math.exp(rng.uniform(math.log(4000), math.log(case["rays"]))) / 6
        width = max(8, int(math.sqrt(pixels * 16 / 9)))
        height = max(8, int(pixels / width))
        if i % 2:
            specs.append(("clutter", max(2, round(tris / 250)), width, height))
        else:
            specs.append(("terrain", max(8, round(math.sqrt(tris / 2))), width, height))
    return specs


@lru_cache(maxsize=8)
def _mesh(size):
    """Terrain vertices, faces and the scene of the mesh, on the GPU."""
    verts, faces = gen.terrain_mesh(size, seed=0)
    v = torch.from_numpy(verts).cuda()
    f = torch.from_numpy(faces.astype(np.int32)).cuda()
    return v, f, diff.scene_for(v, f)


def _gradient_inputs(case, seed):
    """Rays and target distances of a fit: the targets are the distances to
    the terrain plane moved by noise."""
    rays = _primary(case, seed)
    g = torch.Generator().manual_seed(seed)
    noise = (0.02 * torch.randn(rays.shape[0], generator=g)).cuda()
    t = -rays[:, 1].double() / torch.where(rays[:, 5] < -1e-3, rays[:, 5],
                                           torch.full_like(rays[:, 5], -1e-3)).double()
    return rays, (t.clamp(0.0, 10.0).float() + noise)


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "jobs":
        jobs, total, hits_n, occ_n = [], [], 0, 0
        for i, (scene, size, w, h) in enumerate(_job_specs(case)):
            sub = {"scene": scene, "size": size, "width": w, "height": h, "ao": 4}
            sc = _scene(scene, size, case["n"], case["l"])
            rays = _primary(sub, seed * 131 + i)
            shadow, ao = _secondaries(sub, seed * 131 + i, sc, rays)
            for r, k, o in ((rays, "closest", ()), (shadow, "any", ()), (ao, "any", (10, True))):
                total.append((sc, r, k, o))
        hits = torch.empty((sum(r.shape[0] for _, r, k, _ in total if k == "closest"), 4),
                           dtype=torch.float32, device="cuda")
        occ = torch.empty(sum(r.shape[0] for _, r, k, _ in total if k == "any"),
                          dtype=torch.uint8, device="cuda")
        for sc, r, k, o in total:
            m = r.shape[0]
            if k == "closest":
                out, hits_n = hits[hits_n:hits_n + m], hits_n + m
            else:
                out, occ_n = occ[occ_n:occ_n + m], occ_n + m
            jobs.append((sc, r, k, out) + o)
        st.update(jobs=jobs, hits=hits, occ=occ)
        return st
    key = (case["scene"], case["size"], case["n"], case["l"])
    if kind == "closest_fast":
        st.update(manager=_fast_manager(*key), rays=_primary(case, seed))
    elif kind == "visibility":
        st.update(manager=_fast_manager(*key), rays=_segments(case, seed))
    elif kind == "statistics":
        m = _compact_manager(*key)
        rays = _primary(case, seed)
        st.update(manager=m, rays=rays, shadow=_secondaries(case, seed, m.scene, rays)[0])
    elif kind == "manager_frame":
        m = _fast_manager(*key)
        rays = _primary(case, seed)
        st.update(manager=m, rays=rays, ao=_secondaries(case, seed, m.scene, rays)[1])
    elif kind in ("frame", "host"):
        sc = _scene(*key, fmt=case.get("format", "fp32"))
        rays = _primary(case, seed)
        shadow, ao = _secondaries(case, seed, sc, rays)
        st.update(scene=sc)
        if kind == "frame":
            st.update(rays=rays, shadow=shadow, ao=ao)
        else:
            # pinned host buffers for the rays and the results
            batches = []
            for r, k, o in ((rays, "closest", PRIMARY), (shadow, "any", SHADOW), (ao, "any", AO)):
                h = torch.empty(r.shape, dtype=torch.float32).pin_memory()
                h.copy_(r)
                out = (torch.empty((r.shape[0], 4), dtype=torch.float32) if k == "closest"
                       else torch.empty(r.shape[0], dtype=torch.uint8)).pin_memory()
                batches.append((h.numpy(), k, out.numpy(), o))
                st.setdefault("keep", []).extend([h, out])
            st.update(batches=batches)
    elif kind == "rendered":
        cam, target, light, length = _camera(case, seed)
        st.update(scene=_scene(*key), cam=cam, target=target, light=light, length=length,
                  seed=seed)
    elif kind == "gradient":
        v, f, sc = _mesh(case["size"])
        rays, goal = _gradient_inputs(case, seed)
        st.update(scene=sc, verts=v.clone().requires_grad_(True), faces=f,
                  rays=rays.requires_grad_(True), goal=goal)
    return st


# -------------------------------------------------------------------- run --
def _hits(h):
    return {"prim": bg.hit_prims(h), "tuv": h[:, 1:4]}


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "closest_fast":
        return _hits(state["manager"].intersect(state["rays"]))
    if kind == "visibility":
        return state["manager"].intersect_secondary(state["rays"])
    if kind == "statistics":
        m, out = state["manager"], {}
        for name, rays, shadow in (("primary", state["rays"], False),
                                   ("shadow", state["shadow"], True)):
            r = m.intersect_immediately(rays, shadow=shadow)
            res = {"occluded": r["occluded"]} if shadow else _hits(r["hits"])
            out[name] = dict(res, counters=r["counters"], depth=r["depth_hist"],
                             fullness=r["fullness"])
        return out
    if kind == "manager_frame":
        m = state["manager"]
        if case["wide"]:
            return dict(_hits(m.intersect_wide_alternative(state["rays"])),
                        ao=m.intersect_secondary_wide_alternative(state["ao"]))
        return dict(_hits(m.intersect(state["rays"])), ao=m.intersect_secondary(state["ao"]))
    if kind == "frame":
        sc = state["scene"]
        tuned = case["plan"] == "tuned"
        out = _hits(sc.trace(state["rays"], **PRIMARY)["hits"])
        out["shadow"] = sc.trace(state["shadow"], kind="any",
                                 **(SHADOW if tuned else PRIMARY))["occluded"]
        if case["ao"]:
            out["ao"] = sc.trace(state["ao"], kind="any", **(AO if tuned else PRIMARY))["occluded"]
        return out
    if kind == "host":
        h, s, a = state["scene"].trace_host_batches(state["batches"])
        return dict(_hits(h), shadow=s, ao=a)
    if kind == "rendered":
        sc, spp = state["scene"], case["ao"]
        rays = bg.camera_rays(state["cam"], state["target"], case["width"], case["height"])
        hits = sc.trace(rays, **PRIMARY)["hits"]
        shadow, ao = sc.secondary_rays(rays, hits, light=state["light"], ao_samples=spp,
                                       ao_length=state["length"], seed=state["seed"])
        lit = sc.trace(shadow, kind="any", **SHADOW)["occluded"]
        occ = sc.trace(ao, kind="any", **AO)["occluded"]
        return dict(_hits(hits), shadow=lit, ao=occ, factor=bg.ao_factor(occ, spp))
    if kind == "jobs":
        bg.trace_jobs(state["jobs"], policy=2, refill=16)
        return dict(_hits(state["hits"]), occluded=state["occ"])
    t, u, v, prim = diff.ray_hit(state["verts"], state["faces"], state["rays"], state["scene"])
    loss = torch.where(prim >= 0, (t - state["goal"]) ** 2, torch.zeros_like(t)).sum()
    grad_verts, grad_rays = torch.autograd.grad(loss, (state["verts"], state["rays"]))
    return {"t": t.detach(), "u": u.detach(), "v": v.detach(), "prim": prim,
            "verts": grad_verts, "rays": grad_rays}


# ------------------------------------------------------------------- work --
def _triangles(scene, size):
    return 2 * size * size if scene == "terrain" else 768 + 250 * size


def _trace_work(tris, n, l, closest, anyhit):
    """Rays read and results written once, the scene's triangles (36 bytes)
    and one box per leaf (24 bytes) read once; a ray tests at least the boxes
    of one path down the tree (18 operations each) and one triangle (60)."""
    rays = closest + anyhit
    depth = max(1.0, math.log(max(2.0, tris / l)) / math.log(n))
    return (32 * rays + 16 * closest + anyhit + tris * (36 + 24 / l),
            rays * (18.0 * n * depth + 60.0))


def work(case):
    kind = case["kind"]
    if kind == "jobs":
        b = f = 0.0
        for scene, size, w, h in _job_specs(case):
            x, y = _trace_work(_triangles(scene, size), case["n"], case["l"], w * h, 5 * w * h)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    tris = _triangles(case["scene"], case["size"])
    pixels = case["rays"] if kind == "visibility" else case["width"] * case["height"]
    n, l = case["n"], case["l"]
    if kind == "closest_fast":
        b, f = _trace_work(tris, n, l, pixels, 0)
    elif kind == "visibility":
        b, f = _trace_work(tris, n, l, 0, pixels)
    elif kind == "statistics":
        b, f = _trace_work(tris, n, l, pixels, pixels)
        b += 2 * pixels * 32  # the per-ray counters
    elif kind == "manager_frame":
        b, f = _trace_work(tris, n, l, pixels, pixels * case["ao"])
    elif kind == "gradient":
        # hits kept for the backward pass, gradients of hits, rays and
        # vertices; about 300 operations of the reverse pass per ray
        b, f = _trace_work(tris, n, l, pixels, 0)
        b += pixels * (32 + 16 + 12 + 32) + 12 * (case["size"] + 1) ** 2
        f += 300.0 * pixels
    else:
        b, f = _trace_work(tris, n, l, pixels, pixels * (1 + case["ao"]))
        if kind == "rendered":
            # rays written as well as read, the occlusion bytes read again
            b += pixels * (32 * (2 + case["ao"]) + case["ao"] + 4)
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------ exact --
def _group_boxes(lo, hi, size):
    """Boxes of consecutive groups of `size` boxes."""
    pad = -lo.shape[0] % size
    if pad:
        lo = torch.cat([lo, torch.full((pad, 3), math.inf, dtype=lo.dtype, device=lo.device)])
        hi = torch.cat([hi, torch.full((pad, 3), -math.inf, dtype=hi.dtype, device=hi.device)])
    return lo.view(-1, size, 3).amin(1), hi.view(-1, size, 3).amax(1)


def _meets(o, inv, lo, hi, slack):
    a, b = (lo - slack - o) * inv, (hi + slack - o) * inv
    near = torch.minimum(a, b).amax(-1)
    far = torch.maximum(a, b).amin(-1)
    return (near <= far) & (far >= 0)


def _closest(tris, rays, unit, chunk=16384):
    """(triangle, t, b1, b2) of the closest hit of each ray in 64 bits, in
    plain torch: Moller-Trumbore over the triangles whose groups' boxes the
    ray meets (groups of 64 and of 1,024 consecutive triangles). Misses keep
    tMax and triangle -1."""
    dev = rays.device
    p = torch.from_numpy(tris.reshape(-1, 3, 3)).to(dev).double()
    n = p.shape[0]
    lo1, hi1 = _group_boxes(p.amin(1), p.amax(1), 64)
    lo2, hi2 = _group_boxes(lo1, hi1, 16)
    slack = 1e-9 * float((p.amax() - p.amin()).abs())
    tri = torch.full((rays.shape[0],), -1, dtype=torch.int64, device=dev)
    t = rays[:, 3].double().clone()
    b1, b2 = torch.zeros_like(t), torch.zeros_like(t)
    for first in range(0, rays.shape[0], chunk):
        o = rays[first:first + chunk, 0:3].double()
        d = rays[first:first + chunk, 4:7].double()
        if unit:
            d = d / d.norm(dim=1, keepdim=True)
        inv = 1.0 / torch.where(d == 0, torch.full_like(d, 1e-300), d)
        r, g = _meets(o[:, None], inv[:, None], lo2, hi2, slack).nonzero(as_tuple=True)
        g = (g[:, None] * 16 + torch.arange(16, device=dev)).reshape(-1)
        r = r.repeat_interleave(16)
        ok = g < lo1.shape[0]
        r, g = r[ok], g[ok]
        ok = _meets(o[r], inv[r], lo1[g], hi1[g], slack)
        r, g = r[ok], g[ok]
        k = (g[:, None] * 64 + torch.arange(64, device=dev)).reshape(-1)
        r = r.repeat_interleave(64)
        ok = k < n
        r, k = r[ok], k[ok]
        q = p[k]
        e1, e2, dd = q[:, 1] - q[:, 0], q[:, 2] - q[:, 0], d[r]
        s1 = torch.linalg.cross(dd, e2)
        div = (s1 * e1).sum(1)
        s = o[r] - q[:, 0]
        u = (s * s1).sum(1) / div
        s2 = torch.linalg.cross(s, e1)
        v = (dd * s2).sum(1) / div
        tt = (e2 * s2).sum(1) / div
        ok = (div != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (tt > 0) & \
            (tt <= rays[first + r, 3].double())
        r, k, u, v, tt = r[ok], k[ok], u[ok], v[ok], tt[ok]
        best = torch.full((o.shape[0],), math.inf, dtype=torch.float64, device=dev)
        best.scatter_reduce_(0, r, tt, "amin")
        win = tt == best[r]
        r, k, u, v, tt = r[win], k[win], u[win], v[win], tt[win]
        tri[first + r], t[first + r], b1[first + r], b2[first + r] = k, tt, u, v
    return tri, t, b1, b2


def exact(case, seed):
    kind = case["kind"]
    if kind in ("visibility", "jobs"):
        return None  # flags only; too many scenes
    if kind == "gradient":
        rays, goal = _gradient_inputs(case, seed)
        verts, faces = gen.terrain_mesh(case["size"], seed=0)
        tris = verts[faces].reshape(-1, 9)
        tri, t, _, _ = _closest(tris, rays, unit=False)
        v = torch.from_numpy(verts).cuda().double().requires_grad_(True)
        r = rays.double().requires_grad_(True)
        hit = (tri >= 0).nonzero().reshape(-1)
        q = v[torch.from_numpy(faces).cuda()[tri[hit]]]
        o, d = r[hit, 0:3], r[hit, 4:7]
        e1, e2, s = q[:, 1] - q[:, 0], q[:, 2] - q[:, 0], o - q[:, 0]
        s1, s2 = torch.linalg.cross(d, e2), torch.linalg.cross(s, e1)
        div = (s1 * e1).sum(1)
        t_hit = (e2 * s2).sum(1) / div
        gv, gr = torch.autograd.grad(((t_hit - goal.double()[hit]) ** 2).sum(), (v, r))
        u_out, v_out = torch.zeros_like(t), torch.zeros_like(t)
        u_out[hit] = ((s * s1).sum(1) / div).detach()
        v_out[hit] = ((d * s2).sum(1) / div).detach()
        return {"t": t, "u": u_out, "v": v_out, "prim": None, "verts": gv, "rays": gr}
    rays = _primary(case, seed)
    fast = kind in ("closest_fast", "manager_frame")
    _, t, u, v = _closest(_tris(case["scene"], case["size"]), rays, unit=not fast)
    out = {"prim": None, "tuv": torch.stack([t, u, v], 1)}
    if kind == "statistics":
        return {"primary": dict(out, counters=None, depth=None, fullness=None), "shadow": None}
    if kind == "rendered":
        out["factor"] = None
    return out
