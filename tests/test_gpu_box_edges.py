"""Rays aimed at the faces, edges and corners of the boxes and at the triangles'
vertices, with tMax at, just below and just above the target: where the Q8
planes that are moved outward, and the children dropped behind tMax, could
change a result."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import bvhraytracer_gb300 as pkg  # noqa: E402
from bvhraytracer_gb300 import scenes as S  # noqa: E402
from tests.test_gpu_pool import LINE, _same  # noqa: E402

pytestmark = pytest.mark.gpu


def _aimed(tris, arrays, n, seed):
    rng = np.random.default_rng(seed)
    p = tris.reshape(-1, 3)
    lo, hi = p.min(0), p.max(0)
    box = rng.integers(1, len(arrays["lo3"]), n)
    blo = np.asarray(arrays["lo3"], np.float32).reshape(-1, 3)[box]
    bhi = np.asarray(arrays["hi3"], np.float32).reshape(-1, 3)[box]
    # per axis the low plane, the high plane or a point between: 3 planes a
    # corner, 2 an edge, 1 a face
    pick = rng.integers(0, 3, (n, 3))
    between = blo + (bhi - blo) * rng.random((n, 3), dtype=np.float32)
    target = np.where(pick == 0, blo, np.where(pick == 1, bhi, between)).astype(np.float32)
    vertex = rng.random(n) < 0.25
    target[vertex] = p[rng.integers(0, len(p), n)][vertex]
    origin = rng.uniform(lo - 1, hi + 1, (n, 3)).astype(np.float32)
    # a third run along one axis or in one plane of the target
    for a in range(3):
        same = rng.random(n) < 0.25
        origin[same, a] = target[same, a]
    d = target - origin
    length = np.linalg.norm(d.astype(np.float64), axis=1).astype(np.float32)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3], r[:, 4:7] = origin, d
    up, down = np.nextafter(length, np.float32(np.inf)), np.nextafter(length, np.float32(0))
    r[:, 3] = np.choose(rng.integers(0, 4, n), [length, up, down, np.full(n, 1e4, np.float32)])
    unit = rng.random(n) < 0.5  # the fast profile takes directions as they are
    r[unit, 4:7] = d[unit] / np.maximum(length[unit], 1e-30)[:, None]
    return torch.from_numpy(r).cuda()


@pytest.mark.parametrize("n,l", [(4, 4), (8, 8), (8, 1), (12, 12), (16, 4)])
@pytest.mark.parametrize("fmt", ["fp32", "q8"])
def test_rays_through_the_edges_of_boxes(n, l, fmt):
    tris = S.clutter(30, 2)
    bvh = pkg.Bvh(tris, n, l)
    rays = _aimed(tris, bvh.export_compact(), LINE + 321, 7 * n + l)
    scene = pkg.Scene(bvh, node_format=fmt)
    for k in (3000, 40000, 140001, LINE + 321):  # teams, one wave, one thread per ray, the pool
        _same(scene, rays[:k])
    _same(scene, rays, reorder=3)
