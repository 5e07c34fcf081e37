"""Visit histograms (depth_hist, fullness) where the block has room for its
own copy in shared memory and where it has not: equal to the persistent
kernel's, which counts in global memory."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import bvhraytracer_gb300 as pkg  # noqa: E402

pytestmark = pytest.mark.gpu


def _chain(branching, levels, last):
    """Tree of `levels` inner nodes, each with branching - 1 leaves and the
    next inner node, then one inner node with `last` leaves (one triangle per
    leaf): its traversal stack needs 1 + levels * (branching - 1) + last - 1
    entries. Every box is the unit cube; the triangles are small."""
    counts = [branching] * levels + [last]
    lo, hi, cb, cc, pb, pc, tris = [], [], [], [], [], [], []

    def node(begin, count, prim):
        lo.append([0, 0, 0]), hi.append([1, 1, 1])
        cb.append(begin), cc.append(count)
        pb.append(max(prim, 0)), pc.append(0 if prim < 0 else 1)
        return len(cc) - 1

    node(1, counts[0], -1)
    prim = 0
    for i, c in enumerate(counts):
        for j in range(c):
            if i + 1 < len(counts) and j == c - 1:
                node(len(cc) + 1, counts[i + 1], -1)
            else:
                node(0, 0, prim)
                x = 0.9 * (prim + 1) / (sum(counts) + 1)
                tris.append([x, x, 0.5, x + 1e-3, x, 0.5, x, x + 1e-3, 0.5])
                prim += 1
    order = np.tile(np.arange(16, dtype=np.int8), (len(cc), 3))
    return pkg.Bvh.from_compact(
        {"lo3": np.array(lo, np.float32), "hi3": np.array(hi, np.float32),
         "child_begin": cb, "child_count": cc, "prim_begin": pb, "prim_count": pc,
         "order48": order, "prim_ids": np.arange(prim), "prim_tri9": np.array(tris, np.float32)},
        branching, 1)


# Save-distance stacks take cap * 128 * 8 bytes of 227 KiB: at cap 226 the
# histogram's 648 bytes still fit, at 227 they do not.
@pytest.mark.parametrize("last,cap", [(2, 227), (1, 226), (6, 36)])
@pytest.mark.parametrize("n", [1, 127, 128, 1000])
def test_histograms_with_and_without_room(last, cap, n):
    levels = 15 if cap > 36 else 2
    bvh = _chain(16, levels, last)
    assert bvh.info["max_stack"] == cap
    scene = pkg.Scene(bvh)
    rng = np.random.default_rng(n)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3] = rng.uniform(0.2, 0.8, (n, 3))
    rays[:, 2] = 0.6  # away from the triangles: no hit lowers tMax
    rays[:, 3] = 100.0
    rays[:, 4:7] = rng.uniform(0.1, 1.0, (n, 3))
    d = torch.from_numpy(rays).cuda()
    ref = scene.trace(d, scheme="persistent", counters=True, depth_hist=True)
    visits = int(ref["depth_hist"][0].sum())
    assert visits == n * (levels + 1)
    for opts in ({"save_distance": True}, {}):
        got = scene.trace(d, counters=True, depth_hist=True, **opts)
        for k in ("depth_hist", "fullness", "counters"):
            assert torch.equal(got[k], ref[k]), (k, opts)
    scene.status()
