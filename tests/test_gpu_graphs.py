"""Traces recorded into CUDA graphs: large batches of the persistent scheme have
the choice between the packed scene's kernels there too, without memory nodes
in the graph."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")

import bvhraytracer_gb300 as pkg  # noqa: E402
from bvhraytracer_gb300 import scenes as S  # noqa: E402
from tests.test_gpu_pool import LINE, _rays  # noqa: E402

pytestmark = pytest.mark.gpu


def _record(work):
    """(nodes of the graph that `work(stream)` records, the graph)"""
    rt = C.CDLL("libcudart.so.13")
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    torch.cuda.synchronize()
    st, graph, n = C.c_void_p(side.cuda_stream), C.c_void_p(), C.c_size_t()
    assert rt.cudaStreamBeginCapture(st, 2) == 0  # relaxed
    with torch.cuda.stream(side):
        work()
    assert rt.cudaStreamEndCapture(st, C.byref(graph)) == 0
    assert rt.cudaGraphGetNodes(graph, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert rt.cudaGraphGetNodes(graph, nodes, C.byref(n)) == 0
    kinds = []
    for node in nodes:
        kind = C.c_int()
        assert rt.cudaGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        kinds.append(kind.value)
    assert rt.cudaGraphDestroy(graph) == 0
    return kinds


KERNEL = 0  # cudaGraphNodeTypeKernel


@pytest.mark.parametrize("kind", ["closest", "any"])
def test_recorded_kernels(kind):
    """The plan and the two kernels it chooses from, for the persistent scheme
    and for jobs; one thread per ray, in one kernel, for the others."""
    tris = S.clutter(30, 2)
    scene = pkg.Scene(pkg.Bvh(tris, 8, 8))
    rays = _rays(tris, LINE + 5, 1)
    out = scene.trace(rays, kind=kind)["hits" if kind == "closest" else "occluded"]
    assert _record(lambda: scene.trace(rays, kind=kind, scheme="persistent", out=out)) == [KERNEL] * 3
    assert _record(lambda: pkg.trace_jobs([(scene, rays, kind, out)])) == [KERNEL] * 3
    assert _record(lambda: scene.trace(rays, kind=kind, out=out)) == [KERNEL]
    small = rays[:LINE]
    assert _record(lambda: scene.trace(small, kind=kind, scheme="persistent",
                                       out=out[:LINE])) == [KERNEL]


@pytest.mark.parametrize("n,l,fmt", [(8, 8, "fp32"), (4, 4, "q8"), (16, 8, "fp32")])
def test_graphs_of_one_scene_replayed_together(n, l, fmt):
    """Every recorded launch has its own words: graphs of one scene run at the
    same time on different streams, with plain launches among them."""
    tris = S.clutter(40, 3)
    scene = pkg.Scene(pkg.Bvh(tris, n, l), node_format=fmt)
    scattered = _rays(tris, LINE + 9000, n)
    cam, target, _ = S.clutter_viewpoints(40, 3)
    together = pkg.camera_rays(cam, target, 768, 512)
    runs = []
    for rays in (scattered, together, scattered[3000:]):
        for kind in ("closest", "any"):
            key = "hits" if kind == "closest" else "occluded"
            want = scene.trace(rays, kind=kind, scheme="persistent", counters=True)[key]
            out, side, graph = torch.full_like(want, 5), torch.cuda.Stream(), torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            with torch.cuda.graph(graph, stream=side):
                if rays is together:
                    pkg.trace_jobs([(scene, rays, kind, out)])
                else:
                    scene.trace(rays, kind=kind, scheme="persistent", policy=2, out=out)
            runs.append((graph, side, out, want, rays, kind))
    for _ in range(3):
        plain = []
        for graph, _, out, *_ in runs:
            out.fill_(5)
        torch.cuda.synchronize()
        for graph, side, _, want, rays, kind in runs:
            with torch.cuda.stream(side):
                graph.replay()
            key = "hits" if kind == "closest" else "occluded"
            plain.append((scene.trace(rays, kind=kind)[key], want))
        torch.cuda.synchronize()
        for got, want in plain + [r[2:4] for r in runs]:
            assert torch.equal(got.view(torch.uint8), want.view(torch.uint8))
    scene.status()
