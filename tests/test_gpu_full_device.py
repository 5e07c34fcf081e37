"""A large trace on a device without room for its queue words: every ray has a
thread of its own, the call succeeds, and the last error is what it was."""
import subprocess
import sys
from pathlib import Path

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

CODE = """
import ctypes as C
import torch
import bvhraytracer_gb300 as pkg
from bvhraytracer_gb300 import _native as N
from bvhraytracer_gb300 import scenes as S
from tests.test_gpu_pool import LINE, _rays
tris = S.clutter(30, 2)
scene = pkg.Scene(pkg.Bvh(tris, 8, 8))
rays = _rays(tris, LINE + 1000, 1)
want, out = {}, {}
for kind in ("closest", "any"):
    key = "hits" if kind == "closest" else "occluded"
    want[kind] = scene.trace(rays, kind=kind, scheme="persistent", counters=True)[key]
    out[kind] = torch.full_like(want[kind], 5)
    scene.trace(rays[:LINE], kind=kind, out=out[kind][:LINE])  # loads the kernel
    out[kind].fill_(5)
torch.cuda.synchronize()
before = N.lib().bvhgpu_last_error()
# The rest of the device's memory, in pieces down to the driver's smallest.
rt = C.CDLL("libcudart.so.13")
held, size = [], 1 << 36
while size >= 1 << 12:
    p = C.c_void_p()
    if rt.cudaMalloc(C.byref(p), C.c_size_t(size)) == 0:
        held.append(p)
    else:
        rt.cudaGetLastError()
        size >>= 1
for kind in ("closest", "any"):
    scene.trace(rays, kind=kind, out=out[kind])
after = N.lib().bvhgpu_last_error()
rt.cudaDeviceSynchronize()
for p in held:
    rt.cudaFree(p)
torch.cuda.synchronize()
assert held and all(torch.equal(out[k].view(torch.uint8), want[k].view(torch.uint8)) for k in out)
assert after == before, after
scene.status()
print("ok")
"""


def test_trace_without_room_for_queue_words():
    """In a process of its own, whose scratch pool is still empty."""
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0 and r.stdout.split()[-1:] == ["ok"], r.stdout + r.stderr[-2000:]
