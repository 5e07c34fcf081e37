"""Width of the per-block visit histograms: 32-bit words only for trees whose
nodes and leaves, times the rays of a block, they can count (host C++)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "bvhraytracer_gb300" / "csrc"


@pytest.mark.parametrize("inner,leaves,rays,fits", [
    (1, 1, 256, 1), ((1 << 24) - 1, 5, 256, 1), (1 << 24, 5, 256, 0), (5, (1 << 24) - 1, 256, 1),
    (5, 1 << 24, 256, 0), (1 << 26, 1 << 27, 256, 0), (0, (1 << 25) - 1, 128, 1), (0, 1 << 25, 128, 0)])
def test_words_hold_every_visit_of_a_block(tmp_path, inner, leaves, rays, fits):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "fit.cpp"
    src.write_text('#include "bvh_export.hpp"\n#include <cstdio>\n'
                   "int main() { bvhgpu::DeviceLayout L;\n"
                   f"L.n_inner = {inner}u; L.n_leaves = {leaves}u;\n"
                   f'std::printf("%d", (int)L.visits_fit_32({rays})); }}\n')
    exe = tmp_path / "fit"
    subprocess.run([cxx, "-std=c++17", f"-I{CSRC}", f"-I{CSRC.parents[1] / 'include'}", str(src),
                    "-o", str(exe)], check=True)
    got = int(subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout)
    assert got == fits == int(max(inner, leaves) * rays < 1 << 32)
