"""CPU test of the finalize's warp layout (csrc/finalize_shape.h): every number
of keys that a warp takes into its registers as gathered fits its scratch, and
the staged rows fit the same memory."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "similaritysearch.jl_gb300", "csrc")

DRIVER = r"""
#include "finalize_shape.h"
#include <cstdio>
int main() {
    std::printf("%d %d %d\n", 32 * ssg::kWarpKeys, ssg::kWarpStages, ssg::kRowStride);
    for (int need = 1; need <= 64; ++need) std::printf("%d\n", ssg::warp_room(need));
    return 0;
}
"""


def test_warp_room(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    src = tmp_path / "shape.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "shape"
    subprocess.run([gxx, "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = [int(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()]
    held, stages, stride = out[:3]
    for need, room in enumerate(out[3:], 1):
        assert room >= held                                      # gathered keys taken as they stand
        assert 8 * room >= 4 * stages * (need + 1) * stride      # the ring of candidate rows and the query's
        assert (8 * room) % 16 == 0
