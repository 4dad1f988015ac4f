"""How the search for a beamlet's source samples is split: a warp that walks 32
units of depth takes a few dozen steps whatever the beamlet's width, and stays
whole where the launch is large and the beamlets small.  Host code, built here.
"""
import os
import subprocess

from endtoend_gb300 import _build

SOURCE = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include "ee_internal.h"

int main() {
    int bad = 0;
    for (double side : {3.0, 4.0, 6.0, 18.0, 42.0, 130.0})  // cells, with the margin of a cell each way
        for (long long warps : {1ll, 72ll, 2432ll, 30000ll, 1000000ll}) {
            const int n = ee_bl_source_slices(side * side, warps);
            const double steps = 3 * side * side / n;
            if (n < 1 || n > 4096 || steps > 129) bad++, std::printf("%g %lld %d\n", side, warps, n);
            if (n > 1 && steps < 8) bad++;
        }
    if (ee_bl_source_slices(9.0, 30000) != 1 || ee_bl_source_slices(16.0, 30000) != 1) bad++;
    return bad;
}
"""


def test_steps_per_warp(tmp_path):
    src, exe = tmp_path / "slices.cpp", str(tmp_path / "slices")
    src.write_text(SOURCE)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc_path()))), "include")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-w", "-I", cuda, "-I", _build.CSRC, str(src), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
