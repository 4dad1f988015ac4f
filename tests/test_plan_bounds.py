"""A planned beam whose sizes exceed any bound of its plan is refused: the tile
lists, the cones' scratch and the shared arrays are indexed by the sizes that
the device finds, so each bound is compared there, not the arena's alone.  The
comparison is host code too and is built here.
"""
import os
import subprocess

from endtoend_gb300 import _build

SOURCE = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstring>
#include "ee_internal.h"

int main() {
    EeBeamSpec S;
    std::memset(&S, 0, sizeof(S));
    int bad = 0;
    auto expect = [&](bool holds, long long store, int lines, int line) {
        if (ee_plan_holds(S, store, lines, line) != holds) bad++, std::printf("%lld %d %d\n", store, lines, line);
    };
    expect(true, 1ll << 40, 1 << 30, 1024);  // not planned: sized after the read-back
    S.plan_cap = 6400;
    S.plan_lines = 320;
    S.plan_line = 100;
    expect(true, 6400, 320, 100);
    expect(false, 6401, 320, 100);
    expect(false, 6400, 352, 100);
    expect(false, 64, 352, 4);
    expect(false, 6400, 320, 101);
    // a cone of max_lines slots in tiles of 8 x 4 lines fits its list
    for (int n1 = 1; n1 < 70; n1++)
        for (int n2 = 1; n2 < 70; n2++) {
            const int tiles = ((n1 + 7) >> 3) * ((n2 + 3) >> 2), slots = ((n1 + 7) >> 3) * 8 * (((n2 + 3) >> 2) * 4);
            if (tiles > ee_cone_tiles_cap(slots)) bad++;
        }
    return bad;
}
"""


def test_every_bound_is_compared(tmp_path):
    src, exe = tmp_path / "bounds.cpp", str(tmp_path / "bounds")
    src.write_text(SOURCE)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc_path()))), "include")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-w", "-I", cuda, "-I", _build.CSRC, str(src), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    kernels = open(os.path.join(_build.CSRC, "ee_kernels.cu")).read()
    assert "ee_plan_holds(S, off, mls, ml)" in kernels
