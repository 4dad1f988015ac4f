"""The resident warps that a scratch limit leaves the lane cones: a quarter of
the limit, or as much as the arena of a beam that exceeds the limit by itself
(it is taken whatever the limit, and its cones need their warps).  Host code,
built here.
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
    for (int line : {1, 40, 100, 400, 1024})
        for (long long limit : {1ll << 20, 1ll << 24, 1ll << 26, 1ll << 28, 1ll << 30, 8ll << 30})
            for (long long arena : {1ll << 18, 1ll << 24, 1ll << 27, 1ll << 29}) {
                const int warps = ee_cone_warps(line, limit, arena);
                const long long bytes = 1024ll * ee_cone_quads(line) * warps;
                const bool over = arena > limit / 4 * 3;
                const long long room = over ? arena : limit / 4;
                // a warp per SM at least; else within the room, and half of it used or the chip full
                if (warps < 152 || warps > EE_CONE_MAX_WARPS || warps % EE_CONE_BLOCK_WARPS) bad++;
                if (warps > 152 && bytes > room) bad++;
                if (warps < EE_CONE_MAX_WARPS && 2 * bytes < room) bad++;
            }
    return bad;
}
"""


def test_warps_of_a_limit(tmp_path):
    src, exe = tmp_path / "limit.cpp", str(tmp_path / "limit")
    src.write_text(SOURCE)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc_path()))), "include")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-w", "-I", cuda, "-I", _build.CSRC, str(src), "-o", exe])
    assert subprocess.run([exe]).returncode == 0
