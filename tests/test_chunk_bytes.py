"""A chunk's bytes hold its tile lists with its arrays: each list has room for the
tiles of the chunk's largest cone, so one wide beam among many narrow ones makes
all of theirs large.  Host code, built here.
"""
import os
import re
import subprocess

from endtoend_gb300 import _build

SOURCE = r"""
#include <cuda_runtime.h>
#include "ee_internal.h"

int main() {
    int bad = 0;
    for (long long rev : {0ll, 64ll, 1ll << 31})
        for (long long quads : {0ll, 1ll << 29})
            for (long long lists : {0ll, 48ll, 48ll * 32768})
                for (int lines : {32, 1000, 200 * 200}) {
                    const long long cap = ee_cone_tiles_cap(lines);
                    const long long want = 4 * rev + (long long)sizeof(float4) * quads + lists * (long long)sizeof(int) +
                                           lists * cap * (long long)(sizeof(int) + sizeof(unsigned char));
                    if (ee_chunk_bytes(rev, quads, lists, lines) != want) bad++;
                }
    return bad;
}
"""


def test_lists_are_counted(tmp_path):
    src, exe = tmp_path / "bytes.cpp", str(tmp_path / "bytes")
    src.write_text(SOURCE)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc_path()))), "include")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-w", "-I", cuda, "-I", _build.CSRC, str(src), "-o", exe])
    assert subprocess.run([exe]).returncode == 0
    # the direct call and the plan both decide by it
    api = open(os.path.join(_build.CSRC, "ee_api.cpp")).read()
    assert len(re.findall(r"bytes_with\([^;{]*\) >\s*c->max_batch_bytes / 4 \* 3", api)) == 2
