"""The samples that one kernel clears for another to read: k_rev_zero zeroes the
part of each line's gradient that the adjoint cones read, and both kernels work
that part out from the line's geometry.  A compiler may contract the products
and sums of one kernel and not those of the other, so the header that holds this
arithmetic is built here for the host with contraction on and off: what one
build clears has to cover what the other reads, on lines whose ends lie on the
faces of the crop box or the calc bbox, where the last bit decides.
"""
import ctypes as C
import os
import platform
import subprocess

import numpy as np
import pytest

from endtoend_gb300 import _build

SOURCE = r"""
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <cstring>
using std::max;
using std::min;
static inline float __fdividef(float a, float b) { return a / b; }
#include "ee_lines.cuh"

// line: B0 Bx By Bz G0 Gx Gy Gz (3 each), tY, tZ; box: bev, bb0, bbs (3 each);
// out: segment, read span, quads of the field, cleared span
extern "C" void spans(const float* lines, const int* box, int n, int L, int* out) {
    static EeParams P;
    static EeBeamSpec S;
    static EeBeamGeom G;
    for (int i = 0; i < n; i++) {
        const float* f = lines + 26 * i;
        std::memset(&P, 0, sizeof(P));
        std::memset(&S, 0, sizeof(S));
        std::memset((void*)&G, 0, sizeof(G));
        EeRayGeom& R = G.ray[0];
        float* to[8] = {R.B0, R.Bx, R.By, R.Bz, R.G0, R.Gx, R.Gy, R.Gz};
        for (int k = 0; k < 8; k++) std::memcpy(to[k], f + 3 * k, 12);
        const int tY = (int)f[24], tZ = (int)f[25];
        for (int a = 0; a < 3; a++) {
            G.bev[a] = box[9 * i + a];
            P.bb0[a] = box[9 * i + 3 + a];
            P.bbs[a] = box[9 * i + 6 + a];
            R.iB[a] = fabsf(R.Bx[a]) < 1e-6f ? 0.f : 1.f / R.Bx[a];
            R.iG[a] = fabsf(R.Gx[a]) < 1e-6f ? 0.f : 1.f / R.Gx[a];
            R.rev[a] = R.sn[a] = L;
        }
        for (int k = 0; k < 4; k++) R.lit[k][2] = R.side[k][1] = 1.f;  // every sample in the field
        R.front[1] = S.isodist = 100.f;
        int i0, m, c0, c1;
        line_segment(P, G, R, tY, tZ, L, i0, m);
        LineFrame F;
        const LaneSpan s = lane_span(P, S, G, R, tY, tZ, F);
        line_clear_span(P, G, R, tY, tZ, c0, c1);
        const int o[8] = {i0, i0 + m - 1, s.i0, s.i1, s.q0, s.q1, c0, c1};
        std::memcpy(out + 8 * i, o, sizeof(o));
    }
}
"""


@pytest.fixture(scope="module")
def builds(tmp_path_factory):
    d = tmp_path_factory.mktemp("spans")
    src = d / "spans.cpp"
    src.write_text(SOURCE)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc_path()))), "include")
    fma = ["-mfma"] if platform.machine() == "x86_64" else []
    out = []
    for form in ("off", "fast"):
        lib = str(d / f"spans_{form}.so")
        subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-w", *fma, f"-ffp-contract={form}",
                               "-I", cuda, "-I", _build.CSRC, str(src), "-o", lib])
        out.append(C.CDLL(lib))
    return out


def rotations(rng, n):
    q = rng.standard_normal((n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    w, x, y, z = q.T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                     2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                     2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1).reshape(n, 3, 3)


def lines_on_faces(rng, n, L, tilt):
    """Lines that enter or leave a box at a sample 4 q or 4 q - 1, on one of its
    faces to the last bit; tilt: the slope across that face, None: any."""
    B, G = rotations(rng, n), rotations(rng, n)
    box = np.concatenate([rng.integers(40, 90, (n, 3)), rng.integers(0, 9, (n, 3)), rng.integers(40, 90, (n, 3))], 1)
    t = rng.integers(0, L, (n, 2)).astype(np.float64)
    f = np.zeros((n, 26))
    at = 4.0 * rng.integers(6, L // 4 - 6, n) - rng.integers(0, 2, n)  # the sample on the face
    for which, (M, lo, hi) in enumerate(((B, np.zeros((n, 3)), box[:, :3]), (G, box[:, 3:6], box[:, 3:6] + box[:, 6:]))):
        o = 12 * which
        f[:, o + 3:o + 12] = M.transpose(0, 2, 1).reshape(n, 9)
        mid = lo + (hi - lo) * rng.uniform(0.3, 0.7, (n, 3))
        point = np.where(rng.random((n, 3)) < 0.5, lo, hi) * 1.0
        face = rng.integers(0, 3, n)
        on = (np.arange(3)[None] == face[:, None]) & (which == (np.arange(n) % 2))[:, None]
        point = np.where(on, point, mid)
        if tilt is not None:
            f[:, o + 3:o + 6] = np.where(on, tilt * np.sign(f[:, o + 3:o + 6]), f[:, o + 3:o + 6])
        x, y, z = (np.float32(f[:, o + a:o + a + 3]).astype(np.float64) for a in (3, 6, 9))
        f[:, o:o + 3] = point - x * at[:, None] - y * t[:, :1] - z * t[:, 1:]
    f[:, 24:] = t
    return np.ascontiguousarray(f, np.float32), np.ascontiguousarray(box, np.int32)


@pytest.mark.parametrize("tilt", [None, 3e-3, 2e-6])
def test_cleared_samples_cover_those_read(builds, tilt):
    L, n = 160, 40000
    lines, box = lines_on_faces(np.random.default_rng(17), n, L, tilt)
    res = []
    for lib in builds:
        out = np.zeros((n, 8), np.int32)
        lib.spans(lines.ctypes.data_as(C.c_void_p), box.ctypes.data_as(C.c_void_p), n, L, out.ctypes.data_as(C.c_void_p))
        res.append(out)
    assert (res[0][:, 5] >= res[0][:, 4]).sum() > n // 10  # lines with samples
    for clear in res:
        for read in res:
            live = read[:, 5] >= read[:, 4]
            out = live & ((clear[:, 6] >> 2 > read[:, 2] >> 2) | (clear[:, 7] >> 2 < read[:, 3] >> 2))
            assert not out.any(), (int(out.sum()), read[out][:3], clear[out][:3])
    np.testing.assert_array_equal(res[0], res[1])
