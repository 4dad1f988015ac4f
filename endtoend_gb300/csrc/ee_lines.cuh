// ee_lines.cuh -- which samples of a cone's line a kernel visits: the segment
// inside the BEV crop box and the calc bbox, the part the field can reach, the
// part the gathers can read.  Several kernels work these out for the same line.
// No device-only code, so it compiles for the host as well.
#pragma once
#include "ee_internal.h"

namespace {

struct f3 {
    float x, y, z;
};
__device__ __forceinline__ f3 mk(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ f3 operator+(f3 a, f3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ f3 operator-(f3 a, f3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ f3 operator*(f3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ float dot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ f3 ld3(const float* p) { return {p[0], p[1], p[2]}; }
__device__ __forceinline__ f3 mv(const float* M, f3 v) {
    return {M[0] * v.x + M[1] * v.y + M[2] * v.z, M[3] * v.x + M[4] * v.y + M[5] * v.z,
            M[6] * v.x + M[7] * v.y + M[8] * v.z};
}

// The sums below have their roundings written out.  Two kernels that work out
// the same line's samples, one to clear or write what the other reads, have to
// find the same ones, and a compiler may contract a product and a sum in one of
// them and not in the other: on a line along a face of a box the last bit of
// its origin moves the end by several samples.

// c0 + cy fy + cz fz: a point of line (fy, fz).
__device__ __forceinline__ f3 line_point(const float* c0, const float* cy, const float* cz, float fy, float fz) {
    return mk(fmaf(cz[0], fz, fmaf(cy[0], fy, c0[0])), fmaf(cz[1], fz, fmaf(cy[1], fy, c0[1])),
              fmaf(cz[2], fz, fmaf(cy[2], fy, c0[2])));
}
// o + d t
__device__ __forceinline__ f3 along(f3 o, f3 d, float t) { return mk(fmaf(d.x, t, o.x), fmaf(d.y, t, o.y), fmaf(d.z, t, o.z)); }

// The least of a cone's lit forms at lateral REV point (tY, tZ).
__device__ __forceinline__ float lit_form(const EeRayGeom& R, float tY, float tZ) {
    float f = 1e30f;
#pragma unroll
    for (int k = 0; k < 4; k++) f = fminf(f, fmaf(R.lit[k][0], tY, fmaf(R.lit[k][1], tZ, R.lit[k][2])));
    return f;
}

// Samples of REV line (tY, tZ) that can be valid: the line's intersection
// with the BEV crop box and the calc bbox (both convex, so one segment),
// widened by one sample for rounding.  Outside it every sample is a sentinel
// (-3 outside the BEV box, -2 outside the bbox, device.cu:51-70) and its dose
// is zero, so neither the gather nor the scans visit it.
__device__ __forceinline__ void line_segment(const EeParams& P, const EeBeamGeom& G, const EeRayGeom& R, int tY,
                                             int tZ, int L, int& i0, int& n) {
    const f3 bl = line_point(R.B0, R.By, R.Bz, (float)tY, (float)tZ);
    const f3 gl = line_point(R.G0, R.Gy, R.Gz, (float)tY, (float)tZ);
    const float c[6] = {bl.x, bl.y, bl.z, gl.x, gl.y, gl.z};
    const float im[6] = {R.iB[0], R.iB[1], R.iB[2], R.iG[0], R.iG[1], R.iG[2]};
    const float lo[6] = {0.f, 0.f, 0.f, (float)P.bb0[0], (float)P.bb0[1], (float)P.bb0[2]};
    const float hi[6] = {(float)G.bev[0], (float)G.bev[1], (float)G.bev[2], (float)(P.bb0[0] + P.bbs[0]),
                         (float)(P.bb0[1] + P.bbs[1]), (float)(P.bb0[2] + P.bbs[2])};
    float a = 0.f, b = (float)(L - 1);
#pragma unroll
    for (int k = 0; k < 6; k++) {
        if (im[k] == 0.f) {
            if (c[k] < lo[k] - 1e-3f || c[k] > hi[k] + 1e-3f) { n = 0; i0 = 0; return; }
        } else {
            float t0 = (lo[k] - c[k]) * im[k], t1 = (hi[k] - c[k]) * im[k];
            a = fmaxf(a, fminf(t0, t1));
            b = fminf(b, fmaxf(t0, t1));
        }
    }
    if (!(a <= b + 2.f)) { n = 0; i0 = 0; return; }
    i0 = max(R.so[0], (int)floorf(a) - 1);
    int i1 = min(R.so[0] + R.sn[0] - 1, (int)ceilf(b) + 1);
    n = max(0, i1 - i0 + 1);
}

// Samples of a REV line that k_gather can read (and k_gather_T can add to):
// k_gather visits voxels within 2 BEV voxels of the crop box and reads the
// REV cells within one REV step (per axis) of each voxel's REV point, i.e.
// within sum_k |B[a][k]| BEV units per axis a.  So the line's intersection
// with the crop box dilated by 2 + sum_k |B[a][k]| (+0.05, +1 sample each
// side) holds every sample either kernel touches; samples outside it are
// never read and need no zero.  z1 < z0: none.
__device__ __forceinline__ void line_read_span(const EeBeamGeom& G, const EeRayGeom& R, int tY, int tZ, int L,
                                               int& z0, int& z1) {
    const f3 bl = line_point(R.B0, R.By, R.Bz, (float)tY, (float)tZ);
    const float c[3] = {bl.x, bl.y, bl.z};
    float a = 0.f, b = (float)(L - 1);
    z0 = 0;
    z1 = -1;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float D = 2.05f + fabsf(R.Bx[k]) + fabsf(R.By[k]) + fabsf(R.Bz[k]);
        const float lo = -D, hi = (float)G.bev[k] + D, im = R.iB[k];
        if (im == 0.f) {
            if (c[k] < lo || c[k] > hi) return;
        } else {
            const float t0 = (lo - c[k]) * im, t1 = (hi - c[k]) * im;
            a = fmaxf(a, fminf(t0, t1));
            b = fminf(b, fmaxf(t0, t1));
        }
    }
    if (!(a <= b + 2.f)) return;
    z0 = max(R.so[0], (int)floorf(a) - 1);
    z1 = min(R.so[0] + R.sn[0] - 1, (int)ceilf(b) + 1);
}

struct LineFrame {
    f3 gl, gx;  // patient voxel index of sample 0, and its step per sample
};

__device__ __forceinline__ f3 sample_point(const LineFrame& F, int i) { return along(F.gl, F.gx, (float)i); }

// What a lane needs of its line.  [i0, i1]: the samples inside the BEV crop
// box and the calc bbox by the reference's own tests (device.cu:51-70).  Every
// test is a comparison of an affine function of i, which stays monotone in
// FP32, so the samples that pass are one interval: the analytic segment
// trimmed at its ends by the tests themselves, and no sample in between needs
// them again.  [q0, q1]: the quads of [i0, i1] that hold the samples whose
// TERMA corners can lie in the field (field_forms); q1 < q0: no such sample,
// so neither dose nor TERMA gradient.
struct LaneSpan {
    int i0, i1, q0, q1;
};

__device__ __forceinline__ LaneSpan lane_span(const EeParams& P, const EeBeamSpec& S, const EeBeamGeom& G,
                                              const EeRayGeom& R, int tY, int tZ, LineFrame& F) {
    const float fy = (float)tY, fz = (float)tZ;
    F.gl = line_point(R.G0, R.Gy, R.Gz, fy, fz);
    F.gx = ld3(R.Gx);
    LaneSpan s{0, -1, 0, -1};
    if (lit_form(R, fy, fz) < 0.f) return s;
    int n;
    line_segment(P, G, R, tY, tZ, R.rev[0], s.i0, n);
    s.i1 = s.i0 + n - 1;
    if (n <= 0) return s;
    // field span: the four sides, raised by more than their rounding, cut the
    // line to one interval.  The forms hold in front of the source; beamlet_of
    // takes |depth|, so a segment that does not stay in front of it is not
    // restricted
    float lo = -1e9f, hi = 1e9f;
    const float pr = fmaf(R.front[2], fy, fmaf(R.front[3], fz, R.front[1]));
    const bool front = fminf(fmaf(R.front[0], (float)s.i0, pr), fmaf(R.front[0], (float)s.i1, pr)) > 1e-2f * S.isodist;
    if (front) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float al = R.side[k][0], be = fmaf(R.side[k][2], fy, fmaf(R.side[k][3], fz, R.side[k][1]));
            if (fabsf(al) < 1e-20f) {
                if (be < 0.f) { lo = 1e9f; hi = -1e9f; }
            } else {
                const float t = fminf(fmaxf(__fdividef(-be, al), -1e9f), 1e9f);
                if (al > 0.f) lo = fmaxf(lo, t);
                else hi = fminf(hi, t);
            }
        }
    }
    const int f0 = max(s.i0, (int)ceilf(lo - 0.01f)), f1 = min(s.i1, (int)floorf(hi + 0.01f));
    if (f0 > f1) return s;
    const f3 bl = line_point(R.B0, R.By, R.Bz, fy, fz), bx = ld3(R.Bx);
    auto valid = [&](int i) {
        const f3 bev = along(bl, bx, (float)i), g = sample_point(F, i);
        return !(bev.x < 0.f || bev.y < 0.f || bev.z < 0.f || bev.x >= (float)G.bev[0] || bev.y >= (float)G.bev[1] ||
                 bev.z >= (float)G.bev[2] || g.x < (float)P.bb0[0] || g.x >= (float)(P.bb0[0] + P.bbs[0]) ||
                 g.y < (float)P.bb0[1] || g.y >= (float)(P.bb0[1] + P.bbs[1]) || g.z < (float)P.bb0[2] ||
                 g.z >= (float)(P.bb0[2] + P.bbs[2]));
    };
#pragma unroll 1
    while (s.i0 <= s.i1 && !valid(s.i0)) s.i0++;
#pragma unroll 1
    while (s.i1 > s.i0 && !valid(s.i1)) s.i1--;
    if (max(f0, s.i0) > min(f1, s.i1)) return s;
    s.q0 = max(f0, s.i0) >> 2;
    s.q1 = min(f1, s.i1) >> 2;
    return s;
}

// Samples [i0, i1] of line (tY, tZ) to clear in the REV gradient before the
// adjoint gather adds to it: the whole segment of a line that can be lit, of
// which lane_span is a part whatever its end tests decide.
__device__ __forceinline__ void line_clear_span(const EeParams& P, const EeBeamGeom& G, const EeRayGeom& R, int tY,
                                                int tZ, int& i0, int& i1) {
    i0 = 0;
    i1 = -1;
    if (lit_form(R, (float)tY, (float)tZ) < 0.f) return;
    int n;
    line_segment(P, G, R, tY, tZ, R.rev[0], i0, n);
    i1 = i0 + n - 1;
}

}  // namespace
