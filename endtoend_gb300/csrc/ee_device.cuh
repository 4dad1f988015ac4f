// ee_device.cuh -- device helpers shared by the beam-dose kernels
// (ee_kernels.cu) and the beamlet-column kernels (ee_beamlet.cu): vector
// arithmetic, the border-mode trilinear gather, the Siddon radiological path,
// the beamlet lookup and the polyenergetic TERMA of one point.
#pragma once
#include "ee_internal.h"
#include "ee_lines.cuh"
#include <cfloat>

namespace {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ int f2key(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : (i ^ 0x7fffffff);
}
__device__ __forceinline__ float key2f(int k) { return __int_as_float(k >= 0 ? k : (k ^ 0x7fffffff)); }

// ceil() with extents within 1e-3 of an integer snapped to it, so that
// axis-aligned beams (exactly integer crop-box / REV extents) do not flip by
// one voxel with the last bit of the FP32 rotation (the reference's plain
// ceilf at host.cu:469-473, :111-114 is rounding-dependent there).
__device__ __forceinline__ float snap_ceilf(float v) {
    float r = rintf(v);
    return fabsf(v - r) <= 1e-3f ? r : ceilf(v);
}

// Vector reduction of four floats into a 16-byte aligned quad of global
// memory (red.global.add.v4.f32, sm_90+): no value comes back, unlike an
// atomicAdd whose result the caller ignores.
__device__ __forceinline__ void red_v4(float* q, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(q), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}

// ------------------------------------------------ bricked TERMA boxes ----
// Address parts of box element (x, y, z) in the 4x4x4-brick layout
// (ee_brick_vol): the element sits at bk_x(x) + bk_y(y) + bk_z(z).  32-bit:
// ee_set_volume keeps the bricked calc bbox, which bounds every box, below 2^31.
struct Brick {
    int n0, n1, n2;
    int sy, sz;  // 64*nbx, 64*nbx*nby
};
__device__ __forceinline__ Brick brick_of(const int tn[3]) {
    Brick B;
    B.n0 = tn[0]; B.n1 = tn[1]; B.n2 = tn[2];
    B.sy = 64 * ((tn[0] + 3) >> 2);
    B.sz = B.sy * ((tn[1] + 3) >> 2);
    return B;
}
__device__ __forceinline__ int bk_x(int x) { return ((x >> 2) << 6) + (x & 3); }
__device__ __forceinline__ int bk_y(const Brick& B, int y) { return (y >> 2) * B.sy + ((y & 3) << 2); }
__device__ __forceinline__ int bk_z(const Brick& B, int z) { return (z >> 2) * B.sz + ((z & 3) << 4); }

// A cone's REV arrays (dose, dose gradient, cone scratch) are bricked over
// (i, tY, tZ), the sample index along the line fastest: dimensions (rev[0],
// rev[1], rev[2]); ee_brick_vol(rev) cells.  Four consecutive samples of a
// line are one 16-byte brick row, and the 8 x 4 lines of a warp cover two
// whole bricks per quad of samples.
__device__ __forceinline__ Brick rev_brick(int n0, int n1, int n2) {  // n0 = rev[0] (along the line)
    Brick B;
    B.n0 = n0; B.n1 = n1; B.n2 = n2;
    B.sy = 64 * ((n0 + 3) >> 2);
    B.sz = B.sy * ((n1 + 3) >> 2);
    return B;
}
// A cone's REV array as it is kept (EeRayGeom::so, sn): the whole array's
// sizes for the border tests, the kept part's brick strides.
__device__ __forceinline__ Brick rev_store(const EeRayGeom& R) {
    Brick B = rev_brick(R.sn[0], R.sn[1], R.sn[2]);
    B.n0 = R.rev[0]; B.n1 = R.rev[1]; B.n2 = R.rev[2];
    return B;
}
// Offset of line (tY, tZ) in a bricked REV array: its sample i sits at
// rev_line(B, tY, tZ) + bk_x(i).
__device__ __forceinline__ int rev_line(const Brick& B, int tY, int tZ) { return bk_y(B, tY) + bk_z(B, tZ); }

// The cell of a point and whether all its corners lie in the box; the float to
// integer conversion saturates, so a point far outside is outside here too.
__device__ __forceinline__ bool brick_cell(const Brick& B, float x, float y, float z, int& i, int& j, int& k) {
    i = __float2int_rd(x);
    j = __float2int_rd(y);
    k = __float2int_rd(z);
    return (unsigned)i < (unsigned)(B.n0 - 1) && (unsigned)j < (unsigned)(B.n1 - 1) && (unsigned)k < (unsigned)(B.n2 - 1);
}

// tex3D<float> with linear filtering, unnormalised coordinates and border
// addressing, as an explicit FP32 gather from a bricked box, at a point (the
// texel-centre shift of -0.5 taken) whose corners all lie in the box.  The corners are addressed from the first one by per-axis
// steps (+1, +4, +16 inside a brick; +61, +sy - 12, +sz - 48 across a brick
// face), which with one range test per axis saves the forward cone 7 % against a
// brick offset per corner with a test each.
__device__ __forceinline__ float tri_brick_cell(const float* __restrict__ v, const Brick& B, float x, float y, float z,
                                                int i, int j, int k) {
    const float ax = x - (float)i, ay = y - (float)j, az = z - (float)k;
    const float* p = v + (i + 60 * (i >> 2) + 4 * j + (j >> 2) * (B.sy - 16) + 16 * k + (k >> 2) * (B.sz - 64));
    const int dx = (i & 3) == 3 ? 61 : 1, dy = (j & 3) == 3 ? B.sy - 12 : 4, dz = (k & 3) == 3 ? B.sz - 48 : 16;
    const float c000 = __ldg(p), c100 = __ldg(p + dx), c010 = __ldg(p + dy), c110 = __ldg(p + dy + dx);
    const float c001 = __ldg(p + dz), c101 = __ldg(p + dz + dx), c011 = __ldg(p + dz + dy),
                c111 = __ldg(p + dz + dy + dx);
    const float c00 = c000 + ax * (c100 - c000), c10 = c010 + ax * (c110 - c010);
    const float c01 = c001 + ax * (c101 - c001), c11 = c011 + ax * (c111 - c011);
    const float c0 = c00 + ay * (c10 - c00), c1 = c01 + ay * (c11 - c01);
    return c0 + az * (c1 - c0);
}

// The same at any other point: the corner values that
// exist, weighted; 0 from one cell outside the box on.  Callers keep it out of
// their unrolled samples: there it was a quarter of the forward cone's code and
// a third of the gather's, more than the instruction cache holds.
__device__ __forceinline__ float tri_brick_edge(const float* __restrict__ v, const Brick B, float x, float y, float z) {
    if (!(x > -1.f && x < (float)B.n0 && y > -1.f && y < (float)B.n1 && z > -1.f && z < (float)B.n2)) return 0.f;
    const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    const int i = (int)fx, j = (int)fy, k = (int)fz;
    const float ax = x - fx, ay = y - fy, az = z - fz;
    float acc = 0.f;
#pragma unroll
    for (int dk = 0; dk < 2; dk++) {
        int kk = k + dk;
        if (kk < 0 || kk >= B.n2) continue;
        float wz = dk ? az : 1.f - az;
#pragma unroll
        for (int dj = 0; dj < 2; dj++) {
            int jj = j + dj;
            if (jj < 0 || jj >= B.n1) continue;
            float wy = dj ? ay : 1.f - ay;
#pragma unroll
            for (int di = 0; di < 2; di++) {
                int ii = i + di;
                if (ii < 0 || ii >= B.n0) continue;
                float wx = di ? ax : 1.f - ax;
                acc += wx * wy * wz * __ldg(v + bk_x(ii) + bk_y(B, jj) + bk_z(B, kk));
            }
        }
    }
    return acc;
}

// The same at any point.
__device__ __forceinline__ float tri_brick(const float* __restrict__ v, const Brick& B, float x, float y, float z) {
    int i, j, k;
    return brick_cell(B, x, y, z, i, j, k) ? tri_brick_cell(v, B, x, y, z, i, j, k) : tri_brick_edge(v, B, x, y, z);
}

// tri_brick for a point the caller has placed in [0, n0) x [0, n1) x [0, n2):
// no entry or lower-bound tests.  The last cell of an axis goes out of line:
// inlined for four voxels it is a third of the gather's code.  (With
// tri_brick_cell's body the gather at 48 registers spills twice as much: 96
// beams 8.7 -> 9.1 ms.)
__device__ __noinline__ float tri_brick_last(const float* __restrict__ v, const Brick B, float x, float y, float z) {
    return tri_brick_edge(v, B, x, y, z);
}
__device__ __forceinline__ float tri_brick_in(const float* __restrict__ v, const Brick& B, float x, float y, float z) {
    const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    const int i = (int)fx, j = (int)fy, k = (int)fz;
    if (i + 1 < B.n0 && j + 1 < B.n1 && k + 1 < B.n2) {
        const float ax = x - fx, ay = y - fy, az = z - fz;
        const float* p = v + bk_x(i) + bk_y(B, j) + bk_z(B, k);
        const int dx = (i & 3) == 3 ? 61 : 1, dy = (j & 3) == 3 ? B.sy - 12 : 4, dz = (k & 3) == 3 ? B.sz - 48 : 16;
        float c000 = __ldg(p), c100 = __ldg(p + dx), c010 = __ldg(p + dy), c110 = __ldg(p + dy + dx);
        float c001 = __ldg(p + dz), c101 = __ldg(p + dz + dx), c011 = __ldg(p + dz + dy),
              c111 = __ldg(p + dz + dy + dx);
        float c00 = c000 + ax * (c100 - c000), c10 = c010 + ax * (c110 - c010);
        float c01 = c001 + ax * (c101 - c001), c11 = c011 + ax * (c111 - c011);
        float c0 = c00 + ay * (c10 - c00), c1 = c01 + ay * (c11 - c01);
        return c0 + az * (c1 - c0);
    }
    return tri_brick_last(v, B, x, y, z);
}

// Transpose of tri_brick.  Each (y, z)
// corner row takes one vector reduction on the 16-byte brick row of corner
// i, holding both x corners unless the pair straddles a brick edge (i % 4 ==
// 3), and a second one on slot 0 of the next brick row only then (or when
// corner i is outside the box).  The other slots of a quad receive +0.  No
// branch on the slot, so the lanes of a warp issue the same two reductions.
__device__ __forceinline__ void tri_brick_scatter(float* v, const Brick& B, float x, float y, float z, float g) {
    if (!(x > -1.f && x < (float)B.n0 && y > -1.f && y < (float)B.n1 && z > -1.f && z < (float)B.n2)) return;
    float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    int i = (int)fx, j = (int)fy, k = (int)fz;
    float ax = x - fx, ay = y - fy, az = z - fz;
    const bool in0 = i >= 0, in1 = i + 1 < B.n0;
    const int o = i & 3;                        // slot of corner i in its brick row
    const bool both = in0 && in1 && o != 3;     // corner i + 1 in the same row
    const int xa = in0 ? (i >> 2) << 6 : 0;     // brick row of corner i
    const int xb = in1 ? ((i + 1) >> 2) << 6 : 0;  // brick row of corner i + 1 (slot 0 unless both)
    // the x weights in the four slots of corner i's brick row, the same for
    // the four corner rows: each row's reduction is w times this pattern
    const float a0 = 1.f - ax;
    const float p0 = o == 0 ? a0 : 0.f, p1 = o == 1 ? a0 : (o == 0 && both ? ax : 0.f);
    const float p2 = o == 2 ? a0 : (o == 1 && both ? ax : 0.f), p3 = o == 3 ? a0 : (o == 2 && both ? ax : 0.f);
#pragma unroll
    for (int dk = 0; dk < 2; dk++) {
        int kk = k + dk;
        if (kk < 0 || kk >= B.n2) continue;
        float wz = dk ? az : 1.f - az;
#pragma unroll
        for (int dj = 0; dj < 2; dj++) {
            int jj = j + dj;
            if (jj < 0 || jj >= B.n1) continue;
            float w = (dj ? ay : 1.f - ay) * wz * g;
            float* row = v + bk_y(B, jj) + bk_z(B, kk);
            if (in0) red_v4(row + xa, w * p0, w * p1, w * p2, w * p3);
            if (in1 && !both) red_v4(row + xb, w * ax, 0.f, 0.f, 0.f);
        }
    }
}

// The quads of a TERMA gradient (ee_quad_vol): the box's sizes, the quads' brick
// strides.
__device__ __forceinline__ Brick quads_of(const int* tn) {
    Brick B;
    B.n0 = tn[0]; B.n1 = tn[1]; B.n2 = tn[2];
    B.sy = 64 * ((tn[0] + 4) >> 2);
    B.sz = B.sy * ((tn[1] + 4) >> 2);
    return B;
}

// Offset of row z of the quads: unsigned, since a box near the 2^31 voxels that a
// volume may have has more quads than that.
__device__ __forceinline__ unsigned quad_z(const Brick& Q, int z) {
    return (unsigned)(z >> 2) * (unsigned)Q.sz + ((unsigned)(z & 3) << 4);
}

// Transpose of tri_brick: scatter g with the trilinear weights, one 16-byte
// reduction per z corner.  Corners outside the box in x or y fall on values that
// quad_value does not read, those in z are left out.  Against a reduction per
// (y, z) corner row into the voxels, and a second one where the row crosses a
// brick, it moves 32 bytes a sample instead of 80 on average: 6 beams 0.628 ->
// 0.369 ms of adjoint cone, 24 beams 3.55 -> 1.95 ms.
__device__ __forceinline__ void quad_scatter(float4* v, const Brick& Q, float x, float y, float z, float g) {
    if (!(x > -1.f && x < (float)Q.n0 && y > -1.f && y < (float)Q.n1 && z > -1.f && z < (float)Q.n2)) return;
    const int i = __float2int_rd(x), j = __float2int_rd(y), k = __float2int_rd(z);
    const float ax = x - (float)i, ay = y - (float)j, az = z - (float)k;
    const unsigned p = (unsigned)(bk_x(i + 1) + bk_y(Q, j + 1));
    const float g1 = ay * g, g0 = g - g1, g01 = ax * g0, g00 = g0 - g01, g11 = ax * g1, g10 = g1 - g11;
    const float bz = az, cz = 1.f - az;
    if (k >= 0) red_v4(reinterpret_cast<float*>(v + (p + quad_z(Q, k))), cz * g00, cz * g01, cz * g10, cz * g11);
    if (k + 1 < Q.n2) red_v4(reinterpret_cast<float*>(v + (p + quad_z(Q, k + 1))), bz * g00, bz * g01, bz * g10, bz * g11);
}

// The gradient of voxel (x, y, z) of the box from its four cells.
__device__ __forceinline__ float quad_value(const float4* __restrict__ v, const Brick& Q, int x, int y, int z) {
    const float4* const p = v + quad_z(Q, z);
    const int x0 = bk_x(x), x1 = bk_x(x + 1), y0 = bk_y(Q, y), y1 = bk_y(Q, y + 1);
    return (__ldg(&p[x1 + y1].x) + __ldg(&p[x0 + y1].y)) + (__ldg(&p[x1 + y0].z) + __ldg(&p[x0 + y0].w));
}

// ---------------------------------------------------------------- TERMA --
// Radiological path of the ray source -> voxel centre (cudaSiddon.cu:20-115):
// plane crossings advanced from a common a_min, midpoint density samples of
// the border-mode trilinear density at (pos-start)/voxel, segments shorter
// than 1e-3 cm skipped, 5000-iteration cap.  (Nine comparisons per crossing in
// place of the reference's validity logic: k_terma 10.0 -> 9.4 ms on 96 beams.)
// A sample is added while the next one's fetch is under way; the order of the
// sum stays.  Bound by the texture unit's data stage, 72 % busy on average so and
// 66 % with one fetch in flight: 96 beams 8.07 -> 7.81 ms, 4 beams with 27
// centres per voxel 6.29 -> 5.80.
__device__ float siddon_rpl(const EeParams& P, f3 vox, f3 src, bool& iter_cap) {
    const f3 start = mk(P.start[0], P.start[1], P.start[2]);
    const f3 voxel = mk(P.voxel[0], P.voxel[1], P.voxel[2]);
    const f3 end = mk(start.x + P.size[0] * voxel.x, start.y + P.size[1] * voxel.y, start.z + P.size[2] * voxel.z);
    f3 diff = vox - src, sd = start - src, ed = end - src;
    float afx = (sd.x - 0.5f * voxel.x) / diff.x, afy = (sd.y - 0.5f * voxel.y) / diff.y,
          afz = (sd.z - 0.5f * voxel.z) / diff.z;
    float alx = (ed.x + 0.5f * voxel.x) / diff.x, aly = (ed.y + 0.5f * voxel.y) / diff.y,
          alz = (ed.z + 0.5f * voxel.z) / diff.z;
    float a_min = fmaxf(0.f, fmaxf(fmaxf(fminf(afx, alx), fminf(afy, aly)), fminf(afz, alz)));
    float a_max = fminf(1.f, fminf(fminf(fmaxf(afx, alx), fmaxf(afy, aly)), fmaxf(afz, alz)));
    float rpl = 0.f;
    if (!(a_min >= a_max)) {
        float d12 = sqrtf(dot(diff, diff));
        float stx = fabsf(voxel.x / diff.x), sty = fabsf(voxel.y / diff.y), stz = fabsf(voxel.z / diff.z);
        float alpha = a_min, ax = a_min, ay = a_min, az = a_min, next = 0.f;
        const float ivx = 1.f / voxel.x, ivy = 1.f / voxel.y, ivz = 1.f / voxel.z;
        int iter = 0;
        // The reference advances every axis that is valid (its parameter in
        // [0, 1)) and not above the other valid ones, one axis after the other.
        // The parameters start at a_min >= 0 and grow, and an invalid one
        // (>= 1) is above every valid one, so "below 1 and not above the other
        // two" is the same test.
        // the next segment's length (0 below the cut) and sample position
        auto segment = [&](float& len, f3& at) {
            if (!(alpha < a_max && ++iter < 5000)) return false;
            const bool vy = ay < 1.f, vz = az < 1.f;
            const bool cx = ax < 1.f && ax <= ay && ax <= az;
            if (cx) { next = ax; ax += stx; }
            const bool cy = vy && ay <= ax && ay <= az;
            if (cy) { next = ay; ay += sty; }
            const bool cz = vz && az <= ax && az <= ay;
            if (cz) { next = az; az += stz; }
            if (!(cx || cy || cz)) return false;  // no axis valid
            const float isect = fabsf(d12 * (next - alpha));
            len = isect >= 0.001f ? isect : 0.f;
            const float mid = (next + alpha) * 0.5f;
            at = mk((src.x + mid * diff.x - start.x) * ivx, (src.y + mid * diff.y - start.y) * ivy,
                    (src.z + mid * diff.z - start.z) * ivz);
            alpha = next;
            return true;
        };
        // a segment below the cut is fetched with the others but not added: the
        // density there may be infinite, and 0 times that is not 0
        auto add = [&](float len, float rho) {
            if (len > 0.f) rpl = fmaf(len, rho, rpl);
        };
        float l0 = 0.f, r0 = 0.f, l1 = 0.f, r1 = 0.f;
        f3 at;
        for (;;) {
            float len;
            if (!segment(len, at)) break;
            l0 = len;
            r0 = tex3D<float>(P.dens_tex, at.x, at.y, at.z);
            add(l1, r1);
            l1 = 0.f;
            if (!segment(len, at)) break;
            l1 = len;
            r1 = tex3D<float>(P.dens_tex, at.x, at.y, at.z);
            add(l0, r0);
            l0 = 0.f;
        }
        add(l0, r0);
        add(l1, r1);
        if (iter >= 5000) iter_cap = true;
    }
    return rpl;
}

// The beamlet decision of beamlet_of in FP64 (same formula), for voxels
// whose FP32 fluence-map coordinate is within 1e-4 of a beamlet boundary
// (50x the FP32 error of that coordinate):
// there the FP32 rounding of the projection decides which beamlet (of two
// with different fluence) the voxel takes, and the result would not be
// reproducible.  About two voxels per beam take this path.
__device__ __noinline__ int beamlet_point_fp64(const EeBeamSpec& S, double vx, double vy, double vz) {
    const double dx = vx - S.srcd[0], dy = vy - S.srcd[1], dz = vz - S.srcd[2];
    const double pl = dx * S.dird[0] + dy * S.dird[1] + dz * S.dird[2];
    const double rx = dx - pl * S.dird[0], ry = dy - pl * S.dird[1], rz = dz - pl * S.dird[2];
    const double rl = sqrt(rx * rx + ry * ry + rz * rz);
    if (!(rl > 0.0)) return -1;
    const double prl = fabs(pl);
    const double trad = rl * fabs(S.isodistd / prl);
    const double sc = trad / rl;
    const double px = rx * sc, py = ry * sc, pz = rz * sc;
    const double bx = S.MBd[0] * px + S.MBd[1] * py + S.MBd[2] * pz;
    const double bz = S.MBd[6] * px + S.MBd[7] * py + S.MBd[8] * pz;
    const double fx = bx / (double)S.beamlet[0] + S.fmap[0] * 0.5;
    const double fz = bz / (double)S.beamlet[1] + S.fmap[1] * 0.5;
    if (!(fx >= 0.0 && fx < (double)S.fmap[0] && fz >= 0.0 && fz < (double)S.fmap[1])) return -1;
    const int idx = (int)floor(fx) + S.fmap[0] * (int)floor(fz);
    if (idx < 0 || idx >= S.fmap[0] * S.fmap[1]) return -1;
    return idx;
}

__device__ __forceinline__ int beamlet_of_fp64(const EeParams& P, const EeBeamSpec& S, int x, int y, int z) {
    return beamlet_point_fp64(S, (double)P.start[0] + (double)x * (double)P.voxel[0],
                              (double)P.start[1] + (double)y * (double)P.voxel[1],
                              (double)P.start[2] + (double)z * (double)P.voxel[2]);
}

// Beamlet under this voxel (cudaSiddon.cu:143-165), -1 if none.
__device__ __forceinline__ int beamlet_of(const EeBeamSpec& S, f3 vox) {
    f3 src = ld3(S.src), nd = ld3(S.dir);
    f3 diff = vox - src;
    float pl = dot(diff, nd);
    f3 proj = nd * pl;
    f3 rej = diff - proj;
    float rl = sqrtf(dot(rej, rej));
    if (!(rl > 0.f)) return -1;  // normalize(0) is NaN in the reference: no fluence
    float trad = rl * fabsf(S.isodist / sqrtf(dot(proj, proj)));
    f3 pf = rej * (trad / rl);
    f3 pb = mv(S.MB, pf);
    float fx = pb.x / S.beamlet[0] + S.fmap[0] * 0.5f;
    float fz = pb.z / S.beamlet[1] + S.fmap[1] * 0.5f;
    // near a beamlet boundary (integer coordinate): signal the FP64 path
    if (fabsf(fx - rintf(fx)) < 1e-4f || fabsf(fz - rintf(fz)) < 1e-4f) return -2;
    if (!(fx >= 0.f && fx < (float)S.fmap[0] && fz >= 0.f && fz < (float)S.fmap[1])) return -1;
    int idx = (int)floorf(fx) + S.fmap[0] * (int)floorf(fz);
    if (idx < 0 || idx >= S.fmap[0] * S.fmap[1]) return -1;
    return idx;
}

__device__ __forceinline__ float terma_per_fluence(const EeParams& P, float rpl, f3 vox, f3 src, float sad) {
    float tsum = 0.f;
    for (int e = 0; e < P.nE; e++) {
        float mu = P.sp_mu[e];
        tsum += P.sp_fluence[e] * P.sp_energy[e] * mu * expf(-mu * rpl);
    }
    f3 d = vox - src;
    return tsum * (sad * sad) / dot(d, d);
}

}  // namespace
