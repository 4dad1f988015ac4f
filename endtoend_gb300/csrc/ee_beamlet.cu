// ee_beamlet.cu -- beamlet dose columns (the dosecalc-beamlet path) on sm_103a.
//
// Semantics follow CCCS/dosecalc-beamlet/nvbbRayConvolve_host.cu and
// nvbbRayConvolve_device.cu: every active beamlet (fluence > 0) owns a pillar
// -- a box along its own divergent axis spanning the calc bbox plus the
// kernel extent, walled off from its neighbours -- the pillars are packed in
// one grid, and for each of the nphi*ntheta/2 convolution directions the
// grid is resampled into the rotated REV frame, convolved along REV lines with
// the cumulative-kernel walk (walls stop the walk), and gathered back.  Each
// pillar is then unpacked onto the calc bbox and thresholded into one sparse
// column.
//
// GB300 organisation:
//   k_bl_sources one warp, or several where beamlets are wide or few, per
//                direction, pillar and 32 units of depth: the REV samples
//                around that piece of the beamlet's footprint, each with the
//                reference's pillar lookup and beamlet test; samples inside
//                are queued and marked on their line (the reference looks at
//                every sample of the packed grid).
//   k_bl_terma   Siddon TERMA of the queued samples, lane-dense.
//   k_bl_walk    one warp per marked REV line: densities sampled into shared
//                memory, then the outputs of the wall-bounded segments that
//                hold TERMA samples; all other dose is zero.
//   k_bl_gather  packed-grid voxel += trilinear REV dose of one direction, in
//                the band of each pillar that the marked lines sweep.
//   k_bl_rows .. k_bl_emit
//                unpack: per pillar only the calc-bbox rows its oriented box
//                crosses, with the exact x-interval of each row; column max,
//                threshold count, prefix sums and a sorted CSR write, all on
//                the device (the reference copies a dense bbox per beamlet to
//                the host and sparsifies there, sparse_io.cpp:22-59).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <vector>

#include "../../include/ee_cccs.h"
#include "ee_device.cuh"
#include "ee_internal.h"

int ee_internal_fail(int code, const char* msg);

namespace {

constexpr int BL_WALL = 2;  // pillar wall thickness, REV voxels (io_data_structs.h:147)
constexpr int BL_BUF = 2;   // unusable buffer inside the walls (io_data_structs.h:148)
constexpr int BL_WARPS = 4;

// ------------------------------------------------------------- tables ---
struct BlPillar {
    float M[9];        // pillar-index vector -> RCS offset (inverse beamlet, then inverse beam rotation)
    float Mi[9];       // RCS offset -> pillar-index vector
    float ps[3];       // pillar start, RCS cm
    int fidx;          // fluence-map index of the beamlet
    int ix, iz;        // pillar position in the packed grid
    int b0[3], bn[3];  // calc-bbox-index AABB of the pillar's usable region (unpack)
    long long row0;    // first unpack row of this pillar
    // the beamlet's footprint (the rays from the source through the corners
    // of its fluence-map cell) in pillar-index coordinates: corner ray c is
    // x = ex[c] + sx[c] * y, z = ez[c] + sz[c] * y
    float ex[4], sx[4], ez[4], sz[4];
};

struct BlGrid {
    int n;             // pillars in this batch
    int npx, npz;      // pillars along the packed grid's x and z
    int pd[3];         // pillar dims (REV voxels)
    float rpd[2];      // 1 / pd[0], 1 / pd[2]
    int gd[3];         // packed grid dims
    float vs[3];       // REV voxel size (lat, long, lat)
    float kr[EE_MAX_RADII];  // kernel radii: the radial bins' mean radii (host.cu:352-357)
    float kern_extent;
};

// --------------------------------------------- host geometry (FP32) ------
// The reference computes the pillar layout on the host in FP32
// (nvbbRayConvolve_host.cu:180-280, 600-690, 75-155); the pillar and REV
// sizes truncate ratios that are integers in exact arithmetic, so the same
// FP32 operations are kept here to land on the same sizes.
struct v3 {
    float x, y, z;
};
v3 operator+(v3 a, v3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
v3 operator-(v3 a, v3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
v3 operator*(v3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
v3 operator*(v3 a, v3 b) { return {a.x * b.x, a.y * b.y, a.z * b.z}; }
float len(v3 a) { return sqrtf(a.x * a.x + a.y * a.y + a.z * a.z); }
float comp(v3 a, int i) { return i == 0 ? a.x : (i == 1 ? a.y : a.z); }

// Rodrigues rotation of p about the unit axis r by t, in the operation order
// of geometry.cu's rotateAroundAxisAtOriginRHS
v3 rot_axis(v3 p, v3 r, float t) {
    float s = sinf(t), c = cosf(t);
    float d = -r.x * p.x - r.y * p.y - r.z * p.z;
    return {(-r.x * d) * (1 - c) + p.x * c + (-r.z * p.y + r.y * p.z) * s,
            (-r.y * d) * (1 - c) + p.y * c + (+r.z * p.x - r.x * p.z) * s,
            (-r.z * d) * (1 - c) + p.z * c + (-r.y * p.x + r.x * p.y) * s};
}
v3 inv_rot_beam(v3 v, float az, float zen, float coll) {
    v3 t = rot_axis(v, {0.f, 1.f, 0.f}, -(zen + coll));
    return rot_axis(t, {sinf(-zen), 0.f, cosf(-zen)}, az);
}
v3 rot_beam(v3 v, float az, float zen, float coll) {
    v3 t = rot_axis(v, {sinf(-zen), 0.f, cosf(-zen)}, -az);
    return rot_axis(t, {0.f, 1.f, 0.f}, zen + coll);
}
// beamlet frame about the divergence angles (geometry.cu:99-115)
v3 inv_rot_beamlet(v3 v, float th, float ph) { return rot_axis(v, {sinf(-ph), 0.f, cosf(-ph)}, -th); }
v3 rot_beamlet(v3 v, float th, float ph) { return inv_rot_beamlet(v, -th, ph); }
v3 rot_kern(v3 v, float th, float ph) {
    v3 u = rot_axis(v, {cosf(ph), 0.f, -sinf(ph)}, -th);
    return rot_axis(u, {0.f, 1.f, 0.f}, -ph);
}

template <class F>
void matrix(F f, float* M) {
    v3 c[3] = {f({1.f, 0.f, 0.f}), f({0.f, 1.f, 0.f}), f({0.f, 0.f, 1.f})};
    for (int j = 0; j < 3; j++) {
        M[0 * 3 + j] = c[j].x;
        M[1 * 3 + j] = c[j].y;
        M[2 * 3 + j] = c[j].z;
    }
}

struct Beamlet {
    int fidx;
    v3 first, last, biso;
    float th, ph;  // divergence angles
    float length;
};

// calcBeamletAnchors (host.cu:180-280): the beamlet's isocentre, divergence
// angles, and the nearest / farthest crossings of its axis with the calc
// bbox faces (0.05 cm tolerance).  false: the axis misses the bbox.
bool anchors(Beamlet& B, v3 src, v3 iso, int idx, float bsx, float bsy, int fx, int fy, v3 voxel, v3 dstart, v3 bb0,
             v3 bbs, float az, float zen, float coll) {
    const unsigned bx = (unsigned)idx % (unsigned)fx, by = (unsigned)idx / (unsigned)fx;
    const v3 bdiff = {bsx * (-0.5f * fx + bx + 0.5f), 0.f, bsy * (-0.5f * fy + by + 0.5f)};
    B.biso = iso + inv_rot_beam(bdiff, az, zen, coll);
    B.th = acosf(len(iso - src) / len(B.biso - src));
    B.ph = atan2f(bdiff.z, bdiff.x);
    const v3 lo = dstart + voxel * bb0;
    const v3 hi = lo + voxel * bbs;
    const double buf = 0.05;
    const v3 d = B.biso - src;
    v3 hit[6];
    for (int a = 0; a < 3; a++) {
        const double den = comp(d, a);
        const double t1 = (comp(lo, a) - comp(src, a)) / (den + 1e-12);
        const double t2 = (comp(hi, a) - comp(src, a)) / (den + 1e-12);
        hit[2 * a] = src + d * (float)t1;
        hit[2 * a + 1] = src + d * (float)t2;
    }
    B.first = {std::numeric_limits<float>::max(), std::numeric_limits<float>::max(), std::numeric_limits<float>::max()};
    B.last = {std::numeric_limits<float>::min(), std::numeric_limits<float>::min(), std::numeric_limits<float>::min()};
    double dmin = std::numeric_limits<double>::max(), dmax = std::numeric_limits<double>::min();
    for (int a = 0; a < 3; a++)
        for (int s = 0; s < 2; s++) {
            const v3 p = hit[2 * a + s];
            const int u = (a + 1) % 3, v = (a + 2) % 3;
            if (comp(p, u) + buf >= comp(lo, u) && comp(p, u) - buf <= comp(hi, u) && comp(p, v) + buf >= comp(lo, v) &&
                comp(p, v) - buf <= comp(hi, v)) {
                if (len(p - src) < dmin) { B.first = p; dmin = len(B.first - src); }
                if (len(p - src) > dmax) { B.last = p; dmax = len(B.last - src); }
            }
        }
    B.length = len(B.last - B.first);
    return dmin < std::numeric_limits<float>::max() && dmax > std::numeric_limits<float>::min();
}

}  // namespace

namespace {

// ------------------------------------------------------------ kernels ----
// One convolution direction of a batch.  The directions that fit the scratch
// budget together run in one launch per stage: 36 k ray traces of a direction
// alone leave the chip to the latency of single rays.
struct BlRayDev {
    int rev[3];        // REV size: along the line, lateral, lateral
    float rs[3];       // REV box origin (cm, REV frame)
    float rcp[3];      // 1 / REV voxel size
    float MK[9], MKi[9];
    int row_f, row_r;  // kernel rows of the two walk directions
    // this direction's part of the group's buffers: REV dose (which holds the
    // TERMA of a line's sources until the line is walked), flag of each line
    // (1: it carries TERMA samples), source bits of each line [lines][words]
    float* dose;
    int* flag;
    unsigned* bits;
    int words;
};

constexpr int BL_CAPACITY = 2;  // status bit: the source queue was too short

// Counters and lists of a group of directions.
struct BlQueue {
    int* nsrc;    // queued sources
    int* nlines;  // lines that carry them
    int2* src;    // (direction, REV sample)
    int2* line;   // (direction, line)
    int cap;      // entries of src
};

// Linear filtering of one kernel row at texel coordinate x (unnormalised,
// clamp addressing) with the filter weight rounded to 8 fractional bits as
// the texture unit does.
__device__ __forceinline__ float kern_tex(const float* K, int nr, float x) {
    float xb = x - 0.5f;
    float fx = floorf(xb);
    int i = (int)fx;
    float a = xb - fx;
    a = floorf(a * 256.f + 0.5f) * (1.f / 256.f);
    int i0 = min(max(i, 0), nr - 1), i1 = min(max(i + 1, 0), nr - 1);
    return (1.f - a) * K[i0] + a * K[i1];
}

// floorf(x / y) with the quotient rounded to nearest, and fmodf(x, y), for
// 0 <= x < 2^24 and an integer-valued y >= 2, without a division.  r = x - q y
// is exact (q y is an integer, the difference a multiple of ulp(x) below 2 y),
// and rcp = 1 / y leaves q at most one off, so one correction step gives the
// exact floor and remainder.  The rounded quotient has the same floor: it
// could only differ by rounding up to an integer n with x < n y, but then
// x <= n y - ulp(x), and with 2^e <= x < 2^(e+1) the distance of x / y from n
// is at least 2^(e-23) / y > n 2^-24, more than half a unit of the floats at n.
__device__ __forceinline__ float floor_mod(float x, float y, float rcp, float& r) {
    float q = floorf(x * rcp);
    r = fmaf(-q, y, x);
    if (r < 0.f) { r += y; q -= 1.f; }
    else if (r >= y) { r -= y; q += 1.f; }
    return q;
}

// A point of the packed pillar grid (packed-index coordinates): its pillar and
// its pillar index coordinate; false for walls, empty pillars and points
// outside the grid (the reference's INVALID density, -1e-12).
__device__ __forceinline__ bool bl_pillar_point(const BlGrid& G, f3 pb, int& pidx, f3& ip) {
    if (pb.x < 0.f || pb.y < 0.f || pb.z < 0.f || pb.x >= (float)G.gd[0] || pb.y >= (float)G.gd[1] ||
        pb.z >= (float)G.gd[2])
        return false;
    float rx, rz;
    const float qx = floor_mod(pb.x, (float)G.pd[0], G.rpd[0], rx), qz = floor_mod(pb.z, (float)G.pd[2], G.rpd[1], rz);
    pidx = (int)qx + (int)qz * G.npx;
    if (pidx >= G.n) return false;
    // pb.y < pd.y + wall: fmodf(pb.y, pd.y) is pb.y or pb.y - pd.y (exact)
    const float py = pb.y >= (float)G.pd[1] ? pb.y - (float)G.pd[1] : pb.y;
    ip = mk(rx, py, rz);
    if (ip.x < (float)BL_WALL || ip.y < (float)BL_WALL || ip.z < (float)BL_WALL) return false;
    ip = mk(ip.x - 0.5f, ip.y - 0.5f, ip.z - 0.5f);
    return true;
}

// M v with the roundings written out.  Samples exactly on a beamlet's edge are
// common on the rotated lattice and the columns' entries are cut by a
// threshold, so the last bit of a coordinate can decide both; it must not hang
// on how a compiler contracts the sums in one kernel or another.
__device__ __forceinline__ f3 mv_rounded(const float* M, f3 v) {
    return mk(fmaf(M[2], v.z, fmaf(M[0], v.x, __fmul_rn(M[1], v.y))),
              fmaf(M[5], v.z, fmaf(M[3], v.x, __fmul_rn(M[4], v.y))),
              fmaf(M[8], v.z, fmaf(M[6], v.x, __fmul_rn(M[7], v.y))));
}
// the same with the first two products' roles exchanged (densities of a line)
__device__ __forceinline__ f3 mv_rounded_x(const float* M, f3 v) {
    return mk(fmaf(M[2], v.z, fmaf(M[1], v.y, __fmul_rn(M[0], v.x))),
              fmaf(M[5], v.z, fmaf(M[4], v.y, __fmul_rn(M[3], v.x))),
              fmaf(M[8], v.z, fmaf(M[7], v.y, __fmul_rn(M[6], v.x))));
}

__device__ __forceinline__ f3 bl_rev_vector(const BlRayDev& R, int tX, int tY, int tZ) {
    return mk(fmaf(R.rs[0], R.rcp[0], (float)tZ), fmaf(R.rs[1], R.rcp[1], (float)tX),
              fmaf(R.rs[2], R.rcp[2], (float)tY));
}

// One REV sample of the packed pillar grid (cudaBeamletRaytrace,
// device.cu:20-246 with ss_factor 1).
__device__ __forceinline__ bool bl_locate(const BlGrid& G, const BlRayDev& R, int tX, int tY, int tZ, int& pidx,
                                          f3& ip) {
    const f3 pb = mv_rounded(R.MKi, bl_rev_vector(R, tX, tY, tZ));
    return bl_pillar_point(G, mk(pb.x + 0.5f, pb.y + 0.5f, pb.z + 0.5f), pidx, ip);
}

// TERMA point of a sample: pillar index rotated, then scaled, + start
__device__ __forceinline__ f3 bl_terma_point(const BlGrid& G, const BlPillar& Q, f3 ip) {
    const f3 tr = mv_rounded(Q.M, ip);
    return mk(fmaf(tr.x, G.vs[0], Q.ps[0]), fmaf(tr.y, G.vs[1], Q.ps[1]), fmaf(tr.z, G.vs[2], Q.ps[2]));
}

// Can pillar-index point ip lie in the pillar's beamlet?  The footprint's
// cross-section at pillar depth y is inside the box spanned by its four
// corner rays there (a rotation keeps rays straight); 0.05 index units of
// margin keep every point the exact test could accept.
__device__ __forceinline__ bool bl_near_footprint(const BlPillar& Q, f3 ip) {
    float x0 = 1e30f, x1 = -1e30f, z0 = 1e30f, z1 = -1e30f;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const float x = fmaf(Q.sx[c], ip.y, Q.ex[c]), z = fmaf(Q.sz[c], ip.y, Q.ez[c]);
        x0 = fminf(x0, x); x1 = fmaxf(x1, x);
        z0 = fminf(z0, z); z1 = fmaxf(z1, z);
    }
    return ip.x >= x0 - 0.05f && ip.x <= x1 + 0.05f && ip.z >= z0 - 0.05f && ip.z <= z1 + 0.05f;
}

// REV coordinates (tZ, tX, tY) of pillar-index point ip: the inverse of
// bl_locate's map.
__device__ __forceinline__ f3 bl_rev_point(const BlGrid& G, const BlPillar& Q, const BlRayDev& R, f3 ip) {
    const f3 r = mv(R.MK, mk(ip.x + (float)(Q.ix * G.pd[0]), ip.y, ip.z + (float)(Q.iz * G.pd[2])));
    return mk(fmaf(-R.rs[0], R.rcp[0], r.x), fmaf(-R.rs[1], R.rcp[1], r.y), fmaf(-R.rs[2], R.rcp[2], r.z));
}

// Pass 1, `slices` warps per direction, pillar and 32 units of pillar depth.  A
// unit's candidates are the REV samples in the box around that piece of the
// beamlet's footprint (3^3 to 4^3 for a beamlet of a voxel or two): each lane
// sets one unit's box up, and the warp then walks the candidates of all its
// units, 32 at a time, locating and testing each as the reference tests every
// sample.  A sample is taken by the depth unit it falls in, so it is queued
// once.  The first lane of a pillar also writes its band: the interval
// [lo, hi] of n . (tZ, tY) that a voxel must lie in for one of its eight REV
// corners to sit on a flagged line, n normal to the projected pillar axis.
// Samples and lines collect in shared memory, so the two global counters take
// one add per warp or so and not one per sample.  Bound by the instructions of
// the tests.  A thread per REV sample (0.2 % of them are in a beamlet) took
// 272 us per direction of about 110 beamlets on 200 x 200 x 160 at 2 mm, a warp
// per unit 27 us; this takes 5.2 us.
constexpr int BL_SRC_WARPS = 4, BL_SRC_BUF = 128;

__global__ void __launch_bounds__(BL_SRC_WARPS * 32)
    k_bl_sources(const EeBeamSpec* __restrict__ spec, BlGrid G, const BlPillar* __restrict__ pil,
                 const BlRayDev* __restrict__ rays, BlQueue W, int slices, float4* __restrict__ band,
                 int* __restrict__ status) {
    // per warp and unit: box origin (tX, tY, tZ), sizes along tX and tY, first candidate
    __shared__ int s_unit[BL_SRC_WARPS][6][32];
    __shared__ int s_v[BL_SRC_WARPS][BL_SRC_BUF], s_line[BL_SRC_WARPS][BL_SRC_BUF];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int part = blockIdx.y * BL_SRC_WARPS + warp, slice = part % slices;
    const int u0 = part / slices * 32, unit = u0 + lane, j = blockIdx.x, r = blockIdx.z;
    const BlRayDev& R = rays[r];
    const BlPillar& Q = pil[j];
    if (unit == 0 && slice == 0) {
        float n0 = -R.MK[7], n1 = R.MK[1];  // n = (-e_tY, e_tZ), e the pillar axis
        const float l = sqrtf(n0 * n0 + n1 * n1);
        if (l > 1e-3f) { n0 /= l; n1 /= l; }
        else { n0 = 1.f; n1 = 0.f; }
        float lo = 1e30f, hi = -1e30f;
        for (int e = 0; e < 2; e++) {
            const float y = e ? (float)G.pd[1] : 1.f;
            float x0 = 1e30f, x1 = -1e30f, z0 = 1e30f, z1 = -1e30f;
            for (int c = 0; c < 4; c++) {
                const float x = fmaf(Q.sx[c], y, Q.ex[c]), z = fmaf(Q.sz[c], y, Q.ez[c]);
                x0 = fminf(x0, x); x1 = fmaxf(x1, x);
                z0 = fminf(z0, z); z1 = fmaxf(z1, z);
            }
            for (int c = 0; c < 4; c++) {
                const f3 q = bl_rev_point(G, Q, R, mk(c & 1 ? x1 : x0, y, c & 2 ? z1 : z0));
                const float t = n0 * q.x + n1 * q.z;
                lo = fminf(lo, t);
                hi = fmaxf(hi, t);
            }
        }
        // one REV cell of trilinear reach, and the footprint's own margin
        const float m = fabsf(n0) + fabsf(n1) + 0.2f;
        band[(size_t)r * G.n + j] = make_float4(n0, n1, lo - m, hi + m);
    }
    // the depth unit [y0, y0 + 1) of sample coordinates (bl_locate gives
    // ip.y in [1.5, pd.y - 0.5)) and its candidates
    int n = 0;
    if (unit <= G.pd[1] - BL_WALL) {
        const float y0 = (float)BL_WALL - 0.5f + (float)unit, y1 = y0 + 1.f;
        float x0 = 1e30f, x1 = -1e30f, z0 = 1e30f, z1 = -1e30f;
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const float y = (c & 4) ? y1 : y0;
            const float x = fmaf(Q.sx[c & 3], y, Q.ex[c & 3]), z = fmaf(Q.sz[c & 3], y, Q.ez[c & 3]);
            x0 = fminf(x0, x); x1 = fmaxf(x1, x);
            z0 = fminf(z0, z); z1 = fmaxf(z1, z);
        }
        const f3 ctr = bl_rev_point(G, Q, R, mk(0.5f * (x0 + x1), y0 + 0.5f, 0.5f * (z0 + z1)));
        // half sizes: the footprint's 0.05 margin and 0.02 for rounding
        const float hx = 0.5f * (x1 - x0) + 0.07f, hy = 0.52f, hz = 0.5f * (z1 - z0) + 0.07f;
        const float rz = fabsf(R.MK[0]) * hx + fabsf(R.MK[1]) * hy + fabsf(R.MK[2]) * hz;
        const float rx = fabsf(R.MK[3]) * hx + fabsf(R.MK[4]) * hy + fabsf(R.MK[5]) * hz;
        const float ry = fabsf(R.MK[6]) * hx + fabsf(R.MK[7]) * hy + fabsf(R.MK[8]) * hz;
        const int tz0 = max(0, (int)ceilf(ctr.x - rz)), tz1 = min(R.rev[2] - 1, (int)floorf(ctr.x + rz));
        const int tx0 = max(0, (int)ceilf(ctr.y - rx)), tx1 = min(R.rev[0] - 1, (int)floorf(ctr.y + rx));
        const int ty0 = max(0, (int)ceilf(ctr.z - ry)), ty1 = min(R.rev[1] - 1, (int)floorf(ctr.z + ry));
        const int nx = tx1 - tx0 + 1, ny = ty1 - ty0 + 1, nz = tz1 - tz0 + 1;
        if (nx > 0 && ny > 0 && nz > 0) {
            n = nx * ny * nz;
            s_unit[warp][0][lane] = tx0;
            s_unit[warp][1][lane] = ty0;
            s_unit[warp][2][lane] = tz0;
            s_unit[warp][3][lane] = nx;
            s_unit[warp][4][lane] = ny;
        }
    }
    int upto = n;  // candidates up to and with this lane's unit
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, upto, o);
        if (lane >= o) upto += y;
    }
    const int total = __shfl_sync(FULL, upto, 31);
    s_unit[warp][5][lane] = upto - n;
    __syncwarp();
    int* bv = s_v[warp];
    int* bl = s_line[warp];
    int nv = 0, nl = 0;  // collected samples and lines
    auto flush = [&]() {
        __syncwarp();
        int base_v = 0, base_l = 0;
        if (lane == 0 && nv) base_v = atomicAdd(W.nsrc, nv);
        if (lane == 0 && nl) base_l = atomicAdd(W.nlines, nl);
        base_v = __shfl_sync(FULL, base_v, 0);
        base_l = __shfl_sync(FULL, base_l, 0);
        if (base_v + nv > W.cap && lane == 0) atomicOr(status, BL_CAPACITY);
        for (int i = lane; i < nv; i += 32)
            if (base_v + i < W.cap) W.src[base_v + i] = make_int2(r, bv[i]);
        for (int i = lane; i < nl; i += 32) W.line[base_l + i] = make_int2(r, bl[i]);
        nv = nl = 0;
        __syncwarp();
    };
    const int per = ((total + slices - 1) / slices + 31) & ~31, stop = min(total, (slice + 1) * per);
    for (int k0 = slice * per; k0 < stop; k0 += 32) {
        const int k = k0 + lane;
        bool take = false, fresh = false;
        int v = 0, line = 0;
        if (k < stop) {
            int u = 0;  // the last unit that starts at or before k (units without candidates share a start)
#pragma unroll
            for (int o = 16; o; o >>= 1)
                if (s_unit[warp][5][u + o] <= k) u += o;
            const int c = k - s_unit[warp][5][u], nx = s_unit[warp][3][u], ny = s_unit[warp][4][u];
            const int cyz = c / nx, cz = cyz / ny;
            const int tX = s_unit[warp][0][u] + c - cyz * nx, tY = s_unit[warp][1][u] + cyz - cz * ny;
            const int tZ = s_unit[warp][2][u] + cz;
            const float y0 = (float)BL_WALL - 0.5f + (float)(u0 + u);
            int pidx;
            f3 ip;
            if (bl_locate(G, R, tX, tY, tZ, pidx, ip) && pidx == j && ip.y >= y0 && ip.y < y0 + 1.f &&
                bl_near_footprint(Q, ip)) {
                const f3 gt = bl_terma_point(G, Q, ip);
                int b = beamlet_of(*spec, gt);
                if (b == -2) b = beamlet_point_fp64(*spec, (double)gt.x, (double)gt.y, (double)gt.z);
                if (b == Q.fidx) {
                    take = true;
                    line = tY + R.rev[1] * tZ;
                    v = line * R.rev[0] + tX;
                    atomicOr(&R.bits[(size_t)line * R.words + (tX >> 5)], 1u << (tX & 31));
                    fresh = atomicExch(&R.flag[line], 1) == 0;
                }
            }
        }
        const unsigned mv_ = __ballot_sync(FULL, take), ml = __ballot_sync(FULL, fresh), below = (1u << lane) - 1u;
        if (take) bv[nv + __popc(mv_ & below)] = v;
        if (fresh) bl[nl + __popc(ml & below)] = line;
        nv += __popc(mv_);
        nl += __popc(ml);
        if (nv > BL_SRC_BUF - 32) flush();  // nl <= nv
    }
    if (nv) flush();
}

// Density of a sample (pillar index scaled, rotated, + start; the reference's
// INVALID -1e-12 for walls / outside).
__device__ __forceinline__ float bl_density(const EeParams& P, const BlGrid& G, const BlPillar* __restrict__ pil,
                                            const BlRayDev& R, int tX, int tY, int tZ) {
    int pidx;
    f3 ip;
    const f3 pb = mv_rounded_x(R.MKi, bl_rev_vector(R, tX, tY, tZ));
    if (!bl_pillar_point(G, mk(pb.x + 0.5f, pb.y + 0.5f, pb.z + 0.5f), pidx, ip)) return -1e-12f;
    const BlPillar& Q = pil[pidx];
    const f3 gd = mv_rounded(Q.M, mk(ip.x * G.vs[0], ip.y * G.vs[1], ip.z * G.vs[2]));
    const f3 g = mk(gd.x + Q.ps[0], gd.y + Q.ps[1], gd.z + Q.ps[2]);
    return tex3D<float>(P.dens_tex, __fdiv_rn(g.x - P.start[0], P.voxel[0]) + 0.5f,
                        __fdiv_rn(g.y - P.start[1], P.voxel[1]) + 0.5f, __fdiv_rn(g.z - P.start[2], P.voxel[2]) + 0.5f);
}

// Pass 2: Siddon radiological path + polyenergetic TERMA of every queued
// sample (one thread each, so the ray traces run lane-dense).
__global__ void __launch_bounds__(256)
    k_bl_terma(EeParams P, const EeBeamSpec* __restrict__ spec, BlGrid G, const BlPillar* __restrict__ pil,
               const BlRayDev* __restrict__ rays, const float* __restrict__ fluence, BlQueue W,
               int* __restrict__ status) {
    const int nq = min(*W.nsrc, W.cap);
    const EeBeamSpec& S = *spec;
    const f3 src = ld3(S.src);
    bool cap = false;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x) {
        const int2 e = W.src[q];
        const BlRayDev& R = rays[e.x];
        const unsigned v = (unsigned)e.y;
        const unsigned line = v / (unsigned)R.rev[0];
        const int tX = (int)(v - line * (unsigned)R.rev[0]);
        const unsigned zq = line / (unsigned)R.rev[1];
        const int tY = (int)(line - zq * (unsigned)R.rev[1]), tZ = (int)zq;
        int pidx;
        f3 ip;
        if (!bl_locate(G, R, tX, tY, tZ, pidx, ip)) continue;
        const BlPillar& Q = pil[pidx];
        const f3 gt = bl_terma_point(G, Q, ip);
        const float f = __ldg(fluence + Q.fidx);  // an active beamlet's: positive
        const float rpl = siddon_rpl(P, gt, src, cap);
        R.dose[v] = f * terma_per_fluence(P, rpl, gt, src, S.sad);
    }
    if (cap) atomicOr(status, 1);
}

// Cumulative kernel at radiological distance r as PackRowConvolve reads it:
// first mean radius >= r, texture-filtered between the two table entries
// (device.cu:326-339).  inv[j] = 1 / (KR[j] - KR[j-1]).  The search for that
// radius starts at the first one not below the quarter-octave r lies in.
constexpr int BL_BINS = 64;              // quarter octaves from 2^-7 to 2^9 cm
constexpr int BL_BIN0 = (127 - 7) << 2;  // float bits >> 21 of the first

__device__ __forceinline__ int bl_bin(float r) {
    return min(max((__float_as_int(r) >> 21) - BL_BIN0, 0), BL_BINS - 1);
}

__device__ __forceinline__ float bl_ck(const float* K, const float* KR, const float* inv, const int* first, int nr,
                                       float r) {
    int lo = first[bl_bin(r)];  // first index with KR[idx] >= r (r <= KR[nr-1])
    while (lo < nr - 1 && KR[lo] < r) lo++;
    if (lo <= 0) return kern_tex(K, nr, 0.5f) * (r * inv[0]);
    const float interp = (r - KR[lo - 1]) * inv[lo];
    return kern_tex(K, nr, (float)lo - 0.5f + interp);
}

// floats of shared memory one warp of k_bl_walk needs for lines of L samples
__host__ __device__ constexpr int bl_walk_floats(int L) { return 4 * L + 1; }

// Pass 3, one warp per flagged line.  The reference's walk from output i
// visits every sample up to the next wall, adding T_k * (CK(s_k) - CK(s_k'))
// where s_k is the radiological distance between the centres of i and k (half
// of i's own step for k = i) and s_k' that of the previous sample; only
// samples with TERMA contribute.  Here each lane sums those terms directly
// over the TERMA samples of i's wall-bounded segment, with the distances from
// a prefix sum of the radiological steps, under the walk's stopping rules
// (the last radius for s_k, the one before it for s_k').  Only the segments
// that hold TERMA samples have outputs; s_k' of one source is s_k of its
// neighbour, whose kernel value is kept.  The prefix sums start at the line's
// first sample in the packed grid (32-sample groups from a multiple of 32:
// samples outside add exact zeros) and end with the last source's segment.
// The warp writes its whole line, so the dose array needs no clear.
__global__ void __launch_bounds__(BL_WARPS * 32, 7)
    k_bl_walk(EeParams P, BlGrid G, const BlPillar* __restrict__ pil, const BlRayDev* __restrict__ rays, BlQueue W,
              int maxL) {
    extern __shared__ float sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nr = P.nradii;
    float* KR = sm;
    float* inv = KR + EE_MAX_RADII;
    int* first = (int*)(inv + EE_MAX_RADII);  // [BL_BINS] start of bl_ck's search
    float* rows = (float*)(first + BL_BINS);  // [ntheta][nr]
    for (int k = threadIdx.x; k < nr; k += blockDim.x) {
        KR[k] = G.kr[k];
        inv[k] = k ? 1.f / (G.kr[k] - G.kr[k - 1]) : 1.f / G.kr[0];
    }
    for (int k = threadIdx.x; k < P.ntheta * nr; k += blockDim.x) rows[k] = P.cumkern[k];
    for (int k = threadIdx.x; k < BL_BINS; k += blockDim.x) {
        const float low = k ? __int_as_float((k + BL_BIN0) << 21) : 0.f;  // bin 0 holds everything below it
        int j = 0;
        while (j < nr - 1 && G.kr[j] < low) j++;
        first[k] = j;
    }
    __syncthreads();
    // per warp: d[L] (radiological step, -1 for walls), pre[L+1] (prefix of
    // steps), src[L] (sources: sample | walls before it << 16), ts[L] (TERMA)
    float* d = rows + P.ntheta * nr + (size_t)warp * bl_walk_floats(maxL);
    float* pre = d + maxL;
    int* src = (int*)(pre + maxL + 1);
    float* ts = (float*)(src + maxL);
    const float delr = P.lng;
    const float rmax = KR[nr - 1], rstop = KR[nr - 2];
    const float nphi = (float)P.nphi;
    const int nl = *W.nlines;
    for (int q = blockIdx.x * BL_WARPS + warp; q < nl; q += gridDim.x * BL_WARPS) {
        const int2 e = W.line[q];
        const BlRayDev& R = rays[e.x];
        const int line = e.y, L = R.rev[0], words = R.words;
        const int tY = line % R.rev[1], tZ = line / R.rev[1];
        const float* Kf = rows + R.row_f * nr;
        const float* Kr = rows + R.row_r * nr;
        const unsigned* bl = R.bits + (size_t)line * words;
        float* out = R.dose + (size_t)line * L;  // TERMA of the sources, then the dose
        // the line's samples in the packed grid, one more at each end
        int a = 0, b = L - 1;
        {
            const f3 p0 = mv(R.MKi, mk(fmaf(R.rs[0], R.rcp[0], (float)tZ), R.rs[1] * R.rcp[1],
                                       fmaf(R.rs[2], R.rcp[2], (float)tY)));
            const float c[3] = {p0.x, p0.y, p0.z};
            float fa = 0.f, fb = (float)(L - 1);
#pragma unroll
            for (int x = 0; x < 3; x++) {
                const float m = R.MKi[3 * x + 1];
                if (fabsf(m) > 1e-4f) {
                    const float u = (-0.6f - c[x]) / m, v = ((float)G.gd[x] - 0.4f - c[x]) / m;
                    fa = fmaxf(fa, fminf(u, v));
                    fb = fminf(fb, fmaxf(u, v));
                }
            }
            a = min(L - 1, max(0, (int)floorf(fa) - 1));
            b = min(L - 1, (int)ceilf(fb) + 1);
        }
        // the last source
        int last = -1;
        {
            const unsigned w = lane < words ? bl[lane] : 0u;
            const unsigned m = __ballot_sync(FULL, w != 0u);
            const int hw = 31 - __clz((int)m);
            last = 32 * hw + 31 - __clz((int)__shfl_sync(FULL, w, hw));
        }
        // prefix sums (steps of walls count 0) and the TERMA-sample list, in
        // ascending order, 32 samples at a time
        float carry = 0.f;
        int wcarry = 0, ns = 0, end = b + 1;
        if (lane == 0) pre[a & ~31] = 0.f;
        for (int i0 = a & ~31; i0 <= b; i0 += 32) {
            const int i = i0 + lane;
            const float rho = i < L ? bl_density(P, G, pil, R, i, tY, tZ) : 0.f;
            const bool wall = i < L && rho < 0.f;
            const float step = (i < L && !wall) ? delr * rho : 0.f;
            float x = step;
            for (int o = 1; o < 32; o <<= 1) {
                const float y = __shfl_up_sync(FULL, x, o);
                if (lane >= o) x += y;
            }
            const unsigned walls = __ballot_sync(FULL, wall), below = (1u << lane) - 1u;
            if (i < L) {
                d[i] = wall ? -1.f : step;
                pre[i + 1] = carry + x;
            }
            const float t = (bl[i0 >> 5] >> lane) & 1u ? out[i] : 0.f;
            const bool is_src = !wall && t != 0.f;
            const unsigned m = __ballot_sync(FULL, is_src);
            if (is_src) {
                const int p = ns + __popc(m & below);
                src[p] = i | (wcarry + __popc(walls & below)) << 16;
                ts[p] = t;
            }
            ns += __popc(m);
            carry = __shfl_sync(FULL, carry + x, 31);
            wcarry += __popc(walls);
            if (i0 + 31 > last) {  // a wall past the last source ends the line
                const unsigned past = walls & (last >= i0 ? ~((2u << (last - i0)) - 1u) : ~0u);
                if (past) {
                    end = i0 + __ffs((int)past) - 1;
                    break;
                }
            }
        }
        __syncwarp();
        for (int i = lane; i < L; i += 32) out[i] = 0.f;
        __syncwarp();
        end = min(end, L);
        for (int q0 = 0; q0 < ns;) {
            // sources q0 .. q1-1 share a segment; its samples lo .. hi-1
            const int sk0 = src[q0] & 0xffff, sg = src[q0] >> 16;
            int q1 = q0 + 1;
            while (q1 < ns && (src[q1] >> 16) == sg) q1++;
            int lo = sk0, hi = (src[q1 - 1] & 0xffff) + 1;
            for (;;) {
                const int i = lo - 1 - lane;
                const unsigned m = __ballot_sync(FULL, i < a || d[max(i, a)] < 0.f);
                lo -= m ? __ffs((int)m) - 1 : 32;
                if (m) break;
            }
            for (;;) {
                const int i = hi + lane;
                const unsigned m = __ballot_sync(FULL, i >= end || d[min(i, end - 1)] < 0.f);
                hi += m ? __ffs((int)m) - 1 : 32;
                if (m) break;
            }
            for (int i = lo + lane; i < hi; i += 32) {
                const float h = 0.5f * d[i];
                float sum = 0.f;
                // backward walk (kernel row P): sources k <= i
                float ck = 0.f;    // CK of sample kn as a source
                int kn = -1;
                for (int e = q0; e < q1; e++) {
                    const int k = src[e] & 0xffff;
                    if (k > i) break;
                    const float tk = ts[e];
                    if (k == i) {
                        if (h <= rmax) sum += (kn == k ? ck : bl_ck(Kf, KR, inv, first, nr, h)) * tk;
                        continue;
                    }
                    const float sk = h + (pre[i] - pre[k + 1]) + 0.5f * d[k];
                    const float sp = (k + 1 == i) ? h : h + (pre[i] - pre[k + 2]) + 0.5f * d[k + 1];
                    if (sk > rmax || sp > rstop) continue;
                    const float cs = kn == k ? ck : bl_ck(Kf, KR, inv, first, nr, sk);
                    ck = bl_ck(Kf, KR, inv, first, nr, sp);
                    kn = k + 1;
                    sum += (cs - ck) * tk;
                }
                // forward walk (kernel row ntheta-1-P): sources k >= i
                kn = -1;
                for (int e = q1 - 1; e >= q0; e--) {
                    const int k = src[e] & 0xffff;
                    if (k < i) break;
                    const float tk = ts[e];
                    if (k == i) {
                        if (h <= rmax) sum += (kn == k ? ck : bl_ck(Kr, KR, inv, first, nr, h)) * tk;
                        continue;
                    }
                    const float sk = h + (pre[k] - pre[i + 1]) + 0.5f * d[k];
                    const float sp = (k - 1 == i) ? h : h + (pre[k - 1] - pre[i + 1]) + 0.5f * d[k - 1];
                    if (sk > rmax || sp > rstop) continue;
                    const float cs = kn == k ? ck : bl_ck(Kr, KR, inv, first, nr, sk);
                    ck = bl_ck(Kr, KR, inv, first, nr, sp);
                    kn = k - 1;
                    sum += (cs - ck) * tk;
                }
                out[i] = sum / nphi;
            }
            q0 = q1;
        }
        __syncwarp();
    }
}

// tex3D<float> of a linear-memory volume as the texture unit filters it:
// border addressing, linear filtering with each weight rounded to 8
// fractional bits.  (x, y, z) are texel-space coordinates after the -0.5
// texel-centre shift.  The reference's REV-dose and packed-dose fetches go
// through textures (device.cu:423, 511); exact FP32 weights would move
// beamlet columns by ~0.25% of their maximum.
// row_flag (optional): [nz][ny], 0 where the whole row is zero and not stored.
__device__ __forceinline__ float tri_border_q(const float* __restrict__ v, int nx, int ny, int nz, float x, float y,
                                              float z, const int* __restrict__ row_flag = nullptr) {
    if (!(x > -1.f && x < (float)nx && y > -1.f && y < (float)ny && z > -1.f && z < (float)nz)) return 0.f;
    const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    const int i = (int)fx, j = (int)fy, k = (int)fz;
    const float ax = floorf((x - fx) * 256.f + 0.5f) * (1.f / 256.f);
    const float ay = floorf((y - fy) * 256.f + 0.5f) * (1.f / 256.f);
    const float az = floorf((z - fz) * 256.f + 0.5f) * (1.f / 256.f);
    const long long sxy = (long long)nx * ny;
    float acc = 0.f;
    if (i >= 0 && j >= 0 && k >= 0 && i + 1 < nx && j + 1 < ny && k + 1 < nz) {
        // all eight texels: the rows' flags, then the rows' loads, each four
        // at once; the same weights and sums as below
        bool on[4];
        float v0[4], v1[4];
#pragma unroll
        for (int e = 0; e < 4; e++) on[e] = !row_flag || __ldg(row_flag + j + (e & 1) + ny * (k + (e >> 1)));
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float* row = v + i + (long long)nx * (j + (e & 1)) + sxy * (k + (e >> 1));
            v0[e] = on[e] ? __ldg(row) : 0.f;
            v1[e] = on[e] ? __ldg(row + 1) : 0.f;
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float wy = (e & 1) ? ay : 1.f - ay, wz = (e >> 1) ? az : 1.f - az;
            const float w0 = (1.f - ax) * wy * wz, w1 = ax * wy * wz;
            if (w0 != 0.f) acc = fmaf(w0, v0[e], acc);
            if (w1 != 0.f) acc = fmaf(w1, v1[e], acc);
        }
        return acc;
    }
#pragma unroll
    for (int dk = 0; dk < 2; dk++) {
        const int kk = k + dk;
        if (kk < 0 || kk >= nz) continue;
        const float wz = dk ? az : 1.f - az;
#pragma unroll
        for (int dj = 0; dj < 2; dj++) {
            const int jj = j + dj;
            if (jj < 0 || jj >= ny) continue;
            const float wy = dj ? ay : 1.f - ay;
            if (row_flag && !__ldg(row_flag + jj + ny * kk)) continue;
            const float* row = v + (long long)nx * jj + sxy * kk;
#pragma unroll
            for (int di = 0; di < 2; di++) {
                const int ii = i + di;
                if (ii < 0 || ii >= nx) continue;
                const float w = (di ? ax : 1.f - ax) * wy * wz;
                if (w != 0.f) acc = fmaf(w, __ldg(row + ii), acc);
            }
        }
    }
    return acc;
}

// PackedREVtoBEVdose (device.cu:407-431): packed voxel (pX, pY, pZ) += the
// positive trilinear REV dose at its rotated position, direction by direction
// in order.  Packed layout: pY fastest, then pZ, then pX.  A block takes a
// column of a pillar, of the voxels that the unpacking can read (its
// coordinates lie in [4, pd - 2) and reach half a voxel below and above: voxels
// 3 .. pd - 2 of each axis).  In a direction's lateral plane the column is one
// point along the pillar's band normal (k_bl_sources), so the band is tested
// once per column and direction; outside it all eight REV corners sit on
// unflagged lines, whose dose is zero.  About 85 % of the (voxel, direction)
// pairs fall away, and the packed grid is read and written once per group
// instead of once per direction: 282 -> 25 us per direction (k_bl_sources'
// case).
constexpr int BL_GATHER_BLOCK = 128;

__global__ void __launch_bounds__(BL_GATHER_BLOCK)
    k_bl_gather(BlGrid G, const BlRayDev* __restrict__ rays, int nr, const float4* __restrict__ band,
                float* __restrict__ packed) {
    __shared__ unsigned long long s_mask;
    constexpr int lo = BL_WALL + BL_BUF - 1, hi = BL_BUF;
    const int ux = G.pd[0] - hi - lo + 1, uz = G.pd[2] - hi - lo + 1;  // used voxels of a pillar
    const int ix = blockIdx.x / ux, iz = blockIdx.y / uz, j = ix + iz * G.npx;
    if (j >= G.n) return;
    const int pX = ix * G.pd[0] + lo + (int)blockIdx.x % ux, pZ = iz * G.pd[2] + lo + (int)blockIdx.y % uz;
    const int t = threadIdx.x;
    if (t == 0) s_mask = 0ull;
    __syncthreads();
    if (t < nr) {
        const BlRayDev& R = rays[t];
        const float4 bd = band[(size_t)t * G.n + j];
        const f3 rot = mv(R.MK, mk((float)pX, 0.f, (float)pZ));
        const float p = bd.x * fmaf(-R.rs[0], R.rcp[0], rot.x) + bd.y * fmaf(-R.rs[2], R.rcp[2], rot.z);
        if (p >= bd.z && p <= bd.w) atomicOr(&s_mask, 1ull << t);
    }
    __syncthreads();
    const unsigned long long mask = s_mask;
    if (!mask) return;
    float* col = packed + ((size_t)pX * G.gd[2] + pZ) * G.gd[1];
    for (int pY = lo + t; pY <= G.pd[1] - hi; pY += BL_GATHER_BLOCK) {
        const float old = col[pY];
        float acc = old;
        for (unsigned long long m = mask; m; m &= m - 1) {
            const BlRayDev& R = rays[__ffsll((long long)m) - 1];
            const f3 rot = mv_rounded(R.MK, mk((float)pX, (float)pY, (float)pZ));
            const float qx = fmaf(-R.rs[0], R.rcp[0], rot.x), qy = fmaf(-R.rs[1], R.rcp[1], rot.y),
                        qz = fmaf(-R.rs[2], R.rcp[2], rot.z);
            const float d = tri_border_q(R.dose, R.rev[0], R.rev[1], R.rev[2], qy, qz, qx, R.flag);
            if (d > 0.f) acc += d;
        }
        if (acc != old) col[pY] = acc;
    }
}

// ---- unpack (UnpackBEVDosePillar, device.cu:438-521) + sparsification ----
// Pillar-index coordinate of calc-bbox voxel (x, y, z) and the usable-region
// test of the reference.
__device__ __forceinline__ bool bl_unpack_coord(const EeParams& P, const BlGrid& G, const BlPillar& Q, int x, int y,
                                                int z, f3& u) {
    const float gx = ((float)x + (float)P.bb0[0]) * P.voxel[0] + P.start[0];
    const float gy = ((float)y + (float)P.bb0[1]) * P.voxel[1] + P.start[1];
    const float gz = ((float)z + (float)P.bb0[2]) * P.voxel[2] + P.start[2];
    const f3 r = mv(Q.Mi, mk(gx - Q.ps[0], gy - Q.ps[1], gz - Q.ps[2]));
    u = mk(r.x / G.vs[0] + 0.5f, r.y / G.vs[1] + 0.5f, r.z / G.vs[2] + 0.5f);
    const float lo = (float)(BL_WALL + BL_BUF);
    return !(u.x < lo || u.y < lo || u.z < lo || u.x >= (float)(G.pd[0] - BL_BUF) ||
             u.y >= (float)(G.pd[1] - BL_BUF) || u.z >= (float)(G.pd[2] - BL_BUF));
}

__device__ __forceinline__ float bl_unpack_value(const BlGrid& G, const BlPillar& Q, const float* __restrict__ packed,
                                                 f3 u) {
    const float ux = u.x + (float)(Q.ix * G.pd[0]), uz = u.z + (float)(Q.iz * G.pd[2]);
    const float d = tri_border_q(packed, G.gd[1], G.gd[2], G.gd[0], u.y - 0.5f, uz - 0.5f, ux - 0.5f);
    return d > 0.f ? d : 0.f;
}

// Rows (y, z) of each pillar's calc-bbox AABB: conservative x-interval of the
// row inside the pillar's usable region (the region is convex and the
// pillar coordinate is affine along the row).
__global__ void __launch_bounds__(256) k_bl_rows(EeParams P, BlGrid G, const BlPillar* __restrict__ pil,
                                                 int* __restrict__ len, int* __restrict__ xs) {
    const BlPillar& Q = pil[blockIdx.y];
    const int nrows = Q.bn[1] * Q.bn[2];
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += gridDim.x * blockDim.x) {
        const int y = Q.b0[1] + r % Q.bn[1], z = Q.b0[2] + r / Q.bn[1];
        f3 u0, u1;
        bl_unpack_coord(P, G, Q, 0, y, z, u0);
        bl_unpack_coord(P, G, Q, 1, y, z, u1);
        const float du[3] = {u1.x - u0.x, u1.y - u0.y, u1.z - u0.z};
        const float uo[3] = {u0.x, u0.y, u0.z};
        float xlo = -1e30f, xhi = 1e30f;
        bool empty = false;
        for (int a = 0; a < 3; a++) {
            const float lo = (float)(BL_WALL + BL_BUF), hi = (float)(G.pd[a] - BL_BUF);
            if (fabsf(du[a]) < 1e-12f) {
                if (uo[a] < lo - 1e-3f || uo[a] > hi + 1e-3f) empty = true;
                continue;
            }
            float t0 = (lo - uo[a]) / du[a], t1 = (hi - uo[a]) / du[a];
            xlo = fmaxf(xlo, fminf(t0, t1));
            xhi = fminf(xhi, fmaxf(t0, t1));
        }
        int a = 0, b = -1;
        if (!empty && xlo <= xhi + 2.f) {
            a = max(Q.b0[0], (int)floorf(xlo) - 1);
            b = min(Q.b0[0] + Q.bn[0] - 1, (int)ceilf(xhi) + 1);
        }
        len[Q.row0 + r] = max(0, b - a + 1);
        xs[Q.row0 + r] = a;
    }
}

// Pillar of a flat unpack row (rows of a pillar are contiguous).
__device__ __forceinline__ int bl_pillar_of(const BlPillar* __restrict__ pil, int n, long long row) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int m = (lo + hi + 1) >> 1;
        if (pil[m].row0 <= row) lo = m;
        else hi = m - 1;
    }
    return lo;
}

// Unpacked values of every candidate voxel (warp per row) and each column's
// maximum (as the ordered bits of a non-negative float).
__global__ void __launch_bounds__(256) k_bl_values(EeParams P, BlGrid G, const BlPillar* __restrict__ pil,
                                                   const float* __restrict__ packed, long long nrows,
                                                   const int* __restrict__ len, const int* __restrict__ xs,
                                                   const long long* __restrict__ seg, float* __restrict__ vals,
                                                   int* __restrict__ colmax) {
    const int lane = threadIdx.x & 31;
    const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long row = w0; row < nrows; row += nw) {
        const int n = len[row];
        if (n == 0) continue;
        const int j = bl_pillar_of(pil, G.n, row);
        const BlPillar& Q = pil[j];
        const long long r = row - Q.row0;
        const int y = Q.b0[1] + (int)(r % Q.bn[1]), z = Q.b0[2] + (int)(r / Q.bn[1]);
        float m = 0.f;
        for (int k = lane; k < n; k += 32) {
            f3 u;
            float v = 0.f;
            if (bl_unpack_coord(P, G, Q, xs[row] + k, y, z, u)) v = bl_unpack_value(G, Q, packed, u);
            vals[seg[row] + k] = v;
            m = fmaxf(m, v);
        }
        for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(FULL, m, o));
        if (lane == 0 && m > 0.f) atomicMax(colmax + j, __float_as_int(m));
    }
}

// Voxels kept by the reference's threshold (value > thresh * column max).
__global__ void __launch_bounds__(256) k_bl_count(BlGrid G, const BlPillar* __restrict__ pil, long long nrows,
                                                  const int* __restrict__ len, const long long* __restrict__ seg,
                                                  const float* __restrict__ vals, const int* __restrict__ colmax,
                                                  float thresh, int* __restrict__ cnt) {
    const int lane = threadIdx.x & 31;
    const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long row = w0; row < nrows; row += nw) {
        const int n = len[row];
        int c = 0;
        if (n > 0) {
            const float cut = thresh * __int_as_float(colmax[bl_pillar_of(pil, G.n, row)]);
            for (int k = lane; k < n; k += 32) c += vals[seg[row] + k] > cut;
            for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(FULL, c, o);
        }
        if (lane == 0) cnt[row] = c;
    }
}

// Sorted CSR write: rows are in (z, y) order within a pillar and x ascends
// along a row, so the full-grid voxel index ascends within each column.
__global__ void __launch_bounds__(256) k_bl_emit(EeParams P, BlGrid G, const BlPillar* __restrict__ pil,
                                                 long long nrows, const int* __restrict__ len,
                                                 const int* __restrict__ xs, const long long* __restrict__ seg,
                                                 const float* __restrict__ vals, const int* __restrict__ colmax,
                                                 float thresh, const long long* __restrict__ off, long long base,
                                                 int* __restrict__ out_rows, float* __restrict__ out_vals) {
    const int lane = threadIdx.x & 31;
    const long long w0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long row = w0; row < nrows; row += nw) {
        const int n = len[row];
        if (n == 0) continue;
        const int j = bl_pillar_of(pil, G.n, row);
        const BlPillar& Q = pil[j];
        const long long r = row - Q.row0;
        const int y = Q.b0[1] + (int)(r % Q.bn[1]), z = Q.b0[2] + (int)(r / Q.bn[1]);
        const float cut = thresh * __int_as_float(colmax[j]);
        long long pos = base + off[row];
        for (int k0 = 0; k0 < n; k0 += 32) {
            const int k = k0 + lane;
            const float v = k < n ? vals[seg[row] + k] : 0.f;
            const bool keep = k < n && v > cut;
            const unsigned m = __ballot_sync(FULL, keep);
            if (keep) {
                const long long p = pos + __popc(m & ((1u << lane) - 1u));
                const int x = xs[row] + k;
                out_rows[p] = ((z + P.bb0[2]) * P.size[1] + (y + P.bb0[1])) * P.size[0] + (x + P.bb0[0]);
                out_vals[p] = v;
            }
            pos += __popc(m);
        }
    }
}

// ---- exclusive prefix sum (int -> long long), 1024 elements per block ----
__global__ void __launch_bounds__(1024) k_scan_block(const int* __restrict__ in, const long long* __restrict__ in64,
                                                     long long n, long long* __restrict__ out,
                                                     long long* __restrict__ block_sums) {
    __shared__ long long wsum[32];
    const long long i = (long long)blockIdx.x * 1024 + threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long v = i < n ? (in ? (long long)in[i] : in64[i]) : 0;
    long long x = v;
    for (int o = 1; o < 32; o <<= 1) {
        long long y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
        long long s = wsum[lane];
        for (int o = 1; o < 32; o <<= 1) {
            long long y = __shfl_up_sync(FULL, s, o);
            if (lane >= o) s += y;
        }
        wsum[lane] = s;
    }
    __syncthreads();
    const long long excl = x - v + (warp ? wsum[warp - 1] : 0);
    if (i < n) out[i] = excl;
    if (threadIdx.x == 1023) block_sums[blockIdx.x] = wsum[31];
}

__global__ void __launch_bounds__(1024) k_scan_add(long long* __restrict__ out, long long n,
                                                   const long long* __restrict__ block_off) {
    const long long i = (long long)blockIdx.x * 1024 + threadIdx.x;
    if (i < n) out[i] += block_off[blockIdx.x];
}

// col_ptr[c] = CSR offset of pillar c's first row; col_ptr[n] = batch total.
__global__ void k_bl_colptr(const BlPillar* __restrict__ pil, int n, const long long* __restrict__ off,
                            const int* __restrict__ cnt, long long nrows, long long base, long long* __restrict__ colptr) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n) colptr[j] = base + (pil[j].row0 < nrows ? off[pil[j].row0] : (nrows ? off[nrows - 1] + cnt[nrows - 1] : 0));
    if (j == n) colptr[n] = base + (nrows ? off[nrows - 1] + cnt[nrows - 1] : 0);
}

}  // namespace

// ================================================================ host ====
namespace {

template <class T>
struct Dev {
    T* p = nullptr;
    size_t n = 0;
    cudaError_t ensure(size_t count) {
        if (count <= n && p) return cudaSuccess;
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
        size_t want = std::max<size_t>(count, 1);
        cudaError_t e = cudaMalloc((void**)&p, want * sizeof(T));
        if (e == cudaSuccess) n = want;
        return e;
    }
    // grow keeping the first `keep` elements (stream-ordered copy)
    cudaError_t grow_keep(size_t count, size_t keep, cudaStream_t s) {
        if (count <= n && p) return cudaSuccess;
        T* q = nullptr;
        size_t want = std::max<size_t>(std::max(count, n + n / 2), 1);
        cudaError_t e = cudaMalloc((void**)&q, want * sizeof(T));
        if (e != cudaSuccess) return e;
        if (p && keep) e = cudaMemcpyAsync(q, p, keep * sizeof(T), cudaMemcpyDeviceToDevice, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (p) cudaFree(p);
        p = q;
        n = want;
        return e;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
};

struct BlWork {
    Dev<EeBeamSpec> spec;
    Dev<float> fluence, revd, packed, vals, out_vals;
    // a group of directions: REV dose (revd); counters, line flags and source
    // bits (lines); the lists of sources and lines
    Dev<int> lines;
    Dev<int2> queue, line_list;
    Dev<BlRayDev> rays;
    Dev<float4> band;
    Dev<BlPillar> pil;
    Dev<int> len, xs, cnt, colmax, status, out_rows, out_bidx;
    Dev<long long> seg, off, out_colptr;
    Dev<long long> scan_tmp[6];
    long long nnz = 0;
    int ncols = 0;
    void release() {
        spec.release(); fluence.release(); revd.release(); lines.release(); line_list.release();
        queue.release(); rays.release(); band.release(); packed.release(); vals.release(); out_vals.release();
        pil.release(); len.release(); xs.release(); cnt.release(); colmax.release(); status.release();
        out_rows.release(); out_bidx.release(); seg.release(); off.release(); out_colptr.release();
        for (auto& t : scan_tmp) t.release();
    }
};

#define BL_CUDA(call)                                                                                    \
    do {                                                                                                 \
        cudaError_t _e = (call);                                                                         \
        if (_e != cudaSuccess) return fail_cuda(#call, _e);                                              \
    } while (0)

int fail_cuda(const char* what, cudaError_t e) {
    char buf[512];
    snprintf(buf, sizeof(buf), "%s failed: %s", what, cudaGetErrorString(e));
    return ee_internal_fail(EE_ERR_CUDA, buf);
}

// exclusive prefix sum of n ints (or long longs) into out; recursion over the
// per-block totals
cudaError_t scan_excl(BlWork& W, const int* in, const long long* in64, long long n, long long* out, int depth,
                      cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const long long nb = (n + 1023) / 1024;
    cudaError_t e = W.scan_tmp[2 * depth].ensure(nb);
    if (e != cudaSuccess) return e;
    k_scan_block<<<(unsigned)nb, 1024, 0, s>>>(in, in64, n, out, W.scan_tmp[2 * depth].p);
    if (nb == 1) return cudaGetLastError();
    if (2 * depth + 1 >= 6) return cudaErrorInvalidValue;
    if ((e = W.scan_tmp[2 * depth + 1].ensure(nb)) != cudaSuccess) return e;
    if ((e = scan_excl(W, nullptr, W.scan_tmp[2 * depth].p, nb, W.scan_tmp[2 * depth + 1].p, depth + 1, s)) != cudaSuccess)
        return e;
    k_scan_add<<<(unsigned)nb, 1024, 0, s>>>(out, n, W.scan_tmp[2 * depth + 1].p);
    return cudaGetLastError();
}

// last exclusive prefix + last element = total
cudaError_t scan_total(const long long* out, const int* in, long long n, cudaStream_t s, long long* total) {
    *total = 0;
    if (n <= 0) return cudaSuccess;
    long long a = 0;
    int b = 0;
    cudaError_t e = cudaMemcpyAsync(&a, out + n - 1, sizeof(a), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&b, in + n - 1, sizeof(b), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    *total = a + b;
    return e;
}

// allocate_batch_sizes (host.cu:64-76): even split, remainder to the first
std::vector<int> batch_sizes(int n, int nb) {
    std::vector<int> v(nb, n / nb);
    for (int r = n - (n / nb) * nb, k = 0; r > 0; r--) v[(k++) % nb] += 1;
    return v;
}

struct RevBox {
    int size[3];
    v3 mn;
};

// findREV (host.cu:88-155) on the packed grid box [0, gsize]: REV sizes in
// the reference's (line, lateral, lateral) order; false if over max_rev
bool find_rev(v3 gsize, float th, float ph, float lat, float lng, const int max_rev[3], RevBox& R) {
    v3 mn = {std::numeric_limits<float>::max(), std::numeric_limits<float>::max(), std::numeric_limits<float>::max()};
    v3 mx = {std::numeric_limits<float>::min(), std::numeric_limits<float>::min(), std::numeric_limits<float>::min()};
    for (int xo = 0; xo < 2; xo++)
        for (int yo = 0; yo < 2; yo++)
            for (int zo = 0; zo < 2; zo++) {
                v3 o = rot_kern({gsize.x * xo, gsize.y * yo, gsize.z * zo}, th, ph);
                mn = {std::min(mn.x, o.x), std::min(mn.y, o.y), std::min(mn.z, o.z)};
                mx = {std::max(mx.x, o.x), std::max(mx.y, o.y), std::max(mx.z, o.z)};
            }
    R.size[0] = (int)(unsigned)std::ceil(std::fabs(mx.y - mn.y) / lng);
    R.size[1] = (int)(unsigned)std::ceil(std::fabs(mx.z - mn.z) / lat);
    R.size[2] = (int)(unsigned)std::ceil(std::fabs(mx.x - mn.x) / lat);
    R.mn = mn;
    return R.size[0] <= max_rev[0] && R.size[1] <= max_rev[1] && R.size[2] <= max_rev[2];
}

}  // namespace

void ee_beamlet_free(void* ws) {
    if (!ws) return;
    BlWork* W = (BlWork*)ws;
    W->release();
    delete W;
}

// Beamlet columns of one beam (dosecalc-beamlet radconvolveTexture,
// nvbbRayConvolve_host.cu:444-1330, one beam).  Outputs stay in the
// workspace; `out` receives device pointers.
int ee_beamlet_run(const EeParams& P, const EeRayConst* rays, cudaStream_t s, void** ws, const EeBeamletOptions& opt,
                   const ee_beam& beam, const EeBeamSpec& S, const float* fluence_host, float thresh, ee_csr* out) {
    if (!*ws) *ws = new BlWork();
    BlWork& W = *(BlWork*)*ws;
    std::memset(out, 0, sizeof(*out));
    W.nnz = 0;
    W.ncols = 0;
    const int fx = beam.fmap_size[0], fy = beam.fmap_size[1];
    // BEAM::reconfigure in FP32 (beam.cpp:300-321)
    const float PI_F = 3.14159265358979323846f;
    float az = fmodf(beam.azimuth, 2 * PI_F), zen = fmodf(beam.zenith, 2 * PI_F);
    auto close = [](float a, float b) { return fabsf(b - a) <= 1e-6f; };
    if (!close(zen, 0.f) && (close(az, 0.f) || close(az, PI_F))) zen = 0.f;
    const float coll = beam.coll;
    const v3 iso = {beam.isocenter[0], beam.isocenter[1], beam.isocenter[2]};
    const v3 src = inv_rot_beam({0.f, -beam.sad, 0.f}, az, zen, 0.f) + iso;
    const v3 voxel = {P.voxel[0], P.voxel[1], P.voxel[2]}, start = {P.start[0], P.start[1], P.start[2]};
    const v3 bb0 = {(float)P.bb0[0], (float)P.bb0[1], (float)P.bb0[2]}, bbs = {(float)P.bbs[0], (float)P.bbs[1], (float)P.bbs[2]};
    const v3 vs = {P.lat, P.lng, P.lat};

    // active beamlets and anchors (host.cu:573-649)
    std::vector<Beamlet> bl;
    for (int i = 0; i < fx * fy; i++)
        if (fluence_host[i] > 0.f) {
            Beamlet B{};
            B.fidx = i;
            if (!anchors(B, src, iso, i, beam.beamlet_size[0], beam.beamlet_size[1], fx, fy, voxel, start, bb0, bbs, az,
                         zen, coll)) {
                char m[160];
                snprintf(m, sizeof(m), "failed to determine beamlet anchor coordinates for beamlet #%d", i);
                return ee_internal_fail(EE_ERR_INVALID_ARG, m);
            }
            bl.push_back(B);
        }
    const int n = (int)bl.size();
    W.ncols = n;
    BL_CUDA(W.out_colptr.ensure((size_t)n + 1));
    BL_CUDA(cudaMemsetAsync(W.out_colptr.p, 0, sizeof(long long) * ((size_t)n + 1), s));
    BL_CUDA(W.out_bidx.ensure(std::max(n, 1)));
    out->nbeamlets = n;
    out->beamlet_index = W.out_bidx.p;
    out->col_ptr = W.out_colptr.p;
    if (n == 0) return EE_OK;
    {
        std::vector<int> h(n);
        for (int i = 0; i < n; i++) h[i] = bl[i].fidx;
        BL_CUDA(cudaMemcpyAsync(W.out_bidx.p, h.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s));
        BL_CUDA(cudaStreamSynchronize(s));
    }
    float max_len = 0.f, msx = 0.f, msy = 0.f;
    for (auto& B : bl) {
        max_len = std::max(max_len, B.length);
        const float r = len(B.last - src), q = len(B.biso - src);
        msx = std::max(msx, beam.beamlet_size[0] * r / q);
        msy = std::max(msy, beam.beamlet_size[1] * r / q);
    }
    // pillar size: beamlet + 2 kernel extents + a wall, rounded up to whole
    // REV voxels, + the buffers (host.cu:651-662)
    const float ke = opt.kernel_extent;
    const float psl = max_len + 2.f * ke + BL_WALL * vs.y;
    const float ptx = msx + 2.f * ke + BL_WALL * vs.x, pty = msy + 2.f * ke + BL_WALL * vs.x;
    const v3 expand = vs - v3{fmodf(ptx, vs.x), fmodf(psl, vs.y), fmodf(pty, vs.z)};
    const v3 psize = v3{ptx, psl, pty} + expand + vs * (2.f * (float)BL_BUF);
    const int pd[3] = {(int)(psize.x / vs.x), (int)(psize.y / vs.y), (int)(psize.z / vs.z)};
    std::vector<v3> pstart(n);
    std::vector<float> Ms(9 * n), Mis(9 * n);
    for (int i = 0; i < n; i++) {
        const Beamlet& B = bl[i];
        v3 g = {-0.5f * (psize.x + BL_WALL * vs.x), -0.5f * (psize.y - B.length + BL_WALL * vs.y),
                -0.5f * (psize.z + BL_WALL * vs.z)};
        g = inv_rot_beam(inv_rot_beamlet(g, B.th, B.ph), az, zen, coll);
        pstart[i] = B.first + g;
        matrix([&](v3 v) { return inv_rot_beam(inv_rot_beamlet(v, B.th, B.ph), az, zen, coll); }, &Ms[9 * i]);
        matrix([&](v3 v) { return rot_beamlet(rot_beam(v, az, zen, coll), B.th, B.ph); }, &Mis[9 * i]);
    }

    // batching: the fewest batches whose REV arrays all fit max_rev
    // (ArraySizeError re-batching, host.cu:805-819)
    const int nrays = P.nrays;
    int nb = 1;
    std::vector<std::vector<RevBox>> revs;
    for (;; nb++) {
        if (nb > 100) return ee_internal_fail(EE_ERR_REV_SIZE, "beamlet batches exceed the REV size limit");
        std::vector<int> bs = batch_sizes(n, nb);
        revs.assign(nb, std::vector<RevBox>(nrays));
        bool ok = true;
        for (int k = 0; k < nb && ok; k++) {
            const int npx = (int)ceil(sqrt(float(bs[k])));
            const int npz = (int)ceil(float(bs[k]) / npx);
            const v3 gsize = v3{(float)(npx * pd[0] + BL_WALL), (float)(pd[1] + BL_WALL), (float)(npz * pd[2] + BL_WALL)} * vs;
            for (int r = 0; r < nrays && ok; r++) ok = find_rev(gsize, rays[r].th, rays[r].ph, P.lat, P.lng, opt.max_rev, revs[k][r]);
        }
        if (ok) break;
    }
    std::vector<int> bsz = batch_sizes(n, nb);
    for (int k = 0; k < nb; k++)
        for (int r = 0; r < nrays; r++)
            if (revs[k][r].size[0] > EE_MAX_LINE)
                return ee_internal_fail(EE_ERR_REV_SIZE, "size of rev (x-dim) exceeds maximum #threads allowed");

    BL_CUDA(W.spec.ensure(1));
    BL_CUDA(cudaMemcpyAsync(W.spec.p, &S, sizeof(S), cudaMemcpyHostToDevice, s));
    BL_CUDA(W.fluence.ensure((size_t)fx * fy));
    BL_CUDA(cudaMemcpyAsync(W.fluence.p, fluence_host, sizeof(float) * fx * fy, cudaMemcpyHostToDevice, s));
    BL_CUDA(W.status.ensure(1));
    BL_CUDA(cudaMemsetAsync(W.status.p, 0, sizeof(int), s));

    int first = 0;
    for (int k = 0; k < nb; k++) {
        const int m = bsz[k];
        BlGrid G{};
        G.n = m;
        G.npx = (int)ceil(sqrt(float(m)));
        G.npz = (int)ceil(float(m) / G.npx);
        for (int a = 0; a < 3; a++) G.pd[a] = pd[a];
        G.rpd[0] = 1.f / (float)pd[0];
        G.rpd[1] = 1.f / (float)pd[2];
        G.gd[0] = G.npx * pd[0] + BL_WALL;
        G.gd[1] = pd[1] + BL_WALL;
        G.gd[2] = G.npz * pd[2] + BL_WALL;
        G.vs[0] = vs.x; G.vs[1] = vs.y; G.vs[2] = vs.z;
        G.kr[0] = 0.5f * P.radii[0];
        for (int r = 1; r < P.nradii; r++) G.kr[r] = 0.5f * (P.radii[r] + P.radii[r - 1]);
        G.kern_extent = ke;
        // pillar table with the calc-bbox AABB of each usable region
        std::vector<BlPillar> pil(m);
        long long rows = 0;
        for (int i = 0; i < m; i++) {
            BlPillar& Q = pil[i];
            const int gi = first + i;
            std::memcpy(Q.M, &Ms[9 * gi], sizeof(Q.M));
            std::memcpy(Q.Mi, &Mis[9 * gi], sizeof(Q.Mi));
            Q.ps[0] = pstart[gi].x; Q.ps[1] = pstart[gi].y; Q.ps[2] = pstart[gi].z;
            Q.fidx = bl[gi].fidx;
            {
                // corner rays of the beamlet's fluence-map cell in pillar
                // index coordinates, ip = Mi ((p - ps) / vs)
                const int bx = Q.fidx % fx, by = Q.fidx / fx;
                const v3 ps = pstart[gi];
                auto to_pil = [&](v3 p) {
                    const v3 q = (p - ps) * v3{1.f / vs.x, 1.f / vs.y, 1.f / vs.z};
                    const float* Mi = Q.Mi;
                    return v3{Mi[0] * q.x + Mi[1] * q.y + Mi[2] * q.z, Mi[3] * q.x + Mi[4] * q.y + Mi[5] * q.z,
                              Mi[6] * q.x + Mi[7] * q.y + Mi[8] * q.z};
                };
                const v3 a = to_pil(src);
                for (int c = 0; c < 4; c++) {
                    const float cx = beam.beamlet_size[0] * (-0.5f * fx + bx + (c & 1));
                    const float cz = beam.beamlet_size[1] * (-0.5f * fy + by + (c >> 1));
                    const v3 corner = iso + inv_rot_beam({cx, 0.f, cz}, az, zen, coll);
                    const v3 e = to_pil(corner) - a;
                    const float sy = std::fabs(e.y) > 1e-12f ? e.y : 1e-12f;
                    Q.sx[c] = e.x / sy;
                    Q.sz[c] = e.z / sy;
                    Q.ex[c] = a.x - Q.sx[c] * a.y;
                    Q.ez[c] = a.z - Q.sz[c] * a.y;
                }
            }
            Q.ix = i % G.npx;
            Q.iz = i / G.npx;
            double lo[3] = {1e30, 1e30, 1e30}, hi[3] = {-1e30, -1e30, -1e30};
            for (int c = 0; c < 8; c++) {
                double u[3];
                for (int a = 0; a < 3; a++)
                    u[a] = (((c >> a) & 1) ? (double)(pd[a] - BL_BUF) : (double)(BL_WALL + BL_BUF)) - 0.5;
                for (int a = 0; a < 3; a++) {
                    double g = Q.ps[a];
                    for (int b2 = 0; b2 < 3; b2++) g += (double)Q.M[3 * a + b2] * u[b2] * (double)(b2 == 1 ? vs.y : vs.x);
                    double t = (g - (double)P.start[a]) / (double)P.voxel[a] - (double)P.bb0[a];
                    lo[a] = std::min(lo[a], t);
                    hi[a] = std::max(hi[a], t);
                }
            }
            for (int a = 0; a < 3; a++) {
                int l = std::max(0, (int)std::floor(lo[a]) - 1), h = std::min(P.bbs[a] - 1, (int)std::ceil(hi[a]) + 1);
                Q.b0[a] = l;
                Q.bn[a] = std::max(0, h - l + 1);
            }
            Q.row0 = rows;
            rows += (long long)Q.bn[1] * Q.bn[2] * (Q.bn[0] > 0 ? 1 : 0);
            if (Q.bn[0] == 0) Q.bn[1] = Q.bn[2] = 0;
        }
        BL_CUDA(W.pil.ensure(m));
        BL_CUDA(cudaMemcpyAsync(W.pil.p, pil.data(), sizeof(BlPillar) * m, cudaMemcpyHostToDevice, s));
        const long long npk = (long long)G.gd[0] * G.gd[1] * G.gd[2];
        BL_CUDA(W.packed.ensure(npk));
        BL_CUDA(cudaMemsetAsync(W.packed.p, 0, sizeof(float) * npk, s));
        long long rmax = 1;
        for (int r = 0; r < nrays; r++)
            rmax = std::max(rmax, (long long)revs[k][r].size[0] * revs[k][r].size[1] * revs[k][r].size[2]);
        if (rmax >= (1ll << 31) || npk >= (1ll << 31))
            return ee_internal_fail(EE_ERR_REV_SIZE, "beamlet REV / packed grid exceeds 2^31 samples");
        // sources of a pillar and direction: lattice points of spacing 1 in
        // the footprint's prism, so at most the volume of the prism widened by
        // half a cell diagonal each way
        double nsrc = 0;
        for (int i = 0; i < m; i++) {
            double w[2] = {0, 0};
            for (int e = 0; e < 2; e++) {
                const double y = e ? pd[1] : 0;
                double lo[2] = {1e30, 1e30}, hi[2] = {-1e30, -1e30};
                for (int c = 0; c < 4; c++) {
                    const double q[2] = {pil[i].ex[c] + pil[i].sx[c] * y, pil[i].ez[c] + pil[i].sz[c] * y};
                    for (int a = 0; a < 2; a++) {
                        lo[a] = std::min(lo[a], q[a]);
                        hi[a] = std::max(hi[a], q[a]);
                    }
                }
                for (int a = 0; a < 2; a++) w[a] = std::max(w[a], std::min(hi[a] - lo[a], (double)pd[2 * a]));
            }
            nsrc += (w[0] + 2.0) * (w[1] + 2.0) * (pd[1] + 2.0);
        }
        // directions in groups whose buffers fit the scratch budget: the REV
        // arrays, flags and bits of the lines, the lists of sources and lines
        for (int r0 = 0; r0 < nrays;) {
            int r1 = r0;
            long long samples = 0, ints = 2, nlines = 0, maxL = 1, bytes = 0;
            for (; r1 < nrays; r1++) {
                const int* z = revs[k][r1].size;
                const long long lines = (long long)z[1] * z[2], n = lines * z[0], flags = lines * (1 + (z[0] + 31) / 32);
                const long long more = 4 * (n + flags) + (long long)sizeof(int2) * ((long long)nsrc + 1 + lines) +
                                       (long long)sizeof(BlRayDev) + (long long)sizeof(float4) * m;
                if (r1 > r0 && bytes + more > opt.scratch_bytes) break;
                bytes += more;
                samples += n;
                ints += flags;
                nlines += lines;
                maxL = std::max<long long>(maxL, z[0]);
            }
            const int ng = r1 - r0;
            BlQueue Qu{};
            Qu.cap = (int)std::min(nsrc * ng, 2147483647.0);
            BL_CUDA(W.revd.ensure(std::max(samples, 1ll)));
            BL_CUDA(W.lines.ensure(ints));
            BL_CUDA(W.queue.ensure(Qu.cap));
            BL_CUDA(W.line_list.ensure(std::max(nlines, 1ll)));
            BL_CUDA(W.rays.ensure(ng));
            BL_CUDA(W.band.ensure((size_t)ng * m));
            std::vector<BlRayDev> hr(ng);
            long long off = 0, ioff = 2;
            for (int r = r0; r < r1; r++) {
                const RevBox& RB = revs[k][r];
                BlRayDev& R = hr[r - r0];
                std::memset(&R, 0, sizeof(R));
                for (int a = 0; a < 3; a++) R.rev[a] = RB.size[a];
                R.rs[0] = RB.mn.x; R.rs[1] = RB.mn.y; R.rs[2] = RB.mn.z;
                R.rcp[0] = 1.f / vs.x; R.rcp[1] = 1.f / vs.y; R.rcp[2] = 1.f / vs.z;
                std::memcpy(R.MK, rays[r].MK, sizeof(R.MK));
                std::memcpy(R.MKi, rays[r].MKi, sizeof(R.MKi));
                const int kw = r % (P.ntheta / 2);
                R.row_f = kw;
                R.row_r = P.ntheta - kw - 1;
                const long long lines = (long long)R.rev[1] * R.rev[2];
                R.words = (R.rev[0] + 31) / 32;
                R.dose = W.revd.p + off;
                R.flag = W.lines.p + ioff;
                R.bits = (unsigned*)(R.flag + lines);
                off += lines * R.rev[0];
                ioff += lines * (1 + R.words);
            }
            BL_CUDA(cudaMemcpyAsync(W.rays.p, hr.data(), sizeof(BlRayDev) * ng, cudaMemcpyHostToDevice, s));
            BL_CUDA(cudaMemsetAsync(W.lines.p, 0, sizeof(int) * ints, s));
            Qu.nsrc = W.lines.p;
            Qu.nlines = W.lines.p + 1;
            Qu.src = W.queue.p;
            Qu.line = W.line_list.p;
            const int slices = ee_bl_source_slices(nsrc / m / (pd[1] + 2.0), (long long)m * ng * (pd[1] / 32 + 1));
            k_bl_sources<<<dim3(m, (pd[1] / 32 + 1) * slices / BL_SRC_WARPS + 1, ng), BL_SRC_WARPS * 32, 0, s>>>(
                W.spec.p, G, W.pil.p, W.rays.p, Qu, slices, W.band.p, W.status.p);
            BL_CUDA(cudaGetLastError());
            k_bl_terma<<<152 * 8, 256, 0, s>>>(P, W.spec.p, G, W.pil.p, W.rays.p, W.fluence.p, Qu, W.status.p);
            BL_CUDA(cudaGetLastError());
            const size_t smem = sizeof(float) * (2 * EE_MAX_RADII + BL_BINS + (size_t)P.ntheta * P.nradii +
                                                 (size_t)BL_WARPS * bl_walk_floats((int)maxL));
            if (smem > 48 * 1024)
                BL_CUDA(cudaFuncSetAttribute(k_bl_walk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            k_bl_walk<<<(unsigned)std::min<long long>((nlines + BL_WARPS - 1) / BL_WARPS + 1, 152 * 16), BL_WARPS * 32,
                        smem, s>>>(P, G, W.pil.p, W.rays.p, Qu, (int)maxL);
            BL_CUDA(cudaGetLastError());
            const int used[2] = {pd[0] - 2 * BL_BUF - BL_WALL + 2, pd[2] - 2 * BL_BUF - BL_WALL + 2};
            if (used[0] > 0 && used[1] > 0) {
                k_bl_gather<<<dim3(G.npx * used[0], G.npz * used[1]), BL_GATHER_BLOCK, 0, s>>>(G, W.rays.p, ng, W.band.p,
                                                                                             W.packed.p);
                BL_CUDA(cudaGetLastError());
            }
            r0 = r1;
        }
        // unpack + threshold + CSR
        BL_CUDA(W.len.ensure(std::max(rows, 1ll)));
        BL_CUDA(W.xs.ensure(std::max(rows, 1ll)));
        BL_CUDA(W.cnt.ensure(std::max(rows, 1ll)));
        BL_CUDA(W.seg.ensure(std::max(rows, 1ll)));
        BL_CUDA(W.off.ensure(std::max(rows, 1ll)));
        BL_CUDA(W.colmax.ensure(m));
        BL_CUDA(cudaMemsetAsync(W.colmax.p, 0, sizeof(int) * m, s));
        long long nvals = 0, nnz_b = 0;
        if (rows > 0) {
            k_bl_rows<<<dim3(64, m), 256, 0, s>>>(P, G, W.pil.p, W.len.p, W.xs.p);
            BL_CUDA(cudaGetLastError());
            BL_CUDA(scan_excl(W, W.len.p, nullptr, rows, W.seg.p, 0, s));
            BL_CUDA(scan_total(W.seg.p, W.len.p, rows, s, &nvals));
            BL_CUDA(W.vals.ensure(std::max(nvals, 1ll)));
            const unsigned wblocks = (unsigned)std::min<long long>((rows + 7) / 8, 152ll * 64);
            k_bl_values<<<wblocks, 256, 0, s>>>(P, G, W.pil.p, W.packed.p, rows, W.len.p, W.xs.p, W.seg.p, W.vals.p,
                                                W.colmax.p);
            BL_CUDA(cudaGetLastError());
            k_bl_count<<<wblocks, 256, 0, s>>>(G, W.pil.p, rows, W.len.p, W.seg.p, W.vals.p, W.colmax.p, thresh, W.cnt.p);
            BL_CUDA(cudaGetLastError());
            BL_CUDA(scan_excl(W, W.cnt.p, nullptr, rows, W.off.p, 0, s));
            BL_CUDA(scan_total(W.off.p, W.cnt.p, rows, s, &nnz_b));
            BL_CUDA(W.out_rows.grow_keep((size_t)(W.nnz + nnz_b), (size_t)W.nnz, s));
            BL_CUDA(W.out_vals.grow_keep((size_t)(W.nnz + nnz_b), (size_t)W.nnz, s));
            k_bl_emit<<<wblocks, 256, 0, s>>>(P, G, W.pil.p, rows, W.len.p, W.xs.p, W.seg.p, W.vals.p, W.colmax.p,
                                              thresh, W.off.p, W.nnz, W.out_rows.p, W.out_vals.p);
            BL_CUDA(cudaGetLastError());
        }
        k_bl_colptr<<<(m + 1 + 127) / 128, 128, 0, s>>>(W.pil.p, m, W.off.p, W.cnt.p, rows, W.nnz,
                                                       W.out_colptr.p + first);
        BL_CUDA(cudaGetLastError());
        W.nnz += nnz_b;
        first += m;
    }
    int st = 0;
    BL_CUDA(cudaMemcpyAsync(&st, W.status.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    BL_CUDA(cudaStreamSynchronize(s));
    if (st & 1) return ee_internal_fail(EE_ERR_SIDDON_ITER, "Siddon ray trace hit its iteration cap");
    if (st & BL_CAPACITY) return ee_internal_fail(EE_ERR_CAPACITY, "beamlet source queue too short");
    out->nnz = W.nnz;
    out->row_index = W.out_rows.p;
    out->value = W.out_vals.p;
    out->col_ptr = W.out_colptr.p;
    return EE_OK;
}
