// ee_kernels.cu -- sm_103a kernels of the CCCS beam-dose engine.
//
// Stages per beam (forward):
//   k_terma     Siddon radiological path + polyenergetic TERMA of the voxels
//               of the beam's TERMA box, with the crop-box min/max reduction.
//               Restates CCCS/DoseCalcAlgo/cudaSiddon.cu:20-308 and the host
//               extent scan CCCS/dosecalc-beam/nvbbRayConvolve_host.cu:429-499.
//   k_geometry  crop box -> BEV box, findREV for every cone, affine maps
//               (host.cu:460-499, :75-155).
//   k_cone_*    resample of density and TERMA along the rotated lines
//               (nvbbRayConvolve_device.cu:11-80) and the bidirectional line
//               convolution (device.cu:87-218): EE_KERNEL_EXP one lane per line
//               over lists of line tiles (k_cone_tiles, k_cone_lane),
//               EE_KERNEL_TABLE window sums of two lines per warp (k_cone_tab),
//               the step-by-step walk and the allocation-free path one warp per
//               line (k_cone).
//   k_gather    patient voxel <- sum over cones of the trilinear REV dose
//               (device.cu:222-261), all cones of all beams of the batch in
//               registers, one write per voxel.
// Adjoint: k_gather_T (scatter), k_cone_T_* (reverse scans + TERMA scatter),
// k_terma_T (per-beamlet reduction).
#include "ee_internal.h"
#include <algorithm>
#include <cfloat>
#include <cstddef>
#include <mutex>

#include "ee_device.cuh"

namespace {

// Crop-box reduction (host.cu:442-459): min/max of the BEV indices `bi` of a
// warp's voxels with non-zero TERMA (nz) as ordered-int keys, merged into the
// beam's keys by one lane, without a block barrier.
__device__ __forceinline__ void merge_crop_box(EeBeamGeom& G, bool nz, f3 bi, bool cap) {
    int kmin0 = nz ? f2key(bi.x) : INT_MAX, kmin1 = nz ? f2key(bi.y) : INT_MAX, kmin2 = nz ? f2key(bi.z) : INT_MAX;
    int kmax0 = nz ? f2key(bi.x) : INT_MIN, kmax1 = nz ? f2key(bi.y) : INT_MIN, kmax2 = nz ? f2key(bi.z) : INT_MIN;
    const unsigned cnt = __popc(__ballot_sync(FULL, nz));
    const bool anycap = __any_sync(FULL, cap);
    if (cnt == 0 && !anycap) return;
    kmin0 = __reduce_min_sync(FULL, kmin0);
    kmin1 = __reduce_min_sync(FULL, kmin1);
    kmin2 = __reduce_min_sync(FULL, kmin2);
    kmax0 = __reduce_max_sync(FULL, kmax0);
    kmax1 = __reduce_max_sync(FULL, kmax1);
    kmax2 = __reduce_max_sync(FULL, kmax2);
    if ((threadIdx.x & 31) == 0) {
        if (cnt > 0) {
            atomicMin(&G.key_min[0], kmin0); atomicMin(&G.key_min[1], kmin1); atomicMin(&G.key_min[2], kmin2);
            atomicMax(&G.key_max[0], kmax0); atomicMax(&G.key_max[1], kmax1); atomicMax(&G.key_max[2], kmax2);
            atomicAdd(&G.nnz, cnt);
        }
        if (anycap) atomicExch(&G.status, 7 /* EE_ERR_SIDDON_ITER */);
    }
}

// TERMA without supersampling.  A block takes ITEMS of the box's voxels brick by
// brick (4x4x4, ee_brick_vol).  A voxel needs a ray trace when it has a beamlet
// (beamlet_of, cudaSiddon.cu:143-165) whose fluence is positive, or any beamlet
// when the unit TERMA is kept for the adjoint; the rest are written at once.  The
// box is the field's axis-aligned hull, so warps at the field's edge hold both
// kinds: the voxels to trace are first gathered into a shared list, a warp's in
// box order, and the warps take 32 of them at a time, so the Siddon loops run
// with full warps.  Each voxel's arithmetic is unchanged.  The crop box
// (host.cu:442-459) is reduced from the traced voxels with non-zero TERMA:
// min/max of BEV indices as ordered-int keys, one merge per 32 voxels.
// Bound by the texture unit's data stage, where the rays' uneven lengths leave
// it busy: 96 beams of 8^2..40^2 beamlets on 200 x 200 x 160 9.42 ms with 256
// threads per block of 256 voxels, 8.99 with 128 of 128, 7.8 with two fetches in
// flight, 6.3 with 512 voxels per 128 threads (ee_launch_terma: the rule).  40
// resident warps per SM: 48 registers, no spills.
constexpr int TERMA_BLOCK = 128;

template <int ITEMS>
__global__ void __launch_bounds__(TERMA_BLOCK, 1280 / TERMA_BLOCK)
    k_terma(EeParams P, const EeBeamSpec* __restrict__ specs, EeBeamGeom* __restrict__ geoms,
            const float* __restrict__ fluence, float* __restrict__ terma, float* __restrict__ unit,
            int* __restrict__ bl_idx) {
    __shared__ int s_bl[ITEMS], s_n, s_next;
    __shared__ float s_fl[ITEMS];
    __shared__ unsigned short s_v[ITEMS];
    const int b = blockIdx.z;
    const EeBeamSpec& S = specs[b];
    const long long bvol = ee_brick_vol(S.tn);
    const long long vb = (long long)blockIdx.x * ITEMS;
    if (vb >= bvol) return;
    const int nbx = (S.tn[0] + 3) >> 2, nby = (S.tn[1] + 3) >> 2;
    // box indices of bricked box element v
    auto coords = [&](long long v, int& xr, int& yr, int& zr) {
        const long long brick = v >> 6;
        const int w = (int)(v & 63);
        const long long bxy = brick % ((long long)nbx * nby);
        xr = (int)(bxy % nbx) * 4 + (w & 3);
        yr = (int)(bxy / nbx) * 4 + ((w >> 2) & 3);
        zr = (int)(brick / ((long long)nbx * nby)) * 4 + (w >> 4);
    };
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        s_n = 0;
        s_next = TERMA_BLOCK;
    }
    __syncthreads();
    // the list of voxels to trace, a warp's in box order
#pragma unroll 1
    for (int c = threadIdx.x; c < ITEMS; c += TERMA_BLOCK) {
        const long long v = vb + c;
        bool need = false;
        int bl = -1;
        float fl = 0.f;
        if (v < bvol) {
            int xr, yr, zr;
            coords(v, xr, yr, zr);
            // padding of the last bricks: never sampled, kept zero
            const bool inbox = xr < S.tn[0] && yr < S.tn[1] && zr < S.tn[2];
            if (inbox) {
                const int x = S.t0[0] + xr, y = S.t0[1] + yr, z = S.t0[2] + zr;
                const f3 vox = mk(P.start[0] + x * P.voxel[0], P.start[1] + y * P.voxel[1], P.start[2] + z * P.voxel[2]);
                bl = beamlet_of(S, vox);
                if (bl == -2) bl = beamlet_of_fp64(P, S, x, y, z);
                if (bl >= 0) {
                    fl = __ldg(fluence + S.fl_off + bl);
                    need = fl > 0.f || unit;
                }
            }
            if (!need) {
                terma[S.t_off + v] = 0.f;
                if (unit) unit[S.t_off + v] = 0.f;
                if (bl_idx) bl_idx[S.t_off + v] = bl;
            }
        }
        const unsigned m = __ballot_sync(FULL, need);
        int p = 0;
        if (lane == 0 && m) p = atomicAdd(&s_n, __popc(m));
        p = __shfl_sync(FULL, p, 0) + __popc(m & ((1u << lane) - 1u));
        if (need) {
            s_v[p] = (unsigned short)c;
            s_bl[p] = bl;
            s_fl[p] = fl;
        }
    }
    __syncthreads();
    const int total = s_n;
    // 32 voxels to each warp, then the next 32 to the warp that is done
#pragma unroll 1
    for (int k0 = threadIdx.x & ~31; k0 < total;) {
        const int k = k0 + lane;
        bool nz = false, cap = false;
        f3 bi = mk(0.f, 0.f, 0.f);
        if (k < total) {
            const long long vt = vb + s_v[k];
            int xr, yr, zr;
            coords(vt, xr, yr, zr);
            const int x = S.t0[0] + xr, y = S.t0[1] + yr, z = S.t0[2] + zr;
            const f3 vox = mk(P.start[0] + x * P.voxel[0], P.start[1] + y * P.voxel[1], P.start[2] + z * P.voxel[2]);
            const f3 src = ld3(S.src);
            const float flt = s_fl[k];
            const float rpl = siddon_rpl(P, vox, src, cap);
            const float u = terma_per_fluence(P, rpl, vox, src, S.sad);
            const float t = flt > 0.f ? flt * u : 0.f;
            terma[S.t_off + vt] = t;
            if (unit) unit[S.t_off + vt] = u;
            if (bl_idx) bl_idx[S.t_off + vt] = s_bl[k];
            if (t != 0.f) {
                nz = true;
                // crop box works on calc-bbox-relative indices (host.cu:445-448)
                bi = mv(S.MB, mk((float)(x - P.bb0[0]), (float)(y - P.bb0[1]), (float)(z - P.bb0[2])));
            }
        }
        merge_crop_box(geoms[b], nz, bi, cap);
        if (ITEMS == TERMA_BLOCK) return;
        if (lane == 0) k0 = atomicAdd(&s_next, 32);
        k0 = __shfl_sync(FULL, k0, 0);
    }
}

// TERMA with supersampling (ss > 1, cudaSiddon.cu:248-258, 297-306): each
// voxel's TERMA is the mean over ss^3 sub-voxel centres, each with its own
// beamlet lookup and ray trace, summed x fastest.  A block takes one brick of
// the box (4x4x4 voxels) and walks its 64 ss^3 centres in voxel-major order,
// TS_ITEMS at a time: the centres to trace are gathered into a shared list, a
// thread traces one centre, and a thread per voxel adds the results in the
// centres' order.  Neighbouring lanes then trace rays a fraction of a voxel
// apart, so a warp's density fetches share their texels, which is what the
// texture unit is bound by: 4 beams at ss = 3 8.00 ms with a thread per voxel
// that traces its 27 centres in turn, 6.29 ms here, 5.80 with two fetches in
// flight, 5.60 with 2048 centres at a time, which hold all of ss = 3, instead of
// 1024 (ss = 2: 2.01 -> 1.96; 32 centres at a time to the next free warp: the
// same).  (Unit TERMA and beamlets are not kept: k_terma_T_ss recomputes the
// sub-voxel beamlets.)
constexpr int TS_ITEMS = 2048;

__global__ void __launch_bounds__(256, 4) k_terma_ss(EeParams P, const EeBeamSpec* __restrict__ specs,
                                                     EeBeamGeom* __restrict__ geoms, const float* __restrict__ fluence,
                                                     float* __restrict__ terma, float* __restrict__ unit,
                                                     int* __restrict__ bl_idx) {
    __shared__ float s_val[TS_ITEMS];       // fluence of a listed centre, then its fluence x unit TERMA
    __shared__ unsigned short s_list[TS_ITEMS];
    __shared__ int s_n;
    const int b = blockIdx.z;
    const EeBeamSpec& S = specs[b];
    const int nbx = (S.tn[0] + 3) >> 2, nby = (S.tn[1] + 3) >> 2;
    const long long brick = blockIdx.x;
    if (brick >= (ee_brick_vol(S.tn) >> 6)) return;
    const long long bxy = brick % ((long long)nbx * nby);
    const int bx = (int)(bxy % nbx) * 4, by = (int)(bxy / nbx) * 4, bz = (int)(brick / ((long long)nbx * nby)) * 4;
    const int ss = P.ss, nsub = ss * ss * ss;
    const float sv0 = P.voxel[0] / (float)ss, sv1 = P.voxel[1] / (float)ss, sv2 = P.voxel[2] / (float)ss;
    const f3 src = ld3(S.src);
    const int t = threadIdx.x, lane = t & 31;
    // centre `item` of the brick (voxel-major); false outside the box
    auto centre = [&](int item, f3& p) {
        const int w = item / nsub, ii = item - w * nsub;
        const int xr = bx + (w & 3), yr = by + ((w >> 2) & 3), zr = bz + (w >> 4);
        const int sx = ii % ss, sy = (ii / ss) % ss, sz = ii / (ss * ss);
        p = mk(P.start[0] + ((float)(S.t0[0] + xr) - 0.5f) * P.voxel[0] + ((float)sx + 0.5f) * sv0,
               P.start[1] + ((float)(S.t0[1] + yr) - 0.5f) * P.voxel[1] + ((float)sy + 0.5f) * sv1,
               P.start[2] + ((float)(S.t0[2] + zr) - 0.5f) * P.voxel[2] + ((float)sz + 0.5f) * sv2);
        return xr < S.tn[0] && yr < S.tn[1] && zr < S.tn[2];
    };
    float acc = 0.f;  // voxel t of the brick (t < 64)
    bool cap = false;
    for (int i0 = 0; i0 < 64 * nsub; i0 += TS_ITEMS) {
        const int n = min(TS_ITEMS, 64 * nsub - i0);
        if (t == 0) s_n = 0;
        __syncthreads();
        for (int k = t; k < ((n + 255) & ~255); k += 256) {
            float fl = 0.f;
            f3 p;
            if (k < n && centre(i0 + k, p)) {
                int bs = beamlet_of(S, p);
                if (bs == -2) bs = beamlet_point_fp64(S, (double)p.x, (double)p.y, (double)p.z);
                if (bs >= 0) fl = __ldg(fluence + S.fl_off + bs);
            }
            const bool need = fl > 0.f;
            s_val[k] = need ? fl : 0.f;
            const unsigned m = __ballot_sync(FULL, need);
            int base = 0;
            if (lane == 0 && m) base = atomicAdd(&s_n, __popc(m));
            base = __shfl_sync(FULL, base, 0);
            if (need) s_list[base + __popc(m & ((1u << lane) - 1u))] = (unsigned short)k;
        }
        __syncthreads();
        const int nl = s_n;
        for (int k = t; k < nl; k += 256) {
            const int item = s_list[k];
            f3 p;
            centre(i0 + item, p);
            const float rpl = siddon_rpl(P, p, src, cap);
            s_val[item] *= terma_per_fluence(P, rpl, p, src, S.sad);
        }
        __syncthreads();
        if (t < 64) {
            const int lo = max(t * nsub - i0, 0), hi = min((t + 1) * nsub - i0, n);
            for (int k = lo; k < hi; k++) acc += s_val[k];
        }
        __syncthreads();
    }
    bool nz = false;
    f3 bi = mk(0.f, 0.f, 0.f);
    if (t < 64) {
        const float te = acc / (float)nsub;
        const long long o = S.t_off + brick * 64 + t;
        terma[o] = te;  // the padding of the box's last bricks is never sampled and stays zero
        if (unit) unit[o] = 0.f;
        if (bl_idx) bl_idx[o] = -1;
        nz = te != 0.f;
        // crop box works on calc-bbox-relative indices (host.cu:445-448)
        bi = mv(S.MB, mk((float)(S.t0[0] + bx + (t & 3) - P.bb0[0]), (float)(S.t0[1] + by + ((t >> 2) & 3) - P.bb0[1]),
                         (float)(S.t0[2] + bz + (t >> 4) - P.bb0[2])));
    }
    merge_crop_box(geoms[b], nz, bi, cap);
}

// The beam's field as seen by one cone's REV points.  A voxel has a beamlet
// only where its iso-plane projection falls inside the fluence-map rectangle
// (beamlet_of, cudaSiddon.cu:143-165): with diff = p - src, proj = dir.diff
// and u = MB_row.(diff - proj dir), the fluence coordinate is inside iff
// u + k proj >= 0 and k proj - u > 0, k = half the map's width / isodist, per
// BEV axis x and z.  Outside, TERMA is exactly zero (k_terma writes 0 where
// there is no beamlet) and the TERMA adjoint drops the voxel.  The four sides
// are linear in position, so they are affine forms of the REV point (i, tY,
// tZ); each is raised by its change over one voxel per axis (the trilinear
// corners of a sample; half a voxel more for supersampled centres) plus 0.05
// voxel and 1e-3 cm, far above the FP32 error of forms of about 100 cm.
__device__ __forceinline__ void field_forms(const EeParams& P, const EeBeamSpec& S, EeRayGeom& R) {
    const f3 vox = mk(P.voxel[0], P.voxel[1], P.voxel[2]);
    const f3 d0 = mk(P.start[0] + vox.x * R.G0[0] - S.src[0], P.start[1] + vox.y * R.G0[1] - S.src[1],
                     P.start[2] + vox.z * R.G0[2] - S.src[2]);
    const f3 dx = mk(vox.x * R.Gx[0], vox.y * R.Gx[1], vox.z * R.Gx[2]);
    const f3 dy = mk(vox.x * R.Gy[0], vox.y * R.Gy[1], vox.z * R.Gy[2]);
    const f3 dz = mk(vox.x * R.Gz[0], vox.y * R.Gz[1], vox.z * R.Gz[2]);
    const f3 dir = ld3(S.dir);
    R.front[0] = dot(dir, dx);
    R.front[1] = dot(dir, d0);
    R.front[2] = dot(dir, dy);
    R.front[3] = dot(dir, dz);
    const float reach = P.ss > 1 ? 1.55f : 1.05f;  // voxels from a sample to a centre that feeds it
    for (int a = 0; a < 2; a++) {
        const f3 m = ld3(S.MB + (a ? 6 : 0));
        const f3 g = m - dir * dot(m, dir);  // u = g . diff
        const float k = 0.5f * (float)S.fmap[a] * S.beamlet[a] / S.isodist;
        for (int sg = 0; sg < 2; sg++) {
            const f3 gl = g * (sg ? 1.f : -1.f) + dir * k;
            float* f = R.side[2 * a + sg];
            f[0] = dot(gl, dx);
            f[1] = dot(gl, d0) + reach * (fabsf(gl.x) * vox.x + fabsf(gl.y) * vox.y + fabsf(gl.z) * vox.z) + 1e-3f;
            f[2] = dot(gl, dy);
            f[3] = dot(gl, dz);
        }
    }
}

// The lines of a cone that the field can reach (ee_lit_planes).  A crop box
// holds the BEV origin whatever the field (host.cu:442: the maximum starts at
// FLT_MIN), so most of it can lie off the field: of the 1024-beam candidates'
// lines 46 % have no field span.  The field is raised as in field_forms and
// taken between the planes through the calc bbox's nearest and farthest
// corners, so the half-planes depend on the beam alone.  No bound where the
// frustum form does not hold: voxels that are not cubes (the BEV planes are
// then not normal to the beam) and a bbox that reaches the source.
__device__ bool lit_planes(const EeParams& P, const EeBeamSpec& S, const EeBeamGeom& G, EeRayGeom& R) {
    for (int k = 0; k < 4; k++) {
        R.lit[k][0] = R.lit[k][1] = 0.f;
        R.lit[k][2] = 1.f;
    }
    const float vox = P.voxel[0];
    if (P.voxel[1] != vox || P.voxel[2] != vox || !(S.dnear > 0.02f * S.isodist)) return false;
    const f3 src = ld3(S.src), dir = ld3(S.dir), start = ld3(P.start), off = ld3(G.lim_off);
    const float reach = P.ss > 1 ? 1.55f : 1.05f;
    float c[2][3], h[2][2];
    for (int e = 0; e < 2; e++) {
        const float D = e ? S.dfar + 4.f * vox : S.dnear - 4.f * vox;
        const f3 p = mv(S.MB, (src + dir * D - start) * (1.f / vox) - off);
        c[e][0] = p.x; c[e][1] = p.y; c[e][2] = p.z;
        for (int a = 0; a < 2; a++) {
            const f3 m = ld3(S.MB + (a ? 6 : 0));
            const f3 g = m - dir * dot(m, dir);
            const float k = 0.5f * (float)S.fmap[a] * S.beamlet[a] / S.isodist;
            float M = 0.f;
            for (int sg = 0; sg < 2; sg++) {
                const f3 gl = g * (sg ? 1.f : -1.f) + dir * k;
                M = fmaxf(M, reach * (fabsf(gl.x) + fabsf(gl.y) + fabsf(gl.z)) * vox + 1e-3f);
            }
            h[e][a] = (k * D + M) / vox;
        }
    }
    ee_lit_planes<float>(R.M, c, h, R.q0, R.lit);
    return true;
}

// The part of a cone's REV array that the gathers reach: the lines whose lit
// forms are at least EE_LIT_READ, and along them the crop box dilated as in
// line_read_span.  The cells outside it are neither written nor read (of the
// arrays' 84..142 cells per crop-box voxel a little over half remain), so more
// beams share a chunk.
__device__ void kept_part(const EeBeamGeom& G, EeRayGeom& R, bool bounded) {
    float lo[2] = {0.f, 0.f}, hi[2] = {(float)(R.rev[1] - 1), (float)(R.rev[2] - 1)};
    if (bounded) {
        float a[2], b[2];
        ee_lit_rect<float>(R.lit, -EE_LIT_READ, a, b);
        for (int i = 0; i < 2; i++) {
            lo[i] = fmaxf(lo[i], floorf(a[i] - 0.1f));
            hi[i] = fminf(hi[i], ceilf(b[i] + 0.1f));
        }
    }
    float fa = 0.f, fb = (float)(R.rev[0] - 1);
    for (int k = 0; k < 3; k++) {
        const float D = 2.05f + fabsf(R.Bx[k]) + fabsf(R.By[k]) + fabsf(R.Bz[k]), m = R.Bx[k];
        if (fabsf(m) < 1e-6f) continue;
        const float y = R.By[k], z = R.Bz[k];
        const float cmin = R.B0[k] + fminf(y * lo[0], y * hi[0]) + fminf(z * lo[1], z * hi[1]);
        const float cmax = R.B0[k] + fmaxf(y * lo[0], y * hi[0]) + fmaxf(z * lo[1], z * hi[1]);
        const float t0 = (-D - cmax) / m, t1 = ((float)G.bev[k] + D - cmin) / m;
        fa = fmaxf(fa, fminf(t0, t1));
        fb = fminf(fb, fmaxf(t0, t1));
    }
    const bool none = hi[0] < lo[0] || hi[1] < lo[1] || fb < fa - 4.f;
    const int i0 = max(0, (int)floorf(fa) - 4), i1 = min(R.rev[0] - 1, (int)ceilf(fb) + 4);
    R.so[0] = none ? 0 : i0 & ~3;
    R.sn[0] = none ? 0 : i1 - R.so[0] + 1;
    for (int i = 0; i < 2; i++) {
        R.so[1 + i] = none ? 0 : (int)lo[i] & ~3;
        R.sn[1 + i] = none ? 0 : (int)hi[i] - R.so[1 + i] + 1;
    }
    R.nlines = R.sn[1] * R.sn[2];
}

// Lit form k of the cone as an affine form of the crop-box-relative patient
// index (dx, dy, dz): >= 0 where one of the four lines around the voxel can be
// lit (a cell per axis added).
__device__ __forceinline__ float4 lit_voxel_form(const EeRayGeom& R, int k) {
    const float a = R.lit[k][0], b = R.lit[k][1];
    return make_float4(a * R.A[6] + b * R.A[0], a * R.A[7] + b * R.A[1], a * R.A[8] + b * R.A[2],
                       R.lit[k][2] + fabsf(a) + fabsf(b) - a * R.q0[2] - b * R.q0[0]);
}

__global__ void k_geom_init(const EeBeamSpec* __restrict__ specs, EeBeamGeom* g, int n) {
    int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n) return;
    for (int a = 0; a < 3; a++) { g[b].key_min[a] = f2key(FLT_MAX); g[b].key_max[a] = f2key(FLT_MIN); }
    g[b].nnz = 0;
    g[b].status = 0;
    // planned slot, or unbounded (the host sizes the arena after read-back)
    g[b].arena_off = specs[b].plan_off;
    g[b].arena_cap = specs[b].plan_cap;
}

// ------------------------------------------------------------- geometry --
// Crop box (host.cu:460-499) and findREV (host.cu:75-155) for every cone.
__global__ void k_geometry(EeParams P, const EeBeamSpec* __restrict__ specs, EeBeamGeom* __restrict__ geoms) {
    const int b = blockIdx.x;
    EeBeamGeom& G = geoms[b];
    const EeBeamSpec& S = specs[b];
    __shared__ int s_ok;
    if (threadIdx.x == 0) {
        int ok = (G.status == 0);
        if (ok && G.nnz == 0) { G.status = 3; ok = 0; }
        if (ok) {
            float pl = P.penumbra / P.lat, plg = P.penumbra / P.lng;
            float mn[3], mx[3];
            for (int a = 0; a < 3; a++) { mn[a] = key2f(G.key_min[a]); mx[a] = key2f(G.key_max[a]); }
            mn[0] -= pl; mn[1] -= plg; mn[2] -= pl;
            mx[0] += pl; mx[1] += plg; mx[2] += pl;
            for (int a = 0; a < 3; a++) {
                float s = snap_ceilf(fabsf(mx[a] - mn[a]));
                if (!(s > 0.f) || s >= 1000.f) { ok = 0; }
                G.bev[a] = ok ? (int)s : 0;
                G.bmin[a] = mn[a];
            }
            if (!ok) G.status = 3;
            f3 tmn = mv(S.MBi, mk(mn[0], mn[1], mn[2]));
            G.lim_min[0] = P.start[0] + (tmn.x + P.bb0[0]) * P.voxel[0];
            G.lim_min[1] = P.start[1] + (tmn.y + P.bb0[1]) * P.voxel[1];
            G.lim_min[2] = P.start[2] + (tmn.z + P.bb0[2]) * P.voxel[2];
            for (int a = 0; a < 3; a++) G.lim_off[a] = (G.lim_min[a] - P.start[a]) / P.voxel[a];
            G.v_beam = (long long)G.bev[0] * G.bev[1] * G.bev[2];
        }
        s_ok = ok;
    }
    __syncthreads();
    if (!s_ok) return;
    const f3 bd = mk(G.bev[0] * P.lat, G.bev[1] * P.lng, G.bev[2] * P.lat);
    for (int r = threadIdx.x; r < P.nrays; r += blockDim.x) {
        const EeRayConst& RC = P.rays[r];
        EeRayGeom& R = G.ray[r];
        float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {FLT_MIN, FLT_MIN, FLT_MIN};
        for (int c = 0; c < 8; c++) {
            f3 o = mv(RC.MK, mk(bd.x * (c & 1), bd.y * ((c >> 1) & 1), bd.z * ((c >> 2) & 1)));
            mn[0] = fminf(mn[0], o.x); mn[1] = fminf(mn[1], o.y); mn[2] = fminf(mn[2], o.z);
            mx[0] = fmaxf(mx[0], o.x); mx[1] = fmaxf(mx[1], o.y); mx[2] = fmaxf(mx[2], o.z);
        }
        int sz[3] = {(int)snap_ceilf(fabsf(mx[1] - mn[1]) / P.lng), (int)snap_ceilf(fabsf(mx[2] - mn[2]) / P.lat),
                     (int)snap_ceilf(fabsf(mx[0] - mn[0]) / P.lat)};
        bool bad = false;
        for (int a = 0; a < 3; a++) {
            if (P.max_rev[a] > 0 && sz[a] > P.max_rev[a]) bad = true;
            R.rev[a] = sz[a];
        }
        if (sz[0] > EE_MAX_LINE || sz[0] <= 0 || sz[1] <= 0 || sz[2] <= 0) bad = true;
        if (bad) atomicExch(&G.status, 4);
        f3 q0 = mk(mn[0] / P.lat, mn[1] / P.lng, mn[2] / P.lat);
        R.q0[0] = q0.x; R.q0[1] = q0.y; R.q0[2] = q0.z;
        // REV vector (tZ, tX, tY) + q0 -> BEV (inverseRotateKernel)
        f3 B0 = mv(RC.MKi, q0);
        f3 Bx = mk(RC.MKi[1], RC.MKi[4], RC.MKi[7]);  // column for tX (REV y)
        f3 By = mk(RC.MKi[2], RC.MKi[5], RC.MKi[8]);  // column for tY (REV z)
        f3 Bz = mk(RC.MKi[0], RC.MKi[3], RC.MKi[6]);  // column for tZ (REV x)
        f3 lo = mk(G.lim_off[0], G.lim_off[1], G.lim_off[2]);
        f3 G0 = lo + mv(S.MBi, B0), Gx = mv(S.MBi, Bx), Gy = mv(S.MBi, By), Gz = mv(S.MBi, Bz);
        R.B0[0] = B0.x; R.B0[1] = B0.y; R.B0[2] = B0.z;
        R.Bx[0] = Bx.x; R.Bx[1] = Bx.y; R.Bx[2] = Bx.z;
        R.By[0] = By.x; R.By[1] = By.y; R.By[2] = By.z;
        R.Bz[0] = Bz.x; R.Bz[1] = Bz.y; R.Bz[2] = Bz.z;
        R.G0[0] = G0.x; R.G0[1] = G0.y; R.G0[2] = G0.z;
        R.Gx[0] = Gx.x; R.Gx[1] = Gx.y; R.Gx[2] = Gx.z;
        R.Gy[0] = Gy.x; R.Gy[1] = Gy.y; R.Gy[2] = Gy.z;
        R.Gz[0] = Gz.x; R.Gz[1] = Gz.y; R.Gz[2] = Gz.z;
        for (int i = 0; i < 9; i++) R.M[i] = RC.MK[i];
        for (int i = 0; i < 3; i++)
            for (int j = 0; j < 3; j++)
                R.A[3 * i + j] = RC.MK[3 * i] * S.MB[j] + RC.MK[3 * i + 1] * S.MB[3 + j] + RC.MK[3 * i + 2] * S.MB[6 + j];
        for (int a = 0; a < 3; a++) {
            R.iB[a] = fabsf(R.Bx[a]) < 1e-6f ? 0.f : 1.f / R.Bx[a];
            R.iG[a] = fabsf(R.Gx[a]) < 1e-6f ? 0.f : 1.f / R.Gx[a];
        }
        field_forms(P, S, R);
        kept_part(G, R, lit_planes(P, S, G, R));
    }
    __syncthreads();
    if (threadIdx.x == 0 && G.status == 0) {
        // patient-index AABB of the crop box dilated by 2 BEV voxels
        float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        for (int c = 0; c < 8; c++) {
            f3 bc = mk((c & 1) ? G.bev[0] + 2.f : -2.f, ((c >> 1) & 1) ? G.bev[1] + 2.f : -2.f,
                       ((c >> 2) & 1) ? G.bev[2] + 2.f : -2.f);
            f3 t = mv(S.MBi, bc) + mk(G.lim_off[0], G.lim_off[1], G.lim_off[2]);
            lo[0] = fminf(lo[0], t.x); lo[1] = fminf(lo[1], t.y); lo[2] = fminf(lo[2], t.z);
            hi[0] = fmaxf(hi[0], t.x); hi[1] = fmaxf(hi[1], t.y); hi[2] = fmaxf(hi[2], t.z);
        }
        int x0 = max(P.bb0[0], (int)floorf(lo[0]) - 1), x1 = min(P.bb0[0] + P.bbs[0] - 1, (int)ceilf(hi[0]) + 1);
        int y0 = max(P.bb0[1], (int)floorf(lo[1]) - 1), y1 = min(P.bb0[1] + P.bbs[1] - 1, (int)ceilf(hi[1]) + 1);
        int z0 = max(P.bb0[2], (int)floorf(lo[2]) - 1), z1 = min(P.bb0[2] + P.bbs[2] - 1, (int)ceilf(hi[2]) + 1);
        G.gx0 = x0; G.gy0 = y0; G.gz0 = z0;
        G.gnx = max(0, x1 - x0 + 1); G.gny = max(0, y1 - y0 + 1); G.gnz = max(0, z1 - z0 + 1);
        G.rows = (int)ee_gather_groups(G.gny, G.gnz);
        G.tiles = ((G.gnx + 7) / 8) * ((G.gny + 7) / 8) * ((G.gnz + 3) / 4);
        long long off = 0, all = 0;
        int ml = 0, mls = 0;
        for (int r = 0; r < P.nrays; r++) {
            // bricked REV arrays (rev_brick); the lane kernels run one lane
            // slot per line of an 8 (tY) x 4 (tZ) tile
            EeRayGeom& R = G.ray[r];
            const Brick B = rev_store(R);
            R.offset = off - (bk_x(R.so[0]) + bk_y(B, R.so[1]) + bk_z(B, R.so[2]));
            off += ee_brick_vol(R.sn);
            all += ee_brick_vol(R.rev);
            ml = max(ml, R.rev[0]);
            mls = max(mls, ((R.sn[1] + 7) >> 3) * 8 * (((R.sn[2] + 3) >> 2) * 4));
        }
        G.rev_total = all;
        G.store_total = off;
        // the gather addresses a cone's REV array with a 32-bit offset
        if (all > 2147483647ll) G.status = 4;  // EE_ERR_REV_SIZE
        G.max_line = ml;
        G.max_lines = mls;
        if (!ee_plan_holds(S, off, mls, ml)) G.status = 8;  // EE_ERR_CAPACITY
    }
}


// ------------------------------------------------------- cone: gather ----
// Line `line` of a cone's kept part (R.nlines).
__device__ __forceinline__ void kept_line(const EeRayGeom& R, int line, int& tY, int& tZ) {
    tZ = line / R.sn[1];
    tY = R.so[1] + line - tZ * R.sn[1];
    tZ += R.so[2];
}

// Zero the samples of a line's read span outside [i0, i0 + n) (the cone
// writes those): the REV dose arena needs no separate clear.
__device__ __forceinline__ void zero_outside_segment(float* out, const Brick& Bv, int z0, int z1, int i0, int n,
                                                     int first, int stride) {
    const int e0 = n > 0 ? min(z1 + 1, i0) : z1 + 1;  // [z0, e0) before the segment
    const int s1 = n > 0 ? max(z0, i0 + n) : z1 + 1;  // [s1, z1] after it
    for (int i = z0 + first; i < e0; i += stride) out[bk_x(i)] = 0.f;
    for (int i = s1 + first; i <= z1; i += stride) out[bk_x(i)] = 0.f;
}

// REV resample of samples i0..i0+n-1 of one line into shared memory
// (device.cu:47-79): density sentinel -3 outside the BEV crop box, -2 outside
// the calc bbox; TERMA is zero at sentinel samples (never written by the
// reference).
__device__ __forceinline__ void gather_line(const EeParams& P, const EeBeamSpec& S, const EeBeamGeom& G,
                                            const EeRayGeom& R, const float* __restrict__ terma_b, int tY, int tZ,
                                            int i0, int n, int lane, float* rho, float* T, int stride = 32) {
    const f3 bl = line_point(R.B0, R.By, R.Bz, (float)tY, (float)tZ);
    const f3 gl = line_point(R.G0, R.Gy, R.Gz, (float)tY, (float)tZ);
    const f3 bx = ld3(R.Bx), gx = ld3(R.Gx);
    const float bsx = (float)G.bev[0], bsy = (float)G.bev[1], bsz = (float)G.bev[2];
    const float b0x = (float)P.bb0[0], b0y = (float)P.bb0[1], b0z = (float)P.bb0[2];
    const float b1x = (float)(P.bb0[0] + P.bbs[0]), b1y = (float)(P.bb0[1] + P.bbs[1]), b1z = (float)(P.bb0[2] + P.bbs[2]);
    for (int k = lane; k < n; k += stride) {
        const float fi = (float)(i0 + k);
        f3 bev = along(bl, bx, fi);
        float r = -3.f, t = 0.f;
        if (!(bev.x < 0.f || bev.y < 0.f || bev.z < 0.f || bev.x >= bsx || bev.y >= bsy || bev.z >= bsz)) {
            f3 g = along(gl, gx, fi);
            if (g.x < b0x || g.x >= b1x || g.y < b0y || g.y >= b1y || g.z < b0z || g.z >= b1z) {
                r = -2.f;
            } else {
                r = tex3D<float>(P.dens_tex, g.x + 0.5f, g.y + 0.5f, g.z + 0.5f);
                if (terma_b)
                    t = tri_brick(terma_b, brick_of(S.tn), g.x - (float)S.t0[0], g.y - (float)S.t0[1],
                                   g.z - (float)S.t0[2]);
            }
        }
        rho[k] = r;
        if (T) T[k] = t;
    }
}

// --------------------------------------------------- cone: exp scans -----
// Collapsed-cone line convolution with K(r) = A/a (1-e^{-ar}) + B/b (1-e^{-br})
// on the reference discretisation (device.cu:140-211: no self term, radii
// measured from the receiving voxel's boundary to the source voxel's centre):
//   D_i = sum_c A_c/a_c [ Y_i + T_{i-1} (1 - h_{i-1}) ],
//   Y_{i+1} = h_i^2 Y_i + T_{i-1} h_i (1 - h_{i-1} h_i),  h_j = e^{-a p_j/2},
// p = delr*rho, with p = T = 0 at sentinel samples.  Work-efficient warp
// scan: each lane owns a contiguous chunk of the line, composes its chunk's
// affine maps Y -> F Y + U sequentially, one 5-step shuffle scan over the 32
// chunk maps gives every lane its starting Y, and a second sequential pass
// replays the chunk.  Odd chunk lengths keep the lanes' shared-memory
// strides bank-conflict free.  FWD walks ascending i (contributions from
// k < i); the reverse pass adds its part to D and applies 1/nphi.

// inclusive warp scan of affine maps (F, U): lane j gets maps 0..j composed
__device__ __forceinline__ void warp_affine_scan(int lane, float& F1, float& U1, float& F2, float& U2) {
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        float fF1 = __shfl_up_sync(FULL, F1, off), fU1 = __shfl_up_sync(FULL, U1, off);
        float fF2 = __shfl_up_sync(FULL, F2, off), fU2 = __shfl_up_sync(FULL, U2, off);
        if (lane >= off) {
            U1 = fmaf(F1, fU1, U1); F1 *= fF1;
            U2 = fmaf(F2, fU2, U2); F2 *= fF2;
        }
    }
}

template <bool FWD>
__device__ __forceinline__ void line_scan(const float* rho, const float* T, int n, int lane, float delr,
                                          const float* prm, float* D, float inv_nphi) {
    const float c1 = prm[0] / prm[1], c2 = prm[2] / prm[3];
    const float e1 = -0.5f * prm[1] * delr, e2 = -0.5f * prm[3] * delr;  // h = exp(e * rho)
    const int cs = ((n + 31) >> 5) | 1;
    const int w0 = min(n, lane * cs), w1 = min(n, w0 + cs);
    // previous sample (walk order) of the chunk's first step
    float tm0 = 0.f, hm10 = 1.f, hm20 = 1.f;
    if (w0 > 0 && w0 < w1) {
        const int im = FWD ? w0 - 1 : n - w0;
        const float rm = rho[im];
        if (rm >= 0.f) { tm0 = T[im]; hm10 = __expf(e1 * rm); hm20 = __expf(e2 * rm); }
    }
    // pass 1: compose this chunk's steps
    float F1 = 1.f, U1 = 0.f, F2 = 1.f, U2 = 0.f;
    float tm = tm0, hm1 = hm10, hm2 = hm20;
    for (int w = w0; w < w1; w++) {
        const int i = FWD ? w : n - 1 - w;
        const float r = rho[i];
        float t = 0.f, h1 = 1.f, h2 = 1.f;
        if (r >= 0.f) { t = T[i]; h1 = __expf(e1 * r); h2 = __expf(e2 * r); }
        const float f1 = h1 * h1, f2 = h2 * h2;
        U1 = fmaf(f1, U1, tm * h1 * (1.f - hm1 * h1)); F1 *= f1;
        U2 = fmaf(f2, U2, tm * h2 * (1.f - hm2 * h2)); F2 *= f2;
        tm = t; hm1 = h1; hm2 = h2;
    }
    warp_affine_scan(lane, F1, U1, F2, U2);
    // Y at the start of the chunk: the line starts from Y = 0
    float Y1 = __shfl_up_sync(FULL, U1, 1), Y2 = __shfl_up_sync(FULL, U2, 1);
    if (lane == 0) { Y1 = 0.f; Y2 = 0.f; }
    // pass 2: replay
    tm = tm0; hm1 = hm10; hm2 = hm20;
    for (int w = w0; w < w1; w++) {
        const int i = FWD ? w : n - 1 - w;
        const float r = rho[i];
        float t = 0.f, h1 = 1.f, h2 = 1.f;
        if (r >= 0.f) { t = T[i]; h1 = __expf(e1 * r); h2 = __expf(e2 * r); }
        const float d = c1 * (Y1 + tm * (1.f - hm1)) + c2 * (Y2 + tm * (1.f - hm2));
        if (FWD) D[i] = d;
        else D[i] = r >= 0.f ? (D[i] + d) * inv_nphi : 0.f;
        Y1 = fmaf(h1 * h1, Y1, tm * h1 * (1.f - hm1 * h1));
        Y2 = fmaf(h2 * h2, Y2, tm * h2 * (1.f - hm2 * h2));
        tm = t; hm1 = h1; hm2 = h2;
    }
}

// --------------------------------------------------- cone: table walk ----
// RowConvolve walk (device.cu:126-211) over shared memory with exact FP32
// linear interpolation of the cumulative kernel between radial boundaries.
// coef == nullptr: returns sum_k w_k T_k; otherwise adds w_k * gscale into
// coef[k] with shared-memory atomics (adjoint).
__device__ __forceinline__ float table_walk(const float* rho, const float* T, int L, int i, int step, const float* K,
                                            const float* RAD, int nr, float delr, float* coef, float gscale) {
    float sum = 0.f, r_eff = 0.f, cumval = 0.f, last_cumval = 0.f, last_rad = 0.f, next_rad = RAD[0];
    int rad_start = 0, k1 = i;
    do {
        k1 += step;
        if (k1 < 0 || k1 >= L) break;
        float de = delr * rho[k1];
        r_eff += 0.5f * de;
        if (r_eff > RAD[nr - 1]) break;
        while (next_rad < r_eff) {
            if (rad_start == nr - 1) break;
            last_rad = next_rad;
            next_rad = RAD[++rad_start];
        }
        float interp = (r_eff - last_rad) / (next_rad - last_rad);
        if (rad_start == 0) cumval = interp * K[0];
        else cumval = K[rad_start - 1] + interp * (K[rad_start] - K[rad_start - 1]);
        float w = cumval - last_cumval;
        if (coef) atomicAdd(coef + k1, w * gscale);
        else sum += w * T[k1];
        last_cumval = cumval;
        r_eff += 0.5f * de;
    } while (rad_start < nr - 1);
    return sum;
}

// ------------------------------------------------------- cone kernels ----
constexpr int CONE_WARPS = 4;

__global__ void __launch_bounds__(CONE_WARPS * 32) k_cone(EeParams P, const EeBeamSpec* __restrict__ specs,
                                                          const EeBeamGeom* __restrict__ geoms,
                                                          const float* __restrict__ terma, float* __restrict__ rev,
                                                          int maxL) {
    extern __shared__ float sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ray = blockIdx.y, b = blockIdx.z;
    const EeBeamGeom& G = geoms[b];
    float* tabK = sm + (size_t)CONE_WARPS * 3 * maxL;  // [2][nradii] kernel rows + radii
    float* tabR = tabK + 2 * EE_MAX_RADII;
    if (P.mode != EE_KERNEL_EXP) {
        const EeRayConst& RC = P.rays[ray];
        for (int k = threadIdx.x; k < P.nradii; k += blockDim.x) {
            tabK[k] = P.cumkern[RC.row_fwd * P.nradii + k];
            tabK[EE_MAX_RADII + k] = P.cumkern[RC.row_rev * P.nradii + k];
            tabR[k] = P.radii[k];
        }
        __syncthreads();
    }
    if (G.status != 0) return;
    const EeRayGeom& R = G.ray[ray];
    const int line = blockIdx.x * CONE_WARPS + warp;
    if (line >= R.nlines) return;
    const int L = R.rev[0];
    int tY, tZ;
    kept_line(R, line, tY, tZ);
    if (lit_form(R, (float)tY, (float)tZ) < EE_LIT_READ) return;
    float* rho = sm + (size_t)warp * 3 * maxL;
    float* T = rho + maxL;
    float* D = T + maxL;
    // bricked REV arena (rev_brick): sample i at out + bk_x(i)
    const Brick Bv = rev_store(R);
    float* out = rev + G.arena_off + R.offset + rev_line(Bv, tY, tZ);
    int i0, n, z0, z1;
    line_segment(P, G, R, tY, tZ, L, i0, n);
    line_read_span(G, R, tY, tZ, L, z0, z1);
    zero_outside_segment(out, Bv, z0, z1, i0, n, lane, 32);
    if (n > 0) {
        gather_line(P, specs[b], G, R, terma + specs[b].t_off, tY, tZ, i0, n, lane, rho, T);
        __syncwarp();
        const float inv_nphi = 1.f / (float)P.nphi;
        const EeRayConst& RC = P.rays[ray];
        if (P.mode == EE_KERNEL_EXP) {
            line_scan<true>(rho, T, n, lane, P.lng, P.expp + 4 * RC.row_fwd, D, inv_nphi);
            __syncwarp();
            line_scan<false>(rho, T, n, lane, P.lng, P.expp + 4 * RC.row_rev, D, inv_nphi);
        } else {
            for (int k = lane; k < n; k += 32) {
                float v = 0.f;
                if (rho[k] >= 0.f) {
                    v = table_walk(rho, T, n, k, -1, tabK, tabR, P.nradii, P.lng, nullptr, 0.f);
                    v += table_walk(rho, T, n, k, +1, tabK + EE_MAX_RADII, tabR, P.nradii, P.lng, nullptr, 0.f);
                    v = __fdiv_rn(v, (float)P.nphi);
                }
                D[k] = v;
            }
        }
        __syncwarp();
    }
    for (int k = lane; k < n; k += 32) out[bk_x(i0 + k)] = D[k];
}

__device__ __forceinline__ float rho_at(const EeParams& P, f3 g) {
    return tex3D<float>(P.dens_tex, g.x + 0.5f, g.y + 0.5f, g.z + 0.5f);
}

// ------------------------------------- cone: exact table scan, O(n nr) ----
// The reference's RowConvolve walk (device.cu:126-211) with the cumulative
// kernel interpolated linearly between its nr = 24 radial boundaries (the
// reference's N_KERNEL_RADII), evaluated exactly in O(n * nr) per line
// instead of O(n^2).
//
// One walk direction at a time, in walk order w = 0..n-1 (FWD: line order,
// the sources of receiver w are k < w; reverse: the mirrored order).  With
// d_w = delr * rho_w (0 at sentinels), P_w = sum_{m<w} d_m and
// M_w = P_w + d_w / 2, the walk from receiver w gives source k the
// radiological distance c_k = P_w - M_k (half the source voxel plus every
// voxel in between, device.cu:144-164).  It includes every source with
// c_k <= R_{nr-2} plus the first one beyond that, if its c_k <= R_{nr-1} (the
// loop's two exits, device.cu:146-147,171).  With s the last included source
// and V_k = T_k - T_{k-1}, summation by parts of sum T_k (K(c_k) - K(c_{k+1}))
// gives
//   D_w = T_s K(c_s) + sum_{k=s+1}^{w-1} V_k K(c_k).
// K is linear on segment j, (Rm_j, R_j] with Rm_j = R_{j-1} (Rm_0 = 0):
// K(c) = Km_j + beta_j (c - Rm_j), Km_j = K_{j-1} (Km_0 = 0).  The sources of
// segment j form the index window [x_j, x_{j-1}) with x_j = the first k whose
// M_k >= P_w - R_j (x_{-1} = w), so with the prefix sums SV_k = T_{k-1} and
// SVM_k = sum_{m<k} V_m M_m a window costs two lookups, and regrouping the
// windows at their shared ends leaves one per boundary:
//   D_w = T_s K(c_s) + beta_0 (P_w SV_w - SVM_w)
//       + sum_{j=0}^{nr-3} gamma_{j+1} ((P_w - R_j) SV_{x_j} - SVM_{x_j})
//       - coef_{nr-2} SV_{x_{nr-2}} + beta_{nr-2} SVM_{x_{nr-2}},
// gamma_j = beta_j - beta_{j-1}, coef_j = Km_j + beta_j (P_w - Rm_j), every
// x_j clipped below at s + 1 (source s enters through its own term).  Each
// lane walks a contiguous chunk of receivers; the x_j only move forward as w
// grows, so after a binary search for the chunk's first receiver each is
// advanced, not searched.  Plain FP32: the regrouped terms are bounded by
// |gamma| * P * T, measured at <= 2e-5 of the line's maximum against the
// FP64 walk on 1000-sample lines.
//
// Transpose (TERMA gradient from the REV-dose gradient g): with the last
// receiver b_k whose walk reaches source k (P_i - M_{k+1} <= R_{nr-2} and
// P_i - M_k <= R_{nr-1}, or i = k + 1), and
//   Phi_b(m) = sum_{i <= b} g_i K(P_i - m)   (K = 0 for P_i <= m),
// source k receives Tbar_k = Phi_{b_k}(M_k) - Phi_{b_k}(M_{k+1}).  Phi_b(m)
// regroups the same way over the receiver windows y_j = the first i with
// P_i > m + R_j, with prefix sums Sg_i = sum_{m<i} g_m and
// SgP_i = sum_{m<i} g_m P_m; source k evaluates W_k = Phi_{b_k}(M_k) and
// U_k = Phi_{b_{k-1}}(M_k) in one pass over its pointers, and
// Tbar_k = W_k - U_{k+1}.
constexpr int TAB_NR = 24;            // radial boundaries of the fast path
constexpr int TAB_NB = TAB_NR - 1;    // receiver windows of the forward walk

// Per-block kernel-row tables: R, Rm (shared by both rows), then for the
// forward row and for the reverse row Km, beta, gamma and the suffix sums
// SG_j = sum_{m=j}^{nr-2} gamma_{m+1} and SGR_j = sum_{m=j}^{nr-2}
// gamma_{m+1} R_m (EE_MAX_RADII each).  Window ends that cannot move on a
// line (radius at least the line's radiological length) all sit at the same
// position, so their terms are summed in closed form from SG and SGR.
struct TabRow {
    const float *R, *Rm, *Km, *B, *G, *SG, *SGR;
};
constexpr int TAB_SMEM = 12 * EE_MAX_RADII;

// Fills the tables; the caller synchronises the block before using them.
__device__ __forceinline__ void tab_tables(const EeParams& P, const EeRayConst& RC, float* t) {
    for (int k = threadIdx.x; k < TAB_NR * 2; k += blockDim.x) {
        const int row = k < TAB_NR ? RC.row_fwd : RC.row_rev, j = k % TAB_NR;
        const float* Kr = P.cumkern + (size_t)row * P.nradii;
        const float R = P.radii[j], Rm = j ? P.radii[j - 1] : 0.f;
        const float K = Kr[j], Km = j ? Kr[j - 1] : 0.f;
        const float b = (K - Km) / (R - Rm);
        float bm = 0.f;
        if (j) bm = (Km - (j > 1 ? Kr[j - 2] : 0.f)) / (Rm - (j > 1 ? P.radii[j - 2] : 0.f));
        float* o = t + (k < TAB_NR ? 2 : 7) * EE_MAX_RADII;
        o[j] = Km;
        o[EE_MAX_RADII + j] = b;
        o[2 * EE_MAX_RADII + j] = b - bm;
        if (k < TAB_NR) {
            t[j] = R;
            t[EE_MAX_RADII + j] = Rm;
        }
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        float* o = t + (threadIdx.x == 0 ? 2 : 7) * EE_MAX_RADII;
        float sg = 0.f, sgr = 0.f;
        o[3 * EE_MAX_RADII + TAB_NR - 1] = 0.f;
        o[4 * EE_MAX_RADII + TAB_NR - 1] = 0.f;
        for (int j = TAB_NR - 2; j >= 0; j--) {
            sg += o[2 * EE_MAX_RADII + j + 1];
            sgr = fmaf(o[2 * EE_MAX_RADII + j + 1], t[j], sgr);
            o[3 * EE_MAX_RADII + j] = sg;
            o[4 * EE_MAX_RADII + j] = sgr;
        }
    }
}

__device__ __forceinline__ TabRow tab_row(const float* t, bool fwd) {
    const float* o = t + (fwd ? 2 : 7) * EE_MAX_RADII;
    return TabRow{t, t + EE_MAX_RADII, o, o + EE_MAX_RADII, o + 2 * EE_MAX_RADII, o + 3 * EE_MAX_RADII,
                  o + 4 * EE_MAX_RADII};
}

// exclusive prefix sum over the W-lane group of `lane` (W = 32: the warp; W =
// 16: each half separately); all 32 lanes take part
__device__ __forceinline__ float warp_excl_scan(float x, int lane, int W) {
    float s = x;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {  // lane < W: the last step adds nothing when W = 16
        const float y = __shfl_up_sync(FULL, s, off, W);
        if (lane >= off) s += y;
    }
    return s - x;
}

__device__ __forceinline__ int wmap(bool fwd, int w, int n) { return fwd ? w : n - 1 - w; }

// lane chunks of a line over the W lanes that share it: the shortest length
// that covers it, so that as many lanes as possible work (measured faster
// than odd lengths, which spread the lanes' strided shared-memory accesses
// over all the banks but leave up to a third of the lanes idle)
__device__ __forceinline__ void tab_chunk(int W, int n, int lane, int& w0, int& w1) {
    const int cs = max(1, (n + W - 1) / W);
    w0 = min(n, lane * cs);
    w1 = min(n, w0 + cs);
}

// M_w, P_w and SVM_w for w >= a in walk order, P from sample a on (separate
// arrays: lanes reading scattered samples then spread over all the banks); T is
// 0 below a.  SV_w = T_{w-1} is read from T, which has a zero at T[-1] and T[n].
__device__ __forceinline__ void tab_build(bool fwd, int W, const float* rho, const float* T, int n, int a, int lane,
                                          float delr, float* Mv, float* Pv, float* SVMv) {
    int w0, w1;
    tab_chunk(W, n - a, lane, w0, w1);
    w0 += a;
    w1 += a;
    const float tp0 = (w0 > a && w0 < w1) ? T[wmap(fwd, w0 - 1, n)] : 0.f;
    float sd = 0.f, svm = 0.f, tp = tp0;
#pragma unroll 1
    for (int w = w0; w < w1; w++) {  // chunk sums, P local to the chunk
        const int i = wmap(fwd, w, n);
        const float r = rho[i], t = T[i];
        const float d = r >= 0.f ? delr * r : 0.f;
        svm = fmaf(t - tp, fmaf(0.5f, d, sd), svm);
        sd += d;
        tp = t;
    }
    const float Pst = warp_excl_scan(sd, lane, W);
    float S = warp_excl_scan(fmaf(Pst, tp - tp0, svm), lane, W);
    float Pw = Pst;
    tp = tp0;
#pragma unroll 1
    for (int w = w0; w < w1; w++) {
        const int i = wmap(fwd, w, n);
        const float r = rho[i], t = T[i];
        const float d = r >= 0.f ? delr * r : 0.f;
        const float M = fmaf(0.5f, d, Pw);
        Mv[w] = M;
        Pv[w] = Pw;
        SVMv[w] = S;
        S = fmaf(t - tp, M, S);
        Pw += d;
        tp = t;
    }
}

// Receivers of one walk direction, added to D (sources in [a, e], a lane's
// receivers a contiguous chunk of (a, n)).  X: this lane's window ends, X[32 j]
// = x_j (shared memory, so the loops over the window ends stay loops).
//
// Only the ends inside the sources' range cost a step: an end with R_j >= P_w -
// M_a has not left a, where the prefix sums are 0; one past e + 1 (js of them)
// has every source behind it, SV is 0 there and the ends' SVM terms add up to
// beta_js.  So a receiver inside the range visits the radii up to its distance
// from a and one beyond it those between the range's two ends: 5 of the 20 that
// a 40 cm line has, on average, and receivers at and before a none.  Neither
// s nor the clip matter before R_{nr-2} reaches past a: the general form runs
// only there.
__device__ __forceinline__ void tab_receivers(bool fwd, int W, const float* Mv, const float* Pv, const float* T,
                                              const float* SVMv, int n, int a, int e, int lane, const TabRow& K,
                                              unsigned short* X, float* D) {
    int w0, w1;
    tab_chunk(W, n - 1 - a, lane, w0, w1);
    if (w0 >= w1) return;
    w0 += a + 1;
    w1 += a + 1;
    const float Rl = K.R[TAB_NR - 1], m0 = Mv[a];
    auto SV = [&](int w) { return T[wmap(fwd, w - 1, n)]; };
    int ja = 0, js = 0;  // ends that have left a; ends past e + 1
    {   // the chunk's first receiver: binary searches (x_j <= x_{j-1})
        const float Pw = Pv[w0];
        int hi = min(w0, e + 2);
        for (; ja < TAB_NB && K.R[ja] < Pw - m0; ++ja) {
            const float t = Pw - K.R[ja];
            int lo = a, h = hi;
#pragma unroll 1
            while (lo < h) {
                const int mid = (lo + h) >> 1;
                if (Mv[mid] >= t) h = mid;
                else lo = mid + 1;
            }
            X[32 * ja] = (unsigned short)lo;
            hi = lo;
        }
    }
#pragma unroll 1
    for (int w = w0; w < w1; w++) {
        const float Pw = Pv[w];
        const int hi = min(w, e + 2);
        for (; ja < TAB_NB && K.R[ja] < Pw - m0; ++ja) X[32 * ja] = (unsigned short)a;
        float tot;
        if (ja < TAB_NB) {
            if (hi == e + 2)
                while (js < ja && X[32 * js] == hi) ++js;
            tot = K.B[js] * fmaf(Pw, SV(hi), -SVMv[hi]);
#pragma unroll 1
            for (int j = js; j < ja; j++) {
                const float t = Pw - K.R[j];
                int xx = X[32 * j];
#pragma unroll 1
                while (xx < hi && Mv[xx] < t) ++xx;
                X[32 * j] = (unsigned short)xx;
                tot = fmaf(K.G[j + 1], fmaf(t, SV(xx), -SVMv[xx]), tot);
            }
        } else {
            // the last window end (radius R_{nr-2}) decides the last included source s
            tot = 0.f;
            int xs = X[32 * (TAB_NB - 1)];
            {
                const float t = Pw - K.R[TAB_NB - 1];
#pragma unroll 1
                while (xs < hi && Mv[xs] < t) ++xs;
                X[32 * (TAB_NB - 1)] = (unsigned short)xs;
            }
            const bool back = xs > a && Pw - Mv[xs - 1] <= Rl;
            const int s = back ? xs - 1 : xs;
            const int clip = s + 1;  // window ends are clipped below at s + 1
            int seg = 0;
#pragma unroll 1
            for (int j = 0; j < TAB_NB - 1; j++) {
                const float t = Pw - K.R[j];
                int xx = X[32 * j];
#pragma unroll 1
                while (xx < hi && Mv[xx] < t) ++xx;
                X[32 * j] = (unsigned short)xx;
                if (s < w) {
                    seg += xx > s ? 1 : 0;
                    const int lo = max(xx, clip);
                    tot = fmaf(K.G[j + 1], fmaf(t, SV(lo), -SVMv[lo]), tot);
                }
            }
            if (s < w) {
                tot = fmaf(K.B[0], fmaf(Pw, SV(hi), -SVMv[hi]), tot);  // top end
                {   // the lowest window's lower end
                    seg += xs > s ? 1 : 0;
                    const int lo = max(xs, clip);
                    const float coef = fmaf(K.B[TAB_NB - 1], Pw - K.Rm[TAB_NB - 1], K.Km[TAB_NB - 1]);
                    tot = fmaf(K.B[TAB_NB - 1], SVMv[lo], fmaf(-coef, SV(lo), tot));
                }
                const int sg = back ? TAB_NR - 1 : seg;  // segment of c_s
                tot = fmaf(SV(clip), fmaf(K.B[sg], (Pw - Mv[s]) - K.Rm[sg], K.Km[sg]), tot);
            }
        }
        D[wmap(fwd, w, n)] += tot;
    }
}

// P_w, Sg_w, SgP_w (w = a..n, P_n = +inf: pointer stop) and M_w in walk order,
// the sums from sample a on.
__device__ __forceinline__ void tab_build_T(bool fwd, int W, const float* rho, const float* g, int n, int a, int lane,
                                            float delr, float* Pv, float* Sgv, float* SgPv, float* Mv) {
    int w0, w1;
    tab_chunk(W, n - a, lane, w0, w1);
    w0 += a;
    w1 += a;
    float sd = 0.f, sg = 0.f, sgp = 0.f;
#pragma unroll 1
    for (int w = w0; w < w1; w++) {
        const int i = wmap(fwd, w, n);
        const float r = rho[i], gi = g[i];
        sgp = fmaf(gi, sd, sgp);
        sg += gi;
        sd += r >= 0.f ? delr * r : 0.f;
    }
    float Pw = warp_excl_scan(sd, lane, W);
    float Sg = warp_excl_scan(sg, lane, W);
    float SgP = warp_excl_scan(fmaf(Pw, sg, sgp), lane, W);
#pragma unroll 1
    for (int w = w0; w < w1; w++) {
        const int i = wmap(fwd, w, n);
        const float r = rho[i], gi = g[i];
        const float d = r >= 0.f ? delr * r : 0.f;
        Pv[w] = Pw;
        Sgv[w] = Sg;
        SgPv[w] = SgP;
        Mv[w] = fmaf(0.5f, d, Pw);
        SgP = fmaf(gi, Pw, SgP);
        Sg += gi;
        Pw += d;
    }
    if (w1 == n && w0 < w1) {
        Pv[n] = __int_as_float(0x7f800000);
        Sgv[n] = Sg;
        SgPv[n] = SgP;
    }
}

// Sources [a, e] of one walk direction, and e + 1 for its U: Tbar_k = W_k -
// U_{k+1} added to Tb, with W_k = Phi_{b_k}(M_k), U_k = Phi_{b_{k-1}}(M_k) and
// the window ends y_j (Y[32 j], shared memory) clipped above at cap + 1 for each
// cap.  A lane's sources are a contiguous chunk; its first U goes to the lane
// before it (all lanes take part).
__device__ __forceinline__ void tab_sources(bool fwd, int W, const float* Pv, const float* Sgv, const float* SgPv,
                                            const float* Mv, int n, int a, int e, int lane, const TabRow& K,
                                            unsigned short* Y, float* Tb) {
    int w0, w1;
    tab_chunk(W, min(e + 2, n) - a, lane, w0, w1);
    w0 += a;
    w1 += a;
    float first = 0.f;  // U of the chunk's first source
    if (w0 < w1) {
        const float Rl = K.R[TAB_NR - 1], Rl2 = K.R[TAB_NR - 2];
        // window ends with R_j >= P_{n-1} - M_{w0} stay at n for every source
        const float span = Pv[n - 1] - Mv[w0];
        int ja = 0;
        while (ja < TAB_NR && K.R[ja] < span) ++ja;
        int jm = min(ja, TAB_NR - 1);  // moving middle window ends: j < jm
        auto lim_of = [&](int k) {
            float l = Mv[k] + Rl;
            if (k + 1 < n) l = fminf(l, Mv[k + 1] + Rl2);
            return l;
        };
        // the first receiver i in [lo, n] with P_i > v (P_n = +inf)
        auto ub = [&](float v, int lo) {
            int h = n;
#pragma unroll 1
            while (lo < h) {
                const int mid = (lo + h) >> 1;
                if (Pv[mid] > v) h = mid;
                else lo = mid + 1;
            }
            return lo;
        };
        {   // the chunk's first source: binary searches (y_j >= y_{j-1})
            const float m = Mv[w0];
            int lo = min(w0 + 1, n);
            for (int j = 0; j < ja; j++) {
                lo = ub(m + K.R[j], lo);
                Y[32 * j] = (unsigned short)lo;
            }
            for (int j = ja; j < TAB_NR; j++) Y[32 * j] = (unsigned short)n;
        }
        int ylim = ub(lim_of(w0), min(w0 + 1, n));
        int capU = w0 > a ? min(max(ub(lim_of(w0 - 1), w0) - 1, w0), n - 1) : w0;  // b_{w0-1}
#pragma unroll 1
        for (int k = w0; k < w1; k++) {
            const float m = Mv[k];
            {
                const float l = lim_of(k);
#pragma unroll 1
                while (Pv[ylim] <= l) ++ylim;
            }
            const int capW = min(max(ylim - 1, k + 1), n - 1);  // b_k
            float wk = 0.f, uk = 0.f;
            if (k + 1 < n) {
                const float sW = Sgv[capW + 1], sWp = SgPv[capW + 1], sU = Sgv[capU + 1], sUp = SgPv[capU + 1];
                while (jm > 0 && Y[32 * (jm - 1)] == n) --jm;
                // bottom end k + 1: beta_0 (m Sg - SgP)
                wk = K.B[0] * fmaf(m, Sgv[k + 1], -SgPv[k + 1]);
                uk = wk;
#pragma unroll 1
                for (int j = 0; j < jm; j++) {
                    const float t = m + K.R[j];
                    int yy = Y[32 * j];
#pragma unroll 1
                    while (Pv[yy] <= t) ++yy;
                    Y[32 * j] = (unsigned short)yy;
                    const float a = Sgv[yy], ap = SgPv[yy];
                    const bool inW = yy <= capW + 1, inU = yy <= capU + 1;
                    wk = fmaf(K.G[j + 1], fmaf(t, inW ? a : sW, -(inW ? ap : sWp)), wk);
                    uk = fmaf(K.G[j + 1], fmaf(t, inU ? a : sU, -(inU ? ap : sUp)), uk);
                }
                // fixed middle ends j in [jm, nr-2] sit at n: past both caps
                const float sg = K.SG[jm], sgr = K.SGR[jm];
                wk += fmaf(sW, fmaf(m, sg, sgr), -sWp * sg);
                uk += fmaf(sU, fmaf(m, sg, sgr), -sUp * sg);
                {   // top end (radius R_{nr-1}): coef'_{nr-1} Sg + beta_{nr-1} SgP
                    const int j = TAB_NR - 1;
                    int yy = Y[32 * j];
                    if (j < ja) {
#pragma unroll 1
                        while (Pv[yy] <= m + K.R[j]) ++yy;
                        Y[32 * j] = (unsigned short)yy;
                    }
                    const float coef = K.Km[j] - K.B[j] * (m + K.Rm[j]);
                    const bool inW = yy <= capW + 1, inU = yy <= capU + 1;
                    wk = fmaf(coef, inW ? Sgv[yy] : sW, fmaf(K.B[j], inW ? SgPv[yy] : sWp, wk));
                    uk = fmaf(coef, inU ? Sgv[yy] : sU, fmaf(K.B[j], inU ? SgPv[yy] : sUp, uk));
                }
            }
            if (k == w0) first = uk;
            else Tb[wmap(fwd, k - 1, n)] -= uk;
            if (k <= e) Tb[wmap(fwd, k, n)] += wk;
            capU = capW;
        }
    }
    __syncwarp();
    const float next = __shfl_down_sync(FULL, first, 1, W);
    if (w0 < w1 && w1 <= min(e + 1, n - 1)) Tb[wmap(fwd, w1 - 1, n)] -= next;
}

// Exact-table cone kernel (mode EE_KERNEL_TABLE, nr = 24): REV resample of a
// line into shared memory, then the two walk directions.
constexpr int TAB_WARPS = 4;

__host__ __device__ constexpr int tab_lp(int maxL) { return ((maxL + 3) & ~3) + 4; }
__host__ __device__ constexpr int tab_fwd_stride(int maxL) { return 6 * tab_lp(maxL) + 16 * TAB_NB; }
__host__ __device__ constexpr int tab_adj_stride(int maxL) { return 7 * tab_lp(maxL) + 16 * TAB_NR; }

// A line of the table kernels: its samples [i0, i0 + n), of which [a, e]
// (from i0) can have TERMA; line = -1: nothing to write, n = 0: zeros only.
struct TabLine {
    int line, i0, n, a, e, tY, tZ;
    LineFrame F;
};

// Kept line `line`; -1 where its lit forms are below `least`.
__device__ __forceinline__ TabLine tab_line(const EeParams& P, const EeBeamSpec& S, const EeBeamGeom& G,
                                            const EeRayGeom& R, float least, int line) {
    TabLine t;
    t.line = -1;
    t.i0 = t.n = t.a = t.tY = t.tZ = 0;
    t.e = -1;
    if (line < 0) return t;
    kept_line(R, line, t.tY, t.tZ);
    if (lit_form(R, (float)t.tY, (float)t.tZ) < least) return t;
    t.line = line;
    const LaneSpan s = lane_span(P, S, G, R, t.tY, t.tZ, t.F);
    if (s.q1 < s.q0) return t;
    t.i0 = s.i0;
    t.n = s.i1 - s.i0 + 1;
    t.a = max(4 * s.q0, s.i0) - s.i0;
    t.e = min(4 * s.q1 + 3, s.i1) - s.i0;
    return t;
}

// One line of k_cone_tab on the W lanes of its group (`lane` counts within
// the group; W = 32: the whole warp, W = 16: half of it), with the group's
// arrays at `arr`.  A line without samples still takes part in the scans, which
// all 32 lanes execute.
__device__ __forceinline__ void tab_fwd_line(int W, const EeParams& P, const EeBeamSpec& S, const EeBeamGeom& G,
                                             const EeRayGeom& R, const float* __restrict__ terma_b,
                                             float* __restrict__ rev_beam, const TabLine& L, int lane, float* arr,
                                             int Lp, const float* tab, unsigned short* X) {
    float* Mv = arr;
    float* Pv = Mv + Lp;
    float* SVMv = Pv + Lp;
    float* rho = SVMv + Lp;
    float* D = rho + Lp;
    float* T = D + Lp + 1;  // T[-1] = T[n] = 0
    float* out = nullptr;
    const int n = L.n;
    if (L.line >= 0) {
        const Brick Bv = rev_store(R);
        out = rev_beam + R.offset + rev_line(Bv, L.tY, L.tZ);
        int z0, z1;
        line_read_span(G, R, L.tY, L.tZ, R.rev[0], z0, z1);
        zero_outside_segment(out, Bv, z0, z1, L.i0, n, lane, W);
    }
    const f3 t0 = mk((float)S.t0[0], (float)S.t0[1], (float)S.t0[2]);
    const Brick Bt = brick_of(S.tn);
    for (int k = lane; k < n; k += W) {
        const f3 g = sample_point(L.F, L.i0 + k);
        rho[k] = rho_at(P, g);
        T[k] = k >= L.a && k <= L.e ? tri_brick(terma_b, Bt, g.x - t0.x, g.y - t0.y, g.z - t0.z) : 0.f;
        D[k] = 0.f;
    }
    if (lane == 0) T[-1] = T[n] = 0.f;
    __syncwarp();
#pragma unroll 1
    for (int dir = 0; dir < 2; dir++) {
        const bool fwd = dir == 0;
        const int a = fwd ? L.a : max(0, n - 1 - L.e), e = fwd ? L.e : n - 1 - L.a;  // the sources in walk order
        tab_build(fwd, W, rho, T, n, a, lane, P.lng, Mv, Pv, SVMv);
        __syncwarp();
        tab_receivers(fwd, W, Mv, Pv, T, SVMv, n, a, e, lane, tab_row(tab, fwd), X, D);
        __syncwarp();
    }
    const float nphi = (float)P.nphi;
    for (int k = lane; k < n; k += W) out[bk_x(L.i0 + k)] = rho[k] >= 0.f ? __fdiv_rn(D[k], nphi) : 0.f;
}

// A warp takes two neighbouring lines.  When both fit half of its arrays
// (n below Lp / 2 - 1, or - 2), each half-warp runs one of them, 16 lanes per line;
// else the whole warp runs one after the other.  A lane's first receiver costs a
// binary search per window end, so a lane that runs one chunk of a line
// instead of two shorter chunks of two lines saves one set of searches, and
// short lines keep more lanes busy.
//
// Bound by instruction issue and fixed latencies (40 % of the issue slots at 20
// to 24 warps per SM, which the shared arrays allow).  Two 24 x 24 beams on 200 x
// 200 x 160: 6.8 ms with every radius of the line's length at every receiver,
// 3.3 with the ends inside the sources' range only, TERMA sampled there only and
// one copy of the code for both directions and group widths (129 -> 43 KB), 2.45
// with 16-bit window ends and T in place of an SV array (4 -> 6 blocks per SM);
// the adjoint likewise 5.4, 3.0, 2.6 ms.
__global__ void __launch_bounds__(TAB_WARPS * 32) k_cone_tab(EeParams P, const EeBeamSpec* __restrict__ specs,
                                                             const EeBeamGeom* __restrict__ geoms,
                                                             const float* __restrict__ terma, float* __restrict__ rev,
                                                             int maxL) {
    extern __shared__ float4 sm4[];
    float* sm = reinterpret_cast<float*>(sm4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ray = blockIdx.y, b = blockIdx.z;
    const int Lp = tab_lp(maxL);
    float* tab = sm + (size_t)TAB_WARPS * tab_fwd_stride(maxL);
    const EeRayConst& RC = P.rays[ray];
    tab_tables(P, RC, tab);
    __syncthreads();
    const EeBeamGeom& G = geoms[b];
    if (G.status != 0) return;
    const EeRayGeom& R = G.ray[ray];
    int la = 2 * (blockIdx.x * TAB_WARPS + warp);
    if (la >= R.nlines) return;
    const EeBeamSpec& S = specs[b];
    const TabLine A = tab_line(P, S, G, R, EE_LIT_READ, la),
                  B = tab_line(P, S, G, R, EE_LIT_READ, la + 1 < R.nlines ? la + 1 : -1);
    if (A.line < 0 && B.line < 0) return;
    float* arr = sm + (size_t)warp * tab_fwd_stride(maxL);
    unsigned short* X = reinterpret_cast<unsigned short*>(arr + 6 * Lp) + lane;
    const float* terma_b = terma + S.t_off;
    float* rev_beam = rev + G.arena_off;
    // the second half-warp's arrays start one cell past the middle: an odd
    // offset puts the two halves' strided accesses on different banks
    const int half = Lp >> 1;
    const bool both = max(A.n, B.n) < half - 2;  // T takes n + 2 cells
    const int W = both ? 16 : 32, sub = both ? lane >> 4 : 0;
#pragma unroll 1
    for (int k = 0; k < (both ? 1 : 2); k++) {
        const TabLine& L = (both ? sub : k) ? B : A;
        if (!both && L.line < 0) continue;
        tab_fwd_line(W, P, S, G, R, terma_b, rev_beam, L, lane & (W - 1), arr + sub * (half + 1), Lp, tab, X);
        __syncwarp();
    }
}

// One line of k_cone_T_tab on the W lanes of its group (as tab_fwd_line).
__device__ __forceinline__ void tab_adj_line(int W, const EeParams& P, const EeBeamSpec& S, const EeBeamGeom& G,
                                             const EeRayGeom& R, const float* __restrict__ grad_beam,
                                             float4* __restrict__ terma_grad, const TabLine& L, int lane, float* arr,
                                             int Lp, const float* tab, unsigned short* Y) {
    float* Pv = arr;
    float* Sgv = Pv + Lp;
    float* SgPv = Sgv + Lp;
    float* Mv = SgPv + Lp;
    float* rho = Mv + Lp;
    float* g = rho + Lp;
    float* Tb = g + Lp;
    const int n = L.n;
    {
        const float* gin = grad_beam + R.offset + rev_line(rev_store(R), L.tY, L.tZ);
        const float inv_nphi = 1.f / (float)P.nphi;
        for (int k = lane; k < n; k += W) {
            const float r = rho_at(P, sample_point(L.F, L.i0 + k));
            rho[k] = r;
            g[k] = r >= 0.f ? gin[bk_x(L.i0 + k)] * inv_nphi : 0.f;
            Tb[k] = 0.f;
        }
    }
    __syncwarp();
#pragma unroll 1
    for (int dir = 0; dir < 2; dir++) {
        const bool fwd = dir == 0;
        const int a = fwd ? L.a : max(0, n - 1 - L.e), e = fwd ? L.e : n - 1 - L.a;  // the sources in walk order
        tab_build_T(fwd, W, rho, g, n, a, lane, P.lng, Pv, Sgv, SgPv, Mv);
        __syncwarp();
        tab_sources(fwd, W, Pv, Sgv, SgPv, Mv, n, a, e, lane, tab_row(tab, fwd), Y, Tb);
        __syncwarp();
    }
    // transpose of the REV TERMA resample
    float4* tg = terma_grad + S.q_off;
    const Brick Bt = quads_of(S.tn);
    const f3 t0 = mk((float)S.t0[0], (float)S.t0[1], (float)S.t0[2]);
    for (int k = L.a + lane; k <= L.e; k += W) {
        const float v = Tb[k];
        if (rho[k] < 0.f || v == 0.f) continue;
        const f3 p = sample_point(L.F, L.i0 + k);
        quad_scatter(tg, Bt, p.x - t0.x, p.y - t0.y, p.z - t0.z, v);
    }
}

// Its adjoint followed by the transpose of the REV TERMA resample; two lines
// per warp as k_cone_tab.
__global__ void __launch_bounds__(TAB_WARPS * 32) k_cone_T_tab(EeParams P, const EeBeamSpec* __restrict__ specs,
                                                               const EeBeamGeom* __restrict__ geoms,
                                                               const float* __restrict__ rev_grad,
                                                               float4* __restrict__ terma_grad, int maxL) {
    extern __shared__ float4 sm4[];
    float* sm = reinterpret_cast<float*>(sm4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ray = blockIdx.y, b = blockIdx.z;
    const int Lp = tab_lp(maxL);
    float* tab = sm + (size_t)TAB_WARPS * tab_adj_stride(maxL);
    const EeRayConst& RC = P.rays[ray];
    tab_tables(P, RC, tab);
    __syncthreads();
    const EeBeamGeom& G = geoms[b];
    if (G.status != 0) return;
    const EeRayGeom& R = G.ray[ray];
    int la = 2 * (blockIdx.x * TAB_WARPS + warp);
    if (la >= R.nlines) return;
    const EeBeamSpec& S = specs[b];
    const TabLine A = tab_line(P, S, G, R, 0.f, la), B = tab_line(P, S, G, R, 0.f, la + 1 < R.nlines ? la + 1 : -1);
    if (A.n == 0 && B.n == 0) return;
    float* arr = sm + (size_t)warp * tab_adj_stride(maxL);
    unsigned short* Y = reinterpret_cast<unsigned short*>(arr + 7 * Lp) + lane;
    const float* grad_beam = rev_grad + G.arena_off;
    const int half = Lp >> 1;  // second half-warp's arrays at an odd offset, as k_cone_tab
    const bool both = max(A.n, B.n) < half - 1;
    const int W = both ? 16 : 32, sub = both ? lane >> 4 : 0;
#pragma unroll 1
    for (int k = 0; k < (both ? 1 : 2); k++) {
        const TabLine& L = (both ? sub : k) ? B : A;
        if (!both && L.n == 0) continue;
        tab_adj_line(W, P, S, G, R, grad_beam, terma_grad, L, lane & (W - 1), arr + sub * (half + 1), Lp, tab, Y);
        __syncwarp();
    }
}

// ------------------------------------------- cone: one lane per line ----
// EE_KERNEL_EXP fast path.  Each thread owns one REV line (adjacent threads
// own adjacent lines, so their segments and gathers stay close): it computes
// its segment analytically and runs the recurrence sequentially, without
// shuffles or shared memory.  Same operator as line_scan.

// Lane slot -> REV line for the one-lane-per-line kernels: the lanes of a
// warp own an 8 (tY) x 4 (tZ) tile of lines, so at every sample index the
// warp's reads and writes of the bricked REV arrays fall in two 64-byte brick
// slabs.  False for slots of a tile that lie outside the cone's array.
__device__ __forceinline__ bool lane_line(const EeRayGeom& R, int slot, int& tY, int& tZ) {
    const int wt = slot >> 5, l = slot & 31;
    const int nty = (R.sn[1] + 7) >> 3;
    if (nty == 0) return false;
    tY = (wt % nty) * 8 + (l & 7);
    tZ = (wt / nty) * 4 + (l >> 3);
    const bool in = tY < R.sn[1] && tZ < R.sn[2];
    tY += R.so[1];
    tZ += R.so[2];
    return in;
}

// Cone y of a beam's lists: cones with small angles to the beam axis, whose
// lines are the longest, come first.
__device__ __forceinline__ int list_cone(const EeParams& P, int y) {
    return (y % P.nphi) * (P.ntheta / 2) + y / P.nphi;
}

// The tiles of 8 x 4 lines that may hold a line with lit forms of at least
// `least` in the dilated crop box: the lane cones' work lists, a block per
// beam and cone.  touched (adjoint): tiles that the gather added to; the
// gradient of the others' lines is zero (20 beams of 128^2 pixels with a
// target-and-organs gradient: adjoint cone 2.64 -> 0.80 ms; dense gradients
// unchanged).
__global__ void __launch_bounds__(256) k_cone_tiles(EeParams P, const EeBeamGeom* __restrict__ geoms, float least,
                                                    const unsigned char* __restrict__ touched,
                                                    int* __restrict__ counts, int* __restrict__ tiles, int cap) {
    __shared__ int s_n;
    const int b = blockIdx.y, seg = b * P.nrays + blockIdx.x;
    const EeBeamGeom& G = geoms[b];
    if (seg == 0 && threadIdx.x == 0) counts[0] = 0;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    if (G.status == 0) {
        const int cone = list_cone(P, blockIdx.x);
        const EeRayGeom& R = G.ray[cone];
        const unsigned char* const hit = touched ? touched + (size_t)(b * P.nrays + cone) * cap : nullptr;
        const int nty = (R.sn[1] + 7) >> 3, n = nty * ((R.sn[2] + 3) >> 2);
        for (int t0 = 0; t0 < n; t0 += 256) {
            const int tile = t0 + threadIdx.x;
            bool live = tile < n;
            const bool added = !hit || (live && hit[tile]);
            if (live) {
                const float cy = (float)(R.so[1] + (tile % nty) * 8) + 3.5f, cz = (float)(R.so[2] + (tile / nty) * 4) + 1.5f;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const float a = R.lit[k][0], b2 = R.lit[k][1];
                    if (fmaf(a, cy, fmaf(b2, cz, R.lit[k][2])) + 3.5f * fabsf(a) + 1.5f * fabsf(b2) < least) live = false;
                }
                float a = 0.f, e = (float)(R.rev[0] - 1);
#pragma unroll
                for (int k = 0; k < 3; k++) {  // line_read_span, for all lines of the tile
                    const float c = R.B0[k] + R.By[k] * cy + R.Bz[k] * cz;
                    const float D = 2.1f + fabsf(R.Bx[k]) + 4.5f * fabsf(R.By[k]) + 2.5f * fabsf(R.Bz[k]);
                    const float lo = -D - c, hi = (float)G.bev[k] + D - c;
                    if (R.iB[k] == 0.f) {
                        if (lo > 0.f || hi < 0.f) live = false;
                    } else {
                        a = fmaxf(a, fminf(lo * R.iB[k], hi * R.iB[k]));
                        e = fminf(e, fmaxf(lo * R.iB[k], hi * R.iB[k]));
                    }
                }
                if (a > e + 3.f || !added) live = false;
            }
            const unsigned m = __ballot_sync(FULL, live);
            int base = 0;
            if ((threadIdx.x & 31) == 0 && m) base = atomicAdd(&s_n, __popc(m));
            base = __shfl_sync(FULL, base, 0);
            if (live) tiles[(size_t)seg * cap + base + __popc(m & ((1u << (threadIdx.x & 31)) - 1u))] = tile;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) counts[1 + seg] = s_n;
}

// Runs `line` for every listed tile, a lane per line.  The warps are resident
// (24 per SM at 80 registers; 28 and 32 measured the same and 4 % slower, 20 and
// 16 3 % and 6 % slower): each starts on the tile of its number and takes the
// next from the counter when it is done, not before, or the last tiles wait
// behind long ones while other warps idle (one 24 x 24 beam 1.03 against
// 1.15 ms).  Tiles are taken beam by beam, so that the beams in work stay in L2
// (one list of all beams, filled in the order the blocks happened to run: 96
// beams of 8^2..40^2 beamlets 11.1 against 10.5 ms).  So the scratch of a
// tile's samples is a warp's and not a REV array's: 8 of the 12 to 16 bytes
// that a REV cell took, and it stays in L2.  On the same chunks the cones run
// as fast as one block per 128 lines did; more beams fit a chunk.
template <class F>
__device__ __forceinline__ void cone_tiles_run(const EeParams& P, const EeConeWork& W, int nbeams, int cap, F line) {
    const int lane = threadIdx.x & 31, slot = blockIdx.x * EE_CONE_BLOCK_WARPS + (threadIdx.x >> 5);
    float4* scratch = W.scratch + (size_t)slot * W.quads * 64 + lane;
    const int nseg = nbeams * P.nrays;
    // a window of 32 lists: items before it, this lane's list and the items up
    // to and with it
    int seg0 = 0, base = 0, upto = 0, mine = 0;
    auto load = [&]() {
        mine = seg0 + lane < nseg ? W.counts[1 + seg0 + lane] : 0;
        upto = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, upto, o);
            if (lane >= o) upto += y;
        }
    };
    load();
    for (int item = slot;;) {
        int total;
        while (item >= base + (total = __shfl_sync(FULL, upto, 31))) {
            base += total;
            seg0 += 32;
            if (seg0 >= nseg) return;
            load();
        }
        const int l = __ffs((int)__ballot_sync(FULL, item < base + upto)) - 1, seg = seg0 + l;
        const int first = base + __shfl_sync(FULL, upto - mine, l);
        line(seg / P.nrays, list_cone(P, seg % P.nrays), W.tiles[(size_t)seg * cap + item - first] * 32 + lane, scratch);
        if (lane == 0) item = W.warps + atomicAdd(W.counts, 1);
        item = __shfl_sync(FULL, item, 0);
    }
}

// Forward cone, one lane per line.  Both passes walk whole quads of samples
// (4q .. 4q+3): a lane reads and writes a quad's dose and (rho, T) with
// 16-byte accesses, and the warp's 8 x 4 lines cover two whole bricks.
// Only the quads [q0, q1] of the field span have TERMA (0.30 of the samples of
// 64 beams of 8^2..40^2 beamlets; 0.46 are on dark lines, without any).  The
// walk up the line (contributions from k < i) starts at q0, since nothing below
// it has a source, and past q1 it writes the dose itself, since nothing above
// reaches down to it; the walk down the line starts at q1 and takes its
// densities past q0 from the texture.  So each walk visits 0.42 of the
// samples, and the (rho, T) scratch and the partial dose only the span.
// Bound by latency and by the instruction cache (24 warps of 80 registers per
// SM; half of the issue slots; a sample's corners in the TERMA box are
// addressed by steps, and samples at its faces share one loop per quad: 50 ->
// 41 KB of code, 96 beams 10.5 -> 9.4 ms).  Against both walks over the whole
// segment with the box tests at every sample: one 24 x 24 beam 0.427 -> 0.183
// ms, 96 beams of 8^2..40^2 beamlets 27.8 -> 9.4 ms, 20 beams of 128^2 pixels
// 9.7 -> 4.0 ms (200 x 200 x 160 at 2 mm).
// Samples of an end quad outside [i0, i1] get dose 0 (they are inside the
// read span or never read); their zero TERMA and unit factors leave the
// recurrence as it is.
__device__ __forceinline__ void cone_line(const EeParams& P, const EeBeamSpec* __restrict__ specs,
                                          const EeBeamGeom* __restrict__ geoms, const float* __restrict__ terma,
                                          float* __restrict__ rev, int b, int ray, int slot,
                                          float4* __restrict__ smp) {
    const EeBeamGeom& G = geoms[b];
    const EeRayGeom& R = G.ray[ray];
    int tY, tZ;
    if (!lane_line(R, slot, tY, tZ)) return;
    if (lit_form(R, (float)tY, (float)tZ) < EE_LIT_READ) return;  // dark, and never read
    const EeBeamSpec& S = specs[b];
    LineFrame F;
    const LaneSpan s = lane_span(P, S, G, R, tY, tZ, F);
    // bricked REV arena (rev_brick): this line's sample i sits at out + bk_x(i)
    float* out = rev + G.arena_off + R.offset + rev_line(rev_store(R), tY, tZ);
    const bool lit = s.q0 <= s.q1;
    {   // zeros on the rest of the read span, or all of it on a dark line
        int z0, z1;
        line_read_span(G, R, tY, tZ, R.rev[0], z0, z1);
        const int e0 = lit ? s.i0 >> 2 : 0x3fffffff, e1 = lit ? s.i1 >> 2 : 0x3fffffff;
#pragma unroll 1
        for (int q = z0 >> 2; q <= (z1 >> 2); q++) {
            if (q == e0) q = e1;
            else *reinterpret_cast<float4*>(out + 64 * q) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    if (!lit) return;
    const float* tb = terma + S.t_off;
    const Brick Bt = brick_of(S.tn);
    const f3 t0 = mk((float)S.t0[0], (float)S.t0[1], (float)S.t0[2]);
    const EeRayConst& RC = P.rays[ray];
    const float inv_nphi = 1.f / (float)P.nphi;
    const int qe = s.i1 >> 2, qs = s.i0 >> 2;
    {   // up the line: contributions from k < i, kernel row P
        const float* prm = P.expp + 4 * RC.row_fwd;
        const float c1 = prm[0] / prm[1], c2 = prm[2] / prm[3];
        const float e1 = -0.5f * prm[1] * P.lng, e2 = -0.5f * prm[3] * P.lng;
        float Y1 = 0.f, Y2 = 0.f, tm = 0.f, hm1 = 1.f, hm2 = 1.f;
        auto step = [&](float r, float t) {  // a sample's dose from below
            const bool v = r >= 0.f;
            const float h1 = v ? __expf(e1 * r) : 1.f, h2 = v ? __expf(e2 * r) : 1.f;
            const float d = v ? c1 * (Y1 + tm * (1.f - hm1)) + c2 * (Y2 + tm * (1.f - hm2)) : 0.f;
            Y1 = fmaf(h1 * h1, Y1, tm * h1 * (1.f - hm1 * h1));
            Y2 = fmaf(h2 * h2, Y2, tm * h2 * (1.f - hm2 * h2));
            tm = t; hm1 = h1; hm2 = h2;
            return d;
        };
#pragma unroll 1
        for (int q = s.q0; q <= s.q1; q++) {
            // the quad's samples gathered before the recurrence consumes
            // them, so each lane keeps several independent loads in flight
            float rr[4], tt[4], dq[4];
            unsigned edge = 0;  // samples with corners outside the TERMA box
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int i = 4 * q + j;
                const bool in = i >= s.i0 && i <= s.i1;
                const f3 g = sample_point(F, i);
                rr[j] = rho_at(P, g);
                if (!in) rr[j] = -1.f;
                const f3 p = mk(g.x - t0.x, g.y - t0.y, g.z - t0.z);
                int ci, cj, ck;
                const bool cell = brick_cell(Bt, p.x, p.y, p.z, ci, cj, ck);
                tt[j] = cell ? tri_brick_cell(tb, Bt, p.x, p.y, p.z, ci, cj, ck) : 0.f;
                edge |= cell ? 0u : 1u << j;
                if (!(rr[j] >= 0.f)) tt[j] = 0.f;
            }
#pragma unroll 1
            for (; edge; edge &= edge - 1) {
                const int w = __ffs((int)edge) - 1;
                const f3 g = sample_point(F, 4 * q + w);
                const float e = tri_brick_edge(tb, Bt, g.x - t0.x, g.y - t0.y, g.z - t0.z);
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (j == w && rr[j] >= 0.f) tt[j] = e;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) dq[j] = step(rr[j], tt[j]);
            float4* sq = smp + 64 * (q - s.q0);  // (rho, T)
            sq[0] = make_float4(rr[0], tt[0], rr[1], tt[1]);
            sq[32] = make_float4(rr[2], tt[2], rr[3], tt[3]);
            *reinterpret_cast<float4*>(out + 64 * q) = make_float4(dq[0], dq[1], dq[2], dq[3]);
        }
#pragma unroll 1
        for (int q = s.q1 + 1; q <= qe; q++) {
            float rr[4], dq[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int i = 4 * q + j;
                rr[j] = rho_at(P, sample_point(F, i));
                if (i > s.i1) rr[j] = -1.f;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) dq[j] = step(rr[j], 0.f) * inv_nphi;
            *reinterpret_cast<float4*>(out + 64 * q) = make_float4(dq[0], dq[1], dq[2], dq[3]);
        }
    }
    {   // down the line: contributions from k > i, kernel row ntheta-1-P
        const float* prm = P.expp + 4 * RC.row_rev;
        const float c1 = prm[0] / prm[1], c2 = prm[2] / prm[3];
        const float e1 = -0.5f * prm[1] * P.lng, e2 = -0.5f * prm[3] * P.lng;
        float Y1 = 0.f, Y2 = 0.f, tm = 0.f, hm1 = 1.f, hm2 = 1.f;
        auto step = [&](float r, float t, float below) {
            const bool v = r >= 0.f;
            const float h1 = v ? __expf(e1 * r) : 1.f, h2 = v ? __expf(e2 * r) : 1.f;
            const float d = c1 * (Y1 + tm * (1.f - hm1)) + c2 * (Y2 + tm * (1.f - hm2));
            Y1 = fmaf(h1 * h1, Y1, tm * h1 * (1.f - hm1 * h1));
            Y2 = fmaf(h2 * h2, Y2, tm * h2 * (1.f - hm2 * h2));
            tm = t; hm1 = h1; hm2 = h2;
            return v ? (below + d) * inv_nphi : 0.f;
        };
#pragma unroll 1
        for (int q = s.q1; q >= s.q0; q--) {
            const float4* sq = smp + 64 * (q - s.q0);
            const float4 s01 = sq[0], s23 = sq[32];
            const float4 o4 = *reinterpret_cast<const float4*>(out + 64 * q);
            float4 dq;
            dq.w = step(s23.z, s23.w, o4.w);
            dq.z = step(s23.x, s23.y, o4.z);
            dq.y = step(s01.z, s01.w, o4.y);
            dq.x = step(s01.x, s01.y, o4.x);
            *reinterpret_cast<float4*>(out + 64 * q) = dq;
        }
#pragma unroll 1
        for (int q = s.q0 - 1; q >= qs; q--) {
            float rr[4], dq[4];
#pragma unroll
            for (int j = 3; j >= 0; j--) {
                const int i = 4 * q + j;
                rr[j] = rho_at(P, sample_point(F, i));
                if (i < s.i0) rr[j] = -1.f;
            }
#pragma unroll
            for (int j = 3; j >= 0; j--) dq[j] = step(rr[j], 0.f, 0.f);
            *reinterpret_cast<float4*>(out + 64 * q) = make_float4(dq[0], dq[1], dq[2], dq[3]);
        }
    }
}

__global__ void __launch_bounds__(EE_CONE_BLOCK_WARPS * 32, EE_CONE_SM_WARPS / EE_CONE_BLOCK_WARPS)
    k_cone_lane(EeParams P, const EeBeamSpec* __restrict__ specs, const EeBeamGeom* __restrict__ geoms,
                const float* __restrict__ terma, float* __restrict__ rev, EeConeWork W, int nbeams, int cap) {
    cone_tiles_run(P, W, nbeams, cap, [&](int b, int ray, int slot, float4* scratch) {
        cone_line(P, specs, geoms, terma, rev, b, ray, slot, scratch);
    });
}

// Zero the samples of the chunk's REV gradient arena that the adjoint cones
// may read, before k_gather_T adds into it: the quads of each line's
// line_clear_span, which holds the samples that the cones find for themselves
// whatever their own end tests decide (the arena holds the forward's dose
// before that).  k_gather_T also adds into the rest; those cells are never
// read, so they need no zero.  A warp's 16-byte stores cover two whole bricks.
template <int LANE_BLOCK>
__global__ void __launch_bounds__(LANE_BLOCK) k_rev_zero(EeParams P, const EeBeamGeom* __restrict__ geoms,
                                                         float* __restrict__ rev_grad,
                                                         unsigned char* __restrict__ touched, int cap) {
    const int ray = blockIdx.y, b = blockIdx.z;
    if (const int t = blockIdx.x * LANE_BLOCK + threadIdx.x; touched && t < cap)  // none yet
        touched[(size_t)(b * P.nrays + ray) * cap + t] = 0;
    const EeBeamGeom& G = geoms[b];
    if (G.status != 0) return;
    const EeRayGeom& R = G.ray[ray];
    int tY, tZ;
    if (!lane_line(R, blockIdx.x * LANE_BLOCK + threadIdx.x, tY, tZ)) return;
    int i0, i1;
    line_clear_span(P, G, R, tY, tZ, i0, i1);
    float* row = rev_grad + G.arena_off + R.offset + rev_line(rev_store(R), tY, tZ);
    for (int ib = i0 & ~3; ib <= i1; ib += 4)
        *reinterpret_cast<float4*>(row + bk_x(ib)) = make_float4(0.f, 0.f, 0.f, 0.f);
}

// Adjoint of k_cone_lane followed by the transpose of the REV TERMA resample.
// With g_i the incoming REV-dose gradient (/ nphi), each walk carries the
// neighbour it came from (g, h and Z of sample m's neighbour i):
//   Tbar_m += c g_i (1 - h_m) + Z h_i (1 - h_m h_i),   Z <- h_i^2 Z + c g_i.
// Pass A walks down (transpose of the walk up) and keeps its part of Tbar
// with rho in the warp's scratch; pass B walks up, adds its
// part and scatters Tbar into the TERMA-box gradient.  Only the quads [q0, q1]
// of the field span have a TERMA gradient: pass A stops below q0, pass B
// above q1, and outside the span each only updates Z, with the densities of
// the texture; the scratch holds the span alone.  A quad is loaded while the one
// before it is worked on.  Bound by the reductions into the TERMA gradient
// (half of the time) and by latency: one 24 x 24 beam 0.428 -> 0.143 ms, 20
// beams of 128^2 pixels 8.1 -> 2.6 ms, of which 0.247 -> 0.143 and 2.93 -> 2.64
// by reducing into quads (quad_scatter) and loading ahead; 0.8 where only the
// tiles with a gradient are listed (k_cone_tiles).
__device__ __forceinline__ void cone_T_line(const EeParams& P, const EeBeamSpec* __restrict__ specs,
                                            const EeBeamGeom* __restrict__ geoms, const float* __restrict__ rev_grad,
                                            float4* __restrict__ terma_grad, int b, int ray, int slot,
                                            float4* __restrict__ sA) {
    const EeBeamGeom& G = geoms[b];
    const EeRayGeom& R = G.ray[ray];
    int tY, tZ;
    if (!lane_line(R, slot, tY, tZ)) return;
    const EeBeamSpec& S = specs[b];
    LineFrame F;
    const LaneSpan s = lane_span(P, S, G, R, tY, tZ, F);
    if (s.q1 < s.q0) return;
    const float* gin = rev_grad + G.arena_off + R.offset + rev_line(rev_store(R), tY, tZ);
    const EeRayConst& RC = P.rays[ray];
    const float inv_nphi = 1.f / (float)P.nphi;
    // the neighbour's state; Z before the neighbour's own update
    float gn, h1, h2, Z1, Z2, c1, c2, e1, e2;
    auto begin = [&](int row) {
        const float* prm = P.expp + 4 * row;
        c1 = prm[0] / prm[1];
        c2 = prm[2] / prm[3];
        e1 = -0.5f * prm[1] * P.lng;
        e2 = -0.5f * prm[3] * P.lng;
        gn = 0.f; h1 = 1.f; h2 = 1.f; Z1 = 0.f; Z2 = 0.f;
    };
    auto step = [&](float r, float g) {  // the walk's part of sample m's Tbar
        const bool v = r >= 0.f;
        const float hm1 = v ? __expf(e1 * r) : 1.f, hm2 = v ? __expf(e2 * r) : 1.f;
        const float e = v ? c1 * gn * (1.f - hm1) + Z1 * h1 * (1.f - hm1 * h1) + c2 * gn * (1.f - hm2) +
                                Z2 * h2 * (1.f - hm2 * h2)
                          : 0.f;
        Z1 = fmaf(h1 * h1, Z1, c1 * gn);
        Z2 = fmaf(h2 * h2, Z2, c2 * gn);
        gn = v ? g * inv_nphi : 0.f;
        h1 = hm1; h2 = hm2;
        return e;
    };
    // a quad's densities and gradients; the walks load a quad while they work on
    // the one before it
    auto load = [&](int q, float (&r)[4], float4& g) {
        g = *reinterpret_cast<const float4*>(gin + 64 * q);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int i = 4 * q + j;
            r[j] = rho_at(P, sample_point(F, i));
            if (i < s.i0 || i > s.i1) r[j] = -1.f;
        }
    };
    {   // pass A, down from i1
        begin(RC.row_fwd);
        float rn[4];
        float4 gn4;
        load(s.i1 >> 2, rn, gn4);
#pragma unroll 1
        for (int q = s.i1 >> 2; q >= s.q0; q--) {
            const float gl[4] = {gn4.x, gn4.y, gn4.z, gn4.w};
            float rl[4], e[4];
#pragma unroll
            for (int j = 0; j < 4; j++) rl[j] = rn[j];
            if (q > s.q0) load(q - 1, rn, gn4);
#pragma unroll
            for (int j = 3; j >= 0; j--) e[j] = step(rl[j], gl[j]);
            if (q <= s.q1) {
                float4* sq = sA + 64 * (q - s.q0);  // (pass-A part of Tbar, rho)
                sq[0] = make_float4(e[0], rl[0], e[1], rl[1]);
                sq[32] = make_float4(e[2], rl[2], e[3], rl[3]);
            }
        }
    }
    {   // pass B, up from i0; scatter
        begin(RC.row_rev);
#pragma unroll 1
        for (int q = s.i0 >> 2; q < s.q0; q++) {
            const float4 g4 = *reinterpret_cast<const float4*>(gin + 64 * q);
            const float gl[4] = {g4.x, g4.y, g4.z, g4.w};
            float rl[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int i = 4 * q + j;
                rl[j] = rho_at(P, sample_point(F, i));
                if (i < s.i0) rl[j] = -1.f;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) step(rl[j], gl[j]);
        }
        float4* tg = terma_grad + S.q_off;
        const Brick Bt = quads_of(S.tn);
        const f3 t0 = mk((float)S.t0[0], (float)S.t0[1], (float)S.t0[2]);
        float4 n01 = sA[0], n23 = sA[32], n4 = *reinterpret_cast<const float4*>(gin + 64 * s.q0);
#pragma unroll 1
        for (int q = s.q0; q <= s.q1; q++) {
            const float4 s01 = n01, s23 = n23, g4 = n4;
            if (q < s.q1) {
                const float4* sq = sA + 64 * (q + 1 - s.q0);
                n01 = sq[0];
                n23 = sq[32];
                n4 = *reinterpret_cast<const float4*>(gin + 64 * (q + 1));
            }
            const float al[4] = {s01.x, s01.z, s23.x, s23.z}, rl[4] = {s01.y, s01.w, s23.y, s23.w};
            const float gl[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float tot = al[j] + step(rl[j], gl[j]);
                if (rl[j] >= 0.f && tot != 0.f) {
                    const f3 g = sample_point(F, 4 * q + j);
                    quad_scatter(tg, Bt, g.x - t0.x, g.y - t0.y, g.z - t0.z, tot);
                }
            }
        }
    }
}

__global__ void __launch_bounds__(EE_CONE_BLOCK_WARPS * 32, EE_CONE_SM_WARPS / EE_CONE_BLOCK_WARPS)
    k_cone_T_lane(EeParams P, const EeBeamSpec* __restrict__ specs, const EeBeamGeom* __restrict__ geoms,
                  const float* __restrict__ rev_grad, EeConeWork W, int nbeams, int cap,
                  float4* __restrict__ terma_grad) {
    cone_tiles_run(P, W, nbeams, cap, [&](int b, int ray, int slot, float4* scratch) {
        cone_T_line(P, specs, geoms, rev_grad, terma_grad, b, ray, slot, scratch);
    });
}

// Adjoint of k_cone with the table walk, followed by the transpose of the REV TERMA resample:
// terma_grad (bbox grid) += R_T^T C^T rev_grad.
__global__ void __launch_bounds__(CONE_WARPS * 32) k_cone_T(EeParams P, const EeBeamSpec* __restrict__ specs,
                                                            const EeBeamGeom* __restrict__ geoms,
                                                            const float* __restrict__ rev_grad,
                                                            float4* __restrict__ terma_grad, int maxL) {
    extern __shared__ float sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ray = blockIdx.y, b = blockIdx.z;
    const EeBeamGeom& G = geoms[b];
    float* tabK = sm + (size_t)CONE_WARPS * 3 * maxL;
    float* tabR = tabK + 2 * EE_MAX_RADII;
    const EeRayConst& RC = P.rays[ray];
    for (int k = threadIdx.x; k < P.nradii; k += blockDim.x) {
        tabK[k] = P.cumkern[RC.row_fwd * P.nradii + k];
        tabK[EE_MAX_RADII + k] = P.cumkern[RC.row_rev * P.nradii + k];
        tabR[k] = P.radii[k];
    }
    __syncthreads();
    if (G.status != 0) return;
    const EeRayGeom& R = G.ray[ray];
    const int line = blockIdx.x * CONE_WARPS + warp;
    if (line >= R.nlines) return;
    const int L = R.rev[0];
    int tY, tZ;
    kept_line(R, line, tY, tZ);
    if (lit_form(R, (float)tY, (float)tZ) < 0.f) return;
    float* rho = sm + (size_t)warp * 3 * maxL;
    float* g = rho + maxL;
    float* Tb = g + maxL;
    const EeBeamSpec& S = specs[b];
    int i0, n;
    line_segment(P, G, R, tY, tZ, L, i0, n);
    if (n == 0) return;
    gather_line(P, S, G, R, nullptr, tY, tZ, i0, n, lane, rho, nullptr);
    const Brick Bv = rev_store(R);  // bricked REV gradient
    const float* gin = rev_grad + G.arena_off + R.offset + rev_line(Bv, tY, tZ);
    const float inv_nphi = 1.f / (float)P.nphi;
    __syncwarp();
    for (int k = lane; k < n; k += 32) {
        g[k] = rho[k] >= 0.f ? gin[bk_x(i0 + k)] * inv_nphi : 0.f;
        Tb[k] = 0.f;
    }
    __syncwarp();
    for (int k = lane; k < n; k += 32) {
        if (rho[k] >= 0.f && g[k] != 0.f) {
            table_walk(rho, nullptr, n, k, -1, tabK, tabR, P.nradii, P.lng, Tb, g[k]);
            table_walk(rho, nullptr, n, k, +1, tabK + EE_MAX_RADII, tabR, P.nradii, P.lng, Tb, g[k]);
        }
    }
    __syncwarp();
    // transpose of the REV TERMA resample
    const LineFrame F{line_point(R.G0, R.Gy, R.Gz, (float)tY, (float)tZ), ld3(R.Gx)};
    float4* tg = terma_grad + S.q_off;
    for (int k = lane; k < n; k += 32) {
        float v = Tb[k];
        if (rho[k] < 0.f || v == 0.f) continue;
        f3 gp = sample_point(F, i0 + k);
        quad_scatter(tg, quads_of(S.tn), gp.x - (float)S.t0[0], gp.y - (float)S.t0[1],
                           gp.z - (float)S.t0[2], v);
    }
}

// ------------------------------------------------------------- gather ----
// Voxel range [x0, x1] of patient row (y, z) whose BEV index lies within the
// crop box dilated by 2 voxels (the BEV index is affine in x), widened by one
// voxel for rounding and clipped to the calc bbox.
__device__ __forceinline__ bool row_span(const EeParams& P, const EeBeamSpec& S, const EeBeamGeom& G, int y, int z,
                                         int& x0, int& x1) {
    float xa = (float)P.bb0[0], xb = (float)(P.bb0[0] + P.bbs[0] - 1);
    const float dy = (float)y - G.lim_off[1], dz = (float)z - G.lim_off[2];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        float m = S.MB[3 * a];
        float c = S.MB[3 * a + 1] * dy + S.MB[3 * a + 2] * dz - m * G.lim_off[0];
        float lo = -2.f, hi = (float)G.bev[a] + 2.f;
        if (fabsf(m) < 1e-6f) {
            if (c < lo - 1e-3f || c > hi + 1e-3f) return false;
        } else {
            float t0 = (lo - c) / m, t1 = (hi - c) / m;
            xa = fmaxf(xa, fminf(t0, t1));
            xb = fminf(xb, fmaxf(t0, t1));
        }
    }
    if (!(xa <= xb + 2.f)) return false;
    x0 = max(P.bb0[0], (int)floorf(xa) - 1);
    x1 = min(P.bb0[0] + P.bbs[0] - 1, (int)ceilf(xb) + 1);
    return x0 <= x1;
}

constexpr int ROW_WARPS = 8;

// REV2XYZdose (device.cu:222-261) for all cones at once, a cone only at the
// voxels whose lines it can light (lit_planes): the others read zeros.  A warp
// takes a group of PY x PZ patient rows (EE_GATHER_*) of one beam's AABB and sweeps
// the union of their spans in PX x PY x PZ patches, V of them at a time
// (one voxel of each per lane): a compact patch of voxels maps to a compact
// patch of REV cells, so a corner load of the warp touches fewer cache lines
// than a run of 32 voxels along x would.  A voxel sums the trilinear REV dose
// of every cone.  mode 0/1: atomic accumulation into dose; mode 2: dose[b]
// written directly.
//
// Bound by the load/store unit's data pipe (three quarters of its cycles): a
// corner load of 32 scattered words takes two to three passes over the banks.
// One read of a cone's map serves V voxels; five resident blocks (48 registers,
// a few spilled words) beat four without spills, and six.  96 beams of 8^2..40^2
// beamlets on 200 x 200 x 160: 18.1 ms with one voxel per lane (40 registers),
// 17.5 with two, 17.1 with four; 12.6 without the dark cones, 8.7 in chunks of
// 15 beams and more.  gridDim.y blocks share a group's patches, every
// gridDim.y-th V of them each (ee_launch_gather).
template <int V>
__global__ void __launch_bounds__(ROW_WARPS * 32, 5) k_gather(EeParams P, const EeBeamSpec* __restrict__ specs,
                                                           const EeBeamGeom* __restrict__ geoms,
                                                           const float* __restrict__ rev, float* __restrict__ dose,
                                                           int mode, long long nfull) {
    const int b = blockIdx.z;
    const EeBeamGeom& G = geoms[b];
    if (G.status != 0) return;
    // the beam's cone maps, staged once per block: rows of [A | -q0] (REV
    // from crop-box-relative patient index), (rev sizes, arena offset) and
    // the REV array's brick strides
    __shared__ float4 s_ray[EE_MAX_RAYS][5];
    for (int k = threadIdx.x; k < P.nrays * 5; k += blockDim.x) {
        const int r = k / 5, c = k - 5 * r;
        const EeRayGeom& R = G.ray[r];
        float4 v;
        if (c < 3) {
            v = make_float4(R.A[3 * c], R.A[3 * c + 1], R.A[3 * c + 2], -R.q0[c]);
        } else if (c == 4) {
            const Brick Bq = rev_store(R);
            v = make_float4(__int_as_float(Bq.sy), __int_as_float(Bq.sz), 0.f, 0.f);
        } else {
            v = make_float4(__int_as_float(R.rev[0]), __int_as_float(R.rev[1]), __int_as_float(R.rev[2]),
                            __int_as_float((int)R.offset));
        }
        s_ray[r][c] = v;
    }
    // voxels [x, y] of a row (from the group's first) whose lines can be lit
    constexpr int PX = EE_GATHER_PX, PY = EE_GATHER_PY, ROWS = EE_GATHER_PY * EE_GATHER_PZ;
    __shared__ ushort2 s_lit[ROW_WARPS][EE_MAX_RAYS][ROWS];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = blockIdx.x * ROW_WARPS + warp;
    if (grp >= G.rows) return;
    const int ngy = (G.gny + PY - 1) / PY;
    const int lx = lane % PX, row = lane / PX;
    const int yy = (grp % ngy) * PY + row % PY, zz = (grp / ngy) * EE_GATHER_PZ + row / PY;
    const int y = G.gy0 + yy, z = G.gz0 + zz;
    const EeBeamSpec& S = specs[b];
    int x0 = 0, x1 = -1;
    if (yy >= G.gny || zz >= G.gnz || !row_span(P, S, G, y, z, x0, x1)) {
        x0 = 0;
        x1 = -1;
    }
    const int wx0 = __reduce_min_sync(FULL, x0 <= x1 ? x0 : INT_MAX);
    const int wx1 = __reduce_max_sync(FULL, x0 <= x1 ? x1 : INT_MIN);
    if (wx0 > wx1) return;
    float* out = dose + S.out_off + (mode == 2 ? (long long)b * nfull : 0ll);
    const long long rbase = (long long)P.size[0] * (y + (long long)P.size[1] * z);
    const float* base = rev + G.arena_off;
    const float dy = (float)y - G.lim_off[1], dz = (float)z - G.lim_off[2];
    if (wx0 + (int)blockIdx.y * V * PX > wx1) return;
    const float dx0 = (float)wx0 - G.lim_off[0];
    for (int r = lx; r < P.nrays; r += PX) {  // a row's eight lanes take its cones in turn
        float lo = 0.f, hi = 65535.f;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float4 f = lit_voxel_form(G.ray[r], k);
            const float c = fmaf(f.x, dx0, fmaf(f.y, dy, fmaf(f.z, dz, f.w)));
            if (fabsf(f.x) < 1e-6f) {
                if (c < 0.f) hi = -1.f;
            } else {
                const float t = fminf(fmaxf(__fdividef(-c, f.x), -1e6f), 1e6f);
                if (f.x > 0.f) lo = fmaxf(lo, t);
                else hi = fminf(hi, t);
            }
        }
        const int a = min((int)ceilf(lo - 0.01f), 65535), e = (int)floorf(hi + 0.01f);
        s_lit[warp][r][row] = e < 0 ? make_ushort2(1, 0) : make_ushort2((unsigned short)max(a, 0), (unsigned short)min(e, 65535));
    }
    __syncwarp();
    for (int xs = wx0 + lx + blockIdx.y * V * PX; xs - lx <= wx1; xs += gridDim.y * V * PX) {
        float dx[V], acc[V];
        int rel[V];  // from the group's first voxel; -1: nothing to sum
#pragma unroll
        for (int v = 0; v < V; v++) {
            const int x = xs + v * PX;
            dx[v] = (float)x - G.lim_off[0];
            acc[v] = 0.f;
            // voxels more than 2 BEV voxels outside the crop box see no REV dose
            const f3 bi = mv(S.MB, mk(dx[v], dy, dz));
            const bool in = x >= x0 && x <= x1 &&
                            !(bi.x < -2.f || bi.y < -2.f || bi.z < -2.f || bi.x > G.bev[0] + 2.f ||
                              bi.y > G.bev[1] + 2.f || bi.z > G.bev[2] + 2.f);
            rel[v] = in ? min(x - wx0, 65535) : -1;
        }
        for (int r = 0; r < P.nrays; r++) {
            const ushort2 lit = s_lit[warp][r][row];
            bool on[V], any = false;
#pragma unroll
            for (int v = 0; v < V; v++) {
                on[v] = rel[v] >= (int)lit.x && rel[v] <= (int)lit.y;
                any |= on[v];
            }
            if (!__any_sync(FULL, any)) continue;
            const float4 a0 = s_ray[r][0], a1 = s_ray[r][1], a2 = s_ray[r][2], rv = s_ray[r][3], st = s_ray[r][4];
            // bricked REV arrays over (i, tY, tZ): q.y along the line (rev[0]),
            // q.z -> rev[1], q.x -> rev[2]
            Brick Bq;
            Bq.n0 = __float_as_int(rv.x); Bq.n1 = __float_as_int(rv.y); Bq.n2 = __float_as_int(rv.z);
            Bq.sy = __float_as_int(st.x); Bq.sz = __float_as_int(st.y);
            const float* cone = base + __float_as_int(rv.w);
            const float cx = fmaf(a0.y, dy, fmaf(a0.z, dz, a0.w)), cy = fmaf(a1.y, dy, fmaf(a1.z, dz, a1.w)),
                        cz = fmaf(a2.y, dy, fmaf(a2.z, dz, a2.w));
#pragma unroll
            for (int v = 0; v < V; v++) {
                const float qx = fmaf(a0.x, dx[v], cx), qy = fmaf(a1.x, dx[v], cy), qz = fmaf(a2.x, dx[v], cz);
                if (on[v] && !(qy >= (float)Bq.n0 || qz >= (float)Bq.n1 || qx >= (float)Bq.n2 || qx < 0.f ||
                               qy < 0.f || qz < 0.f))
                    acc[v] += tri_brick_in(cone, Bq, qy, qz, qx);
            }
        }
#pragma unroll
        for (int v = 0; v < V; v++) {
            const int x = xs + v * PX;
            if (x < x0 || x > x1) continue;
            if (mode == 2) out[rbase + x] = acc[v];
            else if (acc[v] != 0.f) atomicAdd(out + rbase + x, acc[v]);
        }
    }
}

// Transpose of k_gather's per-voxel sum: rev_grad += S^T dose_grad, one block per
// 8x8x4 tile of patient voxels.  For each cone the tile's trilinear
// footprint in the REV grid (an AABB computed from the tile's corners under
// the affine patient -> REV map) is accumulated in shared memory first, then
// flushed with one global reduction per non-zero quad of REV samples.  The
// footprints of all cones are computed up front; consecutive cones alternate
// between two shared buffers.  The flush clears the quads it sends, so every
// buffer is all zero again when its next cone scatters into it, and one
// barrier per cone (between its scatter and its flush) suffices.
//
// The shared boxes accumulate in 32-bit fixed point: integer adds are native
// shared-memory atomics, while a float add to shared memory is a
// compare-and-swap loop (measured on the whole kernel: 1.41x as long with
// float adds; the integer form within 2 % of non-atomic adds, which give wrong
// sums and served only as a bound).  A cone that cannot light a line near the
// tile is skipped (lit_planes; one 24 x 24 beam 0.208 -> 0.162 ms).  Each tile
// scales its
// gradients by a power of two s with max|g| * s in [2^21, 2^22), so one
// contribution w * g * s (w <= 1) is below 2^22 in magnitude and rounds to
// an integer exactly through the FP32 sum with 1.5 * 2^23; a box cell takes
// at most one contribution per tile voxel, so its sum stays below
// 256 * 2^22 = 2^30.  The rounding error per contribution is at most
// 2^-22 max|g| of the tile, about FP32 rounding at the tile's largest
// gradient; the flush converts each sum back with the exact factor 1 / s.
//
// Bound by instruction issue (three quarters of the slots) and the conversion
// unit, which takes 8 cycles per warp: what is the same for a tile's voxels is
// worked out once per tile and cone, the cells come from roundings at unit
// spacing and the quads' places from multiplications by 2^-20 reciprocals (four
// conversions per quad and three per voxel less: six beams 0.721 -> 0.642 ms,
// 12 beams 1.65 -> 1.48).  Five blocks per SM at 48 registers; four at 56 are
// 2 % slower on those and 5 % faster on one beam.
constexpr int GT_TX = 8, GT_TY = 8, GT_TZ = 4;
// floats per footprint buffer: an 8x8x4 tile spans at most |(7,7,3)| + 2 = 13
// REV cells per axis when the REV spacing equals the voxel size (16 along i
// after the quad alignment; 16 x 13 x 13 = 2704 < 4096).  A box clipped at
// the array's end takes one cell more on that axis, which can pass 4096 only
// for a tile at the array's corner under the widest rotation; such boxes and
// larger footprints (finer REV spacing) take the direct-scatter path
constexpr int GT_BUF = 4096;
constexpr int GT_SMEM = 2 * GT_BUF;

__global__ void __launch_bounds__(GT_TX * GT_TY * GT_TZ, 5) k_gather_T(EeParams P, const EeBeamSpec* __restrict__ specs,
                                                                   const EeBeamGeom* __restrict__ geoms,
                                                                   const float* __restrict__ dose_grad,
                                                                   float* __restrict__ rev_grad,
                                                                   unsigned char* __restrict__ touched, int cap) {
    extern __shared__ int acc_all[];  // two fixed-point footprint boxes
    // per cone, the box of its footprint (origin l, extent n over i, tY and tZ):
    // [0] {l0 | n0 << 16, l1 | n1 << 16, l2 | n2 << 16, row stride s0} until the
    // second step below, then {s0, slab stride, l1 | l2 << 16, 16 l0}; [1] the
    // REV gradient's {sy, sz, offset lo, offset hi}; [2] {rev[0], rev[1], rev[2]
    // as floats, the constant of a voxel's cell}; [3] {k0, k1, k2 | k each, lo |
    // hi << 16} (the box cells inside the kept part, which the flush sends), rows
    // per slab; [4] {quads per row, its and the slab's rows' reciprocals in
    // 2^-20, nquad | 1 << 16 where the box lies in the kept part}
    __shared__ int4 s_p[EE_MAX_RAYS][5];
    __shared__ float4 s_A[EE_MAX_RAYS][3];
    __shared__ int s_list[EE_MAX_RAYS], s_n;  // cones with a box
    // line tiles of the box's kept lines: first and end in tY and tZ, tiles per row
    __shared__ ushort2 s_tile[EE_MAX_RAYS][2];
    __shared__ unsigned short s_nty[EE_MAX_RAYS];
    const int b = blockIdx.z;
    const EeBeamGeom& G = geoms[b];
    if (G.status != 0 || (int)blockIdx.x >= G.tiles) return;
    const EeBeamSpec& S = specs[b];
    const int ntx = (G.gnx + GT_TX - 1) / GT_TX, nty = (G.gny + GT_TY - 1) / GT_TY;
    const int tile = blockIdx.x;
    const int ox = G.gx0 + (tile % ntx) * GT_TX, oy = G.gy0 + ((tile / ntx) % nty) * GT_TY,
              oz = G.gz0 + (tile / (ntx * nty)) * GT_TZ;
    const int t = threadIdx.x;
    const int x = ox + t % GT_TX, y = oy + (t / GT_TX) % GT_TY, z = oz + t / (GT_TX * GT_TY);
    float gd = 0.f;
    const float dx = (float)x - G.lim_off[0], dy = (float)y - G.lim_off[1], dz = (float)z - G.lim_off[2];
    if (x < G.gx0 + G.gnx && y < G.gy0 + G.gny && z < G.gz0 + G.gnz) {
        gd = __ldg(dose_grad + S.out_off + x + (long long)P.size[0] * (y + (long long)P.size[1] * z));
        const f3 bi = mv(S.MB, mk(dx, dy, dz));
        if (bi.x < -2.f || bi.y < -2.f || bi.z < -2.f || bi.x > G.bev[0] + 2.f || bi.y > G.bev[1] + 2.f ||
            bi.z > G.bev[2] + 2.f)
            gd = 0.f;
    }
    __shared__ int s_gmax;  // bits of the tile's largest |gradient| (ordered as ints)
    if (t == 0) s_gmax = 0;
    if (!__syncthreads_or(gd != 0.f)) return;
    {
        const int m = __reduce_max_sync(0xffffffffu, __float_as_int(fabsf(gd)));
        if ((t & 31) == 0 && m != 0) atomicMax(&s_gmax, m);
    }
    // tile origin relative to the crop box, in patient index units
    const float o0 = (float)ox - G.lim_off[0], o1 = (float)oy - G.lim_off[1], o2 = (float)oz - G.lim_off[2];
    // REV footprint of the tile for every cone: q(v) = A (v - lim_off) - q0,
    // one (cone, REV axis) per thread; bounds widened by 1e-3 so that the
    // per-voxel q (formed in another order) never falls outside
    for (int k = t; k < 3 * P.nrays; k += blockDim.x) {
        const int r = k / 3, a = k - 3 * r;
        const EeRayGeom& R = G.ray[r];
        const float ext[3] = {(float)(GT_TX - 1), (float)(GT_TY - 1), (float)(GT_TZ - 1)};
        const float* Ar = R.A + 3 * a;
        float lo = Ar[0] * o0 + Ar[1] * o1 + Ar[2] * o2 - R.q0[a], hi = lo;
#pragma unroll
        for (int e = 0; e < 3; e++) {
            const float d = Ar[e] * ext[e];
            lo += fminf(d, 0.f);
            hi += fmaxf(d, 0.f);
        }
        // REV axes: q.y -> rev[0] (along the line), q.z -> rev[1], q.x -> rev[2]
        const int dim = a == 1 ? R.rev[0] : (a == 2 ? R.rev[1] : R.rev[2]);
        int l = max(0, (int)floorf(lo - 1e-3f));
        int h = min(dim - 1, (int)floorf(hi + 1e-3f) + 1);
        // A voxel's corners are floor(q) - l and the cell above, and floor(q)
        // <= floor(hi + 1e-3), so unclipped they stay inside [0, h - l].  Where
        // the box is clipped at the array's last cell it gets one more, so the
        // upper corner of a voxel in the last cell lands in the box; the flush
        // drops it (the forward reads 0 past the array).
        if (h == dim - 1 && h >= l) h++;
        int w = h - l + 1;
        if (a == 1) {
            // no voxel of the tile next to a line that can be lit: k_cone_T
            // reads nothing that the cone could add, so its box stays empty
            bool dark = false;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float4 f = lit_voxel_form(R, k);
                const float top = f.x * o0 + f.y * o1 + f.z * o2 + f.w + fmaxf(f.x, 0.f) * ext[0] +
                                  fmaxf(f.y, 0.f) * ext[1] + fmaxf(f.z, 0.f) * ext[2];
                dark |= top < 0.f;
            }
            if (dark) w = 0;
        }
        int* sp = reinterpret_cast<int*>(s_p[r]);
        sp[8 + (a == 1 ? 0 : (a == 2 ? 1 : 2))] = __float_as_int((float)dim);
        if (a == 1) {
            int s0 = 0;
            if (w > 0) {
                // i range on whole quads: a box row of 4 samples is one
                // 16-byte brick row of the REV gradient (flushed as one
                // vector reduction); the cells past rev[0] are brick padding
                w = ((h | 3) + 1) - (l & ~3);
                l &= ~3;
                // row stride 4 (mod 8) floats: the rows of adjacent voxels
                // spread over the shared banks; the extra quad of a row is
                // never scattered to, stays zero and is not sent
                s0 = (w & 7) == 0 ? w + 4 : w;
            }
            sp[3] = s0;
        }
        const int d = a == 1 ? 0 : (a == 2 ? 1 : 2);
        sp[d] = l | (max(w, 0) << 16);
        sp[12 + d] = max(0, R.so[d] - l) | max(0, R.so[d] + R.sn[d] - l) << 16;
        if (d > 0) {
            const int first = max(l - R.so[d], 0), end = max(min(l + max(w, 0) - R.so[d], R.sn[d]), 0);
            const int by = d == 1 ? 3 : 2;
            s_tile[r][d - 1] = first < end ? make_ushort2(first >> by, ((end - 1) >> by) + 1) : make_ushort2(0, 0);
            if (d == 1) s_nty[r] = (unsigned short)((R.sn[1] + 7) >> 3);
        }
        if (a == 0) {
            const Brick Bv = rev_store(R);
            sp[4] = Bv.sy;
            sp[5] = Bv.sz;
            sp[6] = (int)(unsigned)(R.offset & 0xffffffffll);
            sp[7] = (int)(R.offset >> 32);
        }
        // this cone's map for the voxels: the row [A | -q0] of REV axis a
        // (the forward gather forms q in the same order)
        s_A[r][a] = make_float4(Ar[0], Ar[1], Ar[2], -R.q0[a]);
    }
    if (t == 0) s_n = 0;
    __syncthreads();
    for (int r = t; r < P.nrays; r += blockDim.x) {
        int4* const sp = s_p[r];
        const int4 p0 = sp[0], p3 = sp[3];
        const int n0 = p0.x >> 16, n1 = p0.y >> 16, n2 = p0.z >> 16, s0 = p0.w;
        if (n0 <= 0 || n1 <= 0 || n2 <= 0) continue;
        // box cell (k0, k1, k2) over (i, tY, tZ) at k0 + s0 * (k1 + n1p * k2); rows
        // per slab: odd, so that the slab stride s0 * n1p is 4 x odd (mod 32) and
        // the slabs of adjacent voxels spread over the banks too; the padding rows
        // (k1 >= n1) are never scattered to
        const int n1p = n1 | 1, nbox = s0 * n1p * n2;
        s_list[atomicAdd(&s_n, 1)] = nbox <= GT_BUF ? r : -1 - r;
        auto all = [](int k, int n) { return (k & 0xffff) == 0 && (k >> 16) >= n; };
        const int l0 = p0.x & 0xffff, l1 = p0.y & 0xffff, l2 = p0.z & 0xffff, ss = s0 * n1p;
        sp[0] = make_int4(s0, ss, l1 | l2 << 16, 16 * l0);
        // the box cell of a voxel from the bits of its rounded coordinates
        sp[2].w = (int)(0u - (0x4B400000u + (unsigned)l0 + (unsigned)s0 * (0x4B400000u + (unsigned)l1) +
                              (unsigned)ss * (0x4B400000u + (unsigned)l2)));
        sp[3].w = n1p;
        // floor(k / d) = k * (2^20 / d + 1) >> 20 for k < 1024, d < 1024
        sp[4] = make_int4(s0 >> 2, (1 << 20) / (s0 >> 2) + 1, (1 << 20) / n1p + 1,
                          nbox >> 2 | (all(p3.x, n0) && all(p3.y, n1) && all(p3.z, n2) ? 1 << 16 : 0));
    }
    int4* const all4 = reinterpret_cast<int4*>(acc_all);
    for (int k = t; k < GT_SMEM / 4; k += blockDim.x) all4[k] = make_int4(0, 0, 0, 0);
    __syncthreads();
    float* base = rev_grad + G.arena_off;
    // fixed-point scale s = 2^(148 - e) for the biased exponent e of max|g|
    // (max|g| < 2^(e - 126)), clamped to normal floats; a NaN or infinite
    // gradient makes 1 / s a NaN, so it reaches the cells the tile touches
    const int ge = (s_gmax >> 23) & 0xff;
    const int se = min(max(275 - ge, 1), 253);
    const float fx_scale = __int_as_float(se << 23);
    const float fx_inv = ge == 0xff ? __int_as_float(0x7fc00000) : __int_as_float((254 - se) << 23);
    const float gds = gd * fx_scale;
    int parity = 0;  // buffer of the next shared-memory cone
    for (int c = 0; c < s_n; c++) {
        const int r = s_list[c];
        if (touched && t >= GT_TX * GT_TY * GT_TZ - 32) {  // a warp's worth of the block marks the box's line tiles
            const int k = r >= 0 ? r : -1 - r;
            unsigned char* const hit = touched + (size_t)(b * P.nrays + k) * cap;
            const ushort2 ty = s_tile[k][0], tz = s_tile[k][1];
            for (int z = tz.x + ((t & 31) >> 3); z < tz.y; z += 4)
                for (int y = ty.x + (t & 7); y < ty.y; y += 8) hit[y + s_nty[k] * z] = 1;
        }
        if (r >= 0) {
            // buffers alternate over the shared-memory cones: the last flush
            // of this buffer (two such cones back) was cleared by every
            // thread before the barrier of the previous cone
            int* acc = acc_all + parity * GT_BUF;
            parity ^= 1;
            const int4 p0 = s_p[r][0], p2 = s_p[r][2];
            if (gd != 0.f) {
                const float4 a0 = s_A[r][0], a1 = s_A[r][1], a2 = s_A[r][2];
                const f3 q = mk(fmaf(a0.x, dx, fmaf(a0.y, dy, fmaf(a0.z, dz, a0.w))),
                                fmaf(a1.x, dx, fmaf(a1.y, dy, fmaf(a1.z, dz, a1.w))),
                                fmaf(a2.x, dx, fmaf(a2.y, dy, fmaf(a2.z, dz, a2.w))));
                // the forward gather skips a cone where q is outside [0, rev)
                if (!(q.x < 0.f || q.y < 0.f || q.z < 0.f || q.y >= __int_as_float(p2.x) ||
                      q.z >= __int_as_float(p2.y) || q.x >= __int_as_float(p2.z))) {
                    // floor by rounding q - 1/2 at unit spacing, off the
                    // conversion unit; an integer q may take the cell below with
                    // weight 1 on its upper corner (never below the box: its
                    // origin is 0 or under the lowest q by 1e-3)
                    const float b0 = (q.y - 0.5f) + 12582912.f, b1 = (q.z - 0.5f) + 12582912.f,
                                b2 = (q.x - 0.5f) + 12582912.f;
                    const float a0 = q.y - (b0 - 12582912.f), a1 = q.z - (b1 - 12582912.f),
                                a2 = q.x - (b2 - 12582912.f);
                    // all eight corners lie in the box (its set-up above);
                    // those past the array's end are dropped by the flush
                    const float w0[2] = {1.f - a0, a0}, w1[2] = {1.f - a1, a1}, w2[2] = {1.f - a2, a2};
                    int* const cell =
                        acc + (int)((unsigned)__float_as_int(b0) + (unsigned)p0.x * (unsigned)__float_as_int(b1) +
                                    (unsigned)p0.y * (unsigned)__float_as_int(b2) + (unsigned)p2.w);
#pragma unroll
                    for (int d2 = 0; d2 < 2; d2++) {
                        const float t2 = w2[d2] * gds;
#pragma unroll
                        for (int d1 = 0; d1 < 2; d1++) {
                            const float t1 = w1[d1] * t2;
                            // w * g * s rounded to an integer: the sum with
                            // 1.5 * 2^23 has unit spacing, its low bits are
                            // the integer (|w g s| < 2^22)
#pragma unroll
                            for (int d0 = 0; d0 < 2; d0++)
                                atomicAdd(cell + d0 + d1 * p0.x + d2 * p0.y,
                                          __float_as_int(fmaf(w0[d0], t1, 12582912.f)) - 0x4B400000);
                        }
                    }
                }
            }
            __syncthreads();
            const int4 p1 = s_p[r][1], p3 = s_p[r][3], p4 = s_p[r][4];
            float* rb = base + (long long)(((unsigned long long)(unsigned)p1.w << 32) | (unsigned)p1.z) + p0.w;
            const int l1 = p0.z & 0xffff, l2 = p0.z >> 16;
            // one box quad (4 samples) per iteration, quad index = kq + nq0 *
            // (k1 + n1p * k2).  A non-zero quad is one 16-byte vector
            // reduction into the bricked REV gradient (brick rows are 16-byte
            // aligned: arena and cone offsets are multiples of 64 floats),
            // and is cleared for the buffer's next cone.
            int4* acc4 = reinterpret_cast<int4*>(acc);  // s0 is a multiple of 4
            const int nquad = p4.w & 0xffff;
            const bool kept = p4.w >> 16;
            for (int k = t; k < nquad; k += blockDim.x) {
                const int4 v = acc4[k];
                if (v.x != 0 || v.y != 0 || v.z != 0 || v.w != 0) {
                    acc4[k] = make_int4(0, 0, 0, 0);
                    const int q1 = k * p4.y >> 20, kq = k - q1 * p4.x;
                    const int k2 = q1 * p4.z >> 20, k1 = q1 - k2 * p3.w;
                    // rows and slabs past the array's end and quads that
                    // start past it hold the forward's border corners (0), and
                    // cells outside the kept part are not read: cleared, not
                    // sent; a quad that starts inside ends in its last brick,
                    // whose padding nothing reads
                    if (kept || (4 * kq >= (p3.x & 0xffff) && 4 * kq < (p3.x >> 16) && k1 >= (p3.y & 0xffff) &&
                                 k1 < (p3.y >> 16) && k2 >= (p3.z & 0xffff) && k2 < (p3.z >> 16))) {
                        const int y = l1 + k1, z = l2 + k2;
                        red_v4(rb + (64 * kq + (y >> 2) * p1.x + ((y & 3) << 2) + (z >> 2) * p1.y + ((z & 3) << 4)),
                               (float)v.x * fx_inv, (float)v.y * fx_inv, (float)v.z * fx_inv, (float)v.w * fx_inv);
                    }
                }
            }
        } else if (gd != 0.f) {
            // footprint too large for a shared buffer (a REV spacing finer
            // than the voxels): scatter directly
            const EeRayGeom& R = G.ray[-1 - r];
            const f3 q = mk(fmaf(R.A[0], dx, fmaf(R.A[1], dy, fmaf(R.A[2], dz, -R.q0[0]))),
                            fmaf(R.A[3], dx, fmaf(R.A[4], dy, fmaf(R.A[5], dz, -R.q0[1]))),
                            fmaf(R.A[6], dx, fmaf(R.A[7], dy, fmaf(R.A[8], dz, -R.q0[2]))));
            if (!(q.y >= (float)R.rev[0] || q.z >= (float)R.rev[1] || q.x >= (float)R.rev[2] || q.x < 0.f ||
                  q.y < 0.f || q.z < 0.f) &&
                lit_form(R, q.z, q.x) >= 0.5f * EE_LIT_READ)  // a line around the voxel can be lit, so all are kept
                tri_brick_scatter(base + R.offset, rev_store(R), q.y, q.z, q.x, gd);
        }
    }
}

// TERMA adjoint with supersampling (ss > 1): the transpose of k_terma_ss,
// whose voxel TERMA is the mean over ss^3 sub-voxel centres of fluence x
// unit TERMA, each centre with its own beamlet lookup and ray trace
// (cudaSiddon.cu:248-258, 297-306).  The forward keeps neither the beamlets
// nor the unit TERMA of the centres, so each voxel with a non-zero TERMA
// gradient recomputes them (the same centres, lookups and traces) and adds
// gradient x unit / ss^3 to its centres' beamlets; consecutive centres that
// share a beamlet add once.  The fluence enters linearly, as in the ss = 1
// adjoint (a centre whose beamlet has zero fluence still has its slope).
__global__ void __launch_bounds__(256) k_terma_T_ss(EeParams P, const EeBeamSpec* __restrict__ specs,
                                                    const float4* __restrict__ terma_grad, float* __restrict__ fgrad) {
    const int b = blockIdx.z;
    const EeBeamSpec& S = specs[b];
    const long long bvol = ee_brick_vol(S.tn);
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= bvol) return;
    const long long brick = v >> 6;
    const int w = (int)(v & 63), nbx = (S.tn[0] + 3) >> 2, nby = (S.tn[1] + 3) >> 2;
    const long long bxy = brick % ((long long)nbx * nby);
    const int xr = (int)(bxy % nbx) * 4 + (w & 3);
    const int yr = (int)(bxy / nbx) * 4 + ((w >> 2) & 3);
    const int zr = (int)(brick / ((long long)nbx * nby)) * 4 + (w >> 4);
    if (xr >= S.tn[0] || yr >= S.tn[1] || zr >= S.tn[2]) return;
    const float g = quad_value(terma_grad + S.q_off, quads_of(S.tn), xr, yr, zr);
    if (g == 0.f) return;
    const int x = S.t0[0] + xr, y = S.t0[1] + yr, z = S.t0[2] + zr;
    const f3 src = ld3(S.src);
    const int ss = P.ss, nsub = ss * ss * ss;
    const float gs = g / (float)nsub;
    const float sv0 = P.voxel[0] / (float)ss, sv1 = P.voxel[1] / (float)ss, sv2 = P.voxel[2] / (float)ss;
    bool cap = false;
    int cur = -1;
    float acc = 0.f;
    for (int ii = 0; ii < nsub; ii++) {
        const int sx = ii % ss, sy = (ii / ss) % ss, sz = ii / (ss * ss);
        const f3 p = mk(P.start[0] + ((float)x - 0.5f) * P.voxel[0] + ((float)sx + 0.5f) * sv0,
                        P.start[1] + ((float)y - 0.5f) * P.voxel[1] + ((float)sy + 0.5f) * sv1,
                        P.start[2] + ((float)z - 0.5f) * P.voxel[2] + ((float)sz + 0.5f) * sv2);
        int bs = beamlet_of(S, p);
        if (bs == -2) bs = beamlet_point_fp64(S, (double)p.x, (double)p.y, (double)p.z);
        if (bs < 0) continue;
        const float rpl = siddon_rpl(P, p, src, cap);
        const float u = terma_per_fluence(P, rpl, p, src, S.sad);
        if (bs != cur) {
            if (cur >= 0 && acc != 0.f) atomicAdd(fgrad + S.fl_off + cur, acc);
            cur = bs;
            acc = 0.f;
        }
        acc = fmaf(gs, u, acc);
    }
    if (cur >= 0 && acc != 0.f) atomicAdd(fgrad + S.fl_off + cur, acc);
}

// TERMA adjoint: fluence_grad[beamlet(v)] += G_v * terma_grad[v].  A block
// takes TT_VPT * 256 consecutive bricked voxels (a run of bricks along x) and
// sums them per beamlet in a shared histogram of the beam's fluence map, then
// adds the non-zero bins to the fluence gradient: one global atomic per
// beamlet the run touches.  Maps above TT_HIST beamlets aggregate per warp
// (lanes of equal beamlet index summed before one atomic) instead.
constexpr int TT_HIST = 4096, TT_VPT = 4;

__global__ void __launch_bounds__(256) k_terma_T(EeParams P, const EeBeamSpec* __restrict__ specs,
                                                 const float* __restrict__ unit, const int* __restrict__ bl_idx,
                                                 const float4* __restrict__ terma_grad, float* __restrict__ fluence_grad) {
    __shared__ float hist[TT_HIST];
    const int b = blockIdx.z;
    const EeBeamSpec& S = specs[b];
    const long long tvol = ee_brick_vol(S.tn);  // padding: bl_idx -1
    const long long v0 = (long long)blockIdx.x * (256 * TT_VPT);
    if (v0 >= tvol) return;
    const int t = threadIdx.x, nfl = S.fmap[0] * S.fmap[1];
    float* fg = fluence_grad + S.fl_off;
    const Brick Q = quads_of(S.tn);
    const int nbx = (S.tn[0] + 3) >> 2, nby = (S.tn[1] + 3) >> 2;
    const float4* const tq = terma_grad + S.q_off;
    auto grad = [&](long long v) {  // of bricked box element v, inside the box
        const unsigned brick = (unsigned)(v >> 6), row = brick / nbx;
        const int w = (int)(v & 63);
        return quad_value(tq, Q, (int)(brick - row * nbx) * 4 + (w & 3), (int)(row % nby) * 4 + ((w >> 2) & 3),
                          (int)(row / nby) * 4 + (w >> 4));
    };
    if (nfl > TT_HIST) {
        for (int j = 0; j < TT_VPT; j++) {
            const long long v = v0 + j * 256 + t;
            int bl = -1;
            float val = 0.f;
            if (v < tvol) {
                const long long o = S.t_off + v;
                bl = bl_idx[o];
                if (bl >= 0) val = unit[o] * grad(v);
            }
            const unsigned peers = __match_any_sync(FULL, bl);
            const int leader = __ffs(peers) - 1;
            float sum = 0.f;
            for (unsigned m = peers; m; m &= m - 1) sum += __shfl_sync(peers, val, __ffs(m) - 1);
            if ((t & 31) == leader && bl >= 0 && sum != 0.f) atomicAdd(fg + bl, sum);
        }
        return;
    }
    for (int k = t; k < nfl; k += 256) hist[k] = 0.f;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < TT_VPT; j++) {
        const long long v = v0 + j * 256 + t;
        if (v < tvol) {
            const long long o = S.t_off + v;
            const int bl = bl_idx[o];
            if (bl >= 0) {
                const float val = unit[o] * grad(v);
                if (val != 0.f) atomicAdd(hist + bl, val);
            }
        }
    }
    __syncthreads();
    for (int k = t; k < nfl; k += 256) {
        const float h = hist[k];
        if (h != 0.f) atomicAdd(fg + k, h);
    }
}

}  // namespace

// ----------------------------------------------------------- launchers ---
static inline unsigned grid1(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

cudaError_t ee_launch_geom_init(const EeBeamSpec* specs, EeBeamGeom* g, int nbeams, cudaStream_t s) {
    k_geom_init<<<grid1(nbeams, 128), 128, 0, s>>>(specs, g, nbeams);
    return cudaGetLastError();
}

cudaError_t ee_copy_status(const EeBeamGeom* geoms, int* status_host, int nbeams, cudaStream_t s) {
    return cudaMemcpy2DAsync(status_host, sizeof(int), (const char*)geoms + offsetof(EeBeamGeomHead, status),
                             sizeof(EeBeamGeom), sizeof(int), nbeams, cudaMemcpyDeviceToHost, s);
}

cudaError_t ee_launch_terma(const EeParams& P, const EeBeamSpec* specs, EeBeamGeom* geoms, const float* fluence,
                            float* terma, float* unit, int* beamlet_idx, int nbeams, long long max_tvol,
                            cudaStream_t s) {
    if (P.ss > 1)
        k_terma_ss<<<dim3(grid1(max_tvol, 64), 1, nbeams), 256, 0, s>>>(P, specs, geoms, fluence, terma, unit,
                                                                        beamlet_idx);
    else {
        // Voxels per block: larger blocks waste fewer lanes, smaller ones spread
        // the rays of a small call over the chip.  128, 256, 512: one 24 x 24 beam
        // 0.114, 0.133, 0.186 ms (4.2 M voxels), three 0.285, 0.293, 0.326, six
        // 0.406, 0.389, 0.393, twelve 1.06, 0.93, 0.91, 96 8.0, 6.8, 6.3 (1024: 6.1).
        const long long all = max_tvol * nbeams;
        auto run = [&](auto kernel, int items) {
            kernel<<<dim3(grid1(max_tvol, items), 1, nbeams), TERMA_BLOCK, 0, s>>>(P, specs, geoms, fluence, terma, unit,
                                                                                beamlet_idx);
        };
        if (all < 18000000) run(k_terma<128>, 128);
        else if (all < 40000000) run(k_terma<256>, 256);
        else run(k_terma<512>, 512);
    }
    return cudaGetLastError();
}

cudaError_t ee_launch_geometry(const EeParams& P, const EeBeamSpec* specs, EeBeamGeom* geoms, int nbeams,
                               cudaStream_t s) {
    k_geometry<<<nbeams, 64, 0, s>>>(P, specs, geoms);
    return cudaGetLastError();
}

// The split of an SM's L1 between shared memory and cache that the kernels ask
// for, on the current device.  An SM takes blocks of another kernel only at
// the split that it has, so the TERMA and the cones, which would ask for 0 to
// 16 KB, ask for the 100 KB that k_gather needs anyway: with three engines on
// their own streams a 24 x 24 beam takes 0.697 against 0.727 ms a pass, 96
// beams of 8^2..40^2 beamlets 26.9 against 27.3 ms; one engine alone loses 1 %
// on the large batches (128 KB and more: 4 % and up; 64 KB: the three engines
// gain nothing on the batches).
void ee_kernel_setup() {
    const void* const fn[] = {(const void*)k_terma<128>,  (const void*)k_terma<256>,  (const void*)k_terma<512>,
                              (const void*)k_cone_tiles, (const void*)k_cone_lane, (const void*)k_cone_T_lane};
    for (const void* f : fn)
        if (cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, 40) != cudaSuccess)
            (void)cudaGetLastError();  // a preference: the launches do not depend on it
}

static size_t cone_smem(int maxL) { return sizeof(float) * ((size_t)CONE_WARPS * 3 * maxL + 2 * EE_MAX_RADII + EE_MAX_RADII); }

// Raise a kernel's dynamic shared-memory limit on the current device.  The
// attribute belongs to the (device, kernel) pair, so the cache of what was
// set is keyed by both; the lock covers concurrent server threads.  The
// first eager launch on a device sets it, before any graph capture.
static cudaError_t smem_attr(const void* fn, size_t smem) {
    if (smem <= 48 * 1024) return cudaSuccess;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    struct Done {
        int dev;
        const void* fn;
        size_t sz;
    };
    static std::mutex mu;
    static Done done[64];
    static int ndone = 0;
    std::lock_guard<std::mutex> lock(mu);
    for (int k = 0; k < ndone; k++)
        if (done[k].dev == dev && done[k].fn == fn && done[k].sz >= smem) return cudaSuccess;
    size_t got = std::max(smem, (size_t)200 * 1024);  // once, to the largest size any line needs
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)got);
    if (e != cudaSuccess) {
        got = smem;
        e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)got);
    }
    if (e != cudaSuccess) return e;
    for (int k = 0; k < ndone; k++)
        if (done[k].dev == dev && done[k].fn == fn) { done[k].sz = got; return cudaSuccess; }
    if (ndone < 64) done[ndone++] = Done{dev, fn, got};
    return cudaSuccess;
}

cudaError_t ee_launch_cone(const EeParams& P, const EeBeamSpec* specs, const EeBeamGeom* geoms, const float* terma,
                           float* rev, const EeConeWork& work, int nbeams, int max_lines, int max_line,
                           cudaStream_t s) {
    if (P.mode == 1 && work.scratch) {  // exp kernel: one lane per line
        const int cap = ee_cone_tiles_cap(max_lines);
        k_cone_tiles<<<dim3(P.nrays, nbeams), 256, 0, s>>>(P, geoms, EE_LIT_READ, nullptr, work.counts, work.tiles, cap);
        k_cone_lane<<<work.warps / EE_CONE_BLOCK_WARPS, EE_CONE_BLOCK_WARPS * 32, 0, s>>>(P, specs, geoms, terma, rev,
                                                                                        work, nbeams, cap);
        return cudaGetLastError();
    }
    if (P.mode == EE_KERNEL_TABLE && P.nradii == TAB_NR) {  // exact O(n nr) table scan
        const size_t smem = sizeof(float) * ((size_t)TAB_WARPS * tab_fwd_stride(max_line) + TAB_SMEM);
        cudaError_t e = smem_attr((const void*)k_cone_tab, smem);
        if (e != cudaSuccess) return e;
        dim3 grid(grid1(max_lines, 2 * TAB_WARPS), P.nrays, nbeams);
        k_cone_tab<<<grid, TAB_WARPS * 32, smem, s>>>(P, specs, geoms, terma, rev, max_line);
        return cudaGetLastError();
    }
    size_t smem = cone_smem(max_line);
    cudaError_t e = smem_attr((const void*)k_cone, smem);
    if (e != cudaSuccess) return e;
    dim3 grid(grid1(max_lines, CONE_WARPS), P.nrays, nbeams);
    k_cone<<<grid, CONE_WARPS * 32, smem, s>>>(P, specs, geoms, terma, rev, max_line);
    return cudaGetLastError();
}

cudaError_t ee_launch_rev_zero(const EeParams& P, const EeBeamGeom* geoms, float* rev_grad, const EeConeWork& work,
                               int nbeams, int max_lines, cudaStream_t s) {
    k_rev_zero<128><<<dim3(grid1(max_lines, 128), P.nrays, nbeams), 128, 0, s>>>(P, geoms, rev_grad, work.touched,
                                                                                 ee_cone_tiles_cap(max_lines));
    return cudaGetLastError();
}

cudaError_t ee_launch_gather(const EeParams& P, const EeBeamSpec* specs, const EeBeamGeom* geoms, const float* rev,
                             float* dose, int nbeams, int dose_mode, int max_rows, cudaStream_t s) {
    const long long nfull = (long long)P.size[0] * P.size[1] * P.size[2];
    // A warp's patches are a chain of loads, and five blocks are resident per SM.
    // Up to 12 rounds of resident blocks, two blocks share the patches of a
    // group, or the last round is long (one 24 x 24 beam, 1000 blocks: 0.199 ->
    // 0.143 ms; six beams, 6000: 0.565 -> 0.477); above, the set-up that each
    // repeats costs more than that (12 beams, 12000: 1.03 -> 1.07; 96: 8.8 ->
    // 9.3).  Below three blocks per SM four blocks take two patches at a time
    // (a 64^3 slab, 96 blocks: 0.086 -> 0.038 ms, 0.058 with two blocks of four
    // patches; 384: 0.119 -> 0.102; 1000: 0.150 against 0.143).
    const int blocks = grid1(max_rows, ROW_WARPS);
    const long long all = (long long)blocks * nbeams;
    if (all < 456)
        k_gather<2><<<dim3(blocks, 4, nbeams), ROW_WARPS * 32, 0, s>>>(P, specs, geoms, rev, dose, dose_mode, nfull);
    else
        k_gather<4><<<dim3(blocks, all < 9120 ? 2 : 1, nbeams), ROW_WARPS * 32, 0, s>>>(P, specs, geoms, rev, dose,
                                                                                       dose_mode, nfull);
    return cudaGetLastError();
}

cudaError_t ee_launch_gather_T(const EeParams& P, const EeBeamSpec* specs, const EeBeamGeom* geoms,
                               const float* dose_grad, float* rev_grad, const EeConeWork& work, int nbeams,
                               int max_lines, int max_tiles, cudaStream_t s) {
    const size_t smem = sizeof(float) * GT_SMEM;
    cudaError_t e = smem_attr((const void*)k_gather_T, smem);
    if (e != cudaSuccess) return e;
    dim3 grid(max(1, max_tiles), 1, nbeams);
    k_gather_T<<<grid, GT_TX * GT_TY * GT_TZ, smem, s>>>(P, specs, geoms, dose_grad, rev_grad, work.touched,
                                                        ee_cone_tiles_cap(max_lines));
    return cudaGetLastError();
}

cudaError_t ee_launch_cone_T(const EeParams& P, const EeBeamSpec* specs, const EeBeamGeom* geoms, const float* rev_grad,
                             const EeConeWork& work, float4* terma_grad, int nbeams, int max_lines, int max_line,
                             cudaStream_t s) {
    if (P.mode == EE_KERNEL_EXP) {
        if (!work.scratch) return cudaErrorInvalidValue;  // no warp-per-line form of the exp adjoint
        const int cap = ee_cone_tiles_cap(max_lines);
        k_cone_tiles<<<dim3(P.nrays, nbeams), 256, 0, s>>>(P, geoms, 0.f, work.touched, work.counts, work.tiles, cap);
        k_cone_T_lane<<<work.warps / EE_CONE_BLOCK_WARPS, EE_CONE_BLOCK_WARPS * 32, 0, s>>>(
            P, specs, geoms, rev_grad, work, nbeams, cap, terma_grad);
        return cudaGetLastError();
    }
    if (P.mode == EE_KERNEL_TABLE && P.nradii == TAB_NR) {
        const size_t smem = sizeof(float) * ((size_t)TAB_WARPS * tab_adj_stride(max_line) + TAB_SMEM);
        cudaError_t e = smem_attr((const void*)k_cone_T_tab, smem);
        if (e != cudaSuccess) return e;
        dim3 grid(grid1(max_lines, 2 * TAB_WARPS), P.nrays, nbeams);
        k_cone_T_tab<<<grid, TAB_WARPS * 32, smem, s>>>(P, specs, geoms, rev_grad, terma_grad, max_line);
        return cudaGetLastError();
    }
    size_t smem = cone_smem(max_line);
    cudaError_t e = smem_attr((const void*)k_cone_T, smem);
    if (e != cudaSuccess) return e;
    dim3 grid(grid1(max_lines, CONE_WARPS), P.nrays, nbeams);
    k_cone_T<<<grid, CONE_WARPS * 32, smem, s>>>(P, specs, geoms, rev_grad, terma_grad, max_line);
    return cudaGetLastError();
}

cudaError_t ee_launch_terma_T(const EeParams& P, const EeBeamSpec* specs, const EeBeamGeom* geoms,
                              const float* unit_terma, const int* beamlet_idx, const float4* terma_grad,
                              float* fluence_grad, int nbeams, long long max_tvol, cudaStream_t s) {
    (void)geoms;
    if (P.ss > 1) {  // supersampled TERMA: recompute the sub-voxel beamlets
        k_terma_T_ss<<<dim3(grid1(max_tvol, 256), 1, nbeams), 256, 0, s>>>(P, specs, terma_grad, fluence_grad);
        return cudaGetLastError();
    }
    dim3 grid(grid1(max_tvol, 256 * TT_VPT), 1, nbeams);
    k_terma_T<<<grid, 256, 0, s>>>(P, specs, unit_terma, beamlet_idx, terma_grad, fluence_grad);
    return cudaGetLastError();
}

// ------------------------------------------------- EndtoEnd loss terms ----
// Dose terms of the EndtoEnd loss (README.md:20):
//   L_d = sum_i w0_i (d_i - t0_i)^2 + sum_i w_i max(d_i - t_i, 0)^2
// and its gradient dL/dd.  acc[0] += PTV term, acc[1] += OAR term.
__global__ void __launch_bounds__(256) k_loss_grad(const float* __restrict__ dose, const float* __restrict__ ptv_w,
                                                   const float* __restrict__ ptv_t, const float* __restrict__ oar_w,
                                                   const float* __restrict__ oar_t, float* __restrict__ grad,
                                                   double* __restrict__ acc, long long n) {
    double lp = 0.0, lo = 0.0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float d = dose[i];
        float g = 0.f;
        if (ptv_w) {
            float w = ptv_w[i], e = d - ptv_t[i];
            lp += (double)w * e * e;
            g += 2.f * w * e;
        }
        if (oar_w) {
            float w = oar_w[i], e = fmaxf(d - oar_t[i], 0.f);
            lo += (double)w * e * e;
            g += 2.f * w * e;
        }
        grad[i] = g;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lp += __shfl_xor_sync(FULL, lp, o);
        lo += __shfl_xor_sync(FULL, lo, o);
    }
    __shared__ double sp[8], so[8];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { sp[w] = lp; so[w] = lo; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0, b = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) { a += sp[k]; b += so[k]; }
        atomicAdd(acc, a);
        atomicAdd(acc + 1, b);
    }
}

// Fluence-map convolution with a normalised 2-D Gaussian (the EndtoEnd
// fluence-spread step, README.md:15-18), zero padding.  The kernel is
// symmetric, so the same launch is its own transpose.  One thread per output
// pixel of beam blockIdx.z.
__global__ void __launch_bounds__(256) k_spread(const EeBeamSpec* __restrict__ specs, const float* __restrict__ in,
                                                float* __restrict__ out, const float* __restrict__ w1d, int R) {
    const EeBeamSpec& S = specs[blockIdx.z];
    const int fx = S.fmap[0], fy = S.fmap[1];
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= fx * fy) return;
    int x = p % fx, y = p / fx;
    const float* src = in + S.fl_off;
    float acc = 0.f;
    for (int dy = -R; dy <= R; dy++) {
        int yy = y + dy;
        if (yy < 0 || yy >= fy) continue;
        float wy = w1d[dy + R];
        for (int dx = -R; dx <= R; dx++) {
            int xx = x + dx;
            if (xx < 0 || xx >= fx) continue;
            acc += wy * w1d[dx + R] * src[xx + fx * yy];
        }
    }
    out[S.fl_off + p] = acc;
}

// eta * ||D x||_1 with D the forward differences along both fluence-map axes
// (BOO/BOO_QL/CreateDxDyFMO.m:1-36); adds eta * D^T sign(D x)
// into grad and the term into acc[2].
__global__ void __launch_bounds__(256) k_smooth(const EeBeamSpec* __restrict__ specs, const float* __restrict__ x,
                                                float* __restrict__ grad, float eta, double* __restrict__ acc) {
    const EeBeamSpec& S = specs[blockIdx.z];
    const int fx = S.fmap[0], fy = S.fmap[1];
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    double l = 0.0;
    if (p < fx * fy) {
        int i = p % fx, j = p / fx;
        const float* m = x + S.fl_off;
        float v = m[p], g = 0.f;
        if (i + 1 < fx) { float d = m[p + 1] - v; l += fabsf(d); g -= (d > 0.f) - (d < 0.f); }
        if (i > 0) { float d = v - m[p - 1]; g += (d > 0.f) - (d < 0.f); }
        if (j + 1 < fy) { float d = m[p + fx] - v; l += fabsf(d); g -= (d > 0.f) - (d < 0.f); }
        if (j > 0) { float d = v - m[p - fx]; g += (d > 0.f) - (d < 0.f); }
        grad[S.fl_off + p] += eta * g;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(FULL, l, o);
    if ((threadIdx.x & 31) == 0 && l != 0.0) atomicAdd(acc + 2, (double)eta * l);
}

cudaError_t ee_launch_loss_grad(const float* dose, const float* ptv_w, const float* ptv_t, const float* oar_w,
                                const float* oar_t, float* grad, double* acc, long long n, cudaStream_t s) {
    k_loss_grad<<<std::min<long long>(grid1(n, 256), 152 * 8), 256, 0, s>>>(dose, ptv_w, ptv_t, oar_w, oar_t, grad, acc, n);
    return cudaGetLastError();
}

cudaError_t ee_launch_spread(const EeBeamSpec* specs, const float* in, float* out, const float* w1d, int R, int nbeams,
                             int max_pix, cudaStream_t s) {
    dim3 grid(grid1(max_pix, 256), 1, nbeams);
    k_spread<<<grid, 256, 0, s>>>(specs, in, out, w1d, R);
    return cudaGetLastError();
}

cudaError_t ee_launch_smooth(const EeBeamSpec* specs, const float* x, float* grad, float eta, double* acc, int nbeams,
                             int max_pix, cudaStream_t s) {
    dim3 grid(grid1(max_pix, 256), 1, nbeams);
    k_smooth<<<grid, 256, 0, s>>>(specs, x, grad, eta, acc);
    return cudaGetLastError();
}
