// Internal structures shared by the CCCS host code (ee_api.cpp) and the
// sm_103a kernels (ee_kernels.cu).  POD only, identical on host and device.
#pragma once
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/ee_cccs.h"

#define EE_MAX_RAYS 64
#define EE_MAX_E 32
#define EE_MAX_RADII 32
#define EE_MAX_THETA 48
#define EE_MAX_LINE 1024  // longest convolution line (reference limit, host.cu:567)

// Per-context constants, passed by value to every kernel.
struct EeParams {
    int size[3];
    float voxel[3];
    float start[3];
    int bb0[3];
    int bbs[3];
    const float* density;  // full grid
    cudaTextureObject_t dens_tex;  // same volume as a 3-D texture: linear filter, border 0,
                                   // unnormalised coordinates (the reference's texDens,
                                   // nvbbRayConvolve_host.cu:229-242)
    int nE;
    float sp_fluence[EE_MAX_E];
    float sp_energy[EE_MAX_E];
    float sp_mu[EE_MAX_E];
    int ntheta, nphi, nradii, nrays;
    float radii[EE_MAX_RADII];
    float lat, lng, penumbra;
    int max_rev[3];
    int mode;                   // ee_kernel_mode
    int ss;                     // TERMA supersampling per axis (1: off)
    const float* cumkern;       // [ntheta][nradii]
    const float* expp;          // [ntheta][4]
    const struct EeRayConst* rays;  // [nrays]
};

// Per-cone constants (angles and rotations), built on the host.
struct EeRayConst {
    float th, ph;
    int row_fwd, row_rev;  // kernel rows for the two walk directions
    float MK[9];           // BEV -> REV   (rotateKernelAtOriginRHS), row-major
    float MKi[9];          // REV -> BEV   (inverseRotateKernelAtOriginRHS)
};

// TERMA boxes, and their unit-TERMA, beamlet-index and gradient companions,
// are stored in 4x4x4 bricks so that the eight corners of a trilinear cell,
// and the cells of neighbouring REV lines, share cache lines whatever the
// cone's direction.  Box element (x, y, z) sits at bx(x) + by(y) + bz(z):
//   bx(x) = (x>>2)*64 + (x&3),  by(y) = (y>>2)*64*nbx + (y&3)*4,
//   bz(z) = (z>>2)*64*nbx*nby + (z&3)*16,   nb* = ceil(n*/4);
// bricks, and so the rows of 4 x-neighbours, start on 256-byte boundaries.
inline __host__ __device__ long long ee_brick_vol(const int tn[3]) {
    return 64ll * ((tn[0] + 3) >> 2) * ((tn[1] + 3) >> 2) * ((tn[2] + 3) >> 2);
}

// The adjoint scatters each sample's TERMA gradient into quads: the four corners
// of a cell in (x, y) at one z as one float4, for the cells from one before the
// box to its last voxel in x and y, bricked over (n0 + 1, n1 + 1, n2).  A voxel's
// gradient is the sum of one value of each of its four cells.
inline __host__ __device__ long long ee_quad_vol(const int tn[3]) {
    return 64ll * ((tn[0] + 4) >> 2) * ((tn[1] + 4) >> 2) * ((tn[2] + 3) >> 2);
}

// The forward gather's warp patch: EE_GATHER_PX x EE_GATHER_PY x EE_GATHER_PZ
// patient voxels (32 lanes); a warp owns a group of PY x PZ patient rows.
constexpr int EE_GATHER_PX = 8, EE_GATHER_PY = 2, EE_GATHER_PZ = 2;
inline __host__ __device__ long long ee_gather_groups(long long ny, long long nz) {
    return ((ny + EE_GATHER_PY - 1) / EE_GATHER_PY) * ((nz + EE_GATHER_PZ - 1) / EE_GATHER_PZ);
}

// Per-beam constants built on the host.
struct EeBeamSpec {
    float src[3];
    float dir[3];          // unit
    float iso[3];
    float az, zen, coll, sad;
    float isodist;         // |iso - src|
    float MB[9];           // RCS -> BEV (rotateBeamAtOriginRHS)
    float MBi[9];          // BEV -> RCS
    int fmap[2];
    float beamlet[2];
    long long fl_off;      // offset of this beam's fluence map
    // TERMA box: axis-aligned patient-index box holding the field frustum
    // (clipped to the calc bbox); TERMA is identically zero outside it.
    int t0[3];             // origin (full-grid voxel index)
    int tn[3];             // size
    long long t_off;       // element offset in the TERMA arena (a multiple of 64: bricks, below)
    long long q_off;       // first quad of the beam's TERMA gradient (ee_quad_vol)
    // FP64 copies for re-deciding the beamlet of voxels whose FP32 fluence-map
    // coordinate lands within 1e-4 of a beamlet boundary
    double srcd[3];
    double dird[3];
    double MBd[9];
    double isodistd;
    // axial distances from the source between which the calc bbox lies (its
    // corners): every voxel with TERMA is between them
    float dnear, dfar;
    // REV arena slot planned from geometric upper bounds (ee_plan);
    // plan_cap == 0: the arena is sized after the geometry read-back
    long long plan_off;
    long long plan_cap;
    int plan_lines;  // line slots per cone that the planned tile lists hold
    int plan_line;   // samples per line that the planned cone scratch holds
    // element offset of this beam's dose (and dose-gradient) volume: grouped
    // outputs of the request server; 0 otherwise
    long long out_off;
};

// Whether a beam's sizes, as the device finds them, fit what was planned for it.
// The lists and the scratch are indexed by the device's own sizes, so a bound
// that failed would be written past; such a beam gets a status instead.
inline __host__ __device__ bool ee_plan_holds(const EeBeamSpec& S, long long store, int max_lines, int max_line) {
    return S.plan_cap == 0 || (store <= S.plan_cap && max_lines <= S.plan_lines && max_line <= S.plan_line);
}

// Per-cone geometry of one beam, computed on the device.
struct EeRayGeom {
    int rev[3];            // (along-line, lateral-1, lateral-2) sizes
    // the part of the REV array that is kept: samples so[0] .. so[0]+sn[0]-1
    // of lines so[1].. x so[2]..; so is whole bricks
    int so[3], sn[3];
    int nlines;            // sn[1]*sn[2]
    long long offset;      // where sample (0, 0, 0) would sit in the beam's REV arena
    float q0[3];           // rev_min / spacing (reference vector order)
    float G0[3], Gx[3], Gy[3], Gz[3];  // REV (tX,tY,tZ) -> patient voxel index
    float B0[3], Bx[3], By[3], Bz[3];  // REV (tX,tY,tZ) -> BEV crop-box index
    float M[9];            // BEV -> REV (copy of MK for the gather)
    float A[9];            // patient index step -> REV step (MK MB), row-major
    float iB[3], iG[3];    // 1 / Bx, 1 / Gx (0 where below 1e-6): line-box intersections without divisions
    // the field frustum's four sides as affine forms of a REV point,
    // [0] i + [1] + [2] tY + [3] tZ >= 0 where its TERMA corners may lie in
    // the field, and the distance in front of the source (k_geometry)
    float side[4][4];
    float front[4];
    // half-planes [0] tY + [1] tZ + [2] >= 0 that hold every line with a field
    // span ("lit"; k_geometry), [0], [1] a unit normal (or 0, 0, 1: no bound)
    float lit[4][3];
};

// Lit half-planes of one cone (EeRayGeom::lit).  In the box the field is a
// frustum; c[e] is its axis at the near (0) and far (1) plane in BEV index
// coordinates, h[e] its half widths there along BEV x and z, q0 the REV
// origin.  Its eight corners projected along the cone bound every lit line:
// k = 0, 1 cut the projection off at its ends, k = 2, 3 follow its silhouette
// from the near to the far plane, or the axis, where that turns away from it
// (axis: bits 0, 1 take the axis for k = 2, 3 in any case).
template <class T>
inline __host__ __device__ void ee_lit_planes(const float* MK, const T c[2][3], const T h[2][2], const T q0[3],
                                              T lit[4][3], int axis = 0) {
    T v[8][2], mid[2][2];  // (tY, tZ)
    for (int e = 0; e < 2; e++)
        for (int a = 0; a < 2; a++) {
            const float* M = MK + (a ? 0 : 6);  // REV vector (tZ, tX, tY)
            const T m = M[0] * c[e][0] + M[1] * c[e][1] + M[2] * c[e][2] - q0[a ? 0 : 2];
            mid[e][a] = m;
            for (int i = 0; i < 4; i++)
                v[4 * e + i][a] = m + (i & 1 ? h[e][0] : -h[e][0]) * M[0] + (i & 2 ? h[e][1] : -h[e][1]) * M[2];
        }
    T ey = mid[1][0] - mid[0][0], ez = mid[1][1] - mid[0][1];
    const T l = sqrt(ey * ey + ez * ez);
    if (l > T(1e-2)) { ey /= l; ez /= l; }
    else { ey = 1; ez = 0; }
    for (int k = 0; k < 4; k++) {
        const T sg = k & 1 ? 1 : -1;
        T ny = sg * ey, nz = sg * ez;
        if (k >= 2) {
            ny = -sg * ez;
            nz = sg * ey;
            T best[2] = {-1e30f, -1e30f}, by[2] = {0, 0}, bz[2] = {0, 0};  // near and far corner farthest along n
            for (int i = 0; i < 8; i++) {
                const T t = ny * v[i][0] + nz * v[i][1];
                if (t > best[i >> 2]) { best[i >> 2] = t; by[i >> 2] = v[i][0]; bz[i >> 2] = v[i][1]; }
            }
            const T dy = by[1] - by[0], dz = bz[1] - bz[0], dl = sqrt(dy * dy + dz * dz);
            const T along = -dz * ny + dy * nz;  // (dz, dy) turned onto n
            if (!(axis >> (k - 2) & 1) && dl > T(1e-2) && fabs(along) > T(0.5) * dl) {
                const T t = (along > 0 ? 1 : -1) / dl;
                ny = -t * dz;
                nz = t * dy;
            }
        }
        T sup = -1e30f;
        for (int i = 0; i < 8; i++) {
            const T t = ny * v[i][0] + nz * v[i][1];
            sup = t > sup ? t : sup;
        }
        lit[k][0] = -ny;
        lit[k][1] = -nz;
        lit[k][2] = sup + T(0.05);
    }
}

// The lateral rectangle [lo, hi] around the points whose lit forms are all >=
// -slack (the corners of an end's and a side's lines, which meet at 30 degrees
// or more).
template <class T>
inline __host__ __device__ void ee_lit_rect(const T lit[4][3], T slack, T lo[2], T hi[2]) {
    lo[0] = lo[1] = 1e30f;
    hi[0] = hi[1] = -1e30f;
    for (int i = 0; i < 2; i++)
        for (int j = 2; j < 4; j++) {
            const T det = lit[i][0] * lit[j][1] - lit[j][0] * lit[i][1], ci = lit[i][2] + slack, cj = lit[j][2] + slack;
            const T p[2] = {(lit[i][1] * cj - lit[j][1] * ci) / det, (lit[j][0] * ci - lit[i][0] * cj) / det};
            for (int a = 0; a < 2; a++) {
                lo[a] = p[a] < lo[a] ? p[a] : lo[a];
                hi[a] = p[a] > hi[a] ? p[a] : hi[a];
            }
        }
}

// A lit line's forms are >= 0.  The gathers visit a voxel and cone only where
// one of the four lines around the voxel can be lit; such a line is within one
// cell per axis of the voxel, the lines that k_gather then reads within one
// more, so a line whose least form is below this is never read.
constexpr float EE_LIT_READ = -2.95f;  // -2 sqrt(2), and rounding

// Per-beam geometry computed on the device: the crop box and the sizes that
// the host reads back,
struct EeBeamGeomHead {
    int key_min[3];        // ordered-int keys for atomic min/max
    int key_max[3];
    unsigned int nnz;
    int status;
    float bmin[3];
    int bev[3];
    float lim_off[3];      // (lim_min - start)/voxel
    float lim_min[3];
    long long v_beam;
    long long rev_total;   // the cones' REV arrays (bricked)
    long long store_total; // their kept parts: the beam's arena
    int max_line;
    int max_lines;
    // patient rows (y,z) whose voxels can see this beam's REV dose: the AABB
    // of the crop box dilated by 2 voxels, clipped to the calc bbox
    int gy0, gz0, gny, gnz;
    int rows;              // row groups of the forward gather (ee_gather_groups)
    int gx0, gnx;          // x range of the same AABB
    int tiles;             // 8x8x4 patient tiles covering the AABB (adjoint gather)
    long long arena_off;   // element offset of this beam's REV arena
    long long arena_cap;   // elements available to this beam
};
// and the cones' REV frames, which stay on the device.
struct EeBeamGeom : EeBeamGeomHead {
    EeRayGeom ray[EE_MAX_RAYS];
};

// Launch wrappers implemented in ee_kernels.cu.  All enqueue on `s`.
cudaError_t ee_launch_geom_init(const EeBeamSpec* specs, EeBeamGeom* g, int nbeams, cudaStream_t s);
// unit/beamlet_idx (both optional) receive TERMA per unit fluence of every
// in-field voxel and its beamlet index (adjoint).
cudaError_t ee_launch_terma(const EeParams& P, const EeBeamSpec* specs, EeBeamGeom* geoms, const float* fluence,
                            float* terma, float* unit, int* beamlet_idx, int nbeams, long long max_tvol,
                            cudaStream_t s);
cudaError_t ee_launch_geometry(const EeParams& P, const EeBeamSpec* specs, EeBeamGeom* geoms, int nbeams,
                               cudaStream_t s);
// Work space of the exp mode's lane cones: each resident warp keeps one tile's
// samples between its two passes (scratch[warp][quad][2][lane]), and takes
// tiles from lists, one per beam and cone, of those that the gathers can see.
struct EeConeWork {
    float4* scratch = nullptr;
    int warps = 0;         // resident warps, a multiple of EE_CONE_BLOCK_WARPS
    int quads = 0;         // quads of samples per warp
    int* counts = nullptr; // [0] tiles taken; [1 + segment] tiles listed, segment = beam * nrays + cone in list order
    int* tiles = nullptr;  // [segment][tiles_cap] tiles of 8 x 4 lines
    unsigned char* touched = nullptr;  // [beam * nrays + cone][tiles_cap] tiles that the adjoint gather adds to
};
constexpr int EE_CONE_BLOCK_WARPS = 2, EE_CONE_SM_WARPS = 24, EE_CONE_MAX_WARPS = 152 * EE_CONE_SM_WARPS;
inline int ee_cone_quads(int max_line) { return (max_line + 3) / 4 + 2; }
// Resident warps whose scratch stays within a quarter of `limit` bytes.  A beam
// whose arena alone exceeds the other three quarters is taken all the same;
// `arena`: bytes of the largest chunk's, and then the scratch may be as large.
// With the quarter in that case too, a limit of 1 MB left one warp per SM: a 24 x
// 24 beam on 200 x 200 x 160, dose and adjoint, 1.91 ms, so 0.62 (0.61 with a
// limit of 512 MB).
inline int ee_cone_warps(int max_line, long long limit, long long arena) {
    const long long per = 1024ll * ee_cone_quads(max_line), n = (arena > limit / 4 * 3 ? arena : limit / 4) / per;
    return (int)(n < 152 ? 152 : (n > EE_CONE_MAX_WARPS ? EE_CONE_MAX_WARPS : n)) & ~(EE_CONE_BLOCK_WARPS - 1);
}
inline int ee_cone_tiles_cap(int max_lines) { return max_lines / 32 + 1; }
// Bytes of a chunk that its scratch limit counts, apart from the warps' scratch:
// REV arena, TERMA gradient, and the lists of the lane cones with a count, the
// tiles and their marks.
inline long long ee_chunk_bytes(long long rev, long long quads, long long lists, int max_lines) {
    return 4 * rev + 16 * quads + lists * (4 + 5ll * ee_cone_tiles_cap(max_lines));
}
// kernel preferences of the current device; before the first launch on it
void ee_kernel_setup();
// the cones write every sample that k_gather reads; without work space (exp
// mode) the warp-per-line kernel runs
cudaError_t ee_launch_cone(const EeParams& P, const EeBeamSpec* specs, const EeBeamGeom* geoms, const float* terma,
                           float* rev, const EeConeWork& work, int nbeams, int max_lines, int max_line,
                           cudaStream_t s);
// dose_mode 0/1 accumulate atomically into dose (the caller zeroes it for
// mode 0); mode 2 writes dose[b] rows (the caller zeroes the volumes).
cudaError_t ee_launch_gather(const EeParams& P, const EeBeamSpec* specs, const EeBeamGeom* geoms, const float* rev,
                             float* dose, int nbeams, int dose_mode, int max_rows, cudaStream_t s);
// adjoint
cudaError_t ee_launch_gather_T(const EeParams& P, const EeBeamSpec* specs, const EeBeamGeom* geoms,
                               const float* dose_grad, float* rev_grad, const EeConeWork& work, int nbeams,
                               int max_lines, int max_tiles, cudaStream_t s);
// (exp mode: with work space only)
cudaError_t ee_launch_cone_T(const EeParams& P, const EeBeamSpec* specs, const EeBeamGeom* geoms, const float* rev_grad,
                             const EeConeWork& work, float4* terma_grad, int nbeams, int max_lines, int max_line,
                             cudaStream_t s);
// zeros on every line's segment of a chunk's REV gradient arena (before
// ee_launch_gather_T; the forward cone kernels zero their own arena)
cudaError_t ee_launch_rev_zero(const EeParams& P, const EeBeamGeom* geoms, float* rev_grad, const EeConeWork& work,
                               int nbeams, int max_lines, cudaStream_t s);
// test option: EE_DEBUG_POISON=1 fills scratch with NaN where the engine
// relies on its kernels, not on a clear, to write every sample it reads
bool ee_debug_poison();
// per-beam status words of a geometry array (strided copy), for plans
cudaError_t ee_copy_status(const EeBeamGeom* geoms, int* status_host, int nbeams, cudaStream_t s);
cudaError_t ee_launch_terma_T(const EeParams& P, const EeBeamSpec* specs, const EeBeamGeom* geoms,
                              const float* unit_terma, const int* beamlet_idx, const float4* terma_grad,
                              float* fluence_grad, int nbeams, long long max_tvol, cudaStream_t s);
// EndtoEnd loss pieces
cudaError_t ee_launch_loss_grad(const float* dose, const float* ptv_w, const float* ptv_t, const float* oar_w,
                                const float* oar_t, float* grad, double* acc, long long n, cudaStream_t s);
cudaError_t ee_launch_spread(const EeBeamSpec* specs, const float* in, float* out, const float* w1d, int R, int nbeams,
                             int max_pix, cudaStream_t s);
cudaError_t ee_launch_smooth(const EeBeamSpec* specs, const float* x, float* grad, float eta, double* acc, int nbeams,
                             int max_pix, cudaStream_t s);

// Beamlet-column path (ee_beamlet.cu).
struct EeBeamletOptions {
    float kernel_extent;  // dose kernel truncation, cm (argparser.h:27: 2 cm)
    int max_rev[3];       // REV size limit that triggers re-batching (argparser.h:29: 500^3)
    long long scratch_bytes = 0;  // the context's scratch budget: directions whose REV arrays share a launch
};
// Warps that share the candidate samples of 32 units of a pillar's depth
// (k_bl_sources).  `area` cells of footprint are about 3 area candidates per
// unit, so as many steps of a warp for its 32 units; `warps`: the launch's
// without a split.  More than 64 steps are split, and down to 8 (the boxes cost
// about as much) while the launch has fewer than 16 warps per SM.  One beamlet of
// 8 cm on 64^3 at 2.5 mm: 53 ms with one warp per 32 units, 3.5 split (a thread
// per sample of the packed grid: 10.1); of 4 cm on 200 x 200 x 160 at 2 mm, a
// direction per launch: 303 ms, 7.8 (14.5).  A batch's usual hundred beamlets of
// a voxel or two stay whole.
inline int ee_bl_source_slices(double area, long long warps) {
    const double steps = 3.0 * area;
    const double few = std::fmin(steps / 8, 152.0 * 16.0 / (double)warps), n = std::fmax(steps / 64, few);
    return n < 1 ? 1 : (n > 4096 ? 4096 : (int)n);
}
int ee_beamlet_run(const EeParams& P, const EeRayConst* rays, cudaStream_t s, void** ws, const EeBeamletOptions& opt,
                   const ee_beam& beam, const EeBeamSpec& S, const float* fluence_host, float thresh, ee_csr* out);
void ee_beamlet_free(void* ws);
