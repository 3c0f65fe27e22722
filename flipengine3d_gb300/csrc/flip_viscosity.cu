// Viscosity (setViscosity; _applyViscosityToVelocityField,
// fluidsimulation.cpp:3592-3640): Batty's variational viscosity as the
// reference's ViscositySolver sets it up (viscositysolver.cpp:49-891),
// solved on the GPU.
//
// The set-up follows the reference operation by operation: face states from
// the solid level set at cell centres (:97-202), liquid cells dilated by two
// layers (:204-238), the liquid volume fractions of the cell, face and edge
// control volumes from the liquid level set at the control volumes' corners
// (:240-368, LevelsetUtils::volumeFraction), the faces in the system
// (:374-464) and each row's coefficients and right-hand side (:466-821).
// A corner value is sampled once, by the first valid control volume in flat
// order that touches it, at that volume's centre plus the corner's offset,
// as the reference's nodal cache does, so the fractions are the reference's
// bit for bit.
//
// The solve differs on purpose.  The reference runs its FP32 MIC(0)-PCG to
// a relative residual of 1e-4 (at most 700 iterations).  Here the system is
// solved by Jacobi-preconditioned CG in FP64 to 1e-9, so the
// result is the system's solution to well inside the reference's own
// tolerance; a reference-exact MIC(0) over this 15-point, three-component
// system would be a sequential triangular solve.  The faces of the system
// then take the solution and every other face is zeroed, as the reference's
// _applySolutionToVelocityField (:856-891) does.
#include <algorithm>
#include <cmath>
#include <string>

#include "../../include/flip3d.h"
#include "flip_device.cuh"

namespace flip {
namespace {

constexpr int TPB = 256;

// ---------------------------------------------------------------- geometry
struct VGrid {   // one control-volume grid: extents and corner offset from the cell centre
    int ni, nj, nk;
    float ox, oy, oz;
};

// LevelsetUtils::volumeFraction (levelsetutils.cpp:213-260, levelsetutils.h:62-104), float
__device__ __forceinline__ void sort4(float &a, float &b, float &c, float &d) {
    float t;
    if (a > b) { t = a; a = b; b = t; }
    if (c > d) { t = c; c = d; d = t; }
    if (a > c) { t = a; a = c; c = t; }
    if (b > d) { t = b; b = d; d = t; }
    if (b > c) { t = b; b = c; c = t; }
}
__device__ __forceinline__ float tet_fraction(float p0, float p1, float p2, float p3) {
    return __fdiv_rn(__fmul_rn(__fmul_rn(p0, p0), p0),
                     __fmul_rn(__fmul_rn(__fsub_rn(p0, p1), __fsub_rn(p0, p2)), __fsub_rn(p0, p3)));
}
__device__ __forceinline__ float prism_fraction(float p0, float p1, float p2, float p3) {
    const float a = __fdiv_rn(p0, __fsub_rn(p0, p2));
    const float b = __fdiv_rn(p0, __fsub_rn(p0, p3));
    const float c = __fdiv_rn(p1, __fsub_rn(p1, p3));
    const float d = __fdiv_rn(p1, __fsub_rn(p1, p2));
    return __fadd_rn(__fadd_rn(__fmul_rn(__fmul_rn(a, b), __fsub_rn(1.0f, d)),
                               __fmul_rn(__fmul_rn(b, __fsub_rn(1.0f, c)), d)),
                     __fmul_rn(c, d));
}
__device__ float tet_volume(float p0, float p1, float p2, float p3) {
    sort4(p0, p1, p2, p3);
    if (p3 <= 0) return 1.0f;
    if (p2 <= 0) return __fsub_rn(1.0f, tet_fraction(p3, p2, p1, p0));
    if (p1 <= 0) return prism_fraction(p0, p1, p2, p3);
    if (p0 <= 0) return tet_fraction(p0, p1, p2, p3);
    return 0.0f;
}
__device__ float cube_volume(float p000, float p100, float p010, float p110, float p001, float p101, float p011,
                             float p111) {
    float s = tet_volume(p000, p001, p101, p011);
    s = __fadd_rn(s, tet_volume(p000, p101, p100, p110));
    s = __fadd_rn(s, tet_volume(p000, p010, p011, p110));
    s = __fadd_rn(s, tet_volume(p101, p011, p111, p110));
    s = __fadd_rn(s, __fmul_rn(2.0f, tet_volume(p000, p011, p101, p110)));
    s = __fadd_rn(s, tet_volume(p100, p101, p001, p111));
    s = __fadd_rn(s, tet_volume(p100, p001, p000, p010));
    s = __fadd_rn(s, tet_volume(p100, p110, p111, p010));
    s = __fadd_rn(s, tet_volume(p001, p111, p011, p010));
    s = __fadd_rn(s, __fmul_rn(2.0f, tet_volume(p100, p111, p001, p010)));
    return __fdiv_rn(s, 12.0f);
}

// ParticleLevelSet::trilinearInterpolate (particlelevelset.cpp:136-138): the
// cell-centred liquid level set, read at p - dx/2 as a nodal grid, FP64
// weights, corners outside the grid 0, rounded to float.
__device__ float liquid_at(const StepConsts &c, const float *phi, float px, float py, float pz) {
    const float h = (float)(0.5 * c.dx);
    SourceGridView g{phi, c.I, c.J, c.K, 0.0f, 0.0f, 0.0f, c.dx};
    return source_phi(g, __fsub_rn(px, h), __fsub_rn(py, h), __fsub_rn(pz, h));
}

// ------------------------------------------------------------------ states
// Face states (viscositysolver.cpp:135-202): solid on the domain's border
// faces and where the solid level set's cell-centre values on the face's two
// sides sum to <= 0; cell-centre value = the mean of the cell's 8 nodes
// (MeshLevelSet::getDistanceAtCellCenter, meshlevelset.cpp:151-162).
__device__ __forceinline__ float solid_centre(const StepConsts &c, const float *S, int i, int j, int k) {
    const int ni = c.I + 1, nj = c.J + 1;
    auto at = [&](int a, int b, int d) { return S[(long long)a + (long long)ni * ((long long)b + (long long)nj * d)]; };
    float s = at(i, j, k);
    s = __fadd_rn(s, at(i + 1, j, k));
    s = __fadd_rn(s, at(i, j + 1, k));
    s = __fadd_rn(s, at(i + 1, j + 1, k));
    s = __fadd_rn(s, at(i, j, k + 1));
    s = __fadd_rn(s, at(i + 1, j, k + 1));
    s = __fadd_rn(s, at(i, j + 1, k + 1));
    s = __fadd_rn(s, at(i + 1, j + 1, k + 1));
    return __fmul_rn(0.125f, s);
}
__global__ void k_visc_states(StepConsts c, const float *S, uint8_t *fluidFace) {
    const long long nu = (long long)(c.I + 1) * c.J * c.K, nv = (long long)c.I * (c.J + 1) * c.K,
                    nw = (long long)c.I * c.J * (c.K + 1);
    const long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nu + nv + nw) return;
    int i, j, k;
    bool fluid;
    if (f < nu) {
        unflatten(f, c.I + 1, c.J, i, j, k);
        fluid = !(i == 0 || i == c.I) &&
                __fadd_rn(solid_centre(c, S, i - 1, j, k), solid_centre(c, S, i, j, k)) > 0.0f;
    } else if (f < nu + nv) {
        unflatten(f - nu, c.I, c.J + 1, i, j, k);
        fluid = !(j == 0 || j == c.J) &&
                __fadd_rn(solid_centre(c, S, i, j - 1, k), solid_centre(c, S, i, j, k)) > 0.0f;
    } else {
        unflatten(f - nu - nv, c.I, c.J, i, j, k);
        fluid = !(k == 0 || k == c.K) &&
                __fadd_rn(solid_centre(c, S, i, j, k - 1), solid_centre(c, S, i, j, k)) > 0.0f;
    }
    fluidFace[f] = fluid ? 1 : 0;
}

// Valid control volumes (viscositysolver.cpp:207-238): cells with liquid
// phi < 0 on an (I+1)(J+1)(K+1) grid, dilated twice over 6 neighbours.
__global__ void k_visc_valid(StepConsts c, const float *phi, uint8_t *valid) {
    const long long n = (long long)(c.I + 1) * (c.J + 1) * (c.K + 1);
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    int i, j, k;
    unflatten(t, c.I + 1, c.J + 1, i, j, k);
    valid[t] = (i < c.I && j < c.J && k < c.K && phi[(long long)i + (long long)c.I * ((long long)j + (long long)c.J * k)] < 0.0f)
                   ? 1 : 0;
}
__global__ void k_visc_dilate(StepConsts c, const uint8_t *in, uint8_t *out) {
    const int ni = c.I + 1, nj = c.J + 1, nk = c.K + 1;
    const long long n = (long long)ni * nj * nk;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    int i, j, k;
    unflatten(t, ni, nj, i, j, k);
    auto v = [&](int a, int b, int d) {
        return a >= 0 && b >= 0 && d >= 0 && a < ni && b < nj && d < nk &&
               in[(long long)a + (long long)ni * ((long long)b + (long long)nj * d)];
    };
    out[t] = (v(i, j, k) || v(i - 1, j, k) || v(i + 1, j, k) || v(i, j - 1, k) || v(i, j + 1, k) || v(i, j, k - 1) ||
              v(i, j, k + 1)) ? 1 : 0;
}

// The control-volume grids, in the order of ViscosityVolumeGrid
// (viscositysolver.h:57-78): centre, U, V, W, edgeU, edgeV, edgeW.  All seven
// go through one launch (blockIdx.y: the grid).
enum { VC = 0, VU, VV, VW, EU, EV, EW, NVOL };
struct VGrids {
    VGrid g[NVOL];
    float *node[NVOL], *vol[NVOL];
};

// Corner values (viscositysolver.cpp:278-368): node (a, b, d) of a grid's
// (ni+1)(nj+1)(nk+1) corners takes its value from the first valid volume in
// flat order among the eight that share it, sampled at that volume's centre
// plus the corner's offset.  The volume is found first and the sample, FP64,
// taken once for all lanes: in the search's loop it ran up to eight times a
// warp (16.5 us a grid at 40^3; all seven now 60 us).
__global__ void __launch_bounds__(TPB) k_visc_corners(StepConsts c, VGrids grids, const uint8_t *valid, const float *phi) {
    const VGrid g = grids.g[blockIdx.y];
    const int ni = g.ni + 1, nj = g.nj + 1, nk = g.nk + 1;
    const long long n = (long long)ni * nj * nk;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    int a, b, d;
    unflatten(t, ni, nj, a, b, d);
    const int vi = c.I + 1, vj = c.J + 1;
    // cells in ascending flat order: lower k first, then lower j, then lower i
    int first = -1;
#pragma unroll
    for (int q = 7; q >= 0; q--) {
        const int ci = a - 1 + (q & 1), cj = b - 1 + (q >> 1 & 1), ck = d - 1 + (q >> 2);
        if (ci < 0 || cj < 0 || ck < 0 || ci >= g.ni || cj >= g.nj || ck >= g.nk) continue;
        if (valid[(long long)ci + (long long)vi * ((long long)cj + (long long)vj * ck)]) first = q;
    }
    float val = 0.0f;
    if (first >= 0) {
        const int dxx = first & 1, dy = first >> 1 & 1, dz = first >> 2;
        const int ci = a - 1 + dxx, cj = b - 1 + dy, ck = d - 1 + dz;
        // centre = centerStart + GridIndexToCellCenter(ci, cj, ck, dx), then +-dx/2
        const float hdx = __fmul_rn(0.5f, (float)c.dx);
        const float cx = __fadd_rn(g.ox, (float)((double)(float)ci * c.dx + 0.5 * c.dx));
        const float cy = __fadd_rn(g.oy, (float)((double)(float)cj * c.dx + 0.5 * c.dx));
        const float cz = __fadd_rn(g.oz, (float)((double)(float)ck * c.dx + 0.5 * c.dx));
        // node (a, b, d) is corner (1 - dxx, 1 - dy, 1 - dz) of this cell
        const float px = __fadd_rn(cx, dxx ? -hdx : hdx);
        const float py = __fadd_rn(cy, dy ? -hdx : hdx);
        const float pz = __fadd_rn(cz, dz ? -hdx : hdx);
        val = liquid_at(c, phi, px, py, pz);
    }
    grids.node[blockIdx.y][t] = val;
}
__global__ void __launch_bounds__(TPB) k_visc_volumes(StepConsts c, VGrids grids, const uint8_t *valid) {
    const VGrid g = grids.g[blockIdx.y];
    const float *node = grids.node[blockIdx.y];
    float *vol = grids.vol[blockIdx.y];
    const long long n = (long long)g.ni * g.nj * g.nk;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    int i, j, k;
    unflatten(t, g.ni, g.nj, i, j, k);
    const int vi = c.I + 1, vj = c.J + 1;
    if (!valid[(long long)i + (long long)vi * ((long long)j + (long long)vj * k)]) {
        vol[t] = 0.0f;
        return;
    }
    const int ni = g.ni + 1, nj = g.nj + 1;
    auto nd = [&](int a, int b, int d) { return node[(long long)a + (long long)ni * ((long long)b + (long long)nj * d)]; };
    const float p000 = nd(i, j, k), p001 = nd(i, j, k + 1), p010 = nd(i, j + 1, k), p011 = nd(i, j + 1, k + 1);
    const float p100 = nd(i + 1, j, k), p101 = nd(i + 1, j, k + 1), p110 = nd(i + 1, j + 1, k),
                p111 = nd(i + 1, j + 1, k + 1);
    float v;
    if (p000 < 0 && p001 < 0 && p010 < 0 && p011 < 0 && p100 < 0 && p101 < 0 && p110 < 0 && p111 < 0) v = 1.0f;
    else if (p000 >= 0 && p001 >= 0 && p010 >= 0 && p011 >= 0 && p100 >= 0 && p101 >= 0 && p110 >= 0 && p111 >= 0)
        v = 0.0f;
    else v = cube_volume(p000, p100, p010, p110, p001, p101, p011, p111);
    vol[t] = v;
}

// ------------------------------------------------------------------ system
struct VolPtrs {
    const float *v[NVOL];
    int ni[NVOL], nj[NVOL];
};
__device__ __forceinline__ float vol(const VolPtrs &p, int g, int i, int j, int k) {
    return p.v[g][(long long)i + (long long)p.ni[g] * ((long long)j + (long long)p.nj[g] * k)];
}
struct FaceIdx {   // flat index of a face over the U, V, W grids, one after the other
    int I, J, K;
    long long nu, nv;
    __device__ long long u(int i, int j, int k) const { return (long long)i + (long long)(I + 1) * ((long long)j + (long long)J * k); }
    __device__ long long v(int i, int j, int k) const { return nu + (long long)i + (long long)I * ((long long)j + (long long)(J + 1) * k); }
    __device__ long long w(int i, int j, int k) const { return nu + nv + (long long)i + (long long)I * ((long long)j + (long long)J * k); }
    __device__ long long of(int d, int i, int j, int k) const { return d == 0 ? u(i, j, k) : d == 1 ? v(i, j, k) : w(i, j, k); }
};
// One coupling of a row, in the order the reference adds them: the face
// (direction, offset), which of the six factors, and its sign.
struct Term { signed char d, di, dj, dk, f, s; };
enum { FR = 0, FL, FT, FB, FF, FK };
struct TermTable {
    Term t[3][14] = {
    {{0, 1, 0, 0, FR, -1}, {0, -1, 0, 0, FL, -1}, {0, 0, 1, 0, FT, -1}, {0, 0, -1, 0, FB, -1}, {0, 0, 0, 1, FF, -1},
     {0, 0, 0, -1, FK, -1}, {1, 0, 1, 0, FT, -1}, {1, -1, 1, 0, FT, 1}, {1, 0, 0, 0, FB, 1}, {1, -1, 0, 0, FB, -1},
     {2, 0, 0, 1, FF, -1}, {2, -1, 0, 1, FF, 1}, {2, 0, 0, 0, FK, 1}, {2, -1, 0, 0, FK, -1}},
    {{1, 1, 0, 0, FR, -1}, {1, -1, 0, 0, FL, -1}, {1, 0, 1, 0, FT, -1}, {1, 0, -1, 0, FB, -1}, {1, 0, 0, 1, FF, -1},
     {1, 0, 0, -1, FK, -1}, {0, 1, 0, 0, FR, -1}, {0, 1, -1, 0, FR, 1}, {0, 0, 0, 0, FL, 1}, {0, 0, -1, 0, FL, -1},
     {2, 0, 0, 1, FF, -1}, {2, 0, -1, 1, FF, 1}, {2, 0, 0, 0, FK, 1}, {2, 0, -1, 0, FK, -1}},
    {{2, 1, 0, 0, FR, -1}, {2, -1, 0, 0, FL, -1}, {2, 0, 1, 0, FT, -1}, {2, 0, -1, 0, FB, -1}, {2, 0, 0, 1, FF, -1},
     {2, 0, 0, -1, FK, -1}, {0, 1, 0, 0, FR, -1}, {0, 1, 0, -1, FR, 1}, {0, 0, 0, 0, FL, 1}, {0, 0, 0, -1, FL, -1},
     {1, 0, 1, 0, FT, -1}, {1, 0, 1, -1, FT, 1}, {1, 0, 0, 0, FB, 1}, {1, 0, 0, -1, FB, -1}}};
};
__constant__ TermTable kTerms;
// The control volume behind each factor of a row of direction d: (grid, di, dj, dk)
__constant__ signed char kVol[3][7][4] = {
    {{VU, 0, 0, 0}, {VC, 0, 0, 0}, {VC, -1, 0, 0}, {EW, 0, 1, 0}, {EW, 0, 0, 0}, {EV, 0, 0, 1}, {EV, 0, 0, 0}},
    {{VV, 0, 0, 0}, {EW, 1, 0, 0}, {EW, 0, 0, 0}, {VC, 0, 0, 0}, {VC, 0, -1, 0}, {EU, 0, 0, 1}, {EU, 0, 0, 0}},
    {{VW, 0, 0, 0}, {EV, 1, 0, 0}, {EV, 0, 0, 0}, {EU, 0, 1, 0}, {EU, 0, 0, 0}, {VC, 0, 0, 0}, {VC, 0, 0, -1}}};

// The rows' coefficients by place in the list: six factors, diagonal, 1 /
// diagonal, each an array; the right-hand side (which becomes the residual).
struct RowCoefs {
    double *base, *rhs;
    long long room;
    __device__ double *at(int q) const { return base + q * room; }
};

struct SysArgs {
    FaceIdx fx;
    VolPtrs vp;
    const uint8_t *fluidFace;
    const float *u, *v, *w;
    float visc;     // the (constant) viscosity
    float factor;   // dt / dx^2 as the reference rounds it
};

__device__ __forceinline__ int face_of(const FaceIdx &fx, long long f, int &i, int &j, int &k) {
    if (f < fx.nu) { unflatten(f, fx.I + 1, fx.J, i, j, k); return 0; }
    if (f < fx.nu + fx.nv) { unflatten(f - fx.nu, fx.I, fx.J + 1, i, j, k); return 1; }
    unflatten(f - fx.nu - fx.nv, fx.I, fx.J, i, j, k);
    return 2;
}
__device__ __forceinline__ void row_volumes(const SysArgs &a, int d, int i, int j, int k, float *vv) {
#pragma unroll
    for (int q = 0; q < 7; q++)
        vv[q] = vol(a.vp, kVol[d][q][0], i + kVol[d][q][1], j + kVol[d][q][2], k + kVol[d][q][3]);
}

// Per face: in the system or not (viscositysolver.cpp:374-464); per block of
// faces, how many are.
__global__ void __launch_bounds__(TPB) k_visc_system(SysArgs a, long long nf, uint8_t *inSys, int *blockRows) {
    const long long f = (long long)blockIdx.x * TPB + threadIdx.x;
    bool in = false;
    if (f < nf) {
        int i, j, k;
        const int d = face_of(a.fx, f, i, j, k);
        if (i >= 1 && j >= 1 && k >= 1 && i < a.fx.I && j < a.fx.J && k < a.fx.K && a.fluidFace[f]) {
            float vv[7];
            row_volumes(a, d, i, j, k, vv);
            in = vv[0] > 0.0f || vv[1] > 0.0f || vv[2] > 0.0f || vv[3] > 0.0f || vv[4] > 0.0f || vv[5] > 0.0f || vv[6] > 0.0f;
        }
        inSys[f] = in;
    }
    const int rows = __syncthreads_count(in);
    if (threadIdx.x == 0) blockRows[blockIdx.x] = rows;
}

// The place of a face in the list of the system's faces, which is in order.
__device__ __forceinline__ int row_place(bool in, const int *start) {
    __shared__ int warps[TPB / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (lane == 0) warps[warp] = __popc(m);
    __syncthreads();
    int at = start[blockIdx.x] + __popc(m & ((1u << lane) - 1u));
    for (int w = 0; w < warp; w++) at += warps[w];
    return at;
}
__global__ void __launch_bounds__(TPB) k_visc_list(const uint8_t *inSys, long long nf, const int *start, int *list) {
    const long long f = (long long)blockIdx.x * TPB + threadIdx.x;
    const bool in = f < nf && inSys[f];
    const int at = row_place(in, start);
    if (in) list[at] = (int)f;
}

// Per row: its six factors, diagonal and right-hand side (:550-821), all in
// float, kept as doubles, which they are multiplied with.
__global__ void __launch_bounds__(TPB) k_visc_rows(SysArgs a, const int *list, const int *listed, RowCoefs c) {
    const int rows = *listed;
    for (int n = blockIdx.x * TPB + threadIdx.x; n < rows; n += gridDim.x * TPB) {
        const long long f = list[n];
        int i, j, k;
        const int d = face_of(a.fx, f, i, j, k);
        float vv[7];
        row_volumes(a, d, i, j, k, vv);
        const float v = a.visc;
        const float vq = __fmul_rn(0.25f, __fadd_rn(__fadd_rn(__fadd_rn(v, v), v), v));
        const float two = __fmul_rn(2.0f, a.factor);
        float F[6];
#pragma unroll
        for (int q = 0; q < 6; q++) {
            // the two factors across the row's own direction use the
            // viscosity at the cell centres, doubled; the others the
            // mean of four
            const bool own = (d == 0 && q < 2) || (d == 1 && (q == 2 || q == 3)) || (d == 2 && q >= 4);
            F[q] = own ? __fmul_rn(__fmul_rn(two, v), vv[q + 1]) : __fmul_rn(__fmul_rn(a.factor, vq), vv[q + 1]);
        }
        float diag = vv[0];
#pragma unroll
        for (int q = 0; q < 6; q++) diag = __fadd_rn(diag, F[q]);
        const float *G[3] = {a.u, a.v, a.w};
        const long long self = f - (d == 0 ? 0 : d == 1 ? a.fx.nu : a.fx.nu + a.fx.nv);
        float rval = __fmul_rn(vv[0], G[d][self]);
        for (int q = 0; q < 14; q++) {
            const Term t = kTerms.t[d][q];
            const long long g = a.fx.of(t.d, i + t.di, j + t.dj, k + t.dk);
            if (a.fluidFace[g]) continue;   // SOLID: the known velocity moves to the right-hand side
            const long long gl = g - (t.d == 0 ? 0 : t.d == 1 ? a.fx.nu : a.fx.nu + a.fx.nv);
            const float entry = t.s < 0 ? -F[t.f] : F[t.f];
            rval = __fsub_rn(rval, __fmul_rn(entry, G[t.d][gl]));
        }
#pragma unroll
        for (int q = 0; q < 6; q++) c.at(q)[n] = (double)F[q];
        c.at(6)[n] = (double)diag;
        c.at(7)[n] = 1.0 / (double)diag;
        c.rhs[n] = (double)rval;
    }
}
// _applySolutionToVelocityField (viscositysolver.cpp:856-891): the field is
// cleared and the system's faces take the solution; without a system it is left
// as it is (:55-58), as it is where a wait of the solver ran out.
__global__ void __launch_bounds__(TPB) k_visc_write(FaceIdx fx, long long nf, const uint8_t *inSys, const int *start,
                                                    const int *listed, const double *x, const double *scal, float *u, float *v,
                                                    float *w) {
    if (*listed == 0 || scal[7] != 0.0) return;
    const long long f = (long long)blockIdx.x * TPB + threadIdx.x;
    const bool in = f < nf && inSys[f];
    const int at = row_place(in, start);
    if (f >= nf) return;
    const float val = in ? (float)x[at] : 0.0f;
    if (f < fx.nu) u[f] = val;
    else if (f < fx.nu + fx.nv) v[f - fx.nu] = val;
    else w[f - fx.nu - fx.nv] = val;
}

// ------------------------------------------------------------------- solve
// Jacobi-preconditioned CG in FP64 over the faces in the system, all
// iterations in one cooperative launch.  The systems are small (41k rows at
// 40^3, a few MB), so what counts are the steps' latencies and FP64, of which an
// SM does two operations a cycle.  As five launches an iteration, two of them a
// sum in one CTA, it took 70 us at 40^3 (apply 24, sums 2 x 13, update 14,
// direction 4); here 15 us.
//   * chunks of 32 rows go to the SMs in turn, so that all have equally many;
//   * p stays implicit off its own row: p = z + beta p_old from the pair
//     {z, p_old} of a neighbour's row, zero off the system, so that a direction
//     needs no step of its own;
//   * products are added with one rounding (fma), and z = r (1 / diagonal);
//   * a sum over the rows is also the barrier: a CTA writes its share into a
//     slot, tagged with the number of the sum, and every CTA reads all slots,
//     in the same order.
// scal: [3] |r|inf  [4] |b|inf  [5] rows  [6] iterations  [7] 1: a wait ran out
constexpr int CG_CTAS = 320, CG_TPB = 512;
constexpr int CG_BATCH = 8;            // |r|inf is compared with the tolerance every so many iterations
constexpr int CG_MAX_ITER = 2000;

struct CgArgs {
    FaceIdx fx;
    RowCoefs c;
    const int *list, *listed;   // the rows' faces; how many
    double *x, *p, *q;          // a row's own, by place in the list (and c.rhs: r)
    double2 *zp;                // {z, p_old} by face
    unsigned long long *slots;  // [2][CG_CTAS][4]
    double *scal;
    unsigned spinLimit;         // looks of a wait before it gives up
    unsigned skew;              // 0; nonzero only to make the waits run out (fault injection)
};

// Sums a0 and takes the maximum of a1 >= 0 over the grid, in a fixed order, and
// is a barrier: what a CTA wrote to global memory before is seen after.  False
// once a wait ran out.
__device__ bool cg_all(const CgArgs &a, unsigned epoch, double &a0, double &a1) {
    constexpr int WARPS = CG_TPB / 32;
    __shared__ double s0[WARPS], t0;
    __shared__ long long s1[WARPS], t1;
    __shared__ int good;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long m = __double_as_longlong(a1);   // as integers in the same order
    auto lanes = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            a0 += __shfl_xor_sync(0xffffffffu, a0, o);
            m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        }
    };
    if (__any_sync(0xffffffffu, a0 != 0.0 || m != 0)) lanes();
    if (lane == 0) {
        s0[warp] = a0;
        s1[warp] = m;
    }
    __syncthreads();
    if (warp == 0) {
        a0 = lane < WARPS ? s0[lane] : 0.0;
        m = lane < WARPS ? s1[lane] : 0;
        lanes();
        // a slot's words: the halves of the two numbers, each with the sum's
        // number, so that a word is new or not as a whole.  Two sets in turn: a
        // CTA writes one again only after every CTA has read it.
        unsigned long long *set = a.slots + (size_t)(epoch & 1) * CG_CTAS * 4;
        // Release: the lanes that write the slot have met the CTA's other threads at
        // the barrier above, and their fence after it puts all that those wrote
        // before the slot.  Acquire: below, after the slots have been seen.
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        if (lane < 4) {
            const unsigned long long v = (unsigned long long)(lane < 2 ? __double_as_longlong(a0) : m);
            asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(set + 4 * blockIdx.x + lane),
                         "l"((unsigned long long)epoch << 32 | (v >> (lane & 1 ? 32 : 0) & 0xffffffffull))
                         : "memory");
        }
        a0 = 0.0;
        m = 0;
        bool ok = true;
        for (int first = lane; ok && first < (int)gridDim.x; first += 128) {   // four slots a lane at a time
            unsigned long long w[4][4];
            for (unsigned spin = 0;; spin++) {
                bool all = true;
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const int t = min(first + 32 * h, (int)gridDim.x - 1);
#pragma unroll
                    for (int q = 0; q < 4; q += 2)
                        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                                     : "=l"(w[h][q]), "=l"(w[h][q + 1])
                                     : "l"(set + 4 * t + q)
                                     : "memory");
                }
#pragma unroll
                for (int h = 0; h < 4; h++)
#pragma unroll
                    for (int q = 0; q < 4; q++) all &= (unsigned)(w[h][q] >> 32) == epoch + a.skew;
                if (all) break;
                if (spin >= a.spinLimit || ((spin & 1023u) == 1023u && *(volatile double *)&a.scal[7] != 0.0)) {
                    ok = false;
                    break;
                }
            }
#pragma unroll
            for (int h = 0; h < 4; h++)
                if (first + 32 * h < (int)gridDim.x) {
                    a0 += __longlong_as_double((long long)((w[h][0] & 0xffffffffull) | w[h][1] << 32));
                    m = max(m, (long long)((w[h][2] & 0xffffffffull) | w[h][3] << 32));
                }
        }
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        if (!ok) *(volatile double *)&a.scal[7] = 1.0;
        ok = __all_sync(0xffffffffu, ok);
        lanes();
        if (lane == 0) {
            t0 = a0;
            t1 = m;
            good = ok;
        }
    }
    __syncthreads();
    a0 = t0;
    a1 = __longlong_as_double(t1);
    return good != 0;   // written again only after the next sum's first barrier
}

// The couplings of row (i, j, k) of direction D, added to y in the reference's
// order: entries times the neighbours' p, which is 0 off the system.
template <int D>
__device__ __forceinline__ double couple(const CgArgs &a, int i, int j, int k, const double *F, double beta, double y) {
    double2 v[14];
#pragma unroll
    for (int q = 0; q < 14; q++) {
        constexpr TermTable T;
        const Term t = T.t[D][q];
        v[q] = __ldcg(&a.zp[a.fx.of(t.d, i + t.di, j + t.dj, k + t.dk)]);
    }
#pragma unroll
    for (int q = 0; q < 14; q++) {
        constexpr TermTable T;
        const Term t = T.t[D][q];
        y = __fma_rn(t.s < 0 ? -F[t.f] : F[t.f], __fma_rn(beta, v[q].y, v[q].x), y);
    }
    return y;
}

__global__ void __launch_bounds__(CG_TPB, 1) k_cg(CgArgs a) {
    const int rows = *a.listed, step = gridDim.x * CG_TPB;
    const int first = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + (threadIdx.x & 31);
    unsigned epoch = 0;
    double rz = 0.0, bmax = 0.0;
    for (int n = first; n < rows; n += step) {
        const double b = a.c.rhs[n], z = b * a.c.at(7)[n];
        rz = __fma_rn(b, z, rz);
        bmax = fmax(bmax, fabs(b));
        a.x[n] = 0.0;
        __stcg(&a.zp[a.list[n]], make_double2(z, 0.0));
    }
    bool ok = cg_all(a, ++epoch, rz, bmax);
    const double tol = 1e-9 * bmax;
    double beta = 0.0, rmax = bmax;
    int it = 0;
    while (ok && it < CG_MAX_ITER && rmax > tol) {
        double pq = 0.0, none = 0.0;
        for (int n = first; n < rows; n += step) {
            const int f = a.list[n];
            int i, j, k;
            const int d = face_of(a.fx, f, i, j, k);
            double F[6];
#pragma unroll
            for (int q = 0; q < 6; q++) F[q] = a.c.at(q)[n];
            const double2 own = __ldcg(&a.zp[f]);
            const double p = __fma_rn(beta, own.y, own.x);
            double y = a.c.at(6)[n] * p;
            y = d == 0 ? couple<0>(a, i, j, k, F, beta, y) : d == 1 ? couple<1>(a, i, j, k, F, beta, y) : couple<2>(a, i, j, k, F, beta, y);
            a.p[n] = p;
            a.q[n] = y;
            pq = __fma_rn(p, y, pq);
        }
        if (!(ok = cg_all(a, ++epoch, pq, none))) break;
        const double alpha = pq != 0.0 ? rz / pq : 0.0;
        double nrz = 0.0, nmax = 0.0;
        for (int n = first; n < rows; n += step) {
            const double p = a.p[n], r = __fma_rn(-alpha, a.q[n], a.c.rhs[n]), z = r * a.c.at(7)[n];
            a.x[n] = __fma_rn(alpha, p, a.x[n]);
            a.c.rhs[n] = r;
            __stcg(&a.zp[a.list[n]], make_double2(z, p));
            nrz = __fma_rn(r, z, nrz);
            nmax = fmax(nmax, fabs(r));
        }
        if (!(ok = cg_all(a, ++epoch, nrz, nmax))) break;
        beta = rz != 0.0 ? nrz / rz : 0.0;
        rz = nrz;
        if (++it % CG_BATCH == 0) rmax = nmax;
    }
    if (first == 0) {
        a.scal[3] = rmax;
        a.scal[4] = bmax;
        a.scal[5] = (double)rows;
        a.scal[6] = (double)it;
    }
}

}  // namespace

void viscosity_buffer_sizes(int I, int J, int K, long long *nf, long long *nn, long long *ncorner,
                            long long vol[7], long long *rowBlocks, long long *slotWords) {
    const long long nu = (long long)(I + 1) * J * K, nv = (long long)I * (J + 1) * K, nw = (long long)I * J * (K + 1);
    *nf = nu + nv + nw;
    *nn = (long long)(I + 1) * (J + 1) * (K + 1);
    *ncorner = (long long)(I + 2) * (J + 2) * (K + 2);
    const long long g[7][3] = {{I, J, K}, {I + 1, J, K}, {I, J + 1, K}, {I, J, K + 1}, {I, J + 1, K + 1},
                               {I + 1, J, K + 1}, {I + 1, J + 1, K}};
    for (int q = 0; q < 7; q++) vol[q] = g[q][0] * g[q][1] * g[q][2];
    const long long blocks = div_up(*nf, TPB);   // their counts, the counts' scan, its total and scratch
    *rowBlocks = 2 * blocks + 2 + scan_scratch_ints((int)blocks);
    *slotWords = 8LL * CG_CTAS;
}

// The viscosity step on the device (buffers from the caller, sized by
// viscosity_buffer_sizes).  Returns FLIP_OK, FLIP_E_DEVICE_TIMEOUT (a wait ran
// out: the field is as it was) or FLIP_E_CUDA.
int viscosity_apply(const StepConsts &c, const ViscosityBuffers &vb, const float *liquidPhi, const float *solidPhi,
                    float *u, float *v, float *w, double visc, double dt, unsigned spinLimit, bool stall,
                    ViscosityResult *res, cudaStream_t s) {
    const long long nu = (long long)(c.I + 1) * c.J * c.K, nv = (long long)c.I * (c.J + 1) * c.K,
                    nw = (long long)c.I * c.J * (c.K + 1), nf = nu + nv + nw;
    const long long nn = (long long)(c.I + 1) * (c.J + 1) * (c.K + 1);
    { FLIP_COUNT(1); k_visc_states<<<div_up(nf, TPB), TPB, 0, s>>>(c, solidPhi, vb.fluidFace); }
    { FLIP_COUNT(1); k_visc_valid<<<div_up(nn, TPB), TPB, 0, s>>>(c, liquidPhi, vb.valid); }
    { FLIP_COUNT(1); k_visc_dilate<<<div_up(nn, TPB), TPB, 0, s>>>(c, vb.valid, vb.valid2); }
    { FLIP_COUNT(1); k_visc_dilate<<<div_up(nn, TPB), TPB, 0, s>>>(c, vb.valid2, vb.valid); }
    // the seven control-volume grids and their corner offsets (viscositysolver.cpp:240-248)
    const float h = (float)(0.5 * c.dx);
    VGrids grids = {{{c.I, c.J, c.K, h, h, h},         {c.I + 1, c.J, c.K, 0, h, h},
                     {c.I, c.J + 1, c.K, h, 0, h},     {c.I, c.J, c.K + 1, h, h, 0},
                     {c.I, c.J + 1, c.K + 1, h, 0, 0}, {c.I + 1, c.J, c.K + 1, 0, h, 0},
                     {c.I + 1, c.J + 1, c.K, 0, 0, h}}, {}, {}};
    VolPtrs vp;
    long long ncorner = 0;   // of the largest grid, which bounds its volumes too
    for (int g = 0; g < NVOL; g++) {
        const VGrid &G = grids.g[g];
        ncorner = std::max(ncorner, (long long)(G.ni + 1) * (G.nj + 1) * (G.nk + 1));
        grids.node[g] = vb.node[g];
        grids.vol[g] = vb.vol[g];
        vp.v[g] = vb.vol[g];
        vp.ni[g] = G.ni;
        vp.nj[g] = G.nj;
    }
    { FLIP_COUNT(1); k_visc_corners<<<dim3(div_up(ncorner, TPB), NVOL), TPB, 0, s>>>(c, grids, vb.valid, liquidPhi); }
    { FLIP_COUNT(1); k_visc_volumes<<<dim3(div_up(ncorner, TPB), NVOL), TPB, 0, s>>>(c, grids, vb.valid); }
    SysArgs sa;
    sa.fx = FaceIdx{c.I, c.J, c.K, nu, nv};
    sa.vp = vp;
    sa.fluidFace = vb.fluidFace;
    sa.u = u;
    sa.v = v;
    sa.w = w;
    sa.visc = (float)visc;
    const float invdx = (float)(1.0 / c.dx);
    sa.factor = (float)(dt * (double)invdx * (double)invdx);
    const int blocks = (int)div_up(nf, TPB);
    int *start = vb.blockRows + blocks, *total = start + blocks + 1;
    const RowCoefs coefs{vb.coefs, vb.r, nf};
    { FLIP_COUNT(1); k_visc_system<<<blocks, TPB, 0, s>>>(sa, nf, vb.inSys, vb.blockRows); }
    launch_scan_cells(vb.blockRows, blocks, start, total + 1, total, s);
    { FLIP_COUNT(1); k_visc_list<<<blocks, TPB, 0, s>>>(vb.inSys, nf, start, vb.list); }
    { FLIP_COUNT(1); k_visc_rows<<<std::min(blocks, 152 * 8), TPB, 0, s>>>(sa, vb.list, total, coefs); }
    // an epoch half the numbers away is never written
    const CgArgs a{sa.fx, coefs, vb.list, total, vb.x, vb.p, vb.q, vb.zp, vb.slots, vb.scal,
                   spinLimit ? spinLimit : DEFAULT_SPIN_LIMIT, stall ? 1u << 31 : 0u};
    cudaError_t e = cudaMemsetAsync(vb.zp, 0, (size_t)nf * sizeof(double2), s);   // off the system
    if (e == cudaSuccess) e = cudaMemsetAsync(vb.slots, 0, sizeof(unsigned long long) * 8 * CG_CTAS, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(vb.scal, 0, 8 * sizeof(double), s);
    // a CTA per SM, fewer where they would have less than a chunk of rows each
    // (one face in five is in a system as a rule)
    int dev = 0, sms = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) {
        const int ctas = std::max(std::min({(int)div_up(nf, 5 * 32), sms, CG_CTAS}), 1);
        void *args[] = {const_cast<CgArgs *>(&a)};
        FLIP_COUNT(1);
        e = cudaLaunchCooperativeKernel((const void *)k_cg, dim3(ctas), dim3(CG_TPB), args, 0, s);
    }
    if (e != cudaSuccess) return record_error(FLIP_E_CUDA, std::string("viscosity: ") + cudaGetErrorString(e));
    { FLIP_COUNT(1); k_visc_write<<<blocks, TPB, 0, s>>>(sa.fx, nf, vb.inSys, start, total, vb.x, vb.scal, u, v, w); }
    double hs[8];
    e = cudaMemcpyAsync(hs, vb.scal, sizeof(hs), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) { FLIP_SYNC_COUNT(); e = cudaStreamSynchronize(s); }
    if (e != cudaSuccess) return record_error(FLIP_E_CUDA, std::string("viscosity: ") + cudaGetErrorString(e));
    if (hs[7] != 0.0) return record_error(FLIP_E_DEVICE_TIMEOUT, "viscosity: a wait of the solver ran out");
    res->rows = (long long)hs[5];
    res->iterations = (int)hs[6];
    res->residual = hs[4] > 0 && res->rows > 0 ? hs[3] / hs[4] : 0.0;
    e = cudaGetLastError();
    if (e != cudaSuccess) return record_error(FLIP_E_CUDA, std::string("viscosity: ") + cudaGetErrorString(e));
    return FLIP_OK;
}

}  // namespace flip
