// FLIP step kernels for GB300 (sm_103a): particle binning, liquid SDF, P2G,
// extrapolation, body force, constrain, and the fused PIC/FLIP + RK3 +
// collision particle update.  Gathers and stencils: the searches, the splat and
// the update are bound by the instructions and the latency of scattered reads,
// the rest by HBM or, on small grids, by launches.  Nothing here is a dense
// contraction, so no tensor cores are involved.
#include <cstdio>
#include <type_traits>

#include "flip_device.cuh"

namespace flip {

namespace {

constexpr int TPB = 256;

struct F3 { float x, y, z; };
__device__ __forceinline__ F3 f3(float x, float y, float z) { F3 r; r.x = x; r.y = y; r.z = z; return r; }
__device__ __forceinline__ F3 add(F3 a, F3 b) { return f3(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z)); }
__device__ __forceinline__ F3 sub(F3 a, F3 b) { return f3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)); }
__device__ __forceinline__ F3 mul(float s, F3 v) { return f3(__fmul_rn(v.x, s), __fmul_rn(v.y, s), __fmul_rn(v.z, s)); }
__device__ __forceinline__ float dot3(F3 a, F3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ float len3(F3 a) { return __fsqrt_rn(dot3(a, a)); }
// vmath operator/ : multiply by (float)(1.0 / s)  (src/engine/vmath.cpp:100-103)
__device__ __forceinline__ F3 normalize3(F3 v) {
    float inv = (float)(1.0 / (double)len3(v));
    return mul(inv, v);
}

// ------------------------------------------------------------------ binning
__global__ void k_keys(ParticleSoA p, int n, StepConsts c, unsigned int *keys) {
    pdl_begin();
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    int i = exact_floor(p.px[t], c.invdx, c.invdxf);
    int j = exact_floor(p.py[t], c.invdx, c.invdxf);
    int k = exact_floor(p.pz[t], c.invdx, c.invdxf);
    Dims d{c.I, c.J, c.K};
    keys[t] = d.in(i, j, k) ? (unsigned int)d.idx(i, j, k) : KEY_SOLID;
}

__global__ void k_bin_count(const unsigned int *keys, int n, int *count) {
    pdl_begin();
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    unsigned int k = keys[t];
    if (k & KEY_SOLID) return;
    atomicAdd(&count[k & KEY_CELL_MASK], 1);
}

// Exclusive scan of n ints: 4096 per block, then the block totals.
constexpr int SCAN_T = 1024, SCAN_PER = 4, SCAN_TILE = SCAN_T * SCAN_PER;

__device__ int block_scan_excl(int v, int *sh, int *total) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = (lane < (int)(blockDim.x >> 5)) ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        sh[lane] = w;
    }
    __syncthreads();
    int base = warp > 0 ? sh[warp - 1] : 0;
    if (total) *total = sh[(blockDim.x >> 5) - 1];
    int r = base + x - v;
    __syncthreads();
    return r;
}

__global__ void k_scan_tiles(const int *in, int n, int *out, int *tileSums) {
    pdl_begin();
    __shared__ int sh[32];
    long long base = (long long)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_PER;
    int v[SCAN_PER];
    int sum = 0;
#pragma unroll
    for (int q = 0; q < SCAN_PER; q++) {
        long long g = base + q;
        v[q] = g < n ? in[g] : 0;
        sum += v[q];
    }
    int total;
    int ex = block_scan_excl(sum, sh, &total);
#pragma unroll
    for (int q = 0; q < SCAN_PER; q++) {
        long long g = base + q;
        if (g < n) out[g] = ex;
        ex += v[q];
    }
    if (threadIdx.x == 0) tileSums[blockIdx.x] = total;
}

__global__ void k_scan_sums(int *tileSums, int ntiles, int *grandTotal) {
    pdl_begin();
    __shared__ int sh[32];
    int v[SCAN_PER];
    int sum = 0;
#pragma unroll
    for (int q = 0; q < SCAN_PER; q++) {
        int g = threadIdx.x * SCAN_PER + q;
        v[q] = g < ntiles ? tileSums[g] : 0;
        sum += v[q];
    }
    int total;
    int ex = block_scan_excl(sum, sh, &total);
#pragma unroll
    for (int q = 0; q < SCAN_PER; q++) {
        int g = threadIdx.x * SCAN_PER + q;
        if (g < ntiles) tileSums[g] = ex;
        ex += v[q];
    }
    if (threadIdx.x == 0) *grandTotal = total;
}

__global__ void k_scan_add(int *out, int n, const int *tileSums, const int *grandTotal) {
    pdl_begin();
    long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g < n) out[g] += tileSums[g / SCAN_TILE];
    if (g == n) out[n] = *grandTotal;
}

__global__ void k_bin_scatter(const unsigned int *keys, int n, const int *start, int *cursor, int *slots) {
    pdl_begin();
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    unsigned int k = keys[t];
    if (k & KEY_SOLID) return;
    int c = (int)(k & KEY_CELL_MASK);
    int pos = start[c] + atomicAdd(&cursor[c], 1);
    slots[pos] = t;
}

// Per cell: order the slots by particle id (the reference's order), then
// apply the 250-per-cell limit (first by id) and the extreme-speed removal,
// as _removeMarkerParticles does (src/engine/fluidsimulation.cpp:4324-4353).
// Kept slots are compacted to the front of the cell's segment.
__global__ void k_cell_sort_select(const int *start, int ncells, int *slots, const unsigned int *ids,
                                   const unsigned int *keys, int maxPerCell, int *survivors) {
    pdl_begin();
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncells) return;
    int b = start[c], e = start[c + 1];
    for (int a = b + 1; a < e; a++) {
        int s = slots[a];
        unsigned int key = ids[s];
        int q = a - 1;
        while (q >= b && ids[slots[q]] > key) {
            slots[q + 1] = slots[q];
            q--;
        }
        slots[q + 1] = s;
    }
    int kept = 0;
    for (int a = b; a < e; a++) {
        int s = slots[a];
        int rank = a - b;
        if (rank >= maxPerCell) continue;
        if (keys[s] & KEY_FAST) continue;
        slots[b + kept] = s;
        kept++;
    }
    survivors[c] = kept;
}

// The kept particles in (cell, id) order, a thread per binned particle: writes are
// coalesced, and reads nearly so, since particles move few cells (a thread per
// cell took 813 us with 14.0M particles, stage "binning", this 537).  Where none was
// removed, which the totals of the two scans tell, particle t of the result is
// slots[t].  Otherwise slots[t] is of the cell whose segment t lies in, kept if its
// place there is among the first ones (300 particles of 256 x 128 x 128 cells, 50 of
// them removed from one: the stage takes 1.25 ms, most of it that cell's sort; a
// thread per cell, as many as there are particles, took 3.3 ms).
__device__ __forceinline__ float gather_one(const ParticleSoA &src, const ParticleSoA &dst, int s, int o) {
    const float vx = src.vx[s], vy = src.vy[s], vz = src.vz[s];
    dst.px[o] = src.px[s];
    dst.py[o] = src.py[s];
    dst.pz[o] = src.pz[s];
    dst.vx[o] = vx;
    dst.vy[o] = vy;
    dst.vz[o] = vz;
    dst.id[o] = src.id[s];
    return __fadd_rn(__fadd_rn(__fmul_rn(vx, vx), __fmul_rn(vy, vy)), __fmul_rn(vz, vz));
}
__global__ void k_gather(ParticleSoA src, ParticleSoA dst, const int *start, const int *slots, const unsigned int *keys,
                         const int *newStart, int ncells, unsigned int *maxSpeedSqBits) {
    pdl_begin();
    const int binned = start[ncells];
    const bool all = newStart[ncells] == binned;
    float best = 0.0f;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < binned; t += gridDim.x * blockDim.x) {
        const int s = slots[t];
        int o = t;
        if (!all) {
            const int c = (int)(keys[s] & KEY_CELL_MASK), place = t - start[c], first = newStart[c];
            if (place >= newStart[c + 1] - first) continue;
            o = first + place;
        }
        best = fmaxf(best, gather_one(src, dst, s, o));
    }
    for (int o = 16; o > 0; o >>= 1) best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((threadIdx.x & 31) == 0 && best > 0.0f) atomicMax(maxSpeedSqBits, __float_as_uint(best));
}

// --------------------------------------------------------------- liquid SDF
// The reference scatters (particlelevelset.cpp:582-629): every particle in the
// list of a block of 10^3 cells (particlelevelset.h:140-142) updates the
// block's cells in its search box with min(|c - p| - r), in the block's own
// float frame.  Min is order-free, and rounded square root and the subtraction
// of r are both monotone, so the smallest squared distance per cell and one
// square root give the reference's bits.  Here each cell looks for its nearest
// particle: its own cell first, then the rows of cells around it, nearest
// first, as long as a row can still hold a nearer one.  A cell inside the
// liquid has a particle within half a cell and stops at its own, and the air
// far from it knows from a look of the warp at the 25 rows around.  Bound by the
// latency and the instructions of the cells near the surface.  The stage in
// frames: 253 us at 128^3 (4.1M particles), 69 at 64^3, 251 at 256x128x128 (14.0M);
// scattering every particle into the ~100 cells of its box through shared-memory
// atomics took 857, 375 and 1947.  64 registers a thread: with 128 the occupancy is
// too low, with 42 small grids lose what large ones gain (the kernel alone, in CTAs
// of 512: 313, 456 and 274 us at 128^3, 68, 94 and 74 at 64^3).
// Then the solid post-process (particlelevelset.cpp:172-196).
constexpr int BW = 10;

// Does the reference's count pass put particle p in block (bx,by,bz)'s list?
// (particlelevelset.cpp:477-532, velocityadvector.cpp:272-329)
__device__ __forceinline__ bool in_block_list(float px, float py, float pz, float sr, float blockdxf,
                                              double invBlock, float invBlockf, const float *blockPosF,
                                              int bx, int by, int bz) {
    int ci = exact_floor(px, invBlock, invBlockf), cj = exact_floor(py, invBlock, invBlockf),
        ck = exact_floor(pz, invBlock, invBlockf);
    // (float)((double)(float)n * (double)blockdxf), tabulated from n = -1
    float bpx = blockPosF[ci + 1], bpy = blockPosF[cj + 1], bpz = blockPosF[ck + 1];
    if (__fsub_rn(px, sr) > bpx && __fsub_rn(py, sr) > bpy && __fsub_rn(pz, sr) > bpz &&
        __fadd_rn(px, sr) < __fadd_rn(bpx, blockdxf) && __fadd_rn(py, sr) < __fadd_rn(bpy, blockdxf) &&
        __fadd_rn(pz, sr) < __fadd_rn(bpz, blockdxf)) {
        return ci == bx && cj == by && ck == bz;
    }
    int i0 = exact_floor(__fsub_rn(px, sr), invBlock, invBlockf), i1 = exact_floor(__fadd_rn(px, sr), invBlock, invBlockf);
    int j0 = exact_floor(__fsub_rn(py, sr), invBlock, invBlockf), j1 = exact_floor(__fadd_rn(py, sr), invBlock, invBlockf);
    int k0 = exact_floor(__fsub_rn(pz, sr), invBlock, invBlockf), k1 = exact_floor(__fadd_rn(pz, sr), invBlock, invBlockf);
    return bx >= i0 && bx <= i1 && by >= j0 && by <= j1 && bz >= k0 && bz <= k1;
}

// Does the reference's scatter take particle p to cell (a, b, cc) of block
// (bx, by, bz)?  lx..lz: p in the block's frame.
__device__ __noinline__ bool sdf_reaches(const StepConsts &c, float px, float py, float pz, float lx, float ly, float lz,
                                         float sr, int bx, int by, int bz, int a, int b, int cc) {
    if (!in_block_list(px, py, pz, sr, c.blockdxf, c.invBlock, c.invBlockf, c.blockPosF, bx, by, bz)) return false;
    return a >= exact_floor(__fsub_rn(lx, sr), c.invdx, c.invdxf) && a <= exact_floor(__fadd_rn(lx, sr), c.invdx, c.invdxf) &&
           b >= exact_floor(__fsub_rn(ly, sr), c.invdx, c.invdxf) && b <= exact_floor(__fadd_rn(ly, sr), c.invdx, c.invdxf) &&
           cc >= exact_floor(__fsub_rn(lz, sr), c.invdx, c.invdxf) && cc <= exact_floor(__fadd_rn(lz, sr), c.invdx, c.invdxf);
}

// The rows of cells around a cell, {offset in y, in z}, nearest first: the
// cell's own row, then those that touch it, then the second ring.
__constant__ signed char kRing[25][2] = {
    {0, 0},  {-1, 0}, {1, 0},  {0, -1},  {0, 1},  {-1, -1}, {1, -1}, {-1, 1}, {1, 1},  {-2, 0}, {2, 0},  {0, -2}, {0, 2},
    {-2, -1}, {2, -1}, {-2, 1}, {2, 1}, {-1, -2}, {1, -2}, {-1, 2}, {1, 2}, {-2, -2}, {2, -2}, {-2, 2}, {2, 2}};

// A tuning knob sets the threads of two CTAs (256, 512 or 1024; default 512).
template <int SDF_TPB>
__global__ void __launch_bounds__(SDF_TPB, 1024 / SDF_TPB) k_liquid_sdf(ParticleSoA ps, const int *cellStart, StepConsts c,
                                                     const uint8_t *solidCC, float *phi) {
    pdl_begin();
    const long long ci = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    Dims cells{c.I, c.J, c.K};
    const bool valid = ci < cells.size();
    int gi, gj, gk;
    unflatten(valid ? ci : 0, c.I, c.J, gi, gj, gk);
    // Which of the rows around hold particles that the warp's cells could reach:
    // where the cells are of one row, a lane looks at a row; no row, no search.
    const int lane = threadIdx.x & 31, gi0 = __shfl_sync(0xffffffffu, gi, 0), gi1 = __shfl_sync(0xffffffffu, gi, 31);
    unsigned rows = 0x1ffffffu;
    if (__all_sync(0xffffffffu, valid && gi == gi0 + lane)) {
        bool any = false;
        if (lane < 25) {
            const int y = gj + kRing[lane][0], z = gk + kRing[lane][1];
            if (y >= 0 && z >= 0 && y < c.J && z < c.K) {
                const long long base = cells.idx(0, y, z);
                any = cellStart[base + max(gi0 - 2, 0)] != cellStart[base + min(gi1 + 2, c.I - 1) + 1];
            }
        }
        rows = __ballot_sync(0xffffffffu, any);
    }
    if (!valid) return;
    const float maxd = c.sdfMax, r = c.radiusf;
    const float sr = __fmul_rn(2.0f, r);
    const int bx = gi / BW, by = gj / BW, bz = gk / BW, a = gi - bx * BW, b = gj - by * BW, cc = gk - bz * BW;
    const float offx = c.blockPos[bx + 1], offy = c.blockPos[by + 1], offz = c.blockPos[bz + 1];
    const float cx = c.centre[a], cy = c.centre[b], cz = c.centre[cc];
    // A particle nearer than this is within the search radius and so in the
    // list and the box, whatever the rounding; farther ones are looked up.
    // The box reaches sr + dx / 2 = 2.2321 dx along an axis.
    const float near = 1.7f * c.dxf, near2 = near * near, reach = 2.24f * c.dxf;
    // Squared distance of the nearest point of a cell 1 or 2 away along an
    // axis, less a margin far above the rounding of the distances below.
    const float h1 = 0.499f * c.dxf, h2 = 1.499f * c.dxf, q1 = h1 * h1, q2 = h2 * h2;
    float best = __uint_as_float(0x7f800000u);   // +inf
    // The cell's centre in the simulation's frame, for a first look: `slack` is far
    // above what the rounding of such coordinates makes of a squared distance.
    const float mx = offx + cx, my = offy + cy, mz = offz + cz, slack = 0.03f * c.dxf * c.dxf;
    // four particles at a time, so that their loads overlap (the last one
    // repeated at the end does not change the minimum)
    auto look = [&](int from, int to) {
        for (int t = from; t < to; t += 4) {
            float x[4], y[4], z[4], d2[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int tq = min(t + q, to - 1);
                x[q] = ps.px[tq];
                y[q] = ps.py[tq];
                z[q] = ps.pz[tq];
            }
            bool hit = false;
            const float bar = best + slack;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float ex = x[q] - mx, ey = y[q] - my, ez = z[q] - mz;
                hit |= __fmaf_rn(ez, ez, __fmaf_rn(ey, ey, ex * ex)) < bar;
            }
            if (!hit) continue;
            hit = false;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float ddx = __fsub_rn(cx, __fsub_rn(x[q], offx)), dy = __fsub_rn(cy, __fsub_rn(y[q], offy)),
                            dz = __fsub_rn(cz, __fsub_rn(z[q], offz));
                d2[q] = __fadd_rn(__fadd_rn(__fmul_rn(ddx, ddx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                // beyond the box along an axis: out, whatever the rounding
                if (fmaxf(fabsf(ddx), fmaxf(fabsf(dy), fabsf(dz))) > reach) d2[q] = __uint_as_float(0x7f800000u);
                hit |= d2[q] < best;
            }
            if (!hit) continue;
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (d2[q] < best && (d2[q] < near2 || sdf_reaches(c, x[q], y[q], z[q], __fsub_rn(x[q], offx),
                                                                 __fsub_rn(y[q], offy), __fsub_rn(z[q], offz), sr, bx, by,
                                                                 bz, a, b, cc)))
                    best = d2[q];
        }
    };
    if (rows & 1) look(cellStart[ci], cellStart[ci + 1]);
    if (best > q1) {
        for (unsigned left = rows; left; left &= left - 1) {
            const int n = __ffs(left) - 1, oy = kRing[n][0], oz = kRing[n][1];
            const float ly = oy == 0 ? 0.0f : (oy == 1 || oy == -1 ? q1 : q2), lz = oz == 0 ? 0.0f : (oz == 1 || oz == -1 ? q1 : q2);
            const float row = ly + lz;   // as near as the row can be
            if (!(best > row)) continue;
            const int y = gj + oy, z = gk + oz;
            if (y < 0 || z < 0 || y >= c.J || z >= c.K) continue;
            const long long base = cells.idx(0, y, z);
            const int w = best > row + q2 ? 2 : (best > row + q1 ? 1 : 0);
            const int x0 = max(gi - w, 0), x1 = min(gi + w, c.I - 1);
            if (n == 0) {   // its own cell is done
                look(cellStart[base + x0], cellStart[ci]);
                look(cellStart[ci + 1], cellStart[base + x1 + 1]);
            } else {
                look(cellStart[base + x0], cellStart[base + x1 + 1]);
            }
        }
    }
    float val = __float_as_uint(best) == 0x7f800000u ? maxd : fminf(maxd, __fsub_rn(__fsqrt_rn(best), r));
    if (val < c.sdfHalf && solidCC[ci]) val = c.sdfNeg;
    if (fabsf(val) < c.sdfEps) val = val > 0 ? c.sdfEps : -c.sdfEps;
    phi[ci] = val;
}

// ---------------------------------------------------------------------- P2G
// Gather form of VelocityAdvector (velocityadvector.cpp:38-459): one thread
// per grid index (i, j, k) for its u, v and w face together; candidate
// particles come from the 27 cells that can hold a particle within r of one of
// them (18 per face); each particle's weight is evaluated in the reference's
// 10^3-block frame, which the three faces share.  Sums run in a fixed (cell,
// id) order, so the result is deterministic (no float atomics).
// Bound by instructions: 144 candidates a face, 22 within r.  So two particles
// at a time, in packed arithmetic (each half rounds as the scalar operation),
// and of each row of cells only the faces it can reach.  The lanes of a warp
// visit different cells, so a load touches 32 lines; positions and velocities
// load in pairs.  The stage in frames, with the extrapolation's seven layers: 587 us
// at 128^3 (4.1M particles), 889 at 256x128x128 (14.0M), the kernel 476 at 128^3
// (cold, in a profile); with a kernel per direction 875 and 2389.  16-byte vectors of
// a particle's coordinates touch four times the lines: slower.
// The reference also requires the face to lie in the particle's local box and
// the particle to be in the block's list, both taken with the support radius
// sr = r + 1e-6.  A particle within r of the face meets both: every coordinate
// of the face is within r of the particle, and the 1e-6 margin is far above
// the rounding of these float expressions (ulp(1) ~ 1.2e-7).
constexpr int P2G_TPB = 128;
__global__ void __launch_bounds__(P2G_TPB, 1024 / P2G_TPB) k_p2g(ParticleSoA p, const int *cellStart, StepConsts c,
                                             float *U, float *V, float *W, uint8_t *vu, uint8_t *vv, uint8_t *vw,
                                             PairOps k2) {
    pdl_begin();
    const int ni = c.I + 1, nj = c.J + 1, nk = c.K + 1;
    const long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= (long long)ni * nj * nk) return;
    int fi, fj, fk;
    unflatten(f, ni, nj, fi, fj, fk);
    const double dx = c.dx;
    const float r = (float)c.radius;
    const float rsq = __fmul_rn(r, r);
    // same expression trees as the reference's coefficient set-up
    const float coef1 = __fmul_rn(4.0f / 9.0f, __fdiv_rn(1.0f, __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(r, r), r), r), r), r)));
    const float coef2 = __fmul_rn(17.0f / 9.0f, __fdiv_rn(1.0f, __fmul_rn(__fmul_rn(__fmul_rn(r, r), r), r)));
    const float coef3 = __fmul_rn(22.0f / 9.0f, __fdiv_rn(1.0f, __fmul_rn(r, r)));
    const float h = (float)(0.5 * dx);
    const int bx = fi / BW, by = fj / BW, bz = fk / BW;
    const float offx = c.blockPos[bx + 1], offy = c.blockPos[by + 1], offz = c.blockPos[bz + 1];
    const float gx = c.nodePos[fi - bx * BW], gy = c.nodePos[fj - by * BW], gz = c.nodePos[fk - bz * BW];
    const bool isU = fj < c.J && fk < c.K, isV = fi < c.I && fk < c.K, isW = fi < c.I && fj < c.J;
    const int cx0 = max(fi - 1, 0), cx1 = min(fi + 1, c.I - 1), cy0 = max(fj - 1, 0), cy1 = min(fj + 1, c.J - 1),
              cz0 = max(fk - 1, 0), cz1 = min(fk + 1, c.K - 1);
    Dims cells{c.I, c.J, c.K};
    const F2 nox = f2(-offx, -offx), noy = f2(-offy, -offy), noz = f2(-offz, -offz), nh = f2(-h, -h);
    const F2 pgx = f2(gx, gx), pgy = f2(gy, gy), pgz = f2(gz, gz);
    const F2 c1 = f2(coef1, coef1), c2 = f2(coef2, coef2), c3 = f2(coef3, coef3), one = PairOps::ONE;
    float sc[3] = {0.0f, 0.0f, 0.0f}, wt[3] = {0.0f, 0.0f, 0.0f};
    // Two particles' shares of a face: weights of the two together, then the
    // sums in the particles' order.
    auto take = [&](int d, F2 d2, const F2 *vel, bool first, bool second) {
        const bool h0 = first && f2_x(d2) < rsq, h1 = second && f2_y(d2) < rsq;
        if (!(h0 | h1)) return;
        const F2 v = *vel;
        const F2 w3 = k2.mul(k2.mul(k2.mul(c1, d2), d2), d2), w2 = k2.mul(k2.mul(c2, d2), d2), w1 = k2.mul(c3, d2);
        const F2 wgt = k2.sub(k2.add(k2.sub(one, w3), w2), w1), wv = k2.mul(wgt, v);
        if (h0) {
            sc[d] = __fadd_rn(sc[d], f2_x(wv));
            wt[d] = __fadd_rn(wt[d], f2_x(wgt));
        }
        if (h1) {
            sc[d] = __fadd_rn(sc[d], f2_y(wv));
            wt[d] = __fadd_rn(wt[d], f2_y(wgt));
        }
    };
    // Particles [from, to) for those of the three faces that they can reach,
    // in pairs as they lie in memory (the planes hold an even number).
    auto row = [&](auto useU, auto useV, auto useW, int from, int to) {
        for (int t = from & ~1; t < to; t += 2) {
            const bool first = t >= from, second = t + 1 < to;
            auto pair = [&](const float *plane) { return reinterpret_cast<const F2 *>(plane + t); };
            const F2 px = *pair(p.px), py = *pair(p.py), pz = *pair(p.pz);
            auto square = [&](F2 g, F2 q, F2 no) {   // (g - (q - off))^2
                const F2 d = k2.sub(g, k2.add(q, no));
                return k2.mul(d, d);
            };
            const F2 xx1 = square(pgx, k2.add(px, nh), nox), yy1 = square(pgy, k2.add(py, nh), noy),
                     zz1 = square(pgz, k2.add(pz, nh), noz);
            if (useU.value) take(0, k2.add(k2.add(square(pgx, px, nox), yy1), zz1), pair(p.vx), first, second);
            if (useV.value) take(1, k2.add(k2.add(xx1, square(pgy, py, noy)), zz1), pair(p.vy), first, second);
            if (useW.value) take(2, k2.add(k2.add(xx1, yy1), square(pgz, pz, noz)), pair(p.vz), first, second);
        }
    };
    using Yes = std::true_type;
    using No = std::false_type;
    for (int cz = cz0; cz <= cz1; cz++)
        for (int cy = cy0; cy <= cy1; cy++) {
            // the row's particles: cells up to fi can reach the u face (those in
            // pb..pu), rows up to fj the v face, up to fk the w face
            const long long base = cells.idx(0, cy, cz);
            const int pb = cellStart[base + cx0], pe = cellStart[base + cx1 + 1];
            if (pb == pe) continue;
            const int pu = isU ? cellStart[base + min(fi, c.I - 1) + 1] : pb;
            const bool rowV = isV && cy <= fj, rowW = isW && cz <= fk;
            if (rowV && rowW) {
                row(Yes{}, Yes{}, Yes{}, pb, pu);
                row(No{}, Yes{}, Yes{}, pu, pe);
            } else if (rowV) {
                row(Yes{}, Yes{}, No{}, pb, pu);
                row(No{}, Yes{}, No{}, pu, pe);
            } else if (rowW) {
                row(Yes{}, No{}, Yes{}, pb, pu);
                row(No{}, No{}, Yes{}, pu, pe);
            } else {
                row(Yes{}, No{}, No{}, pb, pu);
            }
        }
    const float eps = 1e-6f;
    auto put = [&](int d, float *G, uint8_t *valid, long long l) {
        const bool ok = wt[d] > eps;
        G[l] = ok ? __fdiv_rn(sc[d], wt[d]) : sc[d];
        valid[l] = ok ? 1 : 0;
    };
    if (isU) put(0, U, vu, (long long)fi + (long long)(c.I + 1) * (fj + (long long)c.J * fk));
    if (isV) put(1, V, vv, (long long)fi + (long long)c.I * (fj + (long long)(c.J + 1) * fk));
    if (isW) put(2, W, vw, (long long)fi + (long long)c.I * (fj + (long long)c.J * fk));
}

// ------------------------------------------------------------ extrapolation
// Layered BFS of GridUtils::extrapolateGrid (gridutils.cpp:32-228) done in
// place, one launch per layer.  A layer fills every unknown face with a known
// neighbour, known meaning valid input or filled by an earlier layer; the grid
// border is fixed and counts as known in a mean, but fills nothing.  The known
// faces are bits, 32 along x to a word (rows padded to whole words), so a
// layer is a few word operations per 32 faces, and only words with faces to
// fill are looked at face by face, a lane per face.  A status byte and a
// thread per face and layer took 31 us a layer at 128^3, nearly all of it on
// faces with nothing to do (stage "constrain", 7 layers and two passes: 233 ->
// 138 us at 128^3, 335 -> 172 us at 256 x 128 x 128).
__device__ __forceinline__ void face_word(const FaceBits &b, long long t, int &dir, int &wx, int &j, int &k) {
    dir = t < b.base[1] ? 0 : (t < b.base[2] ? 1 : 2);
    unflatten(t - b.base[dir], b.wpr[dir], b.nj[dir], wx, j, k);
}
__global__ void __launch_bounds__(TPB) k_extrap_init(FaceBits b, const uint8_t *vu, const uint8_t *vv, const uint8_t *vw,
                                                     unsigned *known) {
    pdl_begin();
    const int lane = threadIdx.x & 31;
    const long long first = ((long long)blockIdx.x * (TPB / 32) + (threadIdx.x >> 5)) * 8;   // eight words a warp
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const long long t = first + q;
        if (t >= b.words) break;
        int dir, wx, j, k;
        face_word(b, t, dir, wx, j, k);
        const int i = wx * 32 + lane, ni = b.ni[dir];
        const uint8_t *valid = dir == 0 ? vu : (dir == 1 ? vv : vw);
        const bool inner = i >= 1 && i <= ni - 2 && j >= 1 && j <= b.nj[dir] - 2 && k >= 1 && k <= b.nk[dir] - 2;
        const unsigned m =
            __ballot_sync(0xffffffffu, inner && valid[(long long)i + (long long)ni * (j + (long long)b.nj[dir] * k)]);
        if (lane == 0) known[t] = m;
    }
}

// WORDS of a row a CTA and layer
template <int WORDS>
__global__ void __launch_bounds__(TPB) k_extrap_layer(FaceBits b, const unsigned *known, unsigned *next, float *u, float *v,
                                                      float *w) {
    pdl_wait();
    pdl_trigger();
    // The CTA's first threads form a word each and list those with faces to
    // fill (their places and neighbour words); then its warps take turns.
    __shared__ unsigned list[WORDS][7];
    __shared__ int4 place[WORDS];
    __shared__ int listed;
    if (threadIdx.x == 0) listed = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long t = (long long)blockIdx.x * WORDS + threadIdx.x;
    int dir = 0, wx = 0, j = 0, k = 0;
    unsigned own = 0, xm = 0, xp = 0, jm = 0, jp = 0, km = 0, kp = 0, fill = 0;
    if (threadIdx.x < WORDS && t < b.words) {
        face_word(b, t, dir, wx, j, k);
        const int wpr = b.wpr[dir], nj = b.nj[dir], ni = b.ni[dir];
        const long long plane = (long long)wpr * nj;
        if (j >= 1 && k >= 1 && j <= nj - 2 && k <= b.nk[dir] - 2) {
            own = known[t];
            xm = own << 1 | (wx > 0 ? known[t - 1] >> 31 : 0u);
            xp = own >> 1 | (wx + 1 < wpr ? known[t + 1] << 31 : 0u);
            jm = known[t - wpr];
            jp = known[t + wpr];
            km = known[t - plane];
            kp = known[t + plane];
            // faces 1 .. ni - 2 of the row
            const int lo = max(1 - wx * 32, 0), hi = min(ni - 2 - wx * 32, 31);
            const unsigned inner = hi < lo ? 0u : (0xffffffffu >> (31 - hi)) & (0xffffffffu << lo);
            fill = inner & ~own & (xm | xp | jm | jp | km | kp);
            // border faces count in the means
            if (wx == 0) xm |= 2u;
            if (ni - 2 - wx * 32 >= 0 && ni - 2 - wx * 32 < 32) xp |= 1u << (ni - 2 - wx * 32);
            if (j == 1) jm = 0xffffffffu;
            if (j == nj - 2) jp = 0xffffffffu;
            if (k == 1) km = 0xffffffffu;
            if (k == b.nk[dir] - 2) kp = 0xffffffffu;
        }
        next[t] = own | fill;
        if (fill) {
            const int at = atomicAdd(&listed, 1);
            const unsigned v[7] = {fill, xp, xm, jp, jm, kp, km};
#pragma unroll
            for (int q = 0; q < 7; q++) list[at][q] = v[q];
            place[at] = make_int4(dir, wx * 32, j, k);
        }
    }
    __syncthreads();
    for (int at = threadIdx.x >> 5; at < listed; at += TPB / 32) {
        if (!(list[at][0] >> lane & 1u)) continue;
        const int4 p = place[at];
        const int d = p.x, x = p.y, jj = p.z, kk = p.w;
        const unsigned *nb = &list[at][1];
        const long long sy = b.ni[d], sz = sy * b.nj[d], l = (long long)(x + lane) + sy * jj + sz * kk;
        float *G = d == 0 ? u : (d == 1 ? v : w);
        const long long off[6] = {1, -1, sy, -sy, sz, -sz};
        float sum = 0.0f;
        int count = 0;
#pragma unroll
        for (int q = 0; q < 6; q++)
            if (nb[q] >> lane & 1u) {
                sum = __fadd_rn(sum, G[l + off[q]]);
                count++;
            }
        G[l] = __fdiv_rn(sum, (float)count);
    }
}

// -------------------------------------------------- save + body force, constrain
// `ex` (optional, one byte per face over u, v, w): faces an inflow source
// constrains, which the body force skips (fluidsimulation.cpp:3450-3489).
__global__ void k_save_force(long long nu, long long nv, long long nw, float *u, float *v, float *w, float *su,
                             float *sv, float *sw, float fx, float fy, float fz, int ax, int ay, int az,
                             const uint8_t *ex) {
    pdl_begin();
    long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool skip = ex && f < nu + nv + nw && ex[f];
    if (f < nu) {
        float x = u[f]; su[f] = x; if (ax && !skip) u[f] = __fadd_rn(x, fx);
    } else if (f < nu + nv) {
        long long l = f - nu; float x = v[l]; sv[l] = x; if (ay && !skip) v[l] = __fadd_rn(x, fy);
    } else if (f < nu + nv + nw) {
        long long l = f - nu - nv; float x = w[l]; sw[l] = x; if (az && !skip) w[l] = __fadd_rn(x, fz);
    }
}

// Faces with zero fluid weight take the solid velocity, which is zero for
// static solids; partly solid faces blend it with their own velocity by the
// mean friction of the solid objects closest to their four corners
// (src/engine/fluidsimulation.cpp:3785-3846, 3884-3950).  The domain walls
// have no friction: without friction arrays those faces stay as they are.
__global__ void k_constrain(long long nu, long long nv, long long nw, float *u, float *v, float *w, float *su,
                            float *sv, float *sw, const float *wu, const float *wv, const float *ww, const float *fu,
                            const float *fv, const float *fw) {
    pdl_begin();
    long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    float *G, *S;
    const float *W, *F;
    long long l;
    if (f < nu) { G = u; S = su; W = wu; F = fu; l = f; }
    else if (f < nu + nv) { G = v; S = sv; W = wv; F = fv; l = f - nu; }
    else if (f < nu + nv + nw) { G = w; S = sw; W = ww; F = fw; l = f - nu - nv; }
    else return;
    const float wt = W[l];
    if (wt == 0.0f) {   // inside the solid: the solid's velocity (zero for static solids)
        G[l] = 0.0f;
        if (S) S[l] = 0.0f;
    } else if (wt < 1.0f && F) {   // part solid: f usolid + (1 - f) u, usolid = 0
        const float fr = F[l], keep = __fsub_rn(1.0f, fr), us = __fmul_rn(fr, 0.0f);
        G[l] = __fadd_rn(us, __fmul_rn(keep, G[l]));
        if (S) S[l] = __fadd_rn(us, __fmul_rn(keep, S[l]));
    }
}

// ---------------------------------------------------------- particle update
// Trilinear weights of Interpolation::trilinearInterpolate (interpolation.cpp:
// 61-70) with vertex order {000,100,010,001,101,011,110,111}, in FP32.
__device__ __forceinline__ float trilerp_f(const float q[8], float x, float y, float z) {
    float x1 = 1.0f - x, y1 = 1.0f - y, z1 = 1.0f - z;
    float r = q[0] * (x1 * y1 * z1);
    r = __fmaf_rn(q[1], x * y1 * z1, r);
    r = __fmaf_rn(q[2], x1 * y * z1, r);
    r = __fmaf_rn(q[3], x1 * y1 * z, r);
    r = __fmaf_rn(q[4], x * y1 * z, r);
    r = __fmaf_rn(q[5], x1 * y * z, r);
    r = __fmaf_rn(q[6], x * y * z1, r);
    r = __fmaf_rn(q[7], x * y * z, r);
    return r;
}

__device__ __forceinline__ float grid_at(const float *G, int ni, int nj, int nk, int a, int b, int cc) {
    bool in = a >= 0 && b >= 0 && cc >= 0 && a < ni && b < nj && cc < nk;
    return in ? __ldg(&G[(long long)a + (long long)ni * ((long long)b + (long long)nj * cc)]) : 0.0f;
}

// The eight corners of cell (i, j, k) in trilerp_f's order, 0 outside the grid:
// one test and one address for all where the cell lies inside (grids hold fewer
// than 2^31 entries).
__device__ __forceinline__ void corners(const float *G, int ni, int nj, int nk, int i, int j, int k, float q[8]) {
    if ((unsigned)i < (unsigned)(ni - 1) && (unsigned)j < (unsigned)(nj - 1) && (unsigned)k < (unsigned)(nk - 1)) {
        const float *g0 = G + (i + ni * (j + nj * k)), *g1 = g0 + ni * nj;
        q[0] = __ldg(g0); q[1] = __ldg(g0 + 1); q[2] = __ldg(g0 + ni); q[6] = __ldg(g0 + ni + 1);
        q[3] = __ldg(g1); q[4] = __ldg(g1 + 1); q[5] = __ldg(g1 + ni); q[7] = __ldg(g1 + ni + 1);
    } else {
        q[0] = grid_at(G, ni, nj, nk, i, j, k);         q[1] = grid_at(G, ni, nj, nk, i + 1, j, k);
        q[2] = grid_at(G, ni, nj, nk, i, j + 1, k);     q[3] = grid_at(G, ni, nj, nk, i, j, k + 1);
        q[4] = grid_at(G, ni, nj, nk, i + 1, j, k + 1); q[5] = grid_at(G, ni, nj, nk, i, j + 1, k + 1);
        q[6] = grid_at(G, ni, nj, nk, i + 1, j + 1, k); q[7] = grid_at(G, ni, nj, nk, i + 1, j + 1, k + 1);
    }
}

// MAC velocity components at a point, as MACVelocityField::_interpolateLinearU/V/W
// (macvelocityfield.cpp:519-613) but in FP32.  The cell coordinate is
// x*(1/dx) - 1/2 in one fused step, which is exact for power-of-two dx and
// within half an ulp otherwise; the reference evaluates the same in FP64.
// With two fields (H), both at the same point.
template <bool TWO>
__device__ __forceinline__ float2 interp_face(const float *G, const float *H, int ni, int nj, int nk, int dir, F3 p,
                                              float invdxf) {
    float fx = dir == 0 ? __fmul_rn(p.x, invdxf) : __fmaf_rn(p.x, invdxf, -0.5f);
    float fy = dir == 1 ? __fmul_rn(p.y, invdxf) : __fmaf_rn(p.y, invdxf, -0.5f);
    float fz = dir == 2 ? __fmul_rn(p.z, invdxf) : __fmaf_rn(p.z, invdxf, -0.5f);
    float gi = floorf(fx), gj = floorf(fy), gk = floorf(fz);
    int i = (int)gi, j = (int)gj, k = (int)gk;
    float q[8], r[8];
    corners(G, ni, nj, nk, i, j, k, q);
    if (TWO) corners(H, ni, nj, nk, i, j, k, r);
    return make_float2(trilerp_f(q, fx - gi, fy - gj, fz - gk), TWO ? trilerp_f(r, fx - gi, fy - gj, fz - gk) : 0.0f);
}

// isPositionInGrid (grid3d.h:133-135): x >= 0 && x < I dx, with the upper
// bound pre-rounded so the float compare equals the reference's FP64 one.
__device__ __forceinline__ bool in_grid(const StepConsts &c, F3 p) {
    return p.x >= 0.0f && p.y >= 0.0f && p.z >= 0.0f && p.x <= c.gxmax && p.y <= c.gymax && p.z <= c.gzmax;
}

__device__ __forceinline__ F3 eval_vel(const StepConsts &c, const float *u, const float *v, const float *w, F3 p) {
    if (!in_grid(c, p)) return f3(0.0f, 0.0f, 0.0f);
    return f3(interp_face<false>(u, u, c.I + 1, c.J, c.K, 0, p, c.invdxf).x,
              interp_face<false>(v, v, c.I, c.J + 1, c.K, 1, p, c.invdxf).x,
              interp_face<false>(w, w, c.I, c.J, c.K + 1, 2, p, c.invdxf).x);
}
// and in the field (su, sv, sw) at the same point
__device__ __forceinline__ F3 eval_vel2(const StepConsts &c, const float *u, const float *v, const float *w, const float *su,
                                        const float *sv, const float *sw, F3 p, F3 &other) {
    other = f3(0.0f, 0.0f, 0.0f);
    if (!in_grid(c, p)) return other;
    const float2 a = interp_face<true>(u, su, c.I + 1, c.J, c.K, 0, p, c.invdxf),
                 b = interp_face<true>(v, sv, c.I, c.J + 1, c.K, 1, p, c.invdxf),
                 d = interp_face<true>(w, sw, c.I, c.J, c.K + 1, 2, p, c.invdxf);
    other = f3(a.y, b.y, d.y);
    return f3(a.x, b.x, d.x);
}

// Nodal solid SDF at a point (Interpolation::trilinearInterpolate(vec3, dx,
// grid), interpolation.cpp:72-113).  FP32 weights; when the value is within
// rounding of zero the sign is settled by the reference's FP64 evaluation.
__device__ float solid_at(const StepConsts &c, const float *S, F3 p) {
    int i = exact_floor(p.x, c.invdx, c.invdxf), j = exact_floor(p.y, c.invdx, c.invdxf),
        k = exact_floor(p.z, c.invdx, c.invdxf);
    float dxl = __fsub_rn(p.x, c.nodePos[max(i, 0)]), dyl = __fsub_rn(p.y, c.nodePos[max(j, 0)]),
          dzl = __fsub_rn(p.z, c.nodePos[max(k, 0)]);
    int ni = c.I + 1, nj = c.J + 1, nk = c.K + 1;
    float q[8];
    corners(S, ni, nj, nk, i, j, k, q);
    float v = trilerp_f(q, dxl * c.invdxf, dyl * c.invdxf, dzl * c.invdxf);
    float mag = 0.0f;
#pragma unroll
    for (int t = 0; t < 8; t++) mag += fabsf(q[t]);
    if (fabsf(v) > 1e-6f * mag) return v;
    double qd[8];
#pragma unroll
    for (int t = 0; t < 8; t++) qd[t] = q[t];
    double ix = (double)dxl * c.invdx, iy = (double)dyl * c.invdx, iz = (double)dzl * c.invdx;
    return (float)(qd[0] * (1 - ix) * (1 - iy) * (1 - iz) + qd[1] * ix * (1 - iy) * (1 - iz) +
                   qd[2] * (1 - ix) * iy * (1 - iz) + qd[3] * (1 - ix) * (1 - iy) * iz + qd[4] * ix * (1 - iy) * iz +
                   qd[5] * (1 - ix) * iy * iz + qd[6] * ix * iy * (1 - iz) + qd[7] * ix * iy * iz);
}

// Interpolation::trilinearInterpolateGradient (interpolation.cpp:197-258), FP32
__device__ F3 solid_grad(const StepConsts &c, const float *S, F3 p) {
    int i = exact_floor(p.x, c.invdx, c.invdxf), j = exact_floor(p.y, c.invdx, c.invdxf),
        k = exact_floor(p.z, c.invdx, c.invdxf);
    float ix = __fsub_rn(p.x, c.nodePos[max(i, 0)]) * c.invdxf;
    float iy = __fsub_rn(p.y, c.nodePos[max(j, 0)]) * c.invdxf;
    float iz = __fsub_rn(p.z, c.nodePos[max(k, 0)]) * c.invdxf;
    int ni = c.I + 1, nj = c.J + 1, nk = c.K + 1;
    float v000 = grid_at(S, ni, nj, nk, i, j, k), v100 = grid_at(S, ni, nj, nk, i + 1, j, k);
    float v010 = grid_at(S, ni, nj, nk, i, j + 1, k), v001 = grid_at(S, ni, nj, nk, i, j, k + 1);
    float v101 = grid_at(S, ni, nj, nk, i + 1, j, k + 1), v011 = grid_at(S, ni, nj, nk, i, j + 1, k + 1);
    float v110 = grid_at(S, ni, nj, nk, i + 1, j + 1, k), v111 = grid_at(S, ni, nj, nk, i + 1, j + 1, k + 1);
    auto bil = [](float a, float b, float cc, float d, float x, float y) {
        float l1 = (1 - x) * a + x * b;
        float l2 = (1 - x) * cc + x * d;
        return (1 - y) * l1 + y * l2;
    };
    float gx = bil(v100 - v000, v110 - v010, v101 - v001, v111 - v011, iy, iz);
    float gy = bil(v010 - v000, v110 - v100, v011 - v001, v111 - v101, ix, iz);
    float gz = bil(v001 - v000, v101 - v100, v011 - v010, v111 - v110, ix, iy);
    return f3(gx, gy, gz);
}

__device__ __forceinline__ bool box_inside(const StepConsts &c, F3 p) {
    return p.x >= c.bposx && p.y >= c.bposy && p.z >= c.bposz && (double)p.x < (double)c.bposx + c.bw &&
           (double)p.y < (double)c.bposy + c.bh && (double)p.z < (double)c.bposz + c.bd;
}
// AABB::getNearestPointInsideAABB (aabb.cpp:497-518), eps 1e-6
__device__ __forceinline__ F3 box_nearest(const StepConsts &c, F3 p) {
    if (box_inside(c, p)) return p;
    float mxx = __fadd_rn(c.bposx, (float)c.bw);
    float mxy = __fadd_rn(c.bposy, (float)c.bh);
    float mxz = __fadd_rn(c.bposz, (float)c.bd);
    p.x = fmaxf(p.x, c.bposx); p.y = fmaxf(p.y, c.bposy); p.z = fmaxf(p.z, c.bposz);
    p.x = (float)fmin((double)p.x, (double)mxx - 1e-6);
    p.y = (float)fmin((double)p.y, (double)mxy - 1e-6);
    p.z = (float)fmin((double)p.z, (double)mxz - 1e-6);
    return p;
}

__device__ __forceinline__ bool near_solid(const StepConsts &c, const uint8_t *ns, F3 p) {
    int i = exact_floor(p.x, c.invNearCell, c.invNearCellf), j = exact_floor(p.y, c.invNearCell, c.invNearCellf),
        k = exact_floor(p.z, c.invNearCell, c.invNearCellf);
    if (i < 0 || j < 0 || k < 0 || i >= c.nsi || j >= c.nsj || k >= c.nsk) return false;
    return ns[(long long)i + (long long)c.nsi * ((long long)j + (long long)c.nsj * k)] != 0;
}

// FluidSimulation::_resolveCollision (src/engine/fluidsimulation.cpp:4221-4296)
__device__ F3 resolve_collision(const StepConsts &c, const float *S, const uint8_t *ns, F3 oldp, F3 newp) {
    int gi = exact_floor(newp.x, c.invdx, c.invdxf), gj = exact_floor(newp.y, c.invdx, c.invdxf),
        gk = exact_floor(newp.z, c.invdx, c.invdxf);
    if (!(gi >= 0 && gj >= 0 && gk >= 0 && gi < c.I && gj < c.J && gk < c.K)) newp = box_nearest(c, newp);
    if (!near_solid(c, ns, oldp) && !near_solid(c, ns, newp)) return newp;
    const float eps = 1e-6f;
    const float stepDist = __fmul_rn(0.5f, (float)c.dx);
    float travel = len3(sub(newp, oldp));
    if (travel < eps) return newp;
    int nsteps = (int)ceilf(__fdiv_rn(travel, stepDist));
    F3 dir = normalize3(sub(newp, oldp));
    F3 last = oldp, cur = oldp;
    bool found = false;
    float cphi = 0.0f;
    for (int s = 0; s < nsteps; s++) {
        if (s == nsteps - 1) cur = newp;
        else cur = add(oldp, mul(__fmul_rn((float)(s + 1), stepDist), dir));
        float ph = solid_at(c, S, cur);
        if (ph < 0.0f || !box_inside(c, cur)) { cphi = ph; found = true; break; }
        last = cur;
    }
    if (!found) return newp;
    F3 res;
    const float maxDist = (float)(c.cfl * c.dx);
    F3 g = solid_grad(c, S, cur);
    if (len3(g) > eps) {
        g = normalize3(g);
        res = sub(cur, mul((float)((double)cphi - (double)0.1f * c.dx), g));
        float rphi = solid_at(c, S, res);
        float rd = len3(sub(res, cur));
        if (rphi < 0 || rd > maxDist) res = last;
    } else {
        res = last;
    }
    if (!box_inside(c, res)) {
        F3 orig = res;
        res = box_nearest(c, res);
        float rphi = solid_at(c, S, res);
        float rd = len3(sub(res, orig));
        if (rphi < 0.0f || rd > maxDist) res = last;
    }
    return res;
}

// What depends on the time step alone, worked out once: a thread that takes an
// FP64 division of its own for each keeps the FP64 unit busy for most of the
// kernel.
struct AdvectSteps {
    float half, threeQuarters, ninth;   // of the time step
    float invSpeedStep;
    double speedStep;
};

// Fused particle update: PIC/FLIP velocity (fluidsimulation.cpp:4082-4092),
// Ralston RK3 (4191-4198), collision (4221-4296), then the removal tests and
// the new cell key for the next binning.  Bound by instructions and the latency
// of the 104 scattered corner reads a particle: the stage takes 278 us at 128^3 (4.1M
// particles), 817 at 256x128x128 (14.0M).  A bounds test and a 64-bit address per
// corner took 614, 1705; FP64 divisions of the time step by each thread 328, 1112.
__global__ void __launch_bounds__(TPB) k_advect(ParticleSoA p, int n, StepConsts c, const float *u, const float *v,
                                                const float *w, const float *su, const float *sv, const float *sw,
                                                const float *S, const uint8_t *ns, float picRatio, float flipRatio,
                                                const AdvectSteps k, unsigned int *keys, unsigned int *hist,
                                                const InflowConstraint ic) {
    pdl_begin();
    __shared__ unsigned int shist[8];
    if (threadIdx.x < 8) shist[threadIdx.x] = 0;
    __syncthreads();
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) {
        F3 p0 = f3(p.px[t], p.py[t], p.pz[t]);
        F3 v0 = f3(p.vx[t], p.vy[t], p.vz[t]);
        F3 vold;
        F3 vpic = eval_vel2(c, u, v, w, su, sv, sw, p0, vold);
        F3 vflip = sub(add(v0, vpic), vold);
        F3 vn = add(mul(picRatio, vpic), mul(flipRatio, vflip));
        if (ic.count > 0) {
            // _constrainMarkerParticleVelocities (fluidsimulation.cpp:4109-4170):
            // a particle in a cell of the source where the source's level set,
            // read at the particle's position in the level set's own frame (the
            // reference passes the position without the level set's offset), is
            // not positive takes the source's velocity; later sources win
            const int ci = exact_floor(p0.x, c.invdx, c.invdxf), cj = exact_floor(p0.y, c.invdx, c.invdxf),
                      ck = exact_floor(p0.z, c.invdx, c.invdxf);
            const Dims d{c.I, c.J, c.K};
            const unsigned bits = d.in(ci, cj, ck) ? ic.cellBits[d.idx(ci, cj, ck)] : 0u;
            for (int q = 0; q < ic.count; q++)
                if ((bits >> q & 1u) && !(source_phi(ic.g[q], p0.x, p0.y, p0.z) > 0.0f))
                    vn = f3(ic.vx[q], ic.vy[q], ic.vz[q]);
        }
        F3 k1 = vpic;
        F3 k2 = eval_vel(c, u, v, w, add(p0, mul(k.half, k1)));
        F3 k3 = eval_vel(c, u, v, w, add(p0, mul(k.threeQuarters, k2)));
        F3 sum = add(add(mul(2.0f, k1), mul(3.0f, k2)), mul(4.0f, k3));
        F3 p1 = add(p0, mul(k.ninth, sum));
        p1 = resolve_collision(c, S, ns, p0, p1);
        p.px[t] = p1.x; p.py[t] = p1.y; p.pz[t] = p1.z;
        p.vx[t] = vn.x; p.vy[t] = vn.y; p.vz[t] = vn.z;
        float speed = len3(vn);
        // floor(speed / step) as the reference's FP64 division gives it
        float qf = __fmul_rn(speed, k.invSpeedStep);
        float fl = floorf(qf);
        int bin = (qf - fl > 1e-3f && qf - fl < 1.0f - 1e-3f) ? (int)fminf(fl, 5.0f)
                                                               : (int)fmin(floor((double)speed / k.speedStep), 5.0);
        if (speed != speed) bin = 5;
        atomicAdd(&shist[bin], 1u);
        unsigned int key;
        if (solid_at(c, S, p1) < 0.0f) {
            key = KEY_SOLID;
        } else {
            int i = exact_floor(p1.x, c.invdx, c.invdxf), j = exact_floor(p1.y, c.invdx, c.invdxf),
                k = exact_floor(p1.z, c.invdx, c.invdxf);
            Dims d{c.I, c.J, c.K};
            key = d.in(i, j, k) ? (unsigned int)d.idx(i, j, k) : KEY_SOLID;
        }
        keys[t] = key;
    }
    __syncthreads();
    if (threadIdx.x < 6 && shist[threadIdx.x]) atomicAdd(&hist[threadIdx.x], shist[threadIdx.x]);
}

// _getMarkerParticleSpeedLimit (fluidsimulation.cpp:4298-4322), one thread
__global__ void k_speed_limit(const unsigned int *hist, int n, int bins, double step, double maxPct, int maxAbs,
                              float *maxSpeedSq) {
    pdl_begin();
    int maxRemoval = (int)fmin((double)(int)((double)n * maxPct), (double)maxAbs);
    double maxspeed = bins * step;
    int cur = 0;
    for (int i = bins - 1; i > 0; i--) {
        if (cur + (int)hist[i] > maxRemoval) break;
        cur += (int)hist[i];
        maxspeed = i * step;
    }
    float ms = (float)maxspeed;
    *maxSpeedSq = __fmul_rn(ms, ms);
}

__global__ void k_mark_fast(ParticleSoA p, int n, const float *maxSpeedSq, unsigned int *keys) {
    pdl_begin();
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    unsigned int k = keys[t];
    if (k & KEY_SOLID) return;
    F3 v = f3(p.vx[t], p.vy[t], p.vz[t]);
    if (dot3(v, v) > *maxSpeedSq) keys[t] = k | KEY_FAST;
}

}  // namespace

// ------------------------------------------------------------------ launchers
void launch_keys_from_positions(const ParticleSoA &p, int n, const StepConsts &c, unsigned int *keys, cudaStream_t s) {
    if (n > 0) launch_next(k_keys, div_up(n, TPB), TPB, s, p, n, c, keys);
}
void launch_bin_count(const unsigned int *keys, int n, int *cellCount, cudaStream_t s) {
    if (n > 0) launch_next(k_bin_count, div_up(n, TPB), TPB, s, keys, n, cellCount);
}
int scan_scratch_ints(int ncells) { return (int)div_up(ncells + 1, SCAN_TILE) + 2; }
void launch_scan_cells(const int *count, int ncells, int *start, int *scratch, int *total, cudaStream_t s) {
    int ntiles = (int)div_up(ncells, SCAN_TILE);
    launch_next(k_scan_tiles, ntiles, SCAN_T, s, count, ncells, start, scratch);
    launch_next(k_scan_sums, 1, SCAN_T, s, scratch, ntiles, total);
    launch_next(k_scan_add, div_up(ncells + 1, TPB), TPB, s, start, ncells, scratch, total);
}
void launch_bin_scatter(const unsigned int *keys, int n, const int *cellStart, int *cursor, int *slots, cudaStream_t s) {
    if (n > 0) launch_next(k_bin_scatter, div_up(n, TPB), TPB, s, keys, n, cellStart, cursor, slots);
}
void launch_cell_sort_select(const int *cellStart, int ncells, int *slots, const unsigned int *ids,
                             const unsigned int *keys, int maxPerCell, int *survivorCount, cudaStream_t s) {
    launch_next(k_cell_sort_select, div_up(ncells, TPB), TPB, s, cellStart, ncells, slots, ids, keys, maxPerCell, survivorCount);
}
void launch_gather_particles(const ParticleSoA &src, ParticleSoA dst, int n, const int *cellStart, const int *slots,
                             const unsigned int *keys, const int *newStart, int ncells, unsigned int *maxSpeedSqBits,
                             cudaStream_t s) {
    if (n <= 0) return;
    launch_next(k_gather, std::min(div_up(n, TPB), 152u * 16u), TPB, s, src, dst, cellStart, slots, keys, newStart, ncells,
                maxSpeedSqBits);
}
void launch_liquid_sdf(const ParticleSoA &p, const int *cellStart, const StepConsts &c, const uint8_t *solidCC,
                       float *phi, int threads, cudaStream_t s) {
    FLIP_COUNT(1);
    // CTAs of half the knob's threads: a CTA lasts as long as its slowest warp
    // (the kernel alone at 128^3: 223 us with CTAs of 256 threads, 299 with 512, 370
    // with 1024)
    const int cta = threads / 2;
    auto *kernel = cta == 128 ? k_liquid_sdf<128> : cta == 512 ? k_liquid_sdf<512> : k_liquid_sdf<256>;
    kernel<<<div_up((long long)c.I * c.J * c.K, cta), cta, 0, s>>>(p, cellStart, c, solidCC, phi);
}
void launch_p2g(const ParticleSoA &p, const int *cellStart, const StepConsts &c, float *u, float *v,
                float *w, uint8_t *vu, uint8_t *vv, uint8_t *vw, cudaStream_t s) {
    launch_next(k_p2g, div_up((long long)(c.I + 1) * (c.J + 1) * (c.K + 1), P2G_TPB), P2G_TPB, s, p, cellStart, c, u, v, w, vu, vv, vw,
                                                                                                  PairOps{});
}
FaceBits face_bits(int I, int J, int K) {
    FaceBits b;
    long long at = 0;
    for (int d = 0; d < 3; d++) {
        b.ni[d] = I + (d == 0);
        b.nj[d] = J + (d == 1);
        b.nk[d] = K + (d == 2);
        b.wpr[d] = (b.ni[d] + 31) / 32;
        b.base[d] = at;
        at += (long long)b.wpr[d] * b.nj[d] * b.nk[d];
    }
    b.words = at;
    return b;
}
void launch_extrapolate(const StepConsts &c, float *u, float *v, float *w, const uint8_t *vu, const uint8_t *vv,
                        const uint8_t *vw, unsigned *known, int layers, cudaStream_t s) {
    const FaceBits b = face_bits(c.I, c.J, c.K);
    launch_next(k_extrap_init, div_up(b.words, TPB / 4), TPB, s, b, vu, vv, vw, known);
    // Few words: more CTAs, so that their warps share the faces to fill (32^3,
    // 7 layers: 34 us against 48); many: fewer (128^3: 129 us against 187;
    // 64^3, 29000 words: 49 against 53).
    const bool few = b.words < 16384;
    for (int l = 0; l < layers; l++)
        launch_after(true, few ? k_extrap_layer<32> : k_extrap_layer<128>, div_up(b.words, few ? 32 : 128), TPB, 0, s, b,
                     known + (l & 1) * b.words, known + (l & 1 ? 0 : b.words), u, v, w);
}
void launch_save_and_force(const StepConsts &c, float *u, float *v, float *w, float *su, float *sv, float *sw,
                           float fx, float fy, float fz, bool ax, bool ay, bool az, const uint8_t *ex,
                           cudaStream_t s) {
    long long nu = (long long)(c.I + 1) * c.J * c.K, nv = (long long)c.I * (c.J + 1) * c.K,
              nw = (long long)c.I * c.J * (c.K + 1);
    launch_next(k_save_force, div_up(nu + nv + nw, TPB), TPB, s, nu, nv, nw, u, v, w, su, sv, sw, fx, fy, fz, ax, ay, az, ex);
}
void launch_constrain(const StepConsts &c, float *u, float *v, float *w, float *su, float *sv, float *sw,
                      const float *wu, const float *wv, const float *ww, const float *fu, const float *fv,
                      const float *fw, cudaStream_t s) {
    long long nu = (long long)(c.I + 1) * c.J * c.K, nv = (long long)c.I * (c.J + 1) * c.K,
              nw = (long long)c.I * c.J * (c.K + 1);
    launch_next(k_constrain, div_up(nu + nv + nw, TPB), TPB, s, nu, nv, nw, u, v, w, su, sv, sw, wu, wv, ww, fu, fv, fw);
}
void launch_advect(ParticleSoA p, int n, const StepConsts &c, const float *u, const float *v, const float *w,
                   const float *su, const float *sv, const float *sw, const float *solidPhi,
                   const uint8_t *nearSolid, float picRatio, float flipRatio, double dt, unsigned int *keys,
                   unsigned int *speedHist, double speedStep, const InflowConstraint &ic, cudaStream_t s) {
    if (n <= 0) return;
    const AdvectSteps k{(float)(0.5 * dt), (float)(0.75 * dt), (float)(dt / 9.0f), (float)(1.0 / speedStep), speedStep};
    launch_next(k_advect, div_up(n, TPB), TPB, s, p, n, c, u, v, w, su, sv, sw, solidPhi, nearSolid, picRatio, flipRatio, k,
                keys, speedHist, ic);
}
void launch_speed_limit(const unsigned int *hist, int n, int bins, double speedStep, double maxPct, int maxAbs,
                        float *maxSpeedSq, cudaStream_t s) {
    launch_next(k_speed_limit, 1, 1, s, hist, n, bins, speedStep, maxPct, maxAbs, maxSpeedSq);
}
void launch_mark_fast(const ParticleSoA &p, int n, const float *maxSpeedSq, unsigned int *keys, cudaStream_t s) {
    if (n > 0) launch_next(k_mark_fast, div_up(n, TPB), TPB, s, p, n, maxSpeedSq, keys);
}

}  // namespace flip
