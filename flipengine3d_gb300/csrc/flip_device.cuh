// Launch interface of the FLIP step kernels (host side of the CUDA code).
#pragma once
#include <algorithm>
#include <cstdint>
#include <string>
#include <cuda_runtime.h>

#include "flip_common.cuh"

namespace flip {

// Particles, structure of arrays, kept sorted by cell (ascending id inside a
// cell).  `id` is the particle's rank in the reference's load order, which
// the reference preserves through every removal.
struct ParticleSoA {
    float *px, *py, *pz, *vx, *vy, *vz;
    unsigned int *id;
};

struct StepConsts {
    int I, J, K;
    double dx, invdx;
    float invdxf;
    float dxf;
    float gxmax, gymax, gzmax;   // largest float coordinate with (double)x < I dx (J dx, K dx)
    double radius;               // liquid SDF / P2G particle radius, 0.5*sqrt(3)*dx
    double cfl;
    int maxPerCell;
    // the reference's blocks of 10 cells, for its particle lists: float edge, 1 / edge
    float blockdxf, invBlockf;
    float centre[10];   // a cell's centre in its block's frame, by its place there
    // liquid level set: particle radius; 3 dx, the smallest float no less than dx / 2, -dx / 2, 0.005 dx
    float radiusf, sdfMax, sdfHalf, sdfNeg, sdfEps;
    double invBlock;
    // near-solid coarse grid
    int nsi, nsj, nsk;
    double nearCell, invNearCell;
    float invNearCellf;
    // collision boundary AABB (domain inset, then the solid buffer)
    float bposx, bposy, bposz;
    double bw, bh, bd;
    // position tables (device): node n at (float)((double)(float)n * dx);
    // 10-cell block n at (float)((double)(float)n * 10 dx) and at
    // (float)((double)(float)n * (double)(float)(10 dx)), index n + 1
    const float *nodePos;
    const float *blockPos;
    const float *blockPosF;
};

// Pairs of floats in one 64-bit register: each operation rounds each half as the
// scalar one does.  Sums and products are fused multiply-adds that are exact up
// to that one rounding (a 1 + b, a b - 0).  A product's zero comes as a kernel
// argument: the compiler folds a visible one away, and is then free to contract
// the product with the sum after it, which rounds once where the two round twice
// (it did in particle to grid).  A sum has nothing to contract with, so its 1 is
// plain.
using F2 = unsigned long long;
__host__ __device__ constexpr F2 f2_bits(unsigned x, unsigned y) { return x | (F2)y << 32; }
__device__ __forceinline__ F2 f2(float x, float y) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float f2_x(F2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float f2_y(F2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
struct PairOps {
    static constexpr F2 ONE = f2_bits(0x3f800000u, 0x3f800000u), MINUS = f2_bits(0xbf800000u, 0xbf800000u);
    F2 zero = f2_bits(0x80000000u, 0x80000000u);   // (-0, -0)
    __device__ F2 mul(F2 a, F2 b) const { return f2_fma(a, b, zero); }
    __device__ F2 add(F2 a, F2 b) const { return f2_fma(a, ONE, b); }
    __device__ F2 sub(F2 a, F2 b) const { return f2_fma(b, MINUS, a); }
    __device__ F2 neg(F2 a) const { return f2_fma(a, MINUS, f2_bits(0x80000000u, 0x80000000u)); }   // exact
};

// Programmatic dependent launch: a kernel launched with launch_after may start
// while the kernel before it in the stream still runs; what it reads or
// overwrites of that kernel's lies after pdl_wait().  Called after pdl_wait,
// pdl_trigger lets the kernel after it start the same way, which can then
// rely on everything up to the kernel before this one even ahead of its own
// wait.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... P, class... Q>
inline void launch_after(bool overlap, void (*k)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                         Q... args) {
    FLIP_COUNT(1);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

// For kernels that begin with pdl_begin: launched early where they are small, and
// a launch's latency is most of what they take (32^3 frames: 1195 us without, 1142
// with; 48^3: 1982, 1870).  Larger ones would take the place of CTAs of the kernel
// before them (early launches of all sizes cost 64^3 frames 2.4%, 128^3 frames
// 1.5%), and the two instructions alone cost them (k_save_force at 128^3: 27 us
// against 18), so they do without.
__host__ __device__ __forceinline__ bool launched_early(unsigned grid, unsigned block) {
    return (long long)grid * block <= 1 << 17;
}
__device__ __forceinline__ void pdl_begin() {
    if (!launched_early(gridDim.x, blockDim.x)) return;
    pdl_wait();
    pdl_trigger();
}
template <class... P, class... Q>
inline void launch_next(void (*k)(P...), unsigned grid, unsigned block, cudaStream_t s, Q... args) {
    launch_after(launched_early(grid, block), k, grid, block, 0, s, args...);
}

// -- seeding from fluid meshes (flip_seed.cu); mask: one 8-bit sub-cell
// mask per cell, four cells to a word; owner: 8 I J K words, all ones
void launch_mask_particles(const ParticleSoA &p, int n, const StepConsts &c, unsigned int *mask, cudaStream_t s);
// meshPhi: the mesh's level set, sampled at p minus its first node's position
void launch_seed_candidates(const StepConsts &c, const int *cells, long long ncells, const SourceGridView &meshPhi,
                            const float *solidPhi, double jitter, bool jitterSurface, unsigned long long seed,
                            const unsigned int *mask, float4 *cand, unsigned int *owner, int *keep, cudaStream_t s);
void launch_seed_scatter(const StepConsts &c, long long ncand, const float4 *cand, const int *keep, const int *rank,
                         const ParticleSoA &p, int n0, unsigned int id0, float vx, float vy, float vz,
                         unsigned int *mask, cudaStream_t s);

// -- binning (flip_kernels.cu)
void launch_keys_from_positions(const ParticleSoA &p, int n, const StepConsts &c, unsigned int *keys, cudaStream_t s);
void launch_bin_count(const unsigned int *keys, int n, int *cellCount, cudaStream_t s);
void launch_scan_cells(const int *count, int ncells, int *start, int *blockSums, int *total, cudaStream_t s);
int scan_scratch_ints(int ncells);
void launch_bin_scatter(const unsigned int *keys, int n, const int *cellStart, int *cursor, int *slots, cudaStream_t s);
void launch_cell_sort_select(const int *cellStart, int ncells, int *slots, const unsigned int *ids,
                             const unsigned int *keys, int maxPerCell, int *survivorCount, cudaStream_t s);
void launch_gather_particles(const ParticleSoA &src, ParticleSoA dst, int n, const int *cellStart, const int *slots,
                             const unsigned int *keys, const int *newStart, int ncells, unsigned int *maxSpeedSqBits,
                             cudaStream_t s);

// -- grid stages
// threads: the CTA size, 256, 512 (default) or 1024
void launch_liquid_sdf(const ParticleSoA &p, const int *cellStart, const StepConsts &c, const uint8_t *solidCC,
                       float *phi, int threads, cudaStream_t s);
void launch_p2g(const ParticleSoA &p, const int *cellStart, const StepConsts &c, float *u, float *v,
                float *w, uint8_t *vu, uint8_t *vv, uint8_t *vw, cudaStream_t s);
// The faces as bits: per direction the extents, words per row of 32 faces
// along x, and the first word.
struct FaceBits {
    int ni[3], nj[3], nk[3], wpr[3];
    long long base[3], words;
};
FaceBits face_bits(int I, int J, int K);
// known: scratch of 2 * face_bits().words words
void launch_extrapolate(const StepConsts &c, float *u, float *v, float *w, const uint8_t *vu, const uint8_t *vv,
                        const uint8_t *vw, unsigned *known, int layers, cudaStream_t s);
// The force-field grid on the device (flip_forces.cu): faces of an
// ni x nj x nk grid of cell size dx, and the body force it reads outside them
struct ForceFieldView {
    const float *u, *v, *w;
    int ni, nj, nk;
    double dx;
    float gx, gy, gz;
};
void launch_force_field(const StepConsts &c, float *u, float *v, float *w, const ForceFieldView &f, double dt,
                        const uint8_t *ex, cudaStream_t s);
void launch_save_and_force(const StepConsts &c, float *u, float *v, float *w, float *su, float *sv, float *sw,
                           float fx, float fy, float fz, bool ax, bool ay, bool az, const uint8_t *ex,
                           cudaStream_t s);
void launch_constrain(const StepConsts &c, float *u, float *v, float *w, float *su, float *sv, float *sw,
                      const float *wu, const float *wv, const float *ww, const float *fu, const float *fv,
                      const float *fw, cudaStream_t s);

// -- particle update: PIC/FLIP, RK3, collision, removal tests, new keys
void launch_advect(ParticleSoA p, int n, const StepConsts &c, const float *u, const float *v, const float *w,
                   const float *su, const float *sv, const float *sw, const float *solidPhi,
                   const uint8_t *nearSolid, float picRatio, float flipRatio, double dt, unsigned int *keys,
                   unsigned int *speedHist, double speedStep, const InflowConstraint &ic, cudaStream_t s);

// -- mesh fluid sources (flip_sources.cu)
// Faces (u, v, w, one byte each) that enabled inflow sources constraining the
// fluid velocity keep out of the body force: P2G-valid faces where a
// source's level set, read at the face's position in its own frame, is
// negative (fluidsimulation.cpp:3372-3440).
void launch_inflow_faces(const StepConsts &c, const InflowConstraint &ic, const uint8_t *vu, const uint8_t *vv,
                         const uint8_t *vw, uint8_t *ex, cudaStream_t s);
// Outflow (fluidsimulation.cpp:4608-4650): particles in the source's cells
// (or outside them, inversed) where its level set at p - offset is negative
// (non-negative, inversed) are flagged for removal in keys.
void launch_outflow_mark(const ParticleSoA &p, int n, const StepConsts &c, const uint8_t *cellMask, int inversed,
                         const SourceGridView &g, unsigned int *keys, cudaStream_t s);
void launch_speed_limit(const unsigned int *hist, int n, int bins, double speedStep, double maxPct, int maxAbs,
                        float *maxSpeedSq, cudaStream_t s);
void launch_mark_fast(const ParticleSoA &p, int n, const float *maxSpeedSq, unsigned int *keys, cudaStream_t s);

// -- pressure projection (flip_pcg.cu); dense cell-grid vectors, cells
// outside the system hold zeros
// Sweep layout: the vectors of the MIC(0) sweeps (factor rows, right-hand
// side, result) are stored step-major.  The interior pencils along i are cut
// into tiles of SWEEP_WA x SWEEP_WB along axes (a, b) = (j, k), or (k, j) when
// `swap` is set (the orientation is chosen per solve).  Pencil (A, B) of a tile
// holds cell i at forward step tf = i - 1 + A + B: a pencil runs one step
// behind each of its lower neighbours.  A tile is worked by warps of SWEEP_VA x
// SWEEP_VB pencils, one per lane: warp wa + 2 wb, lane la + 8 lb holds pencil
// (8 wa + la, 4 wb + lb), and its entry at step tf is
// (tile * T + tf) * SWEEP_NP + warp * 32 + lane.
// T = I - 2 + (SWEEP_WA - 1) + (SWEEP_WB - 1) up to a multiple of SWEEP_CH, so that
// a chunk of SWEEP_CH steps is one contiguous block in either sweep direction.
// In the chunks that a solve passes over (its items), the factor rows, the rows of
// the matrix and the right-hand side are zero at entries without a cell of the
// system.  Elsewhere the matrix is zero, the factor rows are not read, and z and s
// hold finite values that an earlier solve left, which only ever meet a zero.
constexpr int SWEEP_WA = 16, SWEEP_WB = 8, SWEEP_NP = SWEEP_WA * SWEEP_WB, SWEEP_CH = 8;
constexpr int SWEEP_VA = 8, SWEEP_VB = 4;
constexpr int SWEEP_CA = 2, SWEEP_CB = 4;   // tiles of a thread-block cluster along a and b
struct SweepLayout {
    int nta, ntb, T;   // tiles along a and b, steps per tile
    int swap;          // 0: (a, b) = (j, k); 1: (a, b) = (k, j)
    int EA, EB;        // grid extents along a and b
};
inline SweepLayout sweep_layout(int I, int J, int K, int swap = 0) {
    SweepLayout g;
    g.swap = swap;
    g.EA = swap ? K : J;
    g.EB = swap ? J : K;
    g.nta = (g.EA - 2 + SWEEP_WA - 1) / SWEEP_WA;
    g.ntb = (g.EB - 2 + SWEEP_WB - 1) / SWEEP_WB;
    g.T = ((I - 2) + (SWEEP_WA - 1) + (SWEEP_WB - 1) + SWEEP_CH - 1) / SWEEP_CH * SWEEP_CH;
    return g;
}
// entries of either orientation: the arrays are allocated for the larger
inline long long sweep_layout_size(int I, int J, int K) {
    long long best = 0;
    for (int sw = 0; sw < 2; sw++) {
        SweepLayout g = sweep_layout(I, J, K, sw);
        best = std::max(best, (long long)g.nta * g.ntb * g.T * SWEEP_NP);
    }
    return best;
}
// chunks of either orientation: the most items a solve can have
inline long long sweep_items_max(int I, int J, int K) { return sweep_layout_size(I, J, K) / (SWEEP_CH * SWEEP_NP); }
// entry of interior cell (i, j, k)
__host__ __device__ __forceinline__ long long sweep_index(const SweepLayout &g, int i, int j, int k) {
    const int aa = (g.swap ? k : j) - 1, bb = (g.swap ? j : k) - 1;
    const int A = aa % SWEEP_WA, B = bb % SWEEP_WB;
    const int tile = aa / SWEEP_WA + g.nta * (bb / SWEEP_WB);
    const int warp = A / SWEEP_VA + SWEEP_WA / SWEEP_VA * (B / SWEEP_VB), lane = A % SWEEP_VA + SWEEP_VA * (B % SWEEP_VB);
    return ((long long)tile * g.T + (i - 1 + A + B)) * SWEEP_NP + warp * 32 + lane;
}

// Device-side control of the PCG loop: the convergence test runs on the
// device, so the host enqueues iterations in batches and reads this once per
// batch; every kernel of an iteration returns at once when done is set.
struct PcgCtl {
    int done;      // converged
    int iters;     // iterations to convergence
    int it;        // index of the iteration being run
    unsigned int ticket[4];   // CTAs done, of [1] the first z.r and [3] the true residual
    double resid;  // last residual norm tested
    int batches;     // batches run by the device-side loop
    int maxBatches;  // its limit (maximum iterations / PCG_BATCH)
};
constexpr int PCG_BATCH = 8;   // iterations of a captured batch

struct PressureBuffers {
    uint8_t *fluid;        // interior cell with phi < 0 (a row of the system)
    int *items, *nItems;   // the solve's chunks of the sweep layout, and their number
    double4_32a *Ad;           // rows {diag, to +x, to +y, to +z}, FP64
    double *b;             // right-hand side (negative divergence)
    double *pivotInv;      // reciprocals of the MIC(0) pivots, FP64
    float4 *L;             // {invdiag, Lx, Ly, Lz} for the FP32 sweeps, sweep layout
    // The loop's vectors, in the sweep layout (nsl entries each; A, z, s and s2
    // have a step of zeros after them, planes of A too).  Values kept
    // to ~48 bits are pairs of floats, leading part h and remainder l.
    float *A;              // rows as pairs: 8 planes, h of {diag, +x, +y, +z}, then l (also the factor's pivot weights)
    float *xh, *xl;        // solution
    float *rh, *rl;        // residual (rh: the forward sweep's right-hand side)
    float *qh, *ql;        // A s
    float *z;              // preconditioned residual
    float *s, *s2;         // search direction, double-buffered: an iteration reads one and writes the other
    SweepLayout sl;        // the orientation of the current solve
    long long nsl;         // entries allocated for the sweep layout
    bool stale = true;     // z, s, s2 may hold values that are not finite
    double *partials;      // per-block partial sums of s.q, then of z.r (PCG_MAX_PARTIALS each; deterministic)
    double *scal;          // [1]=the first z.r [2]=|b|inf [3], [7]=rho of even and odd iterations [6]=tol |b|inf
    unsigned long long *rmaxBits;  // [0] |r|inf of the recurrence, [1] of b - A x, as double bits
    PcgCtl *ctl;
    // PCG_BATCH iterations captured as a CUDA graph, replayed per batch;
    // [1] also records the sweep timing events
    cudaGraphExec_t batchGraph[2][2] = {};   // [timed][orientation]
    long long batchKernels[2][2] = {};
    bool noGraphs = false;   // the stream cannot be captured: launch eagerly
    // untimed solves: the batches inside a device-side loop (a conditional
    // WHILE node), one launch and one host wait per solve
    cudaGraphExec_t loopGraph[2] = {};   // [orientation]
    long long loopKernels[2] = {};       // kernels per pass of the loop body
    bool noLoopGraph = false;            // the loop could not be built: batches from the host
    int *levelRange;       // [0]=min(i+j+k) [1]=max(i+j+k) [2]=system size [3..6]=min/max j, min/max k
    unsigned int *factorTicket;
    float *pressure;       // float copy of x for the velocity update
    int nPartials;
};
struct PressureArgs {
    const float *phi, *wu, *wv, *ww;
    float *u, *v, *w;
    uint8_t *vu, *vv, *vw;
    double dt, tol, accTol;
    int maxIter;
    float *dumpPressure;   // host, optional
    double *dumpRhs;       // host, optional
    struct SweepTiming *sweepTiming;   // optional: event-timed sweep launches
    int sweepOrientation;  // -1: chosen per solve; 0: lanes along j; 1: lanes along k
};
// Device time of the preconditioner sweeps, summed over launches.
struct SweepTiming {
    cudaEvent_t ev[2 * (PCG_BATCH + 1)];   // a pair per sweep pair of a batch, plus the first
    double ms;
    long long launches;     // sweep kernels (forward and backward count one each)
    long long cellSweeps;   // sum over launches of the system rows swept
};
struct PressureMail {      // pinned host scalars
    int levelRange[8];
    double bmax, rho, ptol;
    PcgCtl ctl;
    int sweepErr;
    int maxBatches;
};
struct PressureResult {
    int iterations;
    double residual;
    bool applied;
    int cells;
};

// Bounded device waits: poll rounds of at most ~250 ns each before a wait
// gives up and raises the error flag (about a second).
constexpr unsigned int DEFAULT_SPIN_LIMIT = 1u << 22;

// Pipelined wavefront sweeps (flip_wavefront.cu)
struct SweepState {
    int2 *range;             // per tile [first, last] step holding a system cell
    unsigned long long *xchg;  // tile edge exchange words {epoch, value}
    long long xchgWords;       // words allocated for xchg
    unsigned int *ticket;    // [0] forward tile tickets, [1] the sweep pair's epoch, [2] backward tile tickets
    int *err;                // set when a bounded wait gave up
    unsigned int epoch;      // host count of the epochs issued (wrap guard)
    unsigned int spinLimit = 0;   // poll rounds of the factor's, sweeps' and viscous solver's waits (0: DEFAULT_SPIN_LIMIT)
    int stall = 0;           // fault injection: the sweeps' edge waits and the viscous solver's sums await an epoch never published
};
int sweep_tiles_max(int I, int J, int K);           // tiles of the larger orientation
long long sweep_exchange_words(int I, int J, int K);   // for the larger orientation
void launch_sweep_ranges(const StepConsts &c, const SweepLayout &g, const uint8_t *fluid, SweepState &sw,
                         cudaStream_t s);
// Before each sweep pair, by one thread of a kernel that runs before it:
// tile tickets from zero for both sweeps and a fresh epoch for each (the
// forward sweep publishes under ticket[1], the backward under ticket[1]+1).
// Kept on the device so that a captured sequence of pairs replays with new
// epochs.
__device__ __forceinline__ void sweep_prep(unsigned int *ticket) {
    ticket[0] = 0u;
    ticket[2] = 0u;
    ticket[1] += 2u;
}
// z = M^-1 r with the MIC(0) factor L: forward then backward sweep
// The launches return at once when *skip is set (a converged solve).
// `prepped`: a kernel ahead of them on the stream already ran sweep_prep;
// `overlap`: and at least one more lies between, so the forward sweep may set
// up while that one runs.
void launch_sweeps(const StepConsts &c, const SweepLayout &g, const float4 *L, const float *rf, float *z,
                   SweepState &sw, const int *skip, cudaStream_t s, bool prepped = false, bool overlap = false);
void sweep_epoch_guard(const StepConsts &c, SweepState &sw, long long upcoming, cudaStream_t s);

void mic0_factor(const StepConsts &c, const uint8_t *fluid, const double4_32a *Ad, double *E, double *W0, double *W1,
                 double *W2, unsigned int *ticket, int *err, unsigned int spinLimit, cudaStream_t s);
void mic0_inverse_pivots(const uint8_t *fluid, long long n, double *E, cudaStream_t s);
void launch_pivot_functions(int n, const double *d, const float *off, double *recip, double *root, cudaStream_t s);
// The reduction grid of the PCG row kernels: one CTA per `cellsPerCta` grid
// cells (a tuning knob, default 4096), at most PCG_MAX_PARTIALS.
constexpr int PCG_MAX_PARTIALS = 152 * 8;
int pressure_partials_for(int I, int J, int K, int cellsPerCta = 4096);
// Steps of the solve: its items, its vectors' layout, one product (flip_pcg.cu)
void launch_items(const StepConsts &c, PressureBuffers &pb, SweepState &sw, cudaStream_t s);
void launch_layout(const StepConsts &c, const PressureBuffers &pb, SweepState &sw, cudaStream_t s);
void launch_spmv(const PressureBuffers &pb, const float *sIn, float *sOut, SweepState &sw, cudaStream_t s);
// PressureSolver::solve (pressuresolver.cpp:44-76) on the device.  Returns
// FLIP_OK (velocities updated, or nothing to solve), FLIP_E_SOLVER_NOCONV
// (left unchanged), FLIP_E_DEVICE_TIMEOUT or FLIP_E_CUDA.
int pressure_project(const StepConsts &c, const PressureArgs &a, PressureBuffers &pb, SweepState &sw,
                     PressureMail *mail, cudaStream_t s, PressureResult *res, std::string *errMsg);

}  // namespace flip

namespace flip {
// -- viscosity (flip_viscosity.cu)
struct ViscosityBuffers {
    uint8_t *fluidFace, *valid, *valid2, *inSys;   // per face; per node (two); per face
    float *node[7], *vol[7];                       // per control-volume grid: corner values, fractions
    double *coefs;                                 // per row: six factors, diagonal, 1 / diagonal
    double *x, *r, *p, *q, *scal;                  // per row: CG vectors; scalars (8)
    double2 *zp;                                   // per face {z, the last p}
    int *list, *blockRows;                         // the system's faces; counts per block of faces and their scan
    unsigned long long *slots;                     // the CTAs' shares of the CG's sums
};
struct ViscosityResult {
    long long rows;
    int iterations;
    double residual;   // |r|inf / |b|inf
};
void viscosity_buffer_sizes(int I, int J, int K, long long *nf, long long *nn, long long *ncorner,
                            long long vol[7], long long *rowBlocks, long long *slotWords);
int viscosity_apply(const StepConsts &c, const ViscosityBuffers &vb, const float *liquidPhi, const float *solidPhi,
                    float *u, float *v, float *w, double visc, double dt, unsigned spinLimit, bool stall,
                    ViscosityResult *res, cudaStream_t s);

// -- surface reconstruction (flip_mesh.cu)
// The frame of the mesher's one compute chunk: the subdivided grid, its
// blocks of 10^3 nodes, the chunk's nodes and offset, and the particle radii.
struct MeshRow {           // a row of cells around a node's: its offset, and the least squared distance to it
    float least;
    short y, z;
};
struct MeshFrame {
    int I, J, K;
    double dx, invdx, subdx, invsub;
    float dxf, invdxf, subdxf, invsubf;
    double blockdx, invBlock;      // 10 subdx, occupancy pass
    float invBlockf;
    float blockdxF;                // (float)(10 subdx), the count pass's block size
    double invBlockF;
    float invBlockFf;
    int nbI, nbJ, nbK;             // blocks of the subdivided grid
    int ni, nj, nk;                // chunk nodes
    int cbI, cbJ, cbK;             // chunk blocks
    float offx, offy, offz;        // chunk offset
    float r, sr, maxd;             // radius, search radius, initial distance
    // how far along an axis a particle can reach a node, how far it can make one inside, and the squared
    // distance below which its search box surely holds the node
    float reach, signReach, near2, slack;
    // where node a of the chunk lies along an axis with chunk offset off, in cells
    __device__ float cellAt(float off, int a) const { return (off + (float)a * subdxf) * invdxf; }
    const MeshRow *rows;           // rows to search, nearest first
    int nrows;
    int wpr, wpc;                  // words of 32 nodes a row of the chunk, of 32 cells a row of the grid
    float nodePos[10];             // a node's place in its block's frame
    const float *blockPos[3];      // origins of the blocks' frames along each axis
    float bbx, bby, bbz, bhx, bhy, bhz;   // the chunk's expanded box: from bb (inside) to bh (outside)
    int solidMode;                 // 0 interpolated, 1 subdivision 2 at offset 0, 2 same grid
    float scalef, invscalef;
};
struct MeshJob {
    StepConsts c;
    ParticleSoA p;
    int n;
    const int *cellStart;
    const float *solidPhi;
    int subdivisions;
    double radius;                 // marker particle radius x marker particle scale
    double smoothValue;
    int smoothIterations;
};
// Device buffers of the mesher, grown on demand; the mesh is verts[cur]
// (nverts xyz floats) and tris (ntris vertex triples).
struct MeshBuffers {
    long long bytes = 0;
    uint8_t *occ = nullptr, *active = nullptr, *cube = nullptr;
    unsigned *inside = nullptr, *occupied = nullptr;   // nodes inside; cells with particles, cells near those: bits
    int *vstart = nullptr, *totals = nullptr;
    int2 *tiles = nullptr, *adj = nullptr, *adjStart = nullptr;
    int *adjCursor = nullptr, *adjList = nullptr, *tris = nullptr;
    float *verts[2] = {nullptr, nullptr};
    long long occCap = 0, activeCap = 0, cubeCap = 0, insideCap = 0, occupiedCap = 0, vstartCap = 0, totalsCap = 0,
              tilesCap = 0, adjCap = 0, adjStartCap = 0, adjCursorCap = 0, adjListCap = 0, trisCap = 0;
    long long vertsCap[2] = {0, 0};
    int nverts = 0, ntris = 0, cur = 0;
};
// Mesh the particles of `job` into mb (synchronises the stream twice).
int mesh_surface(const MeshJob &job, MeshBuffers &mb, cudaStream_t s);
void mesh_release(MeshBuffers &mb);
int record_error(int code, const std::string &msg);   // sets flip_last_error()

// Packed xyz positions/velocities (either may be null) of the n particles, whose
// ids are dense (0..n-1), in the reference's order.
void launch_readback_order(const ParticleSoA &p, int n, float *pos, float *vel, cudaStream_t s);
// Ids to their ranks 0..n-1: flags and rank hold idSpace+1 ints, scratch
// scan_scratch_ints(idSpace).
void launch_compact_ids(const ParticleSoA &p, int n, int idSpace, int *flags, int *rank, int *scratch, int *total,
                        cudaStream_t s);
}  // namespace flip
