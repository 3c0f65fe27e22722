// Variational pressure projection for GB300 (sm_103a).
//
// The system is the reference's (pressuresolver.cpp:580-808): a 7-point
// matrix over the interior cells with phi < 0, ghost-fluid diagonal terms at
// air neighbours, face weights from the solid level set.  Its rows are built
// in FP64 exactly as the reference builds them and kept as {diag, +x, +y, +z}.
// Preconditioner: the reference's MIC(0) (pcgsolver.h:70-185, tau 0.97,
// pivot floor 0.25) restated for 7-point rows; the factorisation runs as an
// i+j+k wavefront in FP64 and the two triangular sweeps as the pipelined
// FP32 wavefront of flip_wavefront.cu.  CG (pcgsolver.h:248-302): the
// Laplacian apply, the solution and the residual are double-float (exact
// float pairs, ~48 bits, on the FP32 pipe; this GPU's FP64 rate is ~1/64 of
// FP32) and the dot products are summed in double-float per thread and FP64
// across threads, so the recurrence tracks b - A x to far below the
// tolerance; the FP32 parts (preconditioner, search direction) only steer
// the iteration.  Every 25
// iterations, and whenever the recurrence reports convergence, the residual
// is recomputed as b - A x (iterative refinement), and convergence is
// decided on it, with the reference's test |r|inf <= tol * |b|inf.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>

#include "../../include/flip3d.h"
#include "flip_device.cuh"

namespace flip {

namespace {

constexpr int TPB = 256;
constexpr int RBLOCKS = 152 * 8;   // grid of the reduction kernels: 8 CTAs of 256 threads per SM (full occupancy)

__device__ __forceinline__ bool sys_cell(const StepConsts &c, const float *phi, int i, int j, int k) {
    if (i < 1 || j < 1 || k < 1 || i > c.I - 2 || j > c.J - 2 || k > c.K - 2) return false;
    return phi[(long long)i + (long long)c.I * ((long long)j + (long long)c.J * k)] < 0.0f;
}

// The rows' flags, and the extent of their levels i + j + k, their number and
// their extent in j and k (for the sweep tile orientation).  A CTA reduces
// over FLAG_CELLS cells before its seven atomics: one set per warp of 32
// cells was bound by them, all on the same addresses (107 us at 128^3).
constexpr int FLAG_CELLS = 4096;
__global__ void __launch_bounds__(TPB) k_flags(StepConsts c, const float *phi, uint8_t *fluid, int *levelRange) {
    pdl_begin();
    __shared__ int sh[7][TPB / 32];
    const long long base = (long long)blockIdx.x * FLAG_CELLS, n = (long long)c.I * c.J * c.K;
    int v[7] = {0x7fffffff, -1, 0, 0x7fffffff, -1, 0x7fffffff, -1};
#pragma unroll 4
    for (int q = threadIdx.x; q < FLAG_CELLS; q += TPB) {
        const long long t = base + q;
        if (t >= n) break;
        int i, j, k;
        unflatten(t, c.I, c.J, i, j, k);
        const bool f = sys_cell(c, phi, i, j, k);
        fluid[t] = f ? 1 : 0;
        if (!f) continue;
        v[0] = min(v[0], i + j + k);
        v[1] = max(v[1], i + j + k);
        v[2]++;
        v[3] = min(v[3], j);
        v[4] = max(v[4], j);
        v[5] = min(v[5], k);
        v[6] = max(v[6], k);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto reduce = [&](int q, int x) {
        return q == 2 ? __reduce_add_sync(0xffffffffu, x)
                      : (q == 0 || q == 3 || q == 5 ? __reduce_min_sync(0xffffffffu, x) : __reduce_max_sync(0xffffffffu, x));
    };
#pragma unroll
    for (int q = 0; q < 7; q++) {
        const int x = reduce(q, v[q]);
        if (lane == 0) sh[q][warp] = x;
    }
    __syncthreads();
    if (warp != 0) return;
#pragma unroll
    for (int q = 0; q < 7; q++) {
        const int idle = q == 2 ? 0 : (q == 0 || q == 3 || q == 5 ? 0x7fffffff : -1);
        const int x = reduce(q, lane < TPB / 32 ? sh[q][lane] : idle);
        if (lane != 0 || x == idle) continue;
        if (q == 2) atomicAdd(&levelRange[q], x);
        else if (q == 0 || q == 3 || q == 5) atomicMin(&levelRange[q], x);
        else atomicMax(&levelRange[q], x);
    }
}

// One matrix row in FP64, as _calculateMatrixCoefficientsThread builds it
// (pressuresolver.cpp:723-808).  Off-diagonal entries exist only towards
// neighbours that are rows of the system; a liquid neighbour outside the
// interior contributes neither an entry nor a ghost-fluid term (the
// reference's key map drops it).
__device__ double4_32a row_coeffs(const StepConsts &c, const float *phi, const float *wu, const float *wv,
                              const float *ww, double mf, int i, int j, int k) {
    Dims du{c.I + 1, c.J, c.K}, dv{c.I, c.J + 1, c.K}, dw{c.I, c.J, c.K + 1}, dc{c.I, c.J, c.K};
    double vR = wu[du.idx(i + 1, j, k)], vL = wu[du.idx(i, j, k)];
    double vT = wv[dv.idx(i, j + 1, k)], vB = wv[dv.idx(i, j, k)];
    double vF = ww[dw.idx(i, j, k + 1)], vK = ww[dw.idx(i, j, k)];
    double pc = phi[dc.idx(i, j, k)];
    double diag = (vR + vL + vT + vB + vF + vK) * mf;
    double xp = 0.0, yp = 0.0, zp = 0.0;
    const double maxtheta = 25.0, eps = 1e-9;
    const int nb[6][3] = {{i + 1, j, k}, {i - 1, j, k}, {i, j + 1, k}, {i, j - 1, k}, {i, j, k + 1}, {i, j, k - 1}};
    const double vol[6] = {vR, vL, vT, vB, vF, vK};
#pragma unroll
    for (int q = 0; q < 6; q++) {
        double pn = phi[dc.idx(nb[q][0], nb[q][1], nb[q][2])];
        if (pn < 0.0) {
            if (sys_cell(c, phi, nb[q][0], nb[q][1], nb[q][2])) {
                if (q == 0) xp = -vol[q] * mf;
                else if (q == 2) yp = -vol[q] * mf;
                else if (q == 4) zp = -vol[q] * mf;
            }
        } else {
            double theta = pn / (pc + eps);
            theta = fmax(-maxtheta, fmin(theta, maxtheta));
            diag -= vol[q] * mf * theta;
        }
    }
    return make_double4_32a(fmax(diag, 0.0), xp, yp, zp);
}

// Max of non-negative values over the block, then one atomic per block.
// With nanAsInf a NaN reads as +inf (a residual norm that never passes for
// converged); otherwise NaNs are ignored, as fmax ignores them.
__device__ __forceinline__ void block_max_to(double v, unsigned long long *out, bool nanAsInf = true) {
    __shared__ long long sh[32];
    if (v != v) v = nanAsInf ? __longlong_as_double(0x7ff0000000000000ll) : 0.0;
    // as integers, which order non-negative doubles the same way and spare the
    // scarce FP64
    long long m = __double_as_longlong(v);
    if (__any_sync(0xffffffffu, m > 0))
        for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) sh[warp] = m;
    __syncthreads();
    if (warp == 0) {
        m = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0;
        for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0 && m > 0) atomicMax(out, (unsigned long long)m);
    }
}

constexpr long long NOT_YET = -1LL;   // the bits of a pivot's reciprocal before it is found: a NaN that no operation returns

// RHS (pressuresolver.cpp:580-669; the domain walls do not move) and the rows.
__global__ void k_build(StepConsts c, const float *phi, const float *wu, const float *wv, const float *ww,
                        const float *u, const float *v, const float *w, double mf, PressureBuffers pb) {
    pdl_begin();
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    Dims d{c.I, c.J, c.K};
    double bmag = 0.0;
    if (t < d.size()) {
        pb.pivotInv[t] = __longlong_as_double(NOT_YET);
        if (!pb.fluid[t]) {
            pb.b[t] = 0.0;   // the row itself is not read
        } else {
            int i, j, k;
        unflatten(t, c.I, c.J, i, j, k);
            Dims du{c.I + 1, c.J, c.K}, dv{c.I, c.J + 1, c.K}, dw{c.I, c.J, c.K + 1};
            double vR = wu[du.idx(i + 1, j, k)], vL = wu[du.idx(i, j, k)];
            double vT = wv[dv.idx(i, j + 1, k)], vB = wv[dv.idx(i, j, k)];
            double vF = ww[dw.idx(i, j, k + 1)], vK = ww[dw.idx(i, j, k)];
            const double factor = c.invdx;
            double div = 0.0;
            div += -factor * vR * (double)u[du.idx(i + 1, j, k)];
            div += factor * vL * (double)u[du.idx(i, j, k)];
            div += -factor * vT * (double)v[dv.idx(i, j + 1, k)];
            div += factor * vB * (double)v[dv.idx(i, j, k)];
            div += -factor * vF * (double)w[dw.idx(i, j, k + 1)];
            div += factor * vK * (double)w[dw.idx(i, j, k)];
            pb.b[t] = div;
            bmag = fabs(div);
            pb.Ad[t] = row_coeffs(c, phi, wu, wv, ww, mf, i, j, k);
        }
    }
    block_max_to(bmag, (unsigned long long *)pb.scal + 2, false);
}

// MIC(0) pivots in FP64.  For 7-point rows the column-oriented elimination of
// factorModifiedIncompleteColesky0 reduces to:
//   d_c = A_cc - sum over earlier neighbours q of
//         L_cq^2 + 0.97 L_cq (sum of q's other later-neighbour entries L_mq),
//   L_mq = A_mq / sqrt(pivot_q); a pivot below 0.25 A_cc falls back to A_cc.
// Regrouped per earlier neighbour q:
//   L_cq^2 + 0.97 L_cq miss_q = (a_q^2 + 0.97 a_q (m1_q + m2_q)) / pivot_q,
// with a_q the coupling of q to c and m1_q, m2_q q's other later-neighbour
// couplings (0 off the system).  The bracket depends on the rows only; this
// pass computes it for every cell and earlier neighbour, so a level needs
// three multiply-subtracts and a reciprocal.  The FP64 results differ from the
// elimination's order in the last bits; the factor is used rounded to FP32.
__global__ void k_mic0_weights(StepConsts c, const uint8_t *fluid, const double4_32a *Ad, double *W0, double *W1,
                               double *W2) {
    pdl_begin();
    const long long n = (long long)c.I * c.J * c.K;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    double w[3] = {0.0, 0.0, 0.0};
    if (fluid[t]) {   // interior by construction
        const long long sy = c.I, sz = (long long)c.I * c.J;
        const long long back[3] = {t - sz, t - sy, t - 1};
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const long long kk = back[q];
            if (!fluid[kk]) continue;
            const double4_32a ak = Ad[kk];
            if (ak.x == 0.0) continue;
            const double a = q == 0 ? ak.w : (q == 1 ? ak.z : ak.y);
            const double o1 = q == 2 ? ak.z : ak.y, o2 = q == 0 ? ak.z : ak.w;
            const double m1 = fluid[q == 2 ? kk + sy : kk + 1] ? o1 : 0.0;
            const double m2 = fluid[q == 0 ? kk + sy : kk + sz] ? o2 : 0.0;
            w[q] = a * a + 0.97 * a * (m1 + m2);
        }
    }
    W0[t] = w[0];
    W1[t] = w[1];
    W2[t] = w[2];
}

// FP64 to FP32 and back with integer operations, which are far cheaper than the
// FP64 unit's conversions: for magnitudes well inside the range of FP32 (in_fp32),
// rounded towards zero.
__device__ __forceinline__ bool in_fp32(double d) {
    return (unsigned)((__double2hiint(d) >> 20 & 0x7ff) - (1023 - 120)) <= 240u;
}
__device__ __forceinline__ float narrow(double d) {
    const int hi = __double2hiint(d);
    return __int_as_float((hi & 0x80000000) | ((hi & 0x7fffffff) - (896 << 20)) << 3 | (int)((unsigned)__double2loint(d) >> 29));
}
__device__ __forceinline__ double widen(float f) {
    const int b = __float_as_int(f);
    return __hiloint2double((b & 0x80000000) | (((b & 0x7fffffff) >> 3) + (896 << 20)), b << 29);
}
__device__ __forceinline__ float narrow_or_0(double d) { return in_fp32(d) ? narrow(d) : 0.0f; }
// 1 / d from a guess g: one step of the third-order hyperpower iteration (Schulz's
// iteration with the next term of the geometric series), e (1 + r + r^2) with
// r = 1 - d e, which leaves r^3 < 2^-57; the division for a guess with fewer than
// 19 bits.
__device__ __forceinline__ double reciprocal(double d, float g) {
    const double e = widen(g), r = __fma_rn(-d, e, 1.0);
    if ((__double2hiint(r) >> 20 & 0x7ff) >= 1023 - 19) return 1.0 / d;
    return __fma_rn(e, __fma_rn(r, r, r), e);
}
__device__ __forceinline__ float guess_reciprocal(float f) {
    float g;
    asm("rcp.approx.f32 %0, %1;" : "=f"(g) : "f"(f));
    return g;
}
// sqrt(e), e the reciprocal of a pivot: the inverse pivot.  The same way: a
// guess from the FP32 unit, then two steps of Newton's iteration for x^2 = e with
// the slope 1 / 2x kept from the guess.
__device__ __forceinline__ double inverse_pivot(double e) {
    if (!(e > 0.0) || !in_fp32(e)) return sqrt(e);
    const float f = narrow(e);
    float g;
    asm("rsqrt.approx.f32 %0, %1;" : "=f"(g) : "f"(f));
    const double y = widen(0.5f * g);
    double x = widen(f * g);
    x = __fma_rn(__fma_rn(-x, x, e), y, x);
    return __fma_rn(__fma_rn(-x, x, e), y, x);
}

// The factor as a tiled wavefront, with no grid-wide barrier: a CTA per tile of
// FT x FT (j, k) pencils, tiles taken by ticket in diagonal order (a tile only
// waits on tiles with smaller tickets, which are running or done).  E, the
// pivots' reciprocals, is all that the cells exchange.  Within a tile a level
// costs one __syncthreads: the -y and -z neighbours' values of the level before
// sit in shared memory, the -x one in a register.  Between tiles the values
// themselves are the message: every cell starts as NOT_YET, and a tile's edge
// threads read the neighbouring pencil's cells until they are there.  Rows,
// weights and edges are loaded a chunk of FCH levels ahead.  A tile starts at
// its first level with a cell in the system and ends with the last; one
// without cells ends at once.  Every wait is bounded: past the limit the tile
// sets *err and stops, and all tiles that wait on it give up too (the solve
// reports a device timeout).
// Bound by latencies: a level's FP64 chain of two multiply-adds and a reciprocal
// of three more (about 64 cycles each; 820 cycles a level in all) and the hops
// between tiles (L2, about 3 us each).  290 us at 128^3, 127 at 64^3, 42 at 32^3
// with tiles of 8 x 8 and chunks of 2 (16 x 16, 4: 394, 174, 51).  Exchanging
// rsqrt(pivot), with a progress counter per tile released every eight levels,
// took 600 us at 128^3.
#ifndef MIC0_FT
#define MIC0_FT 8
#endif
#ifndef MIC0_FCH
#define MIC0_FCH 2
#endif
constexpr int FT = MIC0_FT, FCH = MIC0_FCH, FTHREADS = (FT * FT + 31) / 32 * 32;
static_assert(FT * FT >= 32 && FT * FT <= 1024, "a tile is one CTA");

__device__ __forceinline__ double ld_value(const double *p) {
    double v;
    asm volatile("ld.relaxed.gpu.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_value(double *p, double v) {
    asm volatile("st.relaxed.gpu.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
struct FactorChunk {
    double ad[FCH], w0[FCH], w1[FCH], w2[FCH], ey[FCH], ez[FCH];
    unsigned cells;   // which of its levels have a cell of this pencil
};

__global__ void __launch_bounds__(FTHREADS) k_mic0_tiles(StepConsts c, const uint8_t *fluid, const double4_32a *Ad,
                                                         const double *W0, const double *W1, const double *W2, double *E,
                                                         unsigned int *ticket, int *err, unsigned int spinLimit) {
    pdl_begin();
    __shared__ double prev[2][FT + 1][FT + 1];   // of the level before; row and column 0 stand for the edges
    __shared__ int tileSh, lvLo, lvHi;
    const int ntj = (c.J - 2 + FT - 1) / FT, ntk = (c.K - 2 + FT - 1) / FT;
    if (threadIdx.x == 0) {
        // ticket -> tile in diagonal order (tj + tk, then tj)
        int q = (int)atomicAdd(ticket, 1u), d = 0;
        for (; d < ntj + ntk - 1; d++) {
            const int n = min(d, ntj - 1) - max(0, d - ntk + 1) + 1;
            if (q < n) break;
            q -= n;
        }
        const bool wrong = d >= ntj + ntk - 1;   // more CTAs than tiles: the launch is wrong
        if (wrong) atomicExch(err, 1);
        const int tj = max(0, d - ntk + 1) + q;
        tileSh = wrong ? -1 : tj + ntj * (d - tj);
        lvLo = 0x7fffffff;
        lvHi = -1;
    }
    __syncthreads();
    const int tile = tileSh;
    if (tile < 0) return;
    const int tj = tile % ntj, tk = tile / ntj;
    const int sy = c.I, sz = c.I * c.J;
    // the levels with cells of this tile, 32 cells of a pencil at a time
    {
        const int lane = threadIdx.x & 31;
        int lo = 0x7fffffff, hi = -1;
        for (int p = threadIdx.x >> 5; p < FT * FT; p += FTHREADS / 32) {
            const int j = 1 + tj * FT + p % FT, k = 1 + tk * FT + p / FT;
            if (j > c.J - 2 || k > c.K - 2) continue;
            for (int i = 1 + lane; i <= c.I - 2; i += 32)
                if (fluid[i + sy * j + sz * k]) {
                    lo = min(lo, i + j + k);
                    hi = max(hi, i + j + k);
                }
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0 && hi >= 0) {
            atomicMin(&lvLo, lo);
            atomicMax(&lvHi, hi);
        }
    }
    for (int q = threadIdx.x; q < 2 * (FT + 1) * (FT + 1); q += FTHREADS) (&prev[0][0][0])[q] = 0.0;
    __syncthreads();
    const int lvStart = lvLo, lvEnd = lvHi;
    const int a = threadIdx.x % FT, b = threadIdx.x / FT;   // j and k within the tile
    const int j = 1 + tj * FT + a, k = 1 + tk * FT + b;
    const bool mine = b < FT && j <= c.J - 2 && k <= c.K - 2;
    const int pencil = sy * j + sz * k - j - k;   // cell of level lv: pencil + lv
    const bool edgeY = mine && a == 0 && tj > 0, edgeZ = mine && b == 0 && tk > 0;
    auto load = [&](int lvc, FactorChunk &n) {
        n.cells = 0;
#pragma unroll
        for (int m = 0; m < FCH; m++) {
            const int i = lvc + m - j - k, t = pencil + lvc + m;
            const bool in = mine && i >= 1 && i <= c.I - 2 && lvc + m <= lvEnd && fluid[t];
            n.cells |= (unsigned)in << m;
            n.ad[m] = in ? Ad[t].x : 0.0;
            n.w0[m] = in ? W0[t] : 0.0;
            n.w1[m] = in ? W1[t] : 0.0;
            n.w2[m] = in ? W2[t] : 0.0;
            n.ey[m] = in && edgeY ? ld_value(E + t - sy) : 0.0;
            n.ez[m] = in && edgeZ ? ld_value(E + t - sz) : 0.0;
        }
    };
    // Edge values that a weight asks for and that were not there when the chunk
    // was loaded, all at once; a cell without weight may be off the system.
    auto await = [&](int lvc, FactorChunk &n) {
        unsigned miss = 0;
#pragma unroll
        for (int m = 0; m < FCH; m++) {
            if (edgeY && n.w1[m] == 0.0) n.ey[m] = 0.0;
            if (edgeZ && n.w0[m] == 0.0) n.ez[m] = 0.0;
            miss |= (unsigned)(__double_as_longlong(n.ey[m]) == NOT_YET) << m;
            miss |= (unsigned)(__double_as_longlong(n.ez[m]) == NOT_YET) << (FCH + m);
        }
        for (unsigned spin = 1; miss; spin++) {
            if (spin >= spinLimit || ((spin & 255u) == 0u && *(volatile const int *)err)) {
                atomicExch(err, 1);
                return false;
            }
#pragma unroll
            for (int m = 0; m < FCH; m++) {
                if (miss >> m & 1u) n.ey[m] = ld_value(E + pencil + lvc + m - sy);
                if (miss >> (FCH + m) & 1u) n.ez[m] = ld_value(E + pencil + lvc + m - sz);
            }
#pragma unroll
            for (int m = 0; m < FCH; m++) {
                if (__double_as_longlong(n.ey[m]) != NOT_YET) miss &= ~(1u << m);
                if (__double_as_longlong(n.ez[m]) != NOT_YET) miss &= ~(1u << (FCH + m));
            }
        }
        return true;
    };
    FactorChunk now, next;
    double own = 0.0;   // this pencil's value of the level before (the -x neighbour's)
    int cur = 0;
    if (lvStart <= lvEnd) load(lvStart, now);
    for (int lvc = lvStart; lvc <= lvEnd; lvc += FCH) {
        load(lvc + FCH, next);
        const bool failed = (edgeY || edgeZ) && !await(lvc, now);
        if (__syncthreads_or(failed)) return;
#pragma unroll
        for (int m = 0; m < FCH; m++) {
            double e = 0.0;
            const float f0 = narrow_or_0(now.w0[m]), f1 = narrow_or_0(now.w1[m]);
            if (now.cells >> m & 1u) {
                const double ad = now.ad[m];
                const double ez = edgeZ ? now.ez[m] : prev[cur ^ 1][b][a + 1];
                const double ey = edgeY ? now.ey[m] : prev[cur ^ 1][b + 1][a];
                double d = __fma_rn(-now.w2[m], own, ad);
                // the guess comes from the same steps in FP32, while FP64 takes them
                const float g = guess_reciprocal(
                    __fmaf_rn(-f1, narrow_or_0(ey), __fmaf_rn(-f0, narrow_or_0(ez), narrow_or_0(d))));
                d = __fma_rn(-now.w0[m], ez, d);
                d = __fma_rn(-now.w1[m], ey, d);
                const double least = 0.25 * ad;
                // positive doubles compare as integers, and a quiet NaN, whatever its sign, is not below
                const bool low = ad > 0.0 ? __double_as_longlong(d) < __double_as_longlong(least) &&
                                                (unsigned)__double2hiint(d) <= 0xfff00000u
                                          : d < least;
                if (low) e = 1.0 / ad;
                else if (ad != 0.0) e = reciprocal(d, g);
                if (__double_as_longlong(e) == NOT_YET) e = __longlong_as_double(NOT_YET - 1);
                st_value(E + pencil + lvc + m, e);
            }
            if (b < FT) prev[cur][b + 1][a + 1] = e;
            own = e;
            cur ^= 1;
            __syncthreads();
        }
        now = next;
    }
}
// The two functions above on their own: 1 / d from the unit's guess times `off`,
// and sqrt(d).
__global__ void k_pivot_functions(int n, const double *d, const float *off, double *recip, double *root) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    recip[t] = reciprocal(d[t], guess_reciprocal(narrow_or_0(d[t])) * off[t]);
    root[t] = inverse_pivot(d[t]);
}
// Pivots' reciprocals to inverse pivots, 0 off the system.
__global__ void k_mic0_inverse(const uint8_t *fluid, long long n, double *E) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) E[t] = fluid[t] ? inverse_pivot(E[t]) : 0.0;
}

// The items of a solve: the chunks (SWEEP_CH steps of a tile, 1024 entries of
// the sweep layout) that the sweeps pass over, tile by tile.  An item is
// tile * (T / SWEEP_CH) + chunk.  One CTA.
__global__ void __launch_bounds__(1024) k_items(SweepLayout g, const int2 *range, int *items, int *nItems) {
    pdl_begin();
    __shared__ int sh[32], base;
    const int nt = g.nta * g.ntb, nch = g.T / SWEEP_CH, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    for (int t0 = 0; t0 < nt; t0 += 1024) {
        const int t = t0 + threadIdx.x;
        const int2 rg = t < nt ? range[t] : make_int2(0, -1);
        const int c0 = rg.x / SWEEP_CH, n = rg.y < rg.x ? 0 : rg.y / SWEEP_CH - c0 + 1;
        int x = n;   // inclusive scan over the CTA
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) sh[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int w = sh[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            sh[lane] = w;
        }
        __syncthreads();
        const int at = base + (warp ? sh[warp - 1] : 0) + x - n;
        for (int q = 0; q < n; q++) items[at + q] = t * nch + c0 + q;
        __syncthreads();
        if (threadIdx.x == 0) base += sh[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) *nItems = base;
}

// The grid cell of entry (tile, step tf, pencil p); false outside the interior.
__device__ __forceinline__ bool entry_cell(const SweepLayout &g, int I, int tile, int tf, int p, int &i, int &j, int &k) {
    const int A = (p & 7) + ((p >> 5) & 1) * SWEEP_VA, B = ((p >> 3) & 3) + (p >> 6) * SWEEP_VB;
    const int aa = tile % g.nta * SWEEP_WA + A + 1, bb = tile / g.nta * SWEEP_WB + B + 1;
    i = tf + 1 - A - B;
    j = g.swap ? bb : aa;
    k = g.swap ? aa : bb;
    return i >= 1 && i <= I - 2 && aa <= g.EA - 2 && bb <= g.EB - 2;
}

// A system's vectors in the sweep layout, an item per CTA, four consecutive
// pencils of a step per thread: the FP32 factor rows, the rows as exact float
// pairs (planes of A: the leading parts of the diagonal and of the couplings
// to +x, +y, +z, then their remainders), r = b as pairs, x = s = 0.  Reads
// gather whole 32-byte rows; all writes are coalesced.
__global__ void __launch_bounds__(TPB) k_layout(StepConsts c, SweepLayout g, const int *items, const int *nItems,
                                                PressureBuffers pb, unsigned int *sweepTicket) {
    if (blockIdx.x == 0 && threadIdx.x == 0) sweep_prep(sweepTicket);   // for the first sweep pair
    const int nch = g.T / SWEEP_CH, p0 = (threadIdx.x & 31) * 4;
    for (int it = blockIdx.x; it < *nItems; it += gridDim.x) {
        const int item = items[it], tile = item / nch, tf = item % nch * SWEEP_CH + (threadIdx.x >> 5);
        const long long e = ((long long)tile * g.T + tf) * SWEEP_NP + p0;
        float4 hi[4], lo[4], L[4];
        float rh[4], rl[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            hi[q] = lo[q] = L[q] = make_float4(0.f, 0.f, 0.f, 0.f);
            rh[q] = rl[q] = 0.0f;
            int i, j, k;
            if (!entry_cell(g, c.I, tile, tf, p0 + q, i, j, k)) continue;
            const long long t = (long long)i + (long long)c.I * (j + (long long)c.J * k);
            if (!pb.fluid[t]) continue;
            const double4_32a a = pb.Ad[t];
            const double inv = inverse_pivot(pb.pivotInv[t]), b = pb.b[t];
            hi[q] = make_float4((float)a.x, (float)a.y, (float)a.z, (float)a.w);
            lo[q] = make_float4((float)(a.x - (double)hi[q].x), (float)(a.y - (double)hi[q].y),
                                (float)(a.z - (double)hi[q].z), (float)(a.w - (double)hi[q].w));
            if (inv != 0.0) L[q] = make_float4((float)inv, (float)(a.y * inv), (float)(a.z * inv), (float)(a.w * inv));
            rh[q] = (float)b;
            rl[q] = (float)(b - (double)rh[q]);
        }
        const long long n = pb.nsl + SWEEP_NP;   // the planes' stride
        auto put = [&](float *p, float v0, float v1, float v2, float v3) {
            *reinterpret_cast<float4 *>(p + e) = make_float4(v0, v1, v2, v3);
        };
#pragma unroll
        for (int q = 0; q < 4; q++) pb.L[e + q] = L[q];
        put(pb.A, hi[0].x, hi[1].x, hi[2].x, hi[3].x);
        put(pb.A + n, hi[0].y, hi[1].y, hi[2].y, hi[3].y);
        put(pb.A + 2 * n, hi[0].z, hi[1].z, hi[2].z, hi[3].z);
        put(pb.A + 3 * n, hi[0].w, hi[1].w, hi[2].w, hi[3].w);
        put(pb.A + 4 * n, lo[0].x, lo[1].x, lo[2].x, lo[3].x);
        put(pb.A + 5 * n, lo[0].y, lo[1].y, lo[2].y, lo[3].y);
        put(pb.A + 6 * n, lo[0].z, lo[1].z, lo[2].z, lo[3].z);
        put(pb.A + 7 * n, lo[0].w, lo[1].w, lo[2].w, lo[3].w);
        put(pb.rh, rh[0], rh[1], rh[2], rh[3]);
        put(pb.rl, rl[0], rl[1], rl[2], rl[3]);
        put(pb.xh, 0.f, 0.f, 0.f, 0.f);
        put(pb.xl, 0.f, 0.f, 0.f, 0.f);
        put(pb.s, 0.f, 0.f, 0.f, 0.f);
    }
}

// Sum over a CTA of TPB threads in a fixed order; thread 0 has the result.
// FP64 runs at 2 lanes a clock on this GPU, so the tree's first steps go
// through shared memory in one warp (12 FP64 instructions a CTA; shuffles in
// every warp took 48).
__device__ __forceinline__ double block_sum(double v, double *sh) {
    sh[threadIdx.x] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < 32) {
        double w[TPB / 32];
#pragma unroll
        for (int q = 0; q < TPB / 32; q++) w[q] = sh[threadIdx.x + 32 * q];
#pragma unroll
        for (int m = TPB / 64; m > 0; m >>= 1)
#pragma unroll
            for (int q = 0; q < m; q++) w[q] += w[q + m];
        s = w[0];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    __syncthreads();
    return s;
}
// Max of non-negative floats over the CTA, a NaN counting as +inf, then one
// atomic on the bits of the double.
__device__ __forceinline__ void block_max_float_to(float v, unsigned long long *out) {
    __shared__ unsigned shm[TPB / 32];
    unsigned m = __reduce_max_sync(0xffffffffu, v != v ? 0x7f800000u : __float_as_uint(v));
    if ((threadIdx.x & 31) == 0) shm[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = __reduce_max_sync(0xffffffffu, threadIdx.x < TPB / 32 ? shm[threadIdx.x] : 0u);
        if (threadIdx.x == 0 && m) atomicMax(out, (unsigned long long)__double_as_longlong((double)__uint_as_float(m)));
    }
}

// The sums of the loop are finished by the kernel that needs them: every one
// of its CTAs adds the block partials of the kernel before it, in the same
// fixed order.  A fence, a ticket and a last CTA that adds them at the end of
// the producer took about 2 us longer per sum.  Where the host needs a
// result, the CTA that takes the last ticket sees all partials (or atomics),
// finishes and resets the ticket for the next launch.
__device__ __forceinline__ bool last_cta(unsigned int *ticket, unsigned int ctas) {
    __shared__ int amLast;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        amLast = atomicAdd(ticket, 1u) == ctas - 1;
        if (amLast) {
            *ticket = 0u;
            __threadfence();
        }
    }
    __syncthreads();
    return amLast;
}
// Sum of the launch's block partials in a fixed order (deterministic);
// thread 0 holds the result.
__device__ __forceinline__ double sum_partials_fixed(const double *partials, int n, double *sh) {
    double v = 0.0;
    for (int q = threadIdx.x; q < n; q += blockDim.x) v += __ldcg(partials + q);
    return block_sum(v, sh);
}
// The same sum for every thread of the CTA.
__device__ __forceinline__ double sum_partials_all(const double *partials, int n, double *sh) {
    const double v = sum_partials_fixed(partials, n, sh);
    if (threadIdx.x == 0) sh[0] = v;
    __syncthreads();
    const double r = sh[0];
    __syncthreads();
    return r;
}
__device__ __forceinline__ double bits_to_resid(const unsigned long long *p) {
    return __longlong_as_double((long long)__ldcg(p));
}

// The row kernels below run over the items of the solve on a fixed grid per
// context (pressure_partials_for CTAs): each thread sums its entries in a fixed
// order, each CTA writes one partial, and whoever needs the sum adds the partials
// in a fixed order, so every sum is deterministic.  Entries without a row hold
// zeros.  The vectors live in the sweep layout: a warp takes one step of a
// tile, whose entries are contiguous, and a row's six neighbours are entries
// of the steps before and after it, so loads are 16-byte and coalesced (a row
// list in cell order gathered every neighbour on its own).  The SpMV, the update
// and z.r, cold in a launch list: 17.7, 11.6 and 6.6 us at 518k rows (18.5, 14.8 and
// 13.9 with the row list).

// Double-float arithmetic on the FP32 pipe (this GPU's FP64 rate is ~1/64
// of FP32): a coefficient a = hi + lo (floats, exact to 48 bits) times an
// FP32 s is hi*s exactly as a rounded product plus its FMA-recovered error,
// plus lo*s; sums carry their rounding errors in a second float (Knuth's
// TwoSum).  A 7-term row sum is exact to ~2^-48 of its terms, where FP64 is
// exact to ~2^-53.
__device__ __forceinline__ float2 df_from(double v) {
    const float h = (float)v;
    return make_float2(h, (float)(v - (double)h));
}
__device__ __forceinline__ double df_to(float2 v) { return (double)v.x + (double)v.y; }
// (h, l) with h = fl(h + l): the pair in normalised form (|l| <= ulp(h) / 2)
__device__ __forceinline__ float2 df_norm(float h, float l) {
    const float s = __fadd_rn(h, l);
    return make_float2(s, __fsub_rn(l, __fsub_rn(s, h)));
}
// a + b for pairs: TwoSum of the leading parts, the rest added to the error
__device__ __forceinline__ float2 df_add(float2 a, float2 b) {
    const float t = __fadd_rn(a.x, b.x);
    const float bb = __fsub_rn(t, a.x);
    const float err = __fadd_rn(__fsub_rn(a.x, __fsub_rn(t, bb)), __fsub_rn(b.x, bb));
    return df_norm(t, __fadd_rn(err, __fadd_rn(a.y, b.y)));
}
// f * v for a float f and a pair v: the leading product exact as its
// rounded value plus its FMA-recovered error
__device__ __forceinline__ float2 df_scale(float f, float2 v) {
    const float ph = __fmul_rn(f, v.x);
    const float pl = __fmaf_rn(f, v.y, __fmaf_rn(f, v.x, -ph));
    return make_float2(ph, pl);
}
// (sh, sl) += (ah, al) s for two cells, ns = -s: the leading product exact as
// its rounded value plus its FMA-recovered error, the sum's rounding error by
// Knuth's TwoSum
__device__ __forceinline__ void df2_mul_add(const PairOps &k, F2 ah, F2 al, F2 sv, F2 ns, F2 &sh, F2 &sl) {
    const F2 nph = k.mul(ah, ns);                         // -(ah s) rounded
    const F2 pl = f2_fma(al, sv, f2_fma(ah, sv, nph));   // its error, plus al s
    const F2 t = k.sub(sh, nph);
    const F2 bb = k.sub(t, sh);
    const F2 err = k.sub(k.sub(sh, k.sub(t, bb)), k.add(nph, bb));   // exact error of the sum
    sl = k.add(sl, k.add(err, pl));
    sh = t;
}
// df_norm, df_add and df_scale for two cells
__device__ __forceinline__ void df2_norm(const PairOps &k, F2 h, F2 l, F2 &oh, F2 &ol) {
    oh = k.add(h, l);
    ol = k.sub(l, k.sub(oh, h));
}
__device__ __forceinline__ void df2_add(const PairOps &k, F2 ah, F2 al, F2 bh, F2 bl, F2 &oh, F2 &ol) {
    const F2 t = k.add(ah, bh);
    const F2 bb = k.sub(t, ah);
    const F2 err = k.add(k.sub(ah, k.sub(t, bb)), k.sub(bh, bb));
    df2_norm(k, t, k.add(err, k.add(al, bl)), oh, ol);
}
__device__ __forceinline__ void df2_scale(const PairOps &k, F2 f, F2 nf, F2 vh, F2 vl, F2 &oh, F2 &ol) {   // nf = -f
    oh = k.mul(f, vh);
    ol = f2_fma(f, vl, k.neg(f2_fma(nf, vh, oh)));
}
__device__ __forceinline__ void ld2x2(const float *p, F2 (&v)[2]) {
    const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(p);
    v[0] = q.x; v[1] = q.y;
}
__device__ __forceinline__ void st2x2(float *p, const F2 (&v)[2]) {
    *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(v[0], v[1]);
}
__device__ __forceinline__ void ld4(const float *p, float (&v)[4]) {
    const float4 q = *reinterpret_cast<const float4 *>(p);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
__device__ __forceinline__ void st4(float *p, const float (&v)[4]) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

// s = z + beta s (pcgsolver.h:295-298, beta rounded to float) fused with
// q = A s over the rows in double-float, stored as a pair; s.q summed in
// double-float per thread and in FP64 across threads.  The new s of a row's
// stencil is formed from the previous iteration's buffer sIn (so no row
// reads a value another thread is writing) and the row's own goes to sOut.
// In the first iteration beta = 0 and sIn = 0, so s = z.  A neighbour that
// is not a row couples with 0 (its entry holds a finite value); one outside
// the layout is the zero padding after it.
//
// An item's operands are whole steps of the layout, contiguous in every
// plane, so one thread brings them to shared memory with ten bulk copies (the
// rows' planes and sIn already while the kernel before this one ends): a
// single latency per item, where loads into registers exposed one per
// coupling.  A
// thread takes four consecutive pencils of a step, two to a packed operation;
// only the neighbours in other tiles are read from global memory.
struct SpmvSmem {
    float S[SWEEP_CH + 2][SWEEP_NP], Z[SWEEP_CH + 2][SWEEP_NP];   // steps -1 .. 8 of the item
    float C[6][SWEEP_CH + 1][SWEEP_NP];   // couplings +x, +y, +z: leading parts, remainders; steps -1 .. 7
    float D[2][SWEEP_CH][SWEEP_NP];       // diagonal
    unsigned long long bar;
    int failed, issued;
};
static_assert(sizeof(SpmvSmem) + sizeof(double) * TPB <= 48 * 1024, "static shared memory");
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bulk_steps(float *dst, const float *src, int steps, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_addr(dst)), "l"(src), "r"(steps * SWEEP_NP * 4), "r"(bar) : "memory");
}
template <bool SWAP>
__global__ void __launch_bounds__(TPB, 3)
    k_spmv_s(SweepLayout g, long long nsl, const int *__restrict__ items, const int *__restrict__ nItems,
             const float *__restrict__ A, const float *__restrict__ z, const float *__restrict__ sIn,
             float *__restrict__ sOut, float *__restrict__ qh, float *__restrict__ ql, const double *zrPartials,
             double *partials, double *scal, PcgCtl *ctl, int *err, PairOps k2) {
    __shared__ __align__(128) SpmvSmem sm;
    __shared__ double sh[TPB];
    const int n = *nItems, T = g.T, nch = T / SWEEP_CH, ctas = min((int)gridDim.x, n);
    constexpr int NP = SWEEP_NP;
    const long long np = nsl + NP;        // stride of the planes of A
    const unsigned bar = smem_addr(&sm.bar);
    // The couplings along a and b are planes 1 + CA and 1 + CB (C[CA], C[CB]).
    constexpr int CA = SWAP ? 2 : 1, CB = SWAP ? 1 : 2;
    auto issue = [&](int it, bool rows, bool zed) {   // one thread
        const int item = items[it], tile = item / nch, t0 = item % nch * SWEEP_CH;
        const int lo = t0 > 0, hi = t0 + SWEEP_CH < T;
        const long long e0 = ((long long)tile * T + t0) * NP;
        if (rows) {
            const unsigned steps = 2 * (SWEEP_CH + lo + hi) + 6 * (SWEEP_CH + lo) + 2 * SWEEP_CH;
            asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}" ::"r"(bar),
                         "r"(steps * (NP * 4)) : "memory");
            for (int q = 0; q < 6; q++)
                bulk_steps(sm.C[q][1 - lo], A + (q < 3 ? 1 + q : 2 + q) * np + e0 - lo * NP, SWEEP_CH + lo, bar);
            bulk_steps(sm.D[0][0], A + e0, SWEEP_CH, bar);
            bulk_steps(sm.D[1][0], A + 4 * np + e0, SWEEP_CH, bar);
            bulk_steps(sm.S[1 - lo], sIn + e0 - lo * NP, SWEEP_CH + lo + hi, bar);
        }
        if (zed) bulk_steps(sm.Z[1 - lo], z + e0 - lo * NP, SWEEP_CH + lo + hi, bar);
    };
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        sm.failed = 0;
        // The rows and sIn were written before the kernel ahead of this one;
        // the flag may still be set, and what is started is waited for.
        sm.issued = (int)blockIdx.x < n && !*(volatile int *)&ctl->done;
        if (sm.issued) issue(blockIdx.x, true, false);
    }
    pdl_wait();
    pdl_trigger();
    __syncthreads();
    const bool done = ctl->done != 0;
    if ((int)blockIdx.x >= n || (done && !sm.issued)) return;
    if (threadIdx.x == 0) issue(blockIdx.x, false, true);
    // rho of this iteration, and beta = rho / rho of the one before as float
    // (pcgsolver.h:295-298); the two alternate between two places
    const int odd = ctl->it & 1;
    const double rho = sum_partials_all(zrPartials, ctas, sh), before = scal[odd ? 3 : 7];
    if (blockIdx.x == 0 && threadIdx.x == 0) scal[odd ? 7 : 3] = rho;
    const float betaf = ctl->it > 0 && before != 0.0 ? (float)(rho / before) : 0.0f;
    const F2 beta = f2(betaf, betaf);
    const int u = threadIdx.x >> 5, p0 = (threadIdx.x & 31) * 4, la0 = p0 & 7, lb = (p0 >> 3) & 3, wa = (p0 >> 5) & 1,
              wb = p0 >> 6;
    F2 dotH = k2.zero, dotL = k2.zero;
    unsigned phase = 0;
    for (int it = blockIdx.x; it < n; it += gridDim.x) {
        if (threadIdx.x == 0 && it != (int)blockIdx.x) issue(it, true, true);
        const int item = items[it], tile = item / nch, tf = item % nch * SWEEP_CH + u;
        const int ta = tile % g.nta, tb = tile / g.nta;
        const long long e = ((long long)tile * T + tf) * NP + p0, none = nsl + p0;
        const bool up = tf + 1 < T, down = tf > 0;
        // Neighbours in other tiles, read while the copies run: a+ of the last
        // pencil, a- of the first; b+ or b- of all four.
        const bool farU = la0 != 0 && wa == 1, farD = la0 == 0 && wa == 0;
        const bool farBU = lb == 3 && wb == 1, farBD = lb == 0 && wb == 0;
        float saU = 0.f, saD = 0.f, caH = 0.f, caL = 0.f;
        F2 fz[2] = {0, 0}, fs[2] = {0, 0}, fh[2] = {0, 0}, fl[2] = {0, 0};
        auto snew_at = [&](long long at) { return __fmaf_rn(betaf, sIn[at], z[at]); };
        if (farU)
            saU = snew_at(ta + 1 < g.nta && tf >= SWEEP_WA - 1 ? e + ((long long)T - (SWEEP_WA - 1)) * NP - 36 : none);
        if (farD) {
            const long long at =
                ta > 0 && tf + SWEEP_WA - 1 < T ? e - ((long long)T - (SWEEP_WA - 1)) * NP + 39 : none;
            saD = snew_at(at);
            caH = A[(1 + CA) * np + at];
            caL = A[(5 + CA) * np + at];
        }
        if (farBU || farBD) {
            const long long step = ((long long)T * g.nta - (SWEEP_WB - 1)) * NP - 88;
            long long at = none;
            if (farBU && tb + 1 < g.ntb && tf >= SWEEP_WB - 1) at = e + step;
            if (farBD && tb > 0 && tf + SWEEP_WB - 1 < T) at = e - step;
            ld2x2(z + at, fz);
            ld2x2(sIn + at, fs);
            if (farBD) {
                ld2x2(A + (1 + CB) * np + at, fh);
                ld2x2(A + (5 + CB) * np + at, fl);
            }
        }
        bool in = false;
        for (unsigned spin = 0; spin < DEFAULT_SPIN_LIMIT && !in; spin++) {
            unsigned ok;
            asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 256;\n selp.u32 %0, 1, 0, p;\n}"
                         : "=r"(ok) : "r"(bar), "r"(phase) : "memory");
            in = ok != 0;
        }
        if (!in) sm.failed = 1;
        phase ^= 1;
        if (done) return;   // what was started is in
        auto from = [&](const float *row, int p, F2 (&v)[2]) { ld2x2(row + p, v); };
        auto snew = [&](int r, int p, F2 (&v)[2]) {   // of step r - 1 of the item
            F2 zz[2], ss[2];
            from(sm.Z[r], p, zz);
            from(sm.S[r], p, ss);
            v[0] = f2_fma(beta, ss[0], zz[0]);
            v[1] = f2_fma(beta, ss[1], zz[1]);
        };
        auto snew1 = [&](int r, int p) { return __fmaf_rn(betaf, sm.S[r][p], sm.Z[r][p]); };
        F2 accH[2] = {k2.zero, k2.zero}, accL[2] = {k2.zero, k2.zero};
        auto couple = [&](const F2 (&h)[2], const F2 (&l)[2], const F2 (&v)[2]) {
#pragma unroll
            for (int q = 0; q < 2; q++) df2_mul_add(k2, h[q], l[q], v[q], k2.neg(v[q]), accH[q], accL[q]);
        };
        // sU, sD: the steps after and before; nothing beyond the tile's ends
        F2 s0[2], sU[2] = {0, 0}, sD[2] = {0, 0}, h[2], l[2], v[2];
        snew(u + 1, p0, s0);
        if (up) {
            snew(u + 2, p0, sU);
            if (!farU) saU = snew1(u + 2, la0 == 0 ? p0 + 4 : p0 + 28);
        }
        if (down) {
            snew(u, p0, sD);
            if (!farD) {
                const int p = la0 != 0 ? p0 - 1 : p0 - 25;
                saD = snew1(u, p);
                caH = sm.C[CA][u][p];
                caL = sm.C[3 + CA][u][p];
            }
        }
        from(sm.D[0][u], p0, h); from(sm.D[1][u], p0, l);
        couple(h, l, s0);
        from(sm.C[0][u + 1], p0, h); from(sm.C[3][u + 1], p0, l);
        couple(h, l, sU);   // +x
        auto plusA = [&] {
            from(sm.C[CA][u + 1], p0, h); from(sm.C[3 + CA][u + 1], p0, l);
            v[0] = f2(f2_y(sU[0]), f2_x(sU[1]));
            v[1] = f2(f2_y(sU[1]), saU);
            couple(h, l, v);
        };
        auto plusB = [&] {
            from(sm.C[CB][u + 1], p0, h); from(sm.C[3 + CB][u + 1], p0, l);
            v[0] = v[1] = 0;
            if (farBU) { v[0] = f2_fma(beta, fs[0], fz[0]); v[1] = f2_fma(beta, fs[1], fz[1]); }
            else if (up) snew(u + 2, lb < 3 ? p0 + 8 : p0 + 40, v);
            couple(h, l, v);
        };
        auto minusA = [&] {
            F2 ch[2] = {0, 0}, cl[2] = {0, 0};
            if (down) { from(sm.C[CA][u], p0, ch); from(sm.C[3 + CA][u], p0, cl); }
            h[0] = f2(caH, f2_x(ch[0])); h[1] = f2(f2_y(ch[0]), f2_x(ch[1]));
            l[0] = f2(caL, f2_x(cl[0])); l[1] = f2(f2_y(cl[0]), f2_x(cl[1]));
            v[0] = f2(saD, f2_x(sD[0]));
            v[1] = f2(f2_y(sD[0]), f2_x(sD[1]));
            couple(h, l, v);
        };
        auto minusB = [&] {
            h[0] = fh[0]; h[1] = fh[1]; l[0] = fl[0]; l[1] = fl[1];
            v[0] = v[1] = 0;
            if (farBD) { v[0] = f2_fma(beta, fs[0], fz[0]); v[1] = f2_fma(beta, fs[1], fz[1]); }
            else if (down) {
                const int p = lb > 0 ? p0 - 8 : p0 - 40;
                from(sm.C[CB][u], p, h); from(sm.C[3 + CB][u], p, l);
                snew(u, p, v);
            }
            couple(h, l, v);
        };
        // +y, +z, then -x, -y, -z
        if (SWAP) { plusB(); plusA(); } else { plusA(); plusB(); }
        h[0] = h[1] = l[0] = l[1] = 0;
        if (down) { from(sm.C[0][u], p0, h); from(sm.C[3][u], p0, l); }
        couple(h, l, sD);
        if (SWAP) { minusB(); minusA(); } else { minusA(); minusB(); }
        F2 oh[2], ol[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            df2_norm(k2, accH[q], accL[q], oh[q], ol[q]);
            F2 ph, pl;
            df2_scale(k2, s0[q], k2.neg(s0[q]), oh[q], ol[q], ph, pl);
            df2_add(k2, dotH, dotL, ph, pl, dotH, dotL);
        }
        st2x2(sOut + e, s0);
        st2x2(qh + e, oh);
        st2x2(ql + e, ol);
        __syncthreads();   // the operands are free again
    }
    if (threadIdx.x == 0 && sm.failed) atomicExch(err, 1);
    double b = block_sum(df_to(make_float2(f2_x(dotH), f2_x(dotL))) + df_to(make_float2(f2_y(dotH), f2_y(dotL))), sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = b;
}

// The partial sums of rho_new = z.r; inside the loop (inLoop) it also begins
// the next iteration: its index, its residual norms cleared.  Before the loop
// the last CTA sums rho for the host.
__global__ void __launch_bounds__(TPB) k_dot_zr(const int *__restrict__ items, const int *__restrict__ nItems,
                                                const float *__restrict__ z, const float *__restrict__ rh,
                                                const float *__restrict__ rl, double *partials, double *scal,
                                                unsigned long long *rmaxBits, PcgCtl *ctl, int inLoop) {
    __shared__ double sh[TPB];
    const int n = *nItems;
    float2 dot = make_float2(0.0f, 0.0f);   // double-float per thread, FP64 across threads
    float h[4], l[4];
    auto entry = [&](int it) { return (long long)items[it] * (SWEEP_CH * SWEEP_NP) + threadIdx.x * 4; };
    const int ctas = min((int)gridDim.x, n);
    if ((int)blockIdx.x < n) {   // r does not depend on the sweeps
        ld4(rh + entry(blockIdx.x), h);
        ld4(rl + entry(blockIdx.x), l);
    }
    pdl_wait();
    pdl_trigger();
    if (ctl->done || (int)blockIdx.x >= n) return;
    for (int it = blockIdx.x; it < n; it += gridDim.x) {
        const long long e = entry(it);
        float zv[4];
        ld4(z + e, zv);
        if (it != (int)blockIdx.x) {
            ld4(rh + e, h);
            ld4(rl + e, l);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) dot = df_add(dot, df_scale(zv[q], make_float2(h[q], l[q])));
    }
    double s = block_sum(df_to(dot), sh);
    if (threadIdx.x == 0) partials[blockIdx.x] = s;
    if (inLoop) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            ctl->it += 1;
            rmaxBits[0] = rmaxBits[1] = 0ull;
        }
    } else if (last_cta(&ctl->ticket[1], ctas)) {
        const double zr = sum_partials_fixed(partials, ctas, sh);
        if (threadIdx.x == 0) scal[1] = zr;
    }
}

// The reference's convergence test |r|inf <= tol |b|inf (pcgsolver.h:
// 263-288) on the device.  On the iterations where r is recomputed as b - A x
// (every 25th) that norm decides; otherwise a pass of the recurrence's norm is
// only a claim, which the recompute of b - A x then settles.
__device__ __forceinline__ void convergence_test(PcgCtl *ctl, double resid, double ptol) {
    ctl->resid = resid;
    if (resid <= ptol) {
        ctl->done = 1;
        ctl->iters = ctl->it + 1;
    }
}

// x += alpha s, r -= alpha q with alpha = rho / s.q passed on as float, as
// BLAS::addScaled(float alpha, ...) does (blaswrapper.h:129-158); |r|inf
__global__ void __launch_bounds__(TPB) k_update_xr(const int *__restrict__ items, const int *__restrict__ nItems,
                                                   float *__restrict__ xh, float *__restrict__ xl,
                                                   float *__restrict__ rh, float *__restrict__ rl,
                                                   const float *__restrict__ s, const float *__restrict__ qh,
                                                   const float *__restrict__ ql, const double *sqPartials,
                                                   const double *scal, unsigned long long *rmaxBits, PcgCtl *ctl,
                                                   unsigned int *sweepTicket) {
    __shared__ double sh[TPB];
    const int n = *nItems;
    float vxh[4], vxl[4], vrh[4], vrl[4];
    auto entry = [&](int it) { return (long long)items[it] * (SWEEP_CH * SWEEP_NP) + threadIdx.x * 4; };
    auto load_xr = [&](long long e) {
        ld4(xh + e, vxh); ld4(xl + e, vxl);
        ld4(rh + e, vrh); ld4(rl + e, vrl);
    };
    if ((int)blockIdx.x < n) load_xr(entry(blockIdx.x));   // the SpMV before does not touch them
    pdl_wait();
    pdl_trigger();
    if (blockIdx.x == 0 && threadIdx.x == 0) sweep_prep(sweepTicket);   // for the sweep pair that follows
    if (ctl->done || (int)blockIdx.x >= n) return;
    const int ctas = min((int)gridDim.x, n);
    const float alpha = (float)(scal[ctl->it & 1 ? 7 : 3] / sum_partials_all(sqPartials, ctas, sh));
    float m = 0.0f;
    for (int it = blockIdx.x; it < n; it += gridDim.x) {
        const long long e = entry(it);
        float vs[4], vqh[4], vql[4];
        if (it != (int)blockIdx.x) load_xr(e);
        ld4(s + e, vs); ld4(qh + e, vqh); ld4(ql + e, vql);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float2 xv = df_add(make_float2(vxh[k], vxl[k]),
                                     df_scale(alpha, make_float2(vs[k], 0.0f)));   // alpha s is exact as a pair
            const float2 rv = df_add(make_float2(vrh[k], vrl[k]), df_scale(-alpha, make_float2(vqh[k], vql[k])));
            vxh[k] = xv.x;
            vxl[k] = xv.y;
            vrh[k] = rv.x;   // normalised: the pair rounded to float, the sweeps' right-hand side
            vrl[k] = rv.y;
            const float av = fabsf(rv.x);
            m = (av != av || av > m) ? av : m;   // a NaN sticks
        }
        st4(xh + e, vxh); st4(xl + e, vxl);
        st4(rh + e, vrh); st4(rl + e, vrl);
    }
    block_max_float_to(m, rmaxBits);
}

// r = b - A x (residual replacement); |r|inf, which the last CTA tests as
// final.  Inside the loop it runs only when needed: on every 25th iteration
// (pcgsolver.h's periodic recompute, here before the test) and when the
// recurrence just claimed convergence (a claim is only made on the other
// iterations, so one launch serves both); never once converged.
__global__ void __launch_bounds__(TPB) k_true_residual(StepConsts c, SweepLayout g, const int *__restrict__ items,
                                                       const int *__restrict__ nItems,
                                                       const uint8_t *__restrict__ fluid,
                                                       const double4_32a *__restrict__ Ad, const double *__restrict__ b,
                                                       const float *__restrict__ xh, const float *__restrict__ xl,
                                                       float *__restrict__ rh, float *__restrict__ rl,
                                                       unsigned long long *rmaxBits, const double *scal, PcgCtl *ctl) {
    pdl_wait();
    pdl_trigger();
    if (ctl->done) return;
    const double claimed = bits_to_resid(rmaxBits);   // of the recurrence
    if ((ctl->it + 1) % 25 != 0 && !(claimed <= scal[6])) {
        if (blockIdx.x == 0 && threadIdx.x == 0) ctl->resid = claimed;
        return;
    }
    const int n = *nItems, nch = g.T / SWEEP_CH;
    const long long sy = c.I, sz = (long long)c.I * c.J;
    double m = 0.0;
    for (long long w = (long long)blockIdx.x * TPB + threadIdx.x; w < (long long)n * (SWEEP_CH * SWEEP_NP);
         w += (long long)gridDim.x * TPB) {
        const int item = items[w / (SWEEP_CH * SWEEP_NP)], in = (int)(w % (SWEEP_CH * SWEEP_NP));
        const int tile = item / nch, tf = item % nch * SWEEP_CH + in / SWEEP_NP, p = in % SWEEP_NP;
        int i, j, k;
        if (!entry_cell(g, c.I, tile, tf, p, i, j, k)) continue;
        const long long t = i + sy * j + sz * k;
        if (!fluid[t]) continue;
        const long long e = ((long long)tile * g.T + tf) * SWEEP_NP + p;
        // x at the row and, where they are rows, at its neighbours
        auto xat = [&](bool row, int ni, int nj, int nk) {
            if (!row) return 0.0;
            const long long en = sweep_index(g, ni, nj, nk);
            return df_to(make_float2(xh[en], xl[en]));
        };
        const double4_32a a = Ad[t];
        double ax = a.x * df_to(make_float2(xh[e], xl[e]));
        ax = fma(a.y, xat(fluid[t + 1], i + 1, j, k), ax);
        ax = fma(a.z, xat(fluid[t + sy], i, j + 1, k), ax);
        ax = fma(a.w, xat(fluid[t + sz], i, j, k + 1), ax);
        if (fluid[t - 1]) ax = fma(Ad[t - 1].y, xat(true, i - 1, j, k), ax);
        if (fluid[t - sy]) ax = fma(Ad[t - sy].z, xat(true, i, j - 1, k), ax);
        if (fluid[t - sz]) ax = fma(Ad[t - sz].w, xat(true, i, j, k - 1), ax);
        const double rv = b[t] - ax;
        const float2 rp = df_from(rv);
        rh[e] = rp.x;
        rl[e] = rp.y;
        const double av = fabs(rv);
        m = (av != av || av > m) ? av : m;
    }
    block_max_to(m, rmaxBits + 1);
    if (last_cta(&ctl->ticket[3], gridDim.x) && threadIdx.x == 0) convergence_test(ctl, bits_to_resid(rmaxBits + 1), scal[6]);
}

// The solution to a float per cell (zero off the rows: cleared before).
__global__ void __launch_bounds__(TPB) k_x_to_cells(StepConsts c, SweepLayout g, const int *items, const int *nItems,
                                                    const uint8_t *fluid, const float *xh, const float *xl, float *P) {
    const int nch = g.T / SWEEP_CH;
    for (int it = blockIdx.x; it < *nItems; it += gridDim.x) {
        const int item = items[it], tile = item / nch;
        for (int in = threadIdx.x; in < SWEEP_CH * SWEEP_NP; in += TPB) {
            const int tf = item % nch * SWEEP_CH + in / SWEEP_NP, p = in % SWEEP_NP;
            int i, j, k;
            if (!entry_cell(g, c.I, tile, tf, p, i, j, k)) continue;
            const long long t = (long long)i + (long long)c.I * (j + (long long)c.J * k);
            if (!fluid[t]) continue;
            const long long e = ((long long)tile * g.T + tf) * SWEEP_NP + p;
            P[t] = (float)df_to(make_float2(xh[e], xl[e]));
        }
    }
}

// _applyPressureToVelocityFieldThread (pressuresolver.cpp:896-1046) without
// surface tension.  Liquid means phi < 0 over all cells (FluidMaterialGrid,
// :849-858); the faces i == 0 and i == I-1 (and the v/w analogues) are
// skipped as the reference skips them.
__global__ void k_apply_pressure(StepConsts c, const float *phi, const float *wu, const float *wv, const float *ww,
                                 const float *P, float factor, float *u, float *v, float *w, uint8_t *vu,
                                 uint8_t *vv, uint8_t *vw) {
    pdl_begin();
    long long nu = (long long)(c.I + 1) * c.J * c.K, nv = (long long)c.I * (c.J + 1) * c.K;
    long long nw = (long long)c.I * c.J * (c.K + 1);
    long long f = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nu + nv + nw) return;
    int dir = f < nu ? 0 : (f < nu + nv ? 1 : 2);
    long long l = dir == 0 ? f : (dir == 1 ? f - nu : f - nu - nv);
    int ni = c.I + (dir == 0), nj = c.J + (dir == 1);
    int i, j, k;
    unflatten(l, ni, nj, i, j, k);
    float *G = dir == 0 ? u : (dir == 1 ? v : w);
    uint8_t *V = dir == 0 ? vu : (dir == 1 ? vv : vw);
    const float *W = dir == 0 ? wu : (dir == 1 ? wv : ww);
    V[l] = 0;
    int g = dir == 0 ? i : (dir == 1 ? j : k);
    int gmax = dir == 0 ? c.I : (dir == 1 ? c.J : c.K);
    if (g == 0 || g == gmax - 1) return;
    Dims dc{c.I, c.J, c.K};
    int ai = i - (dir == 0), aj = j - (dir == 1), ak = k - (dir == 2);
    bool fb = dc.in(i, j, k) && phi[dc.idx(i, j, k)] < 0.0f;
    bool fa = phi[dc.idx(ai, aj, ak)] < 0.0f;
    bool border = (g == gmax) ? fa : (fb || fa);
    if (!(W[l] > 0.0f && border)) {
        G[l] = 0.0f;
        return;
    }
    float p1, p2;
    const float eps = 1e-6f;
    const double maxtheta = 25.0;
    if (fa && fb) {
        p1 = P[dc.idx(ai, aj, ak)];
        p2 = P[dc.idx(i, j, k)];
    } else {
        float phi1 = phi[dc.idx(ai, aj, ak)], phi2 = phi[dc.idx(i, j, k)];
        if (fa) {
            float tp = (float)fmax(-maxtheta, fmin((double)__fdiv_rn(phi2, __fadd_rn(phi1, eps)), maxtheta));
            p1 = P[dc.idx(ai, aj, ak)];
            p2 = __fmul_rn(tp, p1);
        } else {
            float tp = (float)fmax(-maxtheta, fmin((double)__fdiv_rn(phi1, __fadd_rn(phi2, eps)), maxtheta));
            p2 = P[dc.idx(i, j, k)];
            p1 = __fmul_rn(tp, p2);
        }
    }
    G[l] = __fadd_rn(G[l], __fmul_rn(-factor, __fsub_rn(p2, p1)));
    V[l] = 1;
}

int cuda_fail(cudaError_t e, const char *what, std::string *msg) {
    if (msg) *msg = std::string("pressure solve: ") + what + ": " + cudaGetErrorString(e);
    return FLIP_E_CUDA;
}

}  // namespace

// One CTA of the row kernels per `cellsPerCta` grid cells (4096 by default),
// at least 128 where there are as many items, at most the three per SM that
// the SpMV's shared memory leaves resident.  A liquid fills a fraction of the
// grid, so a CTA takes a few items of 1024 entries, and CTAs beyond the items
// leave at once.  The floor of 128: 64^3 frames 3.40 -> 3.30 ms; the cap:
// 128^3 frames 11.63 -> 11.40 ms, 256x128x128 27.2 -> 26.3 ms (a partial last
// wave, and more partials for every CTA to add).
constexpr long long ROW_CTAS = 152 * 3;
int pressure_partials_for(int I, int J, int K, int cellsPerCta) {
    static_assert(RBLOCKS == PCG_MAX_PARTIALS, "the partials buffer holds RBLOCKS sums");
    const long long items = sweep_items_max(I, J, K);
    const long long ctas = std::max<long long>(div_up((long long)I * J * K, std::max(cellsPerCta, 256)), 128);
    return (int)std::max(1LL, std::min({ctas, items, ROW_CTAS}));
}

#define PCK(call)                                               \
    do {                                                        \
        cudaError_t e_ = (call);                                \
        if (e_ != cudaSuccess) return cuda_fail(e_, #call, errMsg); \
    } while (0)

// MIC(0) factor of the rows Ad over the cells flagged in `fluid`: E, the
// pivots' reciprocals (FP64), which starts with all bits set.  W0..W2: n
// doubles each of scratch; err: set when a bounded wait gave up.
void mic0_factor(const StepConsts &c, const uint8_t *fluid, const double4_32a *Ad, double *E, double *W0, double *W1,
                 double *W2, unsigned int *ticket, int *err, unsigned int spinLimit, cudaStream_t s) {
    const long long n = (long long)c.I * c.J * c.K;
    const int ntiles = div_up(c.J - 2, FT) * div_up(c.K - 2, FT);
    cudaMemsetAsync(ticket, 0, sizeof(unsigned int), s);
    launch_next(k_mic0_weights, div_up(n, TPB), TPB, s, c, fluid, Ad, W0, W1, W2);
    // not early: its CTAs should have the SMs to themselves, as evenly as they can
    launch_after(false, k_mic0_tiles, ntiles, FTHREADS, 0, s, c, fluid, Ad, W0, W1, W2, E, ticket, err, spinLimit);
}
// E to inverse pivots, 0 off the system.
void mic0_inverse_pivots(const uint8_t *fluid, long long n, double *E, cudaStream_t s) {
    FLIP_COUNT(1);
    k_mic0_inverse<<<div_up(n, TPB), TPB, 0, s>>>(fluid, n, E);
}

void launch_pivot_functions(int n, const double *d, const float *off, double *recip, double *root, cudaStream_t s) {
    FLIP_COUNT(1);
    k_pivot_functions<<<div_up(n, TPB), TPB, 0, s>>>(n, d, off, recip, root);
}

// The chunks of the sweep layout that the sweeps pass over, and the system's
// vectors there.
static unsigned item_ctas(const StepConsts &c) {
    return (unsigned)std::max(1LL, std::min<long long>(sweep_items_max(c.I, c.J, c.K), RBLOCKS));
}
void launch_items(const StepConsts &c, PressureBuffers &pb, SweepState &sw, cudaStream_t s) {
    launch_sweep_ranges(c, pb.sl, pb.fluid, sw, s);
    launch_next(k_items, 1, 1024, s, pb.sl, sw.range, pb.items, pb.nItems);
}
void launch_layout(const StepConsts &c, const PressureBuffers &pb, SweepState &sw, cudaStream_t s) {
    FLIP_COUNT(1);
    k_layout<<<item_ctas(c), TPB, 0, s>>>(c, pb.sl, pb.items, pb.nItems, pb, sw.ticket);
}
// sOut = z + beta sIn, q = A sOut and the partial sums of sOut.q
void launch_spmv(const PressureBuffers &pb, const float *sIn, float *sOut, SweepState &sw, cudaStream_t s) {
    launch_after(true, pb.sl.swap ? k_spmv_s<true> : k_spmv_s<false>, (unsigned)pb.nPartials, TPB, 0, s, pb.sl, pb.nsl, pb.items,
                 pb.nItems, pb.A, pb.z, sIn, sOut, pb.qh, pb.ql, pb.partials + PCG_MAX_PARTIALS, pb.partials, pb.scal, pb.ctl,
                 sw.err, PairOps{});
}

// The condition of the device-side loop over batches of PCG iterations: one
// more batch while the solve has not converged, no wavefront has given up
// and fewer than maxBatches batches have run (so the loop always ends).
__global__ void k_pcg_loop(cudaGraphConditionalHandle h, PcgCtl *ctl, const int *err) {
    const int ran = ctl->batches + 1;
    ctl->batches = ran;
    const bool more = !ctl->done && !*(volatile const int *)err && ran < ctl->maxBatches;
    cudaGraphSetConditional(h, more ? 1u : 0u);
}

int pressure_project(const StepConsts &c, const PressureArgs &a, PressureBuffers &pb, SweepState &sw,
                     PressureMail *mail, cudaStream_t s, PressureResult *res, std::string *errMsg) {
    const long long n = (long long)c.I * c.J * c.K;
    const unsigned nb = div_up(n, TPB);
    const unsigned rb = (unsigned)pb.nPartials;   // reduction grid
    const double mf = a.dt / (c.dx * c.dx);
    res->iterations = 0;
    res->residual = 0.0;
    res->applied = false;
    res->cells = 0;
    auto sync = [&]() -> cudaError_t {
        FLIP_SYNC_COUNT();
        cudaError_t e = cudaStreamSynchronize(s);
        return e != cudaSuccess ? e : cudaGetLastError();
    };

    static const int lr[8] = {0x7fffffff, -1, 0, 0x7fffffff, -1, 0x7fffffff, -1, 0};
    std::memcpy(mail->levelRange, lr, sizeof(lr));
    PCK(cudaMemcpyAsync(pb.levelRange, mail->levelRange, sizeof(lr), cudaMemcpyHostToDevice, s));
    PCK(cudaMemsetAsync(pb.scal, 0, 8 * sizeof(double), s));
    launch_next(k_flags, div_up(n, FLAG_CELLS), TPB, s, c, a.phi, pb.fluid, pb.levelRange);
    launch_next(k_build, nb, TPB, s, c, a.phi, a.wu, a.wv, a.ww, a.u, a.v, a.w, mf, pb);
    PCK(cudaMemcpyAsync(mail->levelRange, pb.levelRange, 7 * sizeof(int), cudaMemcpyDeviceToHost, s));
    PCK(cudaMemcpyAsync(&mail->bmax, pb.scal + 2, sizeof(double), cudaMemcpyDeviceToHost, s));
    PCK(sync());
    if (a.dumpRhs) PCK(cudaMemcpy(a.dumpRhs, pb.b, n * sizeof(double), cudaMemcpyDeviceToHost));
    const int lo = mail->levelRange[0], hi = mail->levelRange[1];
    res->cells = mail->levelRange[2];
    const double bmax = mail->bmax;
    if (hi < lo || bmax < a.tol) {   // no system, or nothing to project (pressuresolver.cpp:53-56)
        if (a.dumpPressure) std::memset(a.dumpPressure, 0, n * sizeof(float));
        return FLIP_OK;
    }
    const double ptol = fmax(a.tol, 1e-30) * bmax;
    if (sw.xchgWords < sweep_exchange_words(c.I, c.J, c.K)) {   // the sweeps' exchange array must cover every step
        if (errMsg) *errMsg = "sweep exchange array smaller than the grid needs";
        return FLIP_E_RUNTIME;
    }
    // Sweep tile orientation for this solve: the one whose tiles the rows'
    // extent crosses with the shorter chain of hops.  A hop inside a cluster
    // delays the next tile by about 8 steps (a group of edge terms and its way
    // through shared memory), one between clusters by about 24.
    {
        const int jlo = mail->levelRange[3], jhi = mail->levelRange[4];
        const int klo = mail->levelRange[5], khi = mail->levelRange[6];
        auto lag = [](int lo_, int hi_, int w, int tiles) {
            const int hops = (hi_ - 1) / w - (lo_ - 1) / w, far = (hi_ - 1) / (w * tiles) - (lo_ - 1) / (w * tiles);
            return 8 * (hops - far) + 24 * far;
        };
        const int cost0 = lag(jlo, jhi, SWEEP_WA, SWEEP_CA) + lag(klo, khi, SWEEP_WB, SWEEP_CB);
        const int cost1 = lag(klo, khi, SWEEP_WA, SWEEP_CA) + lag(jlo, jhi, SWEEP_WB, SWEEP_CB);
        int want = cost1 < cost0 ? 1 : (cost0 < cost1 ? 0 : pb.sl.swap);
        if (a.sweepOrientation == 0 || a.sweepOrientation == 1) want = a.sweepOrientation;
        if (want != pb.sl.swap) pb.sl = sweep_layout(c.I, c.J, c.K, want);
    }
    const SweepLayout sl = pb.sl;
    launch_items(c, pb, sw, s);

    // MIC(0) factor; the pivot weights go to A's buffer, which is filled after
    // it: zero wherever no item of this solve writes a coupling
    double *W = reinterpret_cast<double *>(pb.A);
    mic0_factor(c, pb.fluid, pb.Ad, pb.pivotInv, W, W + n, W + 2 * n, pb.factorTicket, sw.err,
                sw.spinLimit ? sw.spinLimit : DEFAULT_SPIN_LIMIT, s);
    PCK(cudaMemsetAsync(pb.A, 0, 8 * (pb.nsl + SWEEP_NP) * sizeof(float), s));
    if (pb.stale) {   // entries off this solve's items are read (and multiplied by zero): finite values only
        PCK(cudaMemsetAsync(pb.z, 0, (pb.nsl + SWEEP_NP) * sizeof(float), s));
        PCK(cudaMemsetAsync(pb.s, 0, (pb.nsl + SWEEP_NP) * sizeof(float), s));
        PCK(cudaMemsetAsync(pb.s2, 0, (pb.nsl + SWEEP_NP) * sizeof(float), s));
    }
    pb.stale = true;   // until this solve has converged
    launch_layout(c, pb, sw, s);

    unsigned long long *rmax = pb.rmaxBits;
    double *zrPartials = pb.partials + PCG_MAX_PARTIALS;
    SweepTiming *tm = a.sweepTiming;
    // sweep pairs timed but not yet added: event pair index q
    auto tally_pair = [&](int q) {
        float ms = 0.0f;
        if (cudaEventElapsedTime(&ms, tm->ev[2 * q], tm->ev[2 * q + 1]) == cudaSuccess) {
            tm->ms += ms;
            tm->launches += 2;
            tm->cellSweeps += 2LL * res->cells;
        } else {
            cudaGetLastError();   // a pair that was not recorded is not an error of the solve
        }
    };
    bool capturing = false;
    // inside a capture the events become graph nodes that record on every replay
    auto record = [&](cudaEvent_t e) {
        if (capturing) cudaEventRecordWithFlags(e, s, cudaEventRecordExternal);
        else cudaEventRecord(e, s);
    };
    // z = M^-1 r, then rho_new = z.r; with `timed` the sweeps sit between
    // event pair q (recorded as graph nodes when captured)
    // (the kernels of an iteration overlap with the end of the one before each)
    auto precondition = [&](int q, bool timed) {
        if (timed) record(tm->ev[2 * q]);
        launch_sweeps(c, sl, pb.L, pb.rh, pb.z, sw, &pb.ctl->done, s, true, q > 0);   // prepared by a kernel before
        if (timed) record(tm->ev[2 * q + 1]);
        launch_after(true, k_dot_zr, rb, TPB, 0, s, pb.items, pb.nItems, pb.z, pb.rh, pb.rl, zrPartials, pb.scal, rmax,
                     pb.ctl, q > 0);
    };
    // one PCG iteration (pcgsolver.h:263-300); every launch is the same for
    // every iteration but the search direction's two buffers, which swap
    // roles each iteration (a batch of PCG_BATCH, an even count, ends where
    // it began); the iteration index lives on the device
    int sPar = 0;
    auto iteration = [&](int k, bool timed) {
        float *sIn = sPar ? pb.s2 : pb.s, *sOut = sPar ? pb.s : pb.s2;
        launch_spmv(pb, sIn, sOut, sw, s);
        launch_after(true, k_update_xr, rb, TPB, 0, s, pb.items, pb.nItems, pb.xh, pb.xl, pb.rh, pb.rl, sOut, pb.qh, pb.ql,
                     pb.partials, pb.scal, rmax, pb.ctl, sw.ticket);
        launch_after(true, k_true_residual, rb, TPB, 0, s, c, sl, pb.items, pb.nItems, pb.fluid, pb.Ad, pb.b, pb.xh, pb.xl,
                     pb.rh, pb.rl, rmax, pb.scal, pb.ctl);
        precondition(1 + k, timed);
        sPar ^= 1;
    };
    static_assert(PCG_BATCH % 2 == 0, "a batch must leave the search direction in the buffer it started from");

    mail->ptol = ptol;
    PCK(cudaMemsetAsync(pb.ctl, 0, sizeof(PcgCtl), s));
    PCK(cudaMemsetAsync(rmax, 0, 2 * sizeof(unsigned long long), s));
    PCK(cudaMemcpyAsync(pb.scal + 6, &mail->ptol, sizeof(double), cudaMemcpyHostToDevice, s));
    sweep_epoch_guard(c, sw, 2, s);
    precondition(0, tm != nullptr);
    PCK(cudaMemcpyAsync(&mail->rho, pb.scal + 1, sizeof(double), cudaMemcpyDeviceToHost, s));
    PCK(cudaMemcpyAsync(&mail->sweepErr, sw.err, sizeof(int), cudaMemcpyDeviceToHost, s));
    PCK(sync());
    if (tm) tally_pair(0);
    const double rho0 = mail->rho;
    bool ok = false;
    int iterations = 0;
    double resid = bmax;
    int sweepErr = mail->sweepErr;   // the factor's or the first sweep's bounded wait gave up
    if (!sweepErr && !(rho0 == 0 || rho0 != rho0)) {
        // Iterations go to the device PCG_BATCH at a time, as one CUDA graph
        // (captured on first use, per context): the convergence test runs
        // there and the kernels of iterations after convergence return at
        // once.  Untimed, the full batches run inside a device-side loop (a
        // conditional WHILE node whose body is a batch and k_pcg_loop), so
        // the host launches the solve once and waits once; timed, or where
        // the loop cannot be built, the host reads the outcome once per
        // batch.  The iterations after the last full batch run eagerly.
        const int gi = tm ? 1 : 0, go = pb.sl.swap;
        int it0 = 0;
        const int maxBatches = a.maxIter / PCG_BATCH;
        if (!tm && !pb.noGraphs && !pb.noLoopGraph && maxBatches > 0) {
            sweep_epoch_guard(c, sw, 2LL * PCG_BATCH * maxBatches, s);
            if (!pb.loopGraph[go]) {
                long long &counter = launch_counter();
                const long long before = counter;
                const unsigned int epochBefore = sw.epoch;
                cudaGraph_t graph = nullptr;
                cudaGraphConditionalHandle handle{};
                bool built = false;
                if (cudaGraphCreate(&graph, 0) == cudaSuccess &&
                    cudaGraphConditionalHandleCreate(&handle, graph, 1, cudaGraphCondAssignDefault) == cudaSuccess) {
                    cudaGraphNodeParams cp{};
                    cp.type = cudaGraphNodeTypeConditional;
                    cp.conditional.handle = handle;
                    cp.conditional.type = cudaGraphCondTypeWhile;
                    cp.conditional.size = 1;
                    cudaGraphNode_t node;
                    if (cudaGraphAddNode(&node, graph, nullptr, nullptr, 0, &cp) == cudaSuccess &&
                        cudaStreamBeginCaptureToGraph(s, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                                      cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
                        capturing = true;
                        for (int k = 0; k < PCG_BATCH; k++) iteration(k, false);
                        { FLIP_COUNT(1); k_pcg_loop<<<1, 1, 0, s>>>(handle, pb.ctl, sw.err); }
                        capturing = false;
                        cudaGraph_t body = nullptr;
                        built = cudaStreamEndCapture(s, &body) == cudaSuccess &&
                                cudaGraphInstantiate(&pb.loopGraph[go], graph, 0) == cudaSuccess;
                    }
                }
                if (graph) cudaGraphDestroy(graph);
                if (!built) {
                    cudaGetLastError();   // no device-side loop here: batches from the host
                    pb.loopGraph[go] = nullptr;
                    pb.noLoopGraph = true;
                }
                pb.loopKernels[go] = counter - before;
                counter = before;   // counted when run
                sw.epoch = epochBefore;
            }
            if (pb.loopGraph[go]) {
                mail->maxBatches = maxBatches;
                PCK(cudaMemcpyAsync(&pb.ctl->maxBatches, &mail->maxBatches, sizeof(int), cudaMemcpyHostToDevice, s));
                PCK(cudaGraphLaunch(pb.loopGraph[go], s));
                PCK(cudaMemcpyAsync(&mail->ctl, pb.ctl, sizeof(PcgCtl), cudaMemcpyDeviceToHost, s));
                PCK(cudaMemcpyAsync(&mail->sweepErr, sw.err, sizeof(int), cudaMemcpyDeviceToHost, s));
                PCK(sync());
                const int ran = mail->ctl.batches;
                launch_counter() += ran * pb.loopKernels[go];
                sw.epoch += 2u * PCG_BATCH * (unsigned int)ran;
                sweepErr = mail->sweepErr;
                resid = mail->ctl.resid;
                if (!sweepErr && mail->ctl.done) {
                    ok = true;
                    iterations = mail->ctl.iters;
                }
                it0 = ran * PCG_BATCH;
            }
        }
        while (!ok && !sweepErr && it0 < a.maxIter) {
            const int nit = std::min(PCG_BATCH, a.maxIter - it0);
            sweep_epoch_guard(c, sw, 2LL * nit, s);
            if (nit == PCG_BATCH && !pb.batchGraph[gi][go] && !pb.noGraphs) {
                long long &counter = launch_counter();
                const long long before = counter;
                const unsigned int epochBefore = sw.epoch;
                if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
                    cudaGetLastError();   // e.g. the legacy default stream: no graphs, launch eagerly
                    pb.noGraphs = true;
                } else {
                    cudaGraph_t graph = nullptr;
                    capturing = true;
                    for (int k = 0; k < PCG_BATCH; k++) iteration(k, tm != nullptr);
                    capturing = false;
                    PCK(cudaStreamEndCapture(s, &graph));
                    cudaError_t e = cudaGraphInstantiate(&pb.batchGraph[gi][go], graph, 0);
                    cudaGraphDestroy(graph);
                    PCK(e);
                    pb.batchKernels[gi][go] = counter - before;
                    counter = before;   // counted when replayed
                    sw.epoch = epochBefore;
                }
            }
            if (nit == PCG_BATCH && pb.batchGraph[gi][go]) {
                PCK(cudaGraphLaunch(pb.batchGraph[gi][go], s));
                launch_counter() += pb.batchKernels[gi][go];
                sw.epoch += 2 * PCG_BATCH;
            } else {
                for (int k = 0; k < nit; k++) iteration(k, tm != nullptr);
            }
            PCK(cudaMemcpyAsync(&mail->ctl, pb.ctl, sizeof(PcgCtl), cudaMemcpyDeviceToHost, s));
            PCK(cudaMemcpyAsync(&mail->sweepErr, sw.err, sizeof(int), cudaMemcpyDeviceToHost, s));
            PCK(sync());
            sweepErr = mail->sweepErr;
            resid = mail->ctl.resid;
            if (tm)   // the sweep pairs that ran: all before convergence
                for (int k = 0; k < nit; k++)
                    if (!mail->ctl.done || it0 + k < mail->ctl.iters - 1) tally_pair(1 + k);
            if (sweepErr) break;
            if (mail->ctl.done) {
                ok = true;
                iterations = mail->ctl.iters;
                break;
            }
            it0 += nit;
        }
        if (!ok) iterations = a.maxIter;
    }
    if (sweepErr) {
        cudaMemsetAsync(sw.err, 0, sizeof(int), s);
        cudaMemsetAsync(sw.xchg, 0, sweep_exchange_words(c.I, c.J, c.K) * sizeof(unsigned long long), s);
        cudaMemsetAsync(sw.ticket, 0, 3 * sizeof(unsigned int), s);
        sw.epoch = 0;
        sync();
        if (errMsg) *errMsg = "a wavefront (factor or sweep) gave up waiting for a neighbouring tile";
        return FLIP_E_DEVICE_TIMEOUT;
    }
    res->iterations = iterations;
    res->residual = resid;
    pb.stale = !ok;
    const bool accept = ok || (iterations == a.maxIter && resid < a.accTol);   // pressuresolver.cpp:810-840
    PCK(cudaMemsetAsync(pb.pressure, 0, n * sizeof(float), s));
    { FLIP_COUNT(1); k_x_to_cells<<<item_ctas(c), TPB, 0, s>>>(c, sl, pb.items, pb.nItems, pb.fluid, pb.xh, pb.xl, pb.pressure); }
    if (a.dumpPressure) {
        PCK(sync());
        PCK(cudaMemcpy(a.dumpPressure, pb.pressure, n * sizeof(float), cudaMemcpyDeviceToHost));
    }
    if (!accept) return FLIP_E_SOLVER_NOCONV;
    long long tot = (long long)(c.I + 1) * c.J * c.K + (long long)c.I * (c.J + 1) * c.K + (long long)c.I * c.J * (c.K + 1);
    float factor = (float)(a.dt / c.dx);
    { FLIP_COUNT(1); k_apply_pressure<<<div_up(tot, TPB), TPB, 0, s>>>(c, a.phi, a.wu, a.wv, a.ww, pb.pressure, factor,
                                                                    a.u, a.v, a.w, a.vu, a.vv, a.vw); }
    res->applied = true;
    return FLIP_OK;
}

}  // namespace flip
