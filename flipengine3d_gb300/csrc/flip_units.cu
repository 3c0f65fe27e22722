// Steps of the solvers on their own, through the C ABI, so that each can be
// checked apart from a frame.  The same kernels and launch sequences as inside
// one; only the data comes from host arrays in flat order.
//
// The MIC(0) preconditioner: the factor
// (factorModifiedIncompleteColesky0, pcgsolver.h:70-185) and the two
// triangular sweeps (solveLower / solveLowerTransposeInPlace,
// pcgsolver.h:192-221) that the pressure solve runs, on rows the caller
// gives: arbitrary 7-point matrices.  The product A s of the solve's loop, on such
// rows.  The viscosity step: the field that it
// makes of any level sets and velocities.
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/flip3d.h"
#include "flip_device.cuh"

namespace flip {
int record_error(int code, const std::string &msg);   // sets flip_last_error()
}

using namespace flip;

namespace {

// Device buffers of one call, freed on every exit path.
struct Scratch {
    std::vector<void *> ptrs;
    ~Scratch() {
        for (void *p : ptrs) cudaFree(p);
    }
    template <class T>
    bool get(T **p, size_t count) {
        if (cudaMalloc((void **)p, std::max<size_t>(count, 1) * sizeof(T)) != cudaSuccess) return false;
        ptrs.push_back((void *)*p);
        return true;
    }
};

int cuda_status(cudaError_t e, const char *what) {
    if (e == cudaSuccess) return FLIP_OK;
    return record_error(FLIP_E_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

// The rows must form a system the pressure solve could build: flagged cells
// interior (1..n-2 on every axis) and couplings only between flagged cells.
int check_system(int I, int J, int K, const uint8_t *fluid) {
    if (I < 3 || J < 3 || K < 3) return record_error(FLIP_E_DOMAIN, "grid must be at least 3 cells on each axis");
    if ((long long)I * J * K >= (1LL << 28)) return record_error(FLIP_E_DOMAIN, "grid too large");
    for (int k = 0; k < K; k++)
        for (int j = 0; j < J; j++)
            for (int i = 0; i < I; i++) {
                const bool interior = i >= 1 && j >= 1 && k >= 1 && i <= I - 2 && j <= J - 2 && k <= K - 2;
                if (fluid[i + (size_t)I * (j + (size_t)J * k)] && !interior)
                    return record_error(FLIP_E_DOMAIN, "a flagged cell lies on the grid border");
            }
    return FLIP_OK;
}

StepConsts grid_consts(int I, int J, int K) {
    StepConsts c{};
    c.I = I; c.J = J; c.K = K;
    return c;
}

}  // namespace

extern "C" int flip_mic0_factor(int I, int J, int K, const uint8_t *fluid, const double *rows, double *invdiag) {
    if (!fluid || !rows || !invdiag) return record_error(FLIP_E_NULL, "null pointer");
    int rc = check_system(I, J, K, fluid);
    if (rc) return rc;
    const size_t n = (size_t)I * J * K;
    const bool any = std::find_if(fluid, fluid + n, [](uint8_t f) { return f != 0; }) != fluid + n;
    std::memset(invdiag, 0, n * sizeof(double));
    if (!any) return FLIP_OK;
    Scratch sc;
    uint8_t *dFluid;
    double4_32a *dAd;
    double *dInv, *dW;
    int *dErr;
    unsigned int *dTicket;
    if (!sc.get(&dFluid, n) || !sc.get(&dAd, n) || !sc.get(&dInv, n) || !sc.get(&dW, 3 * n) ||
        !sc.get(&dErr, 1) || !sc.get(&dTicket, 1))
        return record_error(FLIP_E_NOMEM, "cudaMalloc failed");
    cudaStream_t s = nullptr;
    if ((rc = cuda_status(cudaMemcpy(dFluid, fluid, n, cudaMemcpyHostToDevice), "copy flags")) ||
        (rc = cuda_status(cudaMemcpy(dAd, rows, n * sizeof(double4_32a), cudaMemcpyHostToDevice), "copy rows")) ||
        (rc = cuda_status(cudaMemset(dInv, 0xff, n * sizeof(double)), "clear")) ||
        (rc = cuda_status(cudaMemset(dErr, 0, sizeof(int)), "clear")))
        return rc;
    mic0_factor(grid_consts(I, J, K), dFluid, dAd, dInv, dW, dW + n, dW + 2 * n, dTicket, dErr, DEFAULT_SPIN_LIMIT, s);
    mic0_inverse_pivots(dFluid, n, dInv, s);
    if ((rc = cuda_status(cudaDeviceSynchronize(), "factor"))) return rc;
    int err = 0;
    if ((rc = cuda_status(cudaMemcpy(&err, dErr, sizeof(int), cudaMemcpyDeviceToHost), "read flag"))) return rc;
    if (err) return record_error(FLIP_E_DEVICE_TIMEOUT, "the factor's wavefront gave up waiting");
    return cuda_status(cudaMemcpy(invdiag, dInv, n * sizeof(double), cudaMemcpyDeviceToHost), "read pivots");
}

extern "C" int flip_mic0_pivot_functions(int n, const double *d, const float *guess_off, double *reciprocal, double *root) {
    if (n < 0) return record_error(FLIP_E_DOMAIN, "negative count");
    if (n == 0) return FLIP_OK;
    if (!d || !guess_off || !reciprocal || !root) return record_error(FLIP_E_NULL, "null pointer");
    Scratch sc;
    double *dd, *dr, *ds;
    float *doff;
    const size_t bytes = (size_t)n * sizeof(double);
    if (!sc.get(&dd, n) || !sc.get(&dr, n) || !sc.get(&ds, n) || !sc.get(&doff, n))
        return record_error(FLIP_E_NOMEM, "cudaMalloc failed");
    int rc;
    if ((rc = cuda_status(cudaMemcpy(dd, d, bytes, cudaMemcpyHostToDevice), "copy")) ||
        (rc = cuda_status(cudaMemcpy(doff, guess_off, (size_t)n * sizeof(float), cudaMemcpyHostToDevice), "copy")))
        return rc;
    launch_pivot_functions(n, dd, doff, dr, ds, nullptr);
    if ((rc = cuda_status(cudaMemcpy(reciprocal, dr, bytes, cudaMemcpyDeviceToHost), "pivot functions"))) return rc;
    return cuda_status(cudaMemcpy(root, ds, bytes, cudaMemcpyDeviceToHost), "read");
}

extern "C" int flip_mic0_precondition(int I, int J, int K, const uint8_t *fluid, const float *factor, const float *r,
                                      float *z, int orientation) {
    if (!fluid || !factor || !r || !z) return record_error(FLIP_E_NULL, "null pointer");
    if (orientation < 0 || orientation > 1) return record_error(FLIP_E_OUT_OF_RANGE, "orientation must be 0 or 1");
    int rc = check_system(I, J, K, fluid);
    if (rc) return rc;
    const size_t n = (size_t)I * J * K;
    const SweepLayout g = sweep_layout(I, J, K, orientation);
    const long long nsl = sweep_layout_size(I, J, K);
    // the rows and right-hand side of the interior cells into the sweep layout
    std::vector<float4> hL((size_t)nsl, make_float4(0.f, 0.f, 0.f, 0.f));
    std::vector<float> hr((size_t)nsl, 0.0f), hz((size_t)nsl, 0.0f);
    for (int k = 1; k <= K - 2; k++)
        for (int j = 1; j <= J - 2; j++)
            for (int i = 1; i <= I - 2; i++) {
                const size_t t = i + (size_t)I * (j + (size_t)J * k);
                const long long e = sweep_index(g, i, j, k);
                if (fluid[t]) hL[e] = make_float4(factor[4 * t], factor[4 * t + 1], factor[4 * t + 2], factor[4 * t + 3]);
                hr[e] = fluid[t] ? r[t] : 0.0f;
            }
    Scratch sc;
    uint8_t *dFluid;
    float4 *dL;
    float *dR, *dZ;
    int *dSkip;
    SweepState sw{};
    const int nt = sweep_tiles_max(I, J, K);
    const long long nw = sweep_exchange_words(I, J, K);
    if (!sc.get(&dFluid, n) || !sc.get(&dL, nsl) || !sc.get(&dR, nsl) || !sc.get(&dZ, nsl) || !sc.get(&dSkip, 1) ||
        !sc.get(&sw.range, nt) || !sc.get(&sw.xchg, nw) || !sc.get(&sw.ticket, 4) || !sc.get(&sw.err, 4))
        return record_error(FLIP_E_NOMEM, "cudaMalloc failed");
    sw.xchgWords = nw;
    if ((rc = cuda_status(cudaMemcpy(dFluid, fluid, n, cudaMemcpyHostToDevice), "copy flags")) ||
        (rc = cuda_status(cudaMemcpy(dL, hL.data(), nsl * sizeof(float4), cudaMemcpyHostToDevice), "copy rows")) ||
        (rc = cuda_status(cudaMemcpy(dR, hr.data(), nsl * sizeof(float), cudaMemcpyHostToDevice), "copy rhs")) ||
        (rc = cuda_status(cudaMemset(dZ, 0, nsl * sizeof(float)), "clear")) ||
        (rc = cuda_status(cudaMemset(dSkip, 0, sizeof(int)), "clear")) ||
        (rc = cuda_status(cudaMemset(sw.xchg, 0, nw * sizeof(unsigned long long)), "clear")) ||
        (rc = cuda_status(cudaMemset(sw.ticket, 0, 4 * sizeof(unsigned int)), "clear")) ||
        (rc = cuda_status(cudaMemset(sw.err, 0, 4 * sizeof(int)), "clear")))
        return rc;
    const StepConsts c = grid_consts(I, J, K);
    cudaStream_t s = nullptr;
    launch_sweep_ranges(c, g, dFluid, sw, s);
    launch_sweeps(c, g, dL, dR, dZ, sw, dSkip, s);
    if ((rc = cuda_status(cudaDeviceSynchronize(), "sweeps"))) return rc;
    int err = 0;
    if ((rc = cuda_status(cudaMemcpy(&err, sw.err, sizeof(int), cudaMemcpyDeviceToHost), "read flag"))) return rc;
    if (err) return record_error(FLIP_E_DEVICE_TIMEOUT, "a sweep tile gave up waiting");
    if ((rc = cuda_status(cudaMemcpy(hz.data(), dZ, nsl * sizeof(float), cudaMemcpyDeviceToHost), "read result")))
        return rc;
    for (size_t t = 0; t < n; t++) z[t] = 0.0f;
    for (int k = 1; k <= K - 2; k++)
        for (int j = 1; j <= J - 2; j++)
            for (int i = 1; i <= I - 2; i++) {
                const size_t t = i + (size_t)I * (j + (size_t)J * k);
                if (fluid[t]) z[t] = hz[sweep_index(g, i, j, k)];
            }
    return FLIP_OK;
}

extern "C" int flip_pressure_apply(int I, int J, int K, const uint8_t *fluid, const double *rows, const float *z,
                                   const float *s, float beta, int orientation, float *s_out, double *q, double *dot) {
    if (!fluid || !rows || !z || !s || !s_out || !q || !dot) return record_error(FLIP_E_NULL, "null pointer");
    if (orientation < 0 || orientation > 1) return record_error(FLIP_E_OUT_OF_RANGE, "orientation must be 0 or 1");
    int rc = check_system(I, J, K, fluid);
    if (rc) return rc;
    const size_t n = (size_t)I * J * K;
    const SweepLayout g = sweep_layout(I, J, K, orientation);
    const size_t nsl = (size_t)sweep_layout_size(I, J, K), pad = nsl + SWEEP_NP;
    std::vector<float> hz(pad, 0.0f), hs(pad, 0.0f), hq(2 * nsl);
    bool any = false;
    auto rows_of = [&](auto f) {
        for (int k = 1; k <= K - 2; k++)
            for (int j = 1; j <= J - 2; j++)
                for (int i = 1; i <= I - 2; i++) {
                    const size_t t = i + (size_t)I * (j + (size_t)J * k);
                    if (fluid[t]) f(t, (size_t)sweep_index(g, i, j, k));
                }
    };
    rows_of([&](size_t t, size_t e) {
        hz[e] = z[t];
        hs[e] = s[t];
        any = true;
    });
    std::memset(s_out, 0, n * sizeof(float));
    std::memset(q, 0, n * sizeof(double));
    *dot = 0.0;
    if (!any) return FLIP_OK;
    Scratch sc;
    PressureBuffers pb{};
    pb.sl = g;
    pb.nsl = (long long)nsl;
    pb.nPartials = pressure_partials_for(I, J, K);
    SweepState sw{};
    const std::vector<double> ones(n, 1.0);
    if (!sc.get(&pb.fluid, n) || !sc.get(&pb.items, sweep_items_max(I, J, K)) || !sc.get(&pb.nItems, 4) || !sc.get(&pb.Ad, n) ||
        !sc.get(&pb.b, n) || !sc.get(&pb.pivotInv, n) || !sc.get(&pb.L, nsl) || !sc.get(&pb.A, 8 * pad) || !sc.get(&pb.xh, nsl) ||
        !sc.get(&pb.xl, nsl) || !sc.get(&pb.rh, nsl) || !sc.get(&pb.rl, nsl) || !sc.get(&pb.qh, nsl) || !sc.get(&pb.ql, nsl) ||
        !sc.get(&pb.z, pad) || !sc.get(&pb.s, pad) || !sc.get(&pb.s2, pad) || !sc.get(&pb.partials, 2 * PCG_MAX_PARTIALS) ||
        !sc.get(&pb.scal, 8) || !sc.get(&pb.ctl, 1) || !sc.get(&sw.range, sweep_tiles_max(I, J, K)) || !sc.get(&sw.ticket, 4) ||
        !sc.get(&sw.err, 4))
        return record_error(FLIP_E_NOMEM, "cudaMalloc failed");
    auto put = [&](void *to, const void *from, size_t bytes) { return cuda_status(cudaMemcpy(to, from, bytes, cudaMemcpyHostToDevice), "copy"); };
    auto clear = [&](void *p, size_t bytes) { return cuda_status(cudaMemset(p, 0, bytes), "clear"); };
    if ((rc = put(pb.fluid, fluid, n)) || (rc = put(pb.Ad, rows, n * sizeof(double4_32a))) ||
        (rc = put(pb.pivotInv, ones.data(), n * sizeof(double))) || (rc = clear(pb.b, n * sizeof(double))) ||
        (rc = clear(pb.A, 8 * pad * sizeof(float))) || (rc = clear(sw.ticket, 4 * sizeof(unsigned))) || (rc = clear(sw.err, 4 * sizeof(int))))
        return rc;
    StepConsts c = grid_consts(I, J, K);
    cudaStream_t st = nullptr;
    launch_items(c, pb, sw, st);
    launch_layout(c, pb, sw, st);
    // the second iteration of a solve whose z.r was 1 and is beta
    PcgCtl ctl{};
    ctl.it = 1;
    std::vector<double> zr(PCG_MAX_PARTIALS, 0.0), scal(8, 0.0), sums(pb.nPartials);
    zr[0] = beta;
    scal[3] = 1.0;
    if ((rc = put(pb.z, hz.data(), pad * 4)) || (rc = put(pb.s, hs.data(), pad * 4)) || (rc = put(pb.ctl, &ctl, sizeof(ctl))) ||
        (rc = put(pb.partials + PCG_MAX_PARTIALS, zr.data(), zr.size() * 8)) || (rc = put(pb.scal, scal.data(), 64)))
        return rc;
    launch_spmv(pb, pb.s, pb.s2, sw, st);
    if ((rc = cuda_status(cudaDeviceSynchronize(), "product"))) return rc;
    int nItems = 0, err = 0;
    auto get = [&](void *to, const void *from, size_t bytes) { return cuda_status(cudaMemcpy(to, from, bytes, cudaMemcpyDeviceToHost), "read"); };
    if ((rc = get(&nItems, pb.nItems, sizeof(int))) || (rc = get(&err, sw.err, sizeof(int))) || (rc = get(hs.data(), pb.s2, nsl * 4)) ||
        (rc = get(hq.data(), pb.qh, nsl * 4)) || (rc = get(hq.data() + nsl, pb.ql, nsl * 4)) ||
        (rc = get(sums.data(), pb.partials, sums.size() * 8)))
        return rc;
    if (err) return record_error(FLIP_E_DEVICE_TIMEOUT, "a copy into shared memory did not arrive");
    rows_of([&](size_t t, size_t e) {
        s_out[t] = hs[e];
        q[t] = (double)hq[e] + (double)hq[nsl + e];
    });
    for (int b = 0; b < std::min(pb.nPartials, nItems); b++) *dot += sums[b];
    return FLIP_OK;
}

extern "C" int flip_viscosity_step(int I, int J, int K, double dx, const float *liquid_phi, const float *solid_phi, float *u,
                                   float *v, float *w, double viscosity, double dt, long long *rows, int *iterations,
                                   double *residual) {
    if (!liquid_phi || !solid_phi || !u || !v || !w) return record_error(FLIP_E_NULL, "null pointer");
    if (I < 3 || J < 3 || K < 3) return record_error(FLIP_E_DOMAIN, "grid must be at least 3 cells on each axis");
    if ((long long)I * J * K >= (1LL << 28)) return record_error(FLIP_E_DOMAIN, "grid too large");
    if (!(dx > 0.0) || !(viscosity >= 0.0) || !(dt >= 0.0)) return record_error(FLIP_E_DOMAIN, "cell size, viscosity or time step");
    const size_t nodes = (size_t)(I + 1) * (J + 1) * (K + 1), cells = (size_t)I * J * K;
    for (int k = 0; k <= K; k++)
        for (int j = 0; j <= J; j++)
            for (int i = 0; i <= I; i++) {
                const bool wall = i <= 1 || j <= 1 || k <= 1 || i >= I - 1 || j >= J - 1 || k >= K - 1;
                if (wall && !(solid_phi[i + (size_t)(I + 1) * (j + (size_t)(J + 1) * k)] < 0.0f))
                    return record_error(FLIP_E_DOMAIN, "a cell on the grid border is not solid");
            }
    long long nf, nn, ncorner, vol[7], rowBlocks, slotWords;
    viscosity_buffer_sizes(I, J, K, &nf, &nn, &ncorner, vol, &rowBlocks, &slotWords);
    const size_t n[3] = {(size_t)(I + 1) * J * K, (size_t)I * (J + 1) * K, (size_t)I * J * (K + 1)};
    Scratch sc;
    ViscosityBuffers b{};
    float *phi, *solid, *f[3], *host[3] = {u, v, w};
    bool ok = sc.get(&b.fluidFace, nf) && sc.get(&b.valid, nn) && sc.get(&b.valid2, nn) && sc.get(&b.inSys, nf) &&
              sc.get(&b.coefs, 8 * nf) && sc.get(&b.x, nf) && sc.get(&b.r, nf) && sc.get(&b.zp, nf) && sc.get(&b.p, nf) &&
              sc.get(&b.q, nf) && sc.get(&b.list, nf) && sc.get(&b.blockRows, rowBlocks) && sc.get(&b.slots, slotWords) &&
              sc.get(&b.scal, 8) && sc.get(&phi, cells) && sc.get(&solid, nodes);
    for (int g = 0; g < 7; g++) ok = ok && sc.get(&b.vol[g], vol[g]) && sc.get(&b.node[g], ncorner);
    for (int d = 0; d < 3; d++) ok = ok && sc.get(&f[d], n[d]);
    if (!ok) return record_error(FLIP_E_NOMEM, "cudaMalloc failed");
    int rc;
    if ((rc = cuda_status(cudaMemcpy(phi, liquid_phi, cells * 4, cudaMemcpyHostToDevice), "copy level set")) ||
        (rc = cuda_status(cudaMemcpy(solid, solid_phi, nodes * 4, cudaMemcpyHostToDevice), "copy level set")))
        return rc;
    for (int d = 0; d < 3; d++)
        if ((rc = cuda_status(cudaMemcpy(f[d], host[d], n[d] * 4, cudaMemcpyHostToDevice), "copy velocities"))) return rc;
    StepConsts c = grid_consts(I, J, K);
    c.dx = dx;
    ViscosityResult res{};
    if ((rc = viscosity_apply(c, b, phi, solid, f[0], f[1], f[2], viscosity, dt, 0, false, &res, nullptr)))
        return rc;
    for (int d = 0; d < 3; d++)
        if ((rc = cuda_status(cudaMemcpy(host[d], f[d], n[d] * 4, cudaMemcpyDeviceToHost), "read velocities"))) return rc;
    if (rows) *rows = res.rows;
    if (iterations) *iterations = res.iterations;
    if (residual) *residual = res.residual;
    return FLIP_OK;
}
