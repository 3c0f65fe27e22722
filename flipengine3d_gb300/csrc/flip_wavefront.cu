// MIC(0) triangular sweeps as a pipelined wavefront (sm_103a).
//
// The preconditioner solve of the reference, solveLower followed by
// solveLowerTransposeInPlace (pcgsolver.h:192-221), over the 7-point factor:
//   forward   y_c = inv_c * (r_c - Lz_{c-z} y_{c-z} - Ly_{c-y} y_{c-y} - Lx_{c-x} y_{c-x})
//   backward  z_c = inv_c * (y_c - Lx_c z_{c+x} - Ly_c z_{c+y} - Lz_c z_{c+z})
// with the subtractions in the reference's column order and FP32 rounding
// of every product and difference.  A cell depends on its three lower
// (upper) neighbours only, so the cells of a plane i + j + k = const are
// independent: the exact wavefront order.
//
// What bounds it: the dependency chain.  A sweep cannot take fewer steps than
// the system's extent i + j + k; everything above that is time per step and
// the delay with which one tile's edge terms reach the next.
//
// Mapping.  A tile is 16 (a) x 8 (b) pencils along i, worked by four warps of
// 8 x 4 pencils, a pencil per lane.  In the forward sweep pencil (A, B) meets
// cell i = 1 + t - A - B at step t, so a cell's three lower neighbours were
// all formed at step t - 1: in the lane itself, or in the lane before it along
// a or b (two shuffles a step).  The warps of a tile share the step numbers
// and run on four schedulers without a barrier; each waits only for the terms
// of its own edge pencils.  A step is bound by the latencies of one warp's
// instructions (about 85 cycles, and some 30 more for its part of the group's and
// the chunk's waits); bundles of 2 x 2 pencils per lane, one warp a tile, took 205
// cycles a step and saved fewer hops than that costs.  128 pencils
// per CTA rather than more: a step reads 20 and writes 4 bytes per pencil, and
// 3 KB a step is what one SM can draw from L2 in the time of a step.  In the
// forward sweep a cell hands its neighbours the finished products L_c * y_c
// rather than y_c: each product is rounded once, by whichever thread forms
// it, so the bits are the reference's.
//
// Edges.  Every term that crosses to another warp has a word of its own in
// the consumer's shared memory for the whole sweep (so no credit flows back),
// laid out so that one 16-byte load takes a pencil's terms of EC = 4 steps.
// The words start as a bit pattern that no product can have (a NaN payload;
// FP32 products give the canonical NaN only), and the consumer looks at its
// words until the pattern is gone.  Eight tiles (2 x 4: 32 x 32 pencils) form
// a thread-block cluster, in which the edge lanes store straight into the
// consumer's shared memory: a hop costs the group of steps and a few hundred
// cycles.  Between clusters a term travels as one 64-bit word {sweep epoch,
// value} in global memory, indexed by step; the consumer's four edge warps
// poll the words of their groups of steps until the epoch is the current
// sweep's.  Naturally aligned words are seen whole or not at all, so no fence
// or flag sits between producer and consumer.
//
// Data movement.  The factor rows and the right-hand side live in the
// step-major sweep layout (flip_device.cuh), so the 8 steps of a chunk of a
// tile are one contiguous block in either direction.  A loader thread moves
// whole chunks with bulk asynchronous copies into a ring of shared-memory
// slots, and prefetches the chunk one ring further ahead into L2.  Cells
// outside the grid or the system have zero rows, so a step is unpredicated.
//
// Clusters take tickets in dependency order, so a tile only waits for tiles
// that are already running (a cluster's own CTAs run together).  Every wait
// is bounded: on timeout the tile raises the error flag and stops, and the
// host reports FLIP_E_DEVICE_TIMEOUT; no wait can spin forever.  A CTA that
// gives up stays until the other CTAs of its cluster are done, since they may
// still store into its shared memory.
//
// A group of four steps tests its edge words on a vote: the words are loaded two
// steps ahead and the vote taken one step ahead, inside the latency of the step
// before (as the group's first act it cost 170 cycles, two steps' worth), and the
// shuffles a step waits for are issued before the last one's stores.
//
// Measured per launch (events around a pair, in the frames): 128^3 dam break (518k
// rows) 39.0 us, 64^3 (58k rows) 19.6 us, 256 x 128 x 128 tank (1.8M rows) 50.7 us;
// the form before it (tiles of 32 x 8 pencils, four warps in lockstep with a barrier
// a step, every edge through L2) took 53.2, 25.6 and 71.4 us on the same box, and the
// look ahead saved 2.5, 1.2 and 3.4.
#include <atomic>
#include <type_traits>

#include "flip_device.cuh"

namespace flip {

namespace {

constexpr int WA = SWEEP_WA, WB = SWEEP_WB, NP = SWEEP_NP, CH = SWEEP_CH;
constexpr int VA = SWEEP_VA, VB = SWEEP_VB;                 // pencils of a warp along a and b
constexpr int NWA = WA / VA, NWB = WB / VB, NWC = NWA * NWB;   // compute warps of a tile
static_assert(VA == 8 && VB == 4 && NWA == 2 && NWB == 2 && CH == 8, "lane and warp mapping");
constexpr int CA = SWEEP_CA, CB = SWEEP_CB, CL = CA * CB;   // tiles of a cluster along a and b
constexpr int EC = 4;        // steps per group of edge words
#ifndef SWEEP_NBUF
#define SWEEP_NBUF 4   // operand slots in shared memory, 8 steps each
#endif
constexpr int NBUF = SWEEP_NBUF;
static_assert(NBUF >= 2, "the ring needs a slot in flight beside the one in use");
constexpr int NHELP = 4;     // edge warps: groups of steps polled at the same time
constexpr int LOADER = NWC, EDGE = LOADER + 1, NTHREADS = 32 * (EDGE + NHELP);
// The edge words of every step fit beside the operand slots up to this many
// steps; longer grids (I above about 700) keep a ring of RC chunks of them
// instead, and take every term of another tile from global memory.  A warp is
// less than NBUF chunks ahead of the slowest warp of its tile (the operand
// slots) and hands on terms of at most one chunk further.
constexpr int WHOLE_STEPS = 720, RC = NBUF + 2;
constexpr int GW = (VA + VB) * EC;   // edge words of a warp per group: VB a-edge pencils, then VA b-edge pencils
constexpr unsigned ABSENT = 0xffffffffu;   // a word that has not come (the largest unsigned value)
// Waiting for this CTA's own bulk copies in flight (they complete by
// themselves) keeps the default limit, whatever limit the edge waits have.
constexpr unsigned int DRAIN_SPIN_LIMIT = DEFAULT_SPIN_LIMIT;

struct SweepArgs {
    const float4 *L;               // factor rows, sweep layout
    const float *rin;              // right-hand side, sweep layout (backward: the forward result)
    float *out;                    // result, sweep layout (backward: in place over the forward result)
    int T;                         // steps per tile, a multiple of CH
    int nta, ntb, nca;             // tiles along a and b, clusters along a
    int nClusters;
    const int2 *range;             // per tile: first/last step (forward numbering) holding a system cell
    unsigned long long *xchg;      // per tile: T x WB a-edge words, then T x WA b-edge words
    unsigned int *ticket;          // [0] forward cluster tickets, [1] the pair's epoch, [2] backward cluster tickets
                                   // (set by sweep_prep before each pair)
    int *err;
    const int *skip;   // nonzero: return at once
    unsigned int spinLimit;    // poll rounds before a wait gives up
    unsigned int epochSkew;    // 0; nonzero only to make the edge waits run out (fault injection)
};

struct Slot {
    float4 L[CH][NP];   // rows in layout order: forward row q = step q, backward row q = step CH-1-q
    float r[CH][NP];
};
struct SweepSmem {
    Slot slot[NBUF];
    unsigned long long loaded[NBUF], done[NBUF];   // per slot: operand bytes in; chunk done
    int abort;
    int cluster;
    unsigned int epoch;
    int pad;
    float unused[NWC][32 + 2 * GW];   // where lanes and steps without a taker store their terms
};
// after it: per warp, the edge words that come in, [group][pencil][step of the group]
__host__ __device__ constexpr size_t sweep_smem_bytes(int edgeSteps) {
    return sizeof(SweepSmem) + ((size_t)NWC * (edgeSteps / EC) + CH / EC) * GW * 4;   // a chunk more may be read
}
static_assert(sweep_smem_bytes(WHOLE_STEPS) <= 227 * 1024, "the sweep's shared memory fits one CTA");
static_assert(sizeof(SweepSmem) % 16 == 0 && WHOLE_STEPS % CH == 0, "alignment of the edge words");

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void mb_init(unsigned b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(count) : "memory");
}
__device__ __forceinline__ void mb_arrive_relaxed(unsigned on, unsigned b) {
    asm volatile("{\n .reg .b64 st;\n .reg .pred q;\n setp.ne.u32 q, %1, 0;\n"
                 " @q mbarrier.arrive.relaxed.cta.shared::cta.b64 st, [%0];\n}" ::"r"(b), "r"(on) : "memory");
}
__device__ __forceinline__ void mb_arrive_release(unsigned on, unsigned b) {
    asm volatile("{\n .reg .b64 st;\n .reg .pred q;\n setp.ne.u32 q, %1, 0;\n"
                 " @q mbarrier.arrive.release.cta.shared::cta.b64 st, [%0];\n}" ::"r"(b), "r"(on) : "memory");
}
__device__ __forceinline__ void mb_arrive_expect_tx(unsigned b, unsigned bytes) {
    asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 st, [%0], %1;\n}" ::"r"(b), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mb_test(unsigned b, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(b), "r"(parity) : "memory");
    return ok != 0;
}
// A look ahead: the same without ordering anything.
__device__ __forceinline__ unsigned mb_peek(unsigned b, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(b), "r"(parity));
    return ok;
}
// One round of waiting for a phase: the thread is suspended until the phase
// completes or about `ns` nanoseconds pass, so waiting warps take no issue
// slots from the warps that compute on the same scheduler.
__device__ __forceinline__ bool mb_try(unsigned b, unsigned parity, unsigned ns) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
                 " selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(b), "r"(parity), "r"(ns) : "memory");
    return ok != 0;
}
// Bounded wait for a phase of an mbarrier; false on abort or timeout (which
// raises the abort and error flags).
__device__ __noinline__ bool mb_wait_slow(unsigned b, unsigned parity, int *abortFlag, int *err, unsigned int limit) {
    for (unsigned int spin = 0; spin < limit; spin++) {
        if (mb_try(b, parity, 256)) return true;
        if (*(volatile int *)abortFlag) return false;
        if ((spin & 255u) == 255u && *(volatile int *)err) return false;   // another tile gave up
    }
    *(volatile int *)abortFlag = 1;
    atomicExch(err, 1);
    return false;
}
__device__ __forceinline__ bool mb_wait(unsigned b, unsigned parity, int *abortFlag, int *err, unsigned int limit) {
    return mb_try(b, parity, 256) || mb_wait_slow(b, parity, abortFlag, err, limit);
}
// The same for a whole warp, which goes on or stops together.
__device__ __forceinline__ bool warp_wait(unsigned b, unsigned parity, int *abortFlag, int *err, unsigned int limit) {
    if (__all_sync(0xffffffffu, mb_try(b, parity, 256))) return true;
    return __all_sync(0xffffffffu, mb_wait_slow(b, parity, abortFlag, err, limit));
}
// After `spin` looks at edge words that have not come: does the warp stop?
// Looks are about a shared-memory round trip apart, then a suspension; the
// limit counts the suspended ones, as mb_wait does.
__device__ __noinline__ bool edge_gives_up(unsigned spin, int *abortFlag, int *err, unsigned int limit) {
    if (spin < 64) return false;
    __nanosleep(spin < 1024 ? 32 : 256);
    const bool stop = *(volatile int *)abortFlag || ((spin & 255u) == 255u && *(volatile int *)err);
    if (!__any_sync(0xffffffffu, stop || spin - 64 >= limit)) return false;
    if (!__any_sync(0xffffffffu, stop)) atomicExch(err, 1);
    return true;
}
// bulk copy global -> shared, completion counted in bytes on mbarrier b
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, unsigned b) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(b) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void *src, unsigned bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned map_rank(unsigned addr, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ int ld_cluster(unsigned addr) {
    int v;
    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
// An edge term stored into a CTA's shared memory (this one's or another of its
// cluster); and, where `on` holds, as a word of the exchange array.  Ordered
// against nothing else (the reader looks at the word itself), so the compiler
// may move the loads of later steps above them.
template <int OFF>
__device__ __forceinline__ void hand_on(unsigned addr, float v) {
    asm volatile("st.relaxed.cluster.shared::cluster.f32 [%0 + %2], %1;" ::"r"(addr), "f"(v), "n"(OFF));
}
__device__ __forceinline__ void publish(unsigned on, unsigned long long *p, unsigned epoch, float v) {
    asm volatile("{\n .reg .pred q;\n setp.ne.u32 q, %2, 0;\n @q st.relaxed.gpu.global.u64 [%0], %1;\n}"
                 ::"l"(p), "l"(((unsigned long long)epoch << 32) | __float_as_uint(v)), "r"(on));
}
// A pencil's edge words of a group.
__device__ __forceinline__ uint4 ld_edge(unsigned addr) {
    uint4 v;
    asm volatile("ld.volatile.shared::cta.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void clear_edge(unsigned addr) {
    asm volatile("st.volatile.shared::cta.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(addr), "r"(ABSENT) : "memory");
}
__device__ __forceinline__ bool any_absent(uint4 a, uint4 b) {
    return max(max(max(a.x, a.y), max(a.z, a.w)), max(max(b.x, b.y), max(b.z, b.w))) == ABSENT;
}

// What a compute warp works with (see k_wavefront).
struct WarpJob {
    SweepSmem *sm;
    int *err;
    unsigned spinLimit;
    int c0, nChunks, lane;
    const float4 *L;              // this lane's operands in slot 0, row 0
    const float *r;
    float *out;                   // result of this lane at the tile's step 0
    int lastStep;                 // T - 1
    bool inEdgeA, inEdgeB;
    unsigned inA, inB;            // this lane's edge words (of chunk 0)
    unsigned dstA, dstB;          // where it hands terms on: the consumer's words, moved to this warp's chunk 0
    unsigned unused;              // and where to at other steps
    // {first, count} of the chunks whose steps 0-6, and whose step 7, hand a term on
    int2 kA, kA7, kB, kB7;
    unsigned long long *xA, *xB;  // as words of the exchange array,
    int2 pA, pA7, pB, pB7;        // in these
    unsigned epoch;
};

// The steps of one warp.  PUB: it also publishes words for another cluster.
template <bool FWD, bool SWAP, bool WHOLE, bool PUB>
__device__ __forceinline__ bool run_steps(const WarpJob &w) {
    constexpr unsigned CHB = (CH / EC) * GW * 4;   // edge bytes of a chunk
    // forward: the products of the last cell, for the next one along i, a and
    // b; backward: its z, which all three take
    float tx = 0.0f, sA = 0.0f, sB = 0.0f, nA = 0.0f, nB = 0.0f;
    // the edge words of the next group, read ahead
    uint4 na = ld_edge(w.inA + (WHOLE ? w.c0 * CHB : 0)), nb = ld_edge(w.inB + (WHOLE ? w.c0 * CHB : 0));
    unsigned ready = 0;   // the next chunk's operands were seen to be in
    bool miss = __any_sync(0xffffffffu, any_absent(na, nb));   // words of the next group had not come
    float *out = w.out + (ptrdiff_t)(FWD ? w.c0 * CH : w.lastStep - w.c0 * CH) * NP;
    unsigned long long *xA = w.xA + (size_t)w.c0 * CH * WB, *xB = w.xB + (size_t)w.c0 * CH * WA;
    unsigned cw = WHOLE ? w.c0 * CHB : 0;   // the chunk's edge words
#pragma unroll 1
    for (int n = 0; n < w.nChunks; n++) {
        const int b = n % NBUF, c = w.c0 + n;
        if (!__all_sync(0xffffffffu, ready) &&
            !warp_wait(smem_addr(&w.sm->loaded[b]), (n / NBUF) & 1, &w.sm->abort, w.err, w.spinLimit))
            return false;
        asm volatile("" ::: "memory");
        const float4 *L = reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(w.L) + (size_t)b * sizeof(Slot));
        const float *r = reinterpret_cast<const float *>(reinterpret_cast<const char *>(w.r) + (size_t)b * sizeof(Slot));
        // a step's terms are taken one step later: step 7's fall into the next chunk
        const unsigned cw1 = WHOLE ? cw + CHB : ((n + 1) % RC) * CHB;
        // Chunks in which steps 0-6, and in which step 7, hand a term on (the
        // windows start at step 0 or 7 of a chunk and end at its step 6 or 7:
        // ranges are whole chunks, terms move by -1, 7 or 15).
        auto in = [&](int2 k) { return (unsigned)(c - k.x) < (unsigned)k.y; };
        const unsigned dA = in(w.kA) ? w.dstA + cw : w.unused, dA7 = in(w.kA7) ? w.dstA + cw1 : w.unused;
        const unsigned dB = in(w.kB) ? w.dstB + cw : w.unused, dB7 = in(w.kB7) ? w.dstB + cw1 : w.unused;
        const unsigned puA = PUB ? in(w.pA) : 0, puA7 = PUB ? in(w.pA7) : 0;
        const unsigned puB = PUB ? in(w.pB) : 0, puB7 = PUB ? in(w.pB7) : 0;
        // operands of the next step, loaded while the current one computes
        float4 Ln = L[(FWD ? 0 : CH - 1) * NP];
        float rn = r[(FWD ? 0 : CH - 1) * NP];
        float xa[EC], xb[EC];
        bool fine = true;
        // the group's edge words, read ahead or awaited
        auto take_edges = [&](unsigned off, bool miss) {
            for (unsigned spin = 0; miss;) {
                na = ld_edge(w.inA + off);
                nb = ld_edge(w.inB + off);
                miss = __any_sync(0xffffffffu, any_absent(na, nb));
                if (!miss) break;
                __nanosleep(20);   // leaves the issue slots to the kernels of other streams; no cost alone
                if (edge_gives_up(++spin, &w.sm->abort, w.err, w.spinLimit)) { fine = false; return; }
            }
            if (!WHOLE) {   // the ring's words are free again once all warps are done with the chunk
                __syncwarp();
                if (w.inEdgeA) clear_edge(w.inA + off);
                if (w.inEdgeB) clear_edge(w.inB + off);
            }
            xa[0] = __uint_as_float(na.x); xa[1] = __uint_as_float(na.y); xa[2] = __uint_as_float(na.z); xa[3] = __uint_as_float(na.w);
            xb[0] = __uint_as_float(nb.x); xb[1] = __uint_as_float(nb.y); xb[2] = __uint_as_float(nb.z); xb[3] = __uint_as_float(nb.w);
        };
        auto step = [&](auto U) {
            constexpr int u = decltype(U)::value, s = u % EC;
            const float4 Lc = Ln;
            const float rr = rn;
            if (u + 1 < CH) {
                constexpr int q = FWD ? u + 1 : CH - 2 - u;
                Ln = L[q * NP];
                rn = r[q * NP];
            }
            float vA = nA, vB = nB;
            if (w.inEdgeA) vA = xa[s];
            if (w.inEdgeB) vB = xb[s];
            float acc, res;
            if (FWD) {
                acc = __fsub_rn(rr, SWAP ? vA : vB);    // -z
                acc = __fsub_rn(acc, SWAP ? vB : vA);   // -y
                acc = __fsub_rn(acc, tx);               // -x
                res = __fmul_rn(acc, Lc.x);
                tx = __fmul_rn(Lc.y, res);
                sA = __fmul_rn(SWAP ? Lc.w : Lc.z, res);
                sB = __fmul_rn(SWAP ? Lc.z : Lc.w, res);
            } else {
                acc = __fsub_rn(rr, __fmul_rn(Lc.y, tx));                // +x
                acc = __fsub_rn(acc, __fmul_rn(Lc.z, SWAP ? vB : vA));   // +y
                acc = __fsub_rn(acc, __fmul_rn(Lc.w, SWAP ? vA : vB));   // +z
                res = __fmul_rn(acc, Lc.x);
                tx = sA = sB = res;
            }
            nA = FWD ? __shfl_up_sync(0xffffffffu, sA, 1) : __shfl_down_sync(0xffffffffu, sA, 1);
            nB = FWD ? __shfl_up_sync(0xffffffffu, sB, VA) : __shfl_down_sync(0xffffffffu, sB, VA);
            __stcg(out + (FWD ? u : -u) * NP, res);
            constexpr int off = ((u + 1) / EC % (CH / EC)) * GW * 4 + (u + 1) % EC * 4;
            hand_on<off>(u < 7 ? dA : dA7, sA);
            hand_on<off>(u < 7 ? dB : dB7, sB);
            if (PUB) {
                publish(u < 7 ? puA : puA7, xA + u * WB, w.epoch, sA);
                publish(u < 7 ? puB : puB7, xB + u * WA, w.epoch, sB);
            }
        };
        using std::integral_constant;
        take_edges(cw, miss);
        if (!fine) return false;
        step(integral_constant<int, 0>{});
        step(integral_constant<int, 1>{});
        na = ld_edge(w.inA + cw + GW * 4);
        nb = ld_edge(w.inB + cw + GW * 4);
        step(integral_constant<int, 2>{});
        miss = __any_sync(0xffffffffu, any_absent(na, nb));
        step(integral_constant<int, 3>{});
        take_edges(cw + GW * 4, miss);
        if (!fine) return false;
        step(integral_constant<int, 4>{});
        step(integral_constant<int, 5>{});
        na = ld_edge(w.inA + cw1);   // past the last chunk: a place that is not used
        nb = ld_edge(w.inB + cw1);
        ready = mb_peek(smem_addr(&w.sm->loaded[(n + 1) % NBUF]), ((n + 1) / NBUF) & 1);
        step(integral_constant<int, 6>{});
        miss = __any_sync(0xffffffffu, any_absent(na, nb));
        step(integral_constant<int, 7>{});
        out += (FWD ? CH : -CH) * NP;
        cw = cw1;
        if (PUB) { xA += CH * WB; xB += CH * WA; }
        // The slot may be refilled: every value read from it has been used.  A
        // relaxed arrival, since a releasing one waits for the results' stores to
        // reach L2.  In the ring other warps write the words cleared above again, after
        // this arrival or after the copy into the slot that it lets through: there it
        // releases the clears, and so does the loader's (frames of 800x32x32 and
        // 1500x20x20: 4.44 and 4.51 ms either way).
        __syncwarp();
        if (WHOLE) mb_arrive_relaxed(w.lane == 0, smem_addr(&w.sm->done[b]));
        else mb_arrive_release(w.lane == 0, smem_addr(&w.sm->done[b]));
    }
    return true;
}

// SWAP: the tiles' a axis is k and b is j (else a = j, b = k).  The couplings
// that travel along each axis and the order of the subtractions follow:
// forward -z, -y, -x; backward +x, +y, +z.  WHOLE: every step's edge words have
// their own place (and terms inside a cluster are stored there); else a ring.
template <bool FWD, bool SWAP, bool WHOLE>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(NTHREADS) k_wavefront(SweepArgs a) {
    extern __shared__ __align__(128) unsigned char smemRaw[];
    SweepSmem &sm = *reinterpret_cast<SweepSmem *>(smemRaw);
    const int T = a.T;
    const int edgeGroups = (WHOLE ? T : RC * CH) / EC;   // groups of edge words per warp
    float *edge = reinterpret_cast<float *>(smemRaw + sizeof(SweepSmem));   // [warp][group][GW]
    const unsigned rank = cluster_rank();
    if (threadIdx.x == 0) {
        // Nothing to do once converged or after an earlier sweep gave up.  One
        // thread decides for the cluster: the flags may change while its CTAs
        // start, and a CTA must not leave while another reads its shared memory.
        if (rank == 0)
            sm.cluster = *(volatile const int *)a.skip || *(volatile int *)a.err ? -1
                                                                                  : (int)atomicAdd(&a.ticket[FWD ? 0 : 2], 1u);
        sm.abort = 0;
        sm.epoch = *(volatile unsigned int *)&a.ticket[1] + (FWD ? 0u : 1u);   // forward e, backward e + 1
        for (int b = 0; b < NBUF; b++) {
            mb_init(smem_addr(&sm.loaded[b]), 1);   // the loader's arrival, plus the bytes of the chunk
            mb_init(smem_addr(&sm.done[b]), NWC);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cluster_sync();
    const int ticket = ld_cluster(map_rank(smem_addr(&sm.cluster), 0));
    // The cluster and the tile of this CTA; clusters in dependency order.
    const bool live = ticket >= 0 && ticket < a.nClusters;
    const int cl = FWD ? ticket : a.nClusters - 1 - ticket;
    const int ta = live ? (cl % a.nca) * CA + (int)rank % CA : a.nta, tb = live ? (cl / a.nca) * CB + (int)rank / CA : 0;
    const bool exists = live && ta < a.nta && tb < a.ntb;
    const int tile = ta + a.nta * tb;
    // First and last step of a tile in this sweep's numbering, out to whole
    // chunks (the steps added hold zero rows); hi < lo where it holds no cell.
    auto steps_of = [&](int tl) {
        const int2 rg = a.range[tl];
        if (rg.y < rg.x) return make_int2(T, -1);
        const int lo = rg.x & ~(CH - 1), hi = rg.y | (CH - 1);
        return FWD ? make_int2(lo, hi) : make_int2((T - 1) - hi, (T - 1) - lo);
    };
    // The tiles this one takes terms from (up) and hands terms to (down), by
    // axis, and whether they are in the same cluster.  Consumer step te takes
    // the a-edge term of the producer's step te + WA - 1 and the b-edge term
    // of te + WB - 1, in the tiles' own step numbers; between warps of a tile
    // it takes the term of step te - 1.
    const int dir = FWD ? 1 : -1;
    const int2 none = make_int2(T, -1);
    const bool mute = a.epochSkew != 0;   // fault injection: nothing is handed on
    auto range_at = [&](bool in, int tl) { return exists && in ? steps_of(tl) : none; };
    const int2 own = range_at(true, tile);
    const int2 rUA = range_at(ta - dir >= 0 && ta - dir < a.nta, tile - dir);
    const int2 rUB = range_at(tb - dir >= 0 && tb - dir < a.ntb, tile - dir * a.nta);
    const int2 rDA = range_at(ta + dir >= 0 && ta + dir < a.nta && !mute, tile + dir);
    const int2 rDB = range_at(tb + dir >= 0 && tb + dir < a.ntb && !mute, tile + dir * a.nta);
    const int lo = own.x, hi = own.y;
    const bool work = hi >= lo;
    const bool upAcl = WHOLE && (ta - dir) / CA == ta / CA && ta - dir >= 0;
    const bool upBcl = WHOLE && (tb - dir) / CB == tb / CB && tb - dir >= 0;
    const bool dnAcl = WHOLE && (ta + dir) / CA == ta / CA && ta + dir >= 0;
    const bool dnBcl = WHOLE && (tb + dir) / CB == tb / CB && tb + dir >= 0;
    // consumer steps that receive a term of another tile, along each axis
    const int iA0 = max(lo, rUA.x - (WA - 1)), iA1 = min(hi, rUA.y - (WA - 1));
    const int iB0 = max(lo, rUB.x - (WB - 1)), iB1 = min(hi, rUB.y - (WB - 1));
    const bool pollA = iA1 >= iA0 && !upAcl, pollB = iB1 >= iB0 && !upBcl;
    const bool helpers = work && (!WHOLE || pollA || pollB);
    // the first warp along an axis (0 forward) takes the other tiles' terms
    constexpr int W0 = FWD ? 0 : 1;
    const int g0 = lo / EC, c0 = lo / CH, nChunks = (hi + 1) / CH - c0;
    const size_t tileBase = (size_t)tile * T * NP;
    // chunk n into its slot: its 8 steps are one block of the layout
    constexpr unsigned bl = CH * NP * sizeof(float4), br = CH * NP * sizeof(float);
    auto chunk_entry = [&](int n) { return tileBase + (size_t)(FWD ? (c0 + n) * CH : T - (c0 + n + 1) * CH) * NP; };
    auto issue = [&](int n) {
        const int b = n % NBUF;
        const unsigned bar = smem_addr(&sm.loaded[b]);
        mb_arrive_expect_tx(bar, bl + br);
        bulk_load(&sm.slot[b].L, a.L + chunk_entry(n), bl, bar);
        bulk_load(&sm.slot[b].r, a.rin + chunk_entry(n), br, bar);
    };
    auto prefetch = [&](int n) {   // into L2, for its copy one ring later
        if (n >= nChunks) return;
        prefetch_l2(a.L + chunk_entry(n), bl);
        prefetch_l2(a.rin + chunk_entry(n), br);
    };
    if (work) {
        // Words that will come are ABSENT, the others are zero terms.  In the
        // ring everything comes, the other tiles' zero terms too, except a
        // warp's first term from the warp before it.
        const int first = WHOLE ? g0 : 0, count = WHOLE ? (hi + 1) / EC - g0 : edgeGroups;
        for (int q = threadIdx.x; q < NWC * count * (VA + VB); q += NTHREADS) {
            const int pencil = q % (VA + VB), rest = q / (VA + VB), g = first + rest % count, wi = rest / count;
            const bool isA = pencil < VB;
            const bool outside = (isA ? wi % NWA : wi / NWA) == W0;   // its terms come from another tile
            const int w0 = outside ? (isA ? iA0 : iB0) : lo + 1, w1 = outside ? (isA ? iA1 : iB1) : hi;
            unsigned v[EC];
            for (int s = 0; s < EC; s++) {
                const int te = g * EC + s;
                const bool comes = WHOLE ? te >= w0 && te <= w1 : outside || te != 0;
                v[s] = comes ? ABSENT : 0u;
            }
            reinterpret_cast<uint4 *>(edge)[((size_t)wi * edgeGroups + g) * (VA + VB) + pencil] =
                make_uint4(v[0], v[1], v[2], v[3]);
        }
    }
    cluster_sync();   // also keeps rank 0 until every CTA has read its ticket
    // All of the above may run while the kernel before this one ends.
    pdl_wait();
    pdl_trigger();
    if (!work || *(volatile const int *)a.skip) return;   // converged meanwhile: every CTA sees the same now
    const size_t wordsPerTile = (size_t)T * (WA + WB);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (warp == LOADER) {
        // ================================================== loader thread
        if (lane != 0) return;
        int issued = 0;
        for (; issued < nChunks; issued++) {
            const int before = issued - NBUF;
            if (before >= 0 && !mb_wait(smem_addr(&sm.done[before % NBUF]), (before / NBUF) & 1, &sm.abort, a.err, a.spinLimit)) break;
            issue(issued);
            prefetch(issued + NBUF);
        }
        // The copies started must land before the CTA's shared memory is
        // released, also when the compute warps stop early: each slot's
        // phase completes once its bytes are in.
        for (int m = max(0, issued - NBUF); m < issued; m++)
            for (unsigned int spin = 0;
                 spin < DRAIN_SPIN_LIMIT && !mb_test(smem_addr(&sm.loaded[m % NBUF]), (m / NBUF) & 1); spin++)
                __nanosleep(32);
        return;
    }

    if (warp >= EDGE) {
        // ==================================================== edge warps
        // Warp h polls the words of every NHELP-th group of steps: lane e one
        // a-edge word (step e / WB, pencil e % WB) and two b-edge words.
        if (!helpers) return;
        const unsigned int epWait = sm.epoch + a.epochSkew;   // awaited in the neighbours' words
        const unsigned long long *xA = a.xchg + (size_t)(tile - dir) * wordsPerTile + (WA - 1) * WB;
        const unsigned long long *xB =
            a.xchg + (size_t)(tile - dir * a.nta) * wordsPerTile + (size_t)T * WB + (WB - 1) * WA;
        const int nGroups = nChunks * (CH / EC);
        const int s4 = lane / WB, pA = lane % WB, sB0 = lane / WA, pB = lane % WA;
        // the warps whose words these are
        float *wA = edge + (size_t)(W0 + NWA * (pA / VB)) * edgeGroups * GW + (pA % VB) * EC + s4;
        float *wB = edge + (size_t)(pB / VA + NWA * W0) * edgeGroups * GW + (VB + pB % VA) * EC + sB0;
        for (int m = warp - EDGE; m < nGroups; m += NHELP) {
            const int g = WHOLE ? g0 + m : m % edgeGroups;
            if (!WHOLE && m >= 2 * NBUF) {   // the words' last group is done
                const int prev = m / 2 - NBUF;
                if (!mb_wait(smem_addr(&sm.done[prev % NBUF]), (prev / NBUF) & 1, &sm.abort, a.err, a.spinLimit)) return;
            }
            const int t = (g0 + m) * EC, tA = t + s4, tB0 = t + sB0, tB1 = tB0 + EC / 2;
            bool needA = pollA && tA >= iA0 && tA <= iA1;
            bool needB0 = pollB && tB0 >= iB0 && tB0 <= iB1, needB1 = pollB && tB1 >= iB0 && tB1 <= iB1;
            float vA = 0.f, vB0 = 0.f, vB1 = 0.f;
            bool ok = true;
            for (unsigned int spin = 0; needA || needB0 || needB1; spin++) {
                if (spin >= a.spinLimit) {
                    atomicExch(a.err, 1);
                    ok = false;
                    break;
                }
                if (spin > 8) {
                    if (*(volatile int *)&sm.abort || ((spin & 63) == 63 && *(volatile int *)a.err)) { ok = false; break; }
                    if (spin > 64) __nanosleep(32);
                }
                const unsigned long long w2 = needA ? ld_word(xA + (size_t)tA * WB + pA) : 0ull,
                                         w0 = needB0 ? ld_word(xB + (size_t)tB0 * WA + pB) : 0ull,
                                         w1 = needB1 ? ld_word(xB + (size_t)tB1 * WA + pB) : 0ull;
                if (needA && (unsigned)(w2 >> 32) == epWait) { vA = __uint_as_float((unsigned)w2); needA = false; }
                if (needB0 && (unsigned)(w0 >> 32) == epWait) { vB0 = __uint_as_float((unsigned)w0); needB0 = false; }
                if (needB1 && (unsigned)(w1 >> 32) == epWait) { vB1 = __uint_as_float((unsigned)w1); needB1 = false; }
            }
            if (!__all_sync(0xffffffffu, ok)) {
                // the compute warps and the loader see the flag in their waits
                *(volatile int *)&sm.abort = 1;
                return;
            }
            if (!WHOLE || pollA) *(volatile float *)(wA + g * GW) = vA;
            if (!WHOLE || pollB) {
                *(volatile float *)(wB + g * GW) = vB0;
                *(volatile float *)(wB + g * GW + EC / 2) = vB1;
            }
        }
        return;
    }

    // ====================================================== compute warps
    // Warp (wa, wb), lane (la, lb): pencil (8 wa + la, 4 wb + lb) of the tile.
    const int wa = warp % NWA, wb = warp / NWA, la = lane % VA, lb = lane / VA;
    const bool outEdgeA = la == (FWD ? VA - 1 : 0), outEdgeB = lb == (FWD ? VB - 1 : 0);
    WarpJob w;
    w.sm = &sm;
    w.err = a.err;
    w.spinLimit = a.spinLimit;
    w.c0 = c0;
    w.nChunks = nChunks;
    w.lane = lane;
    w.L = &sm.slot[0].L[0][warp * 32 + lane];
    w.r = &sm.slot[0].r[0][warp * 32 + lane];
    w.out = a.out + tileBase + warp * 32 + lane;
    w.lastStep = T - 1;
    w.inEdgeA = la == (FWD ? 0 : VA - 1);
    w.inEdgeB = lb == (FWD ? 0 : VB - 1);
    w.epoch = sm.epoch;
    const unsigned eb = smem_addr(edge), warpBytes = (unsigned)edgeGroups * GW * 4;
    w.inA = eb + warp * warpBytes + lb * EC * 4;
    w.inB = eb + warp * warpBytes + (VB + la) * EC * 4;
    // To the next warp of the tile, or from the last one to the next tile: the
    // words of its first warp there (another CTA of the cluster, by its own
    // steps), or the exchange array.
    const bool lastA = wa == 1 - W0, lastB = wb == 1 - W0;
    const unsigned toA = (unsigned)(lastA ? W0 + NWA * wb : 1 - W0 + NWA * wb) * warpBytes + lb * EC * 4;
    const unsigned toB = (unsigned)(lastB ? wa + NWA * W0 : wa + NWA * (1 - W0)) * warpBytes + (VB + la) * EC * 4;
    constexpr int GB = GW * 4 / EC;   // edge bytes per step
    w.unused = smem_addr(&sm.unused[warp][lane]);
    w.unused = map_rank(w.unused, rank);
    w.dstA = lastA && dnAcl ? map_rank(eb + toA, (unsigned)((int)rank + dir)) - WA * GB : map_rank(eb + toA, rank);
    w.dstB = lastB && dnBcl ? map_rank(eb + toB, (unsigned)((int)rank + dir * CA)) - WB * GB : map_rank(eb + toB, rank);
    const int dA0 = max(lo, rDA.x + WA - 1), dA1 = min(hi, rDA.y + WA - 1);   // steps whose term the next tile takes
    const int dB0 = max(lo, rDB.x + WB - 1), dB1 = min(hi, rDB.y + WB - 1);
    // chunks of a window of steps [s0, s1], by `first` step of the chunk (0: its
    // steps 0-6; 7: step 7)
    auto chunks = [](bool on, int s0, int s1, int first) {
        const int k0 = (s0 - first + CH - 1) >> 3, k1 = (s1 - (first | 6)) >> 3;   // floor division
        return make_int2(k0, on ? max(k1 - k0 + 1, 0) : 0);
    };
    const bool smA = outEdgeA && (!lastA || dnAcl), smB = outEdgeB && (!lastB || dnBcl);   // into shared memory
    const int sA0 = lastA ? dA0 : lo, sA1 = lastA ? dA1 : hi - 1, sB0 = lastB ? dB0 : lo, sB1 = lastB ? dB1 : hi - 1;
    w.kA = chunks(smA, sA0, sA1, 0);
    w.kA7 = chunks(smA, sA0, sA1, 7);
    w.kB = chunks(smB, sB0, sB1, 0);
    w.kB7 = chunks(smB, sB0, sB1, 7);
    w.pA = chunks(outEdgeA && !smA, dA0, dA1, 0);
    w.pA7 = chunks(outEdgeA && !smA, dA0, dA1, 7);
    w.pB = chunks(outEdgeB && !smB, dB0, dB1, 0);
    w.pB7 = chunks(outEdgeB && !smB, dB0, dB1, 7);
    w.xA = a.xchg + (size_t)tile * wordsPerTile + wb * VB + lb;                    // [t][WB]
    w.xB = a.xchg + (size_t)tile * wordsPerTile + (size_t)T * WB + wa * VA + la;   // [t][WA]
    const bool pub = __any_sync(0xffffffffu, w.pA.y + w.pA7.y + w.pB.y + w.pB7.y > 0);
    const bool fine = pub ? run_steps<FWD, SWAP, WHOLE, true>(w) : run_steps<FWD, SWAP, WHOLE, false>(w);
    if (!fine) {
        // Peers may still store into this CTA's shared memory: stop the other
        // warps, let what is in flight land, and stay until the cluster's
        // other threads have ended or got here.
        *(volatile int *)&sm.abort = 1;
        for (int q = 0; q < 32; q++) __nanosleep(1000);
        __syncwarp();
        cluster_sync();
    }
}

// Before a sweep pair without a kernel that prepares it (sweep_prep).
__global__ void k_sweep_prep(unsigned int *ticket) { sweep_prep(ticket); }

__global__ void k_tile_range_init(int2 *range, int n) {
    pdl_begin();
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) range[t] = make_int2(0x7fffffff, -1);
}

// First and last forward step at which a tile meets a system cell
// (lanes of a warp that fall into the same tile reduce before the atomics).
__global__ void k_tile_range(const uint8_t *fluid, int I, int J, int K, SweepLayout g, int2 *range) {
    pdl_begin();
    long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    bool f = t < (long long)I * J * K && fluid[t];
    int tile = -1, step = 0;
    if (f) {
        int i, j, k;
        unflatten(t, I, J, i, j, k);
        const int aa = (g.swap ? k : j) - 1, bb = (g.swap ? j : k) - 1;
        tile = aa / WA + g.nta * (bb / WB);
        step = (i - 1) + aa % WA + bb % WB;
    }
    unsigned int grp = __match_any_sync(0xffffffffu, tile);
    int mn = __reduce_min_sync(grp, f ? step : 0x7fffffff);
    int mx = __reduce_max_sync(grp, f ? step : -1);
    if (f && (int)(threadIdx.x & 31) == __ffs(grp) - 1) {
        atomicMin(&range[tile].x, mn);
        atomicMax(&range[tile].y, mx);
    }
}

}  // namespace

int sweep_tiles_max(int I, int J, int K) {
    int best = 0;
    for (int sw = 0; sw < 2; sw++) {
        const SweepLayout g = sweep_layout(I, J, K, sw);
        best = std::max(best, g.nta * g.ntb);
    }
    return best;
}

// per tile: WB a-edge words and WA b-edge words for each of its T steps
long long sweep_exchange_words(int I, int J, int K) {
    const SweepLayout g = sweep_layout(I, J, K);
    return (long long)sweep_tiles_max(I, J, K) * (WA + WB) * g.T;
}

void launch_sweep_ranges(const StepConsts &c, const SweepLayout &g, const uint8_t *fluid, SweepState &sw,
                         cudaStream_t s) {
    const int n = g.nta * g.ntb;
    launch_next(k_tile_range_init, div_up(n, 256), 256, s, sw.range, n);
    long long nc = (long long)c.I * c.J * c.K;
    launch_next(k_tile_range, div_up(nc, 256), 256, s, fluid, c.I, c.J, c.K, g, sw.range);
}

void launch_sweeps(const StepConsts &c, const SweepLayout &g, const float4 *L, const float *rf, float *z,
                   SweepState &sw, const int *skip, cudaStream_t s, bool prepped, bool overlap) {
    static std::atomic<unsigned long long> smemSet{0};   // devices on which the shared memory is opted in
    int dev = 0;
    cudaGetDevice(&dev);
    // [direction][orientation][whole]
    using Kernel = void (*)(SweepArgs);
    static constexpr Kernel kernels[2][2][2] = {
        {{k_wavefront<true, false, false>, k_wavefront<true, false, true>},
         {k_wavefront<true, true, false>, k_wavefront<true, true, true>}},
        {{k_wavefront<false, false, false>, k_wavefront<false, false, true>},
         {k_wavefront<false, true, false>, k_wavefront<false, true, true>}}};
    if (dev < 64 && !((smemSet.load() >> dev) & 1ull)) {   // idempotent, so a race only repeats it
        for (auto &byDir : kernels)
            for (auto &byOrient : byDir)
                for (Kernel k : byOrient)
                    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sweep_smem_bytes(WHOLE_STEPS));
        smemSet.fetch_or(1ull << dev);
    }
    SweepArgs a;
    a.L = L;
    a.T = g.T;
    a.nta = g.nta; a.ntb = g.ntb;
    a.nca = (g.nta + CA - 1) / CA;
    a.nClusters = a.nca * ((g.ntb + CB - 1) / CB);
    a.range = sw.range; a.xchg = sw.xchg; a.ticket = sw.ticket; a.err = sw.err; a.skip = skip;
    a.spinLimit = sw.spinLimit ? sw.spinLimit : DEFAULT_SPIN_LIMIT;
    a.epochSkew = sw.stall ? 1u : 0u;
    const bool whole = g.T <= WHOLE_STEPS;
    const size_t smem = sweep_smem_bytes(whole ? g.T : RC * CH);
    const unsigned n = (unsigned)a.nClusters * CL;
    if (!prepped) { FLIP_COUNT(1); k_sweep_prep<<<1, 1, 0, s>>>(sw.ticket); }
    // forward: y from r; backward: z from y, in place
    for (int d = 0; d < 2; d++) {
        a.rin = d == 0 ? rf : z;
        a.out = z;
        launch_after(overlap || d == 1, kernels[d][g.swap ? 1 : 0][whole ? 1 : 0], n, NTHREADS, smem, s, a);
    }
    sw.epoch += 2;
}

// Epochs are 32-bit: before they wrap, forget every old word (outside any
// capture: the host calls this between sweeps).
void sweep_epoch_guard(const StepConsts &c, SweepState &sw, long long upcoming, cudaStream_t s) {
    if ((long long)sw.epoch + upcoming < 0xfffffff0LL) return;
    cudaMemsetAsync(sw.xchg, 0, sweep_exchange_words(c.I, c.J, c.K) * sizeof(unsigned long long), s);
    cudaMemsetAsync(sw.ticket, 0, 3 * sizeof(unsigned int), s);
    sw.epoch = 0;
}

}  // namespace flip
