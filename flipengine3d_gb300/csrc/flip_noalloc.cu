// Particle positions in id order, written into caller memory, with no
// allocation by the library.
//
// The same three steps as the context's readback (flag the ids, exclusive
// scan of the flags, scatter), but working in one file-scope device array
// instead of buffers allocated with the context, so that a caller whose
// device memory all comes from its own allocator, or who must not let a
// cudaMalloc stall the device in the middle of a frame loop, can still order
// the particles it holds.
#include <string>

#include "../../include/flip3d.h"
#include "flip_device.cuh"

namespace flip {
int record_error(int code, const std::string &msg);   // sets flip_last_error()
}

// Scratch shared by every call on a device: a bit per id, 32 to a word, and for
// each word the ids below it.  Sized for FLIP_NOALLOC_MAX_IDS ids: 2 x 2^15
// words, 256 KiB, held by every GPU that loads the library until the process
// exits.
static_assert(FLIP_NOALLOC_MAX_IDS % 32 == 0, "whole words");
static __device__ __align__(256) int g_noalloc_scratch[2 * (FLIP_NOALLOC_MAX_IDS / 32)];

namespace {

constexpr int TPB = 256, SCAN_TPB = 1024;

// Ids as bits, 32 to a word, and for each word how many ids lie below it: an id's
// rank is that and the bits below its own.  Four launches of a few microseconds
// each, every one started while the one before it ends.  A call on ids in random
// order takes 15.5 us for 1000, 17 for 300k and 42 for 2^20; with a word per id,
// scanned in three steps, there were six launches (23, 31 and 50), and with the
// words scanned by one CTA 300k took 21 and 2^20 95.
__global__ void __launch_bounds__(TPB) k_na_clear(unsigned *bits, int words) {
    flip::pdl_trigger();
    const int t = blockIdx.x * TPB + threadIdx.x;
    if (t < words) bits[t] = 0;
}

__global__ void __launch_bounds__(TPB) k_na_flag(const unsigned int *ids, int n, int idSpace, unsigned *bits) {
    const int t = blockIdx.x * TPB + threadIdx.x;
    const unsigned id = t < n ? ids[t] : 0xffffffffu;   // the caller's: written before the clear was launched
    flip::pdl_wait();
    flip::pdl_trigger();
    if (id < (unsigned int)idSpace) atomicOr(&bits[id >> 5], 1u << (id & 31));
}

// A word a thread.  A CTA adds up the words before its own itself (at most 31 loads a
// thread, side by side), so that there is nothing to wait for and no launch more.
__global__ void __launch_bounds__(SCAN_TPB) k_na_scan(const unsigned *bits, int words, int *below) {
    __shared__ int warpSums[SCAN_TPB / 32], warpBefore[SCAN_TPB / 32];
    flip::pdl_wait();
    flip::pdl_trigger();
    const int first = blockIdx.x * SCAN_TPB, w = first + threadIdx.x;
    int before = 0;
#pragma unroll 8
    for (int v = threadIdx.x; v < first; v += SCAN_TPB) before += __popc(bits[v]);
    const int own = w < words ? __popc(bits[w]) : 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 31) {
        warpSums[warp] = inc;
        warpBefore[warp] = before;
    }
    __syncthreads();
    // every warp adds up the warps before it, and all of the earlier CTAs' words
    const int sum = __reduce_add_sync(0xffffffffu, warpBefore[lane] + (lane < warp ? warpSums[lane] : 0));
    if (w < words) below[w] = sum + inc - own;
}

__global__ void __launch_bounds__(TPB) k_na_scatter(const float *px, const float *py, const float *pz, const unsigned int *ids,
                                                    int n, int idSpace, const unsigned *bits, const int *below, float *out) {
    const int t = blockIdx.x * TPB + threadIdx.x;
    const unsigned id = t < n ? ids[t] : 0xffffffffu;
    flip::pdl_wait();
    if (id >= (unsigned int)idSpace) return;
    const long long o = 3LL * (below[id >> 5] + __popc(bits[id >> 5] & ((1u << (id & 31)) - 1u)));
    out[o] = px[t];
    out[o + 1] = py[t];
    out[o + 2] = pz[t];
}

// Device address of the scratch array in the current context.  The address
// belongs to the context that loaded this module, not to the device
// ordinal: a host that makes its own driver contexts, or calls
// cudaDeviceReset, gets a new one.  So it is looked up on every call; once
// the module is loaded in the context the lookup allocates nothing.  Under
// lazy module loading the array's 256 KiB are reserved at the first call in a
// context, not when the library loads.
int scratch_for_current_context(int **out) {
    int *ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void **)&ptr, g_noalloc_scratch);
    if (e != cudaSuccess || !ptr)
        return flip::record_error(FLIP_E_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    *out = ptr;
    return FLIP_OK;
}

}  // namespace

extern "C" int flip_order_particles_by_id_noalloc(const float *d_px, const float *d_py, const float *d_pz,
                                                  const unsigned int *d_ids, int n, int id_space,
                                                  float *d_out_xyz, void *stream) {
    if (n < 0 || id_space < 0) return flip::record_error(FLIP_E_DOMAIN, "negative particle count or id space");
    if (id_space > FLIP_NOALLOC_MAX_IDS)
        return flip::record_error(FLIP_E_OUT_OF_RANGE, "id_space " + std::to_string(id_space) +
                                                           " exceeds the no-allocation limit of " +
                                                           std::to_string(FLIP_NOALLOC_MAX_IDS) + " ids");
    if (n > id_space) return flip::record_error(FLIP_E_DOMAIN, "more particles than distinct ids below id_space");
    if (n == 0) return FLIP_OK;
    if (!d_px || !d_py || !d_pz || !d_ids || !d_out_xyz) return flip::record_error(FLIP_E_NULL, "null device pointer");
    int *scratch = nullptr;
    int rc = scratch_for_current_context(&scratch);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const int words = (id_space + 31) / 32;
    unsigned *bits = reinterpret_cast<unsigned *>(scratch);
    int *below = scratch + words;
    // the first one after all of the caller's work, the others overlapping the one before
    flip::launch_after(false, k_na_clear, flip::div_up(words, TPB), TPB, 0, s, bits, words);
    flip::launch_after(true, k_na_flag, flip::div_up(n, TPB), TPB, 0, s, d_ids, n, id_space, bits);
    flip::launch_after(true, k_na_scan, flip::div_up(words, SCAN_TPB), SCAN_TPB, 0, s, bits, words, below);
    flip::launch_after(true, k_na_scatter, flip::div_up(n, TPB), TPB, 0, s, d_px, d_py, d_pz, d_ids, n, id_space, bits, below,
                       d_out_xyz);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return flip::record_error(FLIP_E_CUDA, std::string("launch: ") + cudaGetErrorString(e));
    return FLIP_OK;
}
