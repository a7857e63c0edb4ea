// mpm_cell_order_noalloc: cell keys and the stable order by cell of
// caller-provided device positions, computed without allocating memory.
//
// Some hosts of this engine cannot allocate device memory at the moment they
// need the cell order: code running inside a memory pool or arena that owns
// every byte of the device heap, plug-ins whose host framework forbids
// cudaMalloc/cudaFree on its calling thread (for example between the
// framework's own allocation phases), and latency-critical callers for whom
// an allocation (and the implicit device synchronisation of cudaFree) in the
// loop is not acceptable.  This entry point needs nothing from the caller
// except its inputs and outputs: its working memory (the radix sort's
// ping-pong key/value buffers and digit histograms) lives in one file-scope
// __device__ array below, reserved when the library is loaded and held by
// every GPU that loads it until the process exits.
//
// The result is the same as mpm_cell_order() reports for the same positions
// (same kernels, same stable LSD radix sort).
#include <cuda_runtime.h>

#include <mutex>

#include "kernels.cuh"
#include "mpm_gb300.h"
#include "radix_sort.cuh"

using namespace mpm;

namespace {

constexpr long long NA_MAX = MPM_NOALLOC_MAX_PARTICLES;
constexpr long long NA_TILES = RS_FEW / RS_FEW_TILE > NA_MAX / RS_TILE ? RS_FEW / RS_FEW_TILE : NA_MAX / RS_TILE;
// layout (32-bit words): keysA, valsA, keysB, valsB (NA_MAX each), digit counts
// (256 per tile) and totals (256), then one word k_cell_keys may flag a
// non-finite position in (a write-only sink: such a particle already gets the
// out-of-grid key, and the word is never read), padded to 64 words.
constexpr long long NA_WORDS = 4 * NA_MAX + 256 * (NA_TILES + 1) + 64;

// The scratch: file scope, static storage on every device that loads the library.
__device__ __align__(256) unsigned g_noalloc_scratch[NA_WORDS];

constexpr int NA_MAX_DEVICES = 64;
unsigned* g_scratch_addr[NA_MAX_DEVICES] = {nullptr};
std::mutex g_setup_mutex;

// Once per device, with that device current: the device address of the
// scratch array.  In host code g_noalloc_scratch names a host-side shadow,
// not device memory, so only this address may be handed to kernels.
int scratch_for_current_device(unsigned** out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return MPM_ERR_CUDA;
    if (dev < 0 || dev >= NA_MAX_DEVICES) return MPM_ERR_CUDA;
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    if (!g_scratch_addr[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            cudaGetLastError();
            return MPM_ERR_CUDA;
        }
        g_scratch_addr[dev] = (unsigned*)p;
    }
    *out = g_scratch_addr[dev];
    return MPM_OK;
}

// A kernel that begins with step_enter: its launch overlaps the kernel before it.
template <typename... Ex, typename... Act>
void launch_after(cudaStream_t st, void (*kernel)(Ex...), unsigned grid, unsigned block, Act&&... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Act>(args)...);
}

}  // namespace

extern "C" int mpm_cell_order_noalloc(const mpm_grid_desc* grid, const double* d_pos, int64_t n, uint32_t* d_keys,
                                      uint32_t* d_order, void* stream) {
    if (!grid || n < 0) return MPM_ERR_ARG;
    if (n > NA_MAX) return MPM_ERR_TOO_LARGE;
    if (n == 0) return MPM_OK;
    if (!d_pos || !d_keys || !d_order) return MPM_ERR_ARG;
    Geom g{};
    long long keyspace = 1;
    for (int a = 0; a < 3; ++a) {
        // cells + 2 must fit an int, and the key count a 32-bit key: check each factor before multiplying
        if (!(grid->length[a] > 0.0) || grid->cells[a] < 1 || grid->cells[a] > (1 << 30)) return MPM_ERR_ARG;
        g.h[a] = grid->length[a] / (double)grid->cells[a];
        g.inv_h[a] = 1.0 / g.h[a];
        set_float_geometry(g, a);
        g.nn[a] = grid->cells[a] + 1;
        g.kd[a] = grid->cells[a] + 2;
        keyspace *= (long long)g.kd[a];  // < 2^32 * (2^30 + 2): no overflow
        if (keyspace >= 0xffffffffLL) return MPM_ERR_ARG;
    }
    g.key_max = (unsigned)keyspace;
    // an error left pending by the caller's own work is not this call's to report or to clear
    if (cudaPeekAtLastError() != cudaSuccess) return MPM_ERR_CUDA;
    unsigned* s = nullptr;
    int rc = scratch_for_current_device(&s);
    if (rc) return rc;
    unsigned* keysA = s;
    unsigned* valsA = s + NA_MAX;
    unsigned* keysB = s + 2 * NA_MAX;
    unsigned* valsB = s + 3 * NA_MAX;
    unsigned* counts = s + 4 * NA_MAX;
    unsigned* err = counts + 256 * (NA_TILES + 1);
    cudaStream_t st = (cudaStream_t)stream;
    // every scratch word the sort reads is written first by this call (keys by k_cell_keys, digit counts and
    // totals by each pass), so the previous call's contents need no clearing.  The keys go to the caller's
    // array and are the first pass's input; its values are the identity, the last pass's the caller's order.
    // A caller that wants the order alone may give one array for both: the first pass, which may be the last
    // as well, then reads the keys from the scratch.
    unsigned* first = d_order == d_keys ? keysB : d_keys;
    launch_after(st, k_cell_keys, (unsigned)((n + 255) / 256), 256, d_pos, n, g, first, (unsigned*)nullptr, d_keys, err,
                 (float*)nullptr, (const uint16_t*)nullptr);
    if (cudaGetLastError() != cudaSuccess) return MPM_ERR_CUDA;
    int bits = 1;
    while (bits < 32 && ((unsigned long long)1 << bits) <= (unsigned long long)g.key_max) ++bits;
    const bool few = n <= RS_FEW;
    const int tile = few ? RS_FEW_TILE : RS_TILE, nblocks = (int)((n + tile - 1) / tile);
    const auto hist = few ? k_rs_hist<8, RS_FEW_ITEMS> : k_rs_hist<8, RS_ITEMS>;
    const auto scatter = few ? k_rs_scatter<8, RS_FEW_ITEMS> : k_rs_scatter<8, RS_ITEMS>;
    const unsigned *kin = first, *vin = nullptr;
    unsigned *kout = keysA, *vout = valsA;
    for (int shift = 0; shift < bits; shift += 8) {
        const bool last = shift + 8 >= bits;
        launch_after(st, hist, nblocks, RS_THREADS, kin, n, shift, counts, nblocks);
        launch_after(st, k_rs_scan, 256, RS_SCAN_THREADS, counts, nblocks);
        launch_after(st, scatter, nblocks, RS_THREADS, kin, vin, last ? (unsigned*)nullptr : kout,
                     last ? d_order : vout, n, shift, (const unsigned*)counts, nblocks);
        if (cudaGetLastError() != cudaSuccess) return MPM_ERR_CUDA;
        kin = kout;
        vin = vout;
        kout = kout == keysA ? keysB : keysA;
        vout = vout == valsA ? valsB : valsA;
    }
    return MPM_OK;
}
