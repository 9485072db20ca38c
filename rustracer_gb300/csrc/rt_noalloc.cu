// The photon-grid build for callers that cannot allocate device memory.
//
// rt_stage_photon_grid allocates its device buffers on every call.  Some callers cannot do that: frame
// loops with a hard no-allocation rule (cudaMalloc / cudaFree can synchronise the device and stall a
// frame), hosts whose device memory is handed out by their own allocator (an engine's or a
// framework's pool that owns every byte the process may touch), and processes running close to the
// memory limit, where an allocation could fail in the middle of a frame.  For them,
// rt_stage_photon_grid_noalloc takes device pointers for its input and outputs and keeps its scratch
// -- a word per slot, the slot order, the list of cells to sort, the scan's status words and the totals --
// in one file-scope __device__ array of fixed size.  Every GPU that loads this library holds that
// array (RT_NOALLOC_SCRATCH_BYTES, 9,438,208 bytes) until the process exits.
#include <cuda_runtime.h>

#include "rt_internal.h"
#include "rt_kernels.h"

using rt::set_error;

namespace {

constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kWordsOff = 0;
constexpr size_t kOrderOff = align256(kWordsOff + 4 * (size_t)RT_NOALLOC_MAX_SLOTS);
constexpr size_t kListOff = align256(kOrderOff + 4 * (size_t)RT_NOALLOC_MAX_SLOTS);
constexpr size_t kStatusOff = align256(kListOff + 4 * (size_t)RT_NOALLOC_MAX_CELLS);
constexpr size_t kStatusMax = RT_NOALLOC_MAX_CELLS / 2048 + 2;  // the scan's status words and ticket
constexpr size_t kTotalOff = align256(kStatusOff + 4 * kStatusMax);
constexpr size_t kScratchBytes = align256(kTotalOff + 16);
static_assert(kScratchBytes <= RT_NOALLOC_SCRATCH_BYTES, "scratch layout exceeds the declared size");

}  // namespace

// Shared by every call on a device.  In host code the name is only a handle: the array's device
// address comes from cudaGetSymbolAddress with the device current.
static __device__ __align__(256) unsigned char g_grid_scratch[RT_NOALLOC_SCRATCH_BYTES];

extern "C" int rt_stage_photon_grid_noalloc(const rt_photon *d_photons, const rt_grid_params *gp, uint32_t *d_counts,
                                            uint32_t *d_meta, rt_photon *d_sorted, void *stream) {
    rt::clear_error();
    (void)cudaGetLastError();  // a non-sticky error left by earlier, unrelated work is not this call's
    if (!gp || !d_counts || !d_meta || !d_sorted || (gp->photon_slots && !d_photons)) {
        set_error("rt_stage_photon_grid_noalloc: null argument");
        return RT_ERR_INVALID_ARGUMENT;
    }
    if ((reinterpret_cast<uintptr_t>(d_photons) | reinterpret_cast<uintptr_t>(d_sorted)) % 16u != 0u ||
        (reinterpret_cast<uintptr_t>(d_counts) | reinterpret_cast<uintptr_t>(d_meta)) % 4u != 0u) {
        set_error("rt_stage_photon_grid_noalloc: d_photons / d_sorted must be 16-byte aligned, d_counts / d_meta 4-byte");
        return RT_ERR_INVALID_ARGUMENT;
    }
    if (gp->num_cells == 0 || gp->num_cells > RT_NOALLOC_MAX_CELLS || gp->photon_slots > RT_NOALLOC_MAX_SLOTS) {
        set_error("rt_stage_photon_grid_noalloc: %u slots and %u cells requested; this entry point handles at most "
                  "%u slots and %u cells (use rt_stage_photon_grid beyond that)",
                  gp->photon_slots, gp->num_cells, (unsigned)RT_NOALLOC_MAX_SLOTS, (unsigned)RT_NOALLOC_MAX_CELLS);
        return RT_ERR_INVALID_ARGUMENT;
    }
    if (rtd::grid_scan_partials(gp->num_cells) > kStatusMax) {
        set_error("rt_stage_photon_grid_noalloc: scan status words exceed the scratch layout");
        return RT_ERR_INVALID_ARGUMENT;
    }
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        set_error("rt_stage_photon_grid_noalloc: no usable current device (%s)", cudaGetErrorString(e));
        return RT_ERR_CUDA;
    }
    // The array's address on the current device, looked up on every call: a lookup allocates nothing
    // once the module is loaded, and a fresh one stays right after cudaDeviceReset reloads it.  The
    // first call on a device may load the module (lazy loading), which creates the array.
    void *base = nullptr;
    e = cudaGetSymbolAddress(&base, g_grid_scratch);
    if (e != cudaSuccess || !base) {
        set_error("rt_stage_photon_grid_noalloc: cudaGetSymbolAddress failed on device %d: %s", dev,
                  cudaGetErrorString(e));
        return RT_ERR_CUDA;
    }
    unsigned char *b = static_cast<unsigned char *>(base);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    auto words = [&](size_t off) { return reinterpret_cast<uint32_t *>(b + off); };
    const rtd::SmallGrid g{reinterpret_cast<const float4 *>(d_photons), d_counts, d_meta,
                           reinterpret_cast<float4 *>(d_sorted), words(kWordsOff), words(kOrderOff), words(kListOff),
                           words(kStatusOff), words(kTotalOff)};
    if ((e = rtd::launch_small_grid(g, *gp, st)) != cudaSuccess) {
        set_error("rt_stage_photon_grid_noalloc: launch failed: %s", cudaGetErrorString(e));
        return RT_ERR_CUDA;
    }
    return RT_OK;
}
