// Allocation-free Morton ordering: the key and sort stage of the octree
// build (sph_tree.cu) for callers that must not allocate device memory.
//
// Who needs this: a host that runs under a fixed device-memory budget (an
// embedding application that has handed the rest of the GPU to its own pool
// allocator, or a service that must not grow its footprint while it runs)
// cannot let a library call cudaMalloc / cudaFree, and a cudaFree also
// synchronises the device, which such a host may not allow in the middle of
// a step.  This entry point takes device pointers for its inputs and
// outputs and keeps its scratch in one file-scope device array, sized for at
// most SPH_NOALLOC_MAX_N particles.  That array exists on every GPU that
// loads the library, for the lifetime of the process, whether or not the
// entry point is used.
//
// The array is shared by every call on a device and keeps the last call's
// contents; each call rewrites all of it that it reads, the error word
// among it.  Two calls whose work overlaps on the GPU
// (different streams, no ordering between them) race on the array.  Called
// eagerly, a call ends by reading the error word back to the host, so it
// returns only after its work on `stream` has finished.  Called while
// `stream` is being captured into a CUDA graph, it only records its work
// (kernel launches and nothing else) and returns at once: a replay reports no
// status.
#include <algorithm>
#include <atomic>
#include <mutex>

#include "sph_internal.cuh"

namespace sph {

// the key and sort kernels of sph_tree.cu (declared in sph_internal.cuh) are launched from here unchanged

namespace {

constexpr int NA_MAX = SPH_NOALLOC_MAX_N;
constexpr int NA_TILE = RS_TILE;                  // radix-sort tile (k_rs_scatter)
constexpr int NA_NB = (NA_MAX + NA_TILE - 1) / NA_TILE;
constexpr int NA_BOX = 304;                       // blocks of k_bbox_partial

// byte offsets inside the scratch array (each 256-byte aligned)
constexpr size_t al(size_t b) { return (b + 255) & ~size_t(255); }
constexpr size_t OFF_BOX = 0;                                           // int64 [NA_BOX * 6]
constexpr size_t OFF_RB = OFF_BOX + al(sizeof(double) * NA_BOX * 6);    // double [8 + 22]
constexpr size_t OFF_K0 = OFF_RB + al(sizeof(double) * 32);             // uint64 [NA_MAX]
constexpr size_t OFF_K1 = OFF_K0 + al(sizeof(uint64_t) * NA_MAX);
constexpr size_t OFF_V0 = OFF_K1 + al(sizeof(uint64_t) * NA_MAX);       // uint32 [NA_MAX]
constexpr size_t OFF_V1 = OFF_V0 + al(sizeof(uint32_t) * NA_MAX);
constexpr size_t OFF_HIST = OFF_V1 + al(sizeof(uint32_t) * NA_MAX);     // uint32 [RS_HISTS][NA_NB][256]
constexpr size_t OFF_ERR = OFF_HIST + al(sizeof(uint32_t) * 256 * RS_HISTS * NA_NB);   // int
constexpr size_t NA_BYTES = OFF_ERR + 256;

}  // namespace
}  // namespace sph

// the scratch: about 3.2 MB for SPH_NOALLOC_MAX_N = 131072
static __device__ __align__(256) unsigned char g_noalloc_scratch[sph::NA_BYTES];

namespace {

std::mutex g_na_mu;
int g_na_pageable[64];   // the device writes pageable host memory (set with g_na_ptr)
unsigned char *g_na_ptr[64] = {nullptr};   // device address of the scratch, per device

// once per device, with that device current: the device address of the array
int noalloc_setup(int dev, unsigned char **out, bool *pageable) {
    std::lock_guard<std::mutex> lk(g_na_mu);
    if (dev < 0 || dev >= 64) return SPH_ERR_CUDA;
    if (!g_na_ptr[dev]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p) {
            cudaGetLastError();
            return SPH_ERR_CUDA;
        }
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrPageableMemoryAccess, dev) != cudaSuccess) {
            cudaGetLastError();
            v = 0;
        }
        g_na_pageable[dev] = v == 1;
        g_na_ptr[dev] = static_cast<unsigned char *>(p);
    }
    *pageable = g_na_pageable[dev] != 0;
    *out = g_na_ptr[dev];
    return SPH_OK;
}

// the array's address is known on this device (a capture may not make the first call: it looks
// the address up)
bool noalloc_ready(int dev) {
    std::lock_guard<std::mutex> lk(g_na_mu);
    return dev >= 0 && dev < 64 && g_na_ptr[dev] != nullptr;
}

// Where a call's status is written by a kernel.  Not the caller's frame: when the wait for the stream fails, the kernel may
// still run after the call has returned.  A word is a call's own until then, and is never used again if the wait fails.
constexpr int NA_WORDS = 256;
int g_na_words[NA_WORDS];
std::atomic<bool> g_na_taken[NA_WORDS];

int take_word() {   // -1: all are taken
    for (int k = 0; k < NA_WORDS; ++k)
        if (!g_na_taken[k].exchange(true)) return k;
    return -1;
}

}  // namespace

extern "C" int sph_morton_order_noalloc(const double *x, const double *y, const double *z, int64_t n,
                                        uint64_t *keys_out, int32_t *order_out, void *stream) {
    using namespace sph;
    if (!x || !y || !z || !keys_out || !order_out || n < 1) return SPH_ERR_ARG;
    if (n > NA_MAX) return SPH_ERR_CAPACITY;   // the scratch holds at most SPH_NOALLOC_MAX_N particles
    // An error an earlier call left pending on this thread is reported before any work is queued and left
    // in place for its owner, so the launch checks below see this call's launches only.
    if (cudaPeekAtLastError() != cudaSuccess) return SPH_ERR_CUDA;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return SPH_ERR_CUDA;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capture) != cudaSuccess) {
        cudaGetLastError();
        return SPH_ERR_CUDA;
    }
    const bool capturing = capture == cudaStreamCaptureStatusActive;
    if (capturing && !noalloc_ready(dev)) return SPH_ERR_STATE;   // nothing recorded
    unsigned char *base = nullptr;
    bool pageable = false;
    const int rc = noalloc_setup(dev, &base, &pageable);
    if (rc != SPH_OK) return rc;
    long long *box = reinterpret_cast<long long *>(base + OFF_BOX);
    double *rb = reinterpret_cast<double *>(base + OFF_RB);
    uint64_t *ka = reinterpret_cast<uint64_t *>(base + OFF_K0), *kb = reinterpret_cast<uint64_t *>(base + OFF_K1);
    uint32_t *va = reinterpret_cast<uint32_t *>(base + OFF_V0), *vb = reinterpret_cast<uint32_t *>(base + OFF_V1);
    uint32_t *hist = reinterpret_cast<uint32_t *>(base + OFF_HIST);
    int *err = reinterpret_cast<int *>(base + OFF_ERR);
    const int nn = (int)n;
    const int nb = (nn + NA_TILE - 1) / NA_TILE;
    static_assert(NA_NB <= RS_DIRECT, "every block adds up the tiles' counts itself");
    // root cube and keys exactly as the octree build does (theta does not enter the keys)
    const int box_blocks = std::min(NA_BOX, (nn + 255) / 256);
    const int64_t row = 256 * (int64_t)nb;   // digit counts of one pass
    k_bbox_partial<<<box_blocks, 256, 0, st>>>(x, y, z, nn, box, hist, (int)(2 * row), err);
    launch_after(!capturing, k_bbox_final, 1, 256, 0, st, box, box_blocks, 0.5, rb);
    launch_after(!capturing, k_keys_hist, nb * RS_SUB, RS_THREADS, 0, st, x, y, z, nn, rb, nullptr, nullptr, nb, ka,
                 hist, err);
    // stable LSD radix sort, 8 passes of 8 bits, the last one into the caller's buffers
    for (int pass = 0; pass < RS_PASSES; ++pass) {
        const bool odd = pass & 1, last = pass == RS_PASSES - 1;
        launch_after(!capturing, k_rs_scatter, nb, RS_THREADS, 0, st, odd ? kb : ka,
                     pass == 0 ? nullptr : (odd ? vb : va), last ? keys_out : (odd ? ka : kb),
                     last ? reinterpret_cast<uint32_t *>(order_out) : (odd ? va : vb), nn, 8 * pass,
                     hist + pass % RS_HISTS * row, last ? nullptr : hist + (pass + 1) % RS_HISTS * row,
                     last ? nullptr : hist + (pass + 2) % RS_HISTS * row, nullptr, nullptr, nb, nullptr);
    }
    if (cudaGetLastError() != cudaSuccess) return SPH_ERR_CUDA;
    if (capturing) return SPH_OK;   // recorded; a replay's status is not read back
    // the status: written by a kernel where the device reaches pageable memory (as the functor calls' results are), which
    // saves the copy's detour (100,000 particles 138 -> 123 us; overlapped launches 140 -> 138)
    int herr = 0;
    const int word = pageable ? take_word() : -1;
    if (word >= 0) launch_after(true, k_publish, 1, 64, 0, st, err, 1, g_na_words + word);
    if ((word >= 0 ? cudaGetLastError()
                   : cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return SPH_ERR_CUDA;
    }
    if (word >= 0) {
        herr = *(volatile int *)(g_na_words + word);
        g_na_taken[word].store(false);
    }
    return (herr & ERR_NONFINITE) ? SPH_ERR_NONFINITE : SPH_OK;
}
