// Device memory that a call needs for its own duration.
//
// The device's default pool returns its memory to the system at every
// synchronisation, so a caller that waits for each result (a frame loop, a
// script's run) paid for mapping it again: 115 to 145 us for the 37 MB of a
// full-HD mesh frame.  This pool, one per device and context, keeps at most
// kScratchKept bytes across a synchronisation, and gives those back when an
// allocation of the library fails.
#include <mutex>

#include "fs3d_common.h"

namespace fs3d {
namespace {

// a full-HD mesh frame takes 37 MB, a drop-in run of 512^3 cells 34 MB
constexpr unsigned long long kScratchKept = 64ull << 20;
constexpr int kMaxDevices = 64;

struct ScratchPool {
    unsigned long long ctx = 0;  // the context it was made in (0: none)
    cudaMemPool_t pool = nullptr, standard = nullptr;  // this pool, and the device's default one
};
ScratchPool g_pools[kMaxDevices];
std::mutex g_pools_mu;

// The current device's pool; null if it has none, or while the caller has made
// another pool than the default the device's current one: scratch then comes
// from that, as every stream-ordered allocation does.
cudaMemPool_t scratch_pool() {
    int dev = 0;
    unsigned long long ctx = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices || !current_context_id(&ctx) || !ctx)
        return nullptr;
    cudaMemPool_t current = nullptr;
    if (cudaDeviceGetMemPool(&current, dev) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(g_pools_mu);
    ScratchPool& s = g_pools[dev];
    if (s.ctx == ctx) return current == s.standard ? s.pool : nullptr;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    unsigned long long kept = kScratchKept;
    // (another stream of this thread may be capturing)
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    s.ctx = ctx;
    if (cudaMemPoolCreate(&s.pool, &props) != cudaSuccess) s.pool = nullptr;
    if (s.pool && cudaMemPoolSetAttribute(s.pool, cudaMemPoolAttrReleaseThreshold, &kept) != cudaSuccess) s.pool = nullptr;
    if (s.pool && cudaDeviceGetDefaultMemPool(&s.standard, dev) != cudaSuccess) s.pool = nullptr;
    cudaThreadExchangeStreamCaptureMode(&mode);
    cudaGetLastError();
    return current == s.standard ? s.pool : nullptr;
}

}  // namespace

// Stream-ordered: free with cudaFreeAsync.  While the stream is captured, and
// when the pool cannot serve it, the memory comes from the default pool.
cudaError_t scratch_alloc(void** p, size_t n, cudaStream_t st) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone)
        if (cudaMemPool_t pool = scratch_pool()) {
            if (cudaMallocFromPoolAsync(p, n, pool, st) == cudaSuccess) return cudaSuccess;
            cudaGetLastError();
            scratch_give_back();
        }
    return cudaMallocAsync(p, n, st);
}

void scratch_give_back() {
    int dev = 0;
    unsigned long long ctx = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices || !current_context_id(&ctx)) return;
    std::lock_guard<std::mutex> lock(g_pools_mu);
    if (g_pools[dev].pool && g_pools[dev].ctx == ctx) cudaMemPoolTrimTo(g_pools[dev].pool, 0);
}

cudaError_t device_alloc(void** p, size_t n) {
    cudaError_t e = cudaMalloc(p, n);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    scratch_give_back();
    return cudaMalloc(p, n);
}

}  // namespace fs3d
