// Shared helpers of libfs3d: the counter-based hash of FS3D-rule v1, status
// plumbing and launch accounting.  Host and device see the same definitions.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <string>

#include "../../include/fs3d.h"
#include "per_context.h"

#define FS3D_HD __host__ __device__ __forceinline__

namespace fs3d {

// MurmurHash3 finalizers (Appleby, public domain).
FS3D_HD uint32_t fmix32(uint32_t h) {
    h ^= h >> 16;
    h *= 0x85ebca6bu;
    h ^= h >> 13;
    h *= 0xc2b2ae35u;
    h ^= h >> 16;
    return h;
}

FS3D_HD uint64_t fmix64(uint64_t k) {
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdULL;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ULL;
    k ^= k >> 33;
    return k;
}

// Per (world seed, step) key; computed once per step on the host.
FS3D_HD uint32_t stepkey(uint64_t seed, uint64_t t) {
    uint32_t h = fmix32(0x243F6A88u ^ (uint32_t)seed);
    h = fmix32(h ^ (uint32_t)(seed >> 32));
    h = fmix32(h ^ (uint32_t)t);
    h = fmix32(h ^ (uint32_t)(t >> 32));
    return h;
}

// Per block row (j along y, k along z).
FS3D_HD uint32_t rowkey(uint32_t sk, uint32_t j, uint32_t k) {
    uint32_t h = fmix32(sk ^ (0x85EBCA77u * (j + 1u)));
    return fmix32(h ^ (0xC2B2AE3Du * (k + 1u)));
}

// Random word w of slot s for the 32 blocks i in [32g, 32g+32) of a block
// row: bit (i & 31) belongs to block i.
FS3D_HD uint32_t plane(uint32_t rk, uint32_t g, uint32_t s, uint32_t w) {
    return fmix32(rk + 0x9E3779B9u * (1u + w + 8u * s + 64u * g));
}

FS3D_HD int nblocks(int n, int o) { return (n + o + 1) >> 1; }

// ---- status plumbing ----
fs3d_status set_error(fs3d_status s, const std::string& msg);
fs3d_status cuda_fail(cudaError_t e, const char* what);
void note_launch(uint64_t n = 1);
// Unique id of the calling thread's current CUDA context; false if no context
// is current yet (the runtime makes one current on its first device call) or
// the driver cannot tell.  A device address cached for one context is stale
// in another (after cudaDeviceReset, for example).
bool current_context_id(unsigned long long* id);
// the value of `p` for the current device and context (make: its value there)
template <class T, class Make>
T of_current_context(PerContext<T>& p, Make make) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return T{};
    }
    return p.get(
        dev,
        [] {
            unsigned long long id = 0;
            return current_context_id(&id) ? id : 0ull;
        },
        make);
}

// device memory for a call's own duration, stream-ordered (scratch.cpp)
cudaError_t scratch_alloc(void** p, size_t n, cudaStream_t st);
// unmaps what the scratch pool of the current device keeps unused
void scratch_give_back();
// cudaMalloc; out of memory, once more after scratch_give_back
cudaError_t device_alloc(void** p, size_t n);

// ---- chained launches: a kernel that begins with chain_wait() may be launched
// with launch_chained(), so that its CTAs are placed and its first instructions
// fetched while the kernel before it in the stream ends (programmatic
// dependent launch).  chain_wait() returns once that kernel has run and its
// writes are visible; nothing in global memory may be touched before it.  What
// the kernel before may have written is read with ordinary loads (no __ldg, no
// const __restrict__ parameter): the read-only path takes for granted that the
// data stand still while the kernel lives, which here begins before they do,
// and such a load may be moved ahead of the wait.
// chain_go() lets the next kernel's CTAs be placed; it stands at the end of
// each CTA's work (the end of the kernel does the same): CTAs placed any
// earlier hold registers that other streams' kernels could use (three 1024^3
// worlds stepped and drawn in turn: 315 us a pass with chain_go() first, 222
// with it last; a lone stream's steps take the same either way).
#ifdef __CUDACC__
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... P, class... A>
cudaError_t launch_chained(void (*fn)(P...), dim3 grid, unsigned block, cudaStream_t st, A... args) {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = grid;
    lc.blockDim = dim3(block);
    lc.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, fn, static_cast<P>(args)...);
}
#endif

}  // namespace fs3d

#define FS3D_CUDA(call)                                              \
    do {                                                             \
        cudaError_t e_ = (call);                                     \
        if (e_ != cudaSuccess) return ::fs3d::cuda_fail(e_, #call);  \
    } while (0)

#define FS3D_CHECK_LAUNCH(what)                                      \
    do {                                                             \
        cudaError_t e_ = cudaGetLastError();                         \
        if (e_ != cudaSuccess) return ::fs3d::cuda_fail(e_, what);   \
        ::fs3d::note_launch();                                       \
    } while (0)
