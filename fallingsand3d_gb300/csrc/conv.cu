// Byte grids <-> bit planes, one world or many per launch.  A CTA takes whole
// rows of one world, one 64-cell chunk a thread, so its bytes are one span.
//
// Bound: HBM (admission 1 B read and 0.25 B written a cell, read-back the
// other way; rows of 16 to 48 cells hold 64 in their planes).  Read-back of 700
// mixed worlds, 137 MB: 89 us with a 64-byte chunk a thread, 53 with four
// 16-byte pieces a thread in flight, 43 with two thirds of the set-up (3.2 TB/s
// of bytes and 1.2 of planes).  Ragged rows (256 worlds of sides 10 to 130, 23
// MB): 116 us byte by byte, 21 through the span; admission 27 and 18.
#include <stdint.h>

#include "fs3d_common.h"
#include "planes.h"
#include "span_device.cuh"

namespace fs3d {

namespace {

struct ConvSpan {
    ConvJob jb;
    int64_t row0;
    int rows, bytes;
};

__device__ __forceinline__ ConvSpan conv_span(const ConvJob* jobs, const ConvBlock* blocks, const ConvJob& one,
                                              int chunks, int* j) {
    ConvSpan c;
    if (blocks) {
        const ConvBlock b = blocks[blockIdx.x];
        c.jb = jobs[b.job];
        c.row0 = b.row0;
        *j = b.job;
    } else {
        c.jb = one;
        c.row0 = (int64_t)blockIdx.x * conv_rows(one.nw, chunks);
        *j = 0;
    }
    const int64_t left = (int64_t)c.jb.Y * c.jb.Z - c.row0;
    c.rows = (int)min((int64_t)conv_rows(c.jb.nw, chunks), left);
    c.bytes = c.rows * c.jb.X;
    return c;
}

__device__ __forceinline__ bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

__global__ void __launch_bounds__(kConvThreads) k_bytes_to_planes(const ConvJob* __restrict__ jobs,
                                                                  const ConvBlock* __restrict__ blocks, ConvJob one,
                                                                  int* flags) {
    __shared__ __align__(16) uint8_t span[kConvThreads * 64 + 16];
    int j;
    const ConvSpan c = conv_span(jobs, blocks, one, kConvChunks, &j);
    const int X = c.jb.X, nw = c.jb.nw, tid = threadIdx.x;
    uint8_t* in = c.jb.bytes + c.row0 * X;
    const int r = tid / nw, g = tid - r * nw, n = min(64, X - 64 * g);
    const bool mine = r < c.rows;
    uint32_t w[16];
    if ((X & 15) == 0 && aligned16(in)) {
        if (mine) load_pieces(in + r * X + 64 * g, n, w);
    } else {
        uint8_t* sm = span + (reinterpret_cast<uintptr_t>(in) & 15u);
        move_span<false, kConvThreads>(in, sm, c.bytes, tid);
        __syncthreads();
        if (mine) read_cells(sm + r * X + 64 * g, n, w);
    }
    bool big = false;
    if (mine) {
        big = any_static(w);
        c.jb.rows[c.row0 * nw + tid] = bytes_to_planes64(w, big);
    }
    if (flags && __syncthreads_or(big) && tid == 0) atomicOr(flags + j, 1);  // keep its bytes
}

// A thread converts 16-cell pieces.  Where rows are whole 16-byte pieces it
// writes them straight out, a warp 512 consecutive bytes at a time; others go
// into the span in shared memory and from there out in 16-byte pieces, static
// bytes coming in the same way.  (A 64-byte chunk a thread took 66 registers, so
// 24 warps per SM, and had one load in flight in each.)
__global__ void __launch_bounds__(kConvThreads, 6) k_planes_to_bytes(const ConvJob* __restrict__ jobs,
                                                                     const ConvBlock* __restrict__ blocks, ConvJob one,
                                                                     const int* skip_if_set) {
    __shared__ __align__(16) uint8_t span[kConvChunksBack * 64 + 16];
    if (skip_if_set && *(volatile const int*)skip_if_set) return;
    int j;
    const ConvSpan c = conv_span(jobs, blocks, one, blocks ? kConvChunksBack : kConvChunks, &j);
    const int X = c.jb.X, nw = c.jb.nw, tid = threadIdx.x;
    uint8_t* out = c.jb.bytes + c.row0 * X;
    const uint8_t* st = c.jb.statics;
    if (!st && c.jb.static_flag && *c.jb.static_flag) st = c.jb.static_src;
    if (st) st += c.row0 * X;
    const uint4* __restrict__ rows = c.jb.rows + c.row0 * nw;
    const bool whole = (X & 15) == 0 && aligned16(out) && aligned16(st);
    const bool staged = !whole && st && ((reinterpret_cast<uintptr_t>(st) ^ reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
    uint8_t* sm = span + (reinterpret_cast<uintptr_t>(out) & 15u);
    if (staged) {
        move_span<false, kConvThreads>(const_cast<uint8_t*>(st), sm, c.bytes, tid);
        __syncthreads();
    }
    // piece i: row i / pr, cells 16 (i % pr) on (i < 2^16: the multiply-high divides exactly)
    const int pr = (X + 15) >> 4, np = c.rows * pr;
    const uint32_t magic = c.jb.magic;
    constexpr int kDepth = 4;  // pieces a thread has in flight
    for (int base = tid; base < np; base += kDepth * kConvThreads) {
        uint4 q[kDepth];
        int row[kDepth], px[kDepth];
#pragma unroll
        for (int d = 0; d < kDepth; ++d) {
            const int i = min(base + d * kConvThreads, np - 1);
            row[d] = pr == 1 ? i : (int)__umulhi((uint32_t)i, magic);
            px[d] = i - row[d] * pr;
            q[d] = __ldg(rows + row[d] * nw + (px[d] >> 2));
        }
#pragma unroll
        for (int d = 0; d < kDepth; ++d) {
            const int i = base + d * kConvThreads;
            if (i >= np) break;
            uint32_t t[4];
            planes_transposed(q[d], t);
            // the packed piece u: byte u of each
            const uint32_t u = (uint32_t)px[d] & 3u, s = u | (u + 4u) << 4;
            const uint32_t p = __byte_perm(__byte_perm(t[0], t[1], s), __byte_perm(t[2], t[3], s), 0x5410);
            uint4 v = piece_bytes(p);
            if (whole) {
                if (st) {
                    const uint4 old = reinterpret_cast<const uint4*>(st)[i];
                    v = make_uint4(with_static(v.x, old.x), with_static(v.y, old.y), with_static(v.z, old.z),
                                   with_static(v.w, old.w));
                }
                reinterpret_cast<uint4*>(out)[i] = v;
                continue;
            }
            const int at = row[d] * X + 16 * px[d], n = min(16, X - 16 * px[d]);
            uint32_t w[4] = {v.x, v.y, v.z, v.w};
            if (staged) {
                uint32_t old[4];
                read_cells(sm + at, n, old);
#pragma unroll
                for (int k = 0; k < 4; ++k) w[k] = with_static(w[k], old[k]);
            } else if (st) {
                for (int x = 0; x < n; ++x)
                    if (((w[x >> 2] >> (8 * (x & 3))) & 3u) == 1u) patch_byte(w, x, st[at + x]);
            }
            write_cells(sm + at, n, w);  // (a thread reads and writes its own cells of the span only)
        }
    }
    if (whole) return;
    __syncthreads();
    move_span<true, kConvThreads>(out, sm, c.bytes, tid);
}

static ConvJob one_job(const uint4* rows, const uint8_t* statics, const uint8_t* bytes, int X, int Y, int Z) {
    ConvJob j{};
    j.rows = const_cast<uint4*>(rows);
    j.statics = statics;
    j.bytes = const_cast<uint8_t*>(bytes);
    j.X = X;
    j.Y = Y;
    j.Z = Z;
    j.nw = plane_nw(X);
    j.magic = conv_magic(X);
    return j;
}

fs3d_status planes_from_bytes(const uint8_t* g, int X, int Y, int Z, uint4* rows, cudaStream_t st, int* statics_flag) {
    k_bytes_to_planes<<<(unsigned)conv_blocks(Y, Z, plane_nw(X), kConvChunks), kConvThreads, 0, st>>>(
        nullptr, nullptr, one_job(rows, nullptr, g, X, Y, Z), statics_flag);
    FS3D_CHECK_LAUNCH("bytes->planes launch");
    return FS3D_OK;
}

fs3d_status planes_from_bytes_multi(const ConvJob* jobs, const ConvBlock* blocks, int64_t nblocks, int* flags,
                                    cudaStream_t st) {
    if (nblocks <= 0) return FS3D_OK;
    k_bytes_to_planes<<<(unsigned)nblocks, kConvThreads, 0, st>>>(jobs, blocks, ConvJob{}, flags);
    FS3D_CHECK_LAUNCH("bytes->planes (many worlds) launch");
    return FS3D_OK;
}

fs3d_status planes_to_bytes(const uint4* rows, const uint8_t* statics, int X, int Y, int Z, uint8_t* g,
                            cudaStream_t st, const int* skip_if_set) {
    k_planes_to_bytes<<<(unsigned)conv_blocks(Y, Z, plane_nw(X), kConvChunks), kConvThreads, 0, st>>>(
        nullptr, nullptr, one_job(rows, statics, g, X, Y, Z), skip_if_set);
    FS3D_CHECK_LAUNCH("planes->bytes launch");
    return FS3D_OK;
}

fs3d_status planes_to_bytes_multi(const ConvJob* jobs, const ConvBlock* blocks, int64_t nblocks, cudaStream_t st) {
    if (nblocks <= 0) return FS3D_OK;
    k_planes_to_bytes<<<(unsigned)nblocks, kConvThreads, 0, st>>>(jobs, blocks, ConvJob{}, nullptr);
    FS3D_CHECK_LAUNCH("planes->bytes (many worlds) launch");
    return FS3D_OK;
}

}  // namespace fs3d
