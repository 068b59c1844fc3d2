// Rows of bytes as 64-cell chunks: 16-byte pieces where rows are made of them,
// and for rows of any length and alignment coalesced spans staged in shared
// memory, from which each lane takes its cells as shifted words.
#pragma once

#include <stdint.h>

#include "bulk_device.cuh"
#include "conv_device.cuh"

namespace fs3d {

// bytes of a static material in v, as a byte mask
__device__ __forceinline__ uint32_t static_bytes(uint32_t v) {
    const uint32_t big = v & 0xFCFCFCFCu;
    return (((((big & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | big) & 0x80808080u) >> 7) * 0xFFu;
}

// New bytes of a chunk (w: the cells' codes), but static materials keep their old byte.
__device__ __forceinline__ void merge_statics(const uint32_t (&old)[16], uint32_t (&w)[16]) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const uint32_t keep = static_bytes(old[k]);
        w[k] = (w[k] & ~keep) | (old[k] & keep);
    }
}

// the n cells (a multiple of 16) at p, 16-byte aligned; cells past n as solid
__device__ __forceinline__ void load_pieces(const uint8_t* p, int n, uint32_t (&w)[16]) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        uint4 v = make_uint4(0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u);
        if (16 * u < n) v = reinterpret_cast<const uint4*>(p)[u];
        w[4 * u] = v.x;
        w[4 * u + 1] = v.y;
        w[4 * u + 2] = v.z;
        w[4 * u + 3] = v.w;
    }
}

__device__ __forceinline__ bool any_static(const uint32_t (&w)[16]) {
    uint32_t any = 0;
#pragma unroll
    for (int k = 0; k < 16; ++k) any |= w[k];
    return (any & 0xFCFCFCFCu) != 0;
}

// [g, g + n) between global memory and shared memory at sm, which is congruent
// to g modulo 16; by T threads (id: which of them)
template <bool STORE, int T>
__device__ __forceinline__ void move_span(uint8_t* g, uint8_t* sm, int n, int id) {
    const int head = (int)(-(intptr_t)reinterpret_cast<uintptr_t>(g) & 15);
    const int h = head < n ? head : n, body = (n - h) & ~15, t = h + body;
    const int i0 = id < h ? id : (id >= 16 && t + id - 16 < n ? t + id - 16 : -1);  // a single byte at either end
    if (i0 >= 0) {
        if (STORE) g[i0] = sm[i0];
        else sm[i0] = g[i0];
    }
    for (int i = h + 16 * id; i < t; i += 16 * T) {
        if (STORE) *reinterpret_cast<uint4*>(g + i) = *reinterpret_cast<const uint4*>(sm + i);
        else *reinterpret_cast<uint4*>(sm + i) = *reinterpret_cast<const uint4*>(g + i);
    }
}

// the n cells (at most 4N) at shared-memory address p, cells past n as solid
template <int N>
__device__ __forceinline__ void read_cells(const uint8_t* p, int n, uint32_t (&w)[N]) {
    const uint32_t m = smem_u32(p) & 3u;
    const uint32_t* pa = reinterpret_cast<const uint32_t*>(p - m);
    uint32_t lo = pa[0];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const int left = n - 4 * k;  // cells of the row from this word on
        uint32_t hi = 0;
        if (left + (int)m > 4) hi = pa[k + 1];
        w[k] = __funnelshift_r(lo, hi, 8 * m);
        lo = hi;
        if (left < 4) {
            const uint32_t keep = left <= 0 ? 0u : (1u << (8 * left)) - 1u;
            w[k] = (w[k] & keep) | (0x01010101u & ~keep);
        }
    }
}

// The first n of 4N cells (w) to shared-memory address p: aligned words whole,
// the chunk's ends byte by byte (a word there may hold another lane's cells).
template <int N>
__device__ __forceinline__ void write_cells(uint8_t* p, int n, const uint32_t (&w)[N]) {
    const int m = (int)(smem_u32(p) & 3u);
    uint32_t tail = 0;  // the word with the chunk's last cells
#pragma unroll
    for (int i = 0; i <= N; ++i) {
        const uint32_t before = i > 0 ? w[i - 1] : 0u, now = i < N ? w[i] : 0u;
        const uint32_t word = m ? __funnelshift_r(before, now, 8 * (4 - m)) : now;
        const int at = 4 * i - m;
        if (at >= 0 && at + 4 <= n) *reinterpret_cast<uint32_t*>(p + at) = word;
        else if (at < n && at > 0) tail = word;
    }
    const int e = (n + m) & ~3;  // offset (from p - m) of the word holding the last cells
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (c >= m && m && c - m < n) p[c - m] = (uint8_t)(w[0] >> (8 * (c - m)));
        if (e > 0 && e - m + c < n) p[e - m + c] = (uint8_t)(tail >> (8 * c));
        if (e == 0 && !m && c < n) p[c] = (uint8_t)(w[0] >> (8 * c));
    }
}

}  // namespace fs3d
