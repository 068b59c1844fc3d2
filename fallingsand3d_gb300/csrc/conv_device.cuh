// Byte grid <-> bit-plane conversion of 64-cell chunks with byte-parallel
// (SWAR) arithmetic, shared by the byte step kernel and the conversion
// kernels.  A plane word is {A even, A odd, B even, B odd}: bit m of an even
// word is cell 2m of the chunk, of an odd word cell 2m + 1.  A value 0..3 is
// its own 2-bit code (A = bit 1, B = bit 0); any value >= 4 is static and
// solid, code (0,1).
#pragma once

#include <stdint.h>

namespace fs3d {

// Every byte of v with a static material (>= 4) turned into a solid's code (1).
__device__ __forceinline__ uint32_t statics_to_solid(uint32_t v) {
    const uint32_t big = v & 0xFCFCFCFCu;
    const uint32_t nz = ((big & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | big;  // bit 7 set iff the byte is >= 4
    const uint32_t m = ((nz & 0x80808080u) >> 7) * 0xFFu;
    return (v & ~m) | (0x01010101u & m);
}

// The bytes of four words, transposed: byte g of q[i] = byte i of p[g].
__device__ __forceinline__ void transpose4(const uint32_t (&p)[4], uint32_t (&q)[4]) {
    const uint32_t a = __byte_perm(p[0], p[1], 0x5140), b = __byte_perm(p[2], p[3], 0x5140);
    const uint32_t c = __byte_perm(p[0], p[1], 0x7362), d = __byte_perm(p[2], p[3], 0x7362);
    q[0] = __byte_perm(a, b, 0x5410);
    q[1] = __byte_perm(a, b, 0x7632);
    q[2] = __byte_perm(c, d, 0x5410);
    q[3] = __byte_perm(c, d, 0x7632);
}

// Four words of a 16-cell piece (codes 0..3 in their bytes) in one: byte i
// holds the codes of cells i, 4 + i, 8 + i, 12 + i from its low bits up.
// Multiply-adds, which leave the logic unit free (it bounds the byte step).
__device__ __forceinline__ uint32_t pack_piece(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
    return w0 + 4u * (w1 + 4u * (w2 + 4u * w3));
}

// The four packed pieces of 64 cells -> plane word.  After the transposition
// byte g of t[i] holds cells 16g + i, + 4 + i, + 8 + i, + 12 + i: an even i
// gives even cells, whose plane bits are 8g + 2j + i/2 for j = 0..3.
__device__ __forceinline__ uint4 pieces_to_planes(const uint32_t (&p)[4]) {
    uint32_t t[4];
    transpose4(p, t);
    return make_uint4(((t[0] >> 1) & 0x55555555u) | (t[2] & 0xAAAAAAAAu), ((t[1] >> 1) & 0x55555555u) | (t[3] & 0xAAAAAAAAu),
                      (t[0] & 0x55555555u) | ((t[2] << 1) & 0xAAAAAAAAu), (t[1] & 0x55555555u) | ((t[3] << 1) & 0xAAAAAAAAu));
}

// and back: byte u of t[0..3] are the bytes of packed piece u
__device__ __forceinline__ void planes_transposed(const uint4& q, uint32_t (&t)[4]) {
    t[0] = (q.z & 0x55555555u) | ((q.x << 1) & 0xAAAAAAAAu);
    t[1] = (q.w & 0x55555555u) | ((q.y << 1) & 0xAAAAAAAAu);
    t[2] = ((q.z >> 1) & 0x55555555u) | (q.x & 0xAAAAAAAAu);
    t[3] = ((q.w >> 1) & 0x55555555u) | (q.y & 0xAAAAAAAAu);
}
__device__ __forceinline__ void planes_to_pieces(const uint4& q, uint32_t (&p)[4]) {
    uint32_t t[4];
    planes_transposed(q, t);
    transpose4(t, p);
}

// word j (cells 4j .. 4j + 3) of a packed piece
__device__ __forceinline__ uint32_t piece_word(uint32_t p, int j) { return (p >> (2 * j)) & 0x03030303u; }
__device__ __forceinline__ uint4 piece_bytes(uint32_t p) {
    return make_uint4(piece_word(p, 0), piece_word(p, 1), piece_word(p, 2), piece_word(p, 3));
}

// 64 cells (16 little-endian words, cell 4k + i in byte i of word k) -> plane
// word; `big`: some byte is a static material
__device__ __forceinline__ uint4 bytes_to_planes64(const uint32_t (&w)[16], bool big) {
    uint32_t p[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        uint32_t v[4] = {w[4 * g], w[4 * g + 1], w[4 * g + 2], w[4 * g + 3]};
        if (big)
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = statics_to_solid(v[j]);
        p[g] = pack_piece(v[0], v[1], v[2], v[3]);
    }
    return pieces_to_planes(p);
}

// plane word -> the codes of its 64 cells as 16 little-endian words
__device__ __forceinline__ void planes_to_words64(const uint4& q, uint32_t (&w)[16]) {
    uint32_t p[4];
    planes_to_pieces(q, p);
#pragma unroll
    for (int k = 0; k < 16; ++k) w[k] = piece_word(p[k >> 2], k & 3);
}

// codes with a solid's (1) replaced by its static byte
__device__ __forceinline__ uint32_t with_static(uint32_t codes, uint32_t statics) {
    const uint32_t m = (codes & ~(codes >> 1) & 0x01010101u) * 0xFFu;
    return (codes & ~m) | (statics & m);
}

// cell x of the words w set to byte v (static indexing of w)
template <int N>
__device__ __forceinline__ void patch_byte(uint32_t (&w)[N], int x, uint32_t v) {
#pragma unroll
    for (int k = 0; k < N; ++k)
        if (k == x >> 2) w[k] = (w[k] & ~(0xFFu << (8 * (x & 3)))) | (v << (8 * (x & 3)));
}

}  // namespace fs3d
