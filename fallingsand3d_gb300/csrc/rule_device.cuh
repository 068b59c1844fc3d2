// Device-side FS3D-rule v1: the scalar per-block rule (bytes) and the
// bit-sliced rule that runs 32 blocks per 32-bit word (bit planes).
#pragma once

#include <stdint.h>

#include "fs3d_common.h"

namespace fs3d {

__device__ __forceinline__ uint32_t draw_dev(uint32_t n, uint32_t rk, uint32_t i, uint32_t s) {
    if (n < 2u) return 0u;
    const uint32_t g = i >> 5, b = i & 31u;
    if (n == 2u) return (plane(rk, g, s, 0u) >> b) & 1u;
    uint32_t u = 0;
#pragma unroll
    for (uint32_t w = 0; w < 8u; ++w) u |= ((plane(rk, g, s, w) >> b) & 1u) << w;
    return u < 85u ? 0u : (u < 170u ? 1u : 2u);
}

__device__ __forceinline__ uint32_t has_zero_byte(uint32_t v) {
    return (v - 0x01010101u) & ~v & 0x80808080u;
}

// Can the block (top layer T, bottom layer B; byte q = column q, cells outside
// the grid hold 1) change?  Exact, by the stability property of the rule.
__device__ __forceinline__ bool block_can_move(uint32_t T, uint32_t B) {
    const uint32_t eT = has_zero_byte(T), eB = has_zero_byte(B);
    const uint32_t pT = has_zero_byte((T & 0xFEFEFEFEu) ^ 0x02020202u);
    const uint32_t wT = has_zero_byte(T ^ 0x03030303u), wB = has_zero_byte(B ^ 0x03030303u);
    return (pT && eB) || (wT && eT) || (wB && eB);
}

__device__ __forceinline__ uint32_t get_byte(uint64_t V, int s) { return (uint32_t)(V >> (8 * s)) & 0xFFu; }

// Runs the rule on one block held as 8 bytes (byte s = slot s; slots 0-3 top
// layer, 4-7 bottom layer, column q = dz*2+dx).  Returns the new bytes.
__device__ __forceinline__ uint64_t block_rule(uint64_t V, uint32_t rk, uint32_t i) {
    uint32_t moved = 0;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const uint32_t m = get_byte(V, s);
        if ((m != 2u && m != 3u) || ((moved >> s) & 1u)) continue;
        const int q = s & 3;
        int dst = -1;
        if (s < 4) {
            if (get_byte(V, 4 + q) == 0u) {
                dst = 4 + q;
            } else {
                uint32_t cand = 0;
#pragma unroll
                for (int q2 = 0; q2 < 4; ++q2)
                    if (q2 != q && get_byte(V, 4 + q2) == 0u) cand |= 1u << (4 + q2);
                if (cand) {
                    uint32_t r = draw_dev(__popc(cand), rk, i, (uint32_t)s);
                    while (r--) cand &= cand - 1u;
                    dst = __ffs(cand) - 1;
                }
            }
        }
        if (dst < 0 && m == 3u) {
            const int base = s & 4;
            uint32_t cand = 0;
#pragma unroll
            for (int q2 = 0; q2 < 4; ++q2)
                if (q2 != q && get_byte(V, base + q2) == 0u) cand |= 1u << (base + q2);
            if (cand) {
                uint32_t r = draw_dev(__popc(cand), rk, i, (uint32_t)s);
                while (r--) cand &= cand - 1u;
                dst = __ffs(cand) - 1;
            }
        }
        if (dst >= 0) {
            V &= ~(0xFFull << (8 * s));
            V = (V & ~(0xFFull << (8 * dst))) | ((uint64_t)m << (8 * dst));
            moved |= 1u << dst;
        }
    }
    return V;
}


// ---------------------------------------------------------------------------
// Bit-sliced rule.  Each 32-bit word holds one predicate for 32 consecutive
// blocks i = 32g .. 32g+31 of a block row (bit i & 31).  Per slot s the input
// is (A, B): (0,0) empty, (0,1) solid, (1,0) sand, (1,1) water.
// ---------------------------------------------------------------------------

// Choosing among up to three ordered candidate masks c1..c3 for the blocks in
// `mov` (each has at least one): the r-th candidate, r = draw(n) with n their
// number, from the slot's random words P_w = plane(rk, g, s, w).  draw(2) =
// P_0; draw(3) compares u = sum_w P_w << w with 85 and 170.
//
// The comparisons run from the lowest bit up, so no word is kept: with ge the
// answer for the bits below, a constant's bits 1 then 0 turn it into p1 | (p0 &
// ge) and its bits 0 then 1 into p1 & (p0 | ge); 85 = 0b01010101 and 170 =
// 0b10101010 repeat one of the two four times, one three-input operation per
// pair of words and constant.
__device__ __forceinline__ void draw3(uint32_t rk, uint32_t g, uint32_t s, uint32_t p0, uint32_t& ge85,
                                      uint32_t& ge170) {
    ge85 = ge170 = 0xFFFFFFFFu;
#pragma unroll
    for (uint32_t w = 0; w < 8u; w += 2u) {
        const uint32_t lo = w ? plane(rk, g, s, w) : p0, hi = plane(rk, g, s, w + 1u);
        ge85 = hi | (lo & ge85);
        ge170 = hi & (lo | ge170);
    }
}

// Destination masks, one candidate per block of `mov`, from the blocks that
// pass over their first candidate (past1) and their second too (past2).
__device__ __forceinline__ void bs_pick(uint32_t mov, uint32_t c1, uint32_t c2, uint32_t past1, uint32_t past2,
                                        uint32_t& d1, uint32_t& d2, uint32_t& d3) {
    d1 = mov & c1 & ~past1;
    d2 = mov & c2 & ((c1 & past1 & ~past2) | (~c1 & ~past1));
    d3 = mov & ~d1 & ~d2;
}

// A row-pair word's draws, hashed where a slot needs them (throughput: about
// half of the slots of a settled warp need none).
struct LazyDraws {
    static constexpr bool kReady = false;
    uint32_t rk, g;
    __device__ __forceinline__ void select(uint32_t mov, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t s, uint32_t& d1,
                                           uint32_t& d2, uint32_t& d3) const {
        const uint32_t two = (c1 & c2) | (c1 & c3) | (c2 & c3);
        uint32_t past1 = 0, past2 = 0;
        if (mov & two) {
            const uint32_t three = c1 & c2 & c3;
            const uint32_t p0 = plane(rk, g, s, 0u);
            past1 = two & ~three & p0;
            if (mov & three) {
                uint32_t ge85, ge170;
                draw3(rk, g, s, p0, ge85, ge170);
                past1 |= three & ge85;
                past2 = three & ge170;
            }
        }
        bs_pick(mov, c1, c2, past1, past2, d1, d2, d3);
    }
};

// The draws of all eight slots, hashed beforehand: they depend on the world's
// seed, the step and the place only, so a caller that has to wait for cells
// hashes them meanwhile, and the slots' serial chain runs without branches.
struct ReadyDraws {
    static constexpr bool kReady = true;
    uint32_t p0[8], ge85[8], ge170[8];
    __device__ __forceinline__ void fill(uint32_t rk, uint32_t g) {
#pragma unroll
        for (uint32_t s = 0; s < 8u; ++s) {
            p0[s] = plane(rk, g, s, 0u);
            draw3(rk, g, s, p0[s], ge85[s], ge170[s]);
        }
    }
    __device__ __forceinline__ void select(uint32_t mov, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t s, uint32_t& d1,
                                           uint32_t& d2, uint32_t& d3) const {
        const uint32_t two = (c1 & c2) | (c1 & c3) | (c2 & c3), three = c1 & c2 & c3;
        bs_pick(mov, c1, c2, (three & ge85[s]) | (two & ~three & p0[s]), three & ge170[s], d1, d2, d3);
    }
};

// The three other columns of q, in increasing order.
__host__ __device__ constexpr int other_col(int q, int n) { return n < q ? n : n + 1; }

// The rule's activity mask of 32 blocks (W = water, E = empty per slot): the
// blocks with a particle that has an empty candidate (a top particle over an
// empty bottom cell, or water beside an empty cell of its layer).  A block
// outside the mask does not change, whatever the draws; a block in it does.
__device__ __forceinline__ uint32_t activity_mask(const uint32_t (&A)[8], const uint32_t (&W)[8],
                                                  const uint32_t (&E)[8]) {
    const uint32_t etop = E[0] | E[1] | E[2] | E[3], ebot = E[4] | E[5] | E[6] | E[7];
    return ((A[0] | A[1] | A[2] | A[3]) & ebot) | ((W[0] | W[1] | W[2] | W[3]) & etop) |
           ((W[4] | W[5] | W[6] | W[7]) & ebot);
}

// Runs one step of the rule on 32 blocks.  A[s], B[s] in/out per slot s.
// Returns the mask of blocks that changed.
//
// Bound: the integer instructions of the eight dependent slots, most of them
// the draws' hashes (each slot's words are drawn when any of a warp's 1024
// blocks needs them).  A top slot chooses once for its diagonal and its
// sideways moves together, since a block has candidates of one kind only:
// with a choice for each, the same words were hashed twice.  One choice a slot
// and the comparison from the lowest bit up: 2048 settled worlds' segment and
// snapshot 1260 -> 1073 us, two segments of 512 fresh worlds 2545 -> 2309 us,
// the 512^3 byte step 67.8 -> 64.6 us while everything falls.
template <class Draws>
__device__ __forceinline__ uint32_t bs_rule(uint32_t (&A)[8], uint32_t (&B)[8], const Draws& draws) {
    // Only the empty and water planes change as slots are visited.  A slot
    // acts exactly on the particles it held at the start (A[s]): a particle
    // only ever moves into an empty cell, so a cell's own particle is still
    // there when its slot comes, and a particle that arrives is never moved
    // again.  The particle plane is rebuilt at the end from E and the solids.
    uint32_t W[8], E[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        W[s] = A[s] & B[s];
        E[s] = ~(A[s] | B[s]);
    }
    const uint32_t active = activity_mask(A, W, E);
    if (!active) return 0u;
#pragma unroll
    for (int s = 0; s < 8; ++s) B[s] = ~A[s] & B[s];  // from here on B holds the solids, which never change
    uint32_t changed = 0;  // a block changes iff one of its particles moves
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const int q = s & 3, base = s & 4;
        const uint32_t act = A[s] & active;
        if (!Draws::kReady && !act) continue;
        const uint32_t wat = W[s];  // on the acting blocks: the slot's own water, untouched so far
        // the other cells of the slot's own layer (where water moves sideways) and,
        // for a top slot, of the layer below; a particle takes a diagonal when
        // there is one, so one choice serves both: the candidates of a block are
        // its diagonal ones, or its sideways ones when it has no diagonal
        uint32_t c1 = E[base + other_col(q, 0)], c2 = E[base + other_col(q, 1)], c3 = E[base + other_col(q, 2)];
        uint32_t fall = 0, down = 0, rest = act;
        if (s < 4) {
            const uint32_t g1 = E[4 + other_col(q, 0)], g2 = E[4 + other_col(q, 1)], g3 = E[4 + other_col(q, 2)];
            fall = act & E[4 + q];
            rest = act & ~E[4 + q];
            down = g1 | g2 | g3;  // the blocks with a diagonal
            c1 = g1 | (c1 & ~down);
            c2 = g2 | (c2 & ~down);
            c3 = g3 | (c3 & ~down);
        }
        const uint32_t mov = rest & (down | wat) & (c1 | c2 | c3);
        const uint32_t moved = fall | mov;
        if (!Draws::kReady && !moved) continue;
        changed |= moved;
        W[s] &= ~moved;
        E[s] |= moved;
        uint32_t d1 = 0, d2 = 0, d3 = 0;
        if (Draws::kReady || mov) draws.select(mov, c1, c2, c3, (uint32_t)s, d1, d2, d3);
        if (s < 4) {
            E[4 + q] &= ~fall;
            W[4 + q] |= fall & wat;
            const uint32_t dw = down & wat;
            E[4 + other_col(q, 0)] &= ~(d1 & down);
            W[4 + other_col(q, 0)] |= d1 & dw;
            E[4 + other_col(q, 1)] &= ~(d2 & down);
            W[4 + other_col(q, 1)] |= d2 & dw;
            E[4 + other_col(q, 2)] &= ~(d3 & down);
            W[4 + other_col(q, 2)] |= d3 & dw;
        }
        // only water moves sideways (down is empty for a bottom slot)
        const uint32_t sw = ~down;
        E[base + other_col(q, 0)] &= ~(d1 & sw);
        W[base + other_col(q, 0)] |= d1 & sw;
        E[base + other_col(q, 1)] &= ~(d2 & sw);
        W[base + other_col(q, 1)] |= d2 & sw;
        E[base + other_col(q, 2)] &= ~(d3 & sw);
        W[base + other_col(q, 2)] |= d3 & sw;
    }
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const uint32_t solid = B[s];
        A[s] = ~E[s] & ~solid;
        B[s] = W[s] | solid;
    }
    return changed;
}


__device__ __forceinline__ uint32_t bs_rule(uint32_t (&A)[8], uint32_t (&B)[8], uint32_t rk, uint32_t g) {
    return bs_rule(A, B, LazyDraws{rk, g});
}

// The half block at the right end of an odd-phase row (x = X-1 present,
// x = X outside) has only its dx=0 column: cells r = layer*2 + dz with bit r
// of P (sand or water), W (water), E (empty).  Every candidate set has at
// most one cell there, so no random draw is ever taken.
__device__ __forceinline__ void half_block_rule(uint32_t& P, uint32_t& W, uint32_t& E) {
    uint32_t M = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const uint32_t bit = 1u << r;
        if (!(P & bit) || (M & bit)) continue;
        int dst = -1;
        if (r < 2) {
            const int below = 2 + r, diag = 3 - r;  // straight down, then the other bottom cell
            if (E & (1u << below))
                dst = below;
            else if (E & (1u << diag))
                dst = diag;
        }
        if (dst < 0 && (W & bit)) {
            const int side = r ^ 1;  // the other cell of the same layer
            if (E & (1u << side)) dst = side;
        }
        if (dst >= 0) {
            const uint32_t d = 1u << dst;
            if (W & bit) W |= d;
            W &= ~bit;
            P = (P & ~bit) | d;
            E = (E | bit) & ~d;
            M |= d;
        }
    }
}

// The bit-sliced slots (A, B per slot) of the 32 blocks of a block row-pair
// that lane gl holds, in the layout rowpair_core describes.  Every lane of the
// warp calls this together (the odd phase takes a bit from the left lane).
__device__ __forceinline__ void rowpair_slots(const uint4 (&q)[4], int o, int gl, int G, uint32_t (&A)[8],
                                              uint32_t (&B)[8]) {
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int s0 = (a >> 1) * 4 + (a & 1) * 2;
        if (o == 0) {
            A[s0] = q[a].x;
            B[s0] = q[a].z;
            A[s0 + 1] = q[a].y;
            B[s0 + 1] = q[a].w;
        } else {
            uint32_t ua = 0u, ub = 0xFFFFFFFFu;  // x = -1 lies outside: solid
            if (G > 1) {
                const uint32_t sa = __shfl_up_sync(0xFFFFFFFFu, q[a].y, 1);
                const uint32_t sb = __shfl_up_sync(0xFFFFFFFFu, q[a].w, 1);
                if (gl > 0) {
                    ua = sa;
                    ub = sb;
                }
            }
            A[s0] = (q[a].y << 1) | (ua >> 31);
            B[s0] = (q[a].w << 1) | (ub >> 31);
            A[s0 + 1] = q[a].x;
            B[s0 + 1] = q[a].z;
        }
    }
}

// One step of one block row-pair held as plane words.  The pair's four rows
// (a = layer*2 + dz: top z0, top z1, bottom z0, bottom z1) cover x in
// [64*gl, 64*gl+64): lane gl of a group of G consecutive lanes (G a power of
// two; every lane of the warp must call this together, `has` false for lanes
// without a word).  q[a] = {A even, A odd, B even, B odd}, updated in place;
// rows outside the world are passed as solid.  In the odd phase the dx=0 word
// is the odd word shifted up one bit with bit 31 of the left lane's odd word
// carried in (x = -1 is solid), and the left lane receives its new bit 31
// back; when the row width is a multiple of 64 (`half_at_end`) the last lane
// also runs the half block at x = 64*nw - 1.
template <class Draws>
__device__ __forceinline__ void rowpair_core(uint4 (&q)[4], bool has, int o, const Draws& draws, int gl, int G, int nw,
                                             bool half_at_end) {
    uint32_t A[8], B[8];
    rowpair_slots(q, o, gl, G, A, B);
    if (has) bs_rule(A, B, draws);
    if (o == 0) {
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int s0 = (a >> 1) * 4 + (a & 1) * 2;
            q[a] = make_uint4(A[s0], A[s0 + 1], B[s0], B[s0 + 1]);
        }
        return;
    }
    // new bit 31 of this lane's odd words: from the right neighbour's dx=0
    // word, from the half block, or unchanged (padding past X)
    uint32_t ta = 0, tb = 0;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        ta |= (q[a].y >> 31) << a;
        tb |= (q[a].w >> 31) << a;
    }
    if (has && gl == nw - 1 && half_at_end) {
        uint32_t P = ta, W = ta & tb, E = ~(ta | tb) & 0xFu;
        half_block_rule(P, W, E);
        ta = P;
        tb = (W | (~P & ~E)) & 0xFu;
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int s0 = (a >> 1) * 4 + (a & 1) * 2;
        uint32_t na = (ta >> a) & 1u, nb = (tb >> a) & 1u;
        if (G > 1) {
            const uint32_t da = __shfl_down_sync(0xFFFFFFFFu, A[s0], 1);
            const uint32_t db = __shfl_down_sync(0xFFFFFFFFu, B[s0], 1);
            if (gl < nw - 1) {
                na = da & 1u;
                nb = db & 1u;
            }
        }
        q[a] = make_uint4(A[s0 + 1], (A[s0] >> 1) | (na << 31), B[s0 + 1], (B[s0] >> 1) | (nb << 31));
    }
}

__device__ __forceinline__ void rowpair_core(uint4 (&q)[4], bool has, int o, uint32_t rk, int gl, int G, int nw,
                                             bool half_at_end) {
    rowpair_core(q, has, o, LazyDraws{rk, (uint32_t)gl}, gl, G, nw, half_at_end);
}

// Whether lane gl's blocks of a block row-pair (q as for rowpair_core, only
// read) can change in phase o: the rule's activity mask, and for the half
// block at the end of an odd-phase row (`half_at_end`, last lane) a particle
// and an empty cell in it (a superset of its moves).  Every lane of the warp
// calls this together; lanes with `has` false answer false.
__device__ __forceinline__ bool rowpair_can_change(const uint4 (&q)[4], bool has, int o, int gl, int G, int nw,
                                                   bool half_at_end) {
    uint32_t A[8], B[8], W[8], E[8];
    rowpair_slots(q, o, gl, G, A, B);
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        W[s] = A[s] & B[s];
        E[s] = ~(A[s] | B[s]);
    }
    bool can = has && activity_mask(A, W, E) != 0u;
    if (o == 1 && has && half_at_end && gl == nw - 1) {
        uint32_t ta = 0, tb = 0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            ta |= (q[a].y >> 31) << a;
            tb |= (q[a].w >> 31) << a;
        }
        if (ta != 0u && (~(ta | tb) & 0xFu) != 0u) can = true;
    }
    return can;
}

}  // namespace fs3d
