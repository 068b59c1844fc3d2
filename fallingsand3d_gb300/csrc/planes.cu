// Bit-plane world format and the multi-world bit-sliced step.
//
// Format.  A world of X*Y*Z cells is stored as Y*Z rows (row r = y*Z + z) of
// nw = ceil(X/64) uint4 words; word g of a row covers x in [64g, 64g+64) and
// holds {A even, A odd, B even, B odd}: bit m of an even word is x = 64g+2m,
// of an odd word x = 64g+2m+1.  (A,B) = (0,0) empty, (0,1) solid, (1,0) sand,
// (1,1) water; cells past X are solid.  Static cells never change, so their
// byte values (stone, or any material >= 4) are taken from an optional byte
// copy of the initial grid when the world is read back.
//
// Step.  The blocks of a block row that start in word g (i = 32g .. 32g+31)
// are evaluated together: in the even phase their dx=0 / dx=1 cells are the
// even / odd words of g; in the odd phase (blocks start at odd x) the dx=0
// cells are the odd word shifted up one bit with the top bit of word g-1
// carried in, and the dx=1 cells are the even word.  A lane group of
// G = pow2ceil(nw) lanes handles one block row-pair (4 rows); lane g owns
// storage word g and the carried bit travels by warp shuffle, so each bit is
// read for computation and written by exactly one lane.  When X is a multiple
// of 64 the odd phase has one extra half block per row-pair (cells x = X-1,
// x = X outside), which the last lane runs with the scalar rule.
#include <stdint.h>

#include <algorithm>

#include "fs3d_common.h"
#include "pcg.h"
#include "planes.h"
#include "conv_device.cuh"
#include "rule_device.cuh"
#include "bulk_device.cuh"
#include "bricks_device.cuh"

namespace fs3d {

// ---------------------------------------------------------------------------
// hashes
// ---------------------------------------------------------------------------
// Sum of the hash terms of the chunk of row r at x = 64 w (plane word q).
// Bound: the 64-bit finalizer's instructions (about 25 a cell), so the cells'
// bytes come four at a time from the packed conversion.
__device__ __forceinline__ uint64_t hash_chunk(const uint4& q, const uint8_t* statics, int X, int64_t r, int w) {
    const int64_t idx = r * X + 64 * w;
    const int n = min(64, X - 64 * w);
    uint32_t p[4];
    planes_to_pieces(q, p);
    uint64_t h = 0;
    for (int g = 0; g < 4; ++g) {
        if (16 * g >= n) break;
        const uint32_t pg = g == 0 ? p[0] : (g == 1 ? p[1] : (g == 2 ? p[2] : p[3]));
#pragma unroll
        for (int x = 0; x < 16; ++x) {
            const int64_t i = idx + 16 * g + x;
            uint32_t v = (pg >> (8 * (x & 3) + 2 * (x >> 2))) & 3u;
            if (16 * g + x < n) {
                if (statics && v == 1u) v = statics[i];
                h += fmix64((uint64_t)i * 256u + v);
            }
        }
    }
    return h;
}

__global__ void k_hash_planes(const uint4* __restrict__ rows, const uint8_t* __restrict__ statics, int X, int Y,
                              int Z, int nw, unsigned long long* out) {
    const int64_t n = (int64_t)Y * Z * nw;
    uint64_t h = 0;
    for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n; u += (int64_t)gridDim.x * blockDim.x)
        h += hash_chunk(rows[u], statics, X, u / nw, (int)(u % nw));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) h += __shfl_xor_sync(0xffffffffu, h, off);
    if ((threadIdx.x & 31) == 0 && h) atomicAdd(out, (unsigned long long)h);
}

// Whole-grid hashes of many worlds in one launch: CTA (j, s) sums every
// gridDim.y-th part of world j (jobs[j]) into out[j * gridDim.y + s].  (One CTA
// a world left a poll waiting for its largest, up to 128^3 cells in 256 threads:
// 393 worlds 857 us, in 32 parts each 130; the polls of 1000 served worlds 8.2
// ms together, now 0.7.)
__global__ void __launch_bounds__(256) k_hash_planes_many(const HashJob* __restrict__ jobs,
                                                         unsigned long long* __restrict__ out) {
    const HashJob jb = jobs[blockIdx.x];
    const int64_t n = (int64_t)jb.Y * jb.Z * jb.nw;
    uint64_t h = 0;
    for (int64_t u = blockIdx.y * blockDim.x + threadIdx.x; u < n; u += (int64_t)gridDim.y * blockDim.x)
        h += hash_chunk(jb.rows[u], jb.statics, jb.X, u / jb.nw, (int)(u % jb.nw));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) h += __shfl_xor_sync(0xffffffffu, h, off);
    __shared__ unsigned long long part[8];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = h;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += part[i];
        out[(size_t)blockIdx.x * gridDim.y + blockIdx.y] = t;
    }
}

// the job j with off[j] <= u < off[j + 1]
__device__ __forceinline__ int find_job(const int64_t* __restrict__ unit_off, int njobs, int64_t u) {
    int lo = 0, hi = njobs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(unit_off + mid) <= u)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// The mixed-size batch world generated straight into planes: stone at y < 2,
// empty below Y/2, and above it one PCG32 draw per cell in index order; each
// thread jumps its generator to the first draw of its 64-cell word.
__device__ __forceinline__ uint4 gen_word(const GenJob& g, int64_t r, int w) {
    const int yf = g.Y / 2, y = (int)(r / g.Z), z = (int)(r % g.Z);
    uint32_t ae = 0, ao = 0, be = 0, bo = 0;
    uint64_t st = 0;
    if (y >= yf) st = pcg_jump(g.p.fill_state, ((uint64_t)(y - yf) * g.Z + z) * g.X + 64u * w, g.p.inc);
    for (int m = 0; m < 64; ++m) {
        const int x = 64 * w + m;
        uint32_t v;
        if (x >= g.X || y < 2) {
            v = 1u;
        } else if (y < yf) {
            v = 0u;
        } else {
            const uint32_t d = pcg_output(st);
            st = st * kPcgMult + g.p.inc;
            v = d < g.p.sand_thr ? 2u : (d < g.p.water_thr ? 3u : 0u);
        }
        const uint32_t a = v >> 1, b = v & 1u;  // codes 0..3 are their own (A, B)
        if (m & 1) {
            ao |= a << (m >> 1);
            bo |= b << (m >> 1);
        } else {
            ae |= a << (m >> 1);
            be |= b << (m >> 1);
        }
    }
    return make_uint4(ae, ao, be, bo);
}

// many worlds per launch (blocks as the conversions'), or `one`
__global__ void __launch_bounds__(kConvThreads) k_gen_batch_planes(const GenJob* __restrict__ jobs,
                                                                   const ConvBlock* __restrict__ blocks, GenJob one) {
    int64_t row0 = (int64_t)blockIdx.x * conv_rows(one.nw > 0 ? one.nw : 1, kConvChunks);
    GenJob g = one;
    if (blocks) {
        const ConvBlock b = blocks[blockIdx.x];
        g = jobs[b.job];
        row0 = b.row0;
    }
    const int r = threadIdx.x / g.nw, w = threadIdx.x - r * g.nw;
    if (r >= conv_rows(g.nw, kConvChunks) || row0 + r >= (int64_t)g.Y * g.Z) return;
    g.rows[row0 * g.nw + threadIdx.x] = gen_word(g, row0 + r, w);
}

// ---------------------------------------------------------------------------
// step
// ---------------------------------------------------------------------------
// One block row-pair of one world; lane gl of a group of G lanes.  Every lane
// of the warp calls this (valid = false for groups past the last row-pair).
__device__ __forceinline__ void plane_rowpair(const PlaneWorld& w, int o, uint32_t sk, int rp, bool valid, int gl,
                                              int G) {
    const int NBZ = nblocks(w.Z, o);
    const int j = valid ? rp / NBZ : 0, k = valid ? rp - j * NBZ : 0;
    const uint32_t rk = rowkey(sk, (uint32_t)j, (uint32_t)k);
    const int y0 = 2 * j - o, z0 = 2 * k - o;
    const bool has = valid && gl < w.nw;
    uint4 q[4], q0[4];
    uint4* ptr[4];
    bool in[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int y = (a < 2) ? y0 + 1 : y0, z = z0 + (a & 1);
        in[a] = has && y >= 0 && y < w.Y && z >= 0 && z < w.Z;
        ptr[a] = in[a] ? w.rows + ((int64_t)y * w.Z + z) * w.nw + gl : w.rows;
        q[a] = in[a] ? *ptr[a] : make_uint4(0u, 0u, 0xFFFFFFFFu, 0xFFFFFFFFu);
        q0[a] = q[a];
    }
    rowpair_core(q, has, o, rk, gl, G, w.nw, (w.X & 63) == 0);
#pragma unroll
    for (int a = 0; a < 4; ++a)
        if (in[a] && (q[a].x != q0[a].x || q[a].y != q0[a].y || q[a].z != q0[a].z || q[a].w != q0[a].w)) *ptr[a] = q[a];
}

// One launch = one step (segment step s_seg) of every live world.  Work items
// are warp-sized: item = (world, first row-pair); a warp covers 32 >> lg
// row-pairs of that world.  Warps loop over items; the item count lives in
// device memory so a captured graph keeps working as worlds come and go.
__global__ void __launch_bounds__(256) k_plane_step(const PlaneWorld* __restrict__ worlds,
                                                   const PlaneItem* __restrict__ items,
                                                   const int* __restrict__ n_items_p, int s_seg) {
    const int n_items = *n_items_p;
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int it = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < n_items; it += warps) {
        const PlaneItem item = items[it];
        const PlaneWorld& w = worlds[item.world];
        if (s_seg >= w.steps) continue;
        const uint64_t t = w.t + (uint64_t)s_seg;
        const int o = (int)(t & 1u);
        const int G = 1 << w.lg;
        const int gl = lane & (G - 1);
        const int rp = item.rp0 + (lane >> w.lg);
        const int nrp = nblocks(w.Y, o) * nblocks(w.Z, o);
        plane_rowpair(w, o, stepkey(w.seed, t), rp, rp < nrp, gl, G);
    }
}

// One step of one large world (too large for the resident kernels), skipping
// settled row-pairs exactly.  Per row (y, z) one byte holds the low 8 bits of
// the last step that changed the row.  A block row-pair of phase o at step t
// is evaluated when one of its four rows changed at step t-1 or t-2 (age
// (t - flag) & 255 of 1 or 2; an older change that aliases to those ages only
// adds work).  Otherwise its cells are those it had when last evaluated (at
// t-2, same phase), which changed nothing, and whether a block can change
// depends on its own cells alone, so it would change nothing again.  Each
// row belongs to one row-pair per step, so the row-pair reads and writes its
// rows' bytes with no other reader in the step.  A fresh world starts with
// every byte at t0 - 1 (every row changed just before).  Warps take
// (32 >> lg) row-pairs each in order; a warp whose row-pairs are all settled
// loads nothing.
__device__ __forceinline__ bool rows_changed_recently(const uint8_t* rf, int Y, int Z, int y0, int z0,
                                                      uint32_t tb) {
    bool d = false;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int y = y0 + (a >> 1), z = z0 + (a & 1);
        if (y >= 0 && y < Y && z >= 0 && z < Z) d |= ((tb - (uint32_t)rf[(int64_t)y * Z + z]) & 0xFFu) - 1u < 2u;
    }
    return d;
}

// LIST: more than two items a warp.  It then looks at the flags of its next G
// items together, a row-pair a lane (one after another, the flags' loads took
// most of a settled step), and takes the dirty ones of them (32 >> lg) at a
// time.  1024^3 dunes, steps 60 / 420 / 960: 196 / 97 / 58 us item by item, 184
// / 83 / 42 listed; 512^3 26.5 / 11 / 10.8 and 25.7 / 10 / 9.  With two items a
// warp the list costs what it saves (400x300x350: 11.8 / 7.5 / 7.4 and 12.1 /
// 7.5 / 7.3), with one 0.3 us (200^3: 6.2 and 6.6).
// Three CTAs per SM (80 registers, a few bytes spilled): 24 warps hide the
// rule's dependent chain better than 16 at 118 registers (1024^3 dunes:
// 118 us per step against 133 us, 123 us at four CTAs)
//
// err: the world's error record (nullable); while it is set nothing is stepped.
// Its load runs beside the flags' and is looked at with them.
template <bool LIST>
__global__ void __launch_bounds__(256, 3) k_plane_step_skip(const PlaneWorld w, uint8_t* __restrict__ rflags,
                                                        int* counts, const int* err) {
    chain_wait();
    const int failed = err ? *(volatile const int*)err : 0;
    const uint64_t t = w.t;
    const int o = (int)(t & 1u);
    const int lane = threadIdx.x & 31;
    const int G = 1 << w.lg, per = 32 >> w.lg, gl = lane & (G - 1);
    const int NBZ = nblocks(w.Z, o), nrp = nblocks(w.Y, o) * NBZ, n_items = (nrp + per - 1) / per;
    const uint32_t sk = stepkey(w.seed, t), tb = (uint32_t)t & 0xFFu;
    const uint32_t gmask = G == 32 ? 0xFFFFFFFFu : ((1u << G) - 1u) << (lane & ~(G - 1));
    const bool half_at_end = (w.X & 63) == 0;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    __shared__ int2 s_list[8][LIST ? 32 : 1];
    int2* list = s_list[threadIdx.x >> 5];
    for (int it0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; it0 < n_items; it0 += LIST ? warps * G : warps) {
        int n_dirty = 0, j = 0, k = 0;
        bool dirty = false;
        if (LIST) {
            const int it = it0 + (lane >> (5 - w.lg)) * warps, rp = it * per + (lane & (per - 1));
            if (it < n_items && rp < nrp) {
                j = rp / NBZ;
                k = rp - j * NBZ;
                dirty = rows_changed_recently(rflags, w.Y, w.Z, 2 * j - o, 2 * k - o, tb);
            }
            dirty = dirty && !failed;
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, dirty);
            n_dirty = __popc(m);
            if (dirty) list[__popc(m & ((1u << lane) - 1u))] = make_int2(j, k);
            __syncwarp();
        } else {
            const int rp = it0 * per + (lane >> w.lg);
            if (rp < nrp) {
                j = rp / NBZ;
                k = rp - j * NBZ;
                if (gl == 0) dirty = rows_changed_recently(rflags, w.Y, w.Z, 2 * j - o, 2 * k - o, tb);
            }
            dirty = __shfl_sync(0xFFFFFFFFu, dirty && !failed, lane & ~(G - 1));
            if (__any_sync(0xFFFFFFFFu, dirty)) n_dirty = 1;
        }
        for (int at = 0; at < n_dirty; at += per) {
            if (LIST) {
                const int me = at + (lane >> w.lg);
                dirty = me < n_dirty;
                const int2 jk = dirty ? list[me] : make_int2(0, 0);
                j = jk.x;
                k = jk.y;
            }
            const int y0 = 2 * j - o, z0 = 2 * k - o;
            const bool has = dirty && gl < w.nw;
            uint4 q[4], q0[4];
            uint4* ptr[4];
            bool in[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const int y = (a < 2) ? y0 + 1 : y0, z = z0 + (a & 1);
                in[a] = has && y >= 0 && y < w.Y && z >= 0 && z < w.Z;
                ptr[a] = in[a] ? w.rows + ((int64_t)y * w.Z + z) * w.nw + gl : w.rows;
                q[a] = in[a] ? *ptr[a] : make_uint4(0u, 0u, 0xFFFFFFFFu, 0xFFFFFFFFu);
                q0[a] = q[a];
            }
            rowpair_core(q, has, o, rowkey(sk, (uint32_t)j, (uint32_t)k), gl, G, w.nw, half_at_end);
            bool any = false;
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const bool chg =
                    in[a] && (q[a].x != q0[a].x || q[a].y != q0[a].y || q[a].z != q0[a].z || q[a].w != q0[a].w);
                if (chg) {
                    *ptr[a] = q[a];
                    any = true;
                }
                const uint32_t bal = __ballot_sync(0xFFFFFFFFu, chg);
                if (gl == 0 && (bal & gmask)) {
                    const int y = (a < 2) ? y0 + 1 : y0, z = z0 + (a & 1);
                    rflags[(int64_t)y * w.Z + z] = (uint8_t)tb;
                }
            }
            if (counts && any) count_bricks(counts, w, y0, z0, gl, q, q0, in);
        }
        if (LIST) __syncwarp();  // the list's readers are done
    }
    chain_go();
}

// ---------------------------------------------------------------------------
// change flags of a world with no history, from its cells
// ---------------------------------------------------------------------------
// A world admitted (or loaded, or written) at step t0 has no record of its
// last changes.  Marking every layer or row changed at t0 - 1 makes its first
// two steps evaluate every row-pair.  Instead a layer or row is marked changed
// at t0 - 1 only when a block row-pair of either phase that covers it can
// change (rowpair_can_change), and at t0 - 3 (two steps before the window the
// skip reads) otherwise.  Exact: at t0 and t0 + 1 a skipped pair has no block
// that can change and no row of it changed since t0 (at t0 + 1 a change at t0
// marks it); from t0 + 2 on the skip's usual argument holds, since a pair not
// evaluated at t0 could not change then.

// the four rows of block row-pair (j, k) of phase o for lane gl, solid outside the world
__device__ __forceinline__ void load_rowpair(const uint4* __restrict__ rows, int Y, int Z, int nw, int y0, int z0,
                                             int gl, bool has, uint4 (&q)[4]) {
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int y = (a < 2) ? y0 + 1 : y0, z = z0 + (a & 1);
        const bool in = has && y >= 0 && y < Y && z >= 0 && z < Z;
        q[a] = in ? rows[((int64_t)y * Z + z) * nw + gl] : make_uint4(0u, 0u, 0xFFFFFFFFu, 0xFFFFFFFFu);
    }
}

__device__ __forceinline__ int lanes_lg(int nw) { return nw <= 1 ? 0 : 32 - __clz(nw - 1); }

// One warp per layer y of each job (blockIdx.x: job, blockIdx.y * 8 + warp: y).
// `one` stands for the job table when jobs is null.
__global__ void __launch_bounds__(256) k_layer_flags_from_cells(const ConvJob* __restrict__ jobs, ConvJob one) {
    const ConvJob jb = jobs ? jobs[blockIdx.x] : one;
    const int y = (int)blockIdx.y * 8 + (int)(threadIdx.x >> 5);
    if (!jb.lflags || y >= jb.Y) return;  // warp-uniform
    const int lane = threadIdx.x & 31, lg = lanes_lg(jb.nw);
    const int G = 1 << lg, per = 32 >> lg, gl = lane & (G - 1), gi = lane >> lg;
    const bool half_at_end = (jb.X & 63) == 0;
    bool any = false;
    for (int o = 0; o < 2 && !any; ++o) {
        const int y0 = 2 * ((y + o) >> 1) - o;  // the pair of phase o covering y: layers y0, y0 + 1
        const int nbz = nblocks(jb.Z, o);
        for (int k0 = 0; k0 < nbz && !any; k0 += per) {
            const int k = k0 + gi;
            const bool has = k < nbz && gl < jb.nw;
            uint4 q[4];
            load_rowpair(jb.rows, jb.Y, jb.Z, jb.nw, y0, 2 * k - o, gl, has, q);
            any = __any_sync(0xFFFFFFFFu, rowpair_can_change(q, has, o, gl, G, jb.nw, half_at_end));
        }
    }
    if (lane == 0) jb.lflags[y] = (uint8_t)(jb.t0b - (any ? 1u : 3u));
}

// Row flags, already set to t0 - 3: every block row-pair of both phases that
// can change marks its rows changed at t0 - 1 (rows shared by two such pairs
// get the same value from both).
__global__ void __launch_bounds__(256) k_row_flags_from_cells(const uint4* __restrict__ rows,
                                                              uint8_t* __restrict__ rflags, int X, int Y, int Z,
                                                              int nw, uint32_t t0b, const int* err, int* own) {
    // (loaded here, stored at the end: the warp does not wait for it)
    const bool tells = own && blockIdx.x == 0 && threadIdx.x == 0;
    const int was = tells ? *(volatile const int*)err : 0;
    const int lane = threadIdx.x & 31, lg = lanes_lg(nw);
    const int G = 1 << lg, per = 32 >> lg, gl = lane & (G - 1), gi = lane >> lg;
    const uint32_t gmask = G == 32 ? 0xFFFFFFFFu : ((1u << G) - 1u) << (lane & ~(G - 1));
    const bool half_at_end = (X & 63) == 0;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t first = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    for (int o = 0; o < 2; ++o) {
        const int nbz = nblocks(Z, o), chunks = (nbz + per - 1) / per;
        const int64_t items = (int64_t)nblocks(Y, o) * chunks;
        for (int64_t it = first; it < items; it += warps) {
            const int j = (int)(it / chunks), k = (int)(it - (int64_t)j * chunks) * per + gi;
            const int y0 = 2 * j - o, z0 = 2 * k - o;
            const bool has = k < nbz && gl < nw;
            uint4 q[4];
            load_rowpair(rows, Y, Z, nw, y0, z0, gl, has, q);
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, rowpair_can_change(q, has, o, gl, G, nw, half_at_end));
            if (gl == 0 && k < nbz && (m & gmask)) {
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    const int y = (a < 2) ? y0 + 1 : y0, z = z0 + (a & 1);
                    if (y >= 0 && y < Y && z >= 0 && z < Z) rflags[(int64_t)y * Z + z] = (uint8_t)(t0b - 1u);
                }
            }
        }
    }
    if (tells) *own = was;
}

// ---------------------------------------------------------------------------
// shared-memory resident segment: one CTA steps one whole world
// ---------------------------------------------------------------------------
// Test hook (fs3d_test_inject): extra bytes a single-CTA kernel announces on
// its mbarrier beyond what its bulk copy delivers.  With it set, the copy
// lands in full but the barrier's phase never completes, so each wait runs to
// its iteration limit and reports a timeout; nothing else changes.  0 in
// normal operation.
static __device__ uint32_t g_inject_tx_extra;

// One world held by a CTA: its rows, followed in shared memory (at the next
// 16-byte boundary) by four change buffers of one byte per layer y (buffer t &
// 3: 1 if step t changed a row of the layer) and a list of up to Y/2 + 2 16-bit
// layer-pair indices.  Step t writes buffer t & 3, reads buffers (t-1) & 3 and
// (t-2) & 3 and clears buffer (t+1) & 3, so no buffer is both read and written
// in a step.
struct WorldView {
    uint4* rows;
    uint8_t* flags;
    uint32_t stride;  // of the change buffers
    int Z, nw;
    __device__ __forceinline__ uint4* at(int y, int z, int g) const { return rows + (y * Z + z) * nw + g; }
    __device__ __forceinline__ uint8_t* flag(int y, uint32_t b) const { return flags + b * stride + y; }
    __host__ __device__ static __forceinline__ uint32_t flag_stride(int layers) { return ((uint32_t)layers + 15u) & ~15u; }
};

// shared-memory bytes after a world's planes: change buffers and the layer list
__host__ __device__ __forceinline__ uint32_t slab_aux_bytes(uint32_t layers) {
    return 4u * ((layers + 15u) & ~15u) + ((2u * (layers / 2u + 2u) + 15u) & ~15u);
}

// index of the n-th (from 0) set bit of m; m has more than n set bits
__device__ __forceinline__ int select_bit(uint32_t m, int n) {
    int pos = 0, c = __popc(m & 0xFFFFu);
    if (n >= c) { n -= c; m >>= 16; pos += 16; }
    c = __popc(m & 0xFFu);
    if (n >= c) { n -= c; m >>= 8; pos += 8; }
    c = __popc(m & 0xFu);
    if (n >= c) { n -= c; m >>= 4; pos += 4; }
    c = __popc(m & 0x3u);
    if (n >= c) { n -= c; m >>= 2; pos += 2; }
    return pos + (n >= (int)(m & 1u) ? 1 : 0);
}

// bytes of a world's planes, rounded up so its change buffers start 16-byte aligned
__host__ __device__ __forceinline__ uint32_t slab_flag_offset(uint32_t plane_bytes) {
    return (plane_bytes + 15u) & ~15u;
}

// Whether the block row-pairs of layer pair j (all k) must be evaluated: a
// row of layer 2j - o or 2j - o + 1 changed in one of the two previous steps.
// Otherwise every pair's cells are those of its last evaluation in the same
// phase, two steps back, which changed nothing, and whether a block can
// change depends on its cells alone (the rule's activity mask), so it would
// change nothing again.  A world without kept flags starts with every layer
// changed at steps t0 - 1 and t0 - 2.
__device__ __forceinline__ bool layer_dirty(const WorldView& v, const PlaneWorld& w, int o, uint32_t tb, int j) {
    uint32_t dirty = 0;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        const int y = 2 * j - o + a;
        if (y >= 0 && y < w.Y) dirty |= (uint32_t)*v.flag(y, (tb + 3u) & 3u) | (uint32_t)*v.flag(y, (tb + 2u) & 3u);
    }
    return dirty != 0;
}

// Evaluates block row-pair (j, k) of a world held in shared memory when `run`
// is set.  Every lane of the warp calls this together (the odd phase passes
// carry bits between lanes).  Layers with a changed row get the step's flag.
__device__ __forceinline__ void world_rowpair(const WorldView& v, const PlaneWorld& w, int o, uint32_t sk,
                                             uint32_t tt /* step & 3 */, int j, int k, bool run, int gl,
                                             int G) {
    if (!__any_sync(0xFFFFFFFFu, run)) return;
    const int y0 = 2 * j - o, z0 = 2 * k - o;
    const uint32_t rk = rowkey(sk, (uint32_t)j, (uint32_t)k);
    const bool has = run && gl < w.nw;
    uint4 q[4], q0[4];
    uint4* ptr[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int y = (a < 2) ? y0 + 1 : y0, z = z0 + (a & 1);
        ptr[a] = (has && y >= 0 && y < w.Y && z >= 0 && z < w.Z) ? v.at(y, z, gl) : nullptr;
        q[a] = ptr[a] ? *ptr[a] : make_uint4(0u, 0u, 0xFFFFFFFFu, 0xFFFFFFFFu);
        q0[a] = q[a];
    }
    rowpair_core(q, has, o, rk, gl, G, w.nw, (w.X & 63) == 0);
#pragma unroll
    for (int a = 0; a < 4; ++a)
        if (ptr[a] && (q[a].x != q0[a].x || q[a].y != q0[a].y || q[a].z != q0[a].z || q[a].w != q0[a].w)) {
            *ptr[a] = q[a];
            *v.flag((a < 2) ? y0 + 1 : y0, tt) = 1u;
        }
}

// Persistent resident segment kernel.  A CTA takes worlds of its class, largest
// first, from `counter`, loads a world's planes into shared memory with one
// TMA bulk copy, runs its segment steps (one barrier per step: the next phase
// pairs different rows) and writes it back with one TMA bulk store.  Worlds
// are independent, so CTAs never wait on one another.
// meta: [0] per-step items, [1 + c] resident worlds of class c, [1 + kAllClasses + c] their offset in order[].
// CTAs of each single-CTA class that share an SM (the register cap that lets
// them: 24 warps of at most 80 registers per SM)
template <int NT>
constexpr int resident_ctas_per_sm() {
    return NT == 128 ? 6 : (NT == 256 ? 3 : 1);
}

// GM: the world stays in global memory (L2) and the CTA keeps only the layer
// flags and list in shared memory, so as many worlds are in flight as warps
// allow; no bulk copies.  CTAs per SM of a GM kernel: kGmThreadsPerSm threads.
#ifndef FS3D_GM_THREADS_PER_SM
#define FS3D_GM_THREADS_PER_SM 768
#endif
constexpr int kGmThreadsPerSm = FS3D_GM_THREADS_PER_SM;
template <int NT, bool GM = false>
__global__ void __launch_bounds__(NT, GM ? kGmThreadsPerSm / NT : resident_ctas_per_sm<NT>())
    k_plane_segment_resident(const PlaneWorld* __restrict__ worlds,
                                                             const int* __restrict__ order,
                                                             const int* __restrict__ meta, int cls,
                                                             int* counter, int* err,
                                                             unsigned long long* processed_cells) {
    extern __shared__ __align__(128) uint4 srows[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ int item;
    const int n = meta[1 + cls], off = meta[1 + kAllClasses + cls];
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    const uint32_t tx_extra = g_inject_tx_extra;
    uint32_t phase = 0;
    const int lane = threadIdx.x & 31;
    __shared__ unsigned long long s_processed;  // cell-steps evaluated (the rest were skipped as settled)
    __shared__ int s_count[2];                   // work-list length, by step parity
    constexpr int kKeys = 32;                    // step keys computed together, one per thread
    __shared__ uint32_t s_keys[kKeys];
    // many dirty layer pairs: each warp lists them once a step, so that a pass
    // looks its own up (the families of dense steps; settled worlds have one or
    // two, found from the masks, and the list's round trip made their 2048-world
    // segment and snapshot 946 us instead of 794)
    constexpr bool kListed = !GM || NT >= 768;
    constexpr int kMasked = 96;
    __shared__ uint8_t s_list[NT / 32][kListed ? kMasked : 1];
    // per phase o: the world's block rows along z, and the multiplier that
    // divides by it (e / n = umulhi(e, m), exact for e, n < 2^16)
    __shared__ uint32_t s_nbz[2], s_magic[2];
    if (threadIdx.x == 0) {
        s_processed = 0;
        s_count[0] = s_count[1] = 0;
    }
    for (;;) {
        // after an error no CTA takes another world
        if (threadIdx.x == 0) item = *(volatile int*)err ? n : atomicAdd(counter, 1);
        __syncthreads();
        const int it = item;
        __syncthreads();
        if (it >= n) break;
        const PlaneWorld w = worlds[order[off + it]];
        if (w.steps <= 0) continue;
        const uint32_t bytes = GM ? 0u : (uint32_t)w.Y * (uint32_t)w.Z * (uint32_t)w.nw * 16u;  // bulk-copied bytes
        WorldView v;
        v.rows = GM ? w.rows : srows;
        v.Z = w.Z;
        v.nw = w.nw;
        v.flags = reinterpret_cast<uint8_t*>(srows) + slab_flag_offset(bytes);
        v.stride = WorldView::flag_stride(w.Y);
        if (threadIdx.x == 0 && bytes) bulk_load(srows, w.rows, bytes, bytes + tx_extra, &bar);
        if (threadIdx.x < 2) {
            s_nbz[threadIdx.x] = (uint32_t)nblocks(w.Z, (int)threadIdx.x);
            s_magic[threadIdx.x] = 0xFFFFFFFFu / (uint32_t)nblocks(w.Z, (int)threadIdx.x) + 1u;
        }
        // change buffers from the kept flags (the low 8 bits of the last step
        // that changed the layer), or every layer changed at t0 - 1 and t0 - 2
        {
            const bool kept = w.lflags != nullptr && !w.lflags_fresh;
            const uint32_t t0b = (uint32_t)w.t & 3u, fs = v.stride;
            for (int i = threadIdx.x; i < w.Y; i += NT) {
                const uint32_t age = kept ? (((uint32_t)w.t - (uint32_t)w.lflags[i]) & 0xFFu) : 0u;
                v.flags[((t0b + 3u) & 3u) * fs + i] = kept ? (age == 1u) : 1u;
                v.flags[((t0b + 2u) & 3u) * fs + i] = kept ? (age == 2u) : 1u;
                v.flags[t0b * fs + i] = 0u;
                v.flags[((t0b + 1u) & 3u) * fs + i] = 0u;
            }
        }
        bool ok = true;
        if (bytes) {
            ok = mbar_wait(&bar, phase, tx_extra ? kCopyWaitInjectedNs : kCopyWaitNs);
            phase ^= 1u;
        }
        // A copy that never landed poisons the world: the error record is
        // set (err[0] = 1, err[2..3] = the world's step at the start of this
        // launch, by the first group to fail), this CTA still takes part in
        // every barrier of its group but touches no memory, and the group
        // stops before its next world.
        const bool poisoned = __syncthreads_or(!ok) != 0;
        if (poisoned && threadIdx.x == 0 && atomicCAS(err, 0, 1) == 0)
            *reinterpret_cast<unsigned long long*>(err + 2) = (unsigned long long)w.t;
        const int G = 1 << w.lg, per = NT >> w.lg;
        const int gl = lane & (G - 1);
        // layer pairs to evaluate in a step, after the buffers
        const uint32_t fs = v.stride;
        uint16_t* jlist = reinterpret_cast<uint16_t*>(v.flags + 4u * fs);
        for (int s = 0; s < w.steps; ++s) {
            if ((s & (kKeys - 1)) == 0) {
                // the next kKeys steps' keys, one thread each (the previous step's
                // barrier is behind every reader of the last ones)
                for (int i = threadIdx.x; i < kKeys; i += NT)
                    if (s + i < w.steps) s_keys[i] = stepkey(w.seed, w.t + (uint64_t)(s + i));
                __syncthreads();
            }
            if (poisoned) {
                __syncthreads();
                continue;
            }
            const uint64_t t = w.t + (uint64_t)s;
            const int o = (int)(t & 1u);
            const uint32_t sk = s_keys[s & (kKeys - 1)];
            const int NBZ = (int)s_nbz[o];
            const int nj = nblocks(w.Y, o);
            const uint32_t tb = (uint32_t)t & 3u;
            // the buffer the next step writes: read and written by no one in this step
            for (int i = threadIdx.x; i < w.Y; i += NT) v.flags[((tb + 1u) & 3u) * fs + i] = 0u;
            // dirty layer pairs: up to 96 as bit masks every warp computes for
            // itself (the buffers it reads are not written in this step), more
            // through the shared list
            uint32_t dm0 = 0, dm1 = 0, dm2 = 0;
            int n_layers;
            const bool masked = nj <= kMasked;
            uint8_t* list = s_list[threadIdx.x >> 5];
            if (masked) {
                dm0 = __ballot_sync(0xFFFFFFFFu, lane < nj && layer_dirty(v, w, o, tb, lane));
                if (nj > 32) dm1 = __ballot_sync(0xFFFFFFFFu, lane + 32 < nj && layer_dirty(v, w, o, tb, 32 + lane));
                if (nj > 64) dm2 = __ballot_sync(0xFFFFFFFFu, lane + 64 < nj && layer_dirty(v, w, o, tb, 64 + lane));
                n_layers = __popc(dm0) + __popc(dm1) + __popc(dm2);
                if (kListed) {
                    __syncwarp();  // the last step's readers are done
                    const uint32_t dm[3] = {dm0, dm1, dm2};
                    int at = 0;
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        if ((dm[i] >> lane) & 1u) list[at + __popc(dm[i] & ((1u << lane) - 1u))] = (uint8_t)(32 * i + lane);
                        at += __popc(dm[i]);
                    }
                    __syncwarp();
                }
            } else {
                int* cnt = &s_count[s & 1];
                for (int base = 0; base < nj; base += NT) {
                    const int i = base + (int)threadIdx.x;
                    const bool add = i < nj && layer_dirty(v, w, o, tb, i);
                    const uint32_t m = __ballot_sync(0xFFFFFFFFu, add);
                    if (m) {
                        int pos = 0;
                        if (lane == __ffs(m) - 1) pos = atomicAdd(cnt, __popc(m));
                        pos = __shfl_sync(0xFFFFFFFFu, pos, __ffs(m) - 1) + __popc(m & ((1u << lane) - 1u));
                        if (add) jlist[pos] = (uint16_t)i;
                    }
                }
                __syncthreads();
                n_layers = *cnt;
            }
            if (threadIdx.x == 0) {
                s_count[(s + 1) & 1] = 0;  // the next step's counter (read before this step)
                // cells evaluated: the rows of every dirty layer pair inside the world, X*Z cells each
                int rows = 2 * n_layers;
                if (n_layers) {
                    if (o && layer_dirty(v, w, o, tb, 0)) --rows;
                    if (2 * (nj - 1) - o + 1 >= w.Y && layer_dirty(v, w, o, tb, nj - 1)) --rows;
                }
                s_processed += (unsigned long long)rows * (unsigned long long)(w.X * w.Z);
            }
            const int npairs = n_layers * NBZ;
            const uint32_t nbz_magic = s_magic[o];
            for (int base = 0; base < npairs; base += per) {
                const int e = base + (int)(threadIdx.x >> w.lg);
                const bool valid = e < npairs;
                const int jd =
                    valid ? (NBZ == 1 ? e : (npairs <= 65536 ? (int)__umulhi((uint32_t)e, nbz_magic) : e / NBZ)) : 0;
                const int kk = valid ? e - jd * NBZ : 0;
                int jj = 0;
                if (valid) {
                    if (!masked)
                        jj = (int)jlist[jd];
                    else if (kListed)
                        jj = (int)list[jd];
                    else if (jd == 0 && dm0)
                        jj = __ffs(dm0) - 1;
                    else if (jd < __popc(dm0))
                        jj = select_bit(dm0, jd);
                    else if (jd < __popc(dm0) + __popc(dm1))
                        jj = 32 + select_bit(dm1, jd - __popc(dm0));
                    else
                        jj = 64 + select_bit(dm2, jd - __popc(dm0) - __popc(dm1));
                }
                world_rowpair(v, w, o, sk, tb, jj, kk, valid, gl, G);
            }
            __syncthreads();
        }
        if (w.lflags && !poisoned) {
            // kept for the next segment: the last of the final two steps that changed the layer
            const uint64_t te = w.t + (uint64_t)w.steps;
            const uint32_t b1 = (uint32_t)(te - 1u) & 3u, b2 = (uint32_t)(te - 2u) & 3u;
            for (int i = threadIdx.x; i < w.Y; i += NT)
                w.lflags[i] = (uint8_t)(v.flags[b1 * fs + i] ? te - 1u : (v.flags[b2 * fs + i] ? te - 2u : te - 3u));
        }
        // make the threads' shared-memory writes visible to the bulk copy
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0 && bytes && !poisoned) bulk_store_wait(w.rows, srows, bytes);
        __syncthreads();  // the buffer is free again
    }
    __syncthreads();
    if (threadIdx.x == 0 && processed_cells && s_processed) atomicAdd(processed_cells, s_processed);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
namespace {

struct ResidentCfg {
    int threads, ctas_per_sm;
    int smem;  // dynamic shared memory per CTA (bytes), 0 = class unavailable
    const void* fn;
};

struct ResidentCfgs {
    ResidentCfg c[kSingleCtaClasses] = {};
};

template <int NT>
const void* resident_fn() {
    return reinterpret_cast<const void*>(&k_plane_segment_resident<NT>);
}

ResidentCfgs fill_classes() {
    ResidentCfgs out;
    int dev = 0, per_sm = 0, optin = 0, reserved = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
    const int kStatic = 256;  // the kernel's own shared variables, rounded up
    const ResidentCfg base[kSingleCtaClasses] = {{128, resident_ctas_per_sm<128>(), 0, resident_fn<128>()},
                                                 {256, resident_ctas_per_sm<256>(), 0, resident_fn<256>()},
                                                 {768, resident_ctas_per_sm<768>(), 0, resident_fn<768>()}};
    for (int c = 0; c < kSingleCtaClasses; ++c) {
        ResidentCfg k = base[c];
        int stat = kStatic;
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, k.fn) == cudaSuccess && (int)fa.sharedSizeBytes > stat)
            stat = ((int)fa.sharedSizeBytes + 127) & ~127;
        int smem = per_sm / k.ctas_per_sm - reserved - stat;
        if (smem > optin - stat) smem = optin - stat;
        smem = smem / 16 * 16;
        if (smem <= 0 || cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            smem = 0;
        int fit = 0;
        if (smem && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k.fn, k.threads, smem) != cudaSuccess ||
                     fit < k.ctas_per_sm))
            smem = 0;
        k.smem = smem;
        out.c[c] = k;
    }
    cudaGetLastError();  // a refused attribute leaves the class unused, not an error
    return out;
}

// those of the current device and context (the attribute belongs to them)
ResidentCfgs resident_cfgs() {
    static PerContext<ResidentCfgs> kept;
    return of_current_context(kept, fill_classes);
}

}  // namespace

ResidentLimits resident_limits() {
    const ResidentCfgs k = resident_cfgs();
    ResidentLimits l;
    for (int c = 0; c < kSingleCtaClasses; ++c) l.one_cta[c] = k.c[c].smem;
    batch_slabs_limits(&l);
    return l;
}

int resident_class(const ResidentLimits& l, int X, int Y, int Z) {
    const int64_t planes = (int64_t)Y * Z * plane_nw(X) * 16;
    for (int c = 0; c < kSingleCtaClasses; ++c) {
        // planes, then the layer flags and the layer list
        const int64_t need = ((planes + 15) & ~(int64_t)15) + (int64_t)slab_aux_bytes((uint32_t)Y);
        if (l.one_cta[c] && need <= l.one_cta[c]) return c;
    }
    for (int c = kSingleCtaClasses; c < kResidentClasses; ++c)
        if (batch_slabs_fit(l, X, Y, Z, kClusterSizes[c - kSingleCtaClasses])) return c;
    return -1;
}

// ---- global-memory segment classes: one CTA per world; the planes stay in
// global memory (L2-resident for a batch of a few hundred MB) and shared
// memory holds only the change buffers and the layer list.  A step's work is
// the dirty layer pairs (a few per step: the moving surface), each of
// ceil(Z/2) block row-pairs times the lanes per pair, so the CTA is sized by
// that layer work, not by the world's volume: idle warps would wait at every
// step's barrier.  Each class caps the layers it holds flags for so that its
// CTAs per SM (24 warps in all) fit in shared memory.
int resident_class_gm(int X, int Y, int Z) {
    const int lanes = nblocks(Z, 1) << plane_lg(plane_nw(X));  // lane tasks of one layer pair
    const int c = gm_class_holding(lanes <= 16 ? 0 : (lanes <= 48 ? 1 : (lanes <= 96 ? 2 : 3)), Y);
    return c < kGmDense ? c : -1;
}

template <int NT>
static cudaError_t launch_gm(int cls, int grid, size_t smem, cudaStream_t st, const PlaneWorld* worlds,
                             const int* order, const int* meta, int* counter, int* err,
                             unsigned long long* processed_cells, bool first) {
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)grid);
    lc.blockDim = dim3((unsigned)NT);
    lc.dynamicSmemBytes = smem;
    lc.stream = st;
    cudaLaunchAttribute attr[1];
    if (first) {
        // the greatest priority: its CTAs take the SMs before the other
        // classes' grids, which are pending at the same moment in a segment graph
        static const int greatest = [] {
            int least = 0, g = 0;
            if (cudaDeviceGetStreamPriorityRange(&least, &g) != cudaSuccess) g = 0;
            return g;
        }();
        attr[0].id = cudaLaunchAttributePriority;
        attr[0].val.priority = greatest;
    }
    lc.attrs = attr;
    lc.numAttrs = first ? 1 : 0;
    return cudaLaunchKernelEx(&lc, k_plane_segment_resident<NT, true>, worlds, order, meta,
                              kResidentClasses + cls, counter, err, processed_cells);
}

fs3d_status launch_plane_segment_gm(int cls, const PlaneWorld* worlds, const int* order, const int* meta,
                                    int* counter, int* err, cudaStream_t st, unsigned long long* processed_cells,
                                    bool first) {
    if (cls < 0 || cls >= kGmClasses) return set_error(FS3D_ERR_INVALID_ARG, "global-memory class out of range");
    static PerContext<bool> carved;
    of_current_context(carved, [] {
        // the planes are read through L1: leave most of the unified memory to it
        const void* fns[kGmClasses] = {reinterpret_cast<const void*>(&k_plane_segment_resident<32, true>),
                                       reinterpret_cast<const void*>(&k_plane_segment_resident<64, true>),
                                       reinterpret_cast<const void*>(&k_plane_segment_resident<128, true>),
                                       reinterpret_cast<const void*>(&k_plane_segment_resident<256, true>),
                                       reinterpret_cast<const void*>(&k_plane_segment_resident<768, true>)};
        for (const void* fn : fns) cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 50);
        cudaGetLastError();
        return true;
    });
    FS3D_CUDA(cudaMemsetAsync(counter, 0, sizeof(int), st));
    const int nt = kGmThreads[cls];
    const int grid = sm_count_public() * (kGmThreadsPerSm / nt);
    const size_t smem = slab_aux_bytes((uint32_t)kGmMaxY[cls]);
    cudaError_t e;
    if (nt == 32)
        e = launch_gm<32>(cls, grid, smem, st, worlds, order, meta, counter, err, processed_cells, first);
    else if (nt == 64)
        e = launch_gm<64>(cls, grid, smem, st, worlds, order, meta, counter, err, processed_cells, first);
    else if (nt == 128)
        e = launch_gm<128>(cls, grid, smem, st, worlds, order, meta, counter, err, processed_cells, first);
    else if (nt == 256)
        e = launch_gm<256>(cls, grid, smem, st, worlds, order, meta, counter, err, processed_cells, first);
    else
        e = launch_gm<768>(cls, grid, smem, st, worlds, order, meta, counter, err, processed_cells, first);
    if (e != cudaSuccess) return cuda_fail(e, "global-memory segment launch");
    note_launch();
    return FS3D_OK;
}

fs3d_status set_inject_tx_extra(uint32_t stall) {
    const fs3d_status s = set_slab_stall(stall == kStallOneCta ? (uint32_t)kStallNone : stall);
    if (s != FS3D_OK) return s;
    const uint32_t bytes = stall == kStallAll || stall == kStallOneCta ? 16u : 0u;
    FS3D_CUDA(cudaMemcpyToSymbol(g_inject_tx_extra, &bytes, sizeof(bytes)));
    return FS3D_OK;
}

fs3d_status launch_plane_segment_resident(int cls, const PlaneWorld* worlds, const int* order, const int* meta,
                                          int* counter, int* err, cudaStream_t st,
                                          unsigned long long* processed_cells) {
    if (cls < 0 || cls >= kSingleCtaClasses) return set_error(FS3D_ERR_INVALID_ARG, "resident class out of range");
    const ResidentCfg k = resident_cfgs().c[cls];
    if (!k.smem) return set_error(FS3D_ERR_CUDA, "resident segment kernel unavailable for this class");
    FS3D_CUDA(cudaMemsetAsync(counter, 0, sizeof(int), st));
    const unsigned grid = (unsigned)(sm_count_public() * k.ctas_per_sm);
    auto fn = k.threads == 128 ? &k_plane_segment_resident<128>
                               : (k.threads == 256 ? &k_plane_segment_resident<256> : &k_plane_segment_resident<768>);
    fn<<<grid, (unsigned)k.threads, (size_t)k.smem, st>>>(worlds, order, meta, cls, counter, err, processed_cells);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "resident segment launch");
    note_launch();
    return FS3D_OK;
}

int sm_count_public();

static int conv_grid(int64_t n) {
    const int64_t need = (n + 255) / 256, cap = (int64_t)sm_count_public() * 8;
    return (int)(need < 1 ? 1 : (need < cap ? need : cap));
}

int plane_lg(int nw) {
    int lg = 0;
    while ((1 << lg) < nw) ++lg;
    return lg;
}

int plane_items_for(int Y, int Z, int nw) {
    const int per = 32 >> plane_lg(nw);
    const int nrp = nblocks(Y, 1) * nblocks(Z, 1);
    return (nrp + per - 1) / per;
}

// Each warp moves 2 KB blocks: lane l takes the 16-byte chunks 32i + l of its
// block (contiguous 512 bytes per instruction), all four loads before the
// stores; one job search per block (a block spans at most a few jobs).
__global__ void k_copy_many(const CopyJob* __restrict__ jobs, const int64_t* __restrict__ chunk_off, int njobs,
                            int64_t total) {
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t blk = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; blk * 128 < total; blk += nwarps) {
        int j = find_job(chunk_off, njobs, blk * 128);
        const uint8_t* src[4];
        uint8_t* dst[4];
        int n[4];
        uint4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int64_t u = blk * 128 + 32 * i + lane;
            n[i] = 0;
            if (u >= total) continue;
            while (j + 1 < njobs && __ldg(chunk_off + j + 1) <= u) ++j;
            const CopyJob& jb = jobs[j];
            const int64_t off = (u - __ldg(chunk_off + j)) * 16;
            n[i] = (int)(jb.bytes - off < 16 ? jb.bytes - off : 16);
            src[i] = jb.src + off;
            dst[i] = jb.dst + off;
            if (n[i] == 16 && ((reinterpret_cast<uintptr_t>(src[i]) | reinterpret_cast<uintptr_t>(dst[i])) & 15u) == 0)
                v[i] = *reinterpret_cast<const uint4*>(src[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (!n[i]) continue;
            if (n[i] == 16 && ((reinterpret_cast<uintptr_t>(src[i]) | reinterpret_cast<uintptr_t>(dst[i])) & 15u) == 0)
                *reinterpret_cast<uint4*>(dst[i]) = v[i];
            else
                for (int k = 0; k < n[i]; ++k) dst[i][k] = src[i][k];
        }
    }
}

// A small copy done by the SMs (16-byte pieces, then the last bytes one by
// one): either side may be page-locked host memory the device can address.
__global__ void k_copy_small(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, size_t bytes) {
    const size_t n16 = bytes / 16;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += (size_t)gridDim.x * blockDim.x)
        reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
    if (blockIdx.x == 0 && threadIdx.x == 0)
        for (size_t i = n16 * 16; i < bytes; ++i) dst[i] = src[i];
}

cudaError_t copy_small_async(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    if (bytes == 0) return cudaSuccess;
    if (((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15u) != 0)
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, st);
    const size_t n16 = bytes / 16;
    const int64_t need = (int64_t)((n16 + 255) / 256), cap = (int64_t)sm_count_public() * 2;
    const int grid = (int)(need < 1 ? 1 : (need < cap ? need : cap));
    k_copy_small<<<grid, 256, 0, st>>>(static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), bytes);
    const cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) note_launch();
    return e;
}

fs3d_status copy_many(const CopyJob* jobs, const int64_t* chunk_off, int njobs, int64_t total_chunks,
                      cudaStream_t st) {
    if (njobs <= 0 || total_chunks <= 0) return FS3D_OK;
    const int64_t blocks_needed = (total_chunks + 128 * 8 - 1) / (128 * 8), cap = (int64_t)sm_count_public() * 8;
    const int grid = (int)(blocks_needed < cap ? blocks_needed : cap);
    k_copy_many<<<grid < 1 ? 1 : grid, 256, 0, st>>>(jobs, chunk_off, njobs, total_chunks);
    FS3D_CHECK_LAUNCH("many-copy launch");
    return FS3D_OK;
}

uint8_t* device_view(const void* p) {
    cudaPointerAttributes a{};
    if (!p || cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged)
        return static_cast<uint8_t*>(const_cast<void*>(p));
    if (a.type == cudaMemoryTypeHost && a.devicePointer) return static_cast<uint8_t*>(a.devicePointer);
    return nullptr;
}

bool device_local(const void* p) {
    cudaPointerAttributes a{};
    int dev = -1;
    if (!p || cudaGetDevice(&dev) != cudaSuccess || cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice && a.device == dev;
}

bool alloc_range(const void* p, uintptr_t* start, size_t* bytes) {
    // cuPointerGetAttributes, looked up once through the runtime (no link
    // dependency on the driver library)
    using GetAttrs = int (*)(unsigned int, int*, void**, unsigned long long);
    static GetAttrs fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttributes", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        cudaGetLastError();
        return reinterpret_cast<GetAttrs>(f);
    }();
    if (!fn || !p) return false;
    unsigned long long base = 0, size = 0;
    int attrs[2] = {11, 12};  // CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE
    void* data[2] = {&base, &size};
    if (fn(2, attrs, data, (unsigned long long)reinterpret_cast<uintptr_t>(p)) != 0 || size == 0) return false;
    if (reinterpret_cast<uintptr_t>(p) < base || reinterpret_cast<uintptr_t>(p) >= base + size) return false;
    *start = (uintptr_t)base;
    *bytes = (size_t)size;
    return true;
}

GenJob gen_job(uint64_t world_seed, int X, int Y, int Z, uint4* rows) {
    return GenJob{rows, X, Y, Z, plane_nw(X), batch_world_gen(world_seed)};
}

fs3d_status planes_generate_batch_world(uint64_t world_seed, int X, int Y, int Z, uint4* rows, cudaStream_t st) {
    k_gen_batch_planes<<<(unsigned)conv_blocks(Y, Z, plane_nw(X), kConvChunks), kConvThreads, 0, st>>>(
        nullptr, nullptr, gen_job(world_seed, X, Y, Z, rows));
    FS3D_CHECK_LAUNCH("generate batch world launch");
    return FS3D_OK;
}

fs3d_status planes_generate_multi(const GenJob* jobs, const ConvBlock* blocks, int64_t nblocks, cudaStream_t st) {
    if (nblocks <= 0) return FS3D_OK;
    k_gen_batch_planes<<<(unsigned)nblocks, kConvThreads, 0, st>>>(jobs, blocks, GenJob{});
    FS3D_CHECK_LAUNCH("generate batch worlds launch");
    return FS3D_OK;
}

fs3d_status planes_hash_async(const uint4* rows, const uint8_t* statics, int X, int Y, int Z,
                              unsigned long long* out_dev, cudaStream_t st) {
    const int nw = plane_nw(X);
    FS3D_CUDA(cudaMemsetAsync(out_dev, 0, sizeof(unsigned long long), st));
    k_hash_planes<<<conv_grid((int64_t)Y * Z * nw), 256, 0, st>>>(rows, statics, X, Y, Z, nw, out_dev);
    FS3D_CHECK_LAUNCH("hash planes launch");
    return FS3D_OK;
}

fs3d_status planes_hash_many(const HashJob* jobs, int njobs, int parts, unsigned long long* out_dev, cudaStream_t st) {
    if (njobs <= 0) return FS3D_OK;
    k_hash_planes_many<<<dim3((unsigned)njobs, (unsigned)parts), 256, 0, st>>>(jobs, out_dev);
    FS3D_CHECK_LAUNCH("hash many worlds launch");
    return FS3D_OK;
}

fs3d_status launch_plane_step(const PlaneWorld* worlds, const PlaneItem* items, const int* n_items_dev,
                              int grid, int s_seg, cudaStream_t st) {
    k_plane_step<<<grid, 256, 0, st>>>(worlds, items, n_items_dev, s_seg);
    FS3D_CHECK_LAUNCH("plane step launch");
    return FS3D_OK;
}

__global__ void k_advance_worlds(PlaneWorld* __restrict__ worlds, const int* __restrict__ meta) {
    const int n = meta[kMetaWorlds];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        PlaneWorld& w = worlds[i];
        w.t += (uint64_t)w.steps;
        if (w.lflags) w.lflags_fresh = 0;
    }
}

fs3d_status launch_advance_worlds(PlaneWorld* worlds, const int* meta, cudaStream_t st) {
    k_advance_worlds<<<8, 256, 0, st>>>(worlds, meta);
    FS3D_CHECK_LAUNCH("advance worlds launch");
    return FS3D_OK;
}

fs3d_status init_row_flags(const uint4* rows, uint8_t* rflags, int X, int Y, int Z, uint64_t t0, cudaStream_t st,
                           const int* err, int* own) {
    FS3D_CUDA(cudaMemsetAsync(rflags, (int)((t0 - 3u) & 0xFFu), (size_t)Y * (size_t)Z, st));
    const int nw = plane_nw(X), per = 32 >> plane_lg(nw);
    const int64_t items = (int64_t)nblocks(Y, 0) * ((nblocks(Z, 0) + per - 1) / per);  // the larger phase's
    const int64_t blocks = std::min<int64_t>((items + 7) / 8, (int64_t)sm_count_public() * 8);
    k_row_flags_from_cells<<<(unsigned)std::max<int64_t>(blocks, 1), 256, 0, st>>>(rows, rflags, X, Y, Z, nw,
                                                                                   (uint32_t)t0 & 0xFFu, err, own);
    FS3D_CUDA(cudaGetLastError());
    note_launch();
    return FS3D_OK;
}

fs3d_status layer_flags_from_cells_multi(const ConvJob* jobs, int njobs, int max_Y, cudaStream_t st) {
    if (njobs <= 0 || max_Y <= 0) return FS3D_OK;
    k_layer_flags_from_cells<<<dim3((unsigned)njobs, (unsigned)((max_Y + 7) / 8)), 256, 0, st>>>(jobs, ConvJob{});
    FS3D_CUDA(cudaGetLastError());
    note_launch();
    return FS3D_OK;
}

fs3d_status layer_flags_from_cells(const uint4* rows, uint8_t* lflags, int X, int Y, int Z, uint64_t t0,
                                   cudaStream_t st) {
    ConvJob one{};
    one.rows = const_cast<uint4*>(rows);
    one.X = X;
    one.Y = Y;
    one.Z = Z;
    one.nw = plane_nw(X);
    one.lflags = lflags;
    one.t0b = (uint32_t)t0 & 0xFFu;
    k_layer_flags_from_cells<<<dim3(1u, (unsigned)((Y + 7) / 8)), 256, 0, st>>>(nullptr, one);
    FS3D_CUDA(cudaGetLastError());
    note_launch();
    return FS3D_OK;
}

fs3d_status launch_plane_step_skip(const PlaneWorld& w, uint8_t* rflags, int* counts, const int* err, cudaStream_t st) {
    const int per = 32 >> w.lg;
    const int64_t nrp = (int64_t)nblocks(w.Y, 1) * nblocks(w.Z, 1);
    const int64_t need = ((nrp + per - 1) / per + 7) / 8;  // eight warps per CTA
    const int64_t cap = (int64_t)sm_count_public() * 3;    // the kernel's launch bound
    const int grid = (int)(need < 1 ? 1 : (need < cap ? need : cap));
    const auto fn = need > 2 * cap ? &k_plane_step_skip<true> : &k_plane_step_skip<false>;
    const cudaError_t e = launch_chained(fn, (unsigned)grid, 256, st, w, rflags, counts, err);
    if (e != cudaSuccess) return cuda_fail(e, "plane step (settled skip) launch");
    note_launch();
    return FS3D_OK;
}

// CTAs of the step kernel that fit on one SM at once
int plane_step_ctas_per_sm() {
    static const int n = [] {
        int v = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_plane_step, 256, 0) != cudaSuccess || v < 1) v = 1;
        return v;
    }();
    return n;
}

// persistent grid: every CTA resident, so warps pick items without tail waves
int plane_step_grid(int64_t n_items) {
    const int64_t warps_per_cta = 8;
    const int64_t need = (n_items + warps_per_cta - 1) / warps_per_cta;
    const int64_t cap = (int64_t)sm_count_public() * plane_step_ctas_per_sm();
    return (int)(need < 1 ? 1 : (need < cap ? need : cap));
}

}  // namespace fs3d
