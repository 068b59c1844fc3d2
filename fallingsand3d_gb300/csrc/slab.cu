// Many steps of one world by several CTAs: over the whole GPU (one world in one
// launch) or by one thread-block cluster (a batch's large young worlds).
//
// The world is cut along y or z into slabs of whole layer pairs, one CTA per
// slab, and each CTA keeps its slab's planes and row flags in shared memory
// for all the steps.  Margolus blocks of one step are disjoint, so a step
// needs no other CTA's work except at the cuts: in the even phase every block
// row-pair lies inside a slab; in the odd phase the pairs that straddle a cut
// are taken by the slab above it.  The last layer of a slab (all but the last
// slab's) is therefore touched by its own CTA in even steps and by the next
// CTA in odd steps, and by no one else.  It lives in a global buffer (the
// edge buffer), word by word, as a token that the two CTAs pass to and fro:
// each 32-bit word of a plane word is stored beside a tag in one 64-bit
// store, the tag being the number of steps the word has taken (bit 31: its
// row changed in the last of them).  The CTA whose turn it is reads the word
// until its tag is the step's, and stores it again with the next tag.  A word
// carries its own tag, so no fence, flag or barrier is needed between the
// CTAs, and only the two neighbours of a cut ever wait on one another.  A
// word is stored again by the lane that read it, so a word is never
// overwritten before it was read.
//
// All CTAs of a world are resident at once (a cooperative launch, or a
// cluster).  Every wait is bounded in time; the planes and flags in global
// memory are written only once every CTA has taken all the steps, on one
// decision for the whole world: in a whole-GPU launch the last CTA to arrive
// commits and one that gives up aborts, whichever is first; in a cluster its
// first CTA looks at the batch's error record once.  A world whose launch
// fails is as it was.
//
// Bound: latency.  A step of a small world is a chain of a word's way through
// L2 to the neighbour (the draws hidden in that wait), the slots' serial chain
// and the loads, stores and barrier around it; a warp spends half of its cycles
// at the barrier, that is, waiting for the CTA's slowest one.
// Measured per step (everything falling / settled), against the launch per
// step and, where the world fitted, one CTA or cluster for the whole world:
// 96x80x112 2.5 / 2.4 us against 6.6 and 6.9, 128^3 3.3 / 3.1 against 7.0 and
// 12, 200^3 4.1 / 3.5 against 6.5 / 7.3, 256^3 4.9 / 3.7 against 7.1 / 8.2.
#include <stdint.h>

#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>

#include "fs3d_common.h"
#include "planes.h"
#include "bulk_device.cuh"
#include "rule_device.cuh"

namespace fs3d {

namespace {

constexpr int kSlabKeys = 32;  // step keys computed together
// threads of a batch's cluster CTAs, by the order of their row-pairs (slab_steps).
// By place, 512 threads of 128 registers, without spills, are 5 to 10 % faster
// than 640 on 128^3, 96^3 and 64x64x1024.
template <bool PLACE>
constexpr int batch_slab_threads() { return PLACE ? 512 : 640; }

// Test hook (fs3d_test_inject): which bulk copies are announced with more bytes
// than they deliver (a CopyStall, planes.h).  0 in normal operation.
static __device__ uint32_t g_slab_stall;
constexpr uint32_t kStallBytes = 16;
// bytes announced too many by CTA r, and the limits of its copy's wait and of
// the waits for other CTAs: of the first CTA's stall, theirs run out first
__device__ __forceinline__ uint32_t stall_bytes(uint32_t stall, int r) {
    return stall == kStallAll || (stall == kStallFirstSlab && r == 0) ? kStallBytes : 0u;
}
__device__ __forceinline__ uint64_t copy_limit(uint32_t stall) {
    return stall == 0 ? kCopyWaitNs : (stall == kStallAll ? 1u : 2u) * kCopyWaitInjectedNs;
}
__device__ __forceinline__ uint64_t peer_limit() {
    return *(volatile uint32_t*)&g_slab_stall ? kCopyWaitInjectedNs : kCopyWaitNs;
}

// The launch's shared words, zeroed before it, at the start of the scratch;
// the edge buffer follows at kSlabEdgeOff.
struct SlabState {
    int arrived;  // CTAs that have taken all the steps
    int verdict;  // 0 open, 1 commit, 2 abort
};
constexpr size_t kSlabEdgeOff = 256;

__device__ __forceinline__ void ld_tagged(const unsigned long long* p, unsigned long long& a, unsigned long long& b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_tagged(unsigned long long* p, unsigned long long a, unsigned long long b) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ unsigned long long tagged(uint32_t data, uint32_t tag) {
    return ((unsigned long long)tag << 32) | data;
}

// One edge word (four tagged 32-bit words): true once it has taken `step`
// steps; *changed = its row changed in the last of them.
__device__ __forceinline__ bool edge_try(const unsigned long long* p, uint32_t step, uint4& q, bool& changed) {
    unsigned long long a, b, c, d;
    ld_tagged(p, a, b);
    ld_tagged(p + 2, c, d);
    const uint32_t ta = (uint32_t)(a >> 32), tb = (uint32_t)(b >> 32), tc = (uint32_t)(c >> 32), td = (uint32_t)(d >> 32);
    q = make_uint4((uint32_t)a, (uint32_t)b, (uint32_t)c, (uint32_t)d);
    changed = (ta >> 31) != 0;
    return (((ta ^ step) | (tb ^ step) | (tc ^ step) | (td ^ step)) & 0x7FFFFFFFu) == 0;
}

// Waits for the edge words at p0 and p1 (each nullable) to have taken `step`
// steps.  False if it gave up: the wait's limit, *stop set (a verdict reached
// without this CTA, or an error recorded), or *dead set by another of its
// threads.
__device__ __forceinline__ bool edge_read(const unsigned long long* p0, const unsigned long long* p1, uint32_t step,
                                          const int* stop, const volatile int* dead, uint4& q0, uint4& q1,
                                          bool& ch0, bool& ch1) {
    unsigned long long t0 = 0;
    for (uint32_t it = 0;; ++it) {
        const bool ok0 = !p0 || edge_try(p0, step, q0, ch0), ok1 = !p1 || edge_try(p1, step, q1, ch1);
        if (ok0 && ok1) return true;
        if ((it & 255u) == 255u) {
            if (*dead || *(volatile const int*)stop) return false;
            const unsigned long long now = global_ns();
            if (!t0)
                t0 = now;
            else if (now - t0 > peer_limit())
                return false;
        }
    }
}

__device__ __forceinline__ void edge_write(unsigned long long* p, const uint4& q, uint32_t tag) {
    st_tagged(p, tagged(q.x, tag), tagged(q.y, tag));
    st_tagged(p + 2, tagged(q.z, tag), tagged(q.w, tag));
}

// One lane's part of a block row-pair of a step's phase, worked out once per
// phase when a slab's row-pairs all have a lane group of their own.
struct SlabTask {
    int row;          // shared-memory plane word of row (y0, z0)
    int flag;         // its row flag
    int edge;         // edge-buffer word (in 64-bit units) of row c0 of the cut's layer
    int c0;           // the pair's first row along the other axis
    uint32_t hj, hk;  // the row key's inputs
    uint32_t in;      // bit a: row a lies in the world (0: nothing to do)
    bool cut;         // the pair's rows of one layer are the cut's
};

// What CTA r of C holds of a world cut along z (ZS) or y.
template <bool ZS>
struct SlabGeo {
    int NO;          // the world's size along the other axis
    bool first, last;
    int lo, hi;      // its layers along the cut axis
    int keep;        // layers lo .. keep-1 are held here, layer hi-1 of an inner slab in the edge buffer
    int layers;
    int row_ys, row_off;  // shared-memory row of (y, z): y * row_ys + z + row_off
    int fl_ys, fl_off;    // row flag, of layers lo-1 .. hi-1 (the edge layers' too)
    uint32_t bytes;       // of the planes held
    __device__ __forceinline__ SlabGeo(const PlaneWorld& w, int r, int C) {
        const int NS = ZS ? w.Z : w.Y, NP = (NS + 1) >> 1;
        NO = ZS ? w.Y : w.Z;
        first = r == 0;
        last = r == C - 1;
        lo = 2 * (int)((int64_t)r * NP / C);
        hi = last ? NS : 2 * (int)((int64_t)(r + 1) * NP / C);
        keep = last ? hi : hi - 1;
        layers = keep - lo;
        row_ys = ZS ? layers : w.Z;
        row_off = ZS ? -lo : -lo * w.Z;
        fl_ys = ZS ? hi - lo + 1 : w.Z;
        fl_off = ZS ? 1 - lo : (1 - lo) * w.Z;
        bytes = (uint32_t)layers * (uint32_t)NO * (uint32_t)w.nw * 16u;
    }
    // (y, z) of row flag i
    __device__ __forceinline__ void flag_at(const PlaneWorld& w, int i, int& y, int& z) const {
        y = ZS ? i / fl_ys : lo - 1 + i / w.Z;
        z = ZS ? lo - 1 + i % fl_ys : i % w.Z;
    }
    __device__ __forceinline__ int flags() const { return (hi - lo + 1) * NO; }
    // the planes into shared memory, as bulk copies on `bar` (told to expect them)
    __device__ __forceinline__ void load(const PlaneWorld& w, uint4* srows, uint64_t* bar) const {
        const int pieces = ZS ? w.Y : 1;
        const uint32_t pb = bytes / (uint32_t)pieces;
        for (int i = threadIdx.x; i < pieces; i += blockDim.x) {
            const uint4* src = w.rows + (ZS ? ((int64_t)i * w.Z + lo) * w.nw : (int64_t)lo * w.Z * w.nw);
            bulk_copy_in(reinterpret_cast<uint8_t*>(srows) + (size_t)i * pb, src, pb, bar);
        }
    }
    // the edge layer this CTA took the last step of (-1: none); o: that step's phase
    __device__ __forceinline__ int last_edge(int o) const { return o ? (first ? -1 : lo - 1) : (last ? -1 : hi - 1); }
    // the planes back, and the edge layer el from the edge buffer (r: this CTA, o as above)
    __device__ __forceinline__ void store(const PlaneWorld& w, const uint4* srows, const unsigned long long* edge, int r,
                                          int o) const {
        const int nw = w.nw, el = last_edge(o);
        for (int i = threadIdx.x; i < layers * NO * nw; i += blockDim.x) {
            const int row = i / nw, g = i - row * nw;
            const int y = ZS ? row / layers : lo + row / w.Z, z = ZS ? lo + row % layers : row % w.Z;
            w.rows[((int64_t)y * w.Z + z) * nw + g] = srows[i];
        }
        if (el < 0) return;
        const unsigned long long* eb = edge + (size_t)(o ? r - 1 : r) * NO * nw * 4;
        for (int i = threadIdx.x; i < NO * nw; i += blockDim.x) {
            unsigned long long a, b, c, d;
            ld_tagged(eb + 4 * (size_t)i, a, b);
            ld_tagged(eb + 4 * (size_t)i + 2, c, d);
            const int row = i / nw, g = i - row * nw;
            const int y = ZS ? row : el, z = ZS ? el : row;
            w.rows[((int64_t)y * w.Z + z) * nw + g] = make_uint4((uint32_t)a, (uint32_t)b, (uint32_t)c, (uint32_t)d);
        }
    }
    // whether the row flag of (y, z) is this CTA's to report
    __device__ __forceinline__ bool owns(int y, int z, int o) const {
        const int sl = ZS ? z : y, el = last_edge(o);
        return (sl >= lo && sl < keep) || (el >= 0 && sl == el);
    }
};

// The steps of CTA r's slab (planes in srows, row flags in rf).  ZS, READY: the
// draws of a row-pair are hashed before its cut's words are waited for (few
// warps per SM: a step is one warp's chain of instructions and the words' way
// through L2, and the hashing hides in the latter), else slot by slot where
// needed (more warps: the instructions count).  True if it gave up (or came in
// dead).  rows_done: the rows of the row-pairs this lane evaluated.
// Threads work in lane groups of 1 << lg, one block row-pair at a time, as
// the per-step kernel does; row-pairs none of whose rows changed in the two
// previous steps are skipped (same argument, same row flags).
//
// The cut's layer pair comes first, since the neighbour waits for it, and the
// others after it, one layer pair after another, or (PLACE) the row-pairs of one
// place along the other axis, y, in all of them, then the next place's.  A young
// world falls from the top and rests at the bottom, so with a whole number of
// layer pairs in a pass the same warps have the resting rows in every pass and
// others the falling ones: two 64-step segments of one 128^3 world, 4 CTAs, 1530
// us layer pair by layer pair and 905 by place; 60 worlds of 96^3 over 2 CTAs
// each 1365 and 1070; 64x64x1024 over 8 1362 and 733.  Where a slab's row-pairs
// have a lane group each (most whole-GPU launches) there is but one pass, and
// the row-pair of a group is worked out once per phase.
template <bool ZS, bool READY, bool PLACE>
__device__ __forceinline__ bool slab_steps(const PlaneWorld& w, const SlabGeo<ZS>& geo, int r, uint4* srows, uint8_t* rf,
                                           unsigned long long* edge, const int* stop, volatile int* s_dead,
                                           uint32_t* s_keys, bool dead, uint32_t& rows_done) {
    const int NO = geo.NO, lo = geo.lo, hi = geo.hi, row_ys = geo.row_ys, row_off = geo.row_off, fl_ys = geo.fl_ys,
              fl_off = geo.fl_off;
    const bool first = geo.first, last = geo.last;
    const int tid = threadIdx.x, NT = blockDim.x, nw = w.nw;
    const int lane = tid & 31, lg = w.lg, G = 1 << lg, per = NT >> lg, gl = lane & (G - 1);
    const uint32_t gmask = G == 32 ? 0xFFFFFFFFu : ((1u << G) - 1u) << (lane & ~(G - 1));
    const bool half_at_end = (w.X & 63) == 0;
    auto tasks = [&](int o) {
        const int np = o ? ((hi - lo) >> 1) + (last ? 1 : 0) : (hi - lo + 1) >> 1;
        return np * ((NO + o + 1) >> 1);
    };
    auto task = [&](int o, int e) {
        const int NB = (NO + o + 1) >> 1, n = tasks(o), np = n / NB;
        SlabTask t{};
        if (e >= n || gl >= nw) return t;
        int pi = e / NB, k = e - pi * NB;
        if (PLACE && e >= NB) {
            k = (e - NB) / (np - 1);
            pi = 1 + (e - NB) - k * (np - 1);
        }
        const int p = o ? pi : np - 1 - pi;  // the cut's pair first: its result travels while the rest is done
        const int s0 = lo - o + 2 * p, c0 = 2 * k - o;
        const int y0 = ZS ? c0 : s0, z0 = ZS ? s0 : c0;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int y = a < 2 ? y0 + 1 : y0, z = z0 + (a & 1);
            if (y >= 0 && y < w.Y && z >= 0 && z < w.Z) t.in |= 1u << a;
        }
        // the pair's lower layer is the slab below's edge (odd phase), or its upper layer this slab's
        t.cut = o ? p == 0 && !first : p == np - 1 && !last;
        t.row = (y0 * row_ys + z0 + row_off) * nw + gl;
        t.flag = y0 * fl_ys + z0 + fl_off;
        t.edge = (((o ? r - 1 : r) * NO + c0) * nw + gl) * 4;
        t.c0 = c0;
        t.hj = 0x85EBCA77u * (uint32_t)(((y0 + o) >> 1) + 1);
        t.hk = 0xC2B2AE3Du * (uint32_t)(((z0 + o) >> 1) + 1);
        return t;
    };
    bool gave_up = false;
    // one row-pair of step s (phase O) on every lane group of the warp
    auto evaluate = [&](auto phase, const SlabTask& k, int s, uint32_t tb, uint32_t sk) {
        constexpr int O = decltype(phase)::value;
        // rows a: (y0 + 1 for a < 2, z0 + (a & 1)); the cut's are the pair's lower
        // layer along the cut axis in the odd phase, its upper one in the even
        // phase: row c0 of that layer is a = E0, row c0 + 1 is a = E1
        constexpr int E0 = ZS ? (O ? 2 : 3) : (O ? 2 : 0), E1 = ZS ? (O ? 0 : 1) : (O ? 3 : 1);
        auto row = [&](int a) { return k.row + ((a < 2 ? row_ys : 0) + (a & 1)) * nw; };
        auto flag = [&](int a) { return k.flag + (a < 2 ? fl_ys : 0) + (a & 1); };
        // every lane of a group finds the same answer
        bool dirty = false;
#pragma unroll
        for (int a = 0; a < 4; ++a)
            if ((k.in >> a) & 1u) dirty |= ((tb - (uint32_t)rf[flag(a)]) & 0xFFu) - 1u < 2u;
        bool some = __any_sync(0xFFFFFFFFu, dirty);
        const bool cuts = __any_sync(0xFFFFFFFFu, k.cut);
        if (!some && !cuts) return;
        const uint32_t rk = fmix32(fmix32(sk ^ k.hj) ^ k.hk);
        ReadyDraws ready;
        if (READY && some) ready.fill(rk, (uint32_t)gl);
        uint4 q[4];
        const uint4 solid = make_uint4(0u, 0u, 0xFFFFFFFFu, 0xFFFFFFFFu);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const bool edge_row = k.cut && (a == E0 || a == E1);
            q[a] = dirty && ((k.in >> a) & 1u) && !edge_row ? srows[row(a)] : solid;
        }
        if (cuts) {
            const bool had = some;
            unsigned long long* p0 = k.cut && ((k.in >> E0) & 1u) ? edge + k.edge : nullptr;
            unsigned long long* p1 = k.cut && ((k.in >> E1) & 1u) ? edge + k.edge + 4 * nw : nullptr;
            if (s == 0) {
                // straight from the world
                const int l = O ? lo - 1 : hi - 1;
                auto at = [&](int c) { return w.rows[(ZS ? (int64_t)c * w.Z + l : (int64_t)l * w.Z + c) * nw + gl]; };
                if (p0) q[E0] = at(k.c0);
                if (p1) q[E1] = at(k.c0 + 1);
            } else if ((p0 || p1) && !gave_up) {
                bool ch0 = false, ch1 = false;
                gave_up = !edge_read(p0, p1, (uint32_t)s, stop, s_dead, q[E0], q[E1], ch0, ch1);
                if (ch0) rf[flag(E0)] = (uint8_t)(tb - 1u);
                if (ch1) rf[flag(E1)] = (uint8_t)(tb - 1u);
                if ((ch0 || ch1) && !dirty) {
                    dirty = true;
#pragma unroll
                    for (int a = 0; a < 4; ++a)
                        if (a != E0 && a != E1 && ((k.in >> a) & 1u)) q[a] = srows[row(a)];
                }
            }
            some = __any_sync(0xFFFFFFFFu, dirty);
            if (READY && some && !had) ready.fill(rk, (uint32_t)gl);
        }
        if (dirty && gl == 0) rows_done += __popc(k.in);
        uint32_t chg = 0;  // bit a: row a changed in this lane's word
        if (some) {
            uint4 q0[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) q0[a] = q[a];
            if constexpr (READY)
                rowpair_core(q, dirty, O, ready, gl, G, nw, half_at_end);
            else
                rowpair_core(q, dirty, O, LazyDraws{rk, (uint32_t)gl}, gl, G, nw, half_at_end);
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const bool c = dirty && ((k.in >> a) & 1u) &&
                               (q[a].x != q0[a].x || q[a].y != q0[a].y || q[a].z != q0[a].z || q[a].w != q0[a].w);
                if (c) {
                    chg |= 1u << a;
                    rf[flag(a)] = (uint8_t)tb;
                    if (!(k.cut && (a == E0 || a == E1))) srows[row(a)] = q[a];
                }
            }
        }
        if (cuts) {
            const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, k.cut && ((chg >> E0) & 1u)) & gmask;
            const uint32_t b1 = __ballot_sync(0xFFFFFFFFu, k.cut && ((chg >> E1) & 1u)) & gmask;
            if (k.cut && !gave_up) {
                if ((k.in >> E0) & 1u) edge_write(edge + k.edge, q[E0], (uint32_t)(s + 1) | (b0 ? 0x80000000u : 0u));
                if ((k.in >> E1) & 1u)
                    edge_write(edge + k.edge + 4 * nw, q[E1], (uint32_t)(s + 1) | (b1 ? 0x80000000u : 0u));
            }
        }
    };
    const bool once = !PLACE && max(tasks(0), tasks(1)) <= per;  // a lane group for every row-pair of either phase
    SlabTask even{}, odd{};
    if (once) {
        even = task(0, tid >> lg);
        odd = task(1, tid >> lg);
    }
    for (int s = 0; s < w.steps && !dead; ++s) {
        if ((s & (kSlabKeys - 1)) == 0) {
            // the previous step's barrier is behind every reader of the last keys
            for (int i = tid; i < kSlabKeys; i += NT) s_keys[i] = stepkey(w.seed, w.t + (uint64_t)(s + i));
            __syncthreads();
        }
        const uint64_t t = w.t + (uint64_t)s;
        const uint32_t tb = (uint32_t)t & 0xFFu, sk = s_keys[s & (kSlabKeys - 1)];
        if (t & 1u) {
            if (once)
                evaluate(std::integral_constant<int, 1>(), odd, s, tb, sk);
            else
                for (int e = tid >> lg, n = tasks(1); e - (tid >> lg) < n; e += per)
                    evaluate(std::integral_constant<int, 1>(), task(1, e), s, tb, sk);
        } else {
            if (once)
                evaluate(std::integral_constant<int, 0>(), even, s, tb, sk);
            else
                for (int e = tid >> lg, n = tasks(0); e - (tid >> lg) < n; e += per)
                    evaluate(std::integral_constant<int, 0>(), task(0, e), s, tb, sk);
        }
        if (gave_up) *s_dead = 1;
        dead = __syncthreads_or(gave_up) != 0;
    }
    return dead;
}

// One world over the whole GPU.  MAXT: the most threads.
template <bool ZS, int MAXT, bool READY>
__global__ void __launch_bounds__(MAXT, 1)
    k_plane_slabs(const PlaneWorld w, uint8_t* __restrict__ rflags, SlabState* st, unsigned long long* edge, int* err,
                  int* own) {
    extern __shared__ __align__(128) uint4 srows[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t s_keys[kSlabKeys];
    __shared__ int s_dead, s_verdict;  // s_dead: some thread gave up (a hint to the others' waits)
    const int C = gridDim.x, r = blockIdx.x, tid = threadIdx.x;
    const SlabGeo<ZS> geo(w, r, C);
    const uint32_t stall = g_slab_stall;
    uint8_t* rf = reinterpret_cast<uint8_t*>(srows) + geo.bytes;
    if (tid == 0) {
        mbar_init(&bar, 1);
        s_dead = 0;
        mbar_expect(&bar, geo.bytes + stall_bytes(stall, r));
    }
    // an error recorded earlier: nothing is stepped (and every CTA's load is skipped or waited for)
    bool dead = __syncthreads_or(tid == 0 && *(volatile int*)own != 0) != 0;
    if (!dead) {
        geo.load(w, srows, &bar);
        for (int i = tid; i < geo.flags(); i += blockDim.x) {
            int y, z;
            geo.flag_at(w, i, y, z);
            rf[i] = (y >= 0 && z >= 0) ? rflags[(int64_t)y * w.Z + z] : 0;
        }
        const bool ok = mbar_wait(&bar, 0, copy_limit(stall));
        dead = __syncthreads_or(!ok) != 0;
    }
    uint32_t rows_done = 0;
    dead = slab_steps<ZS, READY, false>(w, geo, r, srows, rf, edge, &st->verdict, &s_dead, s_keys, dead, rows_done);
    // the verdict: commit when every CTA has taken all the steps
    if (tid == 0) {
        if (dead)
            atomicCAS(&st->verdict, 0, 2);
        else if (atomicAdd(&st->arrived, 1) == C - 1)
            atomicCAS(&st->verdict, 0, 1);
        const unsigned long long t0 = global_ns();
        int v;
        while ((v = *(volatile int*)&st->verdict) == 0) {
            if (global_ns() - t0 > peer_limit()) {
                v = atomicCAS(&st->verdict, 0, 2);
                if (v == 0) v = 2;
                break;
            }
        }
        s_verdict = v;
        if (v == 2) {
            if (atomicCAS(err, 0, 1) == 0) *reinterpret_cast<unsigned long long*>(err + 2) = (unsigned long long)w.t;
            *(volatile int*)own = 1;
        }
    }
    __syncthreads();
    if (s_verdict != 1) return;
    const int lasto = (int)((w.t + (uint64_t)w.steps - 1u) & 1u);
    geo.store(w, srows, edge, r, lasto);
    for (int i = tid; i < geo.flags(); i += blockDim.x) {
        int y, z;
        geo.flag_at(w, i, y, z);
        if (geo.owns(y, z, lasto)) rflags[(int64_t)y * w.Z + z] = rf[i];
    }
}

// A batch's worlds of one cluster class: each cluster of CS CTAs takes worlds
// of the class, largest first, from `counter`, and runs each through its
// segment steps, cut along z.  One SM's 24 warps took 850 to 1020 us for the
// 64 dense steps of a 128^3 world, which ended the segment of a batch of few
// such worlds.
template <bool PLACE>
__global__ void __launch_bounds__(batch_slab_threads<PLACE>(), 1)
    k_batch_slabs(const PlaneWorld* __restrict__ worlds, const int* __restrict__ order, const int* __restrict__ meta, int cls,
                  int CS, int* counter, int* err, unsigned long long* processed_cells, unsigned long long* edges) {
    extern __shared__ __align__(128) uint4 srows[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t s_keys[kSlabKeys];
    __shared__ int s_dead, s_write, item;
    __shared__ unsigned long long s_processed;
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();
    const int r = (int)cluster.block_rank(), tid = threadIdx.x, NT = blockDim.x;
    const int n = meta[1 + cls], off = meta[1 + kAllClasses + cls];
    unsigned long long* edge = edges + (size_t)(blockIdx.x / CS) * (size_t)(CS - 1) * kBatchSlabEdgeWords * 4;
    const uint32_t stall = g_slab_stall;
    if (tid == 0) {
        mbar_init(&bar, 1);
        s_processed = 0;
    }
    __syncthreads();
    uint32_t phase = 0;
    for (;;) {
        // the last world's planes and flags were written here with ordinary
        // stores, and the next world's bulk copies write the same bytes through
        // the async proxy: each thread orders its own before the barrier
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        // after an error no cluster takes another world
        if (r == 0 && tid == 0) item = *(volatile int*)err ? n : atomicAdd(counter, 1);
        if (tid == 0) s_dead = 0;
        cluster.sync();
        const int it = *cluster.map_shared_rank(&item, 0);
        cluster.sync();
        if (it >= n) break;
        const PlaneWorld w = worlds[order[off + it]];
        if (w.steps <= 0) continue;
        const SlabGeo<true> geo(w, r, CS);
        uint8_t* rf = reinterpret_cast<uint8_t*>(srows) + geo.bytes;
        if (tid == 0) mbar_expect(&bar, geo.bytes + stall_bytes(stall, r));
        __syncthreads();
        geo.load(w, srows, &bar);
        // row flags from the layers', or every row changed just before
        const bool kept = w.lflags != nullptr && !w.lflags_fresh;
        for (int i = tid; i < geo.flags(); i += NT) {
            int y, z;
            geo.flag_at(w, i, y, z);
            rf[i] = kept ? w.lflags[y] : (uint8_t)(w.t - 1u);
        }
        // this CTA's edge words: no tag of another world's left
        if (!geo.last)
            for (int i = tid; i < geo.NO * w.nw; i += NT) {
                st_tagged(edge + ((size_t)r * geo.NO * w.nw + i) * 4, 0, 0);
                st_tagged(edge + ((size_t)r * geo.NO * w.nw + i) * 4 + 2, 0, 0);
            }
        const bool ok = mbar_wait(&bar, phase, copy_limit(stall));
        phase ^= 1u;
        bool dead = __syncthreads_or(!ok) != 0;
        cluster.sync();
        uint32_t rows_done = 0;
        dead = slab_steps<true, false, PLACE>(w, geo, r, srows, rf, edge, err, &s_dead, s_keys, dead, rows_done);
        if (dead && tid == 0 && atomicCAS(err, 0, 1) == 0)
            *reinterpret_cast<unsigned long long*>(err + 2) = (unsigned long long)w.t;
        rows_done = __reduce_add_sync(0xFFFFFFFFu, rows_done);
        if ((tid & 31) == 0 && rows_done) atomicAdd(&s_processed, (unsigned long long)rows_done * (unsigned long long)w.X);
        // Write back or not is one answer for the whole world: another class's
        // kernel may record an error between two reads of the record, and a
        // world written by some of its CTAs only would be torn.
        cluster.sync();  // this cluster's own failures are recorded
        if (r == 0 && tid == 0) s_write = *(volatile int*)err == 0;
        cluster.sync();
        const bool write = *cluster.map_shared_rank(&s_write, 0) != 0;
        const uint64_t te = w.t + (uint64_t)w.steps;
        const int lasto = (int)((te - 1u) & 1u);
        if (write) geo.store(w, srows, edge, r, lasto);
        // layer flags: the last of the final two steps that changed one of the
        // layer's rows, older ones first (each value by any CTA that has it)
        if (w.lflags) {
            if (write && r == 0)
                for (int y = tid; y < w.Y; y += NT) w.lflags[y] = (uint8_t)(te - 3u);
            for (uint32_t age = 2; age > 0; --age) {
                cluster.sync();
                for (int i = tid; write && i < geo.flags(); i += NT) {
                    int y, z;
                    geo.flag_at(w, i, y, z);
                    if (rf[i] == (uint8_t)(te - age) && geo.owns(y, z, lasto)) w.lflags[y] = (uint8_t)(te - age);
                }
            }
        }
    }
    __syncthreads();
    if (tid == 0 && processed_cells && s_processed) atomicAdd(processed_cells, s_processed);
}

struct SlabLimits {
    int sms = 0;
    int smem = 0;        // dynamic shared memory a CTA may have (0: the kernels cannot run)
    int batch_smem = 0;  // and one of a batch's clusters
    int clusters = 0;    // clusters of 8 that run at once
};

constexpr int kSlabThreadsNarrow = 256, kSlabThreadsWide = 640;

using SlabFn = void (*)(const PlaneWorld, uint8_t*, SlabState*, unsigned long long*, int*, int*);
SlabFn slab_fn(bool zs, bool wide) {
    if (zs) return wide ? &k_plane_slabs<true, kSlabThreadsWide, false> : &k_plane_slabs<true, kSlabThreadsNarrow, true>;
    return wide ? &k_plane_slabs<false, kSlabThreadsWide, false> : &k_plane_slabs<false, kSlabThreadsNarrow, true>;
}

// The limits hold for the current device and context: the attribute that lets a
// kernel have more than 48 KB belongs to them, so each is given it.
SlabLimits slab_limits() {
    static PerContext<SlabLimits> kept;
    return of_current_context(kept, [] {
        SlabLimits l;
        int dev = 0, optin = 0, coop = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&l.sms, cudaDevAttrMultiProcessorCount, dev);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
        const int smem = (optin - 1024) / 16 * 16;  // room for the kernels' own variables
        bool ok = coop && smem > 0 && l.sms > 0;
        for (int i = 0; i < 4; ++i)
            ok = ok && cudaFuncSetAttribute(reinterpret_cast<const void*>(slab_fn(i & 1, i >> 1)),
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess;
        l.smem = ok ? smem : 0;
        for (const void* fn : {reinterpret_cast<const void*>(&k_batch_slabs<false>), reinterpret_cast<const void*>(&k_batch_slabs<true>)})
            ok = ok && cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess;
        if (ok) l.batch_smem = smem;
        if (l.batch_smem) {
            cudaLaunchConfig_t lc = {};
            lc.gridDim = dim3((unsigned)(l.sms / 8 * 8));
            lc.blockDim = dim3(batch_slab_threads<false>());
            lc.dynamicSmemBytes = (size_t)smem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 8;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            lc.attrs = attr;
            lc.numAttrs = 1;
            // (fewer than an eighth of the SMs: a cluster lies within a group of them)
            if (cudaOccupancyMaxActiveClusters(&l.clusters, k_batch_slabs<false>, &lc) != cudaSuccess) l.clusters = 0;
        }
        cudaGetLastError();  // a refused attribute leaves the kernels unused, not an error
        return l;
    });
}

}  // namespace

// test hook: multi-step launches are refused as if the device could not hold them
static std::atomic<bool> g_refuse_slabs{false};

fs3d_status set_slab_stall(uint32_t which) {
    g_refuse_slabs.store(which == kStallRefuse);
    if (which == kStallRefuse) which = kStallNone;
    FS3D_CUDA(cudaMemcpyToSymbol(g_slab_stall, &which, sizeof(which)));
    return FS3D_OK;
}

void batch_slabs_limits(ResidentLimits* out) {
    const SlabLimits l = slab_limits();
    out->cluster = l.batch_smem;
    out->clusters = l.clusters;
}

bool batch_slabs_fit(const ResidentLimits& l, int X, int Y, int Z, int CS) {
    const int smem = l.cluster;
    const int64_t nw = plane_nw(X), NP = (Z + 1) / 2, mp = (NP + CS - 1) / CS;
    return X <= kPlaneMaxX && NP >= CS && Y * nw <= kBatchSlabEdgeWords && 2 * mp * Y * nw * 16 + (2 * mp + 1) * Y <= smem;
}

size_t batch_slab_edge_bytes(int CS) {
    return (size_t)(sm_count_public() / CS) * (size_t)(CS - 1) * kBatchSlabEdgeWords * 32;
}

fs3d_status launch_batch_slabs(int cls, int CS, const PlaneWorld* worlds, const int* order, const int* meta, int* counter,
                               int* err, void* edges, cudaStream_t st, unsigned long long* processed_cells, bool by_place) {
    FS3D_CUDA(cudaMemsetAsync(counter, 0, sizeof(int), st));
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)(sm_count_public() / CS * CS));
    lc.blockDim = dim3((unsigned)(by_place ? batch_slab_threads<true>() : batch_slab_threads<false>()));
    lc.dynamicSmemBytes = (size_t)slab_limits().batch_smem;
    lc.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    // these worlds take the longest: their CTAs are placed before the other classes'
    static const int greatest = [] {
        int least = 0, g = 0;
        if (cudaDeviceGetStreamPriorityRange(&least, &g) != cudaSuccess) g = 0;
        return g;
    }();
    attr[1].id = cudaLaunchAttributePriority;
    attr[1].val.priority = greatest;
    lc.attrs = attr;
    lc.numAttrs = 2;
    const auto fn = by_place ? &k_batch_slabs<true> : &k_batch_slabs<false>;
    const cudaError_t e = cudaLaunchKernelEx(&lc, fn, worlds, order, meta, cls, CS, counter, err, processed_cells,
                                             static_cast<unsigned long long*>(edges));
    if (e != cudaSuccess) return cuda_fail(e, "cluster segment launch");
    note_launch();
    return FS3D_OK;
}

// The cut: along z or y, and how many slabs.  A slab's work is its row-pairs'
// lanes in a step.  Along z the moving layers of a settled world (a water
// surface lies in a few y layers) spread over all the slabs, along y they are
// one slab's work (300^3 settled: 6.2 us a step against 12), so a y-cut has to
// be half as large again to be taken.  As few slabs as leave every row-pair a
// lane group of kSlabThreadsNarrow threads (96x80x112: 28 slabs 2.41 us, 56
// slabs 2.68), or else as many as there are SMs.  Slabs of more than
// kSlabMaxLanes lanes are left to the per-step kernel, which spreads a step's
// work over all SMs evenly: 256^3 (516 lanes) 5.0 us a step here while
// everything falls and 3.8 settled, 7.1 and 8.2 there; 300^3 (1208) 8.2 and
// 6.2, 8.6 and 8.3 there; 400x300x350 (2416) 11.7 and 16, 10.5 and 8.3 there.
bool slab_plan(int X, int Y, int Z, SlabPlan* out) {
    constexpr double kSlabMaxLanes = 1280.0;
    const SlabLimits l = slab_limits();
    if (!l.smem || X > kPlaneMaxX) return false;
    const int64_t nw = plane_nw(X), G = (int64_t)1 << plane_lg((int)nw);
    double best = kSlabMaxLanes;
    bool found = false;
    for (int zs = 1; zs >= 0; --zs) {
        const int64_t NS = zs ? Z : Y, NO = zs ? Y : Z, NP = (NS + 1) / 2, pair = ((NO + 2) / 2) * G;
        // most layer pairs of a slab; the last slab has one more in odd steps
        const int64_t narrow = kSlabThreadsNarrow / pair - 1;
        const int64_t mp = std::max<int64_t>((NP + l.sms - 1) / l.sms, narrow);
        const int C = (int)((NP + mp - 1) / mp);
        const int64_t smem = 2 * mp * NO * nw * 16 + (2 * mp + 1) * NO;
        const int64_t lanes = (mp + 1) * pair;
        // (narrow slabs cost the same whatever their size)
        const double cost = std::max<double>((double)(mp * pair), kSlabThreadsNarrow) * (zs ? 1.0 : 1.5);
        if (smem > l.smem || cost >= best) continue;
        found = true;
        best = cost;
        out->zs = zs;
        out->ctas = C;
        out->threads = (int)std::min<int64_t>((lanes + 31) / 32 * 32, kSlabThreadsWide);
        out->smem = (int)((smem + 15) / 16 * 16);
        out->scratch = kSlabEdgeOff + (size_t)(C - 1) * (size_t)NO * (size_t)nw * 32;
    }
    return found;
}

bool prefer_slabs(int X, int Y, int Z, int n_steps, SlabPlan* out) {
    return n_steps >= 4 && slab_plan(X, Y, Z, out);
}

fs3d_status launch_plane_slabs(const PlaneWorld& w, const SlabPlan& plan, uint8_t* rflags, void* scratch, int* err, int* own,
                               cudaStream_t st, int* taken) {
    *taken = 0;
    // steps are counted in 31 bits of a tag; a launch is kept to a fraction of a second
    constexpr int kMaxSteps = 1 << 15;
    PlaneWorld d = w;
    for (int done = 0; done < w.steps; done += d.steps) {
        d.t = w.t + (uint64_t)done;
        d.steps = std::min(kMaxSteps, w.steps - done);
        FS3D_CUDA(cudaMemsetAsync(scratch, 0, plan.scratch, st));
        SlabState* state = static_cast<SlabState*>(scratch);
        unsigned long long* edge = reinterpret_cast<unsigned long long*>(static_cast<char*>(scratch) + kSlabEdgeOff);
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3((unsigned)plan.ctas);
        lc.blockDim = dim3((unsigned)plan.threads);
        lc.dynamicSmemBytes = (size_t)plan.smem;
        lc.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        lc.attrs = attr;
        lc.numAttrs = 1;
        const SlabFn fn = slab_fn(plan.zs != 0, plan.threads > kSlabThreadsNarrow);
        const cudaError_t e = g_refuse_slabs.load() ? cudaErrorCooperativeLaunchTooLarge
                                                    : cudaLaunchKernelEx(&lc, fn, d, rflags, state, edge, err, own);
        // refused for what the device has free for this process (its SMs may be
        // shared out), before anything ran: the caller takes the rest of the
        // steps a launch at a time
        if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorNotSupported) {
            cudaGetLastError();
            return FS3D_OK;
        }
        if (e != cudaSuccess) return cuda_fail(e, "slab steps launch");
        note_launch();
        *taken = done + d.steps;
    }
    return FS3D_OK;
}

}  // namespace fs3d
