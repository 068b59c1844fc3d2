// Headless render kernels.  Built with --fmad=false: every float expression is
// a sequence of single IEEE operations (+ - * /, sqrtf correctly rounded), in
// the same order as the CPU restatement, so frames are reproducible bit for
// bit on the host.
//
//  * k_render_sdf: shaders/fs_raymarch.frag:10-81 as a CUDA kernel, one thread
//    per pixel: 64-step sphere tracing of a radius-0.5 sphere at the origin,
//    hit at d < 0.001, bail at t > 1000, central-difference normal (h=0.001),
//    diffuse = max(0.05, dot(n, normalize(p - light))) (the shader's vector
//    points away from the light), red surface, black miss, alpha 1.
//    Ray set-up follows fs_raymarch.vert:30-37 (origin = camPos, aspect =
//    aspect.x) and the fullscreen quad of renderer.cpp:1253-1267.
//  * k_render_dda: Amanatides & Woo (1987) traversal of the world grid with
//    the same ray generation and shading conventions; the face normal of the
//    entered voxel is shaded with the material's colour.
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "fs3d_common.h"
#include "planes.h"

namespace fs3d {

struct CamDev {
    float o[3], f[3], r[3], u[3];
    float tan_half_fov, aspect;
    float light[3];
};

__device__ __forceinline__ float dot3(const float* a, const float* b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a[0], b[0]), __fmul_rn(a[1], b[1])), __fmul_rn(a[2], b[2]));
}
__device__ __forceinline__ void normalize3(float* v) {
    const float len = __fsqrt_rn(dot3(v, v));
    v[0] = __fdiv_rn(v[0], len);
    v[1] = __fdiv_rn(v[1], len);
    v[2] = __fdiv_rn(v[2], len);
}
__device__ __forceinline__ void pixel_uv2(int px, int py, int W, int H, float& ux, float& uy) {
    const float u = __fsub_rn(1.0f, __fdiv_rn(__fadd_rn((float)px, 0.5f), (float)W));
    const float v = __fdiv_rn(__fadd_rn((float)py, 0.5f), (float)H);
    ux = __fsub_rn(__fmul_rn(u, 2.0f), 1.0f);
    uy = __fsub_rn(__fmul_rn(v, 2.0f), 1.0f);
}
// Whether the ray o + t d (d of unit length) stays clear of the ball of radius r
// about the origin, by far more than the hit distance (0.001) and the march's
// rounding (relative to |o|) can bridge: marching it would never hit.  False
// for NaN.
__device__ __forceinline__ bool passes_by(const float* o, const float* d, float r) {
    const float along = o[0] * d[0] + o[1] * d[1] + o[2] * d[2];
    const float x = o[0] - along * d[0], y = o[1] - along * d[1], z = o[2] - along * d[2];
    const float far = r + 0.01f + 1e-5f * (fabsf(o[0]) + fabsf(o[1]) + fabsf(o[2]));
    return x * x + y * y + z * z > far * far;
}
__device__ __forceinline__ float sdf_world(float x, float y, float z) {
    return __fsub_rn(__fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z))), 0.5f);
}

// Most of the frame's rays miss the sphere by far (29 us a 1920x1080 frame
// marching all of them, 64 steps or until t > 1000).
__global__ void k_render_sdf(CamDev cam, int W, int H, float4* __restrict__ out) {
    const int px = blockIdx.x * blockDim.x + threadIdx.x;
    const int py = blockIdx.y * blockDim.y + threadIdx.y;
    if (px >= W || py >= H) return;
    float ux, uy;
    pixel_uv2(px, py, W, H, ux, uy);
    uy = __fmul_rn(uy, __fdiv_rn(1.0f, cam.aspect));
    float d[3] = {ux, uy, 1.0f};
    normalize3(d);
    float col = 0.0f, t = 0.0f;
    const int steps = passes_by(cam.o, d, 0.5f) ? 0 : 64;
    for (int it = 0; it < steps; ++it) {
        const float p[3] = {__fadd_rn(cam.o[0], __fmul_rn(t, d[0])), __fadd_rn(cam.o[1], __fmul_rn(t, d[1])),
                            __fadd_rn(cam.o[2], __fmul_rn(t, d[2]))};
        const float dist = sdf_world(p[0], p[1], p[2]);
        if (dist < 0.001f) {
            const float h = 0.001f;
            float n[3] = {
                __fsub_rn(sdf_world(__fadd_rn(p[0], h), p[1], p[2]), sdf_world(__fsub_rn(p[0], h), p[1], p[2])),
                __fsub_rn(sdf_world(p[0], __fadd_rn(p[1], h), p[2]), sdf_world(p[0], __fsub_rn(p[1], h), p[2])),
                __fsub_rn(sdf_world(p[0], p[1], __fadd_rn(p[2], h)), sdf_world(p[0], p[1], __fsub_rn(p[2], h)))};
            normalize3(n);
            float l[3] = {__fsub_rn(p[0], cam.light[0]), __fsub_rn(p[1], cam.light[1]), __fsub_rn(p[2], cam.light[2])};
            normalize3(l);
            col = fmaxf(0.05f, dot3(n, l));
            break;
        } else if (t > 1000.0f) {
            break;
        }
        t = __fadd_rn(t, dist);
    }
    out[(size_t)py * W + px] = make_float4(col, 0.0f, 0.0f, 1.0f);
}

__constant__ float c_palette[5][3] = {
    {0.0f, 0.0f, 0.0f}, {0.50f, 0.50f, 0.52f}, {0.86f, 0.74f, 0.46f}, {0.20f, 0.42f, 0.90f}, {0.65f, 0.35f, 0.30f}};

// Material lookups.  The walk keeps the index of its row (y, z) and moves it by
// row_y / row_z as it steps; I is the index type (32 bits wherever they reach).
template <class I>
struct BytesGrid {
    using Index = I;
    const uint8_t* g;
    int X, Y, Z;
    __device__ __forceinline__ I row_z() const { return (I)X; }
    __device__ __forceinline__ I row_y() const { return (I)X * (I)Z; }
    // a cell fetched, to be looked at later
    struct Cell {
        uint32_t v;
    };
    __device__ __forceinline__ Cell fetch(I row, int x) const { return Cell{g[row + (I)x]}; }
    static __device__ __forceinline__ bool filled(const Cell& c) { return c.v != 0u; }
    __device__ __forceinline__ uint32_t material(const Cell& c, I, int) const { return c.v; }
};

// bit planes (A,B) + optional static byte overlay for solids
template <class I>
struct PlaneGrid {
    using Index = I;
    const uint32_t* p;  // rows of nw x {A even, A odd, B even, B odd}
    const uint8_t* statics;  // nullable: every solid is stone
    int X, Y, Z, nw;
    __device__ __forceinline__ I row_z() const { return (I)(4 * nw); }
    __device__ __forceinline__ I row_y() const { return (I)(4 * nw) * (I)Z; }
    struct Cell {
        uint32_t a, b;
    };
    __device__ __forceinline__ Cell fetch(I row, int x) const {
        const uint32_t* w = p + (row + (I)(((x >> 6) << 2) + (x & 1)));
        const int bit = (x >> 1) & 31;
        return Cell{w[0] >> bit, w[2] >> bit};
    }
    static __device__ __forceinline__ bool filled(const Cell& c) { return ((c.a | c.b) & 1u) != 0u; }
    __device__ __forceinline__ uint32_t material(const Cell& c, I row, int x) const {
        if (c.a & 1u) return 2u + (c.b & 1u);
        return statics ? statics[(int64_t)(row / (I)(4 * nw)) * X + x] : 1u;
    }
};

// Occupancy of 8x8x8 bricks, built per frame: a byte holds eight bricks along
// x (bit bx & 7 of byte (bx >> 3) + BXB*(bz + BZ*by)), set when the brick holds
// a non-empty cell, and one byte per 64^3 super-brick (its 8 x 8 brick bytes)
// says what the walk may cross from there: 0 a brick at a time, 1 the empty
// super-brick, 2 the empty aligned 256^3 cells around it.  The walk crosses
// empty regions at once and visits every other cell, so its hit is exactly the
// flat walk's.  (1024^3 dunes, settled: a ray crossed 13.3 super-bricks and 4.5
// bricks and visited 5.2 cells in the mean.)
struct BrickMap {
    const uint8_t* bits;
    int BXB, BZ;
    const uint8_t* super;
    int SBZ;
};

// One CTA per super-brick (blockIdx: its x, z, y): 64 brick rows of 8 bricks,
// eight lanes each.  SRC(y, z, xb) = bit c set when the 8 cells of chunk 8 xb
// + c of row (y, z) are not all empty; whole bytes are stored, so nothing has
// to be cleared beforehand.  The last CTA of a 256^3 group to finish (the
// group's counter, which wraps to 0 again by itself) raises its super-bricks
// from 1 to 2 when all of them are empty.
template <class SRC>
__device__ __forceinline__ void build_occupancy(const SRC& src, int Y, int Z, uint8_t* bits, int BXB, uint8_t* super,
                                                unsigned* group) {
    const int BY = (Y + 7) >> 3, BZ = (Z + 7) >> 3;
    const int br = threadIdx.x >> 3, l = threadIdx.x & 7;
    const int by = 8 * blockIdx.z + (br >> 3), bz = 8 * blockIdx.y + (br & 7), xb = blockIdx.x;
    uint32_t m = 0;
    if (by < BY && bz < BZ) m = src(by, bz, xb, l);
    m |= __shfl_xor_sync(0xFFFFFFFFu, m, 1);
    m |= __shfl_xor_sync(0xFFFFFFFFu, m, 2);
    m |= __shfl_xor_sync(0xFFFFFFFFu, m, 4);
    if (l == 0 && by < BY && bz < BZ) bits[xb + (int64_t)BXB * (bz + (int64_t)BZ * by)] = (uint8_t)m;
    const int any = __syncthreads_or(m != 0u);
    auto at = [&](int x, int z, int y) { return super + (x + (int64_t)gridDim.x * (z + (int64_t)gridDim.y * y)); };
    if (threadIdx.x >= 32) return;
    // the group's super-bricks (fewer at the world's far faces)
    const int gx = blockIdx.x >> 2, gz = blockIdx.y >> 2, gy = blockIdx.z >> 2;
    const int nx = min(4, (int)gridDim.x - 4 * gx), nz = min(4, (int)gridDim.y - 4 * gz), ny = min(4, (int)gridDim.z - 4 * gy);
    bool last = false;
    if (threadIdx.x == 0) {
        *at(blockIdx.x, blockIdx.y, blockIdx.z) = any ? 0 : 1;
        if (nx * nz * ny > 1) __threadfence();
    }
    if (nx * nz * ny == 1) return;
    if (threadIdx.x == 0) {
        const unsigned n = (unsigned)(nx * nz * ny);
        const int64_t g = gx + (int64_t)((gridDim.x + 3) >> 2) * (gz + (int64_t)((gridDim.y + 3) >> 2) * gy);
        last = atomicInc(group + g, n - 1u) == n - 1u;
        __threadfence();
    }
    if (!__shfl_sync(0xFFFFFFFFu, last, 0)) return;
    bool empty = true;
    for (int i = threadIdx.x; i < nx * nz * ny; i += 32)
        empty = empty && *(volatile uint8_t*)at(4 * gx + i % nx, 4 * gz + i / nx % nz, 4 * gy + i / (nx * nz)) != 0;
    if (__all_sync(0xFFFFFFFFu, empty))
        for (int i = threadIdx.x; i < nx * nz * ny; i += 32) *at(4 * gx + i % nx, 4 * gz + i / nx % nz, 4 * gy + i / (nx * nz)) = 2;
}

// from the planes: lane l reads the rows of layer y = 8 by + l
__global__ void __launch_bounds__(512) k_occupancy_planes(const uint4* rows, int X, int Y, int Z, int nw,
                                                          uint8_t* bits, uint8_t* super, unsigned* group) {
    chain_wait();
    build_occupancy(
        [&](int by, int bz, int xb, int l) {
            const int y = 8 * by + l;
            uint32_t e = 0, o = 0;
            if (y < Y)
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (8 * bz + k < Z) {
                        const uint4 q = rows[((int64_t)y * Z + 8 * bz + k) * nw + xb];
                        e |= q.x | q.z;
                        o |= q.y | q.w;
                    }
            // (cells past X are solid in the planes)
            const int left = X - 64 * xb;
            if (left < 64) {
                e &= (1u << ((left + 1) >> 1)) - 1u;
                o &= (1u << (left >> 1)) - 1u;
            }
            // nibble c -> bit c: bits 0, 4, 8, 12 of a half land on 9 .. 12
            e |= o;
            e |= e >> 2;
            e |= e >> 1;
            e &= 0x11111111u;
            return ((e * 0x249u) >> 9 & 0xFu) | ((((e >> 16) * 0x249u) >> 9 & 0xFu) << 4);
        },
        Y, Z, bits, nw, super, group);
}

// from exact counts of non-empty cells per brick: lane l reads brick 8 xb + l
__global__ void __launch_bounds__(512) k_occupancy_counts(const int* counts, int X, int Y, int Z,
                                                          uint8_t* bits, uint8_t* super, unsigned* group) {
    chain_wait();
    const int BX = (X + 7) >> 3, BZ = (Z + 7) >> 3;
    build_occupancy(
        [&](int by, int bz, int xb, int l) {
            const int bx = 8 * xb + l;
            return bx < BX && counts[bx + (int64_t)BX * (bz + (int64_t)BZ * by)] > 0 ? 1u << l : 0u;
        },
        Y, Z, bits, (X + 63) >> 6, super, group);
}

// from bytes: lane l reads the rows of layer y = 8 by + l
__global__ void __launch_bounds__(512) k_occupancy_bytes(const uint8_t* g, int X, int Y, int Z,
                                                         uint8_t* bits, uint8_t* super, unsigned* group) {
    chain_wait();
    build_occupancy(
        [&](int by, int bz, int xb, int l) {
            const int y = 8 * by + l, n = min(64, X - 64 * xb);
            uint32_t m = 0;
            if (y < Y)
                for (int k = 0; k < 8 && 8 * bz + k < Z; ++k) {
                    const uint8_t* row = g + ((int64_t)y * Z + 8 * bz + k) * X + 64 * xb;
                    if (n == 64 && (reinterpret_cast<uintptr_t>(row) & 15u) == 0) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const uint4 v = reinterpret_cast<const uint4*>(row)[u];
                            m |= ((v.x | v.y) ? 1u : 0u) << (2 * u) | ((v.z | v.w) ? 2u : 0u) << (2 * u);
                        }
                    } else {
                        for (int x = 0; x < n; ++x)
                            if (row[x]) m |= 1u << (x >> 3);
                    }
                }
            return m;
        },
        Y, Z, bits, (X + 63) >> 6, super, group);
}

// Counts of non-empty cells per brick, from the planes (one thread per row word)
__global__ void k_brickcount_planes(const uint4* __restrict__ rows, int X, int Y, int Z, int nw, int* counts, int BX,
                                    int BZ) {
    const int64_t n = (int64_t)Y * Z * nw;
    for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < n; u += (int64_t)gridDim.x * blockDim.x) {
        const int g = (int)(u % nw);
        const int64_t r = u / nw;
        const int y = (int)(r / Z), z = (int)(r % Z);
        const uint4 q = rows[u];
        const uint32_t e = q.x | q.z, o = q.y | q.w;
        if (!(e | o)) continue;
        const int64_t base = (int64_t)BX * ((z >> 3) + (int64_t)BZ * (y >> 3));
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int cnt = __popc((e >> (4 * c)) & 0xFu) + __popc((o >> (4 * c)) & 0xFu);
            if (cnt && 8 * g + c < BX) atomicAdd(counts + base + 8 * g + c, cnt);
        }
    }
}

// Crossing an empty region (an 8^3 brick or a 64^3 super-brick) at once, with
// the cell-by-cell walk's exact result.  The walk steps, at every cell, the
// axis whose next boundary key is smallest; on equal keys z goes before y
// before x.  Axis a's key after n steps is fma(n, e_a, b_a), a non-decreasing
// function of n, so the walk's steps are the merge of the three axes' key
// sequences in that order.  It leaves the region at the first of the three
// axes' leaving steps (axis a's key at step n_a + k_a - 1, k_a the cells to
// the region's face); every step that comes before it in the merge is taken
// (for each other axis a prefix of its keys, found from an estimate and
// checked key by key), and nothing in between can hit, since the region is
// empty.  The state after the crossing (cells, steps, keys, last axis, t) is
// therefore bit for bit the walk's.
__device__ __forceinline__ bool key_before(float p, int pa, float q, int pb) {
    return p < q || (p == q && pa > pb);  // axis index as the tie priority: z (2) > y (1) > x (0)
}

// Small whole numbers between int and float by the float's own bits: the
// conversion instructions run at an eighth of the others' rate.  Step counts
// are kept as floats (whole, below 2^24, so exact).
__device__ __forceinline__ float small_minus1(int k) { return __fsub_rn(__int_as_float(0x4B000000 + k), 8388609.0f); }
__device__ __forceinline__ int small_int(float x) { return __float_as_int(__fadd_rn(x, 8388608.0f)) - 0x4B000000; }

// Takes the steps of one axis at a crossing: of the axis that leaves the region
// (ax) the k = k1 + 1 steps to its face, of another (steps n.., at most k1 of
// them) those whose keys come before the leaving step's key ke.  r: about 1 / e,
// for the estimate of the first step not taken, which its key and the one
// before it confirm or correct.  All three axes run the same instructions, and
// so does a cell's step below: branches by axis made the lanes of a warp wait
// for each other (1024^3 at 1920x1080, young and settled 614 and 246 us a
// frame, now 514 and 199; 395x179x418 at 436x245 483 and 92, now 388 and 74).
__device__ __forceinline__ void take_steps(int& v, int s, float& n, float b, float e, float r, float& m, float k1, int pa,
                                           float ke, int ax) {
    const bool leaves = pa == ax;
    const float top = __fadd_rn(n, k1);
    float j = __fsub_rn(__fadd_rn(__fadd_rn(__fmul_rn(__fsub_rn(ke, b), r), 0.5f), 12582912.0f), 12582912.0f);
    j = fminf(fmaxf(j, n), top);
    if (leaves) j = __fadd_rn(top, 1.0f);
    float at = __fmaf_rn(j, e, b);
    if (!leaves && s &&
        ((j < top && key_before(at, pa, ke, ax)) ||
         (j > n && !key_before(__fmaf_rn(__fsub_rn(j, 1.0f), e, b), pa, ke, ax)))) {
        while (j < top && key_before(__fmaf_rn(j, e, b), pa, ke, ax)) j = __fadd_rn(j, 1.0f);
        while (j > n && !key_before(__fmaf_rn(__fsub_rn(j, 1.0f), e, b), pa, ke, ax)) j = __fsub_rn(j, 1.0f);
        at = __fmaf_rn(j, e, b);
    }
    v += s * small_int(__fsub_rn(j, n));
    n = j;
    m = s ? at : INFINITY;
}

// A warp takes 8 x 4 pixels (its rays stay together longer than a 16 x 2
// strip's), a CTA 8 x 8, so that few finished warps wait for a long ray.  Two
// loops, one crossing empty regions and one walking the cells of an occupied
// brick, so that the lanes of a warp run the same one of the two.
template <class G>
__global__ void __launch_bounds__(64) k_render_dda(G grid, BrickMap bm, CamDev cam, int W, int H, int row0,
                                                   float4* __restrict__ out) {
    chain_wait();
    const int px = blockIdx.x * 8 + (threadIdx.x & 7);
    const int py = row0 + blockIdx.y * 8 + (threadIdx.x >> 3);
    if (px >= W || py >= H) return;
    const int NX = grid.X, NY = grid.Y, NZ = grid.Z;
    float ux, uy;
    pixel_uv2(px, py, W, H, ux, uy);
    const float sx = __fmul_rn(__fmul_rn(ux, cam.tan_half_fov), cam.aspect);
    const float sy = __fmul_rn(uy, cam.tan_half_fov);
    float d[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) d[a] = __fadd_rn(__fadd_rn(cam.f[a], __fmul_rn(cam.r[a], sx)), __fmul_rn(cam.u[a], sy));
    normalize3(d);
    float4 res = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
    // slab entry: per axis in the same order as the CPU restatement
    float inv[3];
    float tmin = 0.0f, tmax = INFINITY;
    int entry_axis = -1;
    bool miss = false;
    const int N[3] = {NX, NY, NZ};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (d[a] == 0.0f) {
            inv[a] = INFINITY;
            if (cam.o[a] < 0.0f || cam.o[a] >= (float)N[a]) miss = true;
            continue;
        }
        inv[a] = __fdiv_rn(1.0f, d[a]);
        float t0 = __fmul_rn(__fsub_rn(0.0f, cam.o[a]), inv[a]);
        float t1 = __fmul_rn(__fsub_rn((float)N[a], cam.o[a]), inv[a]);
        if (t0 > t1) {
            const float tmp = t0;
            t0 = t1;
            t1 = tmp;
        }
        if (t0 > tmin) {
            tmin = t0;
            entry_axis = a;
        }
        if (t1 < tmax) tmax = t1;
    }
    if (!miss && tmin <= tmax) {
        // per-axis state as scalars (no local-memory arrays): cell v, step s, steps
        // taken n, first boundary t b, t per cell e; the next boundary key is
        // m = fma(n, e, b), one rounding, as in the CPU walk
        int v0, v1, v2, s0, s1, s2;
        float n0 = 0.0f, n1 = 0.0f, n2 = 0.0f;
        float b0, b1, b2, e0, e1, e2;
        auto setup = [&](int a, int& v, int& st, float& bt, float& td) {
            const float p = __fadd_rn(cam.o[a], __fmul_rn(d[a], tmin));
            int c = (int)floorf(p);
            c = c < 0 ? 0 : (c > N[a] - 1 ? N[a] - 1 : c);
            v = c;
            st = d[a] > 0.0f ? 1 : (d[a] < 0.0f ? -1 : 0);
            if (d[a] == 0.0f) {
                bt = INFINITY;
                td = INFINITY;
            } else {
                bt = __fmul_rn(__fsub_rn((float)(c + (st > 0 ? 1 : 0)), cam.o[a]), inv[a]);
                td = fabsf(inv[a]);
            }
        };
        setup(0, v0, s0, b0, e0);
        setup(1, v1, s1, b1, e1);
        setup(2, v2, s2, b2, e2);
        float m0 = b0, m1 = b1, m2 = b2;
        int last = entry_axis;
        float tcur = tmin;
        using I = typename G::Index;
        const I ry = grid.row_y(), rz = grid.row_z();
        // f: all ones for a falling axis; (v ^ ~f) + c: the cells from v to
        // the grid's face ahead, N - v or v + 1
        const int f0 = s0 >> 31, f1 = s1 >> 31, f2 = s2 >> 31;
        const int c0 = f0 ? 1 : NX + 1, c1 = f1 ? 1 : NY + 1, c2 = f2 ? 1 : NZ + 1;
        const float r0 = fabsf(d[0]), r1 = fabsf(d[1]), r2 = fabsf(d[2]);
        int left = NX + NY + NZ + 3;  // steps and crossings: more than any walk takes
        for (;;) {
            // cross empty regions until an occupied brick
            int R = 0;
            while (left > 0) {
                // (both levels fetched at once: the asm keeps the first load from
                // sinking below the branch on the second, 64^3 at 320x180 8.1 us
                // a pass instead of 7.85)
                uint32_t big = bm.super[(v0 >> 6) + bm.BXB * ((v2 >> 6) + bm.SBZ * (v1 >> 6))];
                uint32_t small = bm.bits[(v0 >> 6) + bm.BXB * ((v2 >> 3) + bm.BZ * (v1 >> 3))];
                asm volatile("" : "+r"(big), "+r"(small));
                if ((small >> ((v0 >> 3) & 7)) & 1u) break;
                R = big == 0u ? 8 : (big == 1u ? 64 : 256);
                --left;
                // take every step up to and including the first that leaves the
                // region, with the walk's exact keys (see key_before).  Cells axis
                // a takes to leave it: to the region's face, or the grid's if that
                // comes first (g: cells to the grid's)
                const int g0 = (v0 ^ ~f0) + c0, g1 = (v1 ^ ~f1) + c1, g2 = (v2 ^ ~f2) + c2;
                const int k0 = min(R - ((v0 ^ f0) & (R - 1)), g0), k1 = min(R - ((v1 ^ f1) & (R - 1)), g1),
                          k2 = min(R - ((v2 ^ f2) & (R - 1)), g2);
                const float l0 = small_minus1(k0), l1 = small_minus1(k1), l2 = small_minus1(k2);
                // each axis's key at its leaving step
                const float x0 = s0 ? __fmaf_rn(__fadd_rn(n0, l0), e0, b0) : INFINITY;
                const float x1 = s1 ? __fmaf_rn(__fadd_rn(n1, l1), e1, b1) : INFINITY;
                const float x2 = s2 ? __fmaf_rn(__fadd_rn(n2, l2), e2, b2) : INFINITY;
                int ax = 0;
                float ke = x0;
                if (key_before(x1, 1, ke, ax)) { ax = 1; ke = x1; }
                if (key_before(x2, 2, ke, ax)) { ax = 2; ke = x2; }
                // its k-th step, and the other axes' steps that come before it (a prefix of their keys)
                take_steps(v0, s0, n0, b0, e0, r0, m0, l0, 0, ke, ax);
                take_steps(v1, s1, n1, b1, e1, r1, m1, l1, 1, ke, ax);
                take_steps(v2, s2, n2, b2, e2, r2, m2, l2, 2, ke, ax);
                tcur = ke;
                last = ax;
                if (ax == 0 ? k0 == g0 : (ax == 1 ? k1 == g1 : k2 == g2)) left = 0;
            }
            if (left <= 0) break;
            // walk the brick's cells until one is not empty or the walk leaves it
            // (a cell's fetch runs while the next one is found)
            const I dy = s1 > 0 ? ry : (s1 < 0 ? (I)0 - ry : (I)0), dz = s2 > 0 ? rz : (s2 < 0 ? (I)0 - rz : (I)0);
            I row = (I)v1 * ry + (I)v2 * rz;
            uint32_t m = 0;
            bool inside = true;
            while (inside && left > 0) {
                --left;
                const typename G::Cell cell = grid.fetch(row, v0);
                const I at_row = row;
                const int at_x = v0, at_last = last;
                const float at_t = tcur;
                // next cell: the axis whose boundary key comes first (equal keys: z, then y, then x)
                const bool a0 = m0 < m1 && m0 < m2, a1 = !(m0 < m1) && m1 < m2, a2 = !a0 && !a1;
                tcur = a0 ? m0 : (a1 ? m1 : m2);
                last = a0 ? 0 : (a1 ? 1 : 2);
                const int u0 = v0 + (a0 ? s0 : 0), u1 = v1 + (a1 ? s1 : 0), u2 = v2 + (a2 ? s2 : 0);
                inside = (((u0 ^ v0) | (u1 ^ v1) | (u2 ^ v2)) & ~7) == 0;
                if ((unsigned)u0 >= (unsigned)NX || (unsigned)u1 >= (unsigned)NY || (unsigned)u2 >= (unsigned)NZ) left = 0;
                v0 = u0;
                v1 = u1;
                v2 = u2;
                row += a1 ? dy : (a2 ? dz : (I)0);
                n0 = __fadd_rn(n0, a0 ? 1.0f : 0.0f);
                n1 = __fadd_rn(n1, a1 ? 1.0f : 0.0f);
                n2 = __fadd_rn(n2, a2 ? 1.0f : 0.0f);
                m0 = a0 ? __fmaf_rn(n0, e0, b0) : m0;
                m1 = a1 ? __fmaf_rn(n1, e1, b1) : m1;
                m2 = a2 ? __fmaf_rn(n2, e2, b2) : m2;
                if (G::filled(cell)) {
                    m = grid.material(cell, at_row, at_x);
                    last = at_last;
                    tcur = at_t;
                    break;
                }
            }
            if (m != 0u) {
                float n[3] = {0.0f, 0.0f, 0.0f};
                if (last == 0) n[0] = s0 > 0 ? -1.0f : 1.0f;
                if (last == 1) n[1] = s1 > 0 ? -1.0f : 1.0f;
                if (last == 2) n[2] = s2 > 0 ? -1.0f : 1.0f;
                float l[3];
#pragma unroll
                for (int a = 0; a < 3; ++a)
                    l[a] = __fsub_rn(__fadd_rn(cam.o[a], __fmul_rn(d[a], tcur)), cam.light[a]);
                normalize3(l);
                const float diff = fmaxf(0.05f, dot3(n, l));
                const int ci = m < 4u ? (int)m : 4;
                res = make_float4(__fmul_rn(c_palette[ci][0], diff), __fmul_rn(c_palette[ci][1], diff),
                                  __fmul_rn(c_palette[ci][2], diff), 1.0f);
                break;
            }
            if (left <= 0) break;
        }
    }
    out[(size_t)py * W + px] = res;
}

static CamDev to_dev(const fs3d_camera* c) {
    CamDev d;
    for (int a = 0; a < 3; ++a) {
        d.o[a] = c->origin[a];
        d.f[a] = c->forward[a];
        d.r[a] = c->right[a];
        d.u[a] = c->up[a];
        d.light[a] = c->light_pos[a];
    }
    d.tan_half_fov = c->tan_half_fov;
    d.aspect = c->aspect;
    return d;
}

fs3d_status launch_render_sdf(const fs3d_camera* cam, int W, int H, float* rgba_dev, cudaStream_t st) {
    const dim3 blk(16, 16), grd((W + 15) / 16, (H + 15) / 16);
    k_render_sdf<<<grd, blk, 0, st>>>(to_dev(cam), W, H, reinterpret_cast<float4*>(rgba_dev));
    FS3D_CHECK_LAUNCH("render sdf launch");
    return FS3D_OK;
}

static int map_grid(int64_t n) {
    const int64_t need = (n + 255) / 256, cap = (int64_t)sm_count_public() * 8;
    return (int)(need < 1 ? 1 : (need < cap ? need : cap));
}

static int64_t brick_bytes(int X, int Y, int Z) {
    return (int64_t)((X + 63) / 64) * ((Y + 7) / 8) * ((Z + 7) / 8);
}

static size_t super_bytes(int X, int Y, int Z) {
    return (size_t)((X + 63) / 64) * ((Y + 63) / 64) * ((Z + 63) / 64);
}

static BrickMap brick_map(uint8_t* bits, int X, int Y, int Z) {
    return BrickMap{bits, (X + 63) / 64, (Z + 7) / 8, bits + brick_bytes(X, Y, Z), (Z + 63) / 64};
}

// the 256^3 groups' counters, after both levels
static size_t group_offset(int X, int Y, int Z) { return ((size_t)brick_bytes(X, Y, Z) + super_bytes(X, Y, Z) + 3) & ~(size_t)3; }
static unsigned* group_counters(uint8_t* bits, int X, int Y, int Z) {
    return reinterpret_cast<unsigned*>(bits + group_offset(X, Y, Z));
}

// launches one of the occupancy kernels, a CTA per super-brick
template <class... P, class... A>
static cudaError_t launch_occupancy(void (*fn)(P...), int X, int Y, int Z, cudaStream_t st, A... args) {
    return launch_chained(fn, dim3((unsigned)((X + 63) / 64), (unsigned)((Z + 63) / 64), (unsigned)((Y + 63) / 64)), 512, st,
                          args...);
}

template <class G>
static fs3d_status launch_dda(const G& grid, const BrickMap& bm, const fs3d_camera* cam, int W, int H, float* rgba_dev,
                              cudaStream_t st) {
    constexpr int kRows = 65535 * 8;  // of one launch: a grid counts 65535 tiles along y
    for (int row0 = 0; row0 < H; row0 += std::min(kRows, H - row0)) {
        const unsigned tiles = (unsigned)((std::min(kRows, H - row0) + 7) / 8);
        const cudaError_t e = launch_chained(k_render_dda<G>, dim3((unsigned)((W + 7) / 8), tiles), 64, st, grid, bm,
                                             to_dev(cam), W, H, row0, reinterpret_cast<float4*>(rgba_dev));
        if (e != cudaSuccess) return cuda_fail(e, "render dda launch");
        note_launch();
    }
    return FS3D_OK;
}

// bits: brickmap_bytes(X, Y, Z) of device scratch the caller provides, zeroed before its first frame
fs3d_status launch_render_dda_bytes(const uint8_t* g, int X, int Y, int Z, uint8_t* bits, const fs3d_camera* cam,
                                    int W, int H, float* rgba_dev, cudaStream_t st) {
    const BrickMap bm = brick_map(bits, X, Y, Z);
    const cudaError_t e =
        launch_occupancy(k_occupancy_bytes, X, Y, Z, st, g, X, Y, Z, bits, const_cast<uint8_t*>(bm.super),
                         group_counters(bits, X, Y, Z));
    if (e != cudaSuccess) return cuda_fail(e, "occupancy (bytes) launch");
    note_launch();
    if ((int64_t)X * Y * Z < (int64_t)1 << 31)
        return launch_dda(BytesGrid<uint32_t>{g, X, Y, Z}, bm, cam, W, H, rgba_dev, st);
    return launch_dda(BytesGrid<uint64_t>{g, X, Y, Z}, bm, cam, W, H, rgba_dev, st);
}

fs3d_status launch_render_dda_planes(const uint4* rows, const uint8_t* statics, int X, int Y, int Z, int nw,
                                     uint8_t* bits, const fs3d_camera* cam, int W, int H, float* rgba_dev,
                                     cudaStream_t st, int* brick_counts, bool recount) {
    const BrickMap bm = brick_map(bits, X, Y, Z);
    uint8_t* super = const_cast<uint8_t*>(bm.super);
    if (brick_counts && recount) {
        FS3D_CUDA(cudaMemsetAsync(brick_counts, 0, brick_count_bytes(X, Y, Z), st));
        k_brickcount_planes<<<map_grid((int64_t)Y * Z * nw), 256, 0, st>>>(rows, X, Y, Z, nw, brick_counts, (X + 7) / 8,
                                                                          (Z + 7) / 8);
        FS3D_CHECK_LAUNCH("brick counts (planes) launch");
    }
    unsigned* group = group_counters(bits, X, Y, Z);
    const cudaError_t e = brick_counts
                              ? launch_occupancy(k_occupancy_counts, X, Y, Z, st, brick_counts, X, Y, Z, bits, super, group)
                              : launch_occupancy(k_occupancy_planes, X, Y, Z, st, rows, X, Y, Z, nw, bits, super, group);
    if (e != cudaSuccess) return cuda_fail(e, "occupancy (planes) launch");
    note_launch();
    const uint32_t* p = reinterpret_cast<const uint32_t*>(rows);
    if ((int64_t)Y * Z * nw * 4 < (int64_t)1 << 31)
        return launch_dda(PlaneGrid<uint32_t>{p, statics, X, Y, Z, nw}, bm, cam, W, H, rgba_dev, st);
    return launch_dda(PlaneGrid<uint64_t>{p, statics, X, Y, Z, nw}, bm, cam, W, H, rgba_dev, st);
}

size_t brick_count_bytes(int X, int Y, int Z) {
    return (size_t)((X + 7) / 8) * ((Y + 7) / 8) * ((Z + 7) / 8) * sizeof(int);
}

size_t brickmap_bytes(int X, int Y, int Z) {
    return group_offset(X, Y, Z) + sizeof(unsigned) * (size_t)((X + 255) / 256) * ((Y + 255) / 256) * ((Z + 255) / 256);
}

}  // namespace fs3d

extern "C" fs3d_status fs3d_render_sdf(const fs3d_camera* cam, int W, int H, float* rgba_dev, void* stream) {
    if (!cam || !rgba_dev || W <= 0 || H <= 0)
        return fs3d::set_error(FS3D_ERR_INVALID_ARG, "fs3d_render_sdf: bad args");
    return fs3d::launch_render_sdf(cam, W, H, rgba_dev, (cudaStream_t)stream);
}
