// Bit-plane world format: device descriptors and host entry points.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "fs3d_common.h"
#include "pcg.h"

namespace fs3d {

// One world as the step kernel sees it (device memory, 64 bytes).
struct PlaneWorld {
    uint4* rows;      // Y*Z rows of nw uint4 words
    uint64_t seed;
    uint64_t t;       // step counter at the start of the current segment
    int32_t X, Y, Z, nw;
    int32_t steps;    // steps this world takes in the current segment
    int32_t lg;       // log2 of the lane-group size (pow2ceil(nw))
    uint8_t* lflags;       // nullable: per-layer last-changed step (low 8 bits), kept across segments
    int32_t lflags_fresh;  // 1: lflags hold nothing yet (start from "every layer changed")
    int32_t pad;
};
static_assert(sizeof(PlaneWorld) == 64, "PlaneWorld layout");

// Warp-sized work item: 32 >> lg block row-pairs of one world.
struct PlaneItem {
    int32_t world;
    int32_t rp0;
};

inline int plane_nw(int X) { return (X + 63) / 64; }
inline size_t plane_bytes(int X, int Y, int Z) { return (size_t)Y * Z * plane_nw(X) * sizeof(uint4); }
// layer flags stored after a world's planes in the same allocation
inline size_t layer_flag_bytes(int Y) { return ((size_t)Y + 15) & ~(size_t)15; }
constexpr int kPlaneMaxX = 2048;  // lane groups of at most 32 words

// Resident segment classes: worlds whose planes fit in shared memory take
// all their segment steps in one launch.  Classes 0..2 hold a world in one CTA
// of 128 / 256 / 768 threads (6 / 3 / 1 CTAs per SM); classes 3..5 split a
// world into z-slabs over a cluster of 2 / 4 / 8 CTAs.
constexpr int kResidentClasses = 6;
constexpr int kSingleCtaClasses = 3;  // classes 0..2 hold a world in one CTA
constexpr int kClusterSizes[3] = {2, 4, 8};
// Global-memory segment classes (the world stays in L2/HBM; one CTA of
// 32/64/128/256 threads per world, by the work of one layer pair; -1 if the
// world has too many layers), and kGmDense: one CTA of 768 threads per SM
// for a young (dense) world too large for one CTA's shared memory.
constexpr int kGmClasses = 5;
constexpr int kGmDense = 4;
constexpr int kGmThreads[kGmClasses] = {32, 64, 128, 256, 768};
// the most layers of a world in each: its CTAs have shared memory for the flags of so many
constexpr int kGmMaxY[kGmClasses] = {1024, 1024, 2048, 4096, 4096};
// the first class from c on that holds Y layers (kGmClasses: none does)
inline int gm_class_holding(int c, int Y) {
    while (c < kGmClasses && Y > kGmMaxY[c]) ++c;
    return c;
}
// Classes of settled worlds at a batch's level (choose_widen), by their class
// for themselves (`own`, 0..3).  A level may narrow a world's CTA only as far
// as its layers still fit.
constexpr int kPackedLevel = 0, kOwnLevel = 1, kWidestLevel = 4;
constexpr int kWidened[kWidestLevel + 1][kGmDense] = {
    {1, 1, 1, 3}, {0, 1, 2, 3}, {0, 2, 3, 3}, {2, 3, 3, 3}, {3, 3, 3, 3}};
inline int gm_class_at(int level, int own, int Y) { return gm_class_holding(kWidened[level][own], Y); }
int resident_class_gm(int X, int Y, int Z);
// Class ids of a segment's tables: shared-memory classes 0..5, then the
// global-memory classes 6..9.  meta = {per-step items, worlds per class,
// offset of each class in the order array, worlds in the table}.
constexpr int kAllClasses = kResidentClasses + kGmClasses;
constexpr int kMetaWorlds = 1 + 2 * kAllClasses;
constexpr int kMetaInts = kMetaWorlds + 1;
// Dynamic shared memory of a CTA of each shared-memory class (0: the class
// cannot run) in the current device and context.
struct ResidentLimits {
    int one_cta[kSingleCtaClasses] = {};
    int cluster = 0;
    int clusters = 0;  // clusters of 8 CTAs that run at once
};
ResidentLimits resident_limits();
// smallest class that holds a world of these dims, -1 if none does
int resident_class(const ResidentLimits& l, int X, int Y, int Z);
constexpr int kErrInts = 4;  // size of the error record a resident launch is given
// test hook: bulk copies announced with more bytes than they deliver
enum CopyStall : uint32_t {
    kStallNone = 0,
    kStallAll = 1,        // every one
    kStallOneCta = 2,     // those of worlds held by one CTA
    kStallFirstSlab = 3,  // that of the first CTA of a world cut into slabs
    kStallRefuse = 4,     // (none; multi-step launches are refused)
    kStallKinds = 5
};
fs3d_status set_inject_tx_extra(uint32_t stall);
// test hook: the next n stream-ordered allocations of batch admissions fail as out of memory
void set_inject_alloc_failures(int n);
// One launch steps every world of the single-CTA class `cls`
// (order[meta[1+K+cls] ...], meta[1+cls] of them) through its segment steps in
// shared memory.  err
// points to 4 ints (8-byte aligned): a bulk copy that does not complete
// within the wait limit sets err[0] = 1 and err[2..3] = the failing world's
// step at the start of the launch (first failure only); while err[0] is set,
// launches given it step nothing.  Row
// pairs whose rows are settled are skipped; the cell-steps actually evaluated
// are added to *processed_cells when it is not null.
fs3d_status launch_plane_segment_resident(int cls, const PlaneWorld* worlds, const int* order, const int* meta,
                                          int* counter, int* err, cudaStream_t st,
                                          unsigned long long* processed_cells = nullptr);

// `first`: launched with the greatest priority, so that in a segment graph,
// where every class's grid is pending at once, its CTAs are placed first.
fs3d_status launch_plane_segment_gm(int cls, const PlaneWorld* worlds, const int* order, const int* meta,
                                    int* counter, int* err, cudaStream_t st, unsigned long long* processed_cells,
                                    bool first = false);

// One world of a many-world conversion: its planes, its canonical bytes
// (admission: read; read-back: written) and its static bytes (nullable).
struct ConvJob {
    uint4* rows;
    const uint8_t* statics;
    uint8_t* bytes;
    int32_t X, Y, Z, nw;
    // read-back of a world whose static-material flag has not reached the
    // host yet: when *static_flag is set, its static bytes are at static_src
    const int* static_flag;
    const uint8_t* static_src;
    // admission: the world's layer flags (set from its cells by
    // layer_flags_from_cells_multi; null: none) and its first step's low 8 bits
    uint8_t* lflags = nullptr;
    uint32_t t0b = 0;
    uint32_t magic = 0;  // read-back: conv_magic(X)
};
// One CTA of a conversion takes whole rows of one world: as many as make
// `chunks` 64-cell chunks, from row0 on.  Read-backs of many worlds take twice
// the chunks of the others (a CTA's set-up is a third of its instructions).
constexpr int kConvThreads = 256, kConvChunks = kConvThreads, kConvChunksBack = 2 * kConvThreads;
struct ConvBlock {
    int32_t job;
    uint32_t row0;
};
FS3D_HD int conv_rows(int nw, int chunks) { return chunks / nw; }
inline int64_t conv_blocks(int Y, int Z, int nw, int chunks) {
    return ((int64_t)Y * Z + conv_rows(nw, chunks) - 1) / conv_rows(nw, chunks);
}
// the blocks of job j, written to out; returns how many
inline int64_t conv_fill_blocks(int j, int Y, int Z, int nw, int chunks, ConvBlock* out) {
    const int64_t n = conv_blocks(Y, Z, nw, chunks);
    for (int64_t i = 0; i < n; ++i) out[i] = ConvBlock{j, (uint32_t)(i * conv_rows(nw, chunks))};
    return n;
}
// ConvJob::magic: i / ceil(X / 16) = umulhi(i, magic) for i < 2^16
inline uint32_t conv_magic(int X) { return 0xFFFFFFFFu / (uint32_t)((X + 15) / 16) + 1u; }
// bytes -> planes for many worlds in one launch; flags[j] |= 1 when world j
// holds a material >= 4
fs3d_status planes_from_bytes_multi(const ConvJob* jobs, const ConvBlock* blocks, int64_t nblocks, int* flags,
                                    cudaStream_t st);
fs3d_status planes_to_bytes_multi(const ConvJob* jobs, const ConvBlock* blocks, int64_t nblocks, cudaStream_t st);

// Many byte copies in one launch (each thread moves a 16-byte chunk): used
// instead of one cudaMemcpyAsync per world when both sides are addressable
// by the device (device memory, or page-locked host memory, which the GPU
// reads and writes directly).  chunk_off[j] = sum of ceil(bytes/16) before j.
struct CopyJob {
    const uint8_t* src;
    uint8_t* dst;
    int64_t bytes;
};
fs3d_status copy_many(const CopyJob* jobs, const int64_t* chunk_off, int njobs, int64_t total_chunks, cudaStream_t st);
// A small copy (tables, flags) done by a kernel instead of a copy engine, so
// it does not queue behind large transfers on the copy engines.  Both
// pointers must be device-addressable (device memory, or the device view of
// page-locked host memory); pointers not 16-byte aligned take cudaMemcpyAsync.
cudaError_t copy_small_async(void* dst, const void* src, size_t bytes, cudaStream_t st);
// Whether p is memory of the current device (which a kernel may write at full rate).
bool device_local(const void* p);
// A device-addressable alias of p (itself for device or managed memory, the
// mapped address for page-locked host memory), or nullptr for pageable memory.
uint8_t* device_view(const void* p);
// The allocation that holds p (start, bytes), as the driver reports it; false
// if it cannot tell.  A copy over several grids must stay inside one.
bool alloc_range(const void* p, uintptr_t* start, size_t* bytes);

int plane_lg(int nw);
int plane_items_for(int Y, int Z, int nw);
int plane_step_grid(int64_t n_items);
int plane_step_ctas_per_sm();
fs3d_status planes_from_bytes(const uint8_t* g, int X, int Y, int Z, uint4* rows, cudaStream_t st,
                              int* statics_flag = nullptr);
// the batch world of `world_seed` written straight into planes (needs Y >= 4)
fs3d_status planes_generate_batch_world(uint64_t world_seed, int X, int Y, int Z, uint4* rows, cudaStream_t st);
// the same for many worlds in one launch (blocks of kConvChunks chunks, as the admission conversion's)
struct GenJob {
    uint4* rows = nullptr;
    int32_t X = 0, Y = 0, Z = 0, nw = 0;
    BatchWorldGen p = {};
};
GenJob gen_job(uint64_t world_seed, int X, int Y, int Z, uint4* rows);
fs3d_status planes_generate_multi(const GenJob* jobs, const ConvBlock* blocks, int64_t nblocks, cudaStream_t st);
// skip_if_set (nullable): the conversion writes nothing when *skip_if_set is
// non-zero (a drop-in run whose step kernel recorded a failure leaves the
// caller's grid as it was)
fs3d_status planes_to_bytes(const uint4* rows, const uint8_t* statics, int X, int Y, int Z, uint8_t* g,
                            cudaStream_t st, const int* skip_if_set = nullptr);

// ---- per-step kernel of one large world with an exact skip of settled
// row-pairs: one byte per row (y, z) holds the low 8 bits of the last step
// that changed it (Y*Z bytes).  init_row_flags: a world about to take step t0
// with no history: a row is marked changed at t0 - 1 when a block row-pair of
// either phase that covers it can change (the rule's activity mask on its
// cells), else at t0 - 3.  own (nullable): set to *err on the way, the word that
// decides about one drop-in run (see launch_plane_slabs).
fs3d_status init_row_flags(const uint4* rows, uint8_t* rflags, int X, int Y, int Z, uint64_t t0, cudaStream_t st,
                           const int* err = nullptr, int* own = nullptr);

// Layer flags of newly admitted worlds (jobs with lflags set), the same way
// per layer: marked changed at t0 - 1 when a block row-pair of either phase
// covering the layer can change, else at t0 - 3.  max_Y: the largest Y of the jobs.
fs3d_status layer_flags_from_cells_multi(const ConvJob* jobs, int njobs, int max_Y, cudaStream_t st);
// the same for one world
fs3d_status layer_flags_from_cells(const uint4* rows, uint8_t* lflags, int X, int Y, int Z, uint64_t t0,
                                   cudaStream_t st);
// one step (w.t) of the world; counts (nullable): its per-brick counts of
// non-empty cells, kept exact; err (nullable): while *err is set nothing is stepped
fs3d_status launch_plane_step_skip(const PlaneWorld& w, uint8_t* rflags, int* counts, const int* err, cudaStream_t st);
// ---- many steps of one world in one launch over the whole GPU (slab.cu)
struct SlabPlan {
    int zs = 0;          // slabs cut along z (else along y)
    int ctas = 0;        // slabs
    int threads = 0;     // per CTA
    int smem = 0;        // dynamic shared memory per CTA
    size_t scratch = 0;  // device scratch a launch needs (256-byte aligned; the launch clears it)
};
// how a world would be cut; false if its slabs do not fit in shared memory
bool slab_plan(int X, int Y, int Z, SlabPlan* out);
// whether a call of n steps takes them in one such launch rather than in n
// launches of the per-step kernel
bool prefer_slabs(int X, int Y, int Z, int n_steps, SlabPlan* out);
// w.steps steps from w.t; rflags as for launch_plane_step_skip (kept from call
// to call), err as for launch_plane_segment_resident.  own: the word whose being
// set keeps the launch from stepping; a failure sets both.  It is err itself
// where the launches of one stream share err, else a copy of it taken when the
// run began: a failure on another stream that is recorded while this run goes
// on must not change its mind half-way.  *taken: the steps launched, fewer than
// w.steps when the device refuses such a launch.
fs3d_status launch_plane_slabs(const PlaneWorld& w, const SlabPlan& plan, uint8_t* rflags, void* scratch, int* err, int* own,
                               cudaStream_t st, int* taken);
fs3d_status set_slab_stall(uint32_t stall);  // test hook, as set_inject_tx_extra
// ---- a batch's worlds of a cluster class: CS CTAs a world, cut along z
// (slab.cu).  Whether a world's slabs fit; the most words (Y * nw) of a layer
// at a cut; the bytes of edge buffer a class needs; the launch, as
// launch_plane_segment_resident (by_place: the order of a slab's row-pairs).
constexpr int kBatchSlabEdgeWords = 1024;
void batch_slabs_limits(ResidentLimits* out);  // its last two
bool batch_slabs_fit(const ResidentLimits& l, int X, int Y, int Z, int CS);
size_t batch_slab_edge_bytes(int CS);
fs3d_status launch_batch_slabs(int cls, int CS, const PlaneWorld* worlds, const int* order, const int* meta, int* counter,
                               int* err, void* edges, cudaStream_t st, unsigned long long* processed_cells, bool by_place);

fs3d_status planes_hash_async(const uint4* rows, const uint8_t* statics, int X, int Y, int Z,
                              unsigned long long* out_dev, cudaStream_t st);
// whole-grid hashes of njobs worlds in one launch: the hash of jobs[j] is the
// sum (mod 2^64) of out_dev[j * parts .. + parts)
struct HashJob {
    const uint4* rows;
    const uint8_t* statics;  // nullable
    int32_t X, Y, Z, nw;
};
fs3d_status planes_hash_many(const HashJob* jobs, int njobs, int parts, unsigned long long* out_dev, cudaStream_t st);
// One step of many worlds at once (the batch's worlds too large to be
// resident).
fs3d_status launch_plane_step(const PlaneWorld* worlds, const PlaneItem* items, const int* n_items_dev, int grid,
                              int s_seg, cudaStream_t st);

// After a segment: every world of the table (meta[kMetaWorlds] of them) moves
// on by its segment steps, and its layer flags count as kept, so the next
// segment of an unchanged batch reuses the table as it stands.
fs3d_status launch_advance_worlds(PlaneWorld* worlds, const int* meta, cudaStream_t st);

// byte-grid kernels (step_bytes.cu)
fs3d_status launch_step_bytes(uint8_t* grid, int X, int Y, int Z, uint64_t seed, uint64_t t0, int n_steps,
                              cudaStream_t st);
fs3d_status hash_bytes_async(const uint8_t* g, int64_t n, unsigned long long* out_dev, cudaStream_t st);
int sm_count_public();

// render (render.cu)
fs3d_status launch_render_sdf(const fs3d_camera* cam, int W, int H, float* rgba_dev, cudaStream_t st);
// the DDA kernels take a brick occupancy map of brickmap_bytes() bytes, zeroed before its first frame
size_t brickmap_bytes(int X, int Y, int Z);
fs3d_status launch_render_dda_bytes(const uint8_t* g, int X, int Y, int Z, uint8_t* bits, const fs3d_camera* cam,
                                    int W, int H, float* rgba_dev, cudaStream_t st);
// brick_counts (nullable): exact per-brick counts of non-empty cells; the
// frame then derives its brick map from them (rebuild: recount from the
// planes first) instead of a pass over the planes
fs3d_status launch_render_dda_planes(const uint4* rows, const uint8_t* statics, int X, int Y, int Z, int nw,
                                     uint8_t* bits, const fs3d_camera* cam, int W, int H, float* rgba_dev,
                                     cudaStream_t st, int* brick_counts = nullptr, bool recount = true);
size_t brick_count_bytes(int X, int Y, int Z);

// batch.cu: the admissions of a serving loop, many at once
fs3d_status batch_admit_generated_many(fs3d_batch* b, int n, const fs3d_world_spec* specs, uint64_t* tickets,
                                       int* n_admitted);

}  // namespace fs3d
