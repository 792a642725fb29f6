// svo_internal.h -- launch wrappers shared between the kernel files and the C ABI.
#pragma once
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "svo_b200.h"
#include "svo_device.cuh"

namespace svo {

// Counts kernel launches (svo_kernel_launches).
void count_launches(int n);

constexpr int kMaxLevels = 24;
constexpr int kMaxRes = 2048;

// Voxelizer work split (svo_tuning; split, inplace_max and serial_packed have
// no effect).
struct VoxTuning {
    uint32_t serial_max = 64;  // most grid-bbox voxels of a triangle tested by one thread
    uint32_t warp_max = 256;   // queue entries hold a sixteenth as many brick columns
    uint32_t split = 0;
    uint32_t inplace_max = 32;
    uint32_t serial_packed = 0;
};

// Occupancy bitmap pyramid: level 0 is the voxel grid (one bit per Morton
// code), level l+1 bit j = OR of level-l bits 8j..8j+7.  Every level is stored
// as u64 words padded to whole 512-bit blocks, ranked by RankDev.
struct Pyramid {
    int levels = 0;                      // stored levels (>= 5)
    int grid_levels = 0;                 // log2(R) + 1 levels of the real grid
    uint64_t woff[kMaxLevels] = {};      // u64 word offset of level l
    uint64_t words[kMaxLevels] = {};     // u64 words of level l
    uint64_t coff[kMaxLevels + 1] = {};  // 512-bit block offset of level l
    uint64_t total_words = 0;
    uint64_t total_blocks = 0;
    uint32_t ctas = 0;                   // pyramid CTAs (level-0 chunks of 2048 words)
};

Pyramid make_pyramid(int rx, int ry, int rz);

// Ranks of a mesh's 512-bit blocks.  Levels 0..2: the set bits before the
// block in its level-0 region (pre, at coff[l]) on top of the region's prefix
// (base, level l at l * bstride); level 3, half a block per region: the
// region's prefix; levels 4..: pre alone.
struct RankDev {
    const uint32_t *pre;
    const uint32_t *base;
    uint32_t bstride;  // regions of the mesh rounded up to 4
};

// What the counting phase reports about one mesh, in pinned host memory that
// the kernels write directly (no copy after the last kernel); dup is raised by
// the emission.
struct MeshOut {
    GridParams gp;
    uint32_t totals[kMaxLevels];  // set bits per level
    uint64_t any;                 // the code of one surface voxel
    uint32_t queue;               // entries the big-triangle queue needed (the same for all meshes of a batch)
    uint32_t dup;                 // the emission met consecutive duplicates
    uint32_t dedup[4];            // counts of the dedup (dedup_finish)
};

// One mesh of a batch, as the kernels see it (an array in device memory).
// A single build is a batch of one.
struct MeshDev {
    const float *pts;        // device
    const int32_t *tris;     // device; null = soup (3 points per triangle)
    int64_t n_pts;
    int64_t n_tris;
    int res[3];
    int regions;             // 1: level 0 is zeroed and read only in the regions triangles reach
    GridParams *gp;
    uint32_t *mm;            // bbox scratch (8 u32: 6 extremes, blocks finished), zero at the start
    uint64_t *bits;          // this mesh's pyramid (level l at bits + py.woff[l])
    uint32_t *pre;           // block ranks (RankDev)
    uint32_t *base;          // region sums, then their prefixes (RankDev)
    uint32_t bstride;
    uint64_t *any;           // the code of one surface voxel
    const uint32_t *queue;   // big-triangle queue entries of the batch
    MeshOut *out;            // pinned host memory (or device memory of a caller that copies it)
    uint32_t *done;          // pyramid regions finished
    Pyramid py;
};

// Prefix tables over the meshes of a batch (device memory, n + 1 entries).
struct BatchDev {
    const MeshDev *mesh;
    int n;
    const uint64_t *tri_off;   // global index of each mesh's first triangle
    const uint32_t *cta_off;   // first pyramid CTA of each mesh
    const uint32_t *bbox_off;  // first bbox-reduction block of each mesh
    uint8_t *rflag = nullptr;  // per pyramid CTA (a 2048-word region of level 0): a triangle reaches it
    // Batches with a region-mode mesh: the regions that are read (all of the
    // other meshes', the flagged ones of region-mode meshes) in no order, and
    // their number, zeroed.
    uint32_t *rlist = nullptr;
    uint32_t *rcount = nullptr;
    // Host copy of a one-mesh batch's table, or null: the launchers then pass it
    // to the kernels by value and the tables in device memory need not exist.
    const MeshDev *one = nullptr;
};

#if defined(__CUDACC__)
// Chained launches.  A kernel launched by launch_chained may have its blocks
// placed while the last blocks of the kernel before it on the stream are still
// running; chain_begin(), the first thing every block of such a kernel does,
// lets the next chained kernel in and then waits until everything before its
// own kernel is complete and visible.  Since every block waits, a kernel that
// is complete implies that all earlier ones are.  Used where a short kernel
// follows another on the same stream: two plain launches are about 2 us apart.
// With 320 triangles at 32^3 a build took 92.8 us and takes 83.6 this way, with
// 20k at 128^3 120.8 and 108.9, with 5M at 2048^3 4,037 and 4,020.
//
// Such a kernel may be resident while the kernels before it still write.  So it
// reads nothing of theirs as data that is constant over the whole kernel (const
// T *__restrict__, __ldg): the compiler could then use read-only loads, and move
// them before the wait.  Mesh inputs are constant.
__device__ __forceinline__ void chain_begin() {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
}
template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t shmem, cudaStream_t st,
                                  const A &...args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = shmem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// The meshes of a batch as a kernel sees them: the tables in device memory, or
// (ONE) a lone mesh's table in the kernel's parameters, whose fields come from
// the constant bank instead of a chain of loads at the start of every kernel
// (320 triangles at 32^3: 94.5 -> 90.9 us per build; 1M at 1024^3: 837 -> 801).
template <bool ONE>
struct Meshes {
    const BatchDev &bd;
    const MeshDev &one;
    __device__ __forceinline__ const MeshDev &operator[](int m) const { return ONE ? one : bd.mesh[m]; }
    __device__ __forceinline__ int of_tri(uint64_t gid) const;
    __device__ __forceinline__ int of_region(uint32_t g) const;
    __device__ __forceinline__ uint64_t first_tri(int m) const { return ONE ? 0 : bd.tri_off[m]; }
    __device__ __forceinline__ uint32_t first_region(int m) const { return ONE ? 0 : bd.cta_off[m]; }
};
#endif

// Level-0 regions (2048 words: 64 x 64 x 32 voxels) are tracked from this
// level-0 size on (resolution >= 1024).
constexpr uint64_t kRegionWords = 1ull << 24;

// Per-level inputs of the node emission kernel.
struct EmitLevel {
    uint32_t off;          // first node index of the level
    uint32_t n;            // nodes in the level
    const uint64_t *K1;    // sorted codes of level l+1 (the level's groups); level T: its own code
    const uint64_t *bits;  // bitmap of level l
    const uint32_t *wpre;  // rank at each non-empty word of level l (l >= 1)
    uint32_t side;         // grid side at this level (R >> l)
    float width;           // node width
};

// One mesh of an emission pass (an array in device memory).
struct EmitParams {
    int T;                  // top level index (depth - 1)
    uint32_t N;             // total nodes
    uint32_t flags;
    EmitLevel lv[kMaxLevels];
    const GridParams *gp;
    svo_node *nodes;
    svo_vertex *verts;      // may be null (SVO_FLAG_NO_VERT_EDGE)
    svo_edge *edges;
    unsigned long long *dups;  // [0] vertex, [1] edge consecutive duplicates
    uint32_t *dup_flag;        // pinned host memory: set to 1 with the first of them
};

// The meshes of one emission pass: mesh i owns global node slots
// [node_off[i], node_off[i] + N_i), node_off[i] a multiple of 32 (a warp never
// straddles two meshes).
struct EmitBatch {
    const EmitParams *p;
    int n;
    const uint64_t *node_off;  // n + 1 entries
};

// One compaction job: the set bits of levels [l0, l1) of one mesh, level 0
// written to keys, level l >= 1 to out + koff[l]; jobs own consecutive ranges
// of a global word index (word_off, n + 1 entries).
struct CompactJob {
    const uint64_t *bits;
    RankDev rank;
    Pyramid py;
    int l0, l1;
    uint64_t *out;
    uint64_t *keys;
    uint32_t *wpre;  // rank at each non-empty word of levels >= 1 (indexed from woff[1])
    uint64_t koff[kMaxLevels];
    const uint8_t *rflag;  // region-mode mesh: its level-0 region flags (unflagged regions read as empty)
};
struct CompactBatch {
    const CompactJob *job;
    int n;
    const uint64_t *word_off;
};
// The surface-voxel keys of one mesh, from its non-empty level-0 blocks
// (= its level-3 code list).
struct KeyJob {
    const uint64_t *bits;    // level-0 bitmap
    RankDev rank;
    const uint64_t *blocks;  // sorted non-empty block indices
    uint64_t *out;
};
struct KeyBatch {
    const KeyJob *job;
    int n;
    const uint64_t *blk_off;  // prefix of the jobs' block counts
};

// Binary search: the i with off[i] <= x < off[i + 1] (off has n + 1 entries).
template <class T>
__host__ __device__ __forceinline__ int find_segment(const T *off, int n, T x) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= x) lo = mid; else hi = mid - 1;
    }
    return lo;
}

#if defined(__CUDACC__)
template <bool ONE>
__device__ __forceinline__ int Meshes<ONE>::of_tri(uint64_t gid) const {
    return ONE ? 0 : find_segment(bd.tri_off, bd.n, gid);
}
template <bool ONE>
__device__ __forceinline__ int Meshes<ONE>::of_region(uint32_t g) const {
    return ONE ? 0 : find_segment(bd.cta_off, bd.n, g);
}
#endif

// Bounding cube and grid of every mesh (bbox_blocks: bbox_off[n]), beside the
// clearing of the bitmaps of total_ctas regions (0: they are clear already)
// and, with any_regions, of the region flags (padded to whole words).  Every
// mm and gp->status must be zero.
cudaError_t launch_front(const BatchDev &b, uint32_t bbox_blocks, uint32_t total_ctas,
                         bool any_regions, int num_sms, cudaStream_t st);
// mm[0] = min, mm[1] = max of n int32 indices.
cudaError_t launch_index_range(const int32_t *idx, int64_t n, int32_t *mm, cudaStream_t st);
// counters: 2 zeroed u32 (queue entries, queue cursor); big: the queue of
// large triangles, or null: every large triangle is walked by the warp that
// set it up.
cudaError_t launch_voxelize(const BatchDev &b, int64_t total_tris, bool strict, const VoxTuning &tune,
                            uint4 *big, uint32_t big_cap, uint32_t *counters, int num_sms, cudaStream_t st);
// Builds levels 1.. of every mesh's pyramid, the block ranks and the level
// totals; max_ctas: the most regions of any mesh (py.ctas).  done must be zero.
// With b.rlist set only the listed regions are visited.
cudaError_t launch_pyramid(const BatchDev &b, uint32_t total_ctas, uint32_t max_ctas, int num_sms, cudaStream_t st);
// For batches with a region-mode mesh: flags the level-0 regions that its
// triangles reach (rflag zeroed by launch_front), zeroes those and lists the
// regions to read; the unflagged regions get their words of levels 1..4 and
// their region sums here (zeros), and the pyramid only visits the list.
cudaError_t launch_regions(const BatchDev &b, int64_t total_tris, uint32_t total_ctas, int num_sms, cudaStream_t st);
// Exclusive scan of n u32 values; out has n + 1 entries (out[n] = total).
// scratch: >= scan_scratch_words(n) u64 words, zeroed by the call.
size_t scan_scratch_words(uint64_t n);
cudaError_t launch_scan(const uint32_t *in, uint32_t *out, uint64_t n, unsigned long long *scratch,
                        uint32_t *status, cudaStream_t st);
// Self-test of the scan's bounded look-back wait: the single-pass scan with
// its tile counter started at 1, so tile 0 never publishes and every
// look-back that reaches it gives up after spin_limit polls and records
// kStatusScanTimeout in *status.  n must span at least 2 tiles; scratch holds
// scan_stalled_scratch_words(n) words (the CTA that draws index `tiles` has no
// tile and publishes one slot past the last).  out (n + 1 entries) receives
// partial sums.  Synchronises st before the launch.
size_t scan_stalled_scratch_words(uint64_t n);
cudaError_t launch_scan_stalled(const uint32_t *in, uint32_t *out, uint64_t n, unsigned long long *scratch,
                                uint32_t *status, int spin_limit, cudaStream_t st);
// Stream-ordered allocation from one of a context's pools: the one place a
// build allocates device memory (svo_debug_fail_alloc injects failures here).
cudaError_t pool_malloc(void **p, size_t bytes, cudaMemPool_t pool, cudaStream_t st);
// one: the job of a one-job batch (host copy, passed by value), or null.
cudaError_t launch_compact(const CompactBatch &c, const CompactJob *one, uint64_t total_words, cudaStream_t st);
// one: the job of a one-job batch (host copy, passed by value), or null.
cudaError_t launch_compact_keys(const KeyBatch &k, const KeyJob *one, uint64_t total_blocks, cudaStream_t st);
// Levels 1 and 2 of a region-mode job (job.rflag set): its regions are those of
// the batch's list (BatchDev) from cta0 on.
cudaError_t launch_compact_regions(const CompactJob &job, const uint32_t *rlist, const uint32_t *rcount, uint32_t cta0,
                                   uint32_t regions, int num_sms, cudaStream_t st);
// one: the EmitParams of a one-mesh batch (host copy, passed by value to the
// kernel), or null for a batch of several meshes.
cudaError_t launch_emit(const EmitBatch &b, const EmitParams *one, uint64_t total_nodes, uint32_t flags,
                        int num_sms, cudaStream_t st);
// Stable removal of consecutive duplicates (thrust::unique semantics).
cudaError_t launch_unique_vertices(const svo_vertex *in, uint64_t n, svo_vertex *out,
                                   uint32_t *tile_counts, uint32_t *tile_pre,
                                   unsigned long long *scan_scratch, uint32_t *status,
                                   cudaStream_t st);
cudaError_t launch_unique_edges(const svo_edge *in, uint64_t n, svo_edge *out, uint32_t *tile_counts,
                                uint32_t *tile_pre, unsigned long long *scan_scratch,
                                uint32_t *status, cudaStream_t st);
constexpr uint32_t kUniqueTile = 4096;

// Morton-keyed unique vertex/edge/face keys of all nodes (SVO_FLAG_DEDUP), in
// two steps on one stream.  dedup_begin needs only the level bitmaps (bits[l],
// side sides[l], l = 0..T): it takes the scratch and builds the level-1 part
// of the candidate bitmap, so it can run before the code lists exist.
// dedup_finish (after the code lists, ep) writes the keys and frees the run;
// report: 4 words of pinned host memory that the kernels leave counts in.
// dedup_abort frees a run that will not be finished.
struct DedupRun;
int dedup_begin(cudaMemPool_t scratch_pool, cudaStream_t st, int T, const uint64_t *const *bits,
                const uint32_t *sides, int num_sms, uint32_t *report, DedupRun **run);
int dedup_finish(DedupRun *run, cudaMemPool_t out_pool, const EmitParams &ep, uint64_t n_out[3], uint64_t *out[3]);
void dedup_abort(DedupRun *run);

// Blocks of the bbox reduction for a mesh of n points.
inline uint32_t bbox_blocks(int64_t n) {
    return (uint32_t)std::max<int64_t>(1, std::min<int64_t>((n / 4 + 255) / 256, 148 * 4));
}

}  // namespace svo
