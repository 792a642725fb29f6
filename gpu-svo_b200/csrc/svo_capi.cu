// svo_capi.cu -- C ABI: context, build orchestration, results.
//
// One build = (host->device copy of the mesh) -> bounding cube -> voxelize
// into the level-0 bitmap -> pyramid + block ranks, whose last kernel writes
// the level totals to pinned host memory (the only mid-build sync, to size the
// outputs) -> per-level code lists -> one emission pass writing nodes,
// vertices and edges, which raises a flag in pinned host memory when it meets
// duplicates.
// The reference's equivalent (src/SVO.cu:341-735) synchronises with the host
// at least six times per level and reallocates its node array per level.
#include <atomic>
#include <mutex>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <vector>

#include "svo_internal.h"
#include "svo_host.h"
#include "svo_hostcopy.h"

using namespace svo;

// Extra streams over which an emission wave spreads its per-mesh launches
// (fork from and join back to the build stream with events).
struct AuxStreams {
    static constexpr int kCount = 3;
    cudaStream_t s[kCount] = {};
    cudaEvent_t fork = nullptr;
    cudaEvent_t join[kCount] = {};
};

// The pool of the result arrays.  A context and its results share it and the last
// of them destroys it, after every free has completed: later copies of the
// process crashed in the driver once a pool had been destroyed with allocations
// outstanding.
struct OutPool {
    int device;
    cudaMemPool_t pool;
    std::atomic<bool> outlived{false};  // results were left when the context went
    OutPool(int d, cudaMemPool_t p) : device(d), pool(p) {}
    ~OutPool() {
        cudaSetDevice(device);
        if (outlived) cudaDeviceSynchronize();  // the frees may be on several streams
        cudaMemPoolDestroy(pool);
    }
};

struct svo_ctx {
    int device = 0;
    int num_sms = 148;
    cudaMemPool_t pool = nullptr;      // per-build scratch
    cudaMemPool_t out_pool = nullptr;  // result arrays, kept apart so scratch never splits their blocks
    std::shared_ptr<OutPool> out_keep;  // holds out_pool
    VoxTuning tune;                    // read and written under tune_mu
    std::mutex tune_mu;
    std::mutex aux_mu;                 // builds on other threads take sets of their own
    std::vector<AuxStreams *> aux_free, aux_all;
    // Pinned host blocks for the reports of batches in flight (one batch each).
    struct Pinned {
        void *p;
        size_t bytes;
    };
    std::mutex pinned_mu;
    std::vector<Pinned> pinned_free;
    std::shared_ptr<svo::host::CopyPool> copies;  // staged copies of results, shared with them
};

// One device block that holds the output arrays of several results (a wave of
// a batch); freed with the last of them.
struct svo_arena {
    void *base = nullptr;
    std::atomic<int> refs{0};
};

struct svo_result {
    int device = 0;
    cudaStream_t stream = nullptr;
    std::shared_ptr<OutPool> out_keep;  // the pool of its arrays
    int depth = 0;
    std::vector<int64_t> level_counts;
    svo_aabb bbox{};
    float unit[3] = {0.0f, 0.0f, 0.0f};
    uint64_t n_nodes = 0, n_verts = 0, n_edges = 0, n_keys = 0;
    svo_node *nodes = nullptr;
    svo_vertex *verts = nullptr;
    svo_edge *edges = nullptr;
    uint64_t *keys = nullptr;
    uint64_t n_dedup[3] = {0, 0, 0};
    uint64_t *dedup[3] = {nullptr, nullptr, nullptr};
    int n_timings = 0;
    float timings[9] = {};
    svo_arena *arena = nullptr;  // holds nodes/verts/edges/keys when set
    std::shared_ptr<svo::host::CopyPool> copies;
    uint32_t own = 0x7F;         // bit i: array i of {nodes, verts, edges, keys, dedup x3} is freed on its own
};

namespace {

thread_local std::string g_err;

int fail(int code, const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

int cuda_fail(cudaError_t e, const char *what) {
    if (e == cudaErrorMemoryAllocation)
        return fail(SVO_ERR_OUT_OF_MEMORY, "%s: %s", what, cudaGetErrorString(e));
    return fail(SVO_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

#define SVO_TRY(call, what)                               \
    do {                                                  \
        cudaError_t e_ = (call);                          \
        if (e_ != cudaSuccess) return cuda_fail(e_, what); \
    } while (0)

bool is_device_ptr(const void *p) {
    if (!p) return false;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// Ordinary host memory, unknown to CUDA.
bool is_pageable_ptr(const void *p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// Stream-ordered scratch owned by one build; everything is returned to the
// pool at the end of the build.
struct Scratch {
    cudaMemPool_t pool;
    cudaStream_t st;
    std::vector<void *> ptrs;
    cudaError_t err = cudaSuccess;
    template <class T>
    T *get(size_t count) {
        void *p = nullptr;
        if (err != cudaSuccess) return nullptr;
        err = pool_malloc(&p, std::max<size_t>(count * sizeof(T), 256), pool, st);
        if (err != cudaSuccess) return nullptr;
        ptrs.push_back(p);
        return static_cast<T *>(p);
    }
    void release() {
        for (void *p : ptrs) cudaFreeAsync(p, st);
        ptrs.clear();
    }
    ~Scratch() { release(); }
};

template <class T>
T *pool_alloc(cudaMemPool_t pool, cudaStream_t st, size_t count, cudaError_t &err) {
    void *p = nullptr;
    if (err != cudaSuccess) return nullptr;
    err = pool_malloc(&p, std::max<size_t>(count * sizeof(T), 256), pool, st);
    return static_cast<T *>(p);
}

// CUDA events at stage boundaries (SVO_FLAG_TIMINGS).
struct StageTimer {
    enum { kStart, kBbox, kVox, kPyr, kCompact0, kCompact, kKeys, kEmit, kUnique0, kUnique, kDedup0, kDedup, kEnd, kN };
    bool on = false;
    cudaEvent_t ev[kN] = {};
    bool rec[kN] = {};
    explicit StageTimer(bool enable) : on(enable) {
        if (!on) return;
        for (auto &e : ev) cudaEventCreate(&e);
    }
    ~StageTimer() {
        if (!on) return;
        for (auto &e : ev) cudaEventDestroy(e);
    }
    void mark(int i, cudaStream_t st) {
        if (!on) return;
        cudaEventRecord(ev[i], st);
        rec[i] = true;
    }
    float span(int a, int b) const {
        float ms = 0.0f;
        if (on && rec[a] && rec[b]) cudaEventElapsedTime(&ms, ev[a], ev[b]);
        return ms;
    }
};

// ---------------------------------------------------------------------------
// Batches.  Phase A (svo_batch_create) runs for every mesh at once: bounding
// cube, voxelization, a bitmap pyramid that ranks its own blocks, and a report
// with the level totals that the last kernel writes to pinned host memory.  Phase B (svo_batch_emit) writes
// the octrees of any subset of the meshes in one compaction launch and one
// emission launch.  svo_build is a batch of one.
// ---------------------------------------------------------------------------
struct MeshHost {
    const float *h_pts = nullptr;      // caller's pointers
    const int32_t *h_tris = nullptr;
    int64_t n_pts = 0, n_tris = 0;     // n_tris: triangles (soup: n_pts / 3)
    int res[3] = {0, 0, 0};
    const float *d_pts = nullptr;      // device copies or the caller's device pointers
    const int32_t *d_tris = nullptr;
    bool tris_on_device = false;
    Pyramid py;
    uint64_t bits_off = 0, pre_off = 0, base_off = 0;  // into the batch's bitmap / rank buffers
    uint32_t cta0 = 0;                   // first pyramid CTA (level-0 region) in the batch
    int status = SVO_OK;
    std::string error;
    GridParams gp{};
    uint32_t totals[kMaxLevels] = {};
    int T = -1;
    uint64_t n_l[kMaxLevels] = {}, off[kMaxLevels + 1] = {};
    uint64_t N = 0;
    uint64_t top = 0;  // the code of the single level-T node
    bool emitted = false;
};

// Layout of a batch's small device block that starts zeroed: counters, grid
// parameters, bounding-box scratch, duplicate counts.
struct MetaLayout {
    size_t counters = 0, gp = 0, any = 0, mm = 0, done = 0, dups = 0, bytes = 0;
    explicit MetaLayout(int n) {
        auto take = [&](size_t b) {
            const size_t o = (bytes + 255) / 256 * 256;
            bytes = o + b;
            return o;
        };
        counters = take(4 * sizeof(uint32_t));
        gp = take(sizeof(GridParams) * n);
        any = take(sizeof(uint64_t) * n);
        mm = take(sizeof(uint32_t) * 8 * n);
        done = take(sizeof(uint32_t) * n);
        dups = take(sizeof(unsigned long long) * 2 * n);
    }
};

// Host tables laid out in one buffer, filled in place and uploaded with one
// copy: add() every table, then make(), then fill at().  No growing and no second
// copy, since a table of thousands of meshes is megabytes, whose fresh pages cost
// more than their contents: with vectors of jobs and emission parameters that were
// appended to a growing buffer (13.8 KB of fresh pages a mesh, 4.0 this way) a
// batch of 1,000 small meshes at res 8 took 2.8 ms instead of 0.97, one of 300
// 1.12 instead of 0.31, one of 6,000 37 instead of 14.
struct HostPack {
    size_t bytes = 0;
    std::unique_ptr<unsigned char[]> buf;
    template <class T>
    size_t add(size_t count) {
        const size_t off = (bytes + 15) / 16 * 16;
        if (count) bytes = off + count * sizeof(T);
        return off;
    }
    void make() { buf.reset(bytes ? new unsigned char[bytes] : nullptr); }
    template <class T>
    T *at(size_t off) const { return reinterpret_cast<T *>(buf.get() + off); }
};

}  // namespace

struct svo_batch {
    svo_ctx *ctx = nullptr;
    cudaStream_t st = nullptr;
    uint32_t flags = 0;
    VoxTuning tune;                         // the voxelizer split this batch runs with
    std::vector<MeshHost> m;
    std::vector<int> live;                  // meshes with device work
    std::vector<void *> allocs;             // phase A buffers (pool)
    uint64_t *bits = nullptr;
    uint32_t *pre = nullptr, *base = nullptr;  // block ranks, region prefixes (RankDev)
    uint8_t *rflag = nullptr;               // level-0 regions that triangles reach (one byte per pyramid CTA)
    uint32_t *rlist = nullptr, *rcount = nullptr;  // the regions to read (BatchDev)
    unsigned long long *dups = nullptr;     // 2 per live mesh (device, zeroed by phase A)
    svo_ctx::Pinned box{nullptr, 0};        // pinned host memory: a MeshOut per live mesh
    MeshOut *out = nullptr;
    MeshDev *d_mesh = nullptr;
    HostPack tables;                        // the host copy of the mesh tables
    MeshDev *h_mesh = nullptr;              // in tables, one per live mesh
    bool pending = false;                   // the stream may still hold work of this batch
    float timings_a[4] = {};                // total, bbox, voxelize, pyramid
    bool timed = false;
};

namespace {

template <class T>
T *batch_alloc(svo_batch *b, size_t count, cudaError_t &err) {
    T *p = pool_alloc<T>(b->ctx->pool, b->st, count, err);
    if (p) b->allocs.push_back(p);
    return p;
}

// A pinned host block of at least `bytes` (the smallest kept one that holds
// them first); p is null when there is none to be had.  Sizes are powers of two,
// so that batches of about the same number of meshes take each other's blocks.
// Kept for later batches: at most 16 blocks and kPinnedKept bytes (the reports
// of 80,000 meshes), the largest ones; the context frees them.  A block that is
// not kept costs its batch a cudaHostAlloc and a cudaFreeHost, and the latter
// waits for all work on the device, other streams' too.
constexpr size_t kPinnedKept = 16u << 20;

svo_ctx::Pinned pinned_acquire(svo_ctx *ctx, size_t bytes) {
    {
        std::lock_guard<std::mutex> lk(ctx->pinned_mu);
        auto best = ctx->pinned_free.end();
        for (auto it = ctx->pinned_free.begin(); it != ctx->pinned_free.end(); ++it)
            if (it->bytes >= bytes && (best == ctx->pinned_free.end() || it->bytes < best->bytes)) best = it;
        if (best != ctx->pinned_free.end()) {
            const svo_ctx::Pinned b = *best;
            ctx->pinned_free.erase(best);
            return b;
        }
    }
    svo_ctx::Pinned b{nullptr, 1u << 14};
    while (b.bytes < bytes) b.bytes *= 2;
    if (cudaHostAlloc(&b.p, b.bytes, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
        cudaGetLastError();
        b.p = nullptr;
    }
    return b;
}

void pinned_release(svo_ctx *ctx, svo_ctx::Pinned b) {
    if (!b.p) return;
    std::vector<svo_ctx::Pinned> drop;
    {
        std::lock_guard<std::mutex> lk(ctx->pinned_mu);
        std::vector<svo_ctx::Pinned> &kept = ctx->pinned_free;
        kept.push_back(b);
        size_t total = 0;
        for (const svo_ctx::Pinned &k : kept) total += k.bytes;
        auto smaller = [](const svo_ctx::Pinned &x, const svo_ctx::Pinned &y) { return x.bytes < y.bytes; };
        while (kept.size() > 16 || total > kPinnedKept) {
            auto it = b.bytes > kPinnedKept ? kept.end() - 1 : std::min_element(kept.begin(), kept.end(), smaller);
            total -= it->bytes;
            drop.push_back(*it);
            kept.erase(it);
        }
    }
    for (svo_ctx::Pinned &d : drop) cudaFreeHost(d.p);
}

// The batch's stream must have finished (its kernels write to the report).
void batch_release(svo_batch *b) {
    for (void *p : b->allocs) cudaFreeAsync(p, b->st);
    b->allocs.clear();
    pinned_release(b->ctx, b->box);
    b->box = svo_ctx::Pinned{nullptr, 0};
}

int mesh_error(MeshHost &mh, int code, const char *msg) {
    mh.status = code;
    mh.error = msg;
    return code;
}

// Offsets of arrays laid out one after another in one block (256-byte aligned):
// fewer pool allocations per build.
struct Layout {
    size_t bytes = 0;
    template <class T>
    size_t add(size_t count) {
        const size_t at = bytes;
        bytes += (std::max<size_t>(count * sizeof(T), 1) + 255) / 256 * 256;
        return at;
    }
};

// Phase A.  Returns SVO_OK when the batch itself works (individual meshes
// may still carry an error status).
int batch_phase_a(svo_batch *b) {
    svo::host::TraceRange trace("svo: counting phase (voxelize, pyramid)");
    svo_ctx *ctx = b->ctx;
    cudaStream_t st = b->st;
    SVO_TRY(cudaSetDevice(ctx->device), "cudaSetDevice");
    cudaError_t err = cudaSuccess;
    b->pending = true;
    // ---- validation and mesh data on the device ----
    for (int i = 0; i < (int)b->m.size(); ++i) {
        MeshHost &mh = b->m[i];
        if (!mh.h_pts || mh.n_pts <= 0) {
            mesh_error(mh, SVO_ERR_EMPTY, "mesh has no vertices");
            continue;
        }
        if (mh.n_tris < 0 || (!mh.h_tris && mh.n_pts % 3 != 0)) {
            mesh_error(mh, SVO_ERR_INVALID_ARGUMENT, "triangle soup needs 3 points per triangle");
            continue;
        }
        if (!mh.h_tris) mh.n_tris = mh.n_pts / 3;
        if (mh.n_tris > 0x7FFFFFFF) {
            mesh_error(mh, SVO_ERR_UNSUPPORTED, "more than 2^31-1 triangles");
            continue;
        }
        bool bad_res = false;
        for (int a = 0; a < 3; ++a) bad_res |= mh.res[a] < 1 || mh.res[a] > kMaxRes;
        if (bad_res) {
            char msg[96];
            snprintf(msg, sizeof(msg), "resolution outside [1, %d]", kMaxRes);
            mesh_error(mh, SVO_ERR_UNSUPPORTED, msg);
            continue;
        }
        // face indices are checked on the device by the kernels that read them
        // (kStatusBadIndex, reported with the level totals)
        if (mh.h_tris && mh.n_tris > 0) mh.tris_on_device = is_device_ptr(mh.h_tris);
        if (is_device_ptr(mh.h_pts)) {
            mh.d_pts = mh.h_pts;
        } else {
            float *p = batch_alloc<float>(b, (size_t)mh.n_pts * 3, err);
            if (!p) return cuda_fail(err, "alloc points");
            SVO_TRY(cudaMemcpyAsync(p, mh.h_pts, (size_t)mh.n_pts * 12, cudaMemcpyHostToDevice, st), "copy points");
            mh.d_pts = p;
        }
        if (mh.h_tris && mh.n_tris > 0) {
            if (mh.tris_on_device) {
                mh.d_tris = mh.h_tris;
            } else {
                int32_t *p = batch_alloc<int32_t>(b, (size_t)mh.n_tris * 3, err);
                if (!p) return cuda_fail(err, "alloc tris");
                SVO_TRY(cudaMemcpyAsync(p, mh.h_tris, (size_t)mh.n_tris * 12, cudaMemcpyHostToDevice, st),
                        "copy tris");
                mh.d_tris = p;
            }
        }
        b->live.push_back(i);
    }
    const int n = (int)b->live.size();
    if (n == 0) return SVO_OK;
    const MetaLayout ml(n);
    b->box = pinned_acquire(ctx, sizeof(MeshOut) * (size_t)n);
    if (!b->box.p) return fail(SVO_ERR_OUT_OF_MEMORY, "pinned host memory");
    b->out = static_cast<MeshOut *>(b->box.p);
    std::memset(b->box.p, 0, sizeof(MeshOut) * (size_t)n);
    // ---- layout ----
    uint64_t words = 0, blocks = 0, bases = 0, tris = 0;
    uint32_t ctas = 0, max_ctas = 0, bblocks = 0;
    bool any_regions = false;
    HostPack &tables = b->tables;  // mesh table, triangle / CTA / bbox-block offsets
    const size_t p_mesh = tables.add<MeshDev>(n), p_tri = tables.add<uint64_t>(n + 1),
                 p_cta = tables.add<uint32_t>(n + 1), p_bbox = tables.add<uint32_t>(n + 1);
    tables.make();
    b->h_mesh = tables.at<MeshDev>(p_mesh);
    uint64_t *tri_off = tables.at<uint64_t>(p_tri);
    uint32_t *cta_off = tables.at<uint32_t>(p_cta), *bbox_off = tables.at<uint32_t>(p_bbox);
    for (int k = 0; k < n; ++k) {
        MeshHost &mh = b->m[b->live[k]];
        mh.py = make_pyramid(mh.res[0], mh.res[1], mh.res[2]);
        mh.bits_off = words;
        mh.pre_off = blocks;
        mh.base_off = bases;
        words += (mh.py.total_words + 31) / 32 * 32;
        blocks += mh.py.total_blocks;
        bases += 4 * (uint64_t)((mh.py.ctas + 3) & ~3u);
        tri_off[k] = tris;
        cta_off[k] = ctas;
        mh.cta0 = ctas;
        bbox_off[k] = bblocks;
        tris += (uint64_t)mh.n_tris;
        ctas += mh.py.ctas;
        max_ctas = std::max(max_ctas, mh.py.ctas);
        any_regions |= mh.py.words[0] >= kRegionWords;
        bblocks += bbox_blocks(mh.n_pts);
    }
    tri_off[n] = tris;
    cta_off[n] = ctas;
    bbox_off[n] = bblocks;
    // the batch's scratch arrays and its mesh tables: one block, one upload
    uint32_t big_cap = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(2 * tris, 1 << 16), 0x7FFFFFFFu);
    Layout lay;
    const size_t o_meta = lay.add<unsigned char>(ml.bytes);
    const size_t o_bits = lay.add<uint64_t>(words), o_pre = lay.add<uint32_t>(blocks), o_base = lay.add<uint32_t>(bases),
                 o_big = lay.add<uint4>(big_cap),
                 o_rflag = lay.add<uint8_t>(std::max<uint32_t>(ctas, 1)),
                 o_rlist = lay.add<uint32_t>(any_regions ? ctas : 0);
    const size_t o_tables = lay.add<unsigned char>(tables.bytes);
    unsigned char *blk = batch_alloc<unsigned char>(b, lay.bytes, err);
    if (err != cudaSuccess || !blk) return cuda_fail(err, "batch scratch");
    b->bits = reinterpret_cast<uint64_t *>(blk + o_bits);
    b->pre = reinterpret_cast<uint32_t *>(blk + o_pre);
    b->base = reinterpret_cast<uint32_t *>(blk + o_base);
    uint4 *big = reinterpret_cast<uint4 *>(blk + o_big);
    uint8_t *rflag = b->rflag = blk + o_rflag;
    b->rlist = reinterpret_cast<uint32_t *>(blk + o_rlist);
    unsigned char *meta = blk + o_meta;
    GridParams *gp = reinterpret_cast<GridParams *>(meta + ml.gp);
    uint64_t *any = reinterpret_cast<uint64_t *>(meta + ml.any);
    uint32_t *mm = reinterpret_cast<uint32_t *>(meta + ml.mm);
    uint32_t *done = reinterpret_cast<uint32_t *>(meta + ml.done);
    uint32_t *counters = reinterpret_cast<uint32_t *>(meta + ml.counters);
    b->rcount = counters + 2;
    b->dups = reinterpret_cast<unsigned long long *>(meta + ml.dups);
    for (int k = 0; k < n; ++k) {
        const MeshHost &mh = b->m[b->live[k]];
        MeshDev &d = *new (b->h_mesh + k) MeshDev{};
        d.pts = mh.d_pts;
        d.tris = mh.d_tris;
        d.n_pts = mh.n_pts;
        d.n_tris = mh.n_tris;
        for (int a = 0; a < 3; ++a) d.res[a] = mh.res[a];
        d.gp = gp + k;
        d.mm = mm + 8 * k;
        d.bits = b->bits + mh.bits_off;
        d.pre = b->pre + mh.pre_off;
        d.base = b->base + mh.base_off;
        d.bstride = (mh.py.ctas + 3) & ~3u;
        d.any = any + k;
        d.queue = counters;
        d.out = b->out + k;
        d.done = done + k;
        d.py = mh.py;
        d.regions = mh.py.words[0] >= kRegionWords ? 1 : 0;
    }
    unsigned char *dt = blk + o_tables;
    b->d_mesh = reinterpret_cast<MeshDev *>(dt + p_mesh);
    const uint64_t *d_tri_off = reinterpret_cast<const uint64_t *>(dt + p_tri);
    const uint32_t *d_cta_off = reinterpret_cast<const uint32_t *>(dt + p_cta);
    const uint32_t *d_bbox_off = reinterpret_cast<const uint32_t *>(dt + p_bbox);
    if (n > 1)  // a lone mesh's table is passed to the kernels by value
        SVO_TRY(cudaMemcpyAsync(dt, tables.buf.get(), tables.bytes, cudaMemcpyHostToDevice, st), "upload meshes");
    const BatchDev bd{b->d_mesh, n, d_tri_off, d_cta_off, d_bbox_off, rflag, any_regions ? b->rlist : nullptr, b->rcount,
                      n == 1 ? &b->h_mesh[0] : nullptr};
    const bool strict = (b->flags & SVO_FLAG_STRICT_FP) != 0;
    StageTimer tm((b->flags & SVO_FLAG_TIMINGS) != 0);
    for (int attempt = 0; attempt < 2; ++attempt) {
        tm.mark(StageTimer::kStart, st);
        SVO_TRY(cudaMemsetAsync(meta, 0, ml.bytes, st), "memset meta");
        SVO_TRY(launch_front(bd, bblocks, ctas, any_regions, ctx->num_sms, st), "bounding cube");
        tm.mark(StageTimer::kBbox, st);
        if (any_regions) SVO_TRY(launch_regions(bd, (int64_t)tris, ctas, ctx->num_sms, st), "zero regions");
        SVO_TRY(launch_voxelize(bd, (int64_t)tris, strict, b->tune, big, big_cap, counters, ctx->num_sms, st),
                "voxelize");
        tm.mark(StageTimer::kVox, st);
        SVO_TRY(launch_pyramid(bd, ctas, max_ctas, ctx->num_sms, st), "pyramid");
        tm.mark(StageTimer::kPyr, st);
        SVO_TRY(cudaStreamSynchronize(st), "count phase");
        b->pending = false;
        if (b->out[0].queue > big_cap) {  // more big-triangle entries than the queue holds: grow it, redo
            big_cap = b->out[0].queue;
            big = batch_alloc<uint4>(b, big_cap, err);
            if (!big) return cuda_fail(err, "big-triangle queue");
            b->pending = true;
            continue;
        }
        for (int k = 0; k < n; ++k) {
            MeshHost &mh = b->m[b->live[k]];
            mh.gp = b->out[k].gp;
            std::memcpy(mh.totals, b->out[k].totals, sizeof(mh.totals));
            mh.top = b->out[k].any;
        }
        break;
    }
    if (tm.on) {
        b->timed = true;
        b->timings_a[0] = tm.span(StageTimer::kStart, StageTimer::kPyr);
        b->timings_a[1] = tm.span(StageTimer::kStart, StageTimer::kBbox);
        b->timings_a[2] = tm.span(StageTimer::kBbox, StageTimer::kVox);
        b->timings_a[3] = tm.span(StageTimer::kVox, StageTimer::kPyr);
    }
    // ---- level structure per mesh (src/SVO.cu:383-495) ----
    for (int k = 0; k < n; ++k) {
        MeshHost &mh = b->m[b->live[k]];
        if (mh.gp.status & kStatusBadIndex) {
            mesh_error(mh, SVO_ERR_INVALID_ARGUMENT, "triangle index out of range");
            continue;
        }
        if (mh.gp.status & kStatusNonFinite) {
            mesh_error(mh, SVO_ERR_INVALID_ARGUMENT, "non-finite vertex coordinate");
            continue;
        }
        const uint32_t C0 = mh.totals[0];
        if (C0 == 0) {
            mesh_error(mh, SVO_ERR_EMPTY, "no surface voxels");
            continue;
        }
        if (C0 == 1) {
            mesh_error(mh, SVO_ERR_DEGENERATE, "a single surface voxel: the reference's build is undefined");
            continue;
        }
        mh.T = -1;
        for (int l = 0; l < mh.py.levels; ++l)
            if (mh.totals[l] == 1) {
                mh.T = l;
                break;
            }
        if (mh.T < 0) {
            mesh_error(mh, SVO_ERR_CUDA, "octree levels did not converge");
            continue;
        }
        mh.top >>= 3 * mh.T;  // every surface voxel lies under the top node
        for (int l = 0; l <= mh.T; ++l) {
            mh.n_l[l] = l < mh.T ? 8ull * mh.totals[l + 1] : 1ull;
            mh.off[l + 1] = mh.off[l] + mh.n_l[l];
        }
        mh.N = mh.off[mh.T + 1];
        if (mh.N >= 0xFFFFFFFFull) mesh_error(mh, SVO_ERR_UNSUPPORTED, "more than 2^32-2 nodes");
    }
    return SVO_OK;
}

// Bytes of the outputs of one mesh.
uint64_t output_bytes(const MeshHost &mh, uint32_t flags) {
    uint64_t b = mh.N * sizeof(svo_node);
    if (!(flags & SVO_FLAG_NO_VERT_EDGE)) b += mh.N * (8 * sizeof(svo_vertex) + 12 * sizeof(svo_edge));
    if (!(flags & SVO_FLAG_NO_KEYS)) b += (uint64_t)mh.totals[0] * 8;
    return b;
}

AuxStreams *aux_acquire(svo_ctx *ctx) {
    std::lock_guard<std::mutex> lk(ctx->aux_mu);
    if (!ctx->aux_free.empty()) {
        AuxStreams *a = ctx->aux_free.back();
        ctx->aux_free.pop_back();
        return a;
    }
    // The highest stream priority: when a wave's dedup runs beside its
    // emission, the block scheduler places the dedup kernels' CTAs ahead of
    // the emission grid's pending ones instead of after all of them.
    int least = 0, greatest = 0;
    cudaDeviceGetStreamPriorityRange(&least, &greatest);
    auto *a = new AuxStreams();
    bool ok = cudaEventCreateWithFlags(&a->fork, cudaEventDisableTiming) == cudaSuccess;
    for (int i = 0; i < AuxStreams::kCount && ok; ++i)
        ok = cudaStreamCreateWithPriority(&a->s[i], cudaStreamNonBlocking, greatest) == cudaSuccess &&
             cudaEventCreateWithFlags(&a->join[i], cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        for (int i = 0; i < AuxStreams::kCount; ++i) {
            if (a->s[i]) cudaStreamDestroy(a->s[i]);
            if (a->join[i]) cudaEventDestroy(a->join[i]);
        }
        if (a->fork) cudaEventDestroy(a->fork);
        delete a;
        return nullptr;
    }
    ctx->aux_all.push_back(a);
    return a;
}

void aux_release(svo_ctx *ctx, AuxStreams *a) {
    if (!a) return;
    std::lock_guard<std::mutex> lk(ctx->aux_mu);
    ctx->aux_free.push_back(a);
}

size_t arena_round(size_t b) { return (b + 255) / 256 * 256; }

template <class T>
T *arena_take(unsigned char *&at, uint64_t count) {
    T *p = reinterpret_cast<T *>(at);
    at += arena_round(count * sizeof(T));
    return p;
}

// Meshes of at least this many nodes are emitted by a launch of their own.
#ifndef SVO_OWN_EMIT_NODES
#define SVO_OWN_EMIT_NODES (1ull << 17)
#endif
constexpr uint64_t kOwnEmitNodes = SVO_OWN_EMIT_NODES;

// Meshes of up to this many level-0 words (res 256) have their surface-voxel
// keys listed by the launch that lists the other levels; above, a launch of its
// own visits the non-empty level-0 blocks only (k_compact_keys).  Up to res 256
// level 0 is 2 MB and a launch is saved; at res 512 it is 16 MB that hold few
// bits.  Builds of an icosphere, both ways (us, listed with the levels / a launch
// of its own): res 64 70 / 70, res 128 89 / 93 (without vertices and edges 73 /
// 81), res 256 148 / 149 (94 / 95), res 512 394 / 387 (179 / 174).
constexpr uint64_t kDirectKeyWords = 1ull << 18;

// Phase B for meshes [first, first + count).
int batch_phase_b(svo_batch *b, int first, int count, svo_result **out, int *status_out) {
    svo::host::TraceRange trace("svo: emission wave (codes, nodes, vertices, edges, dedup)");
    svo_ctx *ctx = b->ctx;
    cudaStream_t st = b->st;
    const uint32_t flags = b->flags;
    const bool ve = !(flags & SVO_FLAG_NO_VERT_EDGE);
    const bool want_keys = !(flags & SVO_FLAG_NO_KEYS);
    SVO_TRY(cudaSetDevice(ctx->device), "cudaSetDevice");
    std::vector<int> wave;   // batch mesh indices emitted now
    std::vector<int> dev_k;  // their index in b->live
    for (int i = first; i < first + count; ++i) {
        out[i - first] = nullptr;
        MeshHost &mh = b->m[i];
        if (mh.status == SVO_OK && mh.emitted) mesh_error(mh, SVO_ERR_INVALID_ARGUMENT, "mesh already emitted");
        if (mh.status != SVO_OK) continue;
        wave.push_back(i);
        dev_k.push_back((int)(std::find(b->live.begin(), b->live.end(), i) - b->live.begin()));
    }
    const int n = (int)wave.size();
    std::vector<svo_result *> res(n, nullptr);
    int rc = SVO_OK;
    auto check = [&](cudaError_t e, const char *what) {
        if (e != cudaSuccess && rc == SVO_OK) rc = cuda_fail(e, what);
    };
    Scratch S{ctx->pool, st};
    StageTimer tm((flags & SVO_FLAG_TIMINGS) != 0);
    auto free_results = [&]() {
        for (svo_result *&r : res) {
            svo_result_free(r);
            r = nullptr;
        }
    };
    if (n > 0) {
        b->pending = true;
        // The wave body: an error return from it still reaches the per-mesh
        // status loop below, which marks every mesh of the wave as failed.
        const int wave_rc = [&]() -> int {
            cudaError_t err = cudaSuccess;
            // The dedup keys read only the bitmaps and code lists: they run on
            // a stream of their own.  Of grids up to 1024 the first step (the
            // level-1 candidate bitmap, from the bitmaps alone) is forked here and
            // runs while the host prepares the wave; the rest, and the whole dedup
            // of larger grids, follows the code lists and runs beside the
            // emission.  The wave joins the stream before returning.
            const bool dd = (flags & SVO_FLAG_DEDUP) != 0;
            AuxStreams *dset = dd ? aux_acquire(ctx) : nullptr;
            const cudaStream_t ds = dset ? dset->s[0] : st;
            auto join_dedup = [&]() {
                if (!dset) return;
                check(cudaEventRecord(dset->join[0], ds), "join");
                check(cudaStreamWaitEvent(st, dset->join[0], 0), "join");
                aux_release(ctx, dset);
                dset = nullptr;
            };
            std::vector<DedupRun *> druns(n, nullptr);
            std::vector<int> drc(n, SVO_OK);
            std::vector<std::string> dmsg(n);
            std::vector<char> dstarted(n, 0);
            auto dedup_start = [&](int j) {  // the first step of mesh j's dedup (bitmaps only)
                dstarted[j] = 1;
                const MeshHost &mh = b->m[wave[j]];
                const MeshDev &md = b->h_mesh[dev_k[j]];
                const uint32_t R = 1u << (mh.py.grid_levels - 1);
                const uint64_t *bits[kMaxLevels];
                uint32_t sides[kMaxLevels];
                for (int l = 0; l <= mh.T && l < kMaxLevels; ++l) {
                    bits[l] = md.bits + mh.py.woff[l];
                    sides[l] = std::max<uint32_t>(1u, R >> l);
                }
                drc[j] = dedup_begin(ctx->pool, ds, mh.T, bits, sides, ctx->num_sms, b->out[dev_k[j]].dedup, &druns[j]);
                if (drc[j] != SVO_OK) dmsg[j] = svo_last_error();
            };
            struct DedupGuard {  // on every exit: unfinished runs freed, the dedup stream joined
                std::vector<DedupRun *> &runs;
                decltype(join_dedup) &join;
                ~DedupGuard() {
                    for (DedupRun *&r : runs) {
                        dedup_abort(r);
                        r = nullptr;
                    }
                    join();
                }
            } dguard{druns, join_dedup};
            if (dd) {
                if (dset) {
                    check(cudaEventRecord(dset->fork, st), "fork");
                    check(cudaStreamWaitEvent(ds, dset->fork, 0), "fork");
                }
                tm.mark(StageTimer::kDedup0, ds);
                // early starts hold their candidate bitmaps (R^3 / 8 bytes each) until their
                // finish: up to 4 GiB of them; the other meshes start just before they
                // finish, and so do grids above 1024: their candidate pass (110 us at res
                // 2048) holds the compaction up (60 us beside it, 7 without), while their
                // dedup ends long before the emission.  Whole builds, started early / late
                // (us): heightfield at res 2048 4,035 / 4,010; at res 1024 and below both
                // the same (heightfield at res 1024 980 / 985, icosphere 2,477 / 2,476, at
                // res 512 692 / 693), and the early start spares the emission's memory path
                uint64_t early = 0;
                for (int j = 0; j < n; ++j) {
                    const MeshHost &mh = b->m[wave[j]];
                    const uint64_t R = 1ull << (mh.py.grid_levels - 1);
                    if (R > 1024) continue;
                    if (early + R * R * R / 8 > (4ull << 30)) break;
                    early += R * R * R / 8;
                    dedup_start(j);
                }
            }
            // outputs, code lists, job tables
            std::vector<CompactJob> region_jobs;  // region-mode meshes' levels 1-2
            std::vector<std::pair<uint32_t, uint32_t>> region_range;  // first region, regions
            auto regions = [](const MeshHost &mh) { return mh.py.words[0] >= kRegionWords; };
            auto direct_keys = [&](const MeshHost &mh) {
                return want_keys && (mh.T < 3 || mh.py.words[0] <= kDirectKeyWords);
            };
            auto own_emit = [&](const MeshHost &mh) { return n == 1 || mh.N >= kOwnEmitNodes; };
            int n_jobs = 0, n_kjobs = 0, n_own = 0;
            for (int j = 0; j < n; ++j) {
                const MeshHost &mh = b->m[wave[j]];
                n_jobs += regions(mh) ? (direct_keys(mh) ? 1 : 0) + (mh.T >= 3 ? 1 : 0) : 1;
                n_kjobs += want_keys && !direct_keys(mh) ? 1 : 0;
                n_own += own_emit(mh) ? 1 : 0;
            }
            const int n_small = n - n_own;
            // the tables of the wave's kernels: compaction jobs, key jobs, emission
            // parameters of the meshes that share one emission launch
            HostPack wt;
            const size_t p_jobs = wt.add<CompactJob>(n_jobs), p_woff = wt.add<uint64_t>(n_jobs + 1),
                         p_kjobs = wt.add<KeyJob>(n_kjobs), p_boff = wt.add<uint64_t>(n_kjobs + 1),
                         p_eps = wt.add<EmitParams>(n_small), p_offs = wt.add<uint64_t>(n_small + 1);
            wt.make();
            CompactJob *jobs = wt.at<CompactJob>(p_jobs);
            uint64_t *word_off = wt.at<uint64_t>(p_woff);
            KeyJob *kjobs = wt.at<KeyJob>(p_kjobs);
            uint64_t *blk_off = wt.at<uint64_t>(p_boff);
            EmitParams *ep_small = wt.at<EmitParams>(p_eps);
            uint64_t *off_small = wt.at<uint64_t>(p_offs);
            word_off[0] = blk_off[0] = off_small[0] = 0;
            std::vector<EmitParams> ep_own(n_own);  // large meshes' launches of their own take them by value
            std::vector<EmitParams *> ep(n);        // in one of the two
            uint64_t ktot = 0;
            std::vector<uint64_t> kbase(n);
            for (int j = 0; j < n; ++j) {
                const MeshHost &mh = b->m[wave[j]];
                kbase[j] = ktot;
                for (int l = 1; l <= mh.T; ++l) ktot += mh.totals[l];
            }
            // per-word ranks of levels >= 1 (k_compact writes them, rank lookups read them)
            uint64_t wtot = 0;
            std::vector<uint64_t> wbase(n);
            for (int j = 0; j < n; ++j) {
                const MeshHost &mh = b->m[wave[j]];
                wbase[j] = wtot;
                wtot += mh.py.woff[mh.T] + mh.py.words[mh.T] - mh.py.woff[1];
            }
            // code lists, word ranks: one block
            Layout wl;
            const size_t o_K = wl.add<uint64_t>(ktot + 1), o_WP = wl.add<uint32_t>(wtot + 1);
            unsigned char *wblk = S.get<unsigned char>(wl.bytes);
            if (!wblk) return cuda_fail(S.err, "wave scratch");
            uint64_t *K = reinterpret_cast<uint64_t *>(wblk + o_K);
            uint32_t *WP = reinterpret_cast<uint32_t *>(wblk + o_WP);
            // one block for the output arrays of the whole wave
            size_t arena_bytes = 0;
            for (int j = 0; j < n; ++j) {
                const MeshHost &mh = b->m[wave[j]];
                arena_bytes += arena_round(mh.N * sizeof(svo_node));
                if (ve) arena_bytes += arena_round(mh.N * 8 * sizeof(svo_vertex)) + arena_round(mh.N * 12 * sizeof(svo_edge));
                if (want_keys) arena_bytes += arena_round((size_t)mh.totals[0] * 8);
            }
            svo_arena *arena = new svo_arena();
            arena->refs = 1;  // the wave's own reference, dropped below
            if (pool_malloc(&arena->base, std::max<size_t>(arena_bytes, 256), ctx->out_pool, st) != cudaSuccess) {
                delete arena;
                cudaGetLastError();
                return fail(SVO_ERR_OUT_OF_MEMORY, "wave outputs: %zu bytes", arena_bytes);
            }
            unsigned char *arena_at = static_cast<unsigned char *>(arena->base);
            auto drop_arena = [&]() {
                if (arena && arena->refs.fetch_sub(1) == 1) {
                    cudaFreeAsync(arena->base, st);
                    delete arena;
                }
                arena = nullptr;
            };
            for (int j = 0, at_job = 0, at_kjob = 0, at_own = 0, at_small = 0; j < n; ++j) {
                const MeshHost &mh = b->m[wave[j]];
                const MeshDev &md = b->h_mesh[dev_k[j]];
                svo_result *r = new svo_result();
                res[j] = r;
                r->device = ctx->device;
                r->stream = st;
                r->out_keep = ctx->out_keep;
                r->copies = ctx->copies;
                r->depth = mh.T + 1;
                for (int l = 0; l <= mh.T; ++l) r->level_counts.push_back((int64_t)mh.n_l[l]);
                for (int a = 0; a < 3; ++a) {
                    r->bbox.min[a] = mh.gp.bbox[a];
                    r->bbox.max[a] = mh.gp.bbox[3 + a];
                    r->bbox.width[a] = mh.gp.bbox[6 + a];
                    r->unit[a] = mh.gp.unit[a];
                }
                r->n_nodes = mh.N;
                r->nodes = arena_take<svo_node>(arena_at, mh.N);
                if (ve) {
                    r->verts = arena_take<svo_vertex>(arena_at, mh.N * 8);
                    r->edges = arena_take<svo_edge>(arena_at, mh.N * 12);
                    r->n_verts = mh.N * 8;
                    r->n_edges = mh.N * 12;
                }
                if (want_keys) {
                    r->keys = arena_take<uint64_t>(arena_at, mh.totals[0]);
                    r->n_keys = mh.totals[0];
                }
                r->arena = arena;
                r->own = 0x70;
                arena->refs.fetch_add(1);
                // compaction jobs: levels 1..T into K, level 0 into the keys
                CompactJob job{};
                job.bits = md.bits;
                job.rank = RankDev{md.pre, md.base, md.bstride};
                job.py = mh.py;
                job.l0 = 1;
                job.l1 = mh.T + 1;
                job.out = K + kbase[j];
                job.wpre = WP + wbase[j];
                uint64_t ko = 0;
                for (int l = 1; l <= mh.T; ++l) {
                    job.koff[l] = ko;
                    ko += mh.totals[l];
                }
                if (regions(mh)) {
                    // region mode: levels 1-2 region by region (k_compact_regions);
                    // level 3 words of unflagged regions are empty, not read
                    job.rflag = b->rflag + mh.cta0;
                    region_jobs.push_back(job);
                    region_range.push_back({mh.cta0, mh.py.ctas});
                }
                if (direct_keys(mh)) {
                    job.l0 = 0;
                    job.keys = r->keys;
                } else if (want_keys) {
                    // the level-3 code list is the list of non-empty level-0 blocks
                    new (kjobs + at_kjob) KeyJob{md.bits, job.rank, job.out + job.koff[3], r->keys};
                    blk_off[at_kjob + 1] = blk_off[at_kjob] + mh.totals[3];
                    ++at_kjob;
                }
                auto add_job = [&](int l0, int l1) {
                    if (l0 >= l1) return;
                    job.l0 = l0;
                    job.l1 = l1;
                    new (jobs + at_job) CompactJob(job);
                    word_off[at_job + 1] = word_off[at_job] + mh.py.woff[l1 - 1] + mh.py.words[l1 - 1] - mh.py.woff[l0];
                    ++at_job;
                };
                if (job.rflag) {  // levels 1-2 have a launch of their own (region_jobs)
                    if (job.l0 == 0) add_job(0, 1);
                    add_job(3, mh.T + 1);
                } else {
                    add_job(job.l0, mh.T + 1);
                }
                // emission parameters
                const bool own = own_emit(mh);
                ep[j] = own ? &ep_own[at_own++] : new (ep_small + at_small) EmitParams{};
                if (!own) {
                    off_small[at_small + 1] = off_small[at_small] + (mh.N + 31) / 32 * 32;
                    ++at_small;
                }
                EmitParams &P = *ep[j];
                P.T = mh.T;
                P.N = (uint32_t)mh.N;
                P.flags = flags;
                const uint32_t R = 1u << (mh.py.grid_levels - 1);
                float w = mh.gp.unit[0];  // unitVoxelSize.x doubled per level (src/SVO.cu:351,483)
                for (int l = 0; l <= mh.T; ++l) {
                    P.lv[l].off = (uint32_t)mh.off[l];
                    P.lv[l].n = (uint32_t)mh.n_l[l];
                    P.lv[l].K1 = job.out + (l < mh.T ? job.koff[l + 1] : job.koff[mh.T]);
                    P.lv[l].bits = md.bits + mh.py.woff[l];
                    P.lv[l].wpre = l >= 1 ? job.wpre + (mh.py.woff[l] - mh.py.woff[1]) : nullptr;
                    P.lv[l].side = std::max<uint32_t>(1u, R >> l);
                    P.lv[l].width = w;
                    w = w * 2.0f;
                }
                P.gp = md.gp;
                P.nodes = r->nodes;
                P.verts = ve ? r->verts : nullptr;
                P.edges = ve ? r->edges : nullptr;
                P.dups = b->dups + 2 * dev_k[j];
                P.dup_flag = &b->out[dev_k[j]].dup;
            }
            if (err != cudaSuccess) {
                free_results();
                drop_arena();
                return cuda_fail(err, "output allocation");
            }
            // one upload of the tables; what one kernel takes by value (a lone mesh's
            // jobs and emission) needs none
            const bool lone_job = n_jobs == 1, lone_keys = n_kjobs == 1;
            unsigned char *dwt = n_jobs > 1 || n_kjobs > 1 || n_small > 0 ? S.get<unsigned char>(wt.bytes) : nullptr;
            if (S.err != cudaSuccess) {
                free_results();
                drop_arena();
                return cuda_fail(S.err, "wave tables");
            }
            const CompactJob *d_jobs = reinterpret_cast<const CompactJob *>(dwt + p_jobs);
            const uint64_t *d_word_off = reinterpret_cast<const uint64_t *>(dwt + p_woff);
            const KeyJob *d_kjobs = reinterpret_cast<const KeyJob *>(dwt + p_kjobs);
            const uint64_t *d_blk_off = reinterpret_cast<const uint64_t *>(dwt + p_boff);
            if (dwt) check(cudaMemcpyAsync(dwt, wt.buf.get(), wt.bytes, cudaMemcpyHostToDevice, st), "upload");
            tm.mark(StageTimer::kCompact0, st);
            check(launch_compact(CompactBatch{d_jobs, n_jobs, d_word_off}, lone_job ? jobs : nullptr, word_off[n_jobs], st),
                  "compact");
            // The keys need the level-3 lists and nothing needs the keys: they run on
            // a stream of their own beside the remaining lists (320 triangles at res 512
            // 420 us before, 414 this way; heightfield at res 2048, with the later dedup
            // start above, 4,076 and 4,046).  The auxiliary streams have the highest
            // priority, so the keys go before the emission rather than beside it: at res
            // 2048 they take 54 us, and the emission starts 28 us after the last list.
            AuxStreams *kset = n_kjobs == 0 ? nullptr : aux_acquire(ctx);
            const cudaStream_t ks = kset ? kset->s[0] : st;
            if (kset) {
                check(cudaEventRecord(kset->fork, st), "fork");
                check(cudaStreamWaitEvent(ks, kset->fork, 0), "fork");
            }
            if (n_kjobs > 0)
                check(launch_compact_keys(KeyBatch{d_kjobs, n_kjobs, d_blk_off}, lone_keys ? kjobs : nullptr, blk_off[n_kjobs],
                                          ks),
                      "keys");
            if (n_kjobs > 0) tm.mark(StageTimer::kKeys, ks);
            for (size_t i = 0; i < region_jobs.size(); ++i)
                check(launch_compact_regions(region_jobs[i], b->rlist, b->rcount, region_range[i].first,
                                             region_range[i].second, ctx->num_sms, st),
                      "compact");
            tm.mark(StageTimer::kCompact, st);
            // the dedup's coarse marks, states and keys need the code lists
            if (dset) {
                check(cudaEventRecord(dset->fork, st), "fork");
                check(cudaStreamWaitEvent(ds, dset->fork, 0), "fork");
            }
            // With two or more emission launches of their own, they spread round-robin
            // over the build stream and three more, so that one kernel's tail overlaps the next.
            AuxStreams *aux = n_own >= 2 ? aux_acquire(ctx) : nullptr;
            if (aux) {
                check(cudaEventRecord(aux->fork, st), "fork");
                for (int i = 0; i < AuxStreams::kCount; ++i) check(cudaStreamWaitEvent(aux->s[i], aux->fork, 0), "fork");
            }
            int k_own = 0;
            for (int j = 0; j < n; ++j) {
                if (own_emit(b->m[wave[j]])) {
                    const int lane = aux ? k_own % (AuxStreams::kCount + 1) : 0;
                    cudaStream_t es = lane == 0 ? st : aux->s[lane - 1];
                    ++k_own;
                    check(launch_emit(EmitBatch{nullptr, 1, nullptr}, ep[j], ep[j]->N, flags, ctx->num_sms, es), "emit");
                }
            }
            if (aux) {
                for (int i = 0; i < AuxStreams::kCount; ++i) {
                    check(cudaEventRecord(aux->join[i], aux->s[i]), "join");
                    check(cudaStreamWaitEvent(st, aux->join[i], 0), "join");
                }
                aux_release(ctx, aux);
            }
            if (n_small > 0)
                check(launch_emit(EmitBatch{reinterpret_cast<const EmitParams *>(dwt + p_eps), n_small,
                                            reinterpret_cast<const uint64_t *>(dwt + p_offs)},
                                  nullptr, off_small[n_small], flags, ctx->num_sms, st),
                      "emit");
            tm.mark(StageTimer::kEmit, st);
            // Dedup of every mesh on the forked stream (its host-side waits
            // overlap the emission running on the GPU); statuses are applied
            // after the emission's own checks.
            if (dd) {
                for (int j = 0; j < n && rc == SVO_OK; ++j) {
                    if (b->m[wave[j]].status != SVO_OK) continue;
                    if (!dstarted[j]) dedup_start(j);
                    if (!druns[j]) continue;
                    drc[j] = dedup_finish(druns[j], ctx->out_pool, *ep[j], res[j]->n_dedup, res[j]->dedup);
                    druns[j] = nullptr;
                    if (drc[j] != SVO_OK) dmsg[j] = svo_last_error();
                }
                tm.mark(StageTimer::kDedup, ds);
            }
            join_dedup();
            if (kset) {
                check(cudaEventRecord(kset->join[0], ks), "join");
                check(cudaStreamWaitEvent(st, kset->join[0], 0), "join");
                aux_release(ctx, kset);
            }
            check(cudaStreamSynchronize(st), "emit phase");
            tm.mark(StageTimer::kUnique0, st);  // (the wait above is for the dedup and the keys as well)
            bool more = false;  // work launched after this wait
            // the counters of all meshes at once, when some mesh has duplicates (a read
            // and a wait for each mesh: 100 meshes far from the origin at res 64 9.5 ms,
            // 8.15 this way)
            std::vector<unsigned long long> h_dups;
            if (ve && std::any_of(dev_k.begin(), dev_k.end(), [&](int k) { return b->out[k].dup != 0; })) {
                h_dups.resize(2 * b->live.size());
                check(cudaMemcpyAsync(h_dups.data(), b->dups, h_dups.size() * sizeof(h_dups[0]), cudaMemcpyDeviceToHost, st),
                      "read dups");
                check(cudaStreamSynchronize(st), "read dups");
                more = true;
            }
            for (int j = 0; j < n && rc == SVO_OK; ++j) {
                MeshHost &mh = b->m[wave[j]];
                svo_result *r = res[j];
                if (mh.T == 0 || (mh.top & 7) != 0) {
                    mesh_error(mh, SVO_ERR_DEGENERATE,
                               "single top-level node with a non-zero octant: undefined in the reference");
                    continue;
                }
                const unsigned long long vdup = h_dups.empty() ? 0 : h_dups[2 * dev_k[j]],
                                         edup = h_dups.empty() ? 0 : h_dups[2 * dev_k[j] + 1];
                if (vdup || edup) {
                    // consecutive duplicates (degenerate widths or absorbed
                    // coordinates): compact both arrays as thrust::unique does
                    const uint64_t nv = mh.N * 8, ne = mh.N * 12;
                    const uint64_t tiles = (std::max(nv, ne) + kUniqueTile - 1) / kUniqueTile;
                    Scratch U{ctx->pool, st};
                    uint32_t *tc = U.get<uint32_t>(tiles), *tp = U.get<uint32_t>(tiles + 1);
                    unsigned long long *ss = U.get<unsigned long long>(scan_scratch_words(tiles));
                    uint32_t *ustat = U.get<uint32_t>(1);
                    svo_vertex *v2 = vdup ? pool_alloc<svo_vertex>(ctx->out_pool, st, nv, err) : nullptr;
                    svo_edge *e2 = edup ? pool_alloc<svo_edge>(ctx->out_pool, st, ne, err) : nullptr;
                    if (U.err != cudaSuccess || err != cudaSuccess) {
                        rc = cuda_fail(U.err != cudaSuccess ? U.err : err, "unique scratch");
                        break;
                    }
                    check(cudaMemsetAsync(ustat, 0, 4, st), "memset");
                    uint32_t cv = 0, ce = 0;
                    if (v2) {
                        check(launch_unique_vertices(r->verts, nv, v2, tc, tp, ss, ustat, st), "unique v");
                        check(cudaMemcpyAsync(&cv, tp + (nv + kUniqueTile - 1) / kUniqueTile, 4, cudaMemcpyDeviceToHost,
                                              st), "read");
                        check(cudaStreamSynchronize(st), "unique v");
                    }
                    if (e2) {
                        check(launch_unique_edges(r->edges, ne, e2, tc, tp, ss, ustat, st), "unique e");
                        check(cudaMemcpyAsync(&ce, tp + (ne + kUniqueTile - 1) / kUniqueTile, 4, cudaMemcpyDeviceToHost,
                                              st), "read");
                        check(cudaStreamSynchronize(st), "unique e");
                    }
                    if (v2) {
                        if (r->own & 2) cudaFreeAsync(r->verts, st);
                        r->verts = v2;
                        r->own |= 2;
                        r->n_verts = cv;
                    }
                    if (e2) {
                        if (r->own & 4) cudaFreeAsync(r->edges, st);
                        r->edges = e2;
                        r->own |= 4;
                        r->n_edges = ce;
                    }
                }
            }
            tm.mark(StageTimer::kUnique, st);
            if (more) check(cudaStreamSynchronize(st), "unique phase");
            b->pending = rc != SVO_OK;
            for (int j = 0; j < n; ++j) {
                MeshHost &mh = b->m[wave[j]];
                if (mh.status == SVO_OK && drc[j] != SVO_OK) mesh_error(mh, drc[j], dmsg[j].c_str());
            }
            tm.mark(StageTimer::kEnd, st);
            if (tm.on) cudaEventSynchronize(tm.ev[StageTimer::kEnd]);
            drop_arena();
            return SVO_OK;
        }();
        if (wave_rc != SVO_OK && rc == SVO_OK) rc = wave_rc;
    }
    int first_err = rc;
    for (int j = 0; j < n; ++j) {
        MeshHost &mh = b->m[wave[j]];
        if (rc != SVO_OK && mh.status == SVO_OK) mesh_error(mh, rc, svo_last_error());
        if (mh.status == SVO_OK) {
            mh.emitted = true;
            svo_result *r = res[j];
            if (tm.on && b->timed) {
                r->n_timings = 9;
                r->timings[1] = b->timings_a[1];
                r->timings[2] = b->timings_a[2];
                r->timings[3] = b->timings_a[3];
                r->timings[5] = std::max(tm.span(StageTimer::kCompact0, StageTimer::kCompact),
                                         tm.span(StageTimer::kCompact0, StageTimer::kKeys));
                r->timings[6] = tm.span(StageTimer::kCompact, StageTimer::kEmit);
                r->timings[7] = tm.span(StageTimer::kUnique0, StageTimer::kUnique);
                r->timings[8] = tm.span(StageTimer::kDedup0, StageTimer::kDedup);
                r->timings[0] = b->timings_a[0] + tm.span(StageTimer::kCompact0, StageTimer::kEnd);
            }
            out[wave[j] - first] = r;
        } else {
            svo_result_free(res[j]);
        }
    }
    for (int i = first; i < first + count; ++i) {
        if (status_out) status_out[i - first] = b->m[i].status;
        if (b->m[i].status != SVO_OK && first_err == SVO_OK) first_err = b->m[i].status;
    }
    if (first_err != SVO_OK) {
        for (int i = first; i < first + count; ++i)
            if (b->m[i].status != SVO_OK) {
                g_err = b->m[i].error;
                break;
            }
    }
    return first_err;
}

void batch_destroy(svo_batch *b) {
    if (!b) return;
    cudaSetDevice(b->ctx->device);
    if (b->pending) cudaStreamSynchronize(b->st);
    batch_release(b);  // stream-ordered frees
    delete b;
}

// tune: the voxelizer split to use (null: the context's, read once here).
int batch_create(svo_ctx *ctx, const svo_mesh_desc *descs, int n, uint32_t flags, cudaStream_t st,
                 svo_batch **out, const VoxTuning *tune = nullptr) {
    svo_batch *b = new svo_batch();
    b->ctx = ctx;
    b->st = st;
    b->flags = flags;
    if (tune) {
        b->tune = *tune;
    } else {
        std::lock_guard<std::mutex> lk(ctx->tune_mu);
        b->tune = ctx->tune;
    }
    b->m.resize(n);
    for (int i = 0; i < n; ++i) {
        MeshHost &mh = b->m[i];
        mh.h_pts = descs[i].points;
        mh.n_pts = descs[i].n_points;
        mh.h_tris = descs[i].tris;
        mh.n_tris = descs[i].tris ? descs[i].n_tris : 0;
        for (int a = 0; a < 3; ++a) mh.res[a] = descs[i].res[a];
    }
    const int rc = batch_phase_a(b);
    if (rc != SVO_OK) {
        const std::string msg = g_err;
        batch_destroy(b);
        g_err = msg;
        return rc;
    }
    *out = b;
    return SVO_OK;
}

}  // namespace

extern "C" {

const char *svo_last_error(void) { return g_err.c_str(); }

int svo_ctx_create(int device, svo_ctx **out) {
    if (!out) return fail(SVO_ERR_INVALID_ARGUMENT, "null output");
    *out = nullptr;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0) return fail(SVO_ERR_CUDA, "no CUDA device: %s", cudaGetErrorString(e));
    if (device < 0 || device >= n) return fail(SVO_ERR_INVALID_ARGUMENT, "bad device %d", device);
    SVO_TRY(cudaSetDevice(device), "cudaSetDevice");
    cudaDeviceProp prop;
    SVO_TRY(cudaGetDeviceProperties(&prop, device), "properties");
    if (prop.major < 10) return fail(SVO_ERR_UNSUPPORTED, "needs a Blackwell (sm_100) device, got sm_%d%d", prop.major, prop.minor);
    svo_ctx *c = new svo_ctx();
    c->device = device;
    c->num_sms = prop.multiProcessorCount;
    c->copies = svo::host::copy_pool_create(device);
    // Two pools of its own: per-build scratch, and result arrays (kept apart
    // so scratch never splits their blocks).  Freed blocks stay cached.
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    uint64_t keep = UINT64_MAX;
    for (cudaMemPool_t *pp : {&c->pool, &c->out_pool}) {
        if (cudaMemPoolCreate(pp, &props) != cudaSuccess ||
            cudaMemPoolSetAttribute(*pp, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            svo_ctx_destroy(c);
            cudaGetLastError();
            return fail(SVO_ERR_CUDA, "memory pool");
        }
    }
    c->out_keep = std::make_shared<OutPool>(device, c->out_pool);
    *out = c;
    return SVO_OK;
}

int svo_ctx_reserve(svo_ctx *ctx, uint64_t result_bytes, uint64_t scratch_bytes, void *stream) {
    if (!ctx) return fail(SVO_ERR_INVALID_ARGUMENT, "null context");
    SVO_TRY(cudaSetDevice(ctx->device), "cudaSetDevice");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const std::pair<cudaMemPool_t, uint64_t> want[2] = {{ctx->out_pool, result_bytes}, {ctx->pool, scratch_bytes}};
    for (const auto &w : want) {
        if (w.second == 0) continue;
        void *p = nullptr;
        if (cudaMallocFromPoolAsync(&p, w.second, w.first, st) != cudaSuccess) {
            cudaGetLastError();
            return fail(SVO_ERR_OUT_OF_MEMORY, "cannot reserve %llu bytes", (unsigned long long)w.second);
        }
        SVO_TRY(cudaFreeAsync(p, st), "free");
    }
    SVO_TRY(cudaStreamSynchronize(st), "reserve");
    return SVO_OK;
}

int svo_ctx_device(const svo_ctx *ctx, int *device) {
    if (!ctx || !device) return fail(SVO_ERR_INVALID_ARGUMENT, "null argument");
    *device = ctx->device;
    return SVO_OK;
}

// Results may outlive the context: they hold the pool of their arrays (OutPool).
void svo_ctx_destroy(svo_ctx *ctx) {
    if (!ctx) return;
    cudaSetDevice(ctx->device);
    for (AuxStreams *a : ctx->aux_all) {
        for (int i = 0; i < AuxStreams::kCount; ++i) {
            cudaStreamDestroy(a->s[i]);
            cudaEventDestroy(a->join[i]);
        }
        cudaEventDestroy(a->fork);
        delete a;
    }
    for (svo_ctx::Pinned &b : ctx->pinned_free) cudaFreeHost(b.p);
    if (ctx->pool) cudaMemPoolDestroy(ctx->pool);
    if (ctx->out_keep) {
        if (ctx->out_keep.use_count() > 1) ctx->out_keep->outlived = true;
    } else if (ctx->out_pool) {
        cudaMemPoolDestroy(ctx->out_pool);
    }
    delete ctx;
}

int svo_ctx_set_tuning(svo_ctx *ctx, const svo_tuning *t) {
    if (!ctx || !t) return fail(SVO_ERR_INVALID_ARGUMENT, "null argument");
    if (t->warp_max == 0) return fail(SVO_ERR_INVALID_ARGUMENT, "warp_max must be positive");
    if (t->serial_max > (1u << 16)) return fail(SVO_ERR_INVALID_ARGUMENT, "serial_max must be <= 65536");
    if (t->serial_packed > 1) return fail(SVO_ERR_INVALID_ARGUMENT, "serial_packed must be 0 or 1");
    std::lock_guard<std::mutex> lk(ctx->tune_mu);
    ctx->tune.serial_max = t->serial_max;
    ctx->tune.warp_max = t->warp_max;
    ctx->tune.split = t->split;
    ctx->tune.inplace_max = t->inplace_max;
    ctx->tune.serial_packed = t->serial_packed;
    return SVO_OK;
}

int svo_ctx_get_tuning(const svo_ctx *ctx, svo_tuning *t) {
    if (!ctx || !t) return fail(SVO_ERR_INVALID_ARGUMENT, "null argument");
    std::lock_guard<std::mutex> lk(const_cast<svo_ctx *>(ctx)->tune_mu);
    t->serial_max = ctx->tune.serial_max;
    t->warp_max = ctx->tune.warp_max;
    t->split = ctx->tune.split;
    t->inplace_max = ctx->tune.inplace_max;
    t->serial_packed = ctx->tune.serial_packed;
    return SVO_OK;
}

int svo_ctx_memory(const svo_ctx *ctx, uint64_t *scratch_used, uint64_t *result_used) {
    if (!ctx) return fail(SVO_ERR_INVALID_ARGUMENT, "null context");
    uint64_t a = 0, b = 0;  // the attribute is a 64-bit unsigned count
    SVO_TRY(cudaMemPoolGetAttribute(ctx->pool, cudaMemPoolAttrUsedMemCurrent, &a), "pool attribute");
    SVO_TRY(cudaMemPoolGetAttribute(ctx->out_pool, cudaMemPoolAttrUsedMemCurrent, &b), "pool attribute");
    if (scratch_used) *scratch_used = (uint64_t)a;
    if (result_used) *result_used = (uint64_t)b;
    return SVO_OK;
}

int svo_selftest_scan_timeout(svo_ctx *ctx, void *stream) {
    if (!ctx) return fail(SVO_ERR_INVALID_ARGUMENT, "null context");
    SVO_TRY(cudaSetDevice(ctx->device), "cudaSetDevice");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint64_t n = 3 * 4096 + 17;  // four tiles of the single-pass scan
    Scratch S{ctx->pool, st};
    uint32_t *in = S.get<uint32_t>(n), *out = S.get<uint32_t>(n + 1), *status = S.get<uint32_t>(1);
    unsigned long long *scratch = S.get<unsigned long long>(scan_stalled_scratch_words(n));
    if (S.err != cudaSuccess) return cuda_fail(S.err, "self-test scratch");
    SVO_TRY(cudaMemsetAsync(in, 0, n * sizeof(uint32_t), st), "memset");
    SVO_TRY(cudaMemsetAsync(status, 0, sizeof(uint32_t), st), "memset");
    SVO_TRY(launch_scan_stalled(in, out, n, scratch, status, 1 << 12, st), "stalled scan");
    uint32_t h = 0;
    SVO_TRY(cudaMemcpyAsync(&h, status, sizeof(h), cudaMemcpyDeviceToHost, st), "read status");
    SVO_TRY(cudaStreamSynchronize(st), "stalled scan");
    if (h & kStatusScanTimeout) return fail(SVO_ERR_DEVICE_TIMEOUT, "scan look-back timed out (self-test)");
    return SVO_OK;
}

int svo_build(svo_ctx *ctx, const float *points, int64_t n_points, const int32_t *tris, int64_t n_tris,
              int res_x, int res_y, int res_z, uint32_t flags, void *stream, svo_result **out) {
    if (!ctx || !out) return fail(SVO_ERR_INVALID_ARGUMENT, "null context or output");
    *out = nullptr;
    svo_mesh_desc d{points, n_points, tris, n_tris, {res_x, res_y, res_z}, flags};
    svo_batch *b = nullptr;
    int rc = batch_create(ctx, &d, 1, flags, static_cast<cudaStream_t>(stream), &b);
    if (rc != SVO_OK) return rc;
    int st = SVO_OK;
    rc = batch_phase_b(b, 0, 1, out, &st);
    const std::string msg = g_err;
    batch_destroy(b);
    g_err = msg;
    return rc != SVO_OK ? rc : st;
}

int svo_build_batch(svo_ctx *ctx, const svo_mesh_desc *descs, int n, void *stream, svo_result **out,
                    int *status_out) {
    if (!ctx || (!descs && n > 0) || !out) return fail(SVO_ERR_INVALID_ARGUMENT, "null argument");
    // one batch per distinct flags value (the kernels are specialised on them)
    std::vector<uint32_t> kinds;
    for (int i = 0; i < n; ++i)
        if (std::find(kinds.begin(), kinds.end(), descs[i].flags) == kinds.end()) kinds.push_back(descs[i].flags);
    int first = SVO_OK;
    std::string first_msg;
    for (uint32_t f : kinds) {
        std::vector<int> idx;
        std::vector<svo_mesh_desc> sub;
        for (int i = 0; i < n; ++i)
            if (descs[i].flags == f) {
                idx.push_back(i);
                sub.push_back(descs[i]);
            }
        svo_batch *b = nullptr;
        int rc = batch_create(ctx, sub.data(), (int)sub.size(), f, static_cast<cudaStream_t>(stream), &b);
        std::vector<svo_result *> r(sub.size(), nullptr);
        std::vector<int> st(sub.size(), rc);
        if (rc == SVO_OK) {
            rc = batch_phase_b(b, 0, (int)sub.size(), r.data(), st.data());
            const std::string msg = g_err;
            batch_destroy(b);
            g_err = msg;
        }
        for (size_t k = 0; k < sub.size(); ++k) {
            out[idx[k]] = r[k];
            if (status_out) status_out[idx[k]] = st[k];
        }
        if (rc != SVO_OK && first == SVO_OK) {
            first = rc;
            first_msg = g_err;
        }
    }
    if (first != SVO_OK) g_err = first_msg;
    return first;
}

int svo_batch_create(svo_ctx *ctx, const svo_mesh_desc *descs, int n, uint32_t flags, void *stream,
                     svo_batch **out) {
    if (!ctx || (!descs && n > 0) || !out) return fail(SVO_ERR_INVALID_ARGUMENT, "null argument");
    *out = nullptr;
    return batch_create(ctx, descs, n, flags, static_cast<cudaStream_t>(stream), out);
}

int svo_batch_size(const svo_batch *b) { return b ? (int)b->m.size() : 0; }

int svo_batch_mesh_status(const svo_batch *b, int i) {
    if (!b || i < 0 || i >= (int)b->m.size()) return SVO_ERR_INVALID_ARGUMENT;
    return b->m[i].status;
}

int64_t svo_batch_mesh_nodes(const svo_batch *b, int i) {
    if (!b || i < 0 || i >= (int)b->m.size() || b->m[i].status != SVO_OK) return -1;
    return (int64_t)b->m[i].N;
}

int64_t svo_batch_mesh_output_bytes(const svo_batch *b, int i) {
    if (!b || i < 0 || i >= (int)b->m.size() || b->m[i].status != SVO_OK) return -1;
    return (int64_t)output_bytes(b->m[i], b->flags);
}

int svo_batch_emit(svo_batch *b, int first, int count, svo_result **out, int *status_out) {
    if (!b || !out || first < 0 || count < 0 || first + count > (int)b->m.size())
        return fail(SVO_ERR_INVALID_ARGUMENT, "bad batch range");
    return batch_phase_b(b, first, count, out, status_out);
}

void svo_batch_free(svo_batch *b) { batch_destroy(b); }

int svo_ctx_autotune(svo_ctx *ctx, const svo_mesh_desc *descs, int n, uint32_t flags, void *stream,
                     svo_tuning *best) {
    if (!ctx || !descs || n <= 0) return fail(SVO_ERR_INVALID_ARGUMENT, "null argument or empty sample");
    VoxTuning saved;
    {
        std::lock_guard<std::mutex> lk(ctx->tune_mu);
        saved = ctx->tune;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // device ms of the voxelizer stage of the counting phase, best of 2 (after
    // one untimed run); the candidate goes to the measured batches only, so
    // builds on other threads keep the context's split meanwhile
    auto measure = [&](const VoxTuning &t, float &ms) -> int {
        ms = 1e30f;
        for (int rep = 0; rep < 3; ++rep) {
            svo_batch *b = nullptr;
            const int rc = batch_create(ctx, descs, n, flags | SVO_FLAG_TIMINGS, st, &b, &t);
            if (rc != SVO_OK) {
                batch_destroy(b);
                return rc;
            }
            if (rep > 0 && b->timed) ms = std::min(ms, b->timings_a[2]);
            batch_destroy(b);
        }
        return SVO_OK;
    };
    VoxTuning win = saved;
    float best_ms = 1e30f;
    int rc = SVO_OK;
    for (uint32_t sm : {16u, 32u, 64u, 128u}) {
        for (uint32_t wm : {64u, 128u, 256u, 512u, 1024u}) {
            VoxTuning t = saved;
            t.serial_max = sm;
            t.warp_max = wm;
            float ms = 0.0f;
            if ((rc = measure(t, ms)) != SVO_OK) break;
            if (ms < best_ms) {
                best_ms = ms;
                win = t;
            }
        }
        if (rc != SVO_OK) break;
    }
    if (rc != SVO_OK) return rc;
    {
        std::lock_guard<std::mutex> lk(ctx->tune_mu);
        ctx->tune = win;
    }
    if (best) {
        best->serial_max = win.serial_max;
        best->warp_max = win.warp_max;
        best->split = win.split;
        best->inplace_max = win.inplace_max;
        best->serial_packed = win.serial_packed;
    }
    return SVO_OK;
}

void svo_result_free(svo_result *r) {
    if (!r) return;
    cudaSetDevice(r->device);
    void *ptrs[] = {r->nodes, r->verts, r->edges, r->keys, r->dedup[0], r->dedup[1], r->dedup[2]};
    for (int i = 0; i < 7; ++i)
        if (ptrs[i] && ((r->own >> i) & 1)) cudaFreeAsync(ptrs[i], r->stream);
    if (r->arena && r->arena->refs.fetch_sub(1) == 1) {
        cudaFreeAsync(r->arena->base, r->stream);
        delete r->arena;
    }
    delete r;
}

int svo_result_depth(const svo_result *r) { return r ? r->depth : 0; }
int64_t svo_result_num_nodes(const svo_result *r) { return r ? (int64_t)r->n_nodes : 0; }
int64_t svo_result_num_vertices(const svo_result *r) { return r ? (int64_t)r->n_verts : 0; }
int64_t svo_result_num_edges(const svo_result *r) { return r ? (int64_t)r->n_edges : 0; }
int64_t svo_result_num_keys(const svo_result *r) { return r ? (int64_t)r->n_keys : 0; }

int svo_result_level_counts(const svo_result *r, int64_t *counts, int cap) {
    if (!r) return 0;
    const int n = (int)r->level_counts.size();
    for (int i = 0; i < n && i < cap; ++i) counts[i] = r->level_counts[i];
    return n;
}

int svo_result_bbox(const svo_result *r, svo_aabb *out) {
    if (!r || !out) return fail(SVO_ERR_INVALID_ARGUMENT, "null argument");
    *out = r->bbox;
    return SVO_OK;
}

const svo_node *svo_result_nodes_device(const svo_result *r) { return r ? r->nodes : nullptr; }
const svo_vertex *svo_result_vertices_device(const svo_result *r) { return r ? r->verts : nullptr; }
const svo_edge *svo_result_edges_device(const svo_result *r) { return r ? r->edges : nullptr; }
const uint64_t *svo_result_keys_device(const svo_result *r) { return r ? r->keys : nullptr; }

static int copy_out(const svo_result *r, void *dst, const void *src, uint64_t n, int64_t cap, size_t esz,
                    const char *what) {
    if (!r || (!dst && n > 0)) return fail(SVO_ERR_INVALID_ARGUMENT, "null argument");
    if ((uint64_t)cap < n) return fail(SVO_ERR_INVALID_ARGUMENT, "%s: capacity %lld < %llu", what, (long long)cap,
                                       (unsigned long long)n);
    if (n == 0) return SVO_OK;
    if (!src) return fail(SVO_ERR_INVALID_ARGUMENT, "%s were not built", what);
    SVO_TRY(cudaSetDevice(r->device), "cudaSetDevice");
    cudaError_t staged = cudaSuccess;
    if (r->copies && is_pageable_ptr(dst) &&
        svo::host::copy_to_pageable(*r->copies, dst, src, n * esz, r->stream, &staged)) {
        SVO_TRY(staged, what);
        return SVO_OK;
    }
    SVO_TRY(cudaMemcpyAsync(dst, src, n * esz, cudaMemcpyDeviceToHost, r->stream), what);
    SVO_TRY(cudaStreamSynchronize(r->stream), what);
    return SVO_OK;
}

int svo_result_copy_nodes(const svo_result *r, svo_node *dst, int64_t cap) {
    return copy_out(r, dst, r ? r->nodes : nullptr, r ? r->n_nodes : 0, cap, sizeof(svo_node), "nodes");
}
int svo_result_copy_vertices(const svo_result *r, svo_vertex *dst, int64_t cap) {
    return copy_out(r, dst, r ? r->verts : nullptr, r ? r->n_verts : 0, cap, sizeof(svo_vertex), "vertices");
}
int svo_result_copy_edges(const svo_result *r, svo_edge *dst, int64_t cap) {
    return copy_out(r, dst, r ? r->edges : nullptr, r ? r->n_edges : 0, cap, sizeof(svo_edge), "edges");
}
int svo_result_copy_keys(const svo_result *r, uint64_t *dst, int64_t cap) {
    return copy_out(r, dst, r ? r->keys : nullptr, r ? r->n_keys : 0, cap, sizeof(uint64_t), "keys");
}
int svo_result_timings(const svo_result *r, float *ms, int cap) {
    if (!r) return 0;
    for (int i = 0; i < r->n_timings && i < cap; ++i) ms[i] = r->timings[i];
    return r->n_timings;
}

int64_t svo_result_num_dedup(const svo_result *r, int kind) {
    return (r && kind >= 0 && kind < 3) ? (int64_t)r->n_dedup[kind] : -1;
}
int svo_result_copy_dedup(const svo_result *r, int kind, uint64_t *dst, int64_t cap) {
    if (!r || kind < 0 || kind > 2) return fail(SVO_ERR_INVALID_ARGUMENT, "bad kind");
    return copy_out(r, dst, r->dedup[kind], r->n_dedup[kind], cap, sizeof(uint64_t), "dedup keys");
}

int svo_write_tree(const svo_result *r, const char *path) {
    svo::host::TraceRange trace("svo: write tree .obj");
    if (!r || !path) return fail(SVO_ERR_INVALID_ARGUMENT, "null argument");
    std::vector<svo_node> h(r->n_nodes);
    int rc = svo_result_copy_nodes(r, h.data(), (int64_t)h.size());
    if (rc) return rc;
    return svo_write_tree_nodes(h.data(), (int64_t)h.size(), path);
}

int svo_write_voxels(const svo_result *r, const char *path) {
    if (!r || !path) return fail(SVO_ERR_INVALID_ARGUMENT, "null argument");
    std::vector<uint64_t> k(r->n_keys);
    int rc = svo_result_copy_keys(r, k.data(), (int64_t)k.size());
    if (rc) return rc;
    return svo::host::write_voxels(k.data(), (int64_t)k.size(), r->bbox.min, r->unit[0], path);
}

}  // extern "C"

namespace svo::host {
void set_error(const char *msg) { g_err = msg; }
}  // namespace svo::host

namespace svo {
static std::atomic<int64_t> g_launches{0};
void count_launches(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

// Countdown of svo_debug_fail_alloc: when it reaches the allocation it names,
// that allocation reports cudaErrorMemoryAllocation without asking the pool.
static std::atomic<int64_t> g_fail_alloc{0};

cudaError_t pool_malloc(void **p, size_t bytes, cudaMemPool_t pool, cudaStream_t st) {
    int64_t k = g_fail_alloc.load(std::memory_order_relaxed);
    while (k > 0 && !g_fail_alloc.compare_exchange_weak(k, k - 1, std::memory_order_relaxed)) {
    }
    if (k == 1) {
        *p = nullptr;
        return cudaErrorMemoryAllocation;
    }
    return cudaMallocFromPoolAsync(p, bytes, pool, st);
}
}  // namespace svo

extern "C" int64_t svo_kernel_launches(void) { return svo::g_launches.load(std::memory_order_relaxed); }

extern "C" int64_t svo_debug_fail_alloc(int64_t n) {
    return svo::g_fail_alloc.exchange(n > 0 ? n : 0, std::memory_order_relaxed);
}
