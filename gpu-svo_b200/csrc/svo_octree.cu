// svo_octree.cu -- octree levels, node records, vertex/edge arrays.
//
// The reference builds the octree bottom-up one level per host iteration
// (src/SVO.cu:383-495): compact a dense flag array, group codes by parent,
// place each group's 8 siblings, fill missing siblings, link parents and
// children.  Here every level comes out of one occupancy-bitmap pyramid:
//   * level l+1 bit j is the OR of level-l bits 8j..8j+7 (a byte test), so
//     one streaming pass builds all levels (k_pyramid);
//   * the same pass leaves each 512-bit block's rank within its 2048-word
//     region and each region's sums, whose scan gives O(1) rank queries on
//     every level;
//   * the node at local index 8g+k of level l has code 8*K[l+1][g] + k, where
//     K[l+1] is the sorted list of set bits of level l+1 (k_compact); its
//     children start at 8*rank_l(code) in level l-1, its parent sits at
//     8*rank_{l+2}(code >> 6) + ((code >> 3) & 7) in level l+1 -- exactly the
//     indices the reference's scans produce (src/SVO.cu:221-339);
//   * k_emit writes node records, vertex and edge arrays in one pass: records
//     and edges staged per warp in shared memory and stored by bulk copies,
//     vertices as full 512-byte coalesced streaming writes.
#include <cuda/atomic>

#include "svo_internal.h"

namespace svo {

Pyramid make_pyramid(int rx, int ry, int rz) {
    Pyramid py;
    int rmax = std::max(rx, std::max(ry, rz));
    int k = 0;
    while ((1 << k) < rmax) ++k;
    py.grid_levels = k + 1;
    py.levels = std::max(py.grid_levels, 5);
    const uint64_t bits0 = 1ull << (3 * k);
    uint64_t w0 = (bits0 + 63) / 64;
    w0 = std::max<uint64_t>(w0, 2048);
    w0 = (w0 + 2047) / 2048 * 2048;
    auto up8 = [](uint64_t v) { return (v + 7) / 8 * 8; };
    py.words[0] = w0;
    py.words[1] = w0 / 8;
    py.words[2] = w0 / 64;
    py.words[3] = up8(w0 / 512);
    py.words[4] = up8((w0 / 2048 + 1) / 2);
    for (int l = 5; l < py.levels; ++l) py.words[l] = up8((py.words[l - 1] + 7) / 8);
    uint64_t wo = 0, co = 0;
    for (int l = 0; l < py.levels; ++l) {
        py.woff[l] = wo;
        py.coff[l] = co;
        wo += py.words[l];
        co += py.words[l] / 8;
    }
    py.coff[py.levels] = co;
    py.total_words = wo;
    py.total_blocks = co;
    py.ctas = (uint32_t)(w0 / 2048);
    return py;
}

namespace {

// 8-bit mask of the non-zero bytes of v.
__device__ __forceinline__ uint32_t nz_bytes(uint64_t v) {
    uint64_t m = v | (v >> 4);
    m |= m >> 2;
    m |= m >> 1;
    m &= 0x0101010101010101ull;
    return (uint32_t)((m * 0x0102040810204080ull) >> 56);
}

// Exclusive prefix of v over the NT threads of the block, and the block's sum.
// All threads call; s_warp holds NT / 32 words.
template <int NT>
__device__ __forceinline__ uint32_t block_exscan(uint32_t v, uint32_t *s_warp, uint32_t &total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += o;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    const uint32_t w = lane < NT / 32 ? s_warp[lane] : 0u;
    total = __reduce_add_sync(0xFFFFFFFFu, w);
    const uint32_t before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? w : 0u);
    __syncthreads();  // s_warp may be rewritten
    return before + incl - v;
}

// The region sums of one of levels 0..3 (base + level * bstride) become their
// exclusive prefixes in place; the sum goes to out->totals[level].  Padding past
// the mesh's regions (up to the 16-byte stride) is treated as zero.
template <int NT, int ITEMS>
__device__ __forceinline__ void scan_regions(const MeshDev &md, int level, uint32_t *s_warp) {
    uint32_t *a = md.base + (uint64_t)level * md.bstride;
    const uint32_t n = md.py.ctas;
    uint32_t carry = 0;
    for (uint32_t i0 = 0; i0 < n; i0 += NT * ITEMS) {
        const uint32_t i = i0 + threadIdx.x * ITEMS;
        uint32_t v[ITEMS];
        uint32_t sum = 0;
#pragma unroll
        for (int q = 0; q < ITEMS / 4; ++q) {
            uint4 x = make_uint4(0, 0, 0, 0);
            if (i + 4 * q < n) x = __ldcg(reinterpret_cast<const uint4 *>(a + i) + q);
            v[4 * q] = x.x;
            v[4 * q + 1] = x.y;
            v[4 * q + 2] = x.z;
            v[4 * q + 3] = x.w;
        }
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            if (i + k >= n) v[k] = 0;
            sum += v[k];
        }
        uint32_t tot;
        uint32_t run = carry + block_exscan<NT>(sum, s_warp, tot);
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const uint32_t x = v[k];
            v[k] = run;
            run += x;
        }
#pragma unroll
        for (int q = 0; q < ITEMS / 4; ++q)
            if (i + 4 * q < n)
                reinterpret_cast<uint4 *>(a + i)[q] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
        carry += tot;
    }
    if (threadIdx.x == 0) md.out->totals[level] = carry;
}

// scan_regions of the four levels at once for a mesh of at most 4 NT regions:
// one round trip for all loads.
template <int NT>
__device__ __forceinline__ void scan_regions_all(const MeshDev &md, uint32_t *s_warp) {
    const uint32_t n = md.py.ctas, i = threadIdx.x * 4;
    uint4 v[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        v[l] = make_uint4(0, 0, 0, 0);
        if (i < n) v[l] = __ldcg(reinterpret_cast<const uint4 *>(md.base + (uint64_t)l * md.bstride + i));
        if (i + 1 >= n) v[l].y = 0;  // padding
        if (i + 2 >= n) v[l].z = 0;
        if (i + 3 >= n) v[l].w = 0;
    }
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        uint32_t tot;
        const uint32_t a = block_exscan<NT>(v[l].x + v[l].y + v[l].z + v[l].w, s_warp, tot);
        const uint32_t b = a + v[l].x, c = b + v[l].y, d = c + v[l].z;
        if (i < n) *reinterpret_cast<uint4 *>(md.base + (uint64_t)l * md.bstride + i) = make_uint4(a, b, c, d);
        if (threadIdx.x == 0) md.out->totals[l] = tot;
    }
}

// Levels 5.. of a mesh from its level 4, with the scanned block counts and the
// totals of levels 4.., and the rest of the mesh's report.  Levels of at most kTopWords words stay in shared
// memory between the steps, so only the first step waits on global loads.
constexpr uint32_t kTopWords = 512;

template <int NT>
__device__ __forceinline__ void finish_top(const MeshDev &md, uint64_t (*s_top)[kTopWords], uint32_t *s_warp) {
    const Pyramid &py = md.py;
    if (threadIdx.x < sizeof(GridParams) / 4)  // every earlier kernel has left its status bits
        reinterpret_cast<uint32_t *>(&md.out->gp)[threadIdx.x] =
            __ldcg(reinterpret_cast<const uint32_t *>(md.gp) + threadIdx.x);
    if (threadIdx.x == 32) {
        md.out->any = __ldcg(reinterpret_cast<const unsigned long long *>(md.any));
        md.out->queue = __ldcg(md.queue);
    }
    bool held = false;  // level l is in s_top[l & 1]
    for (int l = 4; l < py.levels; ++l) {
        const uint64_t *in = md.bits + py.woff[l];
        const uint32_t nblk = (uint32_t)(py.words[l] / 8);
        const bool has_next = l + 1 < py.levels;
        uint64_t *out = has_next ? md.bits + py.woff[l + 1] : nullptr;
        const bool hold = has_next && py.words[l + 1] <= kTopWords;
        if (hold)
            for (uint32_t j = nblk + threadIdx.x; j < py.words[l + 1]; j += NT) s_top[(l + 1) & 1][j] = 0;  // padding
        uint32_t carry = 0;
        for (uint32_t j0 = 0; j0 < nblk; j0 += NT) {
            const uint32_t j = j0 + threadIdx.x;
            uint64_t w = 0;
            uint32_t c = 0;
            if (j < nblk) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    ulonglong2 v;
                    if (held) v = reinterpret_cast<const ulonglong2 *>(s_top[l & 1] + 8 * j)[q];
                    else v = __ldcg(reinterpret_cast<const ulonglong2 *>(in + 8 * (uint64_t)j) + q);
                    c += __popcll(v.x) + __popcll(v.y);
                    w |= (uint64_t)nz_bytes(v.x) << (16 * q);
                    w |= (uint64_t)nz_bytes(v.y) << (16 * q + 8);
                }
            }
            uint32_t tot;
            const uint32_t ex = carry + block_exscan<NT>(c, s_warp, tot);
            if (j < nblk) {
                md.pre[py.coff[l] + j] = ex;
                if (has_next) out[j] = w;
                if (hold) s_top[(l + 1) & 1][j] = w;
            }
            carry += tot;
        }
        if (threadIdx.x == 0) md.out->totals[l] = carry;
        held = hold;
        __syncthreads();  // level l + 1 is complete (in shared memory, or in global memory for this block)
    }
}

// Levels 1..4 of 2048-word chunks of level 0 (regions), a persistent grid
// taking them in turn (one 512-bit block of level 0 per thread, 16-byte
// streaming loads).  The same pass ranks: every 512-bit block of levels 0..2
// gets the set bits before it in its region (md.pre), and every region its
// set bits of levels 0..3 (md.base), whose prefix over the regions completes
// the rank -- there is no scan over the blocks (19.2M of them at res 2048:
// that scan and the memset before it took 60 us; the scan of 4 x 65,536 region
// sums is part of k_pyramid_finish, 24 us in all).  With a region-mode mesh in the batch only the listed
// regions are visited: the others are empty, not zeroed in memory at level 0
// and dealt with by k_region_prepare.
//
// FUSE: the CTA that finishes a mesh's last region scans the sums and builds
// the levels above 4 as well, which saves a launch (about 5 us of the 213 us
// of a 20k-triangle build at res 128).  One CTA of 256 threads takes 4 region
// sums per thread and level in one step up to kFuseRegions; meshes with more
// regions (res 1024 and up) are finished by k_pyramid_finish, whose five
// 1024-thread CTAs per mesh work side by side, and so are batches with more
// than 8 regions per SM, where the fused variant's 62 to 64 registers (4 CTAs per
// SM instead of 8) cost the streaming pass more than the launch saves.
constexpr uint32_t kFuseRegions = 1024;

template <bool FUSE, bool ONE>
__global__ void __launch_bounds__(256, FUSE ? 4 : 8) k_pyramid(const __grid_constant__ BatchDev bd,
                                                               const __grid_constant__ MeshDev one, uint32_t total) {
    chain_begin();
    const Meshes<ONE> mesh{bd, one};
    __shared__ uint64_t s1[256];
    __shared__ uint64_t s2[32];
    __shared__ uint64_t s3[4];
    __shared__ uint32_t s_warp[8];
    __shared__ uint32_t s_last;
    __shared__ __align__(16) uint64_t s_top[FUSE ? 2 : 1][kTopWords];
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t count = !FUSE && bd.rlist ? *bd.rcount : total;
    for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
        const uint32_t g = !FUSE && bd.rlist ? bd.rlist[i] : i;
        const int m = mesh.of_region(g);
        const MeshDev &md = mesh[m];
        const Pyramid &py = md.py;
        uint64_t *__restrict__ bits = md.bits;
        uint32_t *__restrict__ pre = md.pre;
        const uint32_t b = g - mesh.first_region(m);
        {
            const uint4 *src = reinterpret_cast<const uint4 *>(bits + py.woff[0] + (uint64_t)b * 2048 + t * 8);
            uint64_t w1 = 0;
            uint32_t c0 = 0, first = 0;  // first: bit of the block
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint4 v = __ldcs(src + q);
                const uint64_t a = ((uint64_t)v.y << 32) | v.x, c = ((uint64_t)v.w << 32) | v.z;
                if (a) first = 128 * q + __ffsll((long long)a) - 1;
                else if (c) first = 128 * q + 64 + __ffsll((long long)c) - 1;
                c0 += __popcll(a) + __popcll(c);
                w1 |= (uint64_t)nz_bytes(a) << (16 * q);
                w1 |= (uint64_t)nz_bytes(c) << (16 * q + 8);
            }
            bits[py.woff[1] + (uint64_t)b * 256 + t] = w1;
            s1[t] = w1;
            // one surface voxel of the mesh (any: the last store wins)
            const uint32_t some = __ballot_sync(0xFFFFFFFFu, c0 != 0);
            if (some && lane == __ffs(some) - 1) *md.any = ((uint64_t)b * 256 + t) * 512 + first;
            uint32_t sum0;
            pre[py.coff[0] + (uint64_t)b * 256 + t] = block_exscan<256>(c0, s_warp, sum0);  // s1 is complete after it
            if (warp == 0) {  // levels 2..4 of the region: one warp
                uint64_t w = 0;
                uint32_t c = 0;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint64_t v = s1[8 * t + k];
                    c += __popcll(v);
                    w |= (uint64_t)nz_bytes(v) << (8 * k);
                }
                uint32_t incl = c;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                    if (lane >= d) incl += o;
                }
                const uint32_t sum1 = __shfl_sync(0xFFFFFFFFu, incl, 31);
                pre[py.coff[1] + (uint64_t)b * 32 + t] = incl - c;
                bits[py.woff[2] + (uint64_t)b * 32 + t] = w;
                s2[t] = w;
                __syncwarp();
                w = 0;
                c = 0;
                if (t < 4) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const uint64_t v = s2[8 * t + k];
                        c += __popcll(v);
                        w |= (uint64_t)nz_bytes(v) << (8 * k);
                    }
                    bits[py.woff[3] + (uint64_t)b * 4 + t] = w;
                    s3[t] = w;
                }
                incl = c;
#pragma unroll
                for (int d = 1; d < 4; d <<= 1) {
                    const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                    if (lane >= d) incl += o;
                }
                const uint32_t sum2 = __shfl_sync(0xFFFFFFFFu, incl, 3);
                if (t < 4) pre[py.coff[2] + (uint64_t)b * 4 + t] = incl - c;
                __syncwarp();
                if (t == 0) {
                    uint32_t w4 = 0, sum3 = 0;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        sum3 += __popcll(s3[k]);
                        w4 |= nz_bytes(s3[k]) << (8 * k);
                    }
                    uint32_t *base = md.base + b;
                    base[0] = sum0;
                    base[md.bstride] = sum1;
                    base[2 * (uint64_t)md.bstride] = sum2;
                    base[3 * (uint64_t)md.bstride] = sum3;
                    reinterpret_cast<uint32_t *>(bits + py.woff[4])[b] = w4;
                }
            }
        }
        __syncthreads();  // s1 is rewritten by the next region; the region's stores come before its arrival
        if (FUSE) {
            if (t == 0) {
                __threadfence();
                s_last = atomicAdd(md.done, 1u) == py.ctas - 1 ? 1u : 0u;
                __threadfence();
            }
            __syncthreads();
            if (s_last) {
                scan_regions_all<256>(md, s_warp);
                finish_top<256>(md, s_top, s_warp);
            }
        }
    }
}

// The region sums' prefixes (CTAs 0..3 of a mesh, one level each) and levels
// 5.. (CTA 4) of every mesh.  The mesh is the grid's x: y ends at 65,535, and a
// batch may hold more meshes than that.
template <bool ONE>
__global__ void __launch_bounds__(1024) k_pyramid_finish(const __grid_constant__ BatchDev bd,
                                                         const __grid_constant__ MeshDev one) {
    __shared__ __align__(16) uint64_t s_top[2][kTopWords];
    __shared__ uint32_t s_warp[32];
    chain_begin();
    const Meshes<ONE> mesh{bd, one};
    const MeshDev &md = mesh[blockIdx.x];
    if (blockIdx.y < 4) scan_regions<1024, 16>(md, (int)blockIdx.y, s_warp);
    else finish_top<1024>(md, s_top, s_warp);
}

// ---------------------------------------------------------------------------
// Single-pass exclusive scan (decoupled look-back).  Tile status words hold
// (flag << 32 | value): flag 1 = tile aggregate, 2 = inclusive prefix.  The
// look-back wait is bounded; on timeout the kernel records
// kStatusScanTimeout and the host fails the build.
// ---------------------------------------------------------------------------
constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr uint64_t kScanTile = kScanThreads * kScanItems;
constexpr int kSpinLimit = 1 << 22;
constexpr uint64_t kScanSplitTiles = 64;  // from this many tiles on (aligned data): reduce-then-scan

__device__ __forceinline__ unsigned long long ld_relaxed(unsigned long long *p) {
    return cuda::atomic_ref<unsigned long long, cuda::thread_scope_device>(*p).load(
        cuda::memory_order_relaxed);
}
__device__ __forceinline__ void st_relaxed(unsigned long long *p, unsigned long long v) {
    cuda::atomic_ref<unsigned long long, cuda::thread_scope_device>(*p).store(v, cuda::memory_order_relaxed);
}

__global__ void __launch_bounds__(kScanThreads) k_scan(const uint32_t *__restrict__ in,
                                                       uint32_t *__restrict__ out, uint64_t n,
                                                       unsigned long long *__restrict__ scratch,
                                                       uint32_t *__restrict__ status, int spin_limit) {
    __shared__ uint32_t s_tile, s_prefix;
    __shared__ uint32_t s_warp[kScanThreads / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) s_tile = atomicAdd(reinterpret_cast<unsigned int *>(scratch), 1u);
    __syncthreads();
    const uint64_t tile = s_tile;
    unsigned long long *st = scratch + 1;
    const uint64_t base = tile * kScanTile + (uint64_t)t * kScanItems;
    uint32_t v[kScanItems];
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < n ? in[base + k] : 0u;
        sum += v[k];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += o;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kScanThreads / 32 ? s_warp[lane] : 0u;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, w, d);
            if (lane >= d) w += o;
        }
        if (lane < kScanThreads / 32) s_warp[lane] = w;  // inclusive warp totals
    }
    __syncthreads();
    const uint32_t aggregate = s_warp[kScanThreads / 32 - 1];
    if (warp == 0) {
        uint32_t prefix = 0;
        if (tile == 0) {
            if (lane == 0) st_relaxed(st, (2ull << 32) | aggregate);
        } else {
            if (lane == 0) st_relaxed(st + tile, (1ull << 32) | aggregate);
            int64_t j = (int64_t)tile - 1;
            int spins = 0;
            for (;;) {
                const int64_t q = j - lane;
                const unsigned long long s = q >= 0 ? ld_relaxed(st + q) : (2ull << 32);
                const uint32_t flag = (uint32_t)(s >> 32);
                if (__any_sync(0xFFFFFFFFu, flag == 0)) {
                    if (++spins > spin_limit) {
                        if (lane == 0) atomicOr(status, kStatusScanTimeout);
                        break;
                    }
                    __nanosleep(64);
                    continue;
                }
                const uint32_t m2 = __ballot_sync(0xFFFFFFFFu, flag == 2);
                const int stop = m2 ? __ffs(m2) - 1 : 31;
                uint32_t val = lane <= stop ? (uint32_t)s : 0u;
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) val += __shfl_xor_sync(0xFFFFFFFFu, val, d);
                prefix += val;
                if (m2) break;
                j -= 32;
            }
            if (lane == 0) st_relaxed(st + tile, (2ull << 32) | (prefix + aggregate));
        }
        if (lane == 0) s_prefix = prefix;
    }
    __syncthreads();
    uint32_t run = s_prefix + (warp ? s_warp[warp - 1] : 0u) + (incl - sum);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
    const uint64_t last_tile = (n + kScanTile - 1) / kScanTile - 1;
    if (tile == last_tile && t == kScanThreads - 1) out[n] = s_prefix + aggregate;
}

// Reduce-then-scan for long, 16-byte aligned arrays: tile sums, one CTA
// scanning them, then each tile scanned again with its prefix added.  Three
// streaming passes, no inter-CTA waiting; every thread moves its 16 items
// with 16-byte loads and stores.
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t *s_warp) {
    v = __reduce_add_sync(0xFFFFFFFFu, v);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s_warp[w];
    return t;
}

__device__ __forceinline__ void load_items(const uint32_t *in, uint64_t base, uint64_t n, uint32_t v[kScanItems]) {
    if (base + kScanItems <= n) {
        const uint4 *p = reinterpret_cast<const uint4 *>(in + base);
#pragma unroll
        for (int q = 0; q < kScanItems / 4; ++q) {
            const uint4 x = __ldcs(p + q);
            v[4 * q] = x.x;
            v[4 * q + 1] = x.y;
            v[4 * q + 2] = x.z;
            v[4 * q + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) v[k] = base + k < n ? in[base + k] : 0u;
    }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_reduce(const uint32_t *__restrict__ in, uint64_t n,
                                                              uint32_t *__restrict__ tsum) {
    __shared__ uint32_t s_warp[kScanThreads / 32];
    uint32_t v[kScanItems];
    load_items(in, blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems, n, v);
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) sum += v[k];
    sum = block_sum(sum, s_warp);
    if (threadIdx.x == 0) tsum[blockIdx.x] = sum;
}

// Exclusive prefix of the tile sums (one CTA of 1024 threads) and the grand
// total at *total.
__global__ void __launch_bounds__(1024) k_scan_tiles(const uint32_t *__restrict__ tsum, uint32_t *__restrict__ tpre,
                                                     uint64_t tiles, uint32_t *__restrict__ total) {
    __shared__ uint32_t s_warp[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t carry = 0;
    for (uint64_t base = 0; base < tiles; base += 1024) {
        const uint64_t i = base + t;
        const uint32_t v = i < tiles ? tsum[i] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += o;
        }
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            uint32_t w = s_warp[lane];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, w, d);
                if (lane >= d) w += o;
            }
            s_warp[lane] = w;  // inclusive warp totals
        }
        __syncthreads();
        if (i < tiles) tpre[i] = carry + (warp ? s_warp[warp - 1] : 0u) + incl - v;
        carry += s_warp[31];
        __syncthreads();  // s_warp is rewritten by the next round
    }
    if (t == 0) *total = carry;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_down(const uint32_t *__restrict__ in, uint32_t *__restrict__ out,
                                                            uint64_t n, const uint32_t *__restrict__ tpre) {
    __shared__ uint32_t s_warp[kScanThreads / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint64_t base = blockIdx.x * kScanTile + (uint64_t)t * kScanItems;
    uint32_t v[kScanItems];
    load_items(in, base, n, v);
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) sum += v[k];
    uint32_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += o;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t run = tpre[blockIdx.x] + incl - sum;
    for (int w = 0; w < warp; ++w) run += s_warp[w];
    uint32_t o[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        o[k] = run;
        run += v[k];
    }
    if (base + kScanItems <= n) {
        uint4 *q = reinterpret_cast<uint4 *>(out + base);
#pragma unroll
        for (int j = 0; j < kScanItems / 4; ++j) q[j] = make_uint4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k)
            if (base + k < n) out[base + k] = o[k];
    }
}

// Set bits of level l before its 512-bit block `blk`.
__device__ __forceinline__ uint32_t block_rank(const RankDev &r, const Pyramid &py, int l, uint64_t blk) {
    if (l >= 4) return r.pre[py.coff[l] + blk];
    if (l == 3) return r.base[3 * (uint64_t)r.bstride + 2 * blk];  // a level-3 block spans two regions
    return r.base[(uint64_t)l * r.bstride + (blk >> (8 - 3 * l))] + r.pre[py.coff[l] + blk];
}

// The set-bit codes of the warp's 32 words, whose outputs are one contiguous
// range in lane order (lane i's codes at o, o + 1, ...; lanes without bits
// hold pc = 0): staged in shared memory as (lane, bit) entries, then read in
// order, each turned into its code (the owning lane's b64 + bit) and stored
// coalesced.  All 32 lanes call; lane 0 must hold a word of the range.
__device__ __forceinline__ void warp_codes(uint64_t *out, uint32_t o, uint32_t pc, uint64_t v, uint64_t b64,
                                           uint16_t *stage, int lane) {
    const uint32_t start = __shfl_sync(0xFFFFFFFFu, o, 0);
    const uint32_t tot = __reduce_add_sync(0xFFFFFFFFu, pc);
    uint32_t at = o - start;
    for (uint64_t m = v; m; m &= m - 1) stage[at++] = (uint16_t)((uint32_t)lane << 6 | (uint32_t)(__ffsll((long long)m) - 1));
    __syncwarp();
    const uint32_t blo = (uint32_t)b64, bhi = (uint32_t)(b64 >> 32);
    for (uint32_t i0 = 0; i0 < tot; i0 += 32) {
        const uint32_t i = i0 + lane;
        const uint32_t e = i < tot ? stage[i] : 0u;
        const int src = (int)(e >> 6);
        const uint64_t base = (uint64_t)__shfl_sync(0xFFFFFFFFu, bhi, src) << 32 | __shfl_sync(0xFFFFFFFFu, blo, src);
        if (i < tot) out[start + i] = base + (e & 63u);
    }
    __syncwarp();
}

// Word w of level l holding v (read by the caller; 0 for a lane without a
// word): rank from the block prefix and the 8-lane popcount prefix, then the
// positions.  All 32 lanes of the warp call (8 aligned lanes per block).
__device__ __forceinline__ void compact_word(const CompactJob &job, int l, uint64_t w, uint64_t v) {
    const int sub = threadIdx.x & 7;
    const uint32_t r0 = v ? block_rank(job.rank, job.py, l, w >> 3) : 0u;
    const uint32_t pc = __popcll(v);
    uint32_t x = pc;
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d, 8);
        if (sub >= d) x += y;
    }
    const uint32_t r = r0 + x - pc;
    if (!v) return;
    if (l >= 1) job.wpre[job.py.woff[l] - job.py.woff[1] + w] = r;
    uint64_t *o = (l == 0 ? job.keys : job.out + job.koff[l]) + r;
    const uint64_t b64 = w * 64;
    while (v) {
        *o++ = b64 + __ffsll((long long)v) - 1;
        v &= v - 1;
    }
}

// One thread per 64-bit word of every job's levels; the 8 lanes of a 512-bit
// block are 8 aligned lanes of a warp (every level and job starts on a block
// boundary), so a word's rank in its level is the block's rank plus an 8-lane
// prefix of popcounts.  Writes the sorted set-bit positions and, for levels >= 1,
// the rank at each non-empty word (rank_of's table).
// In a region-mode mesh a word of levels 0-3 lies inside one level-0 region
// (level-l word w covers level-0 words w * 8^l ..): an unflagged one is
// empty and is not read.
// ONE: a single job, passed by value (no upload of its table).
template <bool ONE>
__global__ void __launch_bounds__(256) k_compact(CompactBatch cb, const __grid_constant__ CompactJob one,
                                                 uint64_t total) {
    chain_begin();
    const uint64_t gi = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (gi >= ((total + 31) & ~31ull)) return;  // whole warps stay for the shuffles
    uint64_t v = 0, w = 0;
    int l = 0, j = 0;
    if (gi < total) {
        if (!ONE) j = find_segment(cb.word_off, cb.n, gi);
        const CompactJob &job = ONE ? one : cb.job[j];
        const Pyramid &py = job.py;
        const uint64_t gw = py.woff[job.l0] + (ONE ? gi : gi - cb.word_off[j]);
        l = job.l0;
        while (l + 1 < job.l1 && gw >= py.woff[l + 1]) ++l;
        w = gw - py.woff[l];
        v = (l <= 3 && job.rflag && !job.rflag[w >> (11 - 3 * l)]) ? 0ull : job.bits[gw];
    }
    compact_word(ONE ? one : cb.job[j], l, w, v);
}

// Levels 1 and 2 of a region-mode mesh, listed region by listed region (a
// block takes them in turn): the 256 level-1 and 32 level-2 words above a
// region lie inside it, and the unflagged ones (most of them at res 2048) hold
// none.  The list is the batch's: the mesh's own regions are cta0 on.
__global__ void __launch_bounds__(256) k_compact_regions(const __grid_constant__ CompactJob job,
                                                         const uint32_t *rlist, const uint32_t *rcount,
                                                         uint32_t cta0, uint32_t regions) {
    chain_begin();
    const uint32_t count = *rcount;
    for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
        const uint32_t rg = rlist[i] - cta0;  // wraps for the meshes before
        if (rg >= regions) continue;
        const uint64_t w1 = (uint64_t)rg * 256 + threadIdx.x;
        compact_word(job, 1, w1, job.bits[job.py.woff[1] + w1]);
        if (threadIdx.x < 32 && job.l1 > 2) {  // a two-voxel octree's top is level 1
            const uint64_t w2 = (uint64_t)rg * 32 + threadIdx.x;
            compact_word(job, 2, w2, job.bits[job.py.woff[2] + w2]);
        }
    }
}

// Level-0 set bits (the surface-voxel keys) from the non-empty 512-bit blocks
// only: a mesh's level-3 code list is exactly its non-empty level-0 blocks,
// in order.  8 lanes per block, one word each.
// ONE: a single job, passed by value.
template <bool ONE>
__global__ void __launch_bounds__(256) k_compact_keys(KeyBatch kb, const __grid_constant__ KeyJob one,
                                                      uint64_t total_blocks) {
    __shared__ uint16_t stage[8][2048];  // a warp's 4 blocks x 512 bits
    const uint64_t gi = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint64_t item = gi >> 3;
    if (((gi >> 5) << 2) >= total_blocks) return;  // whole warps stay for the shuffles
    const int sub = threadIdx.x & 7;
    uint64_t v = 0, blk = 0;
    uint32_t r = 0;
    int j = 0;
    if (item < total_blocks) {
        if (!ONE) j = find_segment(kb.blk_off, kb.n, item);
        const KeyJob &job = ONE ? one : kb.job[j];
        blk = job.blocks[ONE ? item : item - kb.blk_off[j]];
        v = job.bits[blk * 8 + sub];
        r = job.rank.base[blk >> 8] + job.rank.pre[blk];
    }
    const uint32_t pc = __popcll(v);
    uint32_t x = pc;
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, d, 8);
        if (sub >= d) x += y;
    }
    // the warp's blocks are consecutive non-empty blocks of one mesh (its
    // outputs one range) unless it straddles two meshes
    const int j0 = __shfl_sync(0xFFFFFFFFu, j, 0);
    if (ONE || __all_sync(0xFFFFFFFFu, item >= total_blocks || j == j0)) {
        warp_codes((ONE ? one : kb.job[j0]).out, item < total_blocks ? r + x - pc : 0xFFFFFFFFu, pc, v, (blk * 8 + sub) * 64,
                   stage[threadIdx.x >> 5], threadIdx.x & 31);
        return;
    }
    if (!v) return;
    uint64_t *o = kb.job[j].out + r + x - pc;
    const uint64_t b64 = (blk * 8 + sub) * 64;
    while (v) {
        *o++ = b64 + __ffsll((long long)v) - 1;
        v &= v - 1;
    }
}

// ---------------------------------------------------------------------------
// Node emission.
// ---------------------------------------------------------------------------
struct NodeInfo {
    uint64_t code;
    uint64_t pc;  // parent code (level l+1)
    int l;
    bool real;
    uint32_t child0;
    uint32_t parent;
    float o[3];
    float w;
};

// Rank of set bit c among level l's set bits (l >= 1): the word's rank from
// k_compact plus the set bits below c in its word.
__device__ __forceinline__ uint32_t rank_of(const EmitParams &P, int l, uint64_t c) {
    const uint64_t w = c >> 6;
    return P.lv[l].wpre[w] + (uint32_t)__popcll(P.lv[l].bits[w] & ((1ull << (c & 63)) - 1ull));
}

template <bool S>
__device__ __forceinline__ void node_info(const EmitParams &P, const float go[3], uint32_t t, NodeInfo &ni) {
    int l = 0;
    while (l < P.T && t >= P.lv[l + 1].off) ++l;
    const uint32_t i = t - P.lv[l].off;
    ni.l = l;
    if (l < P.T) {
        ni.pc = P.lv[l].K1[i >> 3];
        ni.code = (ni.pc << 3) | (i & 7);
    } else {
        ni.code = P.lv[l].K1[0];
        ni.pc = ni.code >> 3;
    }
    ni.real = false;
    ni.child0 = kNone;
    if (l >= 1) {  // one word load serves both the bit test and the rank
        const uint64_t w = ni.code >> 6;
        const uint64_t wd = P.lv[l].bits[w];
        const uint32_t wp = P.lv[l].wpre[w];
        ni.real = (wd >> (ni.code & 63)) & 1ull;
        if (ni.real) ni.child0 = P.lv[l - 1].off + 8u * (wp + (uint32_t)__popcll(wd & ((1ull << (ni.code & 63)) - 1ull)));
    }
    if (l < P.T) {
        const uint32_t pl = (l + 1 < P.T) ? 8u * rank_of(P, l + 2, ni.pc >> 3) + (uint32_t)(ni.pc & 7) : 0u;
        ni.parent = P.lv[l + 1].off + pl;
    } else {
        ni.parent = kNone;
    }
    ni.w = P.lv[l].width;
    const uint32_t x = compact3(ni.code), y = compact3(ni.code >> 1), z = compact3(ni.code >> 2);
    ni.o[0] = Fp<S>::origin(go[0], ni.w, (float)x);
    ni.o[1] = Fp<S>::origin(go[1], ni.w, (float)y);
    ni.o[2] = Fp<S>::origin(go[2], ni.w, (float)z);
}

// Full 27-neighbourhood.  The same-level node at offset d exists iff its
// parent group is a set bit of the next level.  A node with coordinate parity
// s has its neighbours' parents among 8 groups: its own and, per axis, the
// one on the side it borders (-1 where s_i = 0, +1 where s_i = 1); neighbour d
// then lies in group b (b_i = 1 where d crosses into the bordering group) at
// child (s ^ [d != 0]).
// The 8 siblings of a group sit in 8 aligned lanes and need the same 26 groups
// around theirs: lane k ranks groups k, k + 8, k + 16 and k + 24 and leaves
// their first nodes in tab (28 words per group in shared memory), where each
// lane picks its 7.  That is 4 look-ups a lane instead of 7: the emission with
// full neighbours was held up by their scattered loads (L1 80% busy).
// All 32 lanes call; on: the lane holds a node below the top level (the same
// for the 8 lanes of a group).
__device__ __forceinline__ void full_neighbors(const EmitParams &P, const NodeInfo &ni, uint32_t self, bool on, int lane,
                                               uint32_t *tab, uint32_t nb[27]) {
    uint32_t *mine = tab + (lane >> 3) * 28;
    if (on) {
        const int l1 = ni.l + 1;
        const uint64_t pc = ni.pc;
        const uint64_t sx = spread3(P.lv[l1].side);
        const uint64_t m[3] = {pc & kDilX, pc & kDilY, pc & kDilZ};
        const uint64_t lim[3] = {sx, sx << 1, sx << 2};
        const uint64_t msk[3] = {kDilX, kDilY, kDilZ};
        uint64_t dn[3], up[3];
        uint32_t ok = 0;  // bit 3 a + d: step d - 1 along axis a stays in the grid
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            dn[a] = dil_dec(m[a], msk[a]);
            up[a] = dil_inc(m[a], msk[a]);
            ok |= ((m[a] != 0 ? 1u : 0u) | 2u | (up[a] < lim[a] && up[a] != 0 ? 4u : 0u)) << (3 * a);
        }
        const bool top = l1 >= P.T;  // the root level: rank 0
        const uint64_t *bits = P.lv[l1].bits;
        const uint32_t *wpre = P.lv[l1].wpre;
        uint64_t wd[4];
        uint32_t wp[4], sh[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {  // all loads first
            const uint32_t j = (uint32_t)(lane & 7) + 8 * r, d0 = j % 3, d1 = j / 3 % 3, d2 = j / 9;
            const uint64_t q = (d0 == 0 ? dn[0] : d0 == 1 ? m[0] : up[0]) | (d1 == 0 ? dn[1] : d1 == 1 ? m[1] : up[1]) |
                               (d2 == 0 ? dn[2] : d2 == 1 ? m[2] : up[2]);
            const bool in = j < 27 && j != 13 && ((ok >> d0) & (ok >> (3 + d1)) & (ok >> (6 + d2)) & 1u);
            wd[r] = in ? bits[q >> 6] : 0ull;
            wp[r] = in && !top ? wpre[q >> 6] : 0u;
            sh[r] = (uint32_t)(q & 63);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t j = (uint32_t)(lane & 7) + 8 * r;
            const bool ex = (wd[r] >> sh[r]) & 1ull;
            if (j < 27)
                mine[j] = ex ? P.lv[ni.l].off + 8u * (wp[r] + (uint32_t)__popcll(wd[r] & ((1ull << sh[r]) - 1ull))) : kNone;
        }
    }
    __syncwarp();
    if (!on) return;
    const uint32_t s = (uint32_t)(ni.code & 7);
    nb[13] = self;
    uint32_t base[8];
    base[0] = self - s;  // child 0 of the node's own group
    const int ox = (s & 1) ? 1 : -1, oy = (s & 2) ? 3 : -3, oz = (s & 4) ? 9 : -9;
#pragma unroll
    for (int b = 1; b < 8; ++b)
        base[b] = mine[13 + ((b & 1) ? ox : 0) + ((b & 2) ? oy : 0) + ((b & 4) ? oz : 0)];
    // Neighbour d = base[b] | k with, per axis a, (b_a, k_a) = (1, 1), (0, 0),
    // (0, 1) for d_a = -1, 0, +1 when s_a = 0 and (0, 0), (0, 1), (1, 0) when
    // s_a = 1 (every base is a multiple of 8, and kNone | k = kNone): the
    // 3 x 3 x 3 table follows from the 8 bases one axis at a time.
    const uint32_t sxa = s & 1u, sya = (s >> 1) & 1u, sza = (s >> 2) & 1u;
    uint32_t X[3][4];  // [dx + 1][b_y | b_z << 1]
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const uint32_t b0 = base[r << 1], b1 = base[(r << 1) | 1];
        X[0][r] = sxa ? b0 : (b1 | 1u);
        X[1][r] = b0 | sxa;
        X[2][r] = sxa ? b1 : (b0 | 1u);
    }
    uint32_t Y[3][3][2];  // [dx + 1][dy + 1][b_z]
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int z = 0; z < 2; ++z) {
            const uint32_t c0 = X[i][z << 1], c1 = X[i][(z << 1) | 1];
            Y[i][0][z] = sya ? c0 : (c1 | 2u);
            Y[i][1][z] = c0 | (sya << 1);
            Y[i][2][z] = sya ? c1 : (c0 | 2u);
        }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int jy = 0; jy < 3; ++jy) {
            const uint32_t c0 = Y[i][jy][0], c1 = Y[i][jy][1];
            nb[i + 3 * jy] = sza ? c0 : (c1 | 4u);
            nb[i + 3 * jy + 9] = c0 | (sza << 2);
            nb[i + 3 * jy + 18] = sza ? c1 : (c0 | 4u);
        }
}

// Corners (Morton-numbered) joined by edge e, in the reference's edge order
// 02 23 31 10 46 67 75 54 04 26 37 15 (src/SVO.cu:610,638-663).
__host__ __device__ constexpr int edge_corner(int e, int s) {
    return (int)(((s ? 0x576445760132ull : 0x132057641320ull) >> (4 * e)) & 0xFull);
}

// Warp copy of nbytes (multiple of 8) from shared to global memory, in
// 16-byte streaming stores.
__device__ __forceinline__ void warp_copy_out(const uint4 *src, char *dst, uint32_t nbytes, int lane) {
    const uint32_t nv = nbytes / 16;
    uint4 *d4 = reinterpret_cast<uint4 *>(dst);
    for (uint32_t v = lane; v < nv; v += 32) __stcs(d4 + v, src[v]);
    if ((nbytes & 15) && lane == 0) {
        const unsigned long long *s8 = reinterpret_cast<const unsigned long long *>(src);
        __stcs(reinterpret_cast<unsigned long long *>(dst) + nv * 2, s8[nv * 2]);
    }
}

// The warp's staged bytes (shared memory, written by all lanes) to global
// memory as one bulk copy: both addresses 16-byte aligned, nbytes a multiple
// of 16.  The buffer may be rewritten after bulk_wait.
__device__ __forceinline__ void warp_bulk_out(const uint4 *src, char *dst, uint32_t nbytes, int lane) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the lanes' writes, before the copy reads them
    __syncwarp();
    if (lane == 0) {
        uint64_t first;  // evict first: the outputs are not read again here
        asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(first));
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group.L2::cache_hint [%0], [%1], %2, %3;" ::"l"(dst),
                     "r"((uint32_t)__cvta_generic_to_shared(src)), "r"(nbytes), "l"(first)
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
}
__device__ __forceinline__ void bulk_wait(int lane) {
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncwarp();
}

__device__ __forceinline__ bool veq(const float *a, const float *b) {
    return a[0] == b[0] && a[1] == b[1] && a[2] == b[2];
}

// Consecutive duplicates (thrust::unique, src/SVO.cu:679-725) among this node's
// vertices and edges and between them and the previous node's last ones: the
// previous node has width pw and origin po; first: there is none.
__device__ __forceinline__ void count_duplicates(const float *o, float w, const float *po, float pw, bool first,
                                              uint32_t &vdup, uint32_t &edup) {
    float vp[8][3], cp[8][3];
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            vp[c][a] = __fmul_rn(w, (float)((c >> a) & 1));
            cp[c][a] = c == 0 ? o[a] : __fadd_rn(o[a], (c >> a) & 1 ? w : 0.0f);
        }
#pragma unroll
    for (int i = 1; i < 8; ++i) vdup += veq(vp[i], vp[i - 1]);
#pragma unroll
    for (int e = 1; e < 12; ++e) {
        const float *a0 = cp[edge_corner(e - 1, 0)], *a1 = cp[edge_corner(e - 1, 1)];
        const float *b0 = cp[edge_corner(e, 0)], *b1 = cp[edge_corner(e, 1)];
        edup += (veq(a0, b0) && veq(a1, b1)) || (veq(a0, b1) && veq(a1, b0));
    }
    if (first) return;
    const float pv7[3] = {__fmul_rn(pw, 1.0f), __fmul_rn(pw, 1.0f), __fmul_rn(pw, 1.0f)};
    vdup += veq(vp[0], pv7);
    // previous node's edge 11 = (corner 1, corner 5)
    const float q1[3] = {__fadd_rn(po[0], pw), __fadd_rn(po[1], 0.0f), __fadd_rn(po[2], 0.0f)};
    const float q5[3] = {__fadd_rn(po[0], pw), __fadd_rn(po[1], 0.0f), __fadd_rn(po[2], pw)};
    const float *b0 = cp[0], *b1 = cp[2];
    edup += (veq(q1, b0) && veq(q5, b1)) || (veq(q1, b1) && veq(q5, b0));
}

constexpr int kEmitWarps = 4;
constexpr int kEmitBufBytes = 32 * 168;  // per warp: 32 node records, then the edges of 16 nodes at a time
constexpr int kOwnBytes = 32 * 9 * 4;    // vertex owners (full neighbour tables)

// ONE: a single mesh whose parameters travel in the kernel's parameter space
// (`one`, read through the constant cache); otherwise each warp looks up its
// mesh in the batch table (global memory, L1-cached).
// Node records and edges are staged per warp and leave as bulk copies (the
// edges 16 nodes at a time, which halves the stage), vertices straight from
// registers, everything marked to leave L2 first.  The kernel is bound by
// writes: the SMs' path to L2 is 77% busy (32 bytes per clock and SM; 84% with
// full tables) and DRAM 85% (83%).  633 bytes a node: 27.4M nodes in 2,380 us
// (7.3 TB/s), with full neighbour tables, whose look-ups cost the same memory
// pipe, in 2,540 to 2,580 (2,680 with 7 look-ups per node, plain stores and the
// whole edge stage at 5 CTAs per SM).
// 6 CTAs per SM, 80 registers a thread: with full tables a lone mesh's variant
// spills 72 bytes of stores and 108 of loads a thread and the one over a mesh
// table 92 and 232, the others none.  Beside the dedup that still gains
// (heightfield at res 2048 with dedup 4,150 us for the build, 4,255 with 5, 4,240
// before): six leave 4,096 registers of an SM, a dedup CTA takes 11,264 or
// 12,288, so each one displaces an emission CTA, and five stay where four did
// with 5.  The vertex and edge arrays alone gain 1% from 6 instead of 8 (torus
// soup 1,900 us, 1,912), node records alone need 8 (121 us for 3.7M nodes, 139).
// Without the eviction mark the outputs crowd out the bitmaps (heightfield at
// res 1024 864 us, 840 with it).
template <bool S, bool FULL, bool VE, bool ONE>
__global__ void __launch_bounds__(kEmitWarps * 32, FULL || VE ? 6 : 8)
    k_emit(EmitBatch eb, const __grid_constant__ EmitParams one, uint64_t total) {
    chain_begin();
    extern __shared__ __align__(128) uint4 smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kWarpBytes = kEmitBufBytes + (VE && FULL ? kOwnBytes : 0);
    uint4 *wbuf = smem + warp * (kWarpBytes / 16);
    const uint64_t nwarps = (uint64_t)gridDim.x * kEmitWarps;
    for (uint64_t gbase = ((uint64_t)blockIdx.x * kEmitWarps + warp) * 32; gbase < total; gbase += nwarps * 32) {
        const int mj = ONE ? 0 : find_segment(eb.node_off, eb.n, gbase);
        const EmitParams &P = ONE ? one : eb.p[mj];
        const uint64_t base = ONE ? gbase : gbase - eb.node_off[mj];
        if (base >= P.N) continue;  // padding between meshes
        const float go[3] = {P.gp->origin[0], P.gp->origin[1], P.gp->origin[2]};
        const uint32_t t = (uint32_t)(base + lane);
        const bool valid = base + lane < P.N;
        const uint32_t cnt = (uint32_t)(P.N - base < 32 ? P.N - base : 32);
        NodeInfo ni;
        if (valid) node_info<S>(P, go, t, ni);
        if (VE) {
            // Consecutive duplicates need a corner that coincides with another of the
            // same node: consecutive edges differ in some corner, and the previous
            // node's last edge has one y where this node's first has two.  So a node
            // whose width shows in all three coordinates has none, and the previous
            // node is looked up only in the rare rest (degenerate widths, coordinates
            // that absorb the width): that look-up and the 36 comparisons took every
            // warp a sixth of its instructions.
            if (__any_sync(0xFFFFFFFFu, valid && (ni.w == 0.0f || __fadd_rn(ni.o[0], ni.w) == ni.o[0] ||
                                                  __fadd_rn(ni.o[1], ni.w) == ni.o[1] ||
                                                  __fadd_rn(ni.o[2], ni.w) == ni.o[2]))) {
                float pw = __shfl_up_sync(0xFFFFFFFFu, valid ? ni.w : 0.0f, 1);
                float po[3], o[3] = {ni.o[0], ni.o[1], ni.o[2]};
#pragma unroll
                for (int a = 0; a < 3; ++a) po[a] = __shfl_up_sync(0xFFFFFFFFu, valid ? ni.o[a] : 0.0f, 1);
                if (lane == 0 && valid && t > 0) {
                    NodeInfo pn;
                    node_info<S>(P, go, t - 1, pn);
                    pw = pn.w;
                    po[0] = pn.o[0];
                    po[1] = pn.o[1];
                    po[2] = pn.o[2];
                }
                uint32_t vdup = 0, edup = 0;
                if (valid) count_duplicates(o, ni.w, po, pw, t == 0, vdup, edup);
                vdup = __reduce_add_sync(0xFFFFFFFFu, vdup);
                edup = __reduce_add_sync(0xFFFFFFFFu, edup);
                // the first of them raises the host's flag: only then are the counters read back
                if (lane == 0 && vdup && atomicAdd(P.dups, (unsigned long long)vdup) == 0) *P.dup_flag = 1;
                if (lane == 0 && edup && atomicAdd(P.dups + 1, (unsigned long long)edup) == 0) *P.dup_flag = 1;
            }
        }
        uint32_t nb[27];
#pragma unroll
        for (int j = 0; j < 27; ++j) nb[j] = kNone;
        bulk_wait(lane);  // the buffer's last copy has been read
        if (FULL) {
            full_neighbors(P, ni, t, valid && ni.l < P.T, lane, reinterpret_cast<uint32_t *>(wbuf), nb);
            if (valid && ni.l == P.T) nb[13] = t;
            __syncwarp();  // the table is read before the records take its place
        } else if (valid && ni.l == P.T && P.T >= 1) {
            nb[13] = t;  // root self entry, src/SVO.cu:522-529,556-557
        }
        // ---- node records (21 u64 words each) ----
        if (valid) {
            unsigned long long *d = reinterpret_cast<unsigned long long *>(wbuf) + lane * 21;
            const uint32_t leaf = (ni.l == 0 || !ni.real) ? 1u : 0u;
            uint32_t ch[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) ch[k] = ni.real ? ni.child0 + k : kNone;
            auto pk = [](uint32_t lo, uint32_t hi) { return ((unsigned long long)hi << 32) | lo; };
            d[0] = pk((uint32_t)ni.code, leaf);
            d[1] = pk(__float_as_uint(ni.o[0]), __float_as_uint(ni.o[1]));
            d[2] = pk(__float_as_uint(ni.o[2]), __float_as_uint(ni.w));
            d[3] = pk(ni.parent, ch[0]);
            d[4] = pk(ch[1], ch[2]);
            d[5] = pk(ch[3], ch[4]);
            d[6] = pk(ch[5], ch[6]);
            d[7] = pk(ch[7], nb[0]);
#pragma unroll
            for (int k = 0; k < 13; ++k) d[8 + k] = pk(nb[1 + 2 * k], nb[2 + 2 * k]);
        }
        if (cnt == 32) {
            warp_bulk_out(wbuf, reinterpret_cast<char *>(P.nodes) + base * 168, 32 * 168, lane);
        } else {  // the mesh's last nodes
            __syncwarp();
            warp_copy_out(wbuf, reinterpret_cast<char *>(P.nodes) + base * 168, cnt * 168, lane);
            __syncwarp();
        }
        if (!VE) continue;
        // ---- vertices: corner i = width * (i&1, i>>1&1, i>>2&1), src/SVO.cu:586-608 ----
        // Stored in output order straight from registers: lane l writes corner
        // l & 7 of nodes 4j + (l >> 3).  Only the owners of full neighbour
        // tables go through shared memory, beside the node records.
        uint32_t *vown = reinterpret_cast<uint32_t *>(wbuf) + kEmitBufBytes / 4;
        // Owners with full neighbour tables: the smallest node sharing the vertex (8
        // nodes) or the edge (4), one axis at a time: pairs along x, then y, then z.
        // The neighbours come back from the staged record: held in registers across
        // the staging they spilled (12% of the instructions were local loads and
        // stores, beside a memory pipe that is the bottleneck here).
        uint32_t eown[12];
        if (FULL) {
            const unsigned long long *rec = reinterpret_cast<const unsigned long long *>(wbuf) + lane * 21;
            nb[0] = (uint32_t)(rec[7] >> 32);
#pragma unroll
            for (int k = 0; k < 13; ++k) {
                const unsigned long long v = rec[8 + k];
                nb[1 + 2 * k] = (uint32_t)v;
                nb[2 + 2 * k] = (uint32_t)(v >> 32);
            }
            uint32_t px[2][3][3], pxy[2][2][3];  // [x pair][y][z], [x pair][y pair][z]
            uint32_t xe[2][2], ye[2][2], ze[2][2];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    xe[i][j] = min(min(nb[1 + 3 * i + 9 * j], nb[4 + 3 * i + 9 * j]),
                                   min(nb[10 + 3 * i + 9 * j], nb[13 + 3 * i + 9 * j]));
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int y = 0; y < 3; ++y)
#pragma unroll
                    for (int z = 0; z < 3; ++z) px[i][y][z] = min(nb[i + 3 * y + 9 * z], nb[i + 1 + 3 * y + 9 * z]);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    ye[i][j] = min(px[i][1][j], px[i][1][j + 1]);
#pragma unroll
                    for (int z = 0; z < 3; ++z) pxy[i][j][z] = min(px[i][j][z], px[i][j + 1][z]);
                    ze[i][j] = pxy[i][j][1];
                }
#pragma unroll
            for (int c = 0; c < 8; ++c)
                vown[lane * 9 + c] = min(pxy[c & 1][(c >> 1) & 1][c >> 2], pxy[c & 1][(c >> 1) & 1][(c >> 2) + 1]);
#pragma unroll
            for (int e = 0; e < 12; ++e) {
                const int a = edge_corner(e, 0), ax = a ^ edge_corner(e, 1);
                eown[e] = ax == 1 ? xe[(a >> 1) & 1][a >> 2] : ax == 2 ? ye[a & 1][a >> 2] : ze[a & 1][(a >> 1) & 1];
            }
        } else {
#pragma unroll
            for (int e = 0; e < 12; ++e) eown[e] = t;
        }
        if (FULL) __syncwarp();
        {
            uint4 *d4 = reinterpret_cast<uint4 *>(P.verts + base * 8);
            const float mine = valid ? ni.w : 0.0f;
            const int k = lane & 7;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t node = 4 * j + (lane >> 3);
                const float w = __shfl_sync(0xFFFFFFFFu, mine, (int)node);
                const uint32_t own = FULL ? vown[node * 9 + k] : (uint32_t)base + node;
                if (node < cnt)
                    __stcs(d4 + lane + 32 * j, make_uint4(__float_as_uint(__fmul_rn(w, (float)(k & 1))),
                                                          __float_as_uint(__fmul_rn(w, (float)((k >> 1) & 1))),
                                                          __float_as_uint(__fmul_rn(w, (float)((k >> 2) & 1))), own));
            }
        }
        // ---- edges: 12 per node in the reference's order, src/SVO.cu:629-677 ----
        // a corner's coordinates: corner 0 is the origin itself, the others add 0 or the width
        float oz[3], ow[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            oz[a] = __fadd_rn(ni.o[a], 0.0f);
            ow[a] = __fadd_rn(ni.o[a], ni.w);
        }
        // 16 nodes at a time through the buffer, 84 words per node: edge e = p0 (3), p1 (3), owner
#pragma unroll 1
        for (uint32_t h = 0; h < 2; ++h) {
            bulk_wait(lane);  // the node records, or the first half, have been read
            if (valid && (uint32_t)(lane >> 4) == h) {
                uint4 *d = wbuf + (lane & 15) * 21;
#pragma unroll
                for (int j = 0; j < 21; ++j) {
                    uint32_t wv[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int wi = 4 * j + q, e = wi / 7, f = wi % 7;
                        const int c = edge_corner(e, f < 3 ? 0 : 1), a = f % 3;
                        wv[q] = f == 6 ? eown[e] : __float_as_uint(c == 0 ? ni.o[a] : (c >> a) & 1 ? ow[a] : oz[a]);
                    }
                    d[j] = make_uint4(wv[0], wv[1], wv[2], wv[3]);
                }
            }
            char *dst = reinterpret_cast<char *>(P.edges) + (base + 16 * h) * 336;
            if (cnt == 32) {
                warp_bulk_out(wbuf, dst, 16 * 336, lane);
            } else {
                __syncwarp();
                const uint32_t left = cnt > 16 * h ? (cnt - 16 * h < 16 ? cnt - 16 * h : 16) : 0;
                warp_copy_out(wbuf, dst, left * 336, lane);
                __syncwarp();
            }
        }
    }
    bulk_wait(lane);  // shared memory is read to the end before the block leaves
}

// ---------------------------------------------------------------------------
// Stable removal of consecutive duplicates (rare path).
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool same(const svo_vertex &a, const svo_vertex &b) { return veq(a.pos, b.pos); }
__device__ __forceinline__ bool same(const svo_edge &a, const svo_edge &b) {
    return (veq(a.p0, b.p0) && veq(a.p1, b.p1)) || (veq(a.p0, b.p1) && veq(a.p1, b.p0));
}

template <class T>
__global__ void __launch_bounds__(256) k_unique_count(const T *__restrict__ in, uint64_t n,
                                                      uint32_t *__restrict__ tile_counts) {
    __shared__ uint32_t s[8];
    const uint64_t t0 = (uint64_t)blockIdx.x * kUniqueTile;
    uint32_t c = 0;
    for (uint32_t k = threadIdx.x; k < kUniqueTile; k += blockDim.x) {
        const uint64_t i = t0 + k;
        if (i < n) c += (i == 0 || !same(in[i - 1], in[i]));
    }
    c = __reduce_add_sync(0xFFFFFFFFu, c);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t tot = 0;
        for (int w = 0; w < 8; ++w) tot += s[w];
        tile_counts[blockIdx.x] = tot;
    }
}

template <class T>
__global__ void __launch_bounds__(256) k_unique_scatter(const T *__restrict__ in, uint64_t n,
                                                        const uint32_t *__restrict__ tile_pre,
                                                        T *__restrict__ out) {
    __shared__ uint32_t s_w[8];
    const uint64_t t0 = (uint64_t)blockIdx.x * kUniqueTile;
    uint32_t run = tile_pre[blockIdx.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t k0 = 0; k0 < kUniqueTile; k0 += blockDim.x) {
        const uint64_t i = t0 + k0 + threadIdx.x;
        const bool keep = i < n && (i == 0 || !same(in[i - 1], in[i]));
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, keep);
        if (lane == 0) s_w[warp] = __popc(m);
        __syncthreads();
        uint32_t before = 0, tot = 0;
        for (int w = 0; w < 8; ++w) {
            if (w < warp) before += s_w[w];
            tot += s_w[w];
        }
        if (keep) out[run + before + __popc(m & ((1u << lane) - 1u))] = in[i];
        run += tot;
        __syncthreads();
    }
}

template <class T>
cudaError_t unique_impl(const T *in, uint64_t n, T *out, uint32_t *tile_counts, uint32_t *tile_pre,
                        unsigned long long *scan_scratch, uint32_t *status, cudaStream_t st) {
    const uint64_t tiles = (n + kUniqueTile - 1) / kUniqueTile;
    if (tiles == 0) return cudaSuccess;
    k_unique_count<T><<<(unsigned)tiles, 256, 0, st>>>(in, n, tile_counts);
    count_launches(1);
    cudaError_t e = launch_scan(tile_counts, tile_pre, tiles, scan_scratch, status, st);
    if (e != cudaSuccess) return e;
    k_unique_scatter<T><<<(unsigned)tiles, 256, 0, st>>>(in, n, tile_pre, out);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_pyramid(const BatchDev &b, uint32_t total_ctas, uint32_t max_ctas, int num_sms, cudaStream_t st) {
    if (total_ctas == 0) return cudaSuccess;
    const MeshDev one = b.one ? *b.one : MeshDev{};
    if (max_ctas <= kFuseRegions && total_ctas <= (uint32_t)num_sms * 8) {
        const uint32_t blocks = std::min<uint32_t>(total_ctas, (uint32_t)num_sms * 4);
        if (b.one) launch_chained(k_pyramid<true, true>, blocks, 256, 0, st, b, one, total_ctas);
        else launch_chained(k_pyramid<true, false>, blocks, 256, 0, st, b, one, total_ctas);
        count_launches(1);
        return cudaGetLastError();
    }
    const uint32_t blocks = std::min<uint32_t>(total_ctas, (uint32_t)num_sms * 8);
    if (b.one) {
        launch_chained(k_pyramid<false, true>, blocks, 256, 0, st, b, one, total_ctas);
        launch_chained(k_pyramid_finish<true>, dim3(b.n, 5), 1024, 0, st, b, one);
    } else {
        launch_chained(k_pyramid<false, false>, blocks, 256, 0, st, b, one, total_ctas);
        launch_chained(k_pyramid_finish<false>, dim3(b.n, 5), 1024, 0, st, b, one);
    }
    count_launches(2);
    return cudaGetLastError();
}

size_t scan_scratch_words(uint64_t n) { return 1 + (n + kScanTile - 1) / kScanTile; }

cudaError_t launch_scan(const uint32_t *in, uint32_t *out, uint64_t n, unsigned long long *scratch,
                        uint32_t *status, cudaStream_t st) {
    const uint64_t tiles = (n + kScanTile - 1) / kScanTile;
    if (tiles >= kScanSplitTiles && tiles <= 0x7FFFFFFFull &&
        ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
        // tile sums and their prefixes live in the look-back scratch (tiles + 1 u64 words)
        uint32_t *tsum = reinterpret_cast<uint32_t *>(scratch), *tpre = tsum + tiles;
        k_scan_reduce<<<(unsigned)tiles, kScanThreads, 0, st>>>(in, n, tsum);
        k_scan_tiles<<<1, 1024, 0, st>>>(tsum, tpre, tiles, out + n);
        k_scan_down<<<(unsigned)tiles, kScanThreads, 0, st>>>(in, out, n, tpre);
        count_launches(3);
        return cudaGetLastError();
    }
    cudaError_t e = cudaMemsetAsync(scratch, 0, scan_scratch_words(n) * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    if (tiles == 0) return cudaMemsetAsync(out, 0, sizeof(uint32_t), st);
    k_scan<<<(unsigned)tiles, kScanThreads, 0, st>>>(in, out, n, scratch, status, kSpinLimit);
    count_launches(1);
    return cudaGetLastError();
}

size_t scan_stalled_scratch_words(uint64_t n) { return scan_scratch_words(n) + 1; }

cudaError_t launch_scan_stalled(const uint32_t *in, uint32_t *out, uint64_t n, unsigned long long *scratch,
                                uint32_t *status, int spin_limit, cudaStream_t st) {
    const uint64_t tiles = (n + kScanTile - 1) / kScanTile;
    if (tiles < 2 || tiles > 0x7FFFFFFFull || spin_limit < 1) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(scratch, 0, scan_stalled_scratch_words(n) * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    // the tile counter starts at 1: tile 0 is never run and never publishes
    const unsigned long long one = 1;
    if ((e = cudaMemcpyAsync(scratch, &one, sizeof(one), cudaMemcpyHostToDevice, st)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    k_scan<<<(unsigned)tiles, kScanThreads, 0, st>>>(in, out, n, scratch, status, spin_limit);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_compact(const CompactBatch &c, const CompactJob *one, uint64_t total_words, cudaStream_t st) {
    if (total_words == 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((total_words + 255) / 256);
    if (one) k_compact<true><<<blocks, 256, 0, st>>>(c, *one, total_words);
    else k_compact<false><<<blocks, 256, 0, st>>>(c, CompactJob{}, total_words);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_compact_regions(const CompactJob &job, const uint32_t *rlist, const uint32_t *rcount, uint32_t cta0,
                                   uint32_t regions, int num_sms, cudaStream_t st) {
    if (regions == 0) return cudaSuccess;
    launch_chained(k_compact_regions, std::min<uint32_t>(regions, (uint32_t)num_sms * 8), 256, 0, st, job, rlist, rcount,
                   cta0, regions);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_compact_keys(const KeyBatch &k, const KeyJob *one, uint64_t total_blocks, cudaStream_t st) {
    if (total_blocks == 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((total_blocks * 8 + 255) / 256);
    if (one) k_compact_keys<true><<<blocks, 256, 0, st>>>(k, *one, total_blocks);
    else k_compact_keys<false><<<blocks, 256, 0, st>>>(k, KeyJob{}, total_blocks);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_emit(const EmitBatch &b, const EmitParams *one, uint64_t total, uint32_t flags, int num_sms,
                        cudaStream_t st) {
    if (total == 0) return cudaSuccess;
    const uint64_t warps = (total + 31) / 32;
    const unsigned blocks = (unsigned)std::max<uint64_t>(
        1, std::min<uint64_t>((warps + kEmitWarps - 1) / kEmitWarps, 0x7FFFFFFFull));
    const bool s = (flags & SVO_FLAG_STRICT_FP) != 0, f = (flags & SVO_FLAG_FULL_NEIGHBORS) != 0,
               ve = (flags & SVO_FLAG_NO_VERT_EDGE) == 0;
    const size_t shmem = (size_t)kEmitWarps * (kEmitBufBytes + (ve && f ? kOwnBytes : 0));
    const EmitParams p1 = one ? *one : EmitParams{};
#define SVO_EMIT1(S_, F_, V_)                                                                       \
    do {                                                                                             \
        if (one) launch_chained(k_emit<S_, F_, V_, true>, blocks, kEmitWarps * 32, shmem, st, b, p1, total);   \
        else launch_chained(k_emit<S_, F_, V_, false>, blocks, kEmitWarps * 32, shmem, st, b, p1, total);     \
    } while (0)
#define SVO_EMIT(S_, F_, V_) SVO_EMIT1(S_, F_, V_)
    if (s) {
        if (f) { if (ve) SVO_EMIT(true, true, true); else SVO_EMIT(true, true, false); }
        else { if (ve) SVO_EMIT(true, false, true); else SVO_EMIT(true, false, false); }
    } else {
        if (f) { if (ve) SVO_EMIT(false, true, true); else SVO_EMIT(false, true, false); }
        else { if (ve) SVO_EMIT(false, false, true); else SVO_EMIT(false, false, false); }
    }
#undef SVO_EMIT1
#undef SVO_EMIT
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_unique_vertices(const svo_vertex *in, uint64_t n, svo_vertex *out, uint32_t *tile_counts,
                                   uint32_t *tile_pre, unsigned long long *scan_scratch, uint32_t *status,
                                   cudaStream_t st) {
    return unique_impl(in, n, out, tile_counts, tile_pre, scan_scratch, status, st);
}

cudaError_t launch_unique_edges(const svo_edge *in, uint64_t n, svo_edge *out, uint32_t *tile_counts,
                                uint32_t *tile_pre, unsigned long long *scan_scratch, uint32_t *status,
                                cudaStream_t st) {
    return unique_impl(in, n, out, tile_counts, tile_pre, scan_scratch, status, st);
}

}  // namespace svo
