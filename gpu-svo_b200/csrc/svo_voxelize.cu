// svo_voxelize.cu -- bounding cube and conservative surface voxelization.
//
// Restates the reference's BaseModel bounding cube (src/BaseModel.h:24-49,
// 64-73) and surfaceVoxelize (src/SVO.cu:37-188) for sm_100a.  Instead of one
// thread per triangle writing a dense u32 array of res^3 entries, each overlap
// sets one bit of a Morton-ordered occupancy bitmap (res^3 bits); the test
// arithmetic is the reference's, operation for operation (svo_device.cuh Fp).
//
// Work split: a triangle whose grid bbox has at most `serial_max` voxels is
// tested by its own thread: the edge tests of each projection once per
// coordinate pair (bit masks), the plane test only where all three masks
// agree.  Larger triangles are queued and walked by warps: brick columns along
// the triangle's dominant axis (4x4 voxels wide, packed one per lane), the
// 4x4x4 bricks of each column near the triangle's plane (packed one per
// lane), then the voxels of the bricks that survive culling, a brick per lane.
// A brick is 64 consecutive Morton codes, two bitmap words.  Without a
// queue (the allocation-free entry point) the triangle's own warp walks its
// columns in place.
//
// Brick culling is exact.  Every predicate of the voxel test is monotone in
// each grid coordinate separately (each is built from rounded products,
// sums and fmas of p = coordinate * unit, and IEEE rounding is monotone), so
// over a brick an edge test is largest at the corner picked by the signs of
// its two coefficients, and n.p is smallest/largest at the corners picked by
// the signs of n.  A brick is skipped only when one predicate, evaluated at
// its best corner with the voxel test's own arithmetic, already fails.  The
// bricks of a column that are not looked at lie more than a voxel outside the
// plane's slab, far beyond the rounding of the estimate (warp_columns).
// Triangles with any non-finite setup value are never culled.
#include "svo_internal.h"

namespace svo {

namespace {


__device__ __forceinline__ uint32_t f2ord(float f) {
    uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ord2f(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o);
}

// ---------------------------------------------------------------------------
// Bounding box of all vertices (exact min/max through an order-preserving
// integer map), then the bounding cube on one thread.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void bbox_take(float v, int a, uint32_t lo[3], uint32_t hi[3], bool &bad) {
    bad |= !isfinite(v);
    const uint32_t o = f2ord(v);
    lo[a] = min(lo[a], o);
    hi[a] = max(hi[a], o);
}

// Block `blk` of the `nb` blocks of mesh md's reduction.  When the mesh's
// points are 16-byte aligned, 4 points (12 floats, 3 float4) per step; the
// component of float k is k % 3, the same in every 12-float group.  md.mm
// holds the mesh's largest ~key (0..2: the smallest keys) and largest key
// (3..5) so far, so that zero is the start value of all six; returns true in
// every thread of the mesh's last block, with md.mm complete.
__device__ __forceinline__ bool bbox_block(const MeshDev &md, uint32_t blk, uint32_t nb) {
    const float *__restrict__ pts = md.pts;
    const int64_t n = md.n_pts;
    uint32_t lo[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, hi[3] = {0u, 0u, 0u};
    bool bad = false;
    const int64_t tid = blk * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nth = (int64_t)nb * blockDim.x;
    int64_t done = 0;
    if ((reinterpret_cast<uintptr_t>(pts) & 15) == 0) {
        const float4 *p4 = reinterpret_cast<const float4 *>(pts);
        const int64_t groups = n / 4;
        for (int64_t gi = tid; gi < groups; gi += nth) {
            const float4 a = __ldcs(p4 + 3 * gi), b = __ldcs(p4 + 3 * gi + 1), c = __ldcs(p4 + 3 * gi + 2);
            bbox_take(a.x, 0, lo, hi, bad); bbox_take(a.y, 1, lo, hi, bad); bbox_take(a.z, 2, lo, hi, bad);
            bbox_take(a.w, 0, lo, hi, bad); bbox_take(b.x, 1, lo, hi, bad); bbox_take(b.y, 2, lo, hi, bad);
            bbox_take(b.z, 0, lo, hi, bad); bbox_take(b.w, 1, lo, hi, bad); bbox_take(c.x, 2, lo, hi, bad);
            bbox_take(c.y, 0, lo, hi, bad); bbox_take(c.z, 1, lo, hi, bad); bbox_take(c.w, 2, lo, hi, bad);
        }
        done = groups * 4;
    }
    for (int64_t i = done + tid; i < n; i += nth)
#pragma unroll
        for (int a = 0; a < 3; ++a) bbox_take(__ldg(pts + 3 * i + a), a, lo, hi, bad);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = __reduce_min_sync(0xFFFFFFFFu, lo[a]);
        hi[a] = __reduce_max_sync(0xFFFFFFFFu, hi[a]);
    }
    if (__any_sync(0xFFFFFFFFu, bad) && (threadIdx.x & 31) == 0) atomicOr(&md.gp->status, kStatusNonFinite);
    // the block's extremes, then one atomic per value and block (the 6 words
    // are shared by every block of the mesh)
    __shared__ uint32_t wmm[32][6];
    __shared__ uint32_t s_last;
    const int warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            wmm[warp][a] = ~lo[a];
            wmm[warp][3 + a] = hi[a];
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        uint32_t v = wmm[0][threadIdx.x];
        for (int w = 1; w < nwarp; ++w) v = max(v, wmm[w][threadIdx.x]);
        atomicMax(md.mm + threadIdx.x, v);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        s_last = atomicAdd(md.mm + 6, 1u) == nb - 1 ? 1u : 0u;
        __threadfence();
    }
    __syncthreads();
    return s_last != 0;
}

// createMeshBBCube (src/BaseModel.h:24-49) and unitVoxelSize
// (src/SVO.cu:348-350), one thread.  Host code in the reference: no
// contraction there, so every operation is an explicitly rounded intrinsic.
__device__ __forceinline__ void grid_setup(const MeshDev &md) {
    GridParams *gp = md.gp;
    float mn[3], mx[3], len[3], amin[3], amax[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        mn[a] = ord2f(~__ldcg(md.mm + a));
        mx[a] = ord2f(__ldcg(md.mm + 3 + a));
        len[a] = __fsub_rn(mx[a], mn[a]);
        amin[a] = mn[a];
        amax[a] = mx[a];
    }
    const float maxlen = cmaxf(len[0], cmaxf(len[1], len[2]));
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (maxlen == len[a]) continue;
        const float half = __fdiv_rn(__fsub_rn(maxlen, len[a]), 2.0f);
        amin[a] = __fsub_rn(mn[a], half);
        amax[a] = __fadd_rn(mx[a], half);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float eps = __fdiv_rn(__fsub_rn(amax[a], amin[a]), 10001.0f);
        amin[a] = __fsub_rn(amin[a], eps);
        amax[a] = __fadd_rn(amax[a], eps);
        const float w = __fsub_rn(amax[a], amin[a]);
        gp->bbox[a] = amin[a];
        gp->bbox[3 + a] = amax[a];
        gp->bbox[6 + a] = w;
        gp->origin[a] = amin[a];
        gp->unit[a] = __fdiv_rn(w, (float)md.res[a]);
    }
}

// The first kernel of a build, two independent jobs side by side:
//   * blocks [0, bbox_blocks): the bounding cube of every mesh (block b
//     belongs to the mesh whose segment of bbox_off holds b); a mesh's last
//     block sets up its grid;
//   * the other blocks clear the bitmaps: level 0 of the meshes that are not
//     in region mode (those clear their flagged regions later), the level-0
//     region flags, and the words the pyramid does not write whole (level-3
//     padding, level 4, which it writes as 32-bit halves, and levels >= 5).
// (One kernel instead of the five launches it replaces: in a small build the
// host's launches are the critical path.  The meta words are cleared by a memset
// before it: cleared here, by one block up to 2,048 points and by a cluster of
// eight up to 32,768, 320 triangles at 32^3 take 83.2 us against 83.1 and 30k
// at 300 x 200 x 100 143.0 against 137.9, for eight blocks read the points
// slower than the memset costs.)
template <bool ONE>
__global__ void __launch_bounds__(256) k_front(const __grid_constant__ BatchDev bd, const __grid_constant__ MeshDev one,
                                               uint32_t bbox_blocks, uint32_t regions, uint32_t flag_words) {
    chain_begin();
    const Meshes<ONE> mesh{bd, one};
    if (blockIdx.x < bbox_blocks) {
        const int m = ONE ? 0 : find_segment(bd.bbox_off, bd.n, (uint32_t)blockIdx.x);
        const uint32_t b0 = ONE ? 0u : bd.bbox_off[m], nb = ONE ? bbox_blocks : bd.bbox_off[m + 1] - b0;
        if (bbox_block(mesh[m], blockIdx.x - b0, nb) && threadIdx.x == 0) grid_setup(mesh[m]);
        return;
    }
    const uint32_t zb = blockIdx.x - bbox_blocks, nz = gridDim.x - bbox_blocks;
    if (flag_words) {  // some mesh is in region mode: its level 0 is not cleared here
        for (uint32_t i = zb * blockDim.x + threadIdx.x; i < flag_words; i += nz * blockDim.x)
            reinterpret_cast<uint32_t *>(bd.rflag)[i] = 0;
        for (int m = 0; m < bd.n; ++m) {
            const MeshDev &md = mesh[m];
            if (!md.regions) continue;
            const uint64_t end = md.py.total_words, step = (uint64_t)nz * blockDim.x;
            for (uint64_t i = md.py.woff[3] + 4ull * md.py.ctas + zb * blockDim.x + threadIdx.x; i < end; i += step)
                md.bits[i] = 0;
        }
        if (ONE) return;  // (65,536 regions at res 2048: looking through them took 25 us)
    }
    for (uint32_t g = zb; g < regions; g += nz) {
        const int m = mesh.of_region(g);
        const MeshDev &md = mesh[m];
        if (md.regions) continue;
        const uint32_t r = g - mesh.first_region(m);
        uint4 *w = reinterpret_cast<uint4 *>(md.bits + md.py.woff[0] + (uint64_t)r * 2048);
#pragma unroll
        for (int q = 0; q < 4; ++q) w[threadIdx.x + 256 * q] = make_uint4(0, 0, 0, 0);
        const uint64_t z0 = md.py.woff[3] + 4ull * md.py.ctas;
        for (uint64_t i = z0 + (uint64_t)r * 256 + threadIdx.x; i < md.py.total_words; i += (uint64_t)md.py.ctas * 256)
            md.bits[i] = 0;
    }
}

// ---------------------------------------------------------------------------
// Triangle setup (src/SVO.cu:53-149).
// ---------------------------------------------------------------------------
struct Tri {
    float n[3];
    float d1, d2;
    float ea[9], eb[9], ed[9];  // edge test k of plane p at 3p+k: XY, YZ, ZX
    int lo[3], hi[3];
    int cull;                   // all setup values finite: brick culling allowed
};

__device__ __forceinline__ int f2i_rz(float f) { return __float2int_rz(f); }
__device__ __forceinline__ int clampi(int f, int a, int b) { return max(a, min(f, b)); }

// Voxel bbox of a triangle (vertices relative to the grid origin), clamped
// to the grid: src/SVO.cu:58-66.  The region marker and the voxel test use
// this one function, so the regions cover every voxel the test can set.
__device__ __forceinline__ void tri_box(const GridParams &g, const int res[3], const float v[3][3], int lo[3],
                                        int hi[3]) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float mn = cminf(v[0][a], cminf(v[1][a], v[2][a]));
        const float mx = cmaxf(v[0][a], cmaxf(v[1][a], v[2][a]));
        lo[a] = clampi(f2i_rz(__fdiv_rn(mn, g.unit[a])), 0, res[a] - 1);
        hi[a] = clampi(f2i_rz(__fdiv_rn(mx, g.unit[a])), 0, res[a] - 1);
    }
}

template <bool S>
__device__ __forceinline__ void tri_setup(const GridParams &g, const int res[3], const float *p0,
                                          const float *p1, const float *p2, Tri &t) {
    float v[3][3], e[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        v[0][a] = __fsub_rn(p0[a], g.origin[a]);
        v[1][a] = __fsub_rn(p1[a], g.origin[a]);
        v[2][a] = __fsub_rn(p2[a], g.origin[a]);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        e[0][a] = __fsub_rn(v[1][a], v[0][a]);
        e[1][a] = __fsub_rn(v[2][a], v[1][a]);
        e[2][a] = __fsub_rn(v[0][a], v[2][a]);
    }
    // n = e0.cross(e1).normalized()
    float c0 = Fp<S>::diffprod(e[0][1], e[1][2], e[0][2], e[1][1]);
    float c1 = Fp<S>::diffprod(e[0][2], e[1][0], e[0][0], e[1][2]);
    float c2 = Fp<S>::diffprod(e[0][0], e[1][1], e[0][1], e[1][0]);
    // squared norm: c0*c0 + (c1*c1 + c2*c2), the inner sum fusing c2*c2
    const float sq = Fp<S>::dot3_head(c0, c0, Fp<S>::dot2_late(c1, c2, c1, c2));
    if (sq > 0.0f) {
        const float r = __fsqrt_rn(sq);
        c0 = __fdiv_rn(c0, r);
        c1 = __fdiv_rn(c1, r);
        c2 = __fdiv_rn(c2, r);
    }
    t.n[0] = c0;
    t.n[1] = c1;
    t.n[2] = c2;
    const float *u = g.unit;
    tri_box(g, res, v, t.lo, t.hi);
    float ca[3], cb[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float c = t.n[a] > 0.0f ? u[a] : 0.0f;
        ca[a] = __fsub_rn(c, v[0][a]);
        cb[a] = __fsub_rn(__fsub_rn(u[a], c), v[0][a]);
    }
    t.d1 = Fp<S>::dot3(t.n[0], t.n[1], t.n[2], ca[0], ca[1], ca[2]);
    t.d2 = Fp<S>::dot3(t.n[0], t.n[1], t.n[2], cb[0], cb[1], cb[2]);
    // projections: plane (i, j) with flip axis f: XY (0,1,2), YZ (1,2,0), ZX (2,0,1)
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const int i = p == 0 ? 0 : (p == 1 ? 1 : 2);
        const int j = p == 0 ? 1 : (p == 1 ? 2 : 0);
        const int f = p == 0 ? 2 : (p == 1 ? 0 : 1);
        const bool flip = t.n[f] < 0.0f;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            float a0 = -e[k][j];
            float a1 = e[k][i];
            if (flip) {
                a0 = -a0;
                a1 = -a1;
            }
            const float dt = Fp<S>::dot2(a0, a1, v[k][i], v[k][j]);
            t.ea[3 * p + k] = a0;
            t.eb[3 * p + k] = a1;
            // (+ 0: a negative zero becomes a positive one, which no comparison of the sums sees)
            t.ed[3 * p + k] = __fadd_rn(__fadd_rn(__fadd_rn(-dt, cmaxf(0.0f, __fmul_rn(u[i], a0))),
                                                  cmaxf(0.0f, __fmul_rn(u[j], a1))),
                                        0.0f);
        }
    }
    // 0 * x is a zero for every finite x and NaN otherwise
    float fin = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) fin = __fmaf_rn(t.n[k], 0.0f, __fmaf_rn(u[k], 0.0f, fin));
    fin = __fmaf_rn(t.d1, 0.0f, __fmaf_rn(t.d2, 0.0f, fin));
#pragma unroll
    for (int k = 0; k < 9; ++k)
        fin = __fmaf_rn(t.ea[k], 0.0f, __fmaf_rn(t.eb[k], 0.0f, __fmaf_rn(t.ed[k], 0.0f, fin)));
    t.cull = fin == 0.0f ? 1 : 0;
}

// Bits of v (< 2^10) spread to every third bit.
__device__ __forceinline__ uint32_t spread3_small(uint32_t v) {
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    return (v | (v << 2)) & 0x09249249u;
}

// The voxel test (src/SVO.cu:156-177) at p = (x, y, z) * unit: the plane test
// rejects where (n.p + d1) (n.p + d2) > 0, nine edge tests where a sum is
// negative.  One edge test, its two products named by the loop they vary in:
// fast (the fused one) and slow (rounded first).  XY: fast x, slow y; YZ: fast
// y, slow z; ZX: fast x, slow z (in the reference's loop a * p.z does not vary
// with x, is hoisted, and nvcc then fuses the other product).
template <bool S>
__device__ __forceinline__ bool edge_fails(float cf, float pf, float slow, float ed) {
    const float f = S ? __fadd_rn(__fmul_rn(cf, pf), slow) : __fmaf_rn(cf, pf, slow);
    return __fadd_rn(f, ed) < 0.0f;
}

// Deepest box of the serial tier.
constexpr int kSerialDepth = 8;

// The three edge tests of one projection over NF (at most 4, the same in the
// whole warp) pairs along its fast coordinate: bit f is set where one fails.
// A sum is below zero exactly when its sign bit is set: tri_setup leaves no
// negative zero in ed, so no sum is one, and a NaN sum (it does not fail) is
// the canonical positive one.
template <bool S>
__device__ __forceinline__ uint32_t edge_fail_row(const float *cf, const float *cs, const float *ed, const float pf[4],
                                                  float ps, int NF) {
    uint32_t m = 0;
    const float h0 = __fmul_rn(cs[0], ps), h1 = __fmul_rn(cs[1], ps), h2 = __fmul_rn(cs[2], ps);
#pragma unroll
    for (int i = 3; i >= 0; --i) {
        if (i >= NF) continue;
        const float v0 = __fadd_rn(S ? __fadd_rn(__fmul_rn(cf[0], pf[i]), h0) : __fmaf_rn(cf[0], pf[i], h0), ed[0]);
        const float v1 = __fadd_rn(S ? __fadd_rn(__fmul_rn(cf[1], pf[i]), h1) : __fmaf_rn(cf[1], pf[i], h1), ed[1]);
        const float v2 = __fadd_rn(S ? __fadd_rn(__fmul_rn(cf[2], pf[i]), h2) : __fmaf_rn(cf[2], pf[i], h2), ed[2]);
        m = __funnelshift_l(__float_as_uint(fminf(fminf(v0, v1), v2)), m, 1);
    }
    return m;
}

// The serial tier: the warp's lanes each test every voxel of their own
// triangle's bbox (on: the lane has one), at most 4 x 4 x kSerialDepth.  An
// edge test depends on two coordinates only, so the XY tests run once, the ZX
// and YZ tests once per slice, the plane test once per voxel, and the masks
// are combined slice by slice; no branch depends on a lane's own triangle,
// only on the largest box of the warp.
// The hits of a slice pair (a bitmap word holds 4 x 4 x 2 voxels, and the walk
// begins at an even z in every lane) are collected for the 2 x 2 bricks an
// unaligned box can reach and written with at most four atomicOr.
// Bound by issue (73 to 76% of the slots).
// One loop per lane over its own rows and voxels, with their early exits, costs
// the warp its largest triangle's loops: 407 us for the 5M triangles (2-3
// voxels across) of the heightfield at res 2048 against 336 us this way, 90
// against 70 for 1M at res 1024, 160 against 86 for the torus soup.  Wider
// boxes, as several 4 x 4 tiles, are slower here than in the column tier:
// 320 triangles at res 32 31 us against 17 for the whole voxelizer, the torus
// soup 240 against 220.
template <bool S>
__device__ __forceinline__ void serial_tile(const Tri &t, const float unit[3], uint32_t *__restrict__ bm, bool on) {
    const int nx = on ? t.hi[0] - t.lo[0] + 1 : 0, ny = on ? t.hi[1] - t.lo[1] + 1 : 0, z0 = on ? t.lo[2] & ~1 : 0,
              nz = on ? t.hi[2] - z0 + 1 : 0;  // slices from the even z0
    const int NX = (int)__reduce_max_sync(0xFFFFFFFFu, (uint32_t)nx), NY = (int)__reduce_max_sync(0xFFFFFFFFu, (uint32_t)ny),
              NZ = (int)__reduce_max_sync(0xFFFFFFFFu, (uint32_t)nz);
    const int x0 = on ? t.lo[0] : 0, y0 = on ? t.lo[1] : 0;
    const float fx = (float)x0, fy = (float)y0;
    float px[4], py[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // small integers: the sums are exact
        px[k] = __fmul_rn(fx + (float)k, unit[0]);
        py[k] = __fmul_rn(fy + (float)k, unit[1]);
    }
    uint32_t xy = 0;  // bit 4 y + x
#pragma unroll
    for (int y = 3; y >= 0; --y)
        if (y < NY) xy = xy << 4 | edge_fail_row<S>(t.ea, t.eb, t.ed, px, py[y], NX);
    const uint32_t xm = (1u << nx) - 1u;
    xy = ~xy & (xm * 0x1111u) & ((1u << (4 * ny)) - 1u);
    const uint32_t xs = (uint32_t)x0 & 3u, ys8 = ((uint32_t)y0 & 3u) * 8u;
    // dilated brick coordinates of the word index (brick code << 1 | z bit 1)
    constexpr uint32_t kX = 0x09249249u << 1, kY = kX << 1;
    const uint32_t wx0 = spread3_small((uint32_t)x0 >> 2) << 1, wy0 = spread3_small((uint32_t)y0 >> 2) << 2;
    uint32_t a00 = 0, a10 = 0, a01 = 0, a11 = 0;  // a[x brick][y brick] of the current word layer
    float fz = (float)z0;
    uint32_t zz = (uint32_t)z0;
    for (int z = 0; z < NZ; ++z, ++zz, fz += 1.0f) {  // word layers begin at even z: the same step in every lane
        const float pz = __fmul_rn(fz, unit[2]);
        const uint32_t zr = ~edge_fail_row<S>(t.eb + 6, t.ea + 6, t.ed + 6, px, pz, NX) & 15u;
        const uint32_t yr = ~edge_fail_row<S>(t.ea + 3, t.eb + 3, t.ed + 3, py, pz, NY) & 15u;
        const uint32_t rows = (yr | yr << 3 | yr << 6 | yr << 9) & 0x1111u;  // row y at bit 4 y
        // plane: fails where (n.p + d1) (n.p + d2) > 0
        uint32_t fails = 0;
        const float nzp = __fmul_rn(t.n[2], pz);
#pragma unroll
        for (int y = 3; y >= 0; --y) {
            if (y >= NY) continue;
            fails <<= 4 - NX;
            const float inner = S ? __fadd_rn(__fmul_rn(t.n[1], py[y]), nzp) : __fmaf_rn(t.n[1], py[y], nzp);
#pragma unroll
            for (int x = 3; x >= 0; --x) {
                if (x >= NX) continue;
                const float nd = Fp<S>::dot3_head(t.n[0], px[x], inner);
                const float p = __fmul_rn(__fadd_rn(nd, t.d1), __fadd_rn(nd, t.d2));
                fails = __funnelshift_l(__float_as_uint(__fsub_rn(0.0f, p)), fails, 1);  // sign: p > 0
            }
        }
        const uint32_t hit = z < nz && (int)zz >= t.lo[2] ? xy & ~fails & (zr * 0x1111u) & (rows * 15u) : 0u;
        // rows to bytes, moved to the tile's place in an 8 x 8 square (bit 8 y + x)
        uint32_t sq = (hit | hit << 8) & 0x00FF00FFu;
        sq = ((sq | sq << 4) & 0x0F0F0F0Fu) << xs;
        uint32_t q0 = sq << ys8, q1 = __funnelshift_l(sq, 0u, ys8);
        // swap x bit 1 and y bit 0: bits x0, y0, (x brick), x1, y1
        uint32_t w = (q0 ^ (q0 >> 6)) & 0x00CC00CCu;
        q0 ^= w ^ (w << 6);
        w = (q1 ^ (q1 >> 6)) & 0x00CC00CCu;
        q1 ^= w ^ (w << 6);
        const uint32_t sz = (uint32_t)(z & 1) << 2;  // z0 takes the x brick's bit
        a00 |= (q0 & 0x0F0F0F0Fu) << sz;
        a10 |= ((q0 >> 4) & 0x0F0F0F0Fu) << sz;
        a01 |= (q1 & 0x0F0F0F0Fu) << sz;
        a11 |= ((q1 >> 4) & 0x0F0F0F0Fu) << sz;
        if (((z & 1) || z == NZ - 1) && (a00 | a10 | a01 | a11)) {  // the word layer ends
            const uint32_t wx1 = ((wx0 | ~kX) + 2u) & kX, wy1 = ((wy0 | ~kY) + 4u) & kY;
            const uint32_t wz = spread3_small(zz >> 2) << 3 | ((zz >> 1) & 1u);
            if (a00) atomicOr(bm + (wz | wx0 | wy0), a00);
            if (a10) atomicOr(bm + (wz | wx1 | wy0), a10);
            if (a01) atomicOr(bm + (wz | wx0 | wy1), a01);
            if (a11) atomicOr(bm + (wz | wx1 | wy1), a11);
            a00 = a10 = a01 = a11 = 0;
        }
    }
}

// True when no voxel of the box lo..hi (inclusive) can pass: one predicate
// fails at its most favourable corner (see the comment at the top).
template <bool S>
__device__ __forceinline__ bool brick_reject(const Tri &t, const float *unit, const int lo[3], const int hi[3]) {
    float pl[3], ph[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        pl[a] = __fmul_rn((float)lo[a], unit[a]);
        ph[a] = __fmul_rn((float)hi[a], unit[a]);
    }
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const int i = p == 0 ? 0 : (p == 1 ? 1 : 2);
        const int j = p == 0 ? 1 : (p == 1 ? 2 : 0);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float a = t.ea[3 * p + k], b = t.eb[3 * p + k];
            const float pi = a >= 0.0f ? ph[i] : pl[i];
            const float pj = b >= 0.0f ? ph[j] : pl[j];
            const float f = p == 2 ? Fp<S>::dot2_late(a, b, pi, pj) : Fp<S>::dot2(a, b, pi, pj);
            if (__fadd_rn(f, t.ed[3 * p + k]) < 0.0f) return true;
        }
    }
    // n.p at its smallest and largest corners
    const float x0 = t.n[0] >= 0.0f ? pl[0] : ph[0], x1 = t.n[0] >= 0.0f ? ph[0] : pl[0];
    const float y0 = t.n[1] >= 0.0f ? pl[1] : ph[1], y1 = t.n[1] >= 0.0f ? ph[1] : pl[1];
    const float z0 = t.n[2] >= 0.0f ? pl[2] : ph[2], z1 = t.n[2] >= 0.0f ? ph[2] : pl[2];
    const float nd0 = Fp<S>::dot3_head(t.n[0], x0, Fp<S>::dot3_tail(t.n[1], t.n[2], y0, z0));
    const float nd1 = Fp<S>::dot3_head(t.n[0], x1, Fp<S>::dot3_tail(t.n[1], t.n[2], y1, z1));
    const float dlo = t.d1 <= t.d2 ? t.d1 : t.d2, dhi = t.d1 <= t.d2 ? t.d2 : t.d1;
    {  // everything above the slab: both factors positive from the smallest n.p on
        const float sa = __fadd_rn(nd0, dlo), sb = __fadd_rn(nd0, dhi);
        if (sa > 0.0f && __fmul_rn(sa, sb) > 0.0f) return true;
    }
    {  // everything below: both factors negative up to the largest n.p
        const float sa = __fadd_rn(nd1, dlo), sb = __fadd_rn(nd1, dhi);
        if (sb < 0.0f && __fmul_rn(sa, sb) > 0.0f) return true;
    }
    return false;
}

// The bricks of 32 lanes at once, one per lane (on: the lane has one): the
// serial tier's slices over an aligned 4x4x4 box, clipped to the triangle's
// bbox.  Bound by issue.  The form before, a brick per half-warp and a row of
// it per lane, took more instructions a brick (whole voxelizer of a batch of 15 meshes
// 177 us, 124 this way; torus soup 281 and 220).
template <bool S>
__device__ __forceinline__ void brick_lanes(const Tri &t, const float unit[3], uint32_t *__restrict__ bm, int sx, int sy,
                                            int sz, bool on) {
    float px[4], py[4];
    const float fx = (float)(4 * sx), fy = (float)(4 * sy), fz = (float)(4 * sz);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        px[k] = __fmul_rn(fx + (float)k, unit[0]);
        py[k] = __fmul_rn(fy + (float)k, unit[1]);
    }
    // bits lo..hi of each axis, relative to the brick
    auto span = [](int lo, int hi) { return (2u << min(hi, 3)) - (1u << max(lo, 0)); };
    const uint32_t xm = span(t.lo[0] - 4 * sx, t.hi[0] - 4 * sx), ym = span(t.lo[1] - 4 * sy, t.hi[1] - 4 * sy),
                   zm = on ? span(t.lo[2] - 4 * sz, t.hi[2] - 4 * sz) : 0u;
    uint32_t xy = 0;
#pragma unroll
    for (int y = 3; y >= 0; --y) xy = xy << 4 | edge_fail_row<S>(t.ea, t.eb, t.ed, px, py[y], 4);
    xy = ~xy & (xm * 0x1111u) & ((((ym | ym << 3 | ym << 6 | ym << 9) & 0x1111u) * 15u));
    uint32_t layer[2] = {0, 0};
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const float pz = __fmul_rn(fz + (float)z, unit[2]);
        const uint32_t zr = ~edge_fail_row<S>(t.eb + 6, t.ea + 6, t.ed + 6, px, pz, 4) & 15u;
        const uint32_t yr = ~edge_fail_row<S>(t.ea + 3, t.eb + 3, t.ed + 3, py, pz, 4) & 15u;
        const uint32_t rows = (yr | yr << 3 | yr << 6 | yr << 9) & 0x1111u;
        uint32_t fails = 0;
        const float nzp = __fmul_rn(t.n[2], pz);
#pragma unroll
        for (int y = 3; y >= 0; --y) {
            const float inner = S ? __fadd_rn(__fmul_rn(t.n[1], py[y]), nzp) : __fmaf_rn(t.n[1], py[y], nzp);
#pragma unroll
            for (int x = 3; x >= 0; --x) {
                const float nd = Fp<S>::dot3_head(t.n[0], px[x], inner);
                const float p = __fmul_rn(__fadd_rn(nd, t.d1), __fadd_rn(nd, t.d2));
                fails = __funnelshift_l(__float_as_uint(__fsub_rn(0.0f, p)), fails, 1);  // sign: p > 0
            }
        }
        uint32_t hit = (zm >> z) & 1u ? xy & ~fails & (zr * 0x1111u) & (rows * 15u) : 0u;
        // bits x0 x1 y0 y1 -> x0 y0 (z0) x1 y1
        const uint32_t w = (hit ^ (hit >> 2)) & 0x0C0Cu;
        hit ^= w ^ (w << 2);
        hit = (hit | hit << 8) & 0x00FF00FFu;
        layer[z >> 1] |= ((hit | hit << 4) & 0x0F0F0F0Fu) << (4 * (z & 1));
    }
    uint32_t *word = bm + ((spread3_small((uint32_t)sx) | spread3_small((uint32_t)sy) << 1 | spread3_small((uint32_t)sz) << 2) << 1);
    if (layer[0]) atomicOr(word, layer[0]);
    if (layer[1]) atomicOr(word + 1, layer[1]);
}

// The axis along which triangle t's plane is crossed fastest: the columns of
// its walk run along it.
__device__ __forceinline__ int column_axis(const Tri &t, const float unit[3]) {
    const float a = fabsf(t.n[0]) * unit[0], b = fabsf(t.n[1]) * unit[1], c = fabsf(t.n[2]) * unit[2];
    return c >= a && c >= b ? 2 : b >= a ? 1 : 0;
}

// Brick columns of triangle t along axis d.
__device__ __forceinline__ uint32_t column_count(const Tri &t, int d) {
    const uint32_t nx = (uint32_t)((t.hi[0] >> 2) - (t.lo[0] >> 2) + 1), ny = (uint32_t)((t.hi[1] >> 2) - (t.lo[1] >> 2) + 1),
                   nz = (uint32_t)((t.hi[2] >> 2) - (t.lo[2] >> 2) + 1);
    return d == 0 ? ny * nz : d == 1 ? nz * nx : nx * ny;
}

// The vertices of an indexed triangle after checking its indices against the
// mesh's n_pts vertices; false (nothing read) when one is outside.  Soups are
// always in range.
__device__ __forceinline__ bool load_tri_checked(const float *__restrict__ pts, const int32_t *__restrict__ tris,
                                                 int64_t n_pts, int64_t t, float p[3][3]) {
    if (tris) {
        int64_t vi[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) vi[k] = __ldg(tris + 3 * t + k);
        if ((uint64_t)vi[0] >= (uint64_t)n_pts || (uint64_t)vi[1] >= (uint64_t)n_pts ||
            (uint64_t)vi[2] >= (uint64_t)n_pts)
            return false;
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int a = 0; a < 3; ++a) p[k][a] = __ldg(pts + 3 * vi[k] + a);
        return true;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int a = 0; a < 3; ++a) p[k][a] = __ldg(pts + 9 * t + 3 * k + a);
    return true;
}

// The same for a triangle that k_voxelize has already checked.
__device__ __forceinline__ void load_tri(const float *__restrict__ pts, const int32_t *__restrict__ tris,
                                         int64_t t, float p[3][3]) {
    if (tris) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int64_t vi = __ldg(tris + 3 * t + k);
#pragma unroll
            for (int a = 0; a < 3; ++a) p[k][a] = __ldg(pts + 3 * vi + a);
        }
    } else {
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int a = 0; a < 3; ++a) p[k][a] = __ldg(pts + 9 * t + 3 * k + a);
    }
}

// Lane that owns item `item` when lane i owns the items up to incl[i]
// (inclusive counts over the warp): the number of lanes whose count is <= item.
__device__ __forceinline__ int owner_lane(uint32_t incl, uint32_t item) {
    int pos = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
        const uint32_t v = __shfl_sync(0xFFFFFFFFu, incl, pos + step - 1);
        if (v <= item) pos += step;
    }
    return pos;
}

__device__ __forceinline__ uint32_t warp_inclusive(uint32_t v, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, d);
        if (lane >= d) v += y;
    }
    return v;
}

// Walks the warp's triangles st[i] (shared memory; mesh sm[i]): lane i brings
// the cnt brick columns from c0 on of triangle st[i] (cnt = 0: none).  Three
// rounds, each packed across the triangles with one item per lane, so that
// lanes stay busy whatever the triangles' shapes:
//   1. a column (4x4 voxels across, along the triangle's dominant axis d): the
//      three edge tests of the projection along d reject it, or the slab
//      between the test's two planes bounds its bricks to the few the plane
//      crosses -- a triangle L bricks across costs L^2 items here, not L^3;
//   2. a brick of a surviving column: the exact culling test (brick_reject);
//   3. the voxels of the surviving bricks, collected in pend (64 words of
//      shared memory), 32 at a time, one per lane (brick_lanes).
// The slab bound of round 1 is estimated in float: a voxel passes only if
// -dhi <= n.p <= -dlo (dlo, dhi: the test's two offsets), n.p = q * k + a with
// q = n_d * unit_d per voxel and a over the column's footprint.  |q| is the
// largest of the three |n_i| unit_i and a grid has at most 2048 voxels per
// axis, so the rounding of n.p, the offsets and the estimate is below 0.01 |q|;
// the bound is widened by a whole voxel (|q|) on each side.  Without a usable
// q (degenerate or subnormal normals: |q| < 1e-15, where products of two such
// distances could underflow) the whole column is taken.
// Tri's 39-word stride is odd: distinct triangles fall in distinct banks.
template <bool S, bool ONE>
__device__ __forceinline__ void warp_columns(const Meshes<ONE> &mesh, const Tri *st, const int *sm, uint32_t *pend, uint32_t c0,
                                             uint32_t cnt, int lane) {
    const uint32_t incl = warp_inclusive(cnt, lane);
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
    const uint32_t first = c0 - (incl - cnt);  // item i of this lane is column first + i
    uint32_t npend = 0;  // the same in all lanes
    auto flush = [&](uint32_t n) {  // the first n <= 32 pending bricks, one per lane
        const bool on = (uint32_t)lane < n;
        const uint32_t bw = on ? pend[lane] : pend[0];
        const Tri &t = st[bw >> 27];
        const MeshDev &md = mesh[sm[bw >> 27]];
        const float unit[3] = {md.gp->unit[0], md.gp->unit[1], md.gp->unit[2]};
        brick_lanes<S>(t, unit, reinterpret_cast<uint32_t *>(md.bits), (int)(bw & 511u), (int)((bw >> 9) & 511u),
                       (int)((bw >> 18) & 511u), on);
        __syncwarp();
    };
    for (uint32_t base = 0; base < total; base += 32) {
        // ---- round 1: a column per lane ----
        const uint32_t item = base + lane;
        const int pos = owner_lane(incl, item);
        const int src = item < total ? pos : 0;
        const uint32_t c = item + __shfl_sync(0xFFFFFFFFu, first, src);
        uint32_t kn = 0, col = 0;  // bricks to look at; column: bi | bj << 9 | d << 18 | src << 20
        int k0 = 0;
        if (item < total) {
            const Tri &t = st[src];
            const GridParams *gp = mesh[sm[src]].gp;
            const float u[3] = {gp->unit[0], gp->unit[1], gp->unit[2]};
            const int d = column_axis(t, u), i = d == 2 ? 0 : d + 1, j = d == 0 ? 2 : d - 1;
            const int p = i;  // the projection along d: XY (0), YZ (1), ZX (2)
            const float ui = i == 0 ? u[0] : i == 1 ? u[1] : u[2], uj = j == 0 ? u[0] : j == 1 ? u[1] : u[2],
                        ud = d == 0 ? u[0] : d == 1 ? u[1] : u[2];
            const uint32_t nbi = (uint32_t)((t.hi[i] >> 2) - (t.lo[i] >> 2) + 1);
            const uint32_t cj = c / nbi;
            const int bi = (t.lo[i] >> 2) + (int)(c - cj * nbi), bj = (t.lo[j] >> 2) + (int)cj;
            const int lo_d = t.lo[d], hi_d = t.hi[d];
            bool live = true;
            int ka = lo_d, kb = hi_d;  // voxels along d
            if (t.cull) {
                const float pli = __fmul_rn((float)max(4 * bi, t.lo[i]), ui), phi = __fmul_rn((float)min(4 * bi + 3, t.hi[i]), ui);
                const float plj = __fmul_rn((float)max(4 * bj, t.lo[j]), uj), phj = __fmul_rn((float)min(4 * bj + 3, t.hi[j]), uj);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float ea = t.ea[3 * p + k], eb = t.eb[3 * p + k];
                    const float pi = ea >= 0.0f ? phi : pli, pj = eb >= 0.0f ? phj : plj;
                    const float f = p == 2 ? Fp<S>::dot2_late(ea, eb, pi, pj) : Fp<S>::dot2(ea, eb, pi, pj);
                    live &= !(__fadd_rn(f, t.ed[3 * p + k]) < 0.0f);
                }
                const float q = t.n[d] * ud;
                if (fabsf(q) >= 1e-15f) {
                    const float ai = t.n[i] * pli, bi_ = t.n[i] * phi, aj = t.n[j] * plj, bj_ = t.n[j] * phj;
                    const float alo = fminf(ai, bi_) + fminf(aj, bj_), ahi = fmaxf(ai, bi_) + fmaxf(aj, bj_);
                    const float v0 = (-fmaxf(t.d1, t.d2) - ahi) / q, v1 = (-fminf(t.d1, t.d2) - alo) / q;
                    const float va = fminf(v0, v1) - 1.0f, vb = fmaxf(v0, v1) + 1.0f;
                    if (isfinite(va) && isfinite(vb)) {
                        live &= va <= (float)hi_d && vb >= (float)lo_d;
                        ka = (int)fmaxf(floorf(va), (float)lo_d);
                        kb = (int)fminf(ceilf(vb), (float)hi_d);
                    }
                }
            }
            if (live && ka <= kb) {
                k0 = ka >> 2;
                kn = (uint32_t)((kb >> 2) - k0 + 1);
                col = (uint32_t)bi | (uint32_t)bj << 9 | (uint32_t)d << 18 | (uint32_t)src << 20;
            }
        }
        // ---- round 2: a brick per lane ----
        const uint32_t kincl = warp_inclusive(kn, lane);
        const uint32_t ktotal = __shfl_sync(0xFFFFFFFFu, kincl, 31);
        const int kfirst = k0 - (int)(kincl - kn);
        for (uint32_t kbase = 0; kbase < ktotal; kbase += 32) {
            const uint32_t it = kbase + lane;
            const int q = owner_lane(kincl, it);
            const int own = it < ktotal ? q : 0;
            const uint32_t cw = __shfl_sync(0xFFFFFFFFu, col, own);
            const int kz = (int)it + __shfl_sync(0xFFFFFFFFu, kfirst, own);
            bool live = false;
            uint32_t brick = 0;  // bx | by << 9 | bz << 18 | triangle << 27
            if (it < ktotal) {
                const int ts = (int)(cw >> 20), d = (int)((cw >> 18) & 3u), bi = (int)(cw & 511u), bj = (int)((cw >> 9) & 511u);
                const Tri &t = st[ts];
                const int bx = d == 0 ? kz : d == 1 ? bj : bi, by = d == 0 ? bi : d == 1 ? kz : bj,
                          bz = d == 0 ? bj : d == 1 ? bi : kz;
                const int lo[3] = {max(4 * bx, t.lo[0]), max(4 * by, t.lo[1]), max(4 * bz, t.lo[2])};
                const int hi[3] = {min(4 * bx + 3, t.hi[0]), min(4 * by + 3, t.hi[1]), min(4 * bz + 3, t.hi[2])};
                live = !t.cull || !brick_reject<S>(t, mesh[sm[ts]].gp->unit, lo, hi);
                brick = (uint32_t)bx | (uint32_t)by << 9 | (uint32_t)bz << 18 | (uint32_t)ts << 27;
            }
            // ---- round 3: the survivors' voxels ----
            const uint32_t lm = __ballot_sync(0xFFFFFFFFu, live);
            if (live) pend[npend + __popc(lm & ((1u << lane) - 1u))] = brick;
            npend += __popc(lm);
            __syncwarp();
            if (npend >= 32) {
                flush(32);
                npend -= 32;
                const uint32_t keep = (uint32_t)lane < npend ? pend[32 + lane] : 0u;
                __syncwarp();
                if ((uint32_t)lane < npend) pend[lane] = keep;
                __syncwarp();
            }
        }
    }
    if (npend) flush(npend);
}

// One thread per triangle of the batch (global index -> mesh by tri_off):
// setup, then
//   tier 0 (grid bbox of at most serial_max voxels, 4 x 4 x kSerialDepth):
//     every voxel by this thread;
//   tier 1 (larger): queue entries of at most `cols` brick columns for
//     k_voxelize_columns, which balances them across the GPU; INPLACE (no
//     queue), its columns are walked by this warp right away.
template <bool S, bool INPLACE, bool ONE>
__global__ void __launch_bounds__(256, INPLACE ? 2 : 3)
    k_voxelize(const __grid_constant__ BatchDev bd, const __grid_constant__ MeshDev one, int64_t total,
               uint32_t serial_max, uint32_t cols, uint4 *__restrict__ big, uint32_t big_cap,
               uint32_t *__restrict__ big_count) {
    chain_begin();
    const Meshes<ONE> mesh{bd, one};
    __shared__ Tri s_tri[INPLACE ? 8 : 1][32];  // the warp's tier-1 triangles
    __shared__ int s_mesh[INPLACE ? 8 : 1][32];  // their meshes
    __shared__ uint32_t s_pend[INPLACE ? 8 : 1][64];
    const int lane = threadIdx.x & 31;
    const int64_t warp0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) - lane;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = warp0; base < total; base += stride) {
        const int64_t gid = base + lane;
        Tri t;
        uint32_t ncol = 0;
        int tier = -1, m = 0;
        if (gid < total) {
            m = mesh.of_tri((uint64_t)gid);
            const MeshDev &md = mesh[m];
            const GridParams g = *md.gp;
            float p[3][3];
            if (load_tri_checked(md.pts, md.tris, md.n_pts, gid - (int64_t)mesh.first_tri(m), p)) {
                tri_setup<S>(g, md.res, p[0], p[1], p[2], t);
                const int nx = t.hi[0] - t.lo[0] + 1, ny = t.hi[1] - t.lo[1] + 1, nz = t.hi[2] - t.lo[2] + 1;
                tier = nx <= 4 && ny <= 4 && nz <= kSerialDepth && (uint32_t)(nx * ny * nz) <= serial_max ? 0 : 1;
                if (tier == 1) ncol = column_count(t, column_axis(t, g.unit));
            } else {
                atomicOr(&md.gp->status, kStatusBadIndex);  // tier stays -1: the triangle is skipped
            }
        }
        if (__any_sync(0xFFFFFFFFu, tier == 0)) {
            const MeshDev &md = mesh[m];
            const float unit[3] = {md.gp->unit[0], md.gp->unit[1], md.gp->unit[2]};
            serial_tile<S>(t, unit, reinterpret_cast<uint32_t *>(md.bits), tier == 0);
        }
        if (!__any_sync(0xFFFFFFFFu, tier == 1)) continue;
        if (INPLACE) {
            Tri *st = s_tri[threadIdx.x >> 5];
            int *sm = s_mesh[threadIdx.x >> 5];
            if (tier == 1) {
                st[lane] = t;
                sm[lane] = m;
            }
            __syncwarp();
            warp_columns<S, ONE>(mesh, st, sm, s_pend[threadIdx.x >> 5], 0, ncol, lane);
            __syncwarp();  // st is rewritten by the next round
        } else {
            // one append per warp; entries past the queue's end are counted, not
            // written (the host grows the queue and runs the phase again)
            const uint32_t ne = (ncol + cols - 1) / cols;
            const uint32_t incl = warp_inclusive(ne, lane);
            uint32_t at = 0;
            if (lane == 31) at = atomicAdd(big_count, incl);
            at = __shfl_sync(0xFFFFFFFFu, at, 31) + incl - ne;
            for (uint32_t e = 0; e < ne && at + e < big_cap; ++e)
                big[at + e] = make_uint4((uint32_t)gid, e * cols, min(ncol, (e + 1) * cols), (uint32_t)(gid >> 32));
        }
    }
}

// Queued triangles: a warp takes its share of the queue, at most 32 entries
// (triangle, column range) at a time, one per lane to set up, and walks their
// columns together (warp_columns).  A share at once keeps its lanes busy (30k
// triangles on a 300 x 200 x 100 grid: 31 us, with a quarter of it 68); 16
// columns per entry by default, since with 64 the last warps of a batch of 15
// meshes work alone (140 us against 124 with 24 already).  Its end is uneven (a
// batch of 15 meshes: 11 of 16 warps per SM busy on average), but smaller
// shares, the same from the start (6, 8, 16 entries) or falling towards the end
// of the queue, cost as much in setups and half-full rounds: batch 1,709-1,787
// us against 1,709-1,719, torus soup 1,882-1,942 against 1,872-1,882.
template <bool S, bool ONE>
__global__ void __launch_bounds__(256, 2) k_voxelize_columns(const __grid_constant__ BatchDev bd,
                                                             const __grid_constant__ MeshDev one,
                                                             const uint4 *big, const uint32_t *big_count,
                                                             uint32_t big_cap, uint32_t *cursor) {
    chain_begin();
    const Meshes<ONE> mesh{bd, one};
    __shared__ Tri s_tri[8][32];
    __shared__ int s_mesh[8][32];
    __shared__ uint32_t s_pend[8][64];
    const int lane = threadIdx.x & 31;
    Tri *st = s_tri[threadIdx.x >> 5];
    int *sm = s_mesh[threadIdx.x >> 5];
    const uint32_t n = *big_count;
    if (n > big_cap) return;  // reported to the host: the phase is run again
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t chunk = min(32u, (n + warps - 1) / warps);
    for (;;) {
        uint32_t e0 = 0;
        if (lane == 0) e0 = atomicAdd(cursor, chunk);
        e0 = __shfl_sync(0xFFFFFFFFu, e0, 0);
        if (e0 >= n) return;
        uint32_t c0 = 0, cnt = 0;
        if ((uint32_t)lane < chunk && e0 + lane < n) {
            const uint4 ent = big[e0 + lane];
            const int64_t gid = (int64_t)ent.x | ((int64_t)ent.w << 32);
            const int m = mesh.of_tri((uint64_t)gid);
            const MeshDev &md = mesh[m];
            const GridParams g = *md.gp;
            float p[3][3];
            load_tri(md.pts, md.tris, gid - (int64_t)mesh.first_tri(m), p);
            Tri t;
            tri_setup<S>(g, md.res, p[0], p[1], p[2], t);
            st[lane] = t;
            sm[lane] = m;
            c0 = ent.y;
            cnt = ent.z - ent.y;
        }
        __syncwarp();
        warp_columns<S, ONE>(mesh, st, sm, s_pend[threadIdx.x >> 5], c0, cnt, lane);
        __syncwarp();  // st is rewritten by the next chunk
    }
}

__global__ void k_index_init(int32_t *mm) {
    mm[0] = 0x7FFFFFFF;
    mm[1] = (int32_t)0x80000000;
}

__global__ void k_index_range(const int32_t *__restrict__ idx, int64_t n, int32_t *__restrict__ mm) {
    int32_t lo = 0x7FFFFFFF, hi = (int32_t)0x80000000;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = __ldg(idx + i);
        lo = min(lo, v);
        hi = max(hi, v);
    }
    lo = __reduce_min_sync(0xFFFFFFFFu, lo);
    hi = __reduce_max_sync(0xFFFFFFFFu, hi);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(mm, lo);
        atomicMax(mm + 1, hi);
    }
}

}  // namespace

cudaError_t launch_index_range(const int32_t *idx, int64_t n, int32_t *mm, cudaStream_t st) {
    k_index_init<<<1, 1, 0, st>>>(mm);
    count_launches(1);
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 8));
    k_index_range<<<blocks, 256, 0, st>>>(idx, n, mm);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_front(const BatchDev &b, uint32_t bbox_blocks, uint32_t total_ctas, bool any_regions, int num_sms,
                         cudaStream_t st) {
    const uint32_t blocks = bbox_blocks + std::min<uint32_t>(total_ctas, (uint32_t)num_sms * 8);
    const uint32_t flag_words = any_regions ? (total_ctas + 3) / 4 : 0;
    if (b.one) k_front<true><<<blocks, 256, 0, st>>>(b, *b.one, bbox_blocks, total_ctas, flag_words);
    else k_front<false><<<blocks, 256, 0, st>>>(b, MeshDev{}, bbox_blocks, total_ctas, flag_words);
    count_launches(1);
    return cudaGetLastError();
}

namespace {

// Flags the level-0 regions (64 x 64 x 32 voxels, region index =
// morton3(x, y, z) >> 17) that each triangle's voxel bbox overlaps, for
// region-mode meshes.  The bbox is tri_box's widened by one voxel on each side,
// with a product by the reciprocal voxel size in place of the division: the two
// differ by a few ulps at coordinates <= 2048, far less than the margin, so the
// flagged regions cover every voxel the voxel test can set.
// The kernel waits on gathers (indices, then vertices), so each thread takes 3
// triangles at a time and issues all their loads before using them; the mesh's
// grid and reciprocal units are kept while the mesh stays the same.
constexpr int kMarkBatch = 3;

template <bool ONE>
__global__ void __launch_bounds__(256) k_region_mark(const __grid_constant__ BatchDev bd, const __grid_constant__ MeshDev one,
                                                     int64_t total) {
    chain_begin();
    const Meshes<ONE> mesh{bd, one};
    int cur = -1;
    float org[3] = {0, 0, 0}, inv[3] = {0, 0, 0};
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t g0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g0 < total; g0 += stride * kMarkBatch) {
        int mk[kMarkBatch];
        bool live[kMarkBatch];
        int64_t vi[kMarkBatch][3];
#pragma unroll
        for (int k = 0; k < kMarkBatch; ++k) {
            const int64_t gid = g0 + k * stride;
            live[k] = gid < total;
            mk[k] = live[k] ? mesh.of_tri((uint64_t)gid) : 0;
            const MeshDev &md = mesh[mk[k]];
            live[k] = live[k] && md.regions != 0;
            const int64_t t = gid - (int64_t)mesh.first_tri(mk[k]);
#pragma unroll
            for (int j = 0; j < 3; ++j) vi[k][j] = live[k] ? (md.tris ? (int64_t)__ldg(md.tris + 3 * t + j) : 3 * t + j) : 0;
        }
        float p[kMarkBatch][3][3];
#pragma unroll
        for (int k = 0; k < kMarkBatch; ++k) {
            const MeshDev &md = mesh[mk[k]];
            // an index outside the mesh: skipped here, k_voxelize reports it
            live[k] = live[k] && (uint64_t)vi[k][0] < (uint64_t)md.n_pts && (uint64_t)vi[k][1] < (uint64_t)md.n_pts &&
                      (uint64_t)vi[k][2] < (uint64_t)md.n_pts;
#pragma unroll
            for (int j = 0; j < 3; ++j)
#pragma unroll
                for (int a = 0; a < 3; ++a) p[k][j][a] = live[k] ? __ldg(md.pts + 3 * vi[k][j] + a) : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < kMarkBatch; ++k) {
            if (!live[k]) continue;
            const MeshDev &md = mesh[mk[k]];
            if (mk[k] != cur) {
                cur = mk[k];
                // the one-voxel margin absorbs an approximate reciprocal (2 ulp)
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    org[a] = md.gp->origin[a];
                    inv[a] = __fdividef(1.0f, md.gp->unit[a]);
                }
            }
            int lo[3], hi[3];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                const float v0 = __fsub_rn(p[k][0][a], org[a]), v1 = __fsub_rn(p[k][1][a], org[a]),
                            v2 = __fsub_rn(p[k][2][a], org[a]);
                // the margin is applied before the conversion, so +-inf and NaN clamp as in tri_box
                lo[a] = clampi(f2i_rz(__fsub_rn(__fmul_rn(cminf(v0, cminf(v1, v2)), inv[a]), 1.0f)), 0, md.res[a] - 1);
                hi[a] = clampi(f2i_rz(__fadd_rn(__fmul_rn(cmaxf(v0, cmaxf(v1, v2)), inv[a]), 1.0f)), 0, md.res[a] - 1);
            }
            uint8_t *flag = bd.rflag + mesh.first_region(mk[k]);
            // region bits: z at 3i, x at 3i + 1, y at 3i + 2 (z in 32-voxel, x and y in 64-voxel steps)
            for (uint32_t rz = (uint32_t)lo[2] >> 5; rz <= (uint32_t)hi[2] >> 5; ++rz)
                for (uint32_t ry = (uint32_t)lo[1] >> 6; ry <= (uint32_t)hi[1] >> 6; ++ry)
                    for (uint32_t rx = (uint32_t)lo[0] >> 6; rx <= (uint32_t)hi[0] >> 6; ++rx) {
                        uint8_t *f = flag + (spread3_small(rz) | spread3_small(rx) << 1 | spread3_small(ry) << 2);
                        if (!*f) *f = 1;
                    }
        }
    }
}

// The level-0 regions of a batch with a region-mode mesh, 8 at a time per
// block: the regions to read are listed (one append per 8), a region-mode
// mesh's flagged ones zeroed at level 0, and its unflagged ones zeroed at levels
// 1..4 and in the region sums, which the pyramid then need not visit.  At res
// 2048 the heightfield reaches 3,170 of 65,536 regions; a block that looked at
// every region in turn waited for one flag after another (clearing, region
// pass, pyramid and compaction together 217 us, 127 with the list).
constexpr uint32_t kRegionChunk = 8;

template <bool ONE>
__global__ void __launch_bounds__(256) k_region_prepare(const __grid_constant__ BatchDev bd,
                                                        const __grid_constant__ MeshDev one, uint32_t total) {
    chain_begin();
    const Meshes<ONE> mesh{bd, one};
    __shared__ uint32_t s_live, s_zero;  // bits of the chunk: listed; region mode and unflagged
    const uint32_t t = threadIdx.x;
    for (uint32_t g0 = blockIdx.x * kRegionChunk; g0 < total; g0 += gridDim.x * kRegionChunk) {
        if (t < 32) {
            const uint32_t g = g0 + t;
            bool live = false, zero = false;
            if (t < kRegionChunk && g < total) {
                const bool flagged = bd.rflag[g] != 0;
                zero = mesh[mesh.of_region(g)].regions && !flagged;
                live = !zero;
            }
            const uint32_t lm = __ballot_sync(0xFFFFFFFFu, live), zm = __ballot_sync(0xFFFFFFFFu, zero);
            uint32_t at = 0;
            if (t == 0 && lm) at = atomicAdd(bd.rcount, (uint32_t)__popc(lm));
            at = __shfl_sync(0xFFFFFFFFu, at, 0);
            if (live) bd.rlist[at + __popc(lm & ((1u << t) - 1u))] = g;
            if (t == 0) {
                s_live = lm;
                s_zero = zm;
            }
        }
        __syncthreads();
        const uint32_t lm = s_live, zm = s_zero;
        for (uint32_t k = 0; k < kRegionChunk; ++k) {
            if (!(((lm | zm) >> k) & 1u)) continue;
            const uint32_t g = g0 + k;
            const int m = mesh.of_region(g);
            const MeshDev &md = mesh[m];
            const uint32_t b = g - mesh.first_region(m);
            if ((lm >> k) & 1u) {
                if (!md.regions) continue;  // cleared by k_front
                uint4 *w = reinterpret_cast<uint4 *>(md.bits + md.py.woff[0] + (uint64_t)b * 2048);
#pragma unroll
                for (int q = 0; q < 4; ++q) w[t + 256 * q] = make_uint4(0, 0, 0, 0);
            } else {
                uint64_t *bits = md.bits;
                bits[md.py.woff[1] + (uint64_t)b * 256 + t] = 0;
                if (t < 32) bits[md.py.woff[2] + (uint64_t)b * 32 + t] = 0;
                else if (t < 36) bits[md.py.woff[3] + (uint64_t)b * 4 + (t - 32)] = 0;
                else if (t < 40) md.base[(uint64_t)(t - 36) * md.bstride + b] = 0;
                else if (t == 40) reinterpret_cast<uint32_t *>(bits + md.py.woff[4])[b] = 0;
            }
        }
        __syncthreads();  // s_live, s_zero are rewritten by the next chunk
    }
}

}  // namespace

cudaError_t launch_regions(const BatchDev &b, int64_t total_tris, uint32_t total_ctas, int num_sms,
                           cudaStream_t st) {
    if (total_tris > 0) {
        const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((total_tris + 255) / 256, (int64_t)num_sms * 8));
        if (b.one) launch_chained(k_region_mark<true>, blocks, 256, 0, st, b, *b.one, total_tris);
        else launch_chained(k_region_mark<false>, blocks, 256, 0, st, b, MeshDev{}, total_tris);
        count_launches(1);
    }
    const uint32_t blocks = std::min<uint32_t>((total_ctas + kRegionChunk - 1) / kRegionChunk, (uint32_t)num_sms * 16);
    if (b.one) launch_chained(k_region_prepare<true>, blocks, 256, 0, st, b, *b.one, total_ctas);
    else launch_chained(k_region_prepare<false>, blocks, 256, 0, st, b, MeshDev{}, total_ctas);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_voxelize(const BatchDev &b, int64_t total, bool strict, const VoxTuning &tune, uint4 *big,
                            uint32_t big_cap, uint32_t *counters, int num_sms, cudaStream_t st) {
    // counters[0] = queue entries, counters[1] = queue cursor
    if (total > 0) {
        const int64_t want = (total + 255) / 256;
        const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)num_sms * 16));
        const bool inplace = big == nullptr || big_cap == 0;
        const uint32_t cols = std::max<uint32_t>(1, tune.warp_max / 16);
        const MeshDev one = b.one ? *b.one : MeshDev{};
#define SVO_VOX(S_, I_, O_) \
    launch_chained(k_voxelize<S_, I_, O_>, blocks, 256, 0, st, b, one, total, tune.serial_max, cols, big, big_cap, \
                   counters)
#define SVO_COLS(S_, O_) \
    launch_chained(k_voxelize_columns<S_, O_>, num_sms * 2, 256, 0, st, b, one, big, counters, big_cap, counters + 1)
        if (inplace) {  // the allocation-free entry point: one mesh
            if (!b.one) return cudaErrorInvalidValue;
            if (strict) SVO_VOX(true, true, true); else SVO_VOX(false, true, true);
        } else if (strict) {
            if (b.one) SVO_VOX(true, false, true); else SVO_VOX(true, false, false);
        } else {
            if (b.one) SVO_VOX(false, false, true); else SVO_VOX(false, false, false);
        }
        count_launches(1);
        if (!inplace) {
            if (strict) {
                if (b.one) SVO_COLS(true, true); else SVO_COLS(true, false);
            } else {
                if (b.one) SVO_COLS(false, true); else SVO_COLS(false, false);
            }
            count_launches(1);
        }
#undef SVO_COLS
#undef SVO_VOX
    }
    return cudaGetLastError();
}

}  // namespace svo
