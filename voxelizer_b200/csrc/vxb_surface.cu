// Surface voxelization kernels (FP32): classifyTriangles / analyzeBoundingBox
// / encodeTriangleType (src/voxelizer.cu:3040-3221) and the 1D / 2D / 3D
// processing kernels (3306-3955) with processVoxel (2946-2989).
//
// One kernel classifies every triangle (class, dominant axis, voxel box clamped
// to the grid, work units), gives the triangles with work consecutive
// positions, ordered by class and axis inside a block, and writes one set-up
// record per position together with the prefix of its work units.  The work
// list runs over that prefix: rows of up to 32 columns of the dominant
// projection (of a 1D line, up to 32 of its voxels).  Warps find the triangle of each of their
// 32 rows with one coalesced load of 32 offsets, so the work kernel has no
// block-wide barrier.
//
// The reference runs the surface kernels once per material subspace on
// boxes clamped to it.  Subspaces tile the grid, so the columns of the
// grid-clamped box are the union of the subspaces' columns; along the depth
// axis a column still visits each subspace's slice separately, because the
// single-voxel shortcut (no further tests when the clamped depth range is
// one voxel) depends on the slice.
//
// Hits set the voxel's bit in the surface grid and append (bit position,
// material key) to a hit list.  Once all surface bits exist, every surface
// voxel gets a rank (prefix popcount over the surface grid), and the list is
// max-merged into a compact key array indexed by rank; the emit kernels read
// materials from there.  The key orders triangles by class, then material
// (NodeT in vxb_device.cuh), so the merged key names the winning material.
// If the list overflows, a second traversal (mode 1) merges every hit
// directly.  The same second traversal is the whole merge where no list is
// kept (64-bit PartialNode keys, or when the launch-shape tuner measured it
// faster): the first traversal then sets surface bits only (mode 2).

#include "vxb_common.cuh"
#include "vxb_device.cuh"
#include "vxb_kernels.cuh"

#include <algorithm>

namespace vxb {

using namespace detail;

namespace {

constexpr int kBlock = 256;
constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kNone = 0xFFu;

__device__ __forceinline__ void loadTriF(const float* __restrict__ V, const uint32_t* __restrict__ I, uint32_t t,
                                         F3* v) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        uint32_t a = __ldg(I + 3 * t + k);
        v[k] = F3{__ldg(V + 3 * a), __ldg(V + 3 * a + 1), __ldg(V + 3 * a + 2)};
    }
}

__device__ __forceinline__ F3 subF(F3 a, F3 b) { return F3{__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)}; }

template <int M> __device__ __forceinline__ F3 crossF(F3 a, F3 b) {
    return F3{diff2f<M>(a.y, b.z, a.z, b.y), diff2f<M>(a.z, b.x, a.x, b.z), diff2f<M>(a.x, b.y, a.y, b.x)};
}

struct IBox { int lo[3], hi[3]; };

// The division where divByF does not apply.
__device__ __noinline__ float divideF(float x, float d) { return __fdiv_rn(x, d); }

// getTriangleBounds (float3, src/voxelizer.cu:2366-2390) and
// getVoxelBoundsHalf (2471-2492).
__device__ __forceinline__ IBox voxBoundsHalf(const F3* v, const PassGeom& g) {
    F3 mn = v[0], mx = v[0];
#pragma unroll
    for (int i = 1; i < 3; ++i) {
        if (v[i].x < mn.x) mn.x = v[i].x;
        if (v[i].y < mn.y) mn.y = v[i].y;
        if (v[i].z < mn.z) mn.z = v[i].z;
        if (v[i].x > mx.x) mx.x = v[i].x;
        if (v[i].y > mx.y) mx.y = v[i].y;
        if (v[i].z > mx.z) mx.z = v[i].z;
    }
    const float d = g.df, rd = g.rdf;
    const float a[6] = {__fsub_rn(mn.x, g.mnf[0]), __fsub_rn(mn.y, g.mnf[1]), __fsub_rn(mn.z, g.mnf[2]),
                        __fsub_rn(mx.x, g.mnf[0]), __fsub_rn(mx.y, g.mnf[1]), __fsub_rn(mx.z, g.mnf[2])};
    bool ok = rd != 0.0f;
#pragma unroll
    for (int i = 0; i < 6; ++i) ok &= divExactF(a[i]);
    float q[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) q[i] = divByF(a[i], d, rd);
    if (!ok) {
#pragma unroll
        for (int i = 0; i < 6; ++i) q[i] = divideF(a[i], d);
    }
    IBox b;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        b.lo[i] = __float2int_ru(__fsub_rn(q[i], 0.5f));
        b.hi[i] = __float2int_rd(__fadd_rn(q[3 + i], 0.5f));
    }
    return b;
}

// Class (bits 30-31: 0 degenerate, 1 / 2 / 3 for 1D / 2D / 3D boxes) and
// axis (bits 28-29: the line's axis for 1D, the flat axis for 2D, the
// dominant normal axis for 3D) of a triangle, from its unclamped box.
__device__ __forceinline__ uint32_t classifyTri(const F3* v, const IBox& b) {
    const F3 n = crossF<site::CRF_CLS>(subF(v[0], v[2]), subF(v[1], v[0]));
    if (!(n.x != 0.0f || n.y != 0.0f || n.z != 0.0f)) return 0u;
    const int dx = b.hi[0] - b.lo[0], dy = b.hi[1] - b.lo[1], dz = b.hi[2] - b.lo[2];
    uint32_t bb, axis;
    if (dx == 0) {
        if (dy == 0) { bb = 1; axis = dz == 0 ? 0 : 2; }
        else if (dz == 0) { bb = 1; axis = 1; }
        else { bb = 2; axis = 0; }
    } else if (dy == 0) {
        if (dz == 0) { bb = 1; axis = 0; }
        else { bb = 2; axis = 1; }
    } else if (dz == 0) { bb = 2; axis = 2; }
    else {
        bb = 3;
        const float ax = fabsf(n.x), ay = fabsf(n.y), az = fabsf(n.z);
        if (ax > ay && ax > az) axis = 0;
        else if (ay > ax && ay > az) axis = 1;
        else axis = 2;
    }
    return (axis << 28) | (bb << 30);
}

// The box clamped to the grid, i.e. to the union of the material subspaces
// (adjustVoxelRange, src/voxelizer.cu:3963-3993, over all of them).
__device__ __forceinline__ IBox gridClamp(IBox b, const PassGeom& g) {
    const int hi[3] = {(int)g.X - 1, (int)g.resY - 1, (int)g.resZ - 1};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        b.lo[a] = max(b.lo[a], 0);
        b.hi[a] = min(b.hi[a], hi[a]);
    }
    return b;
}

// Columns of the dominant projection (voxels along the axis for 1D boxes); 0
// for an empty (fully outside) box.  *rows: work units, rows of up to 32
// columns (32 voxels of a 1D line).
__device__ __forceinline__ uint32_t surfColumns(const IBox& b, uint32_t code, uint32_t* rows) {
    *rows = 0u;
    if (b.lo[0] > b.hi[0] || b.lo[1] > b.hi[1] || b.lo[2] > b.hi[2]) return 0u;
    const uint32_t bb = code >> 30, axis = (code >> 28) & 3u;
    const uint32_t ex = (uint32_t)(b.hi[0] - b.lo[0] + 1), ey = (uint32_t)(b.hi[1] - b.lo[1] + 1),
                   ez = (uint32_t)(b.hi[2] - b.lo[2] + 1);
    if (bb == 0) return 0u;
    if (bb == 1) {
        const uint32_t length = axis == 0 ? ex : axis == 1 ? ey : ez;
        *rows = (length + 31u) / 32u;
        return length;
    }
    const uint32_t in = axis == 0 ? ey : ex, out = axis == 2 ? ey : ez;
    *rows = (in + 31u) / 32u * out;
    return in * out;
}

// The unit and mesh triangle of work triangle wt.
__device__ __forceinline__ uint32_t workUnit(const Batch& b, uint32_t wt, uint32_t* t) {
    const uint32_t u = unitOf(b.workBase, b.nUnits, wt);
    *t = wt - __ldg(b.workBase + u);
    return u;
}

struct Overlap { float nx[3], ny[3], de[3]; };

// Columns are indexed along the inner and the outer axis of the dominant
// projection and run along the depth axis:
//   axis 0: inner y, outer z, depth x
//   axis 1: inner x, outer z, depth y
//   axis 2: inner x, outer y, depth z
// First record (80 bytes) of a triangle with work: what every column needs.
struct __align__(16) SurfRec {
    // Edge functions of the dominant projection (not for 1D boxes), as the
    // coefficients whose products are evaluated unfused and fused.
    float cu[3], cf[3], de[3];
    int lo[2];          // voxel box clamped to the grid: first inner, outer
    uint32_t ext;       // inner extent
    uint32_t segs;      // work units of a row: its 32-column segments
    uint32_t code;      // class << 30 | axis << 28 | material
    uint32_t unit;      // unit of the batch
    int dlo, hi;        // first depth; last depth (1D, 3D) or outer (2D)
    float m[3];         // minimum corner along inner, outer, depth
};
// Second record (112 bytes) of 3D boxes, in (inner, outer, depth) order.
struct __align__(16) SurfDepth {
    float v0[3], n[3];  // first vertex, normal
    float rn;           // 1 / the normal's depth component (0: divide)
    float pad;
    // The other two projections in the order of their tests: coefficients of
    // the column's coordinate and of the depth.
    float cc1[3], cd1[3], de1[3], cc2[3], cd2[3], de2[3];
    float pad2[2];
};
static_assert(sizeof(SurfRec) == kSurfRecBytes, "record size");
static_assert(sizeof(SurfDepth) == kSurfDepthBytes, "record size");

// The sites that the common forms below rely on: the dominant projection of
// 3D boxes evaluates all edges alike, 2D boxes fuse the outer coordinate, the
// depth loop tests fuse the depth coordinate in the first projection and the
// constant one in the second.
static_assert(site::OT_3D_YZ == 42 && site::OT_3D_ZX == 42 && site::OT_3D_XY == 42, "dominant projection form");
static_assert(site::OT_2D_YZ == 42 && site::OT_2D_ZX == 21 && site::OT_2D_XY == 42, "2D form");
static_assert(site::OT_2DP_YZ == 0 && site::OT_2DP_ZX == 0 && site::OT_2DP_XY == 0, "2D prolog form");
static_assert(site::OT_3DX_ZX == 42 && site::OT_3DY_XY == 42 && site::OT_3DZ_YZ == 42, "first depth test form");
static_assert(site::OT_3DX_XY == 21 && site::OT_3DY_YZ == 21 && site::OT_3DZ_ZX == 21, "second depth test form");
static_assert(site::OT_3DYP_XY == 21 && site::OT_3DZP_YZ == 21, "first depth test prolog form");
static_assert(site::OT_3DXP_XY == 21 && site::OT_3DYP_YZ == 21 && site::OT_3DZP_ZX == 21,
              "second depth test prolog form");
static_assert(site::PC_2D == 1 && site::PC_3D == 1 && site::PC_3DL == 1, "voxel corner form");
static_assert(site::DT_3DY == 3 && site::DT_3DZ == 5, "depth range form");

// Per-edge contraction modes: the three edge expressions of a test are
// separate (unrolled) expressions in the reference, so a site's mode packs
// two bits per edge.
__device__ __forceinline__ float sum2fm(int m, float a, float b, float c, float d) {
    return m == 0 ? sum2f<0>(a, b, c, d) : m == 1 ? sum2f<1>(a, b, c, d) : sum2f<2>(a, b, c, d);
}
// setupYZ / ZX / XYOverlapTest (src/voxelizer.cu:2675-2757): edge functions
// over the coordinates (a, b) of the vertices, oriented by the normal's third
// component.
template <int DE> __device__ __forceinline__ Overlap setupOverlap(const float* a, const float* b, float nn, float d) {
    Overlap o;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float pa = a[i], pb = b[i], qa = a[(i + 1) % 3], qb = b[(i + 1) % 3];
        if (nn >= 0.0f) { o.nx[i] = __fsub_rn(pb, qb); o.ny[i] = __fsub_rn(qa, pa); }
        else { o.nx[i] = __fsub_rn(qb, pb); o.ny[i] = __fsub_rn(pa, qa); }
        const float s = sum2fm((DE >> (2 * i)) & 3, o.nx[i], pa, o.ny[i], pb);
        o.de[i] = __fadd_rn(__fadd_rn(-s, fmaxf(0.0f, __fmul_rn(d, o.nx[i]))), fmaxf(0.0f, __fmul_rn(d, o.ny[i])));
    }
    return o;
}

// (x, y, z) turned so that the axis comes first: [0] depth, then the two
// coordinates of the dominant projection in its order ((y, z), (z, x) or
// (x, y)).  The inner axis is [1], but [2] for axis 1; the outer one the other.
template <class T> __device__ __forceinline__ T turned(uint32_t axis, int k, T x, T y, T z) {
    return k == 0 ? (axis == 0 ? x : axis == 1 ? y : z) : k == 1 ? (axis == 0 ? y : axis == 1 ? z : x)
                                                                 : (axis == 0 ? z : axis == 1 ? x : y);
}

// Set-up records of a triangle (the second one for 3D boxes only).
__device__ __forceinline__ void setupRecord(const Unit& U, uint32_t unit, uint32_t t, const F3* v, const IBox& box,
                                            uint32_t code, SurfRec* rec, SurfDepth* depth) {
    const uint32_t bb = code >> 30, axis = (code >> 28) & 3u;
    const float d = U.g.df;
    const int in = 1, out = 2;   // swapped for axis 1
    SurfRec r;
    int lo[3], hi[3];
    float m[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        r.cu[i] = r.cf[i] = r.de[i] = 0.0f;
        lo[i] = turned(axis, i, box.lo[0], box.lo[1], box.lo[2]);
        hi[i] = turned(axis, i, box.hi[0], box.hi[1], box.hi[2]);
        m[i] = turned(axis, i, U.g.mnf[0], U.g.mnf[1], U.g.mnf[2]);
    }
    const bool turn = axis == 1;
    r.lo[0] = turn ? lo[out] : lo[in];
    r.lo[1] = turn ? lo[in] : lo[out];
    r.m[0] = turn ? m[out] : m[in];
    r.m[1] = turn ? m[in] : m[out];
    r.m[2] = m[0];
    r.dlo = lo[0];
    r.hi = bb != 2 ? hi[0] : turn ? hi[in] : hi[out];
    r.ext = (uint32_t)((turn ? hi[out] : hi[in]) - r.lo[0]) + 1u;
    r.segs = (r.ext + 31u) / 32u;
    r.code = code | (U.M ? __ldg(U.M + t) : 0u);
    r.unit = unit;
    if (bb >= 2) {
        static_assert(site::CRF_2D == site::CRF_3D && site::DE_2D_YZ == site::DE_3D_YZ &&
                          site::DE_3D_ZX == site::DE_3D_YZ && site::DE_3D_XY == site::DE_3D_YZ &&
                          site::DE_2D_ZX == site::DE_3D_YZ && site::DE_2D_XY == site::DE_3D_YZ, "one set-up form");
        const F3 nv = crossF<site::CRF_3D>(subF(v[0], v[2]), subF(v[1], v[0]));
        float n[3], p[3][3];   // p[k]: coordinate k of the three vertices
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            n[k] = turned(axis, k, nv.x, nv.y, nv.z);
#pragma unroll
            for (int i = 0; i < 3; ++i) p[k][i] = turned(axis, k, v[i].x, v[i].y, v[i].z);
        }
        const Overlap o = setupOverlap<site::DE_3D_YZ>(p[1], p[2], n[0], d);
        // 2D boxes: products of the inner coordinate unfused, of the outer one
        // fused; 3D boxes: products of the first coordinate unfused.
        const bool swap = bb == 2 && turn;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            r.cu[i] = swap ? o.ny[i] : o.nx[i];
            r.cf[i] = swap ? o.nx[i] : o.ny[i];
            r.de[i] = o.de[i];
        }
        if (bb == 3) {
            // The other two projections, tested in this order: the second
            // coordinate and the depth, the depth and the first coordinate.
            const Overlap f = setupOverlap<site::DE_3D_YZ>(p[2], p[0], n[1], d);
            const Overlap g = setupOverlap<site::DE_3D_YZ>(p[0], p[1], n[2], d);
            SurfDepth s;
            s.v0[0] = turn ? p[out][0] : p[in][0];
            s.v0[1] = turn ? p[in][0] : p[out][0];
            s.v0[2] = p[0][0];
            s.n[0] = turn ? n[out] : n[in];
            s.n[1] = turn ? n[in] : n[out];
            s.n[2] = n[0];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                s.cc1[i] = f.nx[i];
                s.cd1[i] = f.ny[i];
                s.de1[i] = f.de[i];
                s.cd2[i] = g.nx[i];
                s.cc2[i] = g.ny[i];
                s.de2[i] = g.de[i];
            }
            s.rn = divScaleF(n[0]) ? __frcp_rn(n[0]) : 0.0f;
            s.pad = s.pad2[0] = s.pad2[1] = 0.0f;
            *depth = s;
        }
    }
    *rec = r;
}

// Classification, positions and set-up.  A block takes kPrepThreads
// consecutive work triangles, orders those with work by (class, axis), so that
// the warps of the work kernel rarely mix kinds, and reserves their positions
// and their work units with one 64-bit atomic: *cursor counts triangles above
// bit kUnitBits and units below, so that positions and unit offsets of all
// blocks follow the same order.  offsets[pos] is the first unit of pos.
// *total is the number of columns: past 2^32 - 2 of them the cursor may have
// carried and the work kernel does nothing.  classes[0..3): triangles per
// class.
//
// Bounds: the triangle gathers and the records' stores.  In place of a
// classification, a partition by global (class, axis) cursors that set up the
// records and a three-launch scan of the units, 140 us on the room and 455 on
// a batch of 64 meshes (4.2 M triangles), now 70 and 215 us.  Records staged in
// shared memory and stored in order took 20% more.  Atomics on the shared
// counters are about 1 ns each, so blocks add theirs up over their triangles
// (added per 128 triangles: 245 us) and take 32 sets per SM at the most (64: 5
// us more).
constexpr int kPrepThreads = 128;
constexpr uint32_t kUnitBits = 33;

__global__ void __launch_bounds__(kPrepThreads, 8) surfacePrepareKernel(Batch b, uint32_t nWork,
                                                                     unsigned long long* cursor,
                                                                     unsigned long long* total, uint32_t* classes,
                                                                     uint32_t* __restrict__ offsets,
                                                                     uint32_t* __restrict__ triOf,
                                                                     SurfRec* __restrict__ recs,
                                                                     SurfDepth* __restrict__ depth) {
    constexpr int kW = kPrepThreads / 32;
    __shared__ uint32_t cnt[kSurfaceBuckets * kW + 1];      // triangles per bucket and warp, then their prefix
    __shared__ uint32_t sorted[kPrepThreads];               // units in order of position
    __shared__ unsigned long long warpSum[kW], base;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned long long allColumns = 0;   // of the thread's triangles
    uint32_t ofClass = 0;                // the block's triangles of class threadIdx.x + 1
    for (uint64_t b0 = (uint64_t)blockIdx.x * kPrepThreads; b0 < nWork; b0 += (uint64_t)gridDim.x * kPrepThreads) {
        const uint64_t wt = b0 + threadIdx.x;
        uint32_t t = 0, unit = 0, code = 0, u = 0, columns = 0;
        F3 v[3];
        IBox box;
        if (wt < nWork) {
            unit = workUnit(b, (uint32_t)wt, &t);
            const Unit& U = b.units[unit];
            if (U.materials) {
                loadTriF(U.V, U.I, t, v);
                const IBox full = voxBoundsHalf(v, U.g);
                code = classifyTri(v, full);
                box = gridClamp(full, U.g);
                columns = surfColumns(box, code, &u);
            }
        }
        const uint32_t bucket = u ? ((code >> 30) - 1u) * 3u + ((code >> 28) & 3u) : kNone;
        const uint32_t peers = __match_any_sync(kFull, bucket);
        for (uint32_t i = threadIdx.x; i < kSurfaceBuckets * kW; i += kPrepThreads) cnt[i] = 0u;
        __syncthreads();
        if (u && lane == (uint32_t)(__ffs(peers) - 1)) cnt[bucket * kW + warp] = __popc(peers);
        __syncthreads();
        // Exclusive prefix over (bucket, warp), by the first warp; sum at the end.
        if (warp == 0) {
            uint32_t carry = 0;
            for (uint32_t i0 = 0; i0 < kSurfaceBuckets * kW; i0 += 32u) {
                const uint32_t i = i0 + lane, x = i < kSurfaceBuckets * kW ? cnt[i] : 0u;
                uint32_t incl = x;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t q = __shfl_up_sync(kFull, incl, o);
                    if (lane >= (uint32_t)o) incl += q;
                }
                if (i < kSurfaceBuckets * kW) cnt[i] = carry + incl - x;
                carry += __shfl_sync(kFull, incl, 31);
            }
            if (lane == 0) cnt[kSurfaceBuckets * kW] = carry;
        }
        __syncthreads();
        const uint32_t n = cnt[kSurfaceBuckets * kW];
        if (n == 0) continue;   // as for most sets of a slice (a call on 1 M triangles 138 -> 133 us)
        uint32_t at = 0;
        if (u) {
            at = cnt[bucket * kW + warp] + __popc(peers & laneMaskLt());
            sorted[at] = u;
        }
        __syncthreads();
        const unsigned long long x = threadIdx.x < n ? sorted[threadIdx.x] : 0u;
        unsigned long long incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long q = __shfl_up_sync(kFull, incl, o);
            if (lane >= (uint32_t)o) incl += q;
        }
        if (lane == 31) warpSum[warp] = incl;
        __syncthreads();
        unsigned long long before = 0, sum = 0;
#pragma unroll
        for (uint32_t k = 0; k < kW; ++k) {
            if (k < warp) before += warpSum[k];
            sum += warpSum[k];
        }
        if (threadIdx.x == 0 && n) {
            base = atomicAdd(cursor, ((unsigned long long)n << kUnitBits) + sum);
        }
        allColumns += columns;
        if (threadIdx.x < 3) ofClass += cnt[(threadIdx.x + 1u) * 3u * kW] - cnt[threadIdx.x * 3u * kW];
        __syncthreads();
        // Positions past the arrays are only possible after a carry.
        const uint32_t pos0 = (uint32_t)(base >> kUnitBits), room = pos0 < nWork ? min(n, nWork - pos0) : 0u;
        if (threadIdx.x < room) offsets[pos0 + threadIdx.x] = (uint32_t)(base + before + incl - x);
        if (u && at < room) {
            if (triOf) triOf[pos0 + at] = t;
            setupRecord(b.units[unit], unit, t, v, box, code, recs + pos0 + at, depth + pos0 + at);
        }
        __syncthreads();
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) allColumns += __shfl_down_sync(kFull, allColumns, o);
    if (lane == 0 && allColumns) atomicAdd(total, allColumns);
    if (threadIdx.x < 3 && ofClass) atomicAdd(classes + threadIdx.x, ofClass);
}

// getSingleVoxelBoundsComponent, src/voxelizer.cu:2575-2586.
__device__ __forceinline__ float vbComp(int c, float m, float d) {
    return linf<1>(__fsub_rn((float)c, 0.5f), d, m);
}

// Two values per operation, each rounded as by itself: two columns of a row, or
// the two projections of a voxel of the depth range.  It halves the edge
// functions' instructions; the stress FCC mesh, whose rows are long, takes 71
// instead of 76 us (a call 173 -> 171), the room 447 instead of 450.
__device__ __forceinline__ float2 both(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 vbComp2(int c, float m, float d) {
    const float2 x = __fadd2_rn(make_float2((float)c, (float)(c + 1)), both(-0.5f));
    return __ffma2_rn(x, both(d), both(m));
}

// determineDepthRange{X,Y,Z} (src/voxelizer.cu:3994-4119) with
// intersectWithPlane* and boundsCheck, in (inner, outer, depth) coordinates:
// p the column's corner, t0 the first vertex, n the normal.
__device__ __noinline__ void depthDivide(float a, float b, float nd, float m, float d, int& lo, int& hi) {
    a = __fdiv_rn(a, nd);
    b = __fdiv_rn(b, nd);
    if (a > b) { const float t = a; a = b; b = t; }
    lo = __float2int_ru(__fsub_rn(__fdiv_rn(__fsub_rn(a, m), d), 0.5f));
    hi = __float2int_rd(__fadd_rn(__fdiv_rn(__fsub_rn(b, m), d), 0.5f));
}

template <int K>
__device__ __forceinline__ void depthRange(uint32_t axis, float pi, float po, const float4& q0, const float4& q1,
                                           float m, float d, float rd, int& lo, int& hi) {
    // q0: v0 (inner, outer, depth), n inner; q1: n outer, n depth, 1 / n depth.
    const float ni = q0.w, no = q1.x, nd = q1.y, rn = q1.z;
    const float ui = __fsub_rn(q0.x, __fadd_rn(pi, ni > 0.0f ? d : 0.0f)),
                wi = __fsub_rn(q0.x, __fadd_rn(pi, ni > 0.0f ? 0.0f : d));
    const float uo = __fsub_rn(q0.y, __fadd_rn(po, no > 0.0f ? d : 0.0f)),
                wo = __fsub_rn(q0.y, __fadd_rn(po, no > 0.0f ? 0.0f : d));
    float a, b;
    if (axis == 0) {
        // (x, y, z) = (depth, inner, outer)
        a = sum3f<site::DT_3DX[K]>(q0.z, nd, ui, ni, uo, no);
        b = sum3f<site::DT_3DX[K]>(q0.z, nd, wi, ni, wo, no);
    } else if (axis == 1) {
        a = sum3f<site::DT_3DY>(ui, ni, q0.z, nd, uo, no);
        b = sum3f<site::DT_3DY>(wi, ni, q0.z, nd, wo, no);
    } else {
        a = sum3f<site::DT_3DZ>(ui, ni, uo, no, q0.z, nd);
        b = sum3f<site::DT_3DZ>(wi, ni, wo, no, q0.z, nd);
    }
    const float qa = divByF(a, nd, rn), qb = divByF(b, nd, rn);
    const float x = __fsub_rn(fminf(qa, qb), m), y = __fsub_rn(fmaxf(qa, qb), m);
    lo = __float2int_ru(__fsub_rn(divByF(x, d, rd), 0.5f));
    hi = __float2int_rd(__fadd_rn(divByF(y, d, rd), 0.5f));
    // x and y need no lower bound: a quotient below 2^-30 rounds away against
    // the half voxel.
    constexpr float kBig = 1.1529215046068470e18f;   // 2^60
    if (rn == 0.0f || rd == 0.0f || !divExactF(a) || !divExactF(b) || !(fabsf(x) < kBig) || !(fabsf(y) < kBig))
        depthDivide(a, b, nd, m, d, lo, hi);
}

// The loop of the reference over [lo, hi] along one axis runs inside one
// material subspace (adjustVoxelRange, src/voxelizer.cu:3963-3993): clamps
// [lo, hi] to the subspace slice (sl: nSl (lo, hi) pairs) that holds c.
__device__ __forceinline__ void subspaceRange(const uint32_t* sl, uint32_t nSl, int c, int& lo, int& hi) {
    for (uint32_t s = 0; s < nSl; ++s) {
        const int a = (int)__ldg(sl + 2 * s), b = (int)__ldg(sl + 2 * s + 1) - 1;
        if (c >= a && c <= b) {
            lo = max(lo, a);
            hi = min(hi, b);
            return;
        }
    }
}

// Whether iteration `pos` of a loop of n iterations falls in the prolog of a
// loop the reference build unrolled U times (the prolog runs the first
// n mod U iterations; vxb_sites.inc).
template <int U> __device__ __forceinline__ bool inProlog(int pos, int n) { return U > 1 && pos < n % U; }

// Where the hits of the surface pass (processVoxel) go.
struct Sink {
    uint32_t* bits;            // surface arena
    const WordRank* wordRank;  // complete surface words with their ranks (mode 1)
    void* keys;                // compact key array (mode 1)
    uint32_t keysCap;          // keys at ranks past it are dropped
    unsigned long long* positions;   // arena position of each rank (mode 1, wide keys)
    unsigned long long* list;
    uint32_t* listCount;
    uint32_t listCap;
};

// Hits of one warp are staged in shared memory before they go to the global
// hit list, so that the list takes one atomic per flush.
constexpr uint32_t kStageHits = 256;
constexpr int kWorkThreads = 128;

// The rows of a warp's last two chunks, and the warp's queue of columns that
// pass (slot of the row << 5 | column).
struct SurfWarp {
    int4 a[64];     // inner of the first column, outer, position, code
    int4 b[64];     // unit, first and last depth, minimum corner along the depth
    float2 c[64];   // minimum corner along the inner axis, the row's corner along the outer axis
    uint16_t queue[1024 + 32];
};

// The work list: rows of up to 32 columns of the dominant projection.  Warps
// take batches of `chunksPerBatch` consecutive chunks of 32 rows; within a
// batch the owner of each chunk's first row follows from the previous chunk.
// Every listed triangle has at least one row, so a chunk's rows belong to at
// most 32 consecutive positions: lane l loads off[t0 + l] and a bit mask of
// the triangle starts inside the chunk gives every lane its owner.
//
// A lane takes one row and tests its columns against the dominant projection
// (all of process2DTriangles, src/voxelizer.cu:3418-3596, and the first test
// of process3DTriangles, 3603-3955), about ten operations a column.  The
// columns that pass, about half, are queued and worked 32 at a time, a lane each: a
// depth range from the plane, then per material subspace slice of the depth
// axis either the single voxel or the other two projections per voxel.  The
// products of the column's coordinate do not change along the depth, so a
// depth voxel costs six fused edge values.  The depth loop only marks hits
// (32 voxels at a time in a mask); they are recorded afterwards, one per lane
// and step.  Loops that the reference build unrolled evaluate their first
// iterations in their own forms (instantiated per node type K as there).
//
// Mode 0: set the voxel's bit and append (bit position << 24 | key) to the
// hit list; mode 1: merge the key at the voxel's rank (surface bits are
// complete); mode 2: set the bit only.  PartialNodes have 64-bit keys.
//
// Bounds: issue (about two thirds of the slots) and the latency of the record
// and edge gathers.  With a column per lane, 303 of 570 instructions of a
// chunk of 32 columns found the owner and loaded its record, and half of the
// lanes idled through the rest.  Alone on a B200, a column per lane with hits
// recorded inside the depth loop / marked first / by rows: room (22.3 M
// columns, 19.2 M hits) 582 / 527 / 450 us, stress FCC mesh (slivers) 193 /
// 163 / 76 us, duct 120 / 103 / 95 us; with two columns per operation 447, 71
// and 93 us.  A list of 5,120 triangles takes 18 instead of 14 us.  The stage
// must hold several steps' hits: with 128 or 64 entries instead of 256 the
// waits for the list's counter make it 676 and 967 us; prefetching the next
// chunk's records and larger batches gave nothing (508-540 us with 8 chunks a
// batch).
template <int K, int MODE>
__global__ void __launch_bounds__(kWorkThreads, 8) surfaceWorkKernel(Sink sink, Batch b, const SurfRec* __restrict__ recs,
                                                               const SurfDepth* __restrict__ depth,
                                                               const uint32_t* __restrict__ triOf,
                                                               const uint32_t* __restrict__ off,
                                                               const unsigned long long* __restrict__ cursor,
                                                               const unsigned long long* __restrict__ totalPtr,
                                                               uint32_t chunksPerBatch, uint32_t* queue) {
    constexpr bool kWide = K == kPartial;
    constexpr int kXProlog = site::OT_3DXP_ZX[K];
    static_assert(kXProlog == site::OT_3DX_ZX || kXProlog == 21, "x-dominant prolog form");
    __shared__ unsigned long long stage[kWorkThreads / 32][MODE == 0 ? kStageHits : 1];
    __shared__ SurfWarp shared[kWorkThreads / 32];
    if (*totalPtr >= 0xFFFFFFFFull) return;   // refused by the host
    const unsigned long long listed = *cursor;
    const uint32_t n = (uint32_t)(listed >> kUnitBits), total = (uint32_t)listed;
    const uint32_t lane = threadIdx.x & 31u;
    unsigned long long* const hits = stage[threadIdx.x >> 5];
    SurfWarp& sw = shared[threadIdx.x >> 5];
    uint32_t staged = 0;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nWarps = (gridDim.x * blockDim.x) >> 5;
    // A short list goes to the warps that fit the device, in chunks of fewer
    // rows and a chunk each, before a warp takes several.
    uint32_t rows = 32u;   // per chunk, a power of two
    while (rows > 1u && total / rows < 148u * 32u) rows >>= 1;
    const uint32_t chunks = (total + rows - 1u) / rows;
    chunksPerBatch = min(chunksPerBatch, max(chunks / nWarps, 1u));
    const uint32_t batches = (chunks + chunksPerBatch - 1) / chunksPerBatch;
    // Batches in a fixed grid-stride order, or (queue != NULL) taken from a
    // device work queue, one atomic per batch, so that warps that drew cheap
    // batches keep working while others finish expensive ones.
    auto nextBatch = [&](uint32_t cur) {
        if (!queue) return cur + nWarps;
        uint32_t v = 0;
        if (lane == 0) v = atomicAdd(queue, 1u);
        return __shfl_sync(kFull, v, 0);
    };
    auto flush = [&]() {
        __syncwarp();
        uint32_t base = 0;
        if (lane == 0 && staged) base = atomicAdd(sink.listCount, staged);
        base = __shfl_sync(kFull, base, 0);
        for (uint32_t i = lane; i < staged; i += 32u)
            if (base + i < sink.listCap) sink.list[base + i] = hits[i];
        __syncwarp();
        staged = 0;
    };
    uint32_t bt = queue ? nextBatch(0) : warp, c = 0, c1 = 0, t0 = 0;   // batch, its chunks left, first position
    uint32_t half = 0, head = 0, tail = 0;   // row slots to fill next, queue entries
    bool drain = false;
    for (;;) {
        // Full groups of columns first; a partial one only when its row slots
        // are needed or nothing is left.
        if (tail - head < 32u && !(drain && tail != head)) {
            drain = false;
            if (c == c1) {
                if (bt >= batches) {
                    if (tail == head) break;
                    drain = true;
                    continue;
                }
                c = bt * chunksPerBatch;
                c1 = min(c + chunksPerBatch, chunks);
                t0 = warpFindOwner(off, n, c * rows, lane);
                bt = nextBatch(bt);
            }
            // What is left moves to the front of the queue.
            const uint32_t left = tail - head;
            const uint32_t entry = lane < left ? sw.queue[head + lane] : 0u;
            if (__any_sync(kFull, lane < left && (entry >> 10) == half)) {
                drain = true;
                continue;
            }
            __syncwarp();
            if (lane < left) sw.queue[lane] = (uint16_t)entry;
            head = 0;
            const uint32_t base = c * rows;
            const uint32_t ol = t0 + lane < n ? __ldg(off + t0 + lane) : total;
            const uint32_t o32 = t0 + 32u < n ? __ldg(off + t0 + 32u) : total;
            const uint32_t starts =
                __reduce_or_sync(kFull, (t0 + lane < n && lane >= 1u && ol < base + rows) ? 1u << (ol - base) : 0u);
            const uint32_t k = __popc(starts & ((2u << lane) - 1u));
            const uint32_t ok = __shfl_sync(kFull, ol, k);
            const uint32_t k31 = __popc(starts);
            const uint32_t next = __shfl_sync(kFull, ol, (k31 + 1u) & 31u);
            const uint32_t nextOff = k31 < 31u ? next : o32;
            const uint32_t item = base + lane, pos = t0 + k;
            t0 += k31 + (nextOff == base + rows ? 1u : 0u);
            ++c;
            // The columns of the row that pass the dominant projection.
            uint32_t pass = 0;
            if (lane < rows && item < total) {
                const uint4* rec = reinterpret_cast<const uint4*>(recs + pos);
                const uint4 r2 = __ldg(rec + 2), r3 = __ldg(rec + 3), r4 = __ldg(rec + 4), r0 = __ldg(rec),
                            r1 = __ldg(rec + 1);
                const uint32_t code = r3.y, ext = r2.w, segs = r3.x, axis = (code >> 28) & 3u, bb = code >> 30;
                int inner = (int)r2.y, outer = (int)r2.z, dlo = (int)r3.w, dhi = (int)r4.x;
                float po = 0.0f;
                if (bb == 1) {
                    // 32 voxels of the line: eight lines of 60,000 take 20 us
                    // (with a lane for all of a line 9.6 ms).
                    dlo += (int)(32u * (item - ok));
                    dhi = min(dhi, dlo + 31);
                    pass = 1u;
                } else {
                    const Unit* U = b.units + r3.z;
                    uint32_t row = item - ok, cols = ext;
                    if (segs > 1u) {
                        const uint32_t u = row;
                        row = u / segs;
                        const uint32_t seg = u - row * segs;
                        inner += (int)(32u * seg);
                        cols = min(ext - 32u * seg, 32u);
                    }
                    outer += (int)row;
                    const float d = U->g.df, mI = __uint_as_float(r4.y);
                    po = vbComp(outer, __uint_as_float(r4.z), d);
                    const float cu[3] = {__uint_as_float(r0.x), __uint_as_float(r0.y), __uint_as_float(r0.z)},
                                de[3] = {__uint_as_float(r1.z), __uint_as_float(r1.w), __uint_as_float(r2.x)};
                    float cf[3] = {__uint_as_float(r0.w), __uint_as_float(r1.x), __uint_as_float(r1.y)};
                    if (bb == 3u && axis == 1u) {
                        // Products of the outer coordinate unfused.
                        float k[3];
#pragma unroll
                        for (int i = 0; i < 3; ++i) k[i] = __fmul_rn(cu[i], po);
                        for (uint32_t c2 = 0; c2 < cols; c2 += 2u) {
                            const float2 pi = vbComp2(inner + (int)c2, mI, d);
                            bool h0 = true, h1 = true;
#pragma unroll
                            for (int i = 0; i < 3; ++i) {
                                const float2 e = __fadd2_rn(__ffma2_rn(both(cf[i]), pi, both(k[i])), both(de[i]));
                                h0 &= e.x >= 0.0f;
                                h1 &= e.y >= 0.0f;
                            }
                            pass |= ((h0 ? 1u : 0u) | (h1 ? 2u : 0u)) << c2;
                        }
                    } else {
                        float pf = po;
                        if (bb == 2) {
                            constexpr int UN = site::UNR_2D[K];
                            if (UN > 1) {
                                const uint32_t oa = axis == 2 ? 1u : 2u;   // outer axis
                                int lo = (int)r2.z, hi = dhi;
                                if (U->sliceN[oa] > 1u)
                                    subspaceRange(b.slices + 2 * (U->sliceBase + U->sliceN[0] + (oa == 2u ? U->sliceN[1] : 0u)),
                                                  U->sliceN[oa], outer, lo, hi);
                                if (inProlog<UN>(outer - lo, hi - lo + 1)) {
                                    // Prolog rows are unfused: the outer
                                    // product rounded, then added (times 1).
#pragma unroll
                                    for (int i = 0; i < 3; ++i) cf[i] = __fmul_rn(cf[i], po);
                                    pf = 1.0f;
                                }
                            }
                        }
                        for (uint32_t c2 = 0; c2 < cols; c2 += 2u) {
                            const float2 pi = vbComp2(inner + (int)c2, mI, d);
                            bool h0 = true, h1 = true;
#pragma unroll
                            for (int i = 0; i < 3; ++i) {
                                const float2 e = __fadd2_rn(
                                    __ffma2_rn(both(cf[i]), both(pf), __fmul2_rn(both(cu[i]), pi)), both(de[i]));
                                h0 &= e.x >= 0.0f;
                                h1 &= e.y >= 0.0f;
                            }
                            pass |= ((h0 ? 1u : 0u) | (h1 ? 2u : 0u)) << c2;
                        }
                    }
                    pass &= kFull >> (32u - cols);
                }
                const uint32_t slot = half * 32u + lane;
                sw.a[slot] = make_int4(inner, outer, (int)pos, (int)code);
                sw.b[slot] = make_int4((int)r3.z, dlo, dhi, (int)r4.w);
                sw.c[slot] = make_float2(__uint_as_float(r4.y), po);
            }
            const uint32_t cnt = __popc(pass);
            uint32_t incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t q = __shfl_up_sync(kFull, incl, o);
                if (lane >= (uint32_t)o) incl += q;
            }
            uint32_t at = left + incl - cnt;
            while (pass) {
                sw.queue[at++] = (uint16_t)((half << 10) | (lane << 5) | (__ffs(pass) - 1));
                pass &= pass - 1u;
            }
            tail = left + __shfl_sync(kFull, incl, 31);
            half ^= 1u;
            __syncwarp();
            continue;
        }
        {
            const uint32_t q0 = head, queued = tail;
            head += min(tail - head, 32u);
            // The lane's column and its depth range; `deep` for 3D boxes, whose
            // range comes from the plane.
            const Unit* U = b.units;
            uint32_t code = 0, nSlices = 0, pos = 0;
            int inner = 0, outer = 0, dlo = 0, dhi = -1, blo = 0, bhi = 0;
            float pi = 0.0f, po = 0.0f, mD = 0.0f, d = 0.0f;
            bool deep = false;
            if (q0 + lane < queued) {
                const uint32_t e = sw.queue[q0 + lane], src = e >> 5;
                const int4 ra = sw.a[src], rb = sw.b[src];
                const float2 rc = sw.c[src];
                code = (uint32_t)ra.w;
                pos = (uint32_t)ra.z;
                U = b.units + rb.x;
                inner = ra.x + (int)(e & 31u);
                outer = ra.y;
                dlo = blo = rb.y;
                bhi = rb.z;
                mD = __int_as_float(rb.w);
                const uint32_t bb = code >> 30, axis = (code >> 28) & 3u;
                dhi = bb == 1u ? bhi : dlo;
                if (bb == 3u) {
                    d = U->g.df;
                    pi = vbComp(inner, rc.x, d);
                    po = rc.y;
                    const float4* s = reinterpret_cast<const float4*>(depth + pos);
                    deep = true;
                    nSlices = U->sliceN[axis];
                    depthRange<K>(axis, pi, po, __ldg(s), __ldg(s + 1), mD, d, U->g.rdf, dlo, dhi);
                }
            }
            const uint32_t axis = (code >> 28) & 3u;
            // The hits among voxels a + w0 .. a + w0 + 31 of a range of cnt.
            auto test = [&](int a, uint32_t cnt, uint32_t w0) {
                if (w0 >= cnt) return 0u;
                const uint32_t last = min(cnt - w0, 32u);
                if (!deep || cnt == 1u) return kFull >> (32u - last);
                float e[20];   // cc1 cd1 de1 cc2 cd2 de2
                const float4* f = reinterpret_cast<const float4*>(depth + pos) + 2;
#pragma unroll
                for (int i = 0; i < 5; ++i) {
                    const float4 q = __ldg(f + i);
                    e[4 * i] = q.x; e[4 * i + 1] = q.y; e[4 * i + 2] = q.z; e[4 * i + 3] = q.w;
                }
                const float p1 = axis == 1 ? pi : po, p2 = axis == 1 ? po : pi;
                float k1[3], k2[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    k1[i] = __fmul_rn(e[i], p1);
                    k2[i] = __fmul_rn(e[9 + i], p2);
                }
                uint32_t m = 0u;
                for (uint32_t v = 0; v < last; ++v) {
                    const float pd = vbComp(a + (int)(w0 + v), mD, d);
                    bool hit = true;
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        // Both projections at once.
                        const float2 q = __fadd2_rn(__ffma2_rn(make_float2(e[3 + i], e[12 + i]), both(pd),
                                                               make_float2(k1[i], k2[i])),
                                                    make_float2(e[6 + i], e[15 + i]));
                        hit &= q.x >= 0.0f;
                        hit &= q.y >= 0.0f;
                    }
                    m |= hit ? 1u << v : 0u;
                }
                constexpr int UL = site::UNR_3DL[K];
                static_assert(UL == 0 || UL == 2, "at most one prolog iteration");
                // The prolog iteration in its own form of the first test (the
                // x-dominant one differs by node type).
                if (UL == 2 && w0 == 0u && (cnt & 1u) && (kXProlog == 21 || axis != 0u)) {
                    const float pd = vbComp(a, mD, d);
                    bool hit = true;
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        hit &= __fadd_rn(__fmaf_rn(e[i], p1, __fmul_rn(e[3 + i], pd)), e[6 + i]) >= 0.0f;
                        hit &= __fadd_rn(__fmaf_rn(e[12 + i], pd, k2[i]), e[15 + i]) >= 0.0f;
                    }
                    m = (m & ~1u) | (hit ? 1u : 0u);
                }
                return m;
            };
            // Records the hits m of voxels first + 0 .. 31 along the depth
            // (whole warp).
            auto record = [&](uint32_t m, int first) {
                uint32_t live = __ballot_sync(kFull, m != 0u);
                if (!live) return;
                // Bit position in the unit of the voxel at `first` and its
                // step along the depth.  The allocation holds a voxel one
                // column further along x and padY / padZ rows further along
                // y / z.
                uint32_t at = 0, step = 0;
                uint32_t* bits = sink.bits;
                unsigned long long entry = 0;
                uint64_t wordBase = 0;
                if (m) {
                    const uint32_t X = U->g.X, AY = U->g.AY, pY = U->g.padY, pZ = U->g.padZ;
                    wordBase = U->wordBase;
                    bits += wordBase;
                    entry = (wordBase << 29) | ((code >> 30) << 8) | (code & 255u);
                    const uint32_t zr = axis == 2 ? pZ : (uint32_t)outer + pZ;
                    const uint32_t yr = pY + (axis == 0 ? (uint32_t)inner : axis == 2 ? (uint32_t)outer : 0u);
                    step = axis == 0 ? 1u : axis == 1 ? X : X * AY;
                    at = (zr * AY + yr) * X + (axis == 0 ? 1u : (uint32_t)inner + 1u) + (uint32_t)first * step;
                }
                do {
                    if (m) {
                        const uint32_t v = __ffs(m) - 1;
                        m &= m - 1u;
                        const uint32_t p = at + v * step, bit = p & 31u;
                        if (MODE != 1) {
                            atomicOr(bits + (p >> 5), 0x80000000u >> bit);
                            if (MODE == 0)
                                hits[staged + __popc(live & laneMaskLt())] = entry + ((unsigned long long)p << 24);
                        } else {
                            const uint64_t w = wordBase + (p >> 5);
                            const WordRank wr = sink.wordRank[w];
                            const uint32_t r = wr.rank + (bit ? __popc(wr.bits >> (32u - bit)) : 0u);
                            if (r < sink.keysCap) {
                                const uint32_t cls = code >> 30, mat = code & 255u;
                                if (kWide) {
                                    const unsigned long long key = ((unsigned long long)cls << 40) |
                                                                   ((unsigned long long)mat << 32) | __ldg(triOf + pos);
                                    atomicMax(reinterpret_cast<unsigned long long*>(sink.keys) + r, key);
                                    sink.positions[r] = w * 32u + bit;   // every hit of a voxel stores the same
                                } else {
                                    atomicMax(reinterpret_cast<uint32_t*>(sink.keys) + r, (cls << 8) | mat);
                                }
                            }
                        }
                    }
                    if (MODE == 0) {
                        staged += __popc(live);
                        if (staged > kStageHits - 32u) flush();
                    }
                    live = __ballot_sync(kFull, m != 0u);
                } while (live);
            };
            // The range clamped to the box, one piece per material subspace
            // slice (most ranges lie in one).
            int a = dlo, z = dhi;
            if (deep) {
                a = max(dlo, blo);
                z = min(dhi, bhi);
            }
            do {
                int end = z;
                if (nSlices > 1u && a <= z) {
                    const uint32_t* sl = b.slices + 2 * (U->sliceBase + (axis >= 1u ? U->sliceN[0] : 0u) +
                                                         (axis == 2u ? U->sliceN[1] : 0u)) + 1;
                    uint32_t e = __ldg(sl);
                    while ((uint32_t)a >= e) {
                        sl += 2;
                        e = __ldg(sl);
                    }
                    end = min(z, (int)e - 1);
                }
                const uint32_t cnt = end >= a ? (uint32_t)(end - a) + 1u : 0u;
                uint32_t w0 = 0;
                do {
                    record(test(a, cnt, w0), a + (int)w0);
                    w0 += 32u;
                } while (__any_sync(kFull, w0 < cnt));
                a = end + 1;
            } while (__any_sync(kFull, a <= z));
        }
    }
    if (MODE == 0) flush();
}

// Exclusive popcount prefix over the surface words (ranks of surface voxels)
// in two launches.  The first sums the tiles, and the block that finishes last
// (a counter, nobody waits) turns the sums into their prefix; the second
// writes the ranks (tile offset plus the block's exclusive scan) and zeroes the
// tile's keys.  The words were just written by the surface pass and are read
// from L2 where they stay.  Ranks are only read where there are surface nodes,
// so sectors of four words without any are not written.
//
// Bounds: DRAM.  Sums, ranks and zeroed keys took four launches:
// room (13.5 M words) 64 us, now 60; duct (8.7 M) 43, now 24; batch of 64
// meshes (21 M) 90, now 59; 44,000 words 13, now 8.  With every word's rank
// written by tiles of four steps the room's second launch takes 58 instead of
// 46 us.
constexpr int kRankItems = 8;
constexpr uint32_t kRankStep = kBlock * kRankItems;   // words of a step; a tile has S steps

// Exclusive scan of v over the block, its total in *sum.
__device__ __forceinline__ uint32_t blockScan(uint32_t v, uint32_t* warpSums, uint32_t* sum) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    if (lane == 31) warpSums[warp] = incl;
    __syncthreads();
    uint32_t before = 0, all = 0;
#pragma unroll
    for (uint32_t k = 0; k < kBlock / 32; ++k) {
        if (k < warp) before += warpSums[k];
        all += warpSums[k];
    }
    __syncthreads();
    *sum = all;
    return before + incl - v;
}

__device__ __forceinline__ void rankLoad(const uint32_t* __restrict__ words, uint64_t n, uint64_t base,
                                         uint32_t x[kRankItems]) {
    if (base + kRankItems <= n) {   // 32-byte aligned: kRankItems words per thread
        const uint4 a = __ldg(reinterpret_cast<const uint4*>(words + base));
        const uint4 b = __ldg(reinterpret_cast<const uint4*>(words + base) + 1);
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
        x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < kRankItems; ++i) x[i] = base + i < n ? __ldg(words + base + i) : 0u;
    }
}

// done: zero on entry, the number of blocks that have written their sums.
// stepSums[step]: the surface nodes of the tile's steps before it.
template <int S>
__global__ void __launch_bounds__(kBlock) rankSumKernel(const uint32_t* __restrict__ words, uint64_t n,
                                                        uint32_t* tileSums, uint32_t* __restrict__ stepSums,
                                                        uint32_t* done, uint32_t* total) {
    __shared__ uint32_t warpSums[kBlock / 32], steps[S][kBlock / 32];
    __shared__ bool last;
    uint32_t x[S][kRankItems], all;
#pragma unroll
    for (int k = 0; k < S; ++k)
        rankLoad(words, n, ((uint64_t)blockIdx.x * S + k) * kRankStep + (uint64_t)threadIdx.x * kRankItems, x[k]);
#pragma unroll
    for (int k = 0; k < S; ++k) {
        uint32_t sum = 0;
#pragma unroll
        for (int i = 0; i < kRankItems; ++i) sum += (uint32_t)__popc(x[k][i]);
        sum = __reduce_add_sync(kFull, sum);
        if ((threadIdx.x & 31u) == 0) steps[k][threadIdx.x >> 5] = sum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t sum = 0;
        for (int k = 0; k < S; ++k) {
            stepSums[(uint64_t)blockIdx.x * S + k] = sum;
            for (int w = 0; w < kBlock / 32; ++w) sum += steps[k][w];
        }
        tileSums[blockIdx.x] = sum;
        __threadfence();
        last = atomicAdd(done, 1u) + 1u == gridDim.x;
    }
    __syncthreads();
    if (!last) return;
    uint32_t carry = 0;
    for (uint32_t start = 0; start < gridDim.x; start += kRankStep) {
        const uint32_t i0 = start + threadIdx.x * kRankItems;
        uint32_t v[kRankItems], s = 0;
#pragma unroll
        for (int i = 0; i < kRankItems; ++i) {
            v[i] = i0 + i < gridDim.x ? __ldcg(tileSums + i0 + i) : 0u;
            s += v[i];
        }
        uint32_t ex = carry + blockScan(s, warpSums, &all);
#pragma unroll
        for (int i = 0; i < kRankItems; ++i) {
            if (i0 + i < gridDim.x) tileSums[i0 + i] = ex;
            ex += v[i];
        }
        carry += all;
    }
    if (threadIdx.x == 0) *total = carry;
}

template <bool kWide>
__global__ void __launch_bounds__(kBlock) rankWriteKernel(const uint32_t* __restrict__ words, uint64_t n,
                                                          WordRank* __restrict__ ranks,
                                                          const uint32_t* __restrict__ tileSums,
                                                          const uint32_t* __restrict__ stepSums, uint32_t stepsPerTile,
                                                          void* keys, uint32_t keysCap) {
    __shared__ uint32_t warpSums[kBlock / 32];
    const uint64_t base = (uint64_t)blockIdx.x * kRankStep + (uint64_t)threadIdx.x * kRankItems;
    uint32_t x[kRankItems], sum = 0, all;
    rankLoad(words, n, base, x);
#pragma unroll
    for (int i = 0; i < kRankItems; ++i) sum += (uint32_t)__popc(x[i]);
    const uint32_t first = __ldg(tileSums + blockIdx.x / stepsPerTile) + __ldg(stepSums + blockIdx.x);
    uint32_t ex = first + blockScan(sum, warpSums, &all);
#pragma unroll
    for (int h = 0; h < kRankItems; h += 4) {
        uint32_t r[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            r[i] = ex;
            ex += (uint32_t)__popc(x[h + i]);
        }
        if (ex == r[0]) continue;
        if (base + h + 4 <= n) {
            uint4* out = reinterpret_cast<uint4*>(ranks + base + h);
            out[0] = make_uint4(x[h], r[0], x[h + 1], r[1]);
            out[1] = make_uint4(x[h + 2], r[2], x[h + 3], r[3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (base + h + i < n) ranks[base + h + i] = WordRank{x[h + i], r[i]};
        }
    }
    const uint64_t end = min((uint64_t)first + all, (uint64_t)keysCap);
    for (uint64_t i = (uint64_t)first + threadIdx.x; i < end; i += kBlock) {
        if (kWide) reinterpret_cast<unsigned long long*>(keys)[i] = 0ull;
        else reinterpret_cast<uint32_t*>(keys)[i] = 0u;
    }
}

__global__ void zeroKeysKernel(void* keys, const uint32_t* __restrict__ countPtr, uint32_t cap, int wide) {
    const uint32_t n = min(*countPtr, cap);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (wide) reinterpret_cast<unsigned long long*>(keys)[i] = 0ull;
        else reinterpret_cast<uint32_t*>(keys)[i] = 0u;
    }
}

// Max-merges the hit list into the rank-indexed key array.  Each thread
// takes two pairs of consecutive entries (16-byte loads) per iteration, so
// the scattered word / rank loads of four entries overlap; one 8-byte load
// gives an entry's surface word and rank.
__global__ void mergeKeysKernel(const unsigned long long* __restrict__ list, const uint32_t* __restrict__ countPtr,
                                uint32_t cap, const WordRank* __restrict__ ranks, uint32_t* keys, uint32_t keysCap) {
    constexpr int U = 2;   // entry pairs per thread and iteration
    const uint32_t n = min(*countPtr, cap);
    const uint32_t pairs = (n + 1) / 2;
    const uint32_t stride = gridDim.x * blockDim.x;
    const ulonglong2* list2 = reinterpret_cast<const ulonglong2*>(list);
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < pairs; i0 += U * stride) {
        unsigned long long e[2 * U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t i = i0 + u * stride;
            ulonglong2 q = make_ulonglong2(~0ull, ~0ull);
            if (i < pairs) q = list2[i];
            e[2 * u] = q.x;
            e[2 * u + 1] = 2 * i + 1 < n ? q.y : ~0ull;
        }
        WordRank wr[2 * U];
#pragma unroll
        for (int u = 0; u < 2 * U; ++u)
            if (e[u] != ~0ull) wr[u] = ranks[(e[u] >> 24) >> 5];
#pragma unroll
        for (int u = 0; u < 2 * U; ++u) {
            if (e[u] == ~0ull) continue;
            const uint32_t b = (uint32_t)((e[u] >> 24) & 31u);
            const uint32_t r = wr[u].rank + (b ? __popc(wr[u].bits >> (32 - b)) : 0u);
            if (r < keysCap) atomicMax(keys + r, (uint32_t)(e[u] & 0xFFFFFFull));
        }
    }
}

}  // namespace

void launch_surface_prepare(const Batch& b, uint32_t nWork, unsigned long long* cursor, unsigned long long* total,
                            uint32_t* classes, uint32_t* offsets, uint32_t* triOf, void* recs, void* depth,
                            cudaStream_t s, uint32_t* launches) {
    surfacePrepareKernel<<<gridFor(nWork, kPrepThreads, 148u * 32u), kPrepThreads, 0, s>>>(
        b, nWork, cursor, total, classes, offsets, triOf, static_cast<SurfRec*>(recs), static_cast<SurfDepth*>(depth));
    *launches += 1;
}

template <int K>
static void launchSurfaceWorkKind(int mode, uint32_t grid, const Sink& sink, const Batch& b, const SurfRec* R,
                                  const SurfDepth* D, const uint32_t* triOf, const uint32_t* offsets,
                                  const unsigned long long* cursor, const unsigned long long* total, uint32_t batch,
                                  uint32_t* queue, cudaStream_t s) {
    if (mode == 0)
        surfaceWorkKernel<K, 0><<<grid, kWorkThreads, 0, s>>>(sink, b, R, D, triOf, offsets, cursor, total, batch, queue);
    else if (mode == 1)
        surfaceWorkKernel<K, 1><<<grid, kWorkThreads, 0, s>>>(sink, b, R, D, triOf, offsets, cursor, total, batch, queue);
    else surfaceWorkKernel<K, 2><<<grid, kWorkThreads, 0, s>>>(sink, b, R, D, triOf, offsets, cursor, total, batch, queue);
}

void launch_surface_work(int kind, int mode, const Batch& b, const void* recs, const void* depth, const uint32_t* triOf,
                         const uint32_t* offsets, const unsigned long long* cursor, const unsigned long long* total,
                         uint32_t* surf, const WordRank* ranks, void* keys, uint32_t keysCap,
                         unsigned long long* positions, unsigned long long* list, uint32_t* listCount,
                         uint32_t listCap, uint32_t blocksPerSm, uint32_t batch, uint32_t* queue, cudaStream_t s,
                         uint32_t* launches) {
    if (queue) cudaMemsetAsync(queue, 0, sizeof(uint32_t), s);
    Sink sink;
    sink.bits = surf;
    sink.wordRank = ranks;
    sink.keys = keys;
    sink.keysCap = keysCap;
    sink.positions = positions;
    sink.list = list;
    sink.listCount = listCount;
    sink.listCap = listCap;
    const uint32_t grid = 148u * blocksPerSm * (256u / kWorkThreads);   // shapes count blocks of 256 threads
    const SurfRec* R = static_cast<const SurfRec*>(recs);
    const SurfDepth* D = static_cast<const SurfDepth*>(depth);
    auto launch = kind == kShort ? launchSurfaceWorkKind<kShort>
                : kind == kLong ? launchSurfaceWorkKind<kLong>
                : kind == kPartial ? launchSurfaceWorkKind<kPartial>
                : kind == kShortFcc ? launchSurfaceWorkKind<kShortFcc> : launchSurfaceWorkKind<kLongFcc>;
    // The shapes count chunks of 32 columns; four of them make about one of 32
    // rows.
    launch(mode, grid, sink, b, R, D, triOf, offsets, cursor, total, std::max(batch / 4u, 1u), queue, s);
    *launches += 1;
}

size_t surface_rank_sums(uint64_t words) { return 2 * (size_t)(words / kRankStep + 8); }

void launch_surface_rank(const uint32_t* bits, uint64_t words, WordRank* ranks, uint32_t* sums, uint32_t* done,
                         uint32_t* total, void* keys, uint32_t keysCap, int wide, cudaStream_t s, uint32_t* launches) {
    // Tiles of four steps once there are two blocks of them per SM: fewer sums
    // for the last block to scan.
    const uint32_t S = words >= 148ull * 2 * 4 * kRankStep ? 4u : 1u;
    const uint32_t steps = std::max(1u, (uint32_t)((words + kRankStep - 1) / kRankStep)), tiles = (steps + S - 1) / S;
    uint32_t* stepSums = sums + tiles;   // up to S - 1 entries past `steps` are written
    if (S == 4) rankSumKernel<4><<<tiles, kBlock, 0, s>>>(bits, words, sums, stepSums, done, total);
    else rankSumKernel<1><<<tiles, kBlock, 0, s>>>(bits, words, sums, stepSums, done, total);
    if (wide) rankWriteKernel<true><<<steps, kBlock, 0, s>>>(bits, words, ranks, sums, stepSums, S, keys, keysCap);
    else rankWriteKernel<false><<<steps, kBlock, 0, s>>>(bits, words, ranks, sums, stepSums, S, keys, keysCap);
    *launches += 2;
}

void launch_surface_keys_zero(void* keys, const uint32_t* count, uint32_t cap, int wide, cudaStream_t s,
                              uint32_t* launches) {
    zeroKeysKernel<<<148 * 8, 256, 0, s>>>(keys, count, cap, wide);
    *launches += 1;
}

void launch_surface_merge(const unsigned long long* list, const uint32_t* listCount, uint32_t listCap,
                          const WordRank* ranks, uint32_t* keys, uint32_t keysCap,
                          uint32_t blocksPerSm, uint32_t entries, cudaStream_t s, uint32_t* launches) {
    // blocksPerSm 0: a block per 1,024 of the expected entries, so that blocks
    // retire as they finish and other streams' blocks get room (blocks past
    // the count exit at once; entries past the grid are taken by its
    // grid-stride loop).
    const uint32_t grid = blocksPerSm ? 148u * blocksPerSm : std::max(1u, (entries / 2 + 511) / 512);
    mergeKeysKernel<<<grid, 256, 0, s>>>(list, listCount, listCap, ranks, keys, keysCap);
    *launches += 1;
}

}  // namespace vxb
