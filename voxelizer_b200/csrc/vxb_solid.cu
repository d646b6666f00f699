// Solid (parity) voxelization kernels: calculateTileOverlap /
// constructWorkQueue / generateVoxelization (src/voxelizer.cu:840-1617),
// FP64 as in the reference.
//
// The reference sorts (tile, triangle) pairs and voxelizes one tile per
// block.  Here the work is the flat set of (work triangle, yz subspace, 4x4
// tile) candidates of every unit of the batch; a candidate is a member of
// the tile's list iff one voxel centre of the tile inside the triangle's
// clipped bounding box passes the binning test, and a member toggles, for
// each centre of the tile inside the subspace that passes the strict
// generation test, the bit of its x-intercept voxel in the centre's row.
// Toggles commute (XOR), so no sort is needed; a row prefix XOR then turns
// toggles into solid runs.
//
// No work list is built.  A warp takes a batch of up to 32 consecutive work
// triangles, sets them up one per lane in shared memory (count of candidates
// included) and walks their candidates 32 at a time over a prefix of those
// counts, so nothing is counted, scanned or searched in global memory first
// and no block-wide barrier holds a warp.  A batch with more than kSplit
// candidates keeps its first chunk and is listed with the number of the others,
// which a second launch spreads over all warps (a box wall alone has tens of
// thousands).  The list has room for every batch.  The first listCap chunks are
// also written out one by one: the search of a chunk's batch costs a call whose
// solid pass is mostly chunks 1-1.5% (stress mesh, 171 us).
//
// Bounds: FP64 issue at half rate (48 edge values a candidate) and the latency
// of its chains.  Solid pass alone on a B200 (memset, toggles, row fill), with
// a candidate list staged per block and with this split: room of 1,049,868
// triangles at 1024 voxels 364 -> 192 us, 81,920 triangles at 701 voxels
// 87 -> 52 us, 576 triangles at 32 voxels 48 -> 17 us.  Chunks of 32 or
// 128 candidates took 8 and 36 us more on the room; 32 costs scenes with many
// medium triangles (stress mesh 54 against 45 us) because every chunk sets
// its batch up again.  Five resident blocks of 96 registers: six (80) and
// seven (72) spill and are equal or up to 8% slower.

#include "vxb_common.cuh"
#include "vxb_device.cuh"
#include "vxb_kernels.cuh"

#include <algorithm>

namespace vxb {

using namespace detail;

namespace {

constexpr double kDblMin = 2.2250738585072014e-308;  // DBL_MIN, src/voxelizer.cu:1443
constexpr int kWarps = 4;                     // warps per block of the toggle kernels
constexpr int kBlocks = 5;                    // resident blocks per SM
constexpr uint32_t kSplit = 256;              // candidates of a batch before its chunks are listed
constexpr uint32_t kChunk = 64;               // candidates of one listed chunk
constexpr uint32_t kChunkBits = 33;           // low bits of the list's cursor: chunks; above: batches
constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kSeveral = 0x80000000u;    // a triangle in several subspaces

__device__ __forceinline__ void loadTriD(const float* __restrict__ V, const uint32_t* __restrict__ I, uint32_t t,
                                         D3* v) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        uint32_t a = __ldg(I + 3 * t + k);
        v[k] = D3{(double)__ldg(V + 3 * a), (double)__ldg(V + 3 * a + 1), (double)__ldg(V + 3 * a + 2)};
    }
}

// The division where divBy does not apply.
__device__ __noinline__ double divide(double x, double d) { return __ddiv_rn(x, d); }

// Per-triangle binning setup: calculateTileOverlap / constructWorkQueue,
// src/voxelizer.cu:861-945 and 1086-1144 (getTriangleBounds 2397-2418,
// getVoxelBoundsDouble 2446-2458, tN 882-884).
struct BinTri {
    D3 v[3];
    int vlo[2], vhi[2];
    double tN;
};

__device__ __forceinline__ void binSetup(const float* V, const uint32_t* I, uint32_t t, const PassGeom& g, BinTri& b) {
    loadTriD(V, I, t, b.v);
    double ymin = b.v[0].y, zmin = b.v[0].z, ymax = ymin, zmax = zmin;
#pragma unroll
    for (int i = 1; i < 3; ++i) {
        ymin = b.v[i].y < ymin ? b.v[i].y : ymin;
        zmin = b.v[i].z < zmin ? b.v[i].z : zmin;
        ymax = b.v[i].y > ymax ? b.v[i].y : ymax;
        zmax = b.v[i].z > zmax ? b.v[i].z : zmax;
    }
    const double d = g.d;
    const double rd = g.rd;
    double a0 = __dsub_rn(ymin, g.mn[1]), a1 = __dsub_rn(zmin, g.mn[2]);
    double b0 = __dsub_rn(ymax, g.mn[1]), b1 = __dsub_rn(zmax, g.mn[2]);
    if (rd != 0.0 && divExact(a0) && divExact(a1) && divExact(b0) && divExact(b1)) {
        a0 = divBy(a0, d, rd);
        a1 = divBy(a1, d, rd);
        b0 = divBy(b0, d, rd);
        b1 = divBy(b1, d, rd);
    } else {
        a0 = divide(a0, d);
        a1 = divide(a1, d);
        b0 = divide(b0, d);
        b1 = divide(b1, d);
    }
    b.vlo[0] = __double2int_rz(ceil(a0));
    b.vlo[1] = __double2int_rz(ceil(a1));
    b.vhi[0] = __double2int_rz(__dadd_rn(floor(b0), 1.0));
    b.vhi[1] = __double2int_rz(__dadd_rn(floor(b1), 1.0));
    const D3* v = b.v;
    b.tN = __dsub_rn(sum3<site::TN>(v[0].y, v[1].z, v[2].y, v[0].z, v[2].z, v[1].y),
                     sum3<site::TN>(v[2].y, v[1].z, v[0].z, v[1].y, v[2].z, v[0].y));
}

__device__ __forceinline__ bool binRejected(const BinTri& b) {
    return b.tN == 0.0 || b.vlo[0] >= b.vhi[0] || b.vlo[1] >= b.vhi[1];
}

// commonSpace of a triangle's range [vlo, vhi) and a subspace's [s0, s1) along
// one axis (src/voxelizer.cu:893-926): the number of 4-voxel tiles of the common
// range [*lo, *hi), 0 without one.
__device__ __forceinline__ uint32_t commonTiles(int vlo, int vhi, uint32_t s0, uint32_t s1, uint32_t* lo,
                                                uint32_t* hi) {
    if (vhi <= (int)s0 || vlo >= (int)s1) return 0u;
    *lo = (uint32_t)max((int)s0, vlo);
    *hi = min(s1, (uint32_t)vhi);
    return (*hi - 1) / 4 - *lo / 4 + 1;
}

// The unit and mesh triangle of work triangle wt.
__device__ __forceinline__ uint32_t workUnit(const Batch& b, uint32_t wt, uint32_t* t) {
    const uint32_t u = unitOf(b.workBase, b.nUnits, wt);
    *t = wt - __ldg(b.workBase + u);
    return u;
}

// The centres of a 4x4 tile starting at (ty, tz) that lie in [y0, y1) x
// [z0, z1), as bits 4 * cz + cy.
__device__ __forceinline__ uint32_t clipTile(uint32_t ty, uint32_t tz, uint32_t y0, uint32_t y1, uint32_t z0,
                                             uint32_t z1) {
    auto clip = [](uint32_t t, uint32_t lo, uint32_t hi) {
        const uint32_t l = lo > t ? min(lo - t, 4u) : 0u, h = hi > t ? min(hi - t, 4u) : 0u;
        return ((1u << h) - 1u) & ~((1u << l) - 1u);
    };
    const uint32_t y = clip(ty, y0, y1), z = clip(tz, z0, z1);
    return (y * 0x1111u) & (((z & 1u) | (z & 2u) << 3 | (z & 4u) << 6 | (z & 8u) << 9) * 15u);
}

// The triangles of one warp that have candidates, one slot each, and the
// warp's queue of toggles (lane of the candidate << 4 | centre).
// Field-major, so that lanes reading one field of different slots do not
// conflict.
struct SolidSlots {
    double v0[3][32];
    double n[3][32];                           // cross(v0 - v2, v1 - v0)
    double rn[32];                             // 1 / n.x (0: divide)
    double ex[3][32], ey[3][32], ed[3][32];    // generation edges (oriented by n.x)
    int lo[2][32], hi[2][32];                  // voxel box
    uint32_t wt[32], unit[32];
    uint32_t flags[32];   // bits 0-2: top-left generation edges; bit 3: binning edges are the same
    uint32_t off[32];     // first candidate
    uint32_t sub[32];     // the triangle's only subspace, or its tiles along y of all of them | kSeveral
    uint16_t queue[512];
};

// Candidates of work triangle wt.  The subspaces are a grid of ranges along y
// and along z, so a triangle's tiles are a product, and its candidates (subspace
// after subspace, y inner) are found along z and then along y: 34 ranges instead
// of 289 subspaces at 8192 x 8192 rows, where a look at each subspace per chunk
// of candidates made the solid pass of a box 7.6 ms, now 2.0.  A triangle within
// one subspace keeps its number.
__device__ __forceinline__ uint32_t solidCount(const Batch& b, uint32_t wt, BinTri& bt, uint32_t* unit,
                                               uint32_t* sub) {
    uint32_t t;
    *unit = workUnit(b, wt, &t);
    const Unit& U = b.units[*unit];
    binSetup(U.V, U.I, t, U.g, bt);
    if (binRejected(bt)) return 0u;
    const SplitYZ* __restrict__ splits = b.splits + U.splitBase;
    const uint32_t ny = U.splitN[0], nz = U.splitN[1];
    uint32_t lo, hi;
    const SplitYZ q0 = splits[0];
    uint32_t cy = commonTiles(bt.vlo[0], bt.vhi[0], q0.y0, q0.y1, &lo, &hi);
    uint32_t cz = commonTiles(bt.vlo[1], bt.vhi[1], q0.z0, q0.z1, &lo, &hi);
    uint32_t sy = 0, sz = 0;
    bool several = false;
    for (uint32_t s = 1; s < ny; ++s) {
        const uint32_t n = commonTiles(bt.vlo[0], bt.vhi[0], splits[s].y0, splits[s].y1, &lo, &hi);
        if (!n) continue;
        several |= cy != 0u;
        cy += n;
        sy = s;
    }
    for (uint32_t s = 1; s < nz; ++s) {
        const uint32_t n = commonTiles(bt.vlo[1], bt.vhi[1], splits[s * ny].z0, splits[s * ny].z1, &lo, &hi);
        if (!n) continue;
        several |= cz != 0u;
        cz += n;
        sz = s;
    }
    *sub = several ? kSeveral | cy : sz * ny + sy;
    return cy * cz;
}

__device__ __forceinline__ void solidStage(SolidSlots& st, uint32_t slot, const BinTri& bt, uint32_t unit,
                                           uint32_t wt) {
    const D3* v = bt.v;
    st.v0[0][slot] = v[0].x;
    st.v0[1][slot] = v[0].y;
    st.v0[2][slot] = v[0].z;
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        st.lo[a][slot] = bt.vlo[a];
        st.hi[a][slot] = bt.vhi[a];
    }
    st.wt[slot] = wt;
    st.unit[slot] = unit;
    const D3 A{__dsub_rn(v[0].x, v[2].x), __dsub_rn(v[0].y, v[2].y), __dsub_rn(v[0].z, v[2].z)};
    const D3 W{__dsub_rn(v[1].x, v[0].x), __dsub_rn(v[1].y, v[0].y), __dsub_rn(v[1].z, v[0].z)};
    const D3 n{diff2<site::CR_GEN>(A.y, W.z, A.z, W.y), diff2<site::CR_GEN>(A.z, W.x, A.x, W.z),
               diff2<site::CR_GEN>(A.x, W.y, A.y, W.x)};
    st.n[0][slot] = n.x;
    st.n[1][slot] = n.y;
    st.n[2][slot] = n.z;
    st.rn[slot] = divScale(n.x) ? __drcp_rn(n.x) : 0.0;
    uint32_t flags = (bt.tN > 0.0) == (n.x > 0.0) ? 8u : 0u;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const D3& p = v[i];
        const D3& q = v[(i + 1) % 3];
        double ex, ey;
        if (n.x > 0.0) { ex = __dsub_rn(p.z, q.z); ey = __dsub_rn(q.y, p.y); }
        else { ex = __dsub_rn(q.z, p.z); ey = __dsub_rn(p.y, q.y); }
        st.ex[i][slot] = ex;
        st.ey[i][slot] = ey;
        st.ed[i][slot] = -sum2<site::D_GEN>(ex, p.y, ey, p.z);
        if (ex > 0.0 || (ex == 0.0 && ey < 0.0)) flags |= 1u << i;
    }
    st.flags[slot] = flags;
}

// Sets up batch `batch` (whole warp): the slots of its triangles with
// candidates in order, *off the first candidate of slot `lane` (~0 past the
// last one).  Returns the number of candidates.
__device__ __forceinline__ uint32_t solidBatch(SolidSlots& st, const Batch& b, uint32_t batch, uint32_t perWarp,
                                               uint32_t nWork, uint32_t lane, unsigned long long* mine, uint32_t* off) {
    const uint32_t wt = batch * perWarp + lane;
    BinTri bt;
    uint32_t unit = 0, sub = 0;
    const uint32_t c = lane < perWarp && wt < nWork ? solidCount(b, wt, bt, &unit, &sub) : 0u;
    *mine += c;
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    const uint32_t used = __ballot_sync(kFull, c != 0u);
    if (c) {
        const uint32_t slot = __popc(used & laneMaskLt());
        st.off[slot] = incl - c;
        st.sub[slot] = sub;
        solidStage(st, slot, bt, unit, wt);
    }
    __syncwarp();
    *off = lane < __popc(used) ? st.off[lane] : 0xFFFFFFFFu;
    return __shfl_sync(kFull, incl, 31);
}

// Binning membership of a candidate evaluated from the triangle
// (traverseTilesForOverlaps, src/voxelizer.cu:980-1033): some centre of the
// tile inside the clipped box passes all three binning edges.
__device__ __noinline__ bool binMember(const Batch& b, uint32_t unit, uint32_t wt, uint32_t ty, uint32_t tz,
                                       uint32_t y0, uint32_t y1, uint32_t z0, uint32_t z1) {
    const Unit& U = b.units[unit];
    const PassGeom& g = U.g;
    BinTri bt;
    binSetup(U.V, U.I, wt - __ldg(b.workBase + unit), g, bt);
    const double d = g.d;
    double ex[3], ey[3], ed[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const D3& p = bt.v[i];
        const D3& q = bt.v[(i + 1) % 3];
        if (bt.tN > 0.0) { ex[i] = __dsub_rn(p.z, q.z); ey[i] = __dsub_rn(q.y, p.y); }
        else { ex[i] = __dsub_rn(q.z, p.z); ey[i] = __dsub_rn(p.y, q.y); }
        ed[i] = -sum2<site::D_BIN>(ex[i], p.y, ey[i], p.z);
    }
    for (uint32_t iz = max(tz, z0); iz < min(tz + 4u, z1); ++iz) {
        const double pz = lin<site::P_BIN>((double)iz, d, g.mn[2]);
        for (uint32_t iy = max(ty, y0); iy < min(ty + 4u, y1); ++iy) {
            const double py = lin<site::P_BIN>((double)iy, d, g.mn[1]);
            bool ok = true;
#pragma unroll
            for (int i = 0; i < 3; ++i) ok &= sum2p1<site::E_BIN>(ex[i], py, ey[i], pz, ed[i]) >= 0.0;
            if (ok) return true;
        }
    }
    return false;
}

// Candidate `local` of a slot: the centres it toggles (bits 4 * cz + cy of
// the tile at *ty, *tz; generateVoxelization, src/voxelizer.cu:1344-1440).
//
// The generation edges r > 0 (top-left: r + DBL_MIN > 0, i.e. r > -DBL_MIN)
// imply the binning edges r >= 0 where both sets have the same orientation,
// so a generating centre inside the clipped box makes the candidate a
// member, and a candidate without generating centres needs no membership.
// Only the rest (rounding at degenerate triangles) evaluates the binning
// edges.
__device__ __forceinline__ uint32_t solidCandidate(const SolidSlots& st, uint32_t slot, const Batch& b, uint32_t local,
                                                   uint32_t* ty, uint32_t* tz) {
    const Unit& U = b.units[st.unit[slot]];
    const PassGeom& g = U.g;
    const SplitYZ* __restrict__ splits = b.splits + U.splitBase;
    uint32_t lo[2] = {0, 0}, hi[2] = {1, 1}, nty = 1;
    const int vlo[2] = {st.lo[0][slot], st.lo[1][slot]}, vhi[2] = {st.hi[0][slot], st.hi[1][slot]};
    const uint32_t sub = st.sub[slot];
    SplitYZ sp = splits[sub & kSeveral ? 0u : sub];
    if (!(sub & kSeveral)) {
        nty = commonTiles(vlo[0], vhi[0], sp.y0, sp.y1, &lo[0], &hi[0]);
        commonTiles(vlo[1], vhi[1], sp.z0, sp.z1, &lo[1], &hi[1]);
    } else {
        const uint32_t ny = U.splitN[0], nz = U.splitN[1], tilesY = sub & ~kSeveral;
        uint32_t ntz = 1;
        for (uint32_t s = 0; s < nz; ++s) {
            const SplitYZ q = splits[s * ny];
            const uint32_t n = commonTiles(vlo[1], vhi[1], q.z0, q.z1, &lo[1], &hi[1]);
            if (!n) continue;
            sp.z0 = q.z0;
            sp.z1 = q.z1;
            ntz = n;
            if (local < n * tilesY) break;
            local -= n * tilesY;
        }
        for (uint32_t s = 0; s < ny; ++s) {
            const SplitYZ q = splits[s];
            const uint32_t n = commonTiles(vlo[0], vhi[0], q.y0, q.y1, &lo[0], &hi[0]);
            if (!n) continue;
            sp.y0 = q.y0;
            sp.y1 = q.y1;
            nty = n;
            if (local < n * ntz) break;
            local -= n * ntz;
        }
    }
    const uint32_t row = local / nty;
    const uint32_t y = (lo[0] / 4 + (local - row * nty)) * 4, z = (lo[1] / 4 + row) * 4;
    *ty = y;
    *tz = z;
    static_assert(site::E_BIN == 0 && site::E_GEN == 0, "row products assume the unfused edge forms");
    static_assert(site::P_BIN == site::P_GEN && site::D_BIN == site::D_GEN, "shared edges assume the same forms");
    const double d = g.d, my = g.mn[1], mz = g.mn[2];
    const uint32_t flags = st.flags[slot];
    // The products of the edges with the four columns' coordinates are kept
    // (the same unfused operations as from scratch).
    double least[3], ed[3], ry[3][4];
    {
        double py[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) py[c] = lin<site::P_GEN>(toDouble(y + c), d, my);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const double ex = st.ex[i][slot];
            ed[i] = st.ed[i][slot];
            least[i] = (flags >> i) & 1u ? -kDblMin : 0.0;
#pragma unroll
            for (int c = 0; c < 4; ++c) ry[i][c] = __dmul_rn(ex, py[c]);
        }
    }
    uint32_t gen = 0;
#pragma unroll
    for (int cz = 0; cz < 4; ++cz) {
        const double pz = lin<site::P_GEN>(toDouble(z + cz), d, mz);
        double rz[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) rz[i] = __dmul_rn(st.ey[i][slot], pz);
#pragma unroll
        for (int cy = 0; cy < 4; ++cy) {
            bool in = true;
#pragma unroll
            for (int i = 0; i < 3; ++i) in &= __dadd_rn(__dadd_rn(ry[i][cy], rz[i]), ed[i]) > least[i];
            if (in) gen |= 1u << (4 * cz + cy);
        }
    }
    gen &= clipTile(y, z, sp.y0, sp.y1, sp.z0, sp.z1);
    if (gen && !((flags & 8u) && (gen & clipTile(y, z, lo[0], hi[0], lo[1], hi[1]))) &&
        !binMember(b, st.unit[slot], st.wt[slot], y, z, lo[0], hi[0], lo[1], hi[1]))
        gen = 0u;
    return gen;
}

// The grid word and bit that centre (vy, vz) toggles for a slot's triangle
// (src/voxelizer.cu:1441-1462); a zero bit past the grid.  Straight-line but
// for operands divBy does not take, so that two toggles of a lane overlap.
struct Toggle {
    uint32_t* word;
    uint32_t bit;
};
__device__ __forceinline__ Toggle solidToggle(const SolidSlots& st, uint32_t slot, const Batch& b, uint32_t vy,
                                              uint32_t vz, uint32_t* __restrict__ fill) {
    const Unit& U = b.units[st.unit[slot]];
    const PassGeom& g = U.g;
    const double d = g.d, rd = g.rd;
    const double py = lin<site::P_GEN>(toDouble(vy), d, g.mn[1]), pz = lin<site::P_GEN>(toDouble(vz), d, g.mn[2]);
    const double nx = st.n[0][slot], rn = st.rn[slot];
    const double ax = __dsub_rn(st.v0[0][slot], g.mn[0]), ay = __dsub_rn(st.v0[1][slot], py),
                 az = __dsub_rn(st.v0[2][slot], pz);
    const double B = sum3<site::B_GEN>(ax, nx, ay, st.n[1][slot], az, st.n[2][slot]);
    double px = divBy(B, nx, rn);
    px = px < 0.0 ? 0.0 : px;
    double x = divBy(px, d, rd);
    if (rn == 0.0 || rd == 0.0 || !divExact(B) || !divExact(px)) {
        px = divide(B, nx);
        px = px < 0.0 ? 0.0 : px;
        x = divide(px, d);
    }
    const uint32_t vx = __double2uint_rz(ceil(x)) + 1u;
    const uint32_t row = (vz + g.padZ) * g.AY + (vy + g.padY);
    return Toggle{fill + U.wordBase + (size_t)row * g.ipx + (vx >> 5), vx < g.X ? 0x80000000u >> (vx & 31u) : 0u};
}

// Candidates [first, last) of a warp's slots (whole warp; `off` as
// solidBatch leaves it).  Each step tests the tiles of 32 candidates, queues
// the centres that toggle and then works the queue 32 centres at a time, so
// that the divisions of the intercept run in full warps although a tile
// toggles 2-3 of its 16 centres on average.
__device__ __forceinline__ void solidCandidates(SolidSlots& st, const Batch& b, uint32_t off, uint32_t first,
                                                uint32_t last, uint32_t lane, uint32_t* __restrict__ fill) {
    for (uint32_t base = first; base < last; base += 32u) {
        // Every slot has a candidate, so the slots that start inside the
        // window are consecutive.
        const uint32_t s0 = __popc(__ballot_sync(kFull, off <= base)) - 1u;
        const uint32_t starts = __reduce_or_sync(kFull, off > base && off - base < 32u ? 1u << (off - base) : 0u);
        uint32_t slot = s0 + __popc(starts & ((2u << lane) - 1u));
        const uint32_t o = __shfl_sync(kFull, off, slot);
        const uint32_t item = base + lane;
        uint32_t gen = 0, ty = 0, tz = 0;
        if (item < last) gen = solidCandidate(st, slot, b, item - o, &ty, &tz);
        // Queue positions: exclusive prefix of the lanes' centre counts.
        uint32_t n = __popc(gen), incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(kFull, incl, o);
            if (lane >= (uint32_t)o) incl += t;
        }
        const uint32_t total = __shfl_sync(kFull, incl, 31);
        uint32_t at = incl - n;
        while (gen) {
            st.queue[at++] = (uint16_t)((lane << 4) | (__ffs(gen) - 1));
            gen &= gen - 1u;
        }
        __syncwarp();
        for (uint32_t q = 0; q < total; q += 64u) {
            const bool in0 = q + lane < total, in1 = q + 32u + lane < total;
            const uint32_t e0 = st.queue[in0 ? q + lane : 0u], e1 = st.queue[in1 ? q + 32u + lane : 0u];
            const uint32_t s0 = __shfl_sync(kFull, slot, e0 >> 4), s1 = __shfl_sync(kFull, slot, e1 >> 4);
            const uint32_t y0 = __shfl_sync(kFull, ty, e0 >> 4), y1 = __shfl_sync(kFull, ty, e1 >> 4);
            const uint32_t z0 = __shfl_sync(kFull, tz, e0 >> 4), z1 = __shfl_sync(kFull, tz, e1 >> 4);
            const Toggle t0 = solidToggle(st, s0, b, y0 + (e0 & 3u), z0 + ((e0 >> 2) & 3u), fill);
            if (q + 32u < total) {
                const Toggle t1 = solidToggle(st, s1, b, y1 + (e1 & 3u), z1 + ((e1 >> 2) & 3u), fill);
                if (in1 && t1.bit) atomicXor(t1.word, t1.bit);
            }
            if (in0 && t0.bit) atomicXor(t0.word, t0.bit);
        }
        __syncwarp();
    }
}

// The listed batches and their chunks (launch_solid_toggle).
struct BigList {
    unsigned long long* cursor;   // NULL: nothing is listed
    uint32_t* first;
    uint32_t* batch;
    uint32_t cap;                 // batches
    uint2* list;                  // batch and chunk, for the first listCap chunks
    uint32_t listCap;
};

// Toggles of every work triangle.  A warp takes batches of `perWarp` (a
// power of two up to 32) triangles in a fixed grid-stride order or (queue !=
// NULL) from a device work queue, one atomic per batch.  A batch with more than
// kSplit candidates is listed for its chunks after the first: big.first[k] is the
// number of the first of them among all listed chunks, big.batch[k] the batch.
// One atomic on *cursor gives both k and that number, so the numbers ascend.
// *total counts the candidates.
__global__ void __launch_bounds__(kWarps * 32, kBlocks) solidToggleKernel(Batch b, uint32_t nWork, uint32_t perWarp,
                                                                          unsigned long long* total, BigList big,
                                                                          uint32_t* __restrict__ fill,
                                                                          uint32_t* queue) {
    __shared__ SolidSlots slots[kWarps];
    const uint32_t lane = threadIdx.x & 31u;
    SolidSlots& st = slots[threadIdx.x >> 5];
    const uint32_t batches = (nWork + perWarp - 1) / perWarp;
    const uint32_t nWarps = gridDim.x * kWarps;
    unsigned long long mine = 0;
    uint32_t bt = blockIdx.x * kWarps + (threadIdx.x >> 5);
    auto take = [&]() {
        uint32_t v = 0;
        if (lane == 0) v = atomicAdd(queue, 1u);
        return __shfl_sync(kFull, v, 0);
    };
    if (queue) bt = take();
    while (bt < batches) {
        uint32_t off;
        uint32_t n = solidBatch(st, b, bt, perWarp, nWork, lane, &mine, &off);
        if (n > kSplit && big.cursor) {
            const uint32_t more = (n - 1u) / kChunk;   // chunks 1 .. more
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(big.cursor, (1ull << kChunkBits) + more);
            at = __shfl_sync(kFull, at, 0);
            const uint32_t entry = (uint32_t)(at >> kChunkBits);
            // The batches that reserved 2^26 chunks have 2^32 candidates: the
            // host refuses the call, and the rest would be in vain.  (Past that
            // the chunks may carry into the number of batches.)
            static_assert((unsigned long long)kChunk << 26 == 1ull << 32, "candidates of 2^26 chunks");
            if ((at & ((1ull << kChunkBits) - 1u)) >= 1u << 26 || entry >= big.cap) break;
            if (lane == 0) {
                big.first[entry] = (uint32_t)at;
                big.batch[entry] = bt;
            }
            for (uint32_t k = lane; k < more && (uint32_t)at + k < big.listCap; k += 32u)
                big.list[(uint32_t)at + k] = make_uint2(bt, k + 1u);
            n = kChunk;
        }
        solidCandidates(st, b, off, 0u, n, lane, fill);
        bt = queue ? take() : bt + nWarps;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) mine += __shfl_down_sync(kFull, mine, o);
    if (lane == 0 && mine) atomicAdd(total, mine);
}

// The listed chunks, one warp each.
__global__ void __launch_bounds__(kWarps * 32, kBlocks) solidBigKernel(Batch b, uint32_t nWork, uint32_t perWarp,
                                                                       const unsigned long long* __restrict__ total,
                                                                       BigList big, uint32_t* __restrict__ fill) {
    __shared__ SolidSlots slots[kWarps];
    const unsigned long long listed = *big.cursor, all = *total;   // both in flight
    if (all >= 0xFFFFFFFFull) return;   // refused by the host
    const uint32_t lane = threadIdx.x & 31u;
    SolidSlots& st = slots[threadIdx.x >> 5];
    const uint32_t entries = (uint32_t)(listed >> kChunkBits), chunks = (uint32_t)listed;
    for (uint32_t c = blockIdx.x * kWarps + (threadIdx.x >> 5); c < chunks; c += gridDim.x * kWarps) {
        uint2 at;   // batch, chunk of it
        if (c < big.listCap) {
            at = big.list[c];
        } else {
            const uint32_t e = warpFindOwner(big.first, entries, c, lane);
            at = make_uint2(big.batch[e], c - big.first[e] + 1u);
        }
        unsigned long long mine = 0;
        uint32_t off;
        const uint32_t n = solidBatch(st, b, at.x, perWarp, nWork, lane, &mine, &off);
        const uint32_t first = at.y * kChunk;
        solidCandidates(st, b, off, first, min(n - first, kChunk) + first, lane, fill);
    }
}

// Toggle bits -> solid runs: bit x of a row = XOR of the row's toggles at or
// before x.  A warp takes kFillRows whole rows (consecutive words) and walks
// them as 32-word chunks, one word per lane, so loads and stores are
// coalesced: a lane turns its word into the prefix XOR of its bits and
// inverts it when the words before it in its row hold an odd number of
// toggles.  That parity is a segmented XOR scan over the lanes (a ballot of
// word parities, cut at the lanes that start a row) plus the parity carried
// from the previous chunk for the row that continues into this one.  Bound by
// the loads in flight: kFillAhead chunks are loaded before the first is
// scanned, and a task holds about kFillWords words whatever the row length
// (one chunk ahead and 16 rows a task: room, 13.5 M words, 50 us, duct, 130
// words a row, 50, batch of 64 meshes 95; now 41, 28 and 69).
constexpr uint32_t kFillAhead = 6;
constexpr uint32_t kFillWords = 1152;  // words of a task, about

__global__ void rowFillKernel(Batch b, uint64_t nRows, uint32_t rowsPerTask, uint32_t* __restrict__ fill) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t nWarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t g = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; g * rowsPerTask < nRows; g += nWarps) {
        uint64_t row = g * rowsPerTask;
        const uint64_t rowEnd = min(row + rowsPerTask, nRows);
        while (row < rowEnd) {
            // The rows of [row, rowEnd) in one unit.
            const uint32_t u = b.nUnits > 1 ? unitOf(b.rowBase, b.nUnits, row) : 0u;
            const uint64_t uRow0 = __ldg(b.rowBase + u), uRow1 = __ldg(b.rowBase + u + 1);
            const uint64_t r1 = min(rowEnd, uRow1);
            const Unit& U = b.units[u];
            const uint32_t ipx = U.g.ipx;
            const FastDiv divX = U.g.divX;
            uint32_t* words = fill + U.wordBase;
            const uint32_t w0 = (uint32_t)(row - uRow0) * ipx, w1 = (uint32_t)(r1 - uRow0) * ipx;
            uint32_t carry = 0u;
            for (uint32_t cb = w0; cb < w1; cb += 32u * kFillAhead) {
                uint32_t x[kFillAhead];
#pragma unroll
                for (uint32_t q = 0; q < kFillAhead; ++q) x[q] = cb + 32u * q + lane < w1 ? words[cb + 32u * q + lane] : 0u;
#pragma unroll
                for (uint32_t q = 0; q < kFillAhead; ++q) {
                    const uint32_t w = cb + 32u * q + lane;
                    const bool valid = w < w1;
                    const uint32_t starts = __ballot_sync(0xffffffffu, valid && divX.div(w) * ipx == w);
                    const uint32_t odd = __ballot_sync(0xffffffffu, __popc(x[q]) & 1u);
                    const uint32_t upTo = starts & ((2u << lane) - 1u);   // row starts at lanes <= lane
                    uint32_t below = (1u << lane) - 1u;                  // lanes < lane
                    uint32_t pre;
                    if (upTo) {
                        below &= ~((1u << (31u - __clz(upTo))) - 1u);
                        pre = __popc(odd & below) & 1u;
                    } else {
                        pre = (__popc(odd & below) & 1u) ^ carry;
                    }
                    uint32_t p = x[q];
                    p ^= p >> 1; p ^= p >> 2; p ^= p >> 4; p ^= p >> 8; p ^= p >> 16;
                    if (pre) p = ~p;
                    if (valid && p != x[q]) words[w] = p;
                    carry = __shfl_sync(0xffffffffu, pre ^ (__popc(x[q]) & 1u), 31);
                }
            }
            row = r1;
        }
    }
}

}  // namespace

// Triangles per batch: 32 lanes set up 32, but a small mesh is spread over 8
// warps per SM first (one triangle per warp at the least).
static uint32_t solidPerWarp(uint32_t nWork) {
    uint32_t n = 1;
    while (n < 32u && nWork / (2u * n) >= 148u * 8u) n *= 2u;
    return n;
}

bool solid_may_list(const PassGeom& g, uint64_t nSplits, uint32_t nWork) {
    // A triangle has at most one candidate per 4x4 tile and one more row and
    // column of partial tiles per subspace cut.
    return ((g.resY + 3ull) / 4 + nSplits) * ((g.resZ + 3ull) / 4 + nSplits) * solidPerWarp(nWork) > kSplit;
}

static uint32_t solidBatches(uint32_t nWork) {
    const uint32_t perWarp = solidPerWarp(nWork);
    return (nWork + perWarp - 1) / perWarp;
}

size_t solid_big_bytes(uint32_t nWork, uint32_t listCap) { return 8 * ((size_t)solidBatches(nWork) + listCap); }

void launch_solid_toggle(const Batch& b, uint32_t nWork, unsigned long long* total, void* big,
                         unsigned long long* cursor, uint32_t listCap, uint32_t* fill, uint32_t blocksPerSm,
                         uint32_t* queue, cudaStream_t s, uint32_t* launches) {
    const uint32_t perWarp = solidPerWarp(nWork), batches = solidBatches(nWork);
    BigList l{};
    if (big) {
        l.cursor = cursor;
        l.list = static_cast<uint2*>(big);
        l.listCap = listCap;
        l.first = reinterpret_cast<uint32_t*>(l.list + listCap);
        l.batch = l.first + batches;
        l.cap = batches;
    }
    if (queue) cudaMemsetAsync(queue, 0, sizeof(uint32_t), s);
    const uint32_t grid = gridFor(batches, kWarps, 148u * 8u * blocksPerSm);
    solidToggleKernel<<<grid, kWarps * 32, 0, s>>>(b, nWork, perWarp, total, l, fill, queue);
    *launches += 1;
    if (big) {
        solidBigKernel<<<148 * kBlocks, kWarps * 32, 0, s>>>(b, nWork, perWarp, total, l, fill);
        *launches += 1;
    }
}

void launch_row_fill(const Batch& b, uint64_t nRows, uint64_t totalWords, uint32_t* fill, cudaStream_t s,
                     uint32_t* launches) {
    // About kFillWords words a task (six rounds of loads), less where
    // that leaves fewer than 16 warps per SM.
    const uint64_t rows = std::min(kFillWords * nRows / std::max<uint64_t>(totalWords, 1), nRows / (148u * 16u));
    const uint32_t perTask = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(rows, 1), 512);
    rowFillKernel<<<gridFor((nRows + perTask - 1) / perTask * 32u, 256), 256, 0, s>>>(b, nRows, perTask, fill);
    *launches += 1;
}

}  // namespace vxb
