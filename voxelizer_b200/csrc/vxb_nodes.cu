// Node classification kernels: packed-bit pruning and node emission.
//
// Emission reads three bit grids (final solid, unpruned fill, surface) and
// writes the node grid once, from 32-bit words (32 nodes of a row).  The
// neighbour masks of a word are shifts of it and of the words around it, so a
// word of one id (all empty, or all solid with all six neighbours solid: id 27)
// costs a few bitwise operations; the ids of the others are computed bit-sliced
// (a plane per id bit) and transposed to bytes.  1- and 2-byte nodes: warps walk
// planes along z, store words of one id at once and collect the others until 32
// are there.  PartialNodes and FCC nodes: a lane forms the ids of a word, and the
// warp stores its words' nodes in order, 16 bytes a lane.
//
// Grids of one unit hold fewer than 2^32 voxels, so word indices inside a
// unit fit 32 bits; arena offsets (unit word bases) are 64-bit.

#include "vxb_common.cuh"
#include "vxb_device.cuh"
#include "vxb_kernels.cuh"
#include "vxb_ratio.cuh"

#include <algorithm>

namespace vxb {

using namespace detail;

namespace {

// Pruning (fillNodeList2 and the host loop, src/voxelizer.cu:1790-1913,
// src/host_side.cpp:1183-1206): a solid node stays solid iff each axis has a
// solid neighbour.  The reference repeats in-place passes over one yz
// subspace until nothing changes, then goes on to the next subspace, so a
// subspace sees the earlier ones pruned and the later ones unpruned.
// Neighbours in a later subspace are therefore read from the unpruned grid
// (fill | surf).  With that rule a subspace depends only on itself and on
// earlier ones, and pruning all of them at once reaches the same greatest
// fixed point as pruning them in order: passes only clear bits, and the
// joint fixed point of such a chain is the chain of the fixed points.
//
// Pass 0 reads the unpruned grid and writes the pruned one, so it needs no
// copy first, and lists the words it changed.  Later passes visit only those:
// a node can only die when a neighbour did, and then on that neighbour's
// axis, so a pass tests, for every bit that a listed word has lost, the
// neighbour on each side against the neighbour behind it.  They clear bits
// with atomicAnd (a word may be reached from several sides) and list the
// words whose bits they cleared.
//
// Bounds: pass 0 moves three bit arenas (the neighbour rows hit in L1 / L2);
// the later passes are short gathers.  Pruning alone on a B200, with one pass
// sequence per subspace and all six neighbours of every listed word
// evaluated, and now: room of 13.5 M words (four subspaces) 195 -> 74 us, 4.6 M
// words without materials 112 -> 35 us, 8.7 M words 106 -> 54 us.  Pass 0 alone
// on the room: 134 us with the six neighbours loaded per word, 112 us walking
// planes with the next plane loaded one barrier ahead (4 words a thread, 64
// registers), 62 us with it loaded two barriers ahead and 2 words a thread
// (40 registers): it is bound by the loads in flight.
struct PruneView {
    uint32_t* S;
    const uint32_t* F;
    const uint32_t* Sf;        // NULL without materials
    const uint8_t* yLater;
    const uint8_t* zLater;
    uint32_t ipx, AY, AZ, nWords;
    FastDiv divX, divY;
};

__device__ __forceinline__ PruneView pruneView(const Batch& b, uint32_t unit, uint32_t* solid, const uint32_t* fill,
                                               const uint32_t* surf) {
    const Unit& U = b.units[unit];
    PruneView v;
    v.S = solid + U.wordBase;
    v.F = fill + U.wordBase;
    v.Sf = (surf && U.materials) ? surf + U.wordBase : nullptr;
    v.yLater = b.later + U.laterBase;
    v.ipx = U.g.ipx;
    v.AY = U.g.AY;
    v.AZ = U.g.AZ;
    v.nWords = v.ipx * v.AY * v.AZ;
    v.zLater = v.yLater + v.AY;
    v.divX = U.g.divX;
    v.divY = U.g.divY;
    return v;
}

__device__ __forceinline__ uint32_t unpruned(const PruneView& v, uint32_t idx) {
    return __ldg(v.F + idx) | (v.Sf ? __ldg(v.Sf + idx) : 0u);
}

// The nodes of a word that keep a neighbour on each axis.
__device__ __forceinline__ uint32_t prunedWord(uint32_t w, uint32_t prev, uint32_t next, uint32_t in, uint32_t out,
                                               uint32_t dn, uint32_t up) {
    return w & ((w >> 1) | (prev << 31) | (w << 1) | (next >> 31)) & (in | out) & (dn | up);
}

// Pass 0.  A block takes kPruneSpan consecutive words of a plane (across
// rows) and walks `planes` planes along z: a thread keeps its words of the
// planes below, at and above the current one in registers, the current plane
// goes through shared memory for the neighbours along x and y, and only those
// outside the span are read again from memory.  So each word of the two
// arenas is loaded once per block instead of seven times, and the positions
// are divided out once per block.
//
// A unit whose planes are thin (kPruneThin words at the most) would leave most
// of such a block idle.  In a launch of its own, its threads take one word each,
// across planes, and load its neighbours: pruning of a rod of 60,002 planes of 7
// words 256 us walking planes, 15 this way; 4,002 planes of 512 words 34 and 27;
// a batch of 2,000 meshes of 16-24 voxels 434 and 137 us.
constexpr int kPruneThreads = 512;
constexpr int kPruneWords = 2;   // words per thread and plane
constexpr uint32_t kPruneSpan = kPruneThreads * kPruneWords;
constexpr uint32_t kPruneThin = kPruneSpan / 2;
constexpr uint32_t kThinThreads = 256;
constexpr uint32_t kPruneKeep = 512;   // changed words a block collects before it lists them one by one

template <bool kThin>
__global__ void __launch_bounds__(kThin ? kThinThreads : kPruneThreads) pruneFirstKernel(Batch b, const uint32_t* __restrict__ blockBase,
                                                                  uint32_t planes, uint32_t* __restrict__ solid,
                                                                  const uint32_t* __restrict__ fill,
                                                                  const uint32_t* __restrict__ surf,
                                                                  unsigned long long* list, uint32_t* count,
                                                                  uint32_t cap, uint32_t* overflow) {
    __shared__ uint32_t buf[2][kPruneSpan];
    __shared__ uint32_t kept[kPruneKeep];
    __shared__ uint32_t nKept, listAt;
    if (threadIdx.x == 0) nKept = 0;
    const uint32_t u = b.nUnits > 1 ? unitOf(blockBase, b.nUnits, blockIdx.x) : 0u;
    const PruneView v = pruneView(b, u, solid, fill, surf);
    const uint32_t plane = v.ipx * v.AY, spans = (plane + kPruneSpan - 1) / kPruneSpan;
    const uint32_t t = blockIdx.x - __ldg(blockBase + u);
    // Lists a changed word.
    auto keep = [&](uint32_t idx) {
        const uint32_t k = atomicAdd(&nKept, 1u);
        if (k < kPruneKeep) {
            kept[k] = idx;
            return;
        }
        const uint32_t g = atomicAdd(count, 1u);
        if (g < cap) list[g] = ((unsigned long long)u << 32) | idx;
        else *overflow = 1u;
    };
    // The block's collected words go to the list together (whole block).
    auto listKept = [&]() {
        __syncthreads();
        const uint32_t nList = min(nKept, kPruneKeep);
        if (threadIdx.x == 0 && nList) listAt = atomicAdd(count, nList);
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < nList; k += kThin ? kThinThreads : kPruneThreads) {
            if (listAt + k < cap) list[listAt + k] = ((unsigned long long)u << 32) | kept[k];
            else *overflow = 1u;
        }
    };
    if (kThin) {
        __syncthreads();   // nKept
        const uint32_t idx = t * kThinThreads + threadIdx.x;
        if (idx < v.nWords) {
            const uint32_t w = unpruned(v, idx);
            uint32_t nw = 0u;
            if (w) {
                const uint32_t row = v.divX.div(idx), k = idx - row * v.ipx, z = v.divY.div(row), y = row - z * v.AY;
                auto at = [&](bool there, uint32_t i) { return there ? unpruned(v, i) : 0u; };
                nw = prunedWord(w, at(k > 0, idx - 1), at(k + 1 < v.ipx, idx + 1), at(y > 0, idx - v.ipx),
                                at(y + 1 < v.AY, idx + v.ipx), at(z > 0, idx - plane), at(z + 1 < v.AZ, idx + plane));
                if (nw != w) keep(idx);
            }
            v.S[idx] = nw;
        }
        listKept();
        return;
    }
    const uint32_t zc = t / spans;
    const uint32_t s0 = (t - zc * spans) * kPruneSpan;
    const uint32_t z0 = zc * planes, z1 = min(z0 + planes, v.AZ), n = min(kPruneSpan, plane - s0);
    uint32_t sides[kPruneWords];   // bits 0-3: a neighbour at x - 1, x + 1, y - 1, y + 1
    // The words below and at the current plane, and the two arenas' words of
    // the next plane, whose loads are issued a plane ahead.
    uint32_t below[kPruneWords], mid[kPruneWords], nextF[kPruneWords], nextS[kPruneWords];
    auto loadPlane = [&](uint32_t z, int q, uint32_t& f, uint32_t& sf) {
        const uint32_t l = threadIdx.x + q * kPruneThreads;
        const bool ok = l < n && z < v.AZ;
        const uint32_t i = z * plane + s0 + l;
        f = ok ? __ldg(v.F + i) : 0u;
        sf = ok && v.Sf ? __ldg(v.Sf + i) : 0u;
    };
#pragma unroll
    for (int q = 0; q < kPruneWords; ++q) {
        const uint32_t l = threadIdx.x + q * kPruneThreads, j = s0 + l;
        const uint32_t y = v.divX.div(j), k = j - y * v.ipx;
        sides[q] = (k > 0) | (k + 1 < v.ipx) << 1 | (y > 0) << 2 | (y + 1 < v.AY) << 3;
        uint32_t f, sf, f0 = 0u, sf0 = 0u;
        if (z0 > 0) loadPlane(z0 - 1, q, f0, sf0);
        loadPlane(z0, q, f, sf);
        loadPlane(z0 + 1, q, nextF[q], nextS[q]);
        below[q] = f0 | sf0;
        mid[q] = f | sf;
    }
    for (uint32_t z = z0; z < z1; ++z) {
        const uint32_t base = z * plane + s0;
        uint32_t* cur = buf[z & 1u];
        uint32_t up[kPruneWords];
#pragma unroll
        for (int q = 0; q < kPruneWords; ++q) {
            up[q] = nextF[q] | nextS[q];
            if (z + 1 < z1) loadPlane(z + 2, q, nextF[q], nextS[q]);
            cur[threadIdx.x + q * kPruneThreads] = mid[q];
        }
        __syncthreads();   // one barrier a plane: the buffers alternate
#pragma unroll
        for (int q = 0; q < kPruneWords; ++q) {
            const uint32_t l = threadIdx.x + q * kPruneThreads;
            if (l >= n) break;
            const uint32_t w = mid[q];
            uint32_t nw = 0u;
            if (w) {
                auto at = [&](uint32_t side, bool inside, int step) {
                    if (!((sides[q] >> side) & 1u)) return 0u;
                    return inside ? cur[(int)l + step] : unpruned(v, base + l + step);
                };
                nw = prunedWord(w, at(0, l > 0, -1), at(1, l + 1 < n, 1), at(2, l >= v.ipx, -(int)v.ipx),
                                at(3, l + v.ipx < n, (int)v.ipx), below[q], up[q]);
                if (nw != w) keep(base + l);
            }
            v.S[base + l] = nw;
            below[q] = w;
        }
#pragma unroll
        for (int q = 0; q < kPruneWords; ++q) mid[q] = up[q];
    }
    listKept();
}

// Clears `dead` of word idx and lists the word when that took a bit.
__device__ __forceinline__ void pruneClear(const PruneView& v, uint32_t idx, uint32_t dead, unsigned long long unit,
                                           unsigned long long* out, uint32_t* outCount, uint32_t cap,
                                           uint32_t* overflow) {
    if (!dead || !(atomicAnd(v.S + idx, ~dead) & dead)) return;
    const uint32_t at = atomicAdd(outCount, 1u);
    if (at < cap) out[at] = (unit << 32) | idx;
    else *overflow = 1u;
}

// One listed word: `lost` bits of it are gone, so each of their neighbours
// dies unless its neighbour on the other side is solid.  Solid words are read
// past L1 (other threads clear bits meanwhile; a bit cleared after it was
// read here lists its word, whose visit then finds this side empty).
__device__ __forceinline__ void pruneListed(const Batch& b, uint32_t* solid, const uint32_t* __restrict__ fill,
                                            const uint32_t* __restrict__ surf, unsigned long long ent,
                                            unsigned long long* out, uint32_t* outCount, uint32_t cap,
                                            uint32_t* overflow) {
    const uint32_t unit = (uint32_t)(ent >> 32), idx = (uint32_t)ent;
    const PruneView v = pruneView(b, unit, solid, fill, surf);
    const uint32_t plane = v.ipx * v.AY;
    const uint32_t row = v.divX.div(idx), k = idx - row * v.ipx, z = v.divY.div(row), y = row - z * v.AY;
    auto ld = [&](uint32_t i) { return __ldcg(v.S + i); };
    const uint32_t w = ld(idx), lost = unpruned(v, idx) & ~w;
    const uint32_t prev = k > 0 ? ld(idx - 1) : 0u, next = k + 1 < v.ipx ? ld(idx + 1) : 0u;
    const uint32_t yAfter = y + 1 < v.AY ? ld(idx + v.ipx) : 0u, yBefore = y > 0 ? ld(idx - v.ipx) : 0u;
    const uint32_t zAfter = z + 1 < v.AZ ? ld(idx + plane) : 0u, zBefore = z > 0 ? ld(idx - plane) : 0u;
    auto clear = [&](uint32_t i, uint32_t dead) { pruneClear(v, i, dead, unit, out, outCount, cap, overflow); };
    // x: inside the word, the last node of the previous word and the first
    // of the next.
    clear(idx, w & ~((w >> 1) | (prev << 31) | (w << 1) | (next >> 31)));
    if ((lost & 0x80000000u) && (prev & 3u) == 1u) clear(idx - 1, 1u);
    if ((lost & 1u) && (next & 0xC0000000u) == 0x80000000u) clear(idx + 1, 0x80000000u);
    // y, z: the row (plane) before sees this word's unpruned bits when this
    // one belongs to a later subspace.
    auto side = [&](uint32_t at, uint32_t step, uint32_t n, const uint8_t* later, uint32_t after, uint32_t before) {
        if (after & lost) {
            uint32_t far = 0u;
            if (at + 2 < n) far = later[at + 1] ? unpruned(v, idx + 2 * step) : ld(idx + 2 * step);
            clear(idx + step, after & lost & ~far);
        }
        if ((before & lost) && !later[at - 1])
            clear(idx - step, before & lost & ~(at > 1 ? ld(idx - 2 * step) : 0u));
    };
    side(y, v.ipx, v.AY, v.yLater, yAfter, yBefore);
    side(z, plane, v.AZ, v.zLater, zAfter, zBefore);
}

constexpr uint32_t kLoopBlocks = 8, kLoopThreads = 512;

// Pass 1 over the whole device.
__global__ void __launch_bounds__(256) pruneListKernel(Batch b, uint32_t* solid, const uint32_t* __restrict__ fill,
                                                       const uint32_t* __restrict__ surf,
                                                       const unsigned long long* __restrict__ in,
                                                       const uint32_t* __restrict__ inCount, unsigned long long* out,
                                                       uint32_t* outCount, uint32_t cap, uint32_t* overflow) {
    const uint32_t nIn = min(*inCount, cap);
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < nIn; e += gridDim.x * blockDim.x)
        pruneListed(b, solid, fill, surf, in[e], out, outCount, cap, overflow);
}

// Passes firstPass .. passes - 1 in one cluster of blocks, with a cluster
// barrier between passes (the lists alternate).  It stops once a list is
// empty.  A list longer than `escapeAt` is left to the host (*overflow); the
// list of pass 1 is taken whole.  Every block reads the same counts, which
// the barrier before a pass has made final, so all leave together.
__global__ void __cluster_dims__(kLoopBlocks, 1, 1) __launch_bounds__(kLoopThreads)
    pruneListLoopKernel(Batch b, uint32_t* solid, const uint32_t* __restrict__ fill,
                        const uint32_t* __restrict__ surf, uint32_t passes, uint32_t firstPass,
                        unsigned long long* list0, unsigned long long* list1, uint32_t* counts, uint32_t cap,
                        uint32_t escapeAt, uint32_t* overflow) {
    for (uint32_t pass = firstPass; pass < passes; ++pass) {
        if (pass > firstPass) {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
        const uint32_t nIn = min(__ldcg(counts + pass - 1), cap);
        if (nIn == 0) return;
        if (pass > 1 && nIn > escapeAt) {
            if (blockIdx.x == 0 && threadIdx.x == 0) *overflow = 1u;
            return;
        }
        const unsigned long long* in = (pass - 1) & 1u ? list1 : list0;
        unsigned long long* out = pass & 1u ? list1 : list0;
        for (uint32_t e = blockIdx.x * kLoopThreads + threadIdx.x; e < nIn; e += kLoopBlocks * kLoopThreads)
            pruneListed(b, solid, fill, surf, __ldcg(in + e), out, counts + pass, cap, overflow);
        __syncwarp();   // the barrier above wants whole warps
    }
}

// One in-place pass over every word; *changed is set when a bit was cleared.
__global__ void pruneFullKernel(Batch b, uint64_t totalWords, uint32_t* solid, const uint32_t* __restrict__ fill,
                                const uint32_t* __restrict__ surf, uint32_t* changed) {
    bool any = false;
    for (uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; g < totalWords;
         g += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t u = b.nUnits > 1 ? unitOf(b.wordBase, b.nUnits, g) : 0u;
        const PruneView v = pruneView(b, u, solid, fill, surf);
        const uint32_t idx = (uint32_t)(g - __ldg(b.wordBase + u));
        if (idx >= v.nWords) continue;
        const uint32_t w = v.S[idx];
        if (w == 0u) continue;
        const uint32_t plane = v.ipx * v.AY;
        const uint32_t row = v.divX.div(idx), k = idx - row * v.ipx, z = v.divY.div(row), y = row - z * v.AY;
        const uint32_t nw = prunedWord(
            w, k > 0 ? v.S[idx - 1] : 0u, k + 1 < v.ipx ? v.S[idx + 1] : 0u, y > 0 ? v.S[idx - v.ipx] : 0u,
            y + 1 < v.AY ? (v.yLater[y] ? unpruned(v, idx + v.ipx) : v.S[idx + v.ipx]) : 0u,
            z > 0 ? v.S[idx - plane] : 0u,
            z + 1 < v.AZ ? (v.zLater[z] ? unpruned(v, idx + plane) : v.S[idx + plane]) : 0u);
        if (nw != w) {
            v.S[idx] = nw;
            any = true;
        }
    }
    if (any) *changed = 1u;
}

// The words of one unit a kernel reads.
struct UnitWords {
    const uint32_t* fin;
    const uint32_t* fill;
    const uint32_t* surf;     // NULL without materials
    const uint8_t* yLater;
    const uint8_t* zLater;
    uint32_t ipx, AY, AZ, border;
};

// Nodes of word w that zeroPadding (src/voxelizer.cu:4811-4844) clears in a
// device space with neighbours: every node on a face of the allocation.
__device__ __forceinline__ uint32_t borderMask(const UnitWords& u, uint32_t w) {
    if (!u.border) return 0u;
    const uint32_t row = w / u.ipx, k = w - row * u.ipx;
    const uint32_t z = row / u.AY, y = row - z * u.AY;
    if (y == 0 || y + 1 == u.AY || z == 0 || z + 1 == u.AZ) return 0xFFFFFFFFu;
    return (k == 0 ? 0x80000000u : 0u) | (k + 1 == u.ipx ? 1u : 0u);
}

struct EmitArgs {
    Batch b;
    const uint32_t* fin;     // pruned solid arena
    const uint32_t* fill;    // parity fill arena (unpruned)
    const uint32_t* surf;    // surface arena
    const WordRank* ranks;   // surface words with their ranks (arena-wide)
    const void* keys;        // merged material keys by rank
    uint32_t keysCap;        // keys past it read as 0
    const unsigned long long* values;   // PartialNode surface nodes without their ids, by rank
};

__device__ __forceinline__ UnitWords unitWords(const EmitArgs& a, const Unit& U) {
    UnitWords uw;
    uw.fin = a.fin + U.wordBase;
    uw.fill = a.fill + U.wordBase;
    uw.surf = U.materials ? a.surf + U.wordBase : nullptr;
    uw.yLater = a.b.later + U.laterBase;
    uw.zLater = uw.yLater + U.g.AY;
    uw.ipx = U.g.ipx;
    uw.AY = U.g.AY;
    uw.AZ = U.g.AZ;
    uw.border = U.g.border;
    return uw;
}

// Node emission, Cartesian lattices.  Boundary ids follow fillNodeList2 in
// split order: a neighbour in a later yz subspace is read from the unpruned
// grid (its subspace was still unpruned when this one converged), every
// other neighbour from the final grid.  Pruned surface nodes keep their
// material (node.bid(0) keeps mat, include/node_types.h).
struct WordNbrs {
    uint32_t c, s0, f0, L, R, In, Out, Dn, Up;
};

template <int K>
__device__ __forceinline__ WordNbrs loadNbrs(const UnitWords& u, uint32_t w) {
    typedef NodeT<K> NT;
    WordNbrs n;
    n.c = __ldg(u.fin + w);
    n.s0 = u.surf ? __ldg(u.surf + w) : 0u;
    n.f0 = NT::bytes == 8 ? __ldg(u.fill + w) : 0u;
    n.L = n.R = n.In = n.Out = n.Dn = n.Up = 0u;
    if (n.c | n.s0 | n.f0) {
        const uint32_t row = w / u.ipx;
        const uint32_t k = w - row * u.ipx;
        const uint32_t z = row / u.AY, y = row - z * u.AY;
        const uint32_t plane = u.ipx * u.AY;
        const uint32_t prev = k > 0 ? __ldg(u.fin + w - 1) : 0u;
        const uint32_t next = k + 1 < u.ipx ? __ldg(u.fin + w + 1) : 0u;
        n.L = (n.c >> 1) | (prev << 31);
        n.R = (n.c << 1) | (next >> 31);
        n.In = y > 0 ? __ldg(u.fin + w - u.ipx) : 0u;
        if (y + 1 < u.AY)
            n.Out = u.yLater[y] ? (__ldg(u.fill + w + u.ipx) | (u.surf ? __ldg(u.surf + w + u.ipx) : 0u))
                                : __ldg(u.fin + w + u.ipx);
        n.Dn = z > 0 ? __ldg(u.fin + w - plane) : 0u;
        if (z + 1 < u.AZ)
            n.Up = u.zLater[z] ? (__ldg(u.fill + w + plane) | (u.surf ? __ldg(u.surf + w + plane) : 0u))
                               : __ldg(u.fin + w + plane);
    }
    return n;
}

// Boundary ids of the nodes `cm` of a word as five bit planes: plane k holds
// bit k of every node's id.  Along each axis a node has a solid neighbour
// below only (1), above only (2) or on both sides (3); the id is
// kOrientTable[x | y << 2 | z << 4] for those three codes (0 when an axis has
// none), and each plane is the union of the code combinations whose id has
// that bit set, evaluated on whole words at once.
__device__ __forceinline__ void idPlanes(uint32_t L, uint32_t R, uint32_t In, uint32_t Out, uint32_t Dn, uint32_t Up,
                                         uint32_t cm, uint32_t P[5]) {
    const uint32_t X1 = L & ~R, X3 = L & R, Xo = L ^ R, Xa = L | R, X2 = R & ~L;
    const uint32_t Y1 = In & ~Out, Y2 = Out & ~In, Y3 = In & Out, Ya = In | Out;
    const uint32_t Z1 = Dn & ~Up, Z2 = Up & ~Dn, Z3 = Dn & Up, Za = Dn | Up, Zo = Dn ^ Up;
    P[0] = ((Za & ((Y1 & L) | (Y2 & X1))) | (Y3 & ((Dn & L) | (Z2 & X1)))) & cm;
    P[1] = ((Y1 & ((Zo & X2) | (Z3 & R))) | (Za & Y2 & L) | (Y3 & ((Z1 & X1) | (Z2 & L) | (Z3 & X3)))) & cm;
    P[2] = ((Z1 & ((Y2 & X2) | (Y3 & R))) | (Z2 & ((Y1 & Xa) | (Y2 & L) | (Y3 & X1))) | (Z3 & ((Y1 & X3) | (Y2 & R)))) &
           cm;
    P[3] = ((Z1 & (((Y1 | Y2) & X3) | (Y3 & Xo))) | (Z2 & ((Y1 & X3) | (Y2 & R) | (Y3 & L))) | (Z3 & Y3 & Xa)) & cm;
    P[4] = ((Y3 & ((Z1 & X3) | (Z2 & R))) | (Z3 & Ya & Xa)) & cm;
}

// NP <= 8 bit planes as bytes in node order: N[m] holds the bytes of nodes
// 4m .. 4m+3 (node t of a word is bit 31 - t), plane k in bit k.  An 8x8 bit
// transpose in each byte lane of the bit-reversed planes leaves the byte of
// node 8b + i in byte b of row i; 4x4 byte transposes put the nodes in order.
template <int NP> __device__ __forceinline__ void planeBytes(const uint32_t* P, uint32_t N[8]) {
    uint32_t r[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) r[k] = k < NP ? __brev(P[k]) : 0u;
#pragma unroll
    for (int s = 4; s >= 1; s >>= 1) {
        const uint32_t m = s == 4 ? 0x0F0F0F0Fu : s == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if ((k / s) % 2 == 0) {
                const uint32_t t = ((r[k] >> s) ^ r[k + s]) & m;
                r[k + s] ^= t;
                r[k] ^= t << s;
            }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t t0 = __byte_perm(r[4 * h], r[4 * h + 1], 0x5140), t1 = __byte_perm(r[4 * h], r[4 * h + 1], 0x7362);
        const uint32_t t2 = __byte_perm(r[4 * h + 2], r[4 * h + 3], 0x5140),
                       t3 = __byte_perm(r[4 * h + 2], r[4 * h + 3], 0x7362);
        N[h] = __byte_perm(t0, t2, 0x5410);
        N[2 + h] = __byte_perm(t0, t2, 0x7632);
        N[4 + h] = __byte_perm(t1, t3, 0x5410);
        N[6 + h] = __byte_perm(t1, t3, 0x7632);
    }
}

// 1- and 2-byte nodes.  A warp takes 32 consecutive words of a plane, a lane
// one of them, and walks `planes` planes along z: the words of the planes
// below, at and above the current one stay in registers, positions are
// divided out once, and a plane's loads are issued a plane ahead.
//
// Words of one id without surface nodes (none solid, or every node solid with
// six solid neighbours: id 27) are stored at once.  The others, 2-26% of the
// words but spread over a third to all of the chunks, are collected with
// their neighbour words; once 32 are there, a lane takes each: its ids come
// from the bit planes of idPlanes, the materials of its surface nodes from
// the merged keys, which are consecutive by rank.  So the planes, transposes
// and key loads run in full warps.
//
// Bounds: the store of the grid (131 us of the room's 864 MB), then issue of
// integer instructions.  With every lane forming its own word at once the
// room took 371 us (materials 126, ids and neighbours 86), 558 MB of a duct
// 197 us, 143 MB without materials 72 us; with words collected but positions
// and neighbours found per word 328, 172 and 58 us; now 259, 127 and 52 us.
// The plane ahead is only in flight with 64 registers (four blocks per SM):
// with 48 (five) the same code takes 320, 156 and 54 us.
constexpr int kEmitWarps = 8;

constexpr uint32_t kSparse = 4;   // most surface nodes of a sparse word
constexpr uint32_t kSlots = 96;

// The collected words of a warp: those with at most kSparse surface nodes
// from slot 0 on, the others from the last slot down, so that the lanes of a
// group need about as many key loads.  32 of a kind leave together, and a
// step collects 32 at the most: 96 slots hold both.
// a: index | flags << 27, solid, surface, rank of the first surface node;
// b: the neighbour words In, Out, Dn, Up.
struct EmitSlots {
    uint4 a[kSlots], b[kSlots];
};
enum : uint32_t {
    kHasPrev = 1u << 27,    // solid node before the first, after the last
    kHasNext = 1u << 28,
    kNoFirst = 1u << 29,    // first, last node cleared (border words)
    kNoLast = 1u << 30,
    kIndexMask = (1u << 27) - 1u
};

// The nodes of the n <= 32 words in slots [from, from + n) (whole warp).
template <int K>
__device__ __forceinline__ void emitWords(const EmitArgs& args, const EmitSlots& slots, uint32_t from, uint32_t n,
                                          uint32_t* __restrict__ stage, uint8_t* __restrict__ uOut, uint32_t lane) {
    typedef NodeT<K> NT;
    constexpr uint32_t NB = NT::bytes;
    constexpr uint32_t CH = 2 * NB;              // 16-byte chunks of a word
    constexpr uint32_t PITCH = 8 * NB + 4;       // 32-bit words of a padded row
    uint32_t* const row = stage + lane * PITCH;
    uint4 a = make_uint4(0u, 0u, 0u, 0u), b = a;
    if (lane < n) {
        a = slots.a[from + lane];
        b = slots.b[from + lane];
    }
    const uint32_t zero = (a.x & kNoFirst ? 0x80000000u : 0u) | (a.x & kNoLast ? 1u : 0u);
    const uint32_t c = a.y, s0 = a.z;
    {
        uint32_t P[5], N[8];
        idPlanes((c >> 1) | (a.x & kHasPrev ? 0x80000000u : 0u), (c << 1) | (a.x & kHasNext ? 1u : 0u), b.x, b.y, b.z,
                 b.w, c & ~zero, P);
        planeBytes<5>(P, N);
#pragma unroll
        for (int q = 0; q < 8; q += 2) {
            if (NB == 1)
                *reinterpret_cast<uint2*>(row + q) = make_uint2(N[q], N[q + 1]);
            else
                *reinterpret_cast<uint4*>(row + 2 * q) =
                    make_uint4(__byte_perm(N[q], 0u, 0x4140), __byte_perm(N[q], 0u, 0x4342),
                               __byte_perm(N[q + 1], 0u, 0x4140), __byte_perm(N[q + 1], 0u, 0x4342));
        }
    }
    // Four surface nodes per step, so that their key loads are in flight
    // together; keys past keysCap read as 0.
    const uint32_t* const keys = reinterpret_cast<const uint32_t*>(args.keys);
    uint8_t* const my = reinterpret_cast<uint8_t*>(row);
    uint32_t r = a.w + (s0 & zero & 0x80000000u ? 1u : 0u);   // a cleared first node has a key too
    for (uint32_t rest = s0 & ~zero; rest; r += 4) {
        uint32_t bt[4], mat[4];
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            bt[q] = __clz(rest);                 // node index in the word (32: none left)
            rest &= ~(0x80000000u >> (bt[q] & 31u));
            mat[q] = bt[q] < 32u && r + q < args.keysCap ? NT::keyMat(__ldg(keys + r + q)) : 0u;
        }
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            if (bt[q] == 32u) break;
            if (NB == 1) my[bt[q]] |= (uint8_t)(mat[q] << 5);
            else my[2 * bt[q] + 1] = (uint8_t)mat[q];
        }
    }
    __syncwarp();
#pragma unroll
    for (uint32_t k = 0; k < CH; ++k) {
        const uint32_t l = (k * 32u + lane) / CH, q = lane % CH;   // word and 16-byte chunk of it
        const uint32_t w = __shfl_sync(0xffffffffu, a.x & kIndexMask, l);
        if (l < n)
            *reinterpret_cast<uint4*>(uOut + (size_t)w * (32u * NB) + 16u * q) =
                *reinterpret_cast<const uint4*>(stage + l * PITCH + 4u * q);
    }
    __syncwarp();
}

// A task covers a chunk of 32 words (kPacked, one warp) or kEmitWarps of them
// (one block) over `planes` planes.  Tasks are numbered through: along a plane,
// groups of planes, units (taskBase), so that no block of a batch is without
// work whatever its units' shapes (1,000 meshes of 36 planes beside one of 4,098:
// 1,250 us a call with the tallest unit's planes for all, now 227).  Where planes
// are so thin that the warps of a block would idle (emit_packed), tasks are
// warps': 60,002 planes of 7 words 27 us, 58 with blocks; 2,000 meshes of 16-24
// voxels 142 us a call and 178.  One unit of wide planes (kUnit) has its groups
// of planes along the grid's y, which keeps z out of the vector registers: 1-3%
// of a call (room, duct) against a division of the block's number.  They are
// fewer than the 65,535 blocks that y takes: emit_planes leaves at most twice as
// many tasks as blocks share the grid (2 * 148 * 2 * 32 with the widest launch
// shape), or groups of 64 planes, and 65,535 of those with planes this wide (more
// than five chunks) are more words than a grid may have.
enum EmitTasks { kUnit, kBlocks, kPacked };

template <int K, EmitTasks T>
__global__ void __launch_bounds__(kEmitWarps * 32, 4) emitNarrowKernel(EmitArgs a, const uint32_t* __restrict__ taskBase,
                                                                       uint32_t tasks, uint32_t planes,
                                                                       uint32_t zBegin, uint32_t zEnd) {
    typedef NodeT<K> NT;
    static_assert(NT::bytes <= 2, "narrow nodes only");
    constexpr uint32_t NB = NT::bytes;
    constexpr uint32_t CH = 2 * NB;
    constexpr uint32_t kFull = 0xffffffffu;
    __shared__ __align__(16) uint32_t stageAll[kEmitWarps][32 * (8 * NB + 4)];
    __shared__ EmitSlots slotsAll[kEmitWarps];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t task = T == kPacked ? blockIdx.x * kEmitWarps + warp : blockIdx.x;
    if (task >= tasks) return;   // whole warp
    const uint32_t u = T != kUnit && taskBase ? unitOf(taskBase, a.b.nUnits, task) : 0u;
    const Unit& U = a.b.units[u];
    const uint32_t ipx = U.g.ipx, AY = U.g.AY, AZ = U.g.AZ, plane = ipx * AY;
    constexpr uint32_t kSpan = T == kPacked ? 32u : 32u * kEmitWarps;
    uint32_t span = task, group = blockIdx.y;
    if (T != kUnit) {
        const uint32_t perPlane = (plane + kSpan - 1u) / kSpan;
        span -= taskBase ? __ldg(taskBase + u) : 0u;
        group = span / perPlane;
        span -= group * perPlane;
    }
    const uint32_t z0 = zBegin + group * planes, z1 = min(z0 + planes, min(AZ, zEnd));
    const uint32_t first = span * kSpan + (T == kPacked ? 0u : warp * 32u);
    if (z0 >= z1 || first >= plane) return;   // whole warp
    EmitSlots& slots = slotsAll[warp];
    uint32_t* const stage = stageAll[warp];
    uint8_t* const uOut = static_cast<uint8_t*>(U.out);
    const uint32_t* const fin = a.fin + U.wordBase;
    const uint32_t* const fill = a.fill + U.wordBase;
    const uint32_t* const surf = U.materials ? a.surf + U.wordBase : nullptr;
    const WordRank* const ranks = a.ranks + U.wordBase;
    const uint8_t* const zLater = a.b.later + U.laterBase + AY;
    const bool border = U.g.border != 0u;
    // The lane's word (clamped to the plane) and its neighbours: offsets in
    // the plane, and masks for those that do not exist.  Loads need no
    // conditions that way; lanes past the plane are left out of every ballot.
    const uint32_t j = min(first + lane, plane - 1u), y = U.g.divX.div(j), k = j - y * ipx;
    const uint32_t wend = min(plane - first, 32u);
    const uint32_t dead = wend < 32u ? kFull << wend : 0u;
    const uint32_t mPrev = k > 0 ? 1u : 0u, mNext = k + 1 < ipx ? 1u : 0u;   // masks of one bit
    const uint32_t mIn = y > 0 ? kFull : 0u, mOut = y + 1 < AY ? kFull : 0u;
    const uint32_t jIn = y > 0 ? j - ipx : j, jOut = y + 1 < AY ? j + ipx : j;
    const bool outLater = y + 1 < AY && a.b.later[U.laterBase + y];
    const bool anyLater = __any_sync(kFull, outLater);
    // Neighbour words along x are in the next lanes; the first and last lane
    // load theirs.
    const uint32_t jEdge = lane == 0 && k > 0 ? j - 1u : lane == 31 && k + 1 < ipx ? j + 1u : j;
    // Planes of [z0, z1) that lie below a later subspace (at most 64).
    uint64_t later = 0;
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
        const uint32_t z = z0 + 32u * h + lane;
        later |= (uint64_t)__ballot_sync(kFull, z < z1 && z + 1 < AZ && zLater[z]) << (32u * h);
    }
    struct Plane {
        uint32_t In, Out, edge, up;   // `up`: the word of the plane above
    };
    auto load = [&](uint32_t z) {
        const uint32_t* __restrict__ f = fin + (size_t)z * plane;
        Plane p;
        p.In = __ldg(f + jIn);
        p.Out = __ldg(f + jOut);
        p.edge = __ldg(f + jEdge);
        p.up = z + 1 < AZ ? __ldg(f + plane + j) : 0u;
        return p;
    };
    const uint32_t v27 = NB == 1 ? 27u * 0x01010101u : 27u * 0x00010001u;
    uint32_t nSparse = 0, nDense = 0;   // collected words
    uint32_t Dn = z0 > 0 ? __ldg(fin + (size_t)(z0 - 1) * plane + j) : 0u;
    uint32_t c = __ldg(fin + (size_t)z0 * plane + j);
    uint4* out = reinterpret_cast<uint4*>(uOut) + ((size_t)(z0 * plane + first) * CH + lane);
    Plane next = load(z0);
    // Surface words are loaded two planes ahead, so that the rank of a word
    // that has surface nodes can be loaded one plane ahead.
    auto surfAt = [&](uint32_t z) { return surf && z < z1 ? __ldg(surf + (size_t)z * plane + j) : 0u; };
    auto rankAt = [&](uint32_t z, uint32_t word) { return word ? __ldg(&ranks[z * plane + j].rank) : 0u; };
    uint32_t s0 = surfAt(z0), nextS = surfAt(z0 + 1u), rank = rankAt(z0, s0);
    for (uint32_t z = z0; z < z1; ++z, out += (size_t)plane * CH) {
        const Plane p = next;
        const uint32_t w = z * plane + j;
        next = load(min(z + 1, z1 - 1u));
        const uint32_t nextRank = rankAt(z + 1u, nextS), afterS = surfAt(z + 2u);
        uint32_t Out = p.Out & mOut, Up = p.up;
        const uint32_t In = p.In & mIn;
        // Rows and planes that start a later pruning subspace are read from
        // the unpruned grid.
        if (anyLater && outLater) Out = __ldg(fill + (w + ipx)) | (surf ? __ldg(surf + (w + ipx)) : 0u);
        if ((later >> (z - z0)) & 1ull) Up = __ldg(fill + (w + plane)) | (surf ? __ldg(surf + (w + plane)) : 0u);
        uint32_t before = __shfl_up_sync(kFull, c, 1), after = __shfl_down_sync(kFull, c, 1);
        before = (lane == 0 ? p.edge : before) & mPrev;
        after = ((lane == 31 ? p.edge : after) >> 31) & mNext;
        uint32_t zero = 0u, flags = (before ? kHasPrev : 0u) | (after ? kHasNext : 0u);
        if (border) {
            // zeroPadding (src/voxelizer.cu:4811-4844).
            zero = mIn == 0u || mOut == 0u || z == 0 || z + 1 == AZ ? kFull : (mPrev ^ 1u) << 31 | (mNext ^ 1u);
            flags |= (mPrev ? 0u : kNoFirst) | (mNext ? 0u : kNoLast);
        }
        const uint32_t cm = c & ~zero, sm = s0 & ~zero;
        const bool full = (cm & ((c >> 1) | before << 31) & ((c << 1) | after) & In & Out & Dn & Up) == kFull;
        const uint32_t rest = __ballot_sync(kFull, sm != 0u || (cm != 0u && !full)) & ~dead;
        const uint32_t fulls = __ballot_sync(kFull, full);
        if ((rest | dead) == 0u && (fulls == 0u || fulls == kFull)) {
            const uint32_t v = fulls ? v27 : 0u;
#pragma unroll
            for (uint32_t q = 0; q < CH; ++q) out[q * 32u] = make_uint4(v, v, v, v);
        } else {
            // 16-byte chunk q * 32 + lane belongs to word q * (32 / CH) + lane / CH.
            const uint32_t skip = (rest | dead) >> (lane / CH), ones = fulls >> (lane / CH);
#pragma unroll
            for (uint32_t q = 0; q < CH; ++q) {
                const uint32_t v = (ones >> (q * (32u / CH))) & 1u ? v27 : 0u;
                if (!((skip >> (q * (32u / CH))) & 1u)) out[q * 32u] = make_uint4(v, v, v, v);
            }
            if (rest) {
                const uint32_t dense = __ballot_sync(kFull, __popc(s0) > (int)kSparse) & rest;
                if ((rest >> lane) & 1u) {
                    const uint32_t below = laneMaskLt();
                    const uint32_t at = (dense >> lane) & 1u ? kSlots - 1u - nDense - __popc(dense & below)
                                                             : nSparse + __popc(rest & ~dense & below);
                    slots.a[at] = make_uint4(w | flags, c, s0, rank);
                    slots.b[at] = make_uint4(In, Out, Dn, Up);
                }
                nDense += __popc(dense);
                nSparse += __popc(rest & ~dense);
                __syncwarp();
                if (nSparse >= 32u) {
                    nSparse -= 32u;
                    emitWords<K>(a, slots, nSparse, 32u, stage, uOut, lane);
                }
                if (nDense >= 32u) {
                    nDense -= 32u;
                    emitWords<K>(a, slots, kSlots - 32u - nDense, 32u, stage, uOut, lane);
                }
            }
        }
        Dn = c;
        c = p.up;
        s0 = nextS;
        nextS = afterS;
        rank = nextRank;
    }
    // The rest, both kinds together where they fit one group.
    if (nSparse + nDense <= 32u && nDense) {
        if (lane < nDense) {
            slots.a[nSparse + lane] = slots.a[kSlots - 1u - lane];
            slots.b[nSparse + lane] = slots.b[kSlots - 1u - lane];
        }
        __syncwarp();
        nSparse += nDense;
        nDense = 0u;
    }
    if (nSparse) emitWords<K>(a, slots, 0u, nSparse, stage, uOut, lane);
    if (nDense) emitWords<K>(a, slots, kSlots - nDense, nDense, stage, uOut, lane);
}

// Values of PartialNode surface nodes by rank (the node without its id): the
// material of the merged key and the volume ratio cut by its triangle, a few
// hundred operations that a thread per surface node shares out evenly over
// the device.  On entry values[r] is the arena position (word * 32 + node) of
// surface node r.
__global__ void __launch_bounds__(128) partialValuesKernel(Batch b, const unsigned long long* __restrict__ keys,
                                                           const uint32_t* __restrict__ countPtr, uint32_t cap,
                                                           unsigned long long* __restrict__ values) {
    const uint32_t n = min(*countPtr, cap);
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        const unsigned long long key = keys[r], at = values[r];
        const uint32_t u = b.nUnits > 1 ? unitOf(b.wordBase, b.nUnits, (uint64_t)(at >> 5)) : 0u;
        const Unit& U = b.units[u];
        const PassGeom& g = U.g;
        const uint32_t w = (uint32_t)((at >> 5) - U.wordBase), bt = (uint32_t)at & 31u;
        const uint32_t row = g.divX.div(w), z = g.divY.div(row);
        const float ratio = ratio::nodeRatio(U.V, U.I, (uint32_t)key, (uint32_t)(key >> 40),
                                             (int)((w - row * g.ipx) * 32u + bt), (int)(row - z * g.AY), (int)z,
                                             detail::F3{g.mnf[0], g.mnf[1], g.mnf[2]}, g.df);
        values[r] = NodeT<kPartial>::pack(0u, NodeT<kPartial>::keyMat(key), ratio);
    }
}

// 8-byte PartialNodes.  Each lane forms the ids of one word (bit-sliced, as
// for the narrow nodes); the warp's 1,024 nodes are then stored in order, two
// nodes (16 bytes) a lane, with the values of surface nodes loaded by rank.
// The ratio of any other node is 1 where the parity fill is set.
//
// With one thread per word that computed the ratios of its surface nodes, 2-3
// lanes of a warp worked at a time: 4.5 M nodes (36 MB) with 118,463 surface
// nodes took 395 us; now 27 us of values and 14 us of emission.  Sharing the
// ratios out inside blocks of 128 words instead took 75 us (64 words: 90).
__global__ void __launch_bounds__(256) emitPartialKernel(EmitArgs a, uint64_t totalWords, uint32_t zBegin, uint32_t zEnd) {
    typedef NodeT<kPartial> NT;
    __shared__ uint32_t ids[8][32][9];          // 32 ids a word, padded
    __shared__ uint4 masks[8][32];              // surface, surface less cleared nodes, fill, rank
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (uint64_t gbase = ((uint64_t)blockIdx.x * 8u + warp) * 32u; gbase < totalWords;
         gbase += (uint64_t)gridDim.x * 8u * 32u) {
        const uint32_t u = a.b.nUnits > 1 ? unitOf(a.b.wordBase, a.b.nUnits, gbase) : 0u;
        const Unit& U = a.b.units[u];
        // The words of planes [zBegin, zEnd).
        const uint32_t plane = U.g.ipx * U.g.AY, wLo = min(zBegin, U.g.AZ) * plane, nWords = min(zEnd, U.g.AZ) * plane;
        const uint32_t wbase = (uint32_t)(gbase - U.wordBase);
        if (wbase >= nWords || wbase + 32u <= wLo) continue;   // whole warp
        const uint32_t w = wbase + lane, wbeg = wLo > wbase ? wLo - wbase : 0u;
        WordNbrs n{};
        uint32_t zero = 0u;
        if (w >= wLo && w < nWords) {
            const UnitWords uw = unitWords(a, U);
            n = loadNbrs<kPartial>(uw, w);
            zero = borderMask(uw, w);
        }
        const uint32_t cm = n.c & ~zero, sm = n.s0 & ~zero, fm = n.f0 & ~zero;
        uint4* out = reinterpret_cast<uint4*>(U.out) + (size_t)wbase * 16u;
        const uint32_t wend = min(nWords - wbase, 32u);
        if (!__any_sync(0xffffffffu, (cm | sm | fm) != 0u)) {
            for (uint32_t i = wbeg * 16u + lane; i < wend * 16u; i += 32u) out[i] = make_uint4(0u, 0u, 0u, 0u);
            continue;
        }
        {
            uint32_t N[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
            if (cm) {
                uint32_t P[5];
                idPlanes(n.L, n.R, n.In, n.Out, n.Dn, n.Up, cm, P);
                planeBytes<5>(P, N);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) ids[warp][lane][i] = N[i];
        }
        masks[warp][lane] = make_uint4(n.s0, sm, fm, sm ? a.ranks[U.wordBase + w].rank : 0u);
        __syncwarp();
#pragma unroll 4
        for (uint32_t i = wbeg * 16u + lane; i < wend * 16u; i += 32u) {
            const uint32_t l = i >> 4, p = (i & 15u) * 2u;   // word and its first node
            const uint32_t id2 = reinterpret_cast<const uint16_t*>(ids[warp][l])[p >> 1];
            const uint4 m = masks[warp][l];
            uint64_t v[2];
#pragma unroll
            for (uint32_t j = 0; j < 2; ++j) {
                const uint32_t t = p + j;
                // Ranks count every surface node of the word, cleared ones
                // included; ranks past the key array have no value.
                const uint32_t r = m.w + (t ? __popc(m.x >> (32u - t)) : 0u);
                v[j] = NT::pack(0u, 0u, (m.z << t) & 0x80000000u ? 1.0f : 0.0f);
                if (((m.y << t) & 0x80000000u) && r < a.keysCap) v[j] = __ldg(a.values + r);
                v[j] |= (id2 >> (8u * j)) & 255u;
            }
            out[i] = make_uint4((uint32_t)v[0], (uint32_t)(v[0] >> 32), (uint32_t)v[1], (uint32_t)(v[1] >> 32));
        }
        __syncwarp();
    }
}

struct FccArgs {
    Batch b;
    const FccMesh* meshes;
    const uint64_t* pairBase;
    uint32_t nMeshes;
    const uint32_t* fill;
    const uint32_t* surf;
    const WordRank* ranks;
    const void* keys;
    uint32_t keysCap;
    uint32_t raw;   // nodes before the boundaries: id = solid bit, no face clearing
};

// Node emission, FCC lattices (convertToFCCGrid + calculateFCCBoundaries,
// src/voxelizer.cu:1710-1776, 1929-2048).  FCC node (X, y, Z) belongs to
// sub-lattice (X & 1) + 2 * (Z & 1) at voxel (X / 2, y, Z / 2); its id is the
// 12-bit mask of solid FCC neighbours.  The neighbour relation is symmetric,
// so the reference's in-place pass equals this snapshot evaluation.
//
// All 12 neighbours of a word of one sub-lattice lie in words of the other
// three, at the same x or one node beside it, so a lane takes one word and
// forms the 12 bits of its 32 nodes as 12 word planes (24 loads instead of
// up to 24 per node), which are transposed to 16-bit ids.  A pair of lanes
// holds the two words whose nodes alternate along X; a warp's 16 pairs are
// 1,024 consecutive nodes, stored 16 bytes a lane with the materials of
// surface nodes loaded by rank.
//
// Node by node (12 neighbour tests of two loads each, 16 bytes a thread) 8.2 M
// LongFCC nodes (33 MB) took 115 us and 1.7 M ShortFCC nodes 39 us; now 21 and
// 13 us.
template <int K>
__global__ void __launch_bounds__(256) emitFccKernel(FccArgs A, uint64_t totalPairs) {
    typedef NodeT<K> NT;
    constexpr uint32_t NPC = 16 / NT::bytes;      // nodes of a 16-byte chunk
    constexpr uint32_t CPP = 64 / NPC;            // chunks of a pair
    __shared__ __align__(16) uint32_t ids[8][32][18];   // 32 16-bit ids a word, padded
    __shared__ __align__(16) uint4 masks[8][32];        // surface nodes, those not cleared, rank
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t px = lane & 1u;
    for (uint64_t g0 = ((uint64_t)blockIdx.x * 8u + warp) * 16u; g0 < totalPairs; g0 += (uint64_t)gridDim.x * 8u * 16u) {
        // Mesh pair bases are multiples of 16.
        const uint32_t m = A.nMeshes > 1 ? unitOf(A.pairBase, A.nMeshes, g0) : 0u;
        const FccMesh M = A.meshes[m];
        const PassGeom& g = A.b.units[M.unit0].g;
        const uint32_t ipx = g.ipx, AY = g.AY, AZ = g.AZ;
        const uint32_t p0 = (uint32_t)(g0 - __ldg(A.pairBase + m)), nPairs = 2u * AZ * AY * ipx;
        if (p0 >= nPairs) continue;               // padding after the mesh (whole warp)
        const uint32_t pair = p0 + (lane >> 1), last = min(nPairs - p0, 16u);
        uint32_t c = 0u, s0 = 0u, zero = 0u, rank = 0u;
        uint32_t N[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) N[i] = 0u;
        if (pair < nPairs) {
            const uint32_t row = g.divX.div(pair), k = pair - row * ipx;
            const uint32_t Z2 = g.divY.div(row), y = row - Z2 * AY, z = Z2 >> 1, pz = Z2 & 1u;
            auto lattice = [&](uint32_t x1, uint32_t z1) -> const Unit& { return A.b.units[M.unit0 + x1 + 2u * z1]; };
            const Unit& U = lattice(px, pz);
            const uint32_t w = (z * AY + y) * ipx + k;
            s0 = U.materials ? __ldg(A.surf + U.wordBase + w) : 0u;
            c = __ldg(A.fill + U.wordBase + w) | s0;
            if (g.border && !A.raw)
                // zeroPadding of an FCC device space with neighbours
                // (src/voxelizer.cu:4827-4834): two node layers at the x and
                // z faces, one at the y faces.
                zero = y == 0 || y + 1 == AY || z == 0 || z + 1 == AZ
                           ? 0xFFFFFFFFu
                           : (k == 0 ? 0x80000000u : 0u) | (k + 1 == ipx ? 1u : 0u);
            const uint32_t cm = c & ~zero;
            if (s0 & ~zero) rank = A.ranks[U.wordBase + w].rank;
            if (cm && A.raw) {
                const uint32_t P[1] = {cm};
                uint32_t lo[8];
                planeBytes<1>(P, lo);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    N[2 * i] = __byte_perm(lo[i], 0u, 0x4140);
                    N[2 * i + 1] = __byte_perm(lo[i], 0u, 0x4342);
                }
            } else if (cm) {
                const bool xe = px == pz;
                // Rows before and after along y of the neighbours that differ
                // in y (y - xe and y + !xe), planes below and above.
                const bool in = !xe || y > 0, out = xe || y + 1 < AY;
                const bool down = pz != 0u || z > 0, up = pz == 0u || z + 1 < AZ;
                const uint32_t ym = xe ? y - 1 : y, yp = xe ? y : y + 1, zd = pz ? z : z - 1, zu = pz ? z + 1 : z;
                auto word = [&](const Unit& L, bool ok, uint32_t zz, uint32_t yy, uint32_t kk) {
                    if (!ok) return 0u;
                    const uint64_t i = L.wordBase + ((zz * AY + yy) * ipx + kk);
                    return __ldg(A.fill + i) | (L.materials ? __ldg(A.surf + i) : 0u);
                };
                const Unit& LA = lattice(px, 1u - pz);
                const Unit& LB = lattice(1u - px, 1u - pz);
                const Unit& LC = lattice(1u - px, pz);
                uint32_t P[12];
                P[0] = word(LA, down && in, zd, ym, k);
                P[3] = word(LA, down && out, zd, yp, k);
                P[8] = word(LA, up && in, zu, ym, k);
                P[11] = word(LA, up && out, zu, yp, k);
                // The other x parity: X - 1 and X + 1 are the same voxel and
                // the one beside it (the previous for even X, the next for
                // odd X).
                const bool edge = px ? k + 1 < ipx : k > 0;
                const uint32_t kn = px ? k + 1 : k - 1;
                auto sides = [&](const Unit& L, bool ok, uint32_t zz, uint32_t yy, uint32_t& left, uint32_t& right) {
                    const uint32_t same = word(L, ok, zz, yy, k), beside = word(L, ok && edge, zz, yy, kn);
                    left = px ? same : (same >> 1) | (beside << 31);
                    right = px ? (same << 1) | (beside >> 31) : same;
                };
                sides(LB, down, zd, y, P[1], P[2]);
                sides(LC, in, z, ym, P[4], P[5]);
                sides(LC, out, z, yp, P[6], P[7]);
                sides(LB, up, zu, y, P[9], P[10]);
                uint32_t all = cm;
#pragma unroll
                for (int i = 0; i < 12; ++i) {
                    P[i] &= cm;
                    all &= P[i];
                }
                if (all == 0xFFFFFFFFu) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) N[i] = 0x0FFF0FFFu;
                } else {
                    uint32_t lo[8], hi[8];
                    planeBytes<8>(P, lo);
                    planeBytes<4>(P + 8, hi);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        N[2 * i] = __byte_perm(lo[i], hi[i], 0x5140);
                        N[2 * i + 1] = __byte_perm(lo[i], hi[i], 0x7362);
                    }
                }
            }
        }
        uint4* out = reinterpret_cast<uint4*>(M.out) + (size_t)p0 * CPP;
        if (!__any_sync(0xffffffffu, (c & ~zero) != 0u)) {
            for (uint32_t i = lane; i < last * CPP; i += 32u) out[i] = make_uint4(0u, 0u, 0u, 0u);
            continue;
        }
#pragma unroll
        for (int i = 0; i < 16; i += 2)
            *reinterpret_cast<uint2*>(&ids[warp][lane][i]) = make_uint2(N[i], N[i + 1]);
        masks[warp][lane] = make_uint4(s0, s0 & ~zero, rank, 0u);
        __syncwarp();
#pragma unroll 2
        for (uint32_t i = lane; i < last * CPP; i += 32u) {
            const uint32_t l = (i / CPP) * 2u, t0 = (i % CPP) * (NPC / 2u);   // even word's lane, its first node
            uint32_t v[4];
            const uint4 m0 = masks[warp][l], m1 = masks[warp][l + 1];
            uint32_t mat[NPC];
#pragma unroll
            for (uint32_t j = 0; j < NPC; ++j) {
                const uint4& q = j & 1u ? m1 : m0;
                const uint32_t t = t0 + j / 2u, r = q.z + (t ? __popc(q.x >> (32u - t)) : 0u);
                mat[j] = ((q.y << t) & 0x80000000u) && r < A.keysCap
                             ? NT::keyMat(__ldg(reinterpret_cast<const uint32_t*>(A.keys) + r))
                             : 0u;
            }
            const uint16_t* e = reinterpret_cast<const uint16_t*>(ids[warp][l]) + t0;
            const uint16_t* o = reinterpret_cast<const uint16_t*>(ids[warp][l + 1]) + t0;
            if (NT::bytes == 2) {
                const uint2 a2 = *reinterpret_cast<const uint2*>(e), b2 = *reinterpret_cast<const uint2*>(o);
                v[0] = __byte_perm(a2.x, b2.x, 0x5410) | (mat[0] << 12) | (mat[1] << 28);
                v[1] = __byte_perm(a2.x, b2.x, 0x7632) | (mat[2] << 12) | (mat[3] << 28);
                v[2] = __byte_perm(a2.y, b2.y, 0x5410) | (mat[NPC - 4] << 12) | (mat[NPC - 3] << 28);
                v[3] = __byte_perm(a2.y, b2.y, 0x7632) | (mat[NPC - 2] << 12) | (mat[NPC - 1] << 28);
            } else {
                const uint32_t a1 = *reinterpret_cast<const uint32_t*>(e), b1 = *reinterpret_cast<const uint32_t*>(o);
                v[0] = (a1 & 0xFFFFu) | (mat[0] << 16);
                v[1] = (b1 & 0xFFFFu) | (mat[1] << 16);
                v[2] = (a1 >> 16) | (mat[2] << 16);
                v[3] = (b1 >> 16) | (mat[3] << 16);
            }
            out[i] = make_uint4(v[0], v[1], v[2], v[3]);
        }
        __syncwarp();
    }
}

}  // namespace

uint32_t prune_planes(uint64_t totalWords) {
    // Planes per block: as many as leave 8 blocks per SM (a block loads two
    // planes more than it prunes).
    return (uint32_t)std::min<uint64_t>(32, std::max<uint64_t>(1, totalWords / kPruneSpan / (148u * 8u)));
}

uint32_t prune_blocks(const PassGeom& g, uint32_t planes, bool thin) {
    const uint32_t plane = g.ipx * g.AY, spans = (plane + kPruneSpan - 1) / kPruneSpan;
    if (thin != (plane <= kPruneThin)) return 0u;
    return thin ? (plane * g.AZ + kThinThreads - 1) / kThinThreads : spans * ((g.AZ + planes - 1) / planes);
}

void launch_prune(const Batch& b, uint64_t totalWords, const uint32_t* const blockBase[2], const uint32_t blocks[2],
                  uint32_t planes, uint32_t* solid, const uint32_t* fill, const uint32_t* surf, uint32_t passes,
                  unsigned long long* list0, unsigned long long* list1, uint32_t* counts, uint32_t cap,
                  uint32_t escapeAt, uint32_t* overflow, cudaStream_t s, uint32_t* launches) {
    for (int thin = 0; thin < 2; ++thin) {
        if (!blocks[thin]) continue;
        auto kernel = thin ? pruneFirstKernel<true> : pruneFirstKernel<false>;
        kernel<<<blocks[thin], thin ? kThinThreads : kPruneThreads, 0, s>>>(b, blockBase[thin], planes, solid, fill,
                                                                            surf, list0, counts, cap, overflow);
        *launches += 1;
    }
    // Few words change.  Up to 64 K words one cluster takes every list (a launch
    // less: 11.6 us of pruning instead of 13.6 at 128^3); larger grids take
    // pass 1 on the whole device, a thread per 16 words at the most.
    uint32_t first = 1;
    if (totalWords > 65536u) {
        pruneListKernel<<<gridFor((totalWords + 15) / 16, 256, 148u * 8u), 256, 0, s>>>(
            b, solid, fill, surf, list0, counts, list1, counts + 1, cap, overflow);
        *launches += 1;
        first = 2;
    }
    pruneListLoopKernel<<<kLoopBlocks, kLoopThreads, 0, s>>>(b, solid, fill, surf, passes, first, list0, list1,
                                                             counts, cap, escapeAt, overflow);
    *launches += 1;
}

void launch_prune_full(const Batch& b, uint64_t totalWords, uint32_t* solid, const uint32_t* fill,
                       const uint32_t* surf, uint32_t* changed, cudaStream_t s, uint32_t* launches) {
    pruneFullKernel<<<gridFor(totalWords, 256, 148u * 8u), 256, 0, s>>>(b, totalWords, solid, fill, surf, changed);
    *launches += 1;
}

uint32_t emit_tasks(const PassGeom& g, bool packed) {
    const uint32_t span = packed ? 32u : 32u * kEmitWarps;
    return (g.ipx * g.AY + span - 1) / span;
}

bool emit_packed(uint64_t chunkPlanes, uint64_t blockPlanes) {
    // Half again as many warps as chunks.  The same within 2-4 us for 13 chunks
    // on 16 warps (54 us packed, 56 in blocks), 10 on 16 (52, 56) and 4 on 8 (31,
    // 29); 1 on 8 is 27 and 58.
    return 2 * kEmitWarps * blockPlanes > 3 * chunkPlanes;
}

uint32_t emit_planes(uint64_t taskPlanes, bool packed, uint32_t blocksPerSm) {
    // Planes per task: 2 * blocksPerSm blocks per SM share the grid (their work
    // differs, so more of them balance better), but a warp's set-up pays for 8
    // planes where 8 blocks per SM remain.
    const uint64_t blocks = packed ? taskPlanes / kEmitWarps : taskPlanes;
    const uint64_t share = blocks / (148u * 2u * (uint64_t)blocksPerSm), least = std::min<uint64_t>(8, blocks / (148u * 8u));
    return (uint32_t)std::min<uint64_t>(64, std::max<uint64_t>(1, std::max(share, least)));
}

void launch_emit_cartesian(int nodeKind, const Batch& b, uint64_t totalWords, const uint32_t* taskBase, uint32_t tasks,
                           bool packed, uint32_t planes, uint32_t zBegin, uint32_t zEnd, const uint32_t* finalSolid,
                           const uint32_t* fill, const uint32_t* surf, const WordRank* ranks, const void* keys,
                           uint32_t keysCap, const unsigned long long* values, cudaStream_t s, uint32_t* launches) {
    EmitArgs a;
    a.keysCap = keysCap;
    a.b = b;
    a.fin = finalSolid;
    a.fill = fill;
    a.surf = surf;
    a.ranks = ranks;
    a.keys = keys;
    a.values = values;
    if (nodeKind == kPartial) {
        emitPartialKernel<<<gridFor(totalWords, 256, 148u * 64u), 256, 0, s>>>(a, totalWords, zBegin, zEnd);
    } else {
        dim3 grid(packed ? (tasks + kEmitWarps - 1) / kEmitWarps : tasks);
        auto kernel = nodeKind == kShort ? emitNarrowKernel<kShort, kBlocks> : emitNarrowKernel<kLong, kBlocks>;
        if (packed) {
            kernel = nodeKind == kShort ? emitNarrowKernel<kShort, kPacked> : emitNarrowKernel<kLong, kPacked>;
        } else if (!taskBase) {
            const uint32_t groups = (zEnd - zBegin + planes - 1) / planes;
            grid = dim3(tasks /= groups, groups);
            kernel = nodeKind == kShort ? emitNarrowKernel<kShort, kUnit> : emitNarrowKernel<kLong, kUnit>;
        }
        kernel<<<grid, kEmitWarps * 32, 0, s>>>(a, taskBase, tasks, planes, zBegin, zEnd);
    }
    *launches += 1;
}

void launch_partial_values(const Batch& b, const void* keys, const uint32_t* count, uint32_t cap,
                           unsigned long long* values, cudaStream_t s, uint32_t* launches) {
    partialValuesKernel<<<148 * 16, 128, 0, s>>>(b, static_cast<const unsigned long long*>(keys), count, cap, values);
    *launches += 1;
}

void launch_emit_fcc(int nodeKind, const Batch& b, const FccMesh* meshes, const uint64_t* pairBase,
                     uint32_t nMeshes, uint64_t totalPairs, const uint32_t* fill, const uint32_t* surf,
                     const WordRank* ranks, const void* keys, uint32_t keysCap, bool raw, cudaStream_t s,
                     uint32_t* launches) {
    FccArgs A;
    A.keysCap = keysCap;
    A.raw = raw ? 1u : 0u;
    A.b = b;
    A.meshes = meshes;
    A.pairBase = pairBase;
    A.nMeshes = nMeshes;
    A.fill = fill;
    A.surf = surf;
    A.ranks = ranks;
    A.keys = keys;
    const uint32_t grid = gridFor(totalPairs, 8u * 16u, 148u * 64u);
    if (nodeKind == kShortFcc) emitFccKernel<kShortFcc><<<grid, 256, 0, s>>>(A, totalPairs);
    else emitFccKernel<kLongFcc><<<grid, 256, 0, s>>>(A, totalPairs);
    *launches += 1;
}

}  // namespace vxb
