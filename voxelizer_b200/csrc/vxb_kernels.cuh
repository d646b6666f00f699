// Kernel declarations and the plain structs the host engine passes to them.
//
// Every kernel works on a batch of units.  A unit is one mesh voxelized on
// one lattice (a Cartesian mesh is one unit, an FCC mesh four: one per
// shifted sub-lattice).  The batch concatenates what its units need into
// shared arrays: work triangles (the units' triangle lists back to back, so
// an FCC mesh's triangles appear once per sub-lattice), bit-grid words (each
// unit's grids start at a multiple of 32 words), subspace tables and flags.
// Meshes stay in their own device arrays.  A single voxelization is a batch
// of one mesh.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace vxb {

// Division of word and row numbers below 2^27 (a grid holds fewer than 2^32
// voxels) by a constant d: with 2^L >= d, m = floor(2^(27 + L) / d) + 1
// exceeds the exact reciprocal by less than 2^-27 of itself, so n * m >> (27 +
// L) is n / d for n < 2^27 (Granlund and Montgomery 1994).  mul holds m << 4,
// which leaves a shift of L - 1 after the high word; d = 1 has mul 0.
struct FastDiv {
    uint32_t mul, shift;
    static FastDiv of(uint32_t d) {
        FastDiv f{0u, 0u};
        if (d <= 1u) return f;
        uint32_t L = 1;
        while (L < 27u && (1u << L) < d) ++L;
        f.mul = (uint32_t)(((1ull << (27 + L)) / d + 1ull) << 4);
        f.shift = L - 1u;
        return f;
    }
#ifdef __CUDACC__
    __device__ __forceinline__ uint32_t div(uint32_t n) const { return mul ? __umulhi(n, mul) >> shift : n; }
#endif
};

// Geometry of one unit.  For FCC lattices each of the four sub-lattices has
// its own shifted minimum corner.
struct PassGeom {
    double mn[3];        // minimum corner (FP64, as the reference's extMinVertex)
    double d;            // voxel length
    double rd;           // 1 / d, or 0 (divBy)
    float mnf[3];        // float(mn) for the FP32 surface path
    float df;            // float(d)
    float rdf;           // 1 / df, or 0 (divByF)
    uint32_t X;          // voxels along x (padded and rounded to 32 * xSplits)
    uint32_t resY, resZ; // voxels along y / z before the 1-voxel padding
    uint32_t AY, AZ;     // allocated rows: resY + 2, resZ + 2
    uint32_t ipx;        // 32-bit words per row: X / 32
    uint32_t padY, padZ; // allocation row / plane of local voxel row / plane 0 (1, or 0 next to a neighbour)
    uint32_t border;     // zero the allocation's faces in the node output (a device space with neighbours)
    FastDiv divX, divY;  // by ipx and by AY
};

struct SplitYZ { uint32_t y0, y1, z0, z1; };

struct Unit {
    PassGeom g;
    const float* V;       // the mesh: vertices (3 floats each),
    const uint32_t* I;    // indices into V (3 per triangle),
    const uint8_t* M;     // material per triangle (NULL without materials)
    uint32_t nT;          // triangles of the mesh
    uint32_t splitBase;   // solid yz subspaces: splitN[0] * splitN[1] SplitYZ entries, y inner
    uint32_t splitN[2];   // subspaces along y, along z
    uint32_t sliceBase;   // material subspace slices: (lo, hi) pairs, x then y then z
    uint32_t sliceN[3];
    uint32_t laterBase;   // AY + AZ flags: row y + 1 / plane z + 1 starts a later pruning subspace
    uint32_t materials;   // surface pass and material output enabled
    uint64_t wordBase;    // first word of the unit's bit grids (a multiple of 32)
    void* out;            // node output (Cartesian units)
};

// A surface word and the rank of its first surface voxel (the exclusive
// popcount prefix of the surface words before it, arena-wide), side by side
// so that one 8-byte load gives both.
struct __align__(8) WordRank {
    uint32_t bits, rank;
};

// Device tables of a batch.  Bases have nUnits + 1 entries (the last one is
// the total), so that the unit of an element is a binary search away.
struct Batch {
    const Unit* units;
    uint32_t nUnits;
    const uint32_t* workBase;   // first work triangle of each unit
    const uint64_t* rowBase;    // first grid row (y, z) of each unit
    const uint64_t* wordBase;   // first grid word of each unit
    const SplitYZ* splits;
    const uint32_t* slices;
    const uint8_t* later;
};

// Exclusive offsets (n + 1 entries) and the grand total of n counts
// (vxb_scan_counts).
void launch_scan(const uint32_t* in, uint32_t* offsets, uint32_t n, uint32_t* blockSums, uint32_t* total,
                 uint32_t* overflow, cudaStream_t s, uint32_t* launches);

// ---- Solid (parity) voxelization: src/voxelizer.cu:840-1617 ----
// The toggles of every candidate into the `fill` arena, then the row prefix
// XOR over all rows of the batch.  *total (zero on entry) receives the number
// of candidates.  `big` (solid_big_bytes; *cursor zero on entry) lists the batches
// of triangles with very many candidates, and the first listCap chunks of them
// one by one; it may be NULL where solid_may_list answers false for every unit,
// and the call then takes one launch instead of two.
// blocksPerSm: launch shape (the autotuner's choice; results do not depend
// on it), here and in the launchers below that take one.  queue: NULL for
// a fixed grid-stride order, else a device word the launcher zeroes and the
// kernel's warps take batches of work from.
bool solid_may_list(const PassGeom& g, uint64_t nSplits, uint32_t nWork);
size_t solid_big_bytes(uint32_t nWork, uint32_t listCap);
void launch_solid_toggle(const Batch& b, uint32_t nWork, unsigned long long* total, void* big,
                         unsigned long long* cursor, uint32_t listCap, uint32_t* fill, uint32_t blocksPerSm,
                         uint32_t* queue, cudaStream_t s, uint32_t* launches);
void launch_row_fill(const Batch& b, uint64_t nRows, uint64_t totalWords, uint32_t* fill, cudaStream_t s,
                     uint32_t* launches);

// ---- Surface voxelization: src/voxelizer.cu:2358-2989, 3040-4201 ----
// Triangles with surface work get consecutive positions (ordered by (class,
// axis) inside each block of the set-up kernel), each with a kSurfRecBytes
// record and, for 3D boxes, a kSurfDepthBytes one.
constexpr uint32_t kSurfaceBuckets = 9;
constexpr size_t kSurfRecBytes = 80;
constexpr size_t kSurfDepthBytes = 112;

// Classification and set-up of the work triangles of units with materials:
// records, first work unit per position (offsets), mesh triangle per position
// (triOf, may be NULL).  *cursor, *total (the exact number of columns) and
// classes[0..3) (triangles per class) are zero on entry.
void launch_surface_prepare(const Batch& b, uint32_t nWork, unsigned long long* cursor, unsigned long long* total,
                            uint32_t* classes, uint32_t* offsets, uint32_t* triOf, void* recs, void* depth,
                            cudaStream_t s, uint32_t* launches);
// Surface work over what launch_surface_prepare wrote, a lane per row of up to
// 32 columns and then a lane per column that passes.
// mode 0: set bits in the `surf` arena and append (bit position << 24 | key)
// to `list` (entries past listCap are counted, not stored); mode 1: merge
// every hit's key at its rank (needs complete bits and their `ranks`) and, for
// PartialNodes (64-bit keys), store its arena position in `positions`; mode 2:
// set bits only.  kind: the node type, whose instantiation of the class
// kernels the arithmetic follows.  batch: chunks of 32 columns a warp takes at
// a time (four make a chunk of 32 rows).  queue: as for launch_solid_toggle.  Nothing is done when *total is
// 2^32 - 1 or more.
void launch_surface_work(int kind, int mode, const Batch& b, const void* recs, const void* depth, const uint32_t* triOf,
                         const uint32_t* offsets, const unsigned long long* cursor, const unsigned long long* total,
                         uint32_t* surf, const WordRank* ranks, void* keys, uint32_t keysCap,
                         unsigned long long* positions, unsigned long long* list, uint32_t* listCount,
                         uint32_t listCap, uint32_t blocksPerSm, uint32_t batch, uint32_t* queue, cudaStream_t s,
                         uint32_t* launches);
// Exclusive popcount prefix over `words` surface words, stored beside each
// word (words of sectors without surface nodes are left out); *total = surface
// voxels; the keys of all of them (at most keysCap) are zeroed.  *done is zero
// on entry; `sums` has room for surface_rank_sums(words) entries.
size_t surface_rank_sums(uint64_t words);
void launch_surface_rank(const uint32_t* bits, uint64_t words, WordRank* ranks, uint32_t* sums, uint32_t* done,
                         uint32_t* total, void* keys, uint32_t keysCap, int wide, cudaStream_t s, uint32_t* launches);
// Zeroes min(*count, cap) keys.
void launch_surface_keys_zero(void* keys, const uint32_t* count, uint32_t cap, int wide, cudaStream_t s,
                              uint32_t* launches);
// Keys at ranks >= keysCap are dropped (the host re-merges after growing).
// blocksPerSm 0 sizes the grid for `entries` entries, a block per 1,024
// (non-persistent).
void launch_surface_merge(const unsigned long long* list, const uint32_t* listCount, uint32_t listCap,
                          const WordRank* ranks, uint32_t* keys, uint32_t keysCap,
                          uint32_t blocksPerSm, uint32_t entries, cudaStream_t s, uint32_t* launches);

// Mesh checks of vxb_create (vxb_meshcheck.cu): hostOut[0..2] / [3..5]
// name the first vertex (after vertex 0) holding the smallest / largest
// non-NaN coordinate per axis as (order code << 32 | vertex), ~0 if none;
// hostOut[6] is the largest index, hostOut[7] the first position of an
// index >= nV (~0 if none).  Synchronizes `s`.
int meshCheck(const float* dV, uint32_t nV, const uint32_t* dI, uint64_t nIdx, unsigned long long* dOut,
              unsigned long long* hostOut, cudaStream_t s);

// ---- Node classification: src/voxelizer.cu:1626-2048 ----
// Pruning of every unit (Cartesian node grids): `solid` from fill | surf
// (surf may be NULL).  counts[p], p < passes, is the length of pass p's
// change list and *overflow a flag, all zero on entry.  Pass 0 goes over all
// words, pass 1 over the words it changed (list0), the others in one cluster
// with alternating lists of at most `cap` (unit << 32 | word) entries.
// blockBase[k]: exclusive prefix over the units of prune_blocks for thin = k
// (nUnits + 1 entries) and `planes` = prune_planes(totalWords); blocks[k] is their
// sum.  The grid is pruned unless counts[passes - 1] or *overflow is set (a list
// longer than cap or, after pass 1, than escapeAt): then launch_prune_full passes,
// which set *changed, finish it.
uint32_t prune_planes(uint64_t totalWords);
uint32_t prune_blocks(const PassGeom& g, uint32_t planes, bool thin);
void launch_prune(const Batch& b, uint64_t totalWords, const uint32_t* const blockBase[2], const uint32_t blocks[2],
                  uint32_t planes, uint32_t* solid, const uint32_t* fill, const uint32_t* surf, uint32_t passes,
                  unsigned long long* list0, unsigned long long* list1, uint32_t* counts, uint32_t cap,
                  uint32_t escapeAt, uint32_t* overflow, cudaStream_t s, uint32_t* launches);
void launch_prune_full(const Batch& b, uint64_t totalWords, uint32_t* solid, const uint32_t* fill,
                       const uint32_t* surf, uint32_t* changed, cudaStream_t s, uint32_t* launches);
// Slices along x (vxb_xslice.cu): vertex rotation, the node array before
// the boundary ids, un-rotation, one in-place boundary-id pass over a yz
// subspace (sets *changed when a node loses its id) and face zeroing.  The
// node kernels treat nodes as `nodeBytes` bytes with the id in byte 0
// (masked by idMask).
void launch_rotate_vertices(const float* V, float* R, uint32_t n, double a, double b, cudaStream_t s,
                            uint32_t* launches);
void launch_emit_raw(int nodeKind, const Batch& b, uint64_t totalWords, const uint32_t* fill, const uint32_t* surf,
                     const WordRank* ranks, const void* keys, uint32_t keysCap, const unsigned long long* values,
                     cudaStream_t s, uint32_t* launches);
void launch_unrotate(const void* in, void* out, uint32_t X, uint32_t Y, uint32_t Z, uint32_t nodeBytes,
                     cudaStream_t s, uint32_t* launches);
void launch_id_pass(void* nodes, uint32_t X, uint32_t Y, uint32_t Z, uint32_t nodeBytes, uint32_t idMask,
                    uint32_t y0, uint32_t y1, uint32_t z0, uint32_t z1, uint32_t* changed, cudaStream_t s,
                    uint32_t* launches);
void launch_zero_faces(void* nodes, uint32_t X, uint32_t Y, uint32_t Z, uint32_t nodeBytes, bool fcc, cudaStream_t s,
                       uint32_t* launches);
// FCC lattices: unRotateNodes' FCC branch (X x Y x Z -> 2Y x X/2 x Z) and
// calculateFCCBoundaries in place.
void launch_unrotate_fcc(const void* in, void* out, uint32_t X, uint32_t Y, uint32_t Z, uint32_t nodeBytes,
                         cudaStream_t s, uint32_t* launches);
void launch_fcc_boundaries(void* nodes, uint32_t X, uint32_t Y, uint32_t Z, uint32_t nodeBytes, cudaStream_t s,
                           uint32_t* launches);
// PartialNodes: values[r] (cap entries) from the arena position of surface
// node r to its node without the id, for r < min(*count, cap).
void launch_partial_values(const Batch& b, const void* keys, const uint32_t* count, uint32_t cap,
                           unsigned long long* values, cudaStream_t s, uint32_t* launches);
// Keys (PartialNodes: values) at ranks >= keysCap read as 0.
// Planes [zBegin, zEnd) of every unit.  1- and 2-byte nodes: a task is a span of
// a plane's words (emit_tasks in a plane; packed: of one warp, else of a block)
// over `planes` planes, at most 64; emit_planes gives that number from the tasks
// of all single planes of all units, emit_packed the kind of task from those of
// both kinds.  `tasks` is the number of tasks and taskBase their exclusive prefix
// over the units (nUnits + 1 entries; NULL for one unit).
constexpr uint32_t kEmitLevels = 7;   // planes 1, 2, .. 64
uint32_t emit_tasks(const PassGeom& g, bool packed);
bool emit_packed(uint64_t chunkPlanes, uint64_t blockPlanes);
uint32_t emit_planes(uint64_t taskPlanes, bool packed, uint32_t blocksPerSm);
void launch_emit_cartesian(int nodeKind, const Batch& b, uint64_t totalWords, const uint32_t* taskBase, uint32_t tasks,
                           bool packed, uint32_t planes, uint32_t zBegin, uint32_t zEnd, const uint32_t* finalSolid,
                           const uint32_t* fill, const uint32_t* surf, const WordRank* ranks, const void* keys,
                           uint32_t keysCap, const unsigned long long* values, cudaStream_t s, uint32_t* launches);

// An FCC mesh: its four sub-lattice units are units [unit0, unit0 + 4).
struct FccMesh {
    uint32_t unit0;
    void* out;
};
// FCC node grids; pairBase[m] is the first pair of words (64 nodes of a row)
// of mesh m, a multiple of 16 (nMeshes + 1 entries).  raw: the nodes before calculateFCCBoundaries (id =
// solid bit, the surface material), for slices along x.
void launch_emit_fcc(int nodeKind, const Batch& b, const FccMesh* meshes, const uint64_t* pairBase,
                     uint32_t nMeshes, uint64_t totalPairs, const uint32_t* fill, const uint32_t* surf,
                     const WordRank* ranks, const void* keys, uint32_t keysCap, bool raw, cudaStream_t s,
                     uint32_t* launches);

}  // namespace vxb
