// The voxelization pipeline of one batch (vxb_pipeline.h).
//
// All units of a batch go through each stage in one launch: solid
// voxelization, surface voxelization with its hit list and ranks,
// split-ordered pruning, material merge and node emission.  Pruning queues
// kPasses passes (the later ones over lists of changed words, ending with an
// empty list); the host checks their counts after the batch and adds passes
// only where they had not converged.

#include "vxb_pipeline.h"

#include "vxb_common.cuh"

#include <algorithm>
#include <cstring>

namespace vxb {

namespace {

// Slots of the status buffer; pruning flags follow at kFlags.
// kSolidTotal and kSolidHigh are the low and high word of one 64-bit count.
// kSurfTotal and kSurfHigh likewise; the cursors take two words.
enum : int { kSolidTotal = 0, kSolidHigh = 1, kSurfTotal = 2, kSurfHigh = 3, kSurfCursor = 4, kHitCount = 6,
             kSurfaceVoxels = 7, kSurfQueue = 8, kToggleQueue = 9, kBigCursor = 10,
             kSurfClasses = 12, kRankDone = 15, kPruneOverflow = 16, kPruneCounts = 17 };

// The work counts take 32 bits: totals of 2^32 - 1 or more are refused.
bool countOverflow(const uint32_t* h) { return h[1] || h[0] == 0xFFFFFFFFu; }

const uint32_t kNodeBytes[5] = {1, 2, 8, 2, 4};

bool isFccType(int t) { return t == VXB_SHORT_FCC_NODE || t == VXB_LONG_FCC_NODE; }

size_t align16(size_t v) { return (v + 15) & ~size_t(15); }

template <class T> size_t append(std::vector<uint8_t>& blob, const std::vector<T>& v) {
    const size_t off = align16(blob.size());
    blob.resize(off + v.size() * sizeof(T));
    if (!v.empty()) memcpy(blob.data() + off, v.data(), v.size() * sizeof(T));
    return off;
}

}  // namespace

int gridInfo(const Plan& p, int nodeType, int nodes, vxb_grid_info* info) {
    const bool fcc = isFccType(nodeType);
    vxb_grid_info gi;
    memset(&gi, 0, sizeof(gi));
    if (nodes) {
        gi.dim.x = fcc ? 2 * p.alloc[0] : p.alloc[0];
        gi.dim.y = p.alloc[1];
        gi.dim.z = fcc ? 2 * p.alloc[2] : p.alloc[2];
        gi.count = (uint64_t)gi.dim.x * gi.dim.y * gi.dim.z;
        gi.bytes = gi.count * kNodeBytes[nodeType];
        // The reference indexes nodes with 32-bit unsigned integers.
        if (gi.count > 0xFFFFFFFFull)
            return failf(VXB_EOVERFLOW, "node grid of %llu nodes exceeds 32-bit indexing",
                         (unsigned long long)gi.count);
    } else {
        gi.dim.x = p.alloc[0];
        gi.dim.y = p.alloc[1];
        gi.dim.z = p.alloc[2];
        gi.count = (uint64_t)p.alloc[0] * p.alloc[1] * p.alloc[2] / 32;
        gi.bytes = gi.count * 4;
        if ((uint64_t)p.alloc[0] * p.alloc[1] * p.alloc[2] > 0xFFFFFFFFull)
            return failf(VXB_EOVERFLOW, "voxel grid exceeds 32-bit indexing");
    }
    gi.voxel_length = p.d;
    for (int a = 0; a < 3; ++a) {
        gi.min_vertex[a] = p.mnHost[a];
        gi.max_vertex[a] = p.mx[a];
    }
    for (int k = 0; k < 4; ++k) gi.partition[k] = p.part[k];
    gi.resolution.x = p.res[0];
    gi.resolution.y = p.res[1];
    gi.resolution.z = p.res[2];
    gi.x_splits = p.xSplits;
    if (info) *info = gi;
    return 0;
}

// Shifts of the four FCC sub-lattices by their slot in the FCC array (slot
// 1 + (x & 1) + 2 (z & 1), src/host_side.cpp:1438-1462).  For a turned mesh
// (slices along x) the reference shifts grid g by the z-swapped pattern and
// writes it to slot (g + 1) % 4 + 1, which toggles each slot's y shift.
PassGeom makeGeom(const Plan& p, int lattice, bool turned) {
    const double h = p.d / 2.0;
    const double sh[4][3] = {{0.0, 0.0, 0.0}, {h, h, 0.0}, {0.0, h, h}, {h, 0.0, h}};
    const double shTurned[4][3] = {{0.0, h, 0.0}, {h, 0.0, 0.0}, {0.0, 0.0, h}, {h, h, h}};
    PassGeom g;
    for (int a = 0; a < 3; ++a) {
        g.mn[a] = p.mn[a] + (turned ? shTurned : sh)[lattice][a];
        g.mnf[a] = (float)g.mn[a];
    }
    g.d = p.d;
    g.rd = detail::divReciprocal(p.d);
    g.df = (float)p.d;
    g.rdf = detail::divReciprocalF(g.df);
    g.X = p.res[0];
    g.resY = p.res[1];
    g.resZ = p.res[2];
    g.AY = p.alloc[1];
    g.AZ = p.alloc[2];
    g.ipx = p.res[0] / 32;
    g.padY = p.padY;
    g.padZ = p.padZ;
    g.border = p.border ? 1u : 0u;
    g.divX = FastDiv::of(g.ipx);
    g.divY = FastDiv::of(g.AY);
    return g;
}

void StageTimer::mark(int stage, bool end, cudaStream_t s) {
    if (!enabled) return;
    if (!ev[0])
        for (auto& e : ev) cudaEventCreate(&e);
    cudaEventRecord(ev[2 * stage + (end ? 1 : 0)], s);
    used[stage] = true;
}

StageTimer::~StageTimer() {
    for (auto& e : ev)
        if (e) cudaEventDestroy(e);
}

Batch Pipeline::batch() {
    const uint8_t* t = tables.as<uint8_t>();
    Batch b;
    b.units = reinterpret_cast<const Unit*>(t + oUnits_);
    b.nUnits = (uint32_t)units_.size();
    b.workBase = reinterpret_cast<const uint32_t*>(t + oWork_);
    b.rowBase = reinterpret_cast<const uint64_t*>(t + oRow_);
    b.wordBase = reinterpret_cast<const uint64_t*>(t + oWord_);
    b.splits = reinterpret_cast<const SplitYZ*>(t + oSplits_);
    b.slices = reinterpret_cast<const uint32_t*>(t + oSlices_);
    b.later = t + oLater_;
    return b;
}

int Pipeline::prepare(const std::vector<MeshJob>& jobs, cudaStream_t s) {
    if (jobs.empty()) return failf(VXB_EINVAL, "empty batch");
    jobs_ = jobs;
    nodeKind_ = jobs[0].nodeType;
    nodes_ = jobs[0].nodes;
    for (const MeshJob& j : jobs)
        if (j.nodeType != nodeKind_ || j.nodes != nodes_)
            return failf(VXB_EINVAL, "all meshes of a batch need the same node type and output kind");
    const bool fcc = isFccType(nodeKind_);
    wide_ = nodeKind_ == VXB_PARTIAL_NODE;
    raw_ = jobs[0].raw != 0;
    for (const MeshJob& j : jobs)
        if ((j.raw != 0) != raw_ || (raw_ && !j.nodes))
            return failf(VXB_EINVAL, "raw node output is for node grids of a whole batch");
    units_.clear();
    std::vector<uint32_t> workBase{0};
    std::vector<uint64_t> rowBase{0}, wordBase{0};
    std::vector<SplitYZ> splits;
    std::vector<uint32_t> slices;
    std::vector<uint8_t> later;
    std::vector<FccMesh> fccMeshes;
    std::vector<uint64_t> pairBase{0};
    anyMaterials_ = false;
    anyCartesian_ = false;
    uint64_t nodeCount = 0;
    for (const MeshJob& j : jobs) {
        Plan p;
        const uint32_t vs[3] = {j.req.vox_split_res.x, j.req.vox_split_res.y, j.req.vox_split_res.z};
        const uint32_t ms[3] = {j.req.mat_split_res.x, j.req.mat_split_res.y, j.req.mat_split_res.z};
        if (makePlan(j.mn, j.mx, j.req.by_cube_length, j.req.max_dimension, j.req.cube_length, vs, ms, p))
            return failf(VXB_EINVAL, "invalid request (maxDimension >= 2 or cubeLength > 0, split sizes > 0 and an x "
                                     "pass of at most 1024 voxels are required)");
        if (j.space) {
            Plan full = p;
            if (devicePlan(full, j.part[0], j.part[1], j.part[2], j.part[3], vs, ms, p))
                return failf(VXB_EINVAL, "empty or out-of-range partition");
        }
        vxb_grid_info gi;
        if (int rc = gridInfo(p, j.nodeType, j.nodes, &gi)) return rc;
        if (!j.out) return failf(VXB_EINVAL, "output buffer is NULL");
        if (j.outBytes < gi.bytes)
            return failf(VXB_EINVAL, "output buffer holds %llu bytes, %llu needed", (unsigned long long)j.outBytes,
                         (unsigned long long)gi.bytes);
        nodeCount += gi.count;
        const int lattices = (j.nodes && fcc) ? 4 : 1;
        const uint32_t firstUnit = (uint32_t)units_.size();
        for (int l = 0; l < lattices; ++l) {
            Unit u;
            memset(&u, 0, sizeof(u));
            u.g = makeGeom(p, l, fcc && j.turned);
            u.V = j.V;
            u.I = j.I;
            u.M = j.M;
            u.nT = j.nT;
            u.splitBase = (uint32_t)splits.size();
            for (const auto& z : p.zSplitsExt)
                for (const auto& y : p.ySplitsExt) splits.push_back(SplitYZ{y.lo, y.hi, z.lo, z.hi});
            u.splitN[0] = (uint32_t)p.ySplitsExt.size();
            u.splitN[1] = (uint32_t)p.zSplitsExt.size();
            u.sliceBase = (uint32_t)(slices.size() / 2);
            const std::vector<Range>* axes[3] = {&p.xMat, &p.yMat, &p.zMat};
            for (int a = 0; a < 3; ++a) {
                u.sliceN[a] = (uint32_t)axes[a]->size();
                for (const auto& r : *axes[a]) {
                    slices.push_back(r.lo);
                    slices.push_back(r.hi);
                }
            }
            u.laterBase = (uint32_t)later.size();
            later.resize(later.size() + p.alloc[1] + p.alloc[2], 0);
            for (size_t i = 1; i < p.ySplitsAlloc.size(); ++i) later[u.laterBase + p.ySplitsAlloc[i].lo - 1] = 1;
            for (size_t i = 1; i < p.zSplitsAlloc.size(); ++i)
                later[u.laterBase + p.alloc[1] + p.zSplitsAlloc[i].lo - 1] = 1;
            u.materials = (j.nodes && j.M) ? 1u : 0u;
            anyMaterials_ |= u.materials != 0;
            u.wordBase = wordBase.back();
            u.out = l == 0 ? j.out : nullptr;
            const uint64_t nWords = (uint64_t)u.g.ipx * u.g.AY * u.g.AZ;
            wordBase.push_back(u.wordBase + ((nWords + 31) & ~uint64_t(31)));
            rowBase.push_back(rowBase.back() + (uint64_t)u.g.AY * u.g.AZ);
            if ((uint64_t)workBase.back() + j.nT > 0xFFFFFFFFull)
                return failf(VXB_EOVERFLOW, "batch of more than 2^32 work triangles");
            workBase.push_back(workBase.back() + j.nT);
            units_.push_back(u);
            anyCartesian_ |= j.nodes && !fcc;
        }
        if (j.nodes && fcc) {
            fccMeshes.push_back(FccMesh{firstUnit, j.out});
            pairBase.push_back(pairBase.back() + ((gi.count / 64 + 15) & ~uint64_t(15)));
        }
    }
    nWork_ = workBase.back();
    totalWords_ = wordBase.back();
    totalRows_ = rowBase.back();
    nFcc_ = (uint32_t)fccMeshes.size();
    totalPairs_ = pairBase.back();
    // Blocks of the first pruning pass, of wide and of thin units.
    std::vector<uint32_t> pruneBase[2];
    prunePlanes_ = prune_planes(totalWords_);
    for (int thin = 0; thin < 2; ++thin) {
        uint64_t blocks = 0;
        if (anyCartesian_)
            for (const Unit& u : units_) {
                pruneBase[thin].push_back((uint32_t)blocks);
                blocks += prune_blocks(u.g, prunePlanes_, thin != 0);
                if (blocks > 0x7FFFFFFFull) return failf(VXB_EOVERFLOW, "pruning launch of more than 2^31 blocks");
            }
        pruneBase[thin].push_back((uint32_t)blocks);
        pruneBlocks_[thin] = (uint32_t)blocks;
    }
    // Tasks of the emission.  The planes of a task follow from the launch shape
    // of each run; one unit takes any number, several units a power of two,
    // whose prefixes over the units are laid out here.
    std::vector<uint32_t> emitBase;
    uint64_t taskPlanes[2] = {0, 0};
    maxPlanes_ = 0;
    for (const Unit& u : units_) {
        for (int k = 0; k < 2; ++k) taskPlanes[k] += (uint64_t)emit_tasks(u.g, k != 0) * u.g.AZ;
        maxPlanes_ = std::max(maxPlanes_, u.g.AZ);
    }
    emitPacked_ = emit_packed(taskPlanes[1], taskPlanes[0]);
    taskPlanes_ = taskPlanes[emitPacked_];
    if (anyCartesian_ && units_.size() > 1)
        for (uint32_t level = 0; level < kEmitLevels; ++level) {
            uint64_t tasks = 0;
            for (const Unit& u : units_) {
                emitBase.push_back((uint32_t)tasks);
                tasks += (uint64_t)emit_tasks(u.g, emitPacked_) * ((u.g.AZ + (1u << level) - 1u) >> level);
            }
            emitBase.push_back((uint32_t)tasks);
            emitTasks_[level] = tasks <= 0x7FFFFFFFull ? (uint32_t)tasks : 0u;   // 0: too many for this level
        }
    // A single plain voxelization writes its solid grid straight into the
    // caller's buffer.
    aliasFill_ = !nodes_ && jobs.size() == 1;
    // Tables.
    blob_.clear();
    oUnits_ = append(blob_, units_);
    oWork_ = append(blob_, workBase);
    oRow_ = append(blob_, rowBase);
    oWord_ = append(blob_, wordBase);
    oSplits_ = append(blob_, splits);
    oSlices_ = append(blob_, slices);
    oLater_ = append(blob_, later);
    for (int thin = 0; thin < 2; ++thin) oPrune_[thin] = append(blob_, pruneBase[thin]);
    oEmit_ = append(blob_, emitBase);
    oFcc_ = append(blob_, fccMeshes);
    oPairBase_ = append(blob_, pairBase);
    // Buffers.
    int rc;
    const size_t wordBytes = 4 * (size_t)totalWords_;
    if ((rc = tables.ensure(blob_.size() + 64))) return rc;
    if ((rc = status.ensure(4 * (kPruneCounts + (size_t)kPasses)))) return rc;
    mayList_ = false;
    for (const Unit& u : units_) mayList_ |= solid_may_list(u.g, (uint64_t)u.splitN[0] * u.splitN[1], nWork_);
    if (mayList_ && (rc = bigList.ensure(solid_big_bytes(nWork_, kBigChunks)))) return rc;
    if (!aliasFill_ && (rc = fill.ensure(wordBytes))) return rc;
    if (anyCartesian_ && (rc = fin.ensure(wordBytes))) return rc;
    // Change lists of the pruning passes: the first pass lists every word it
    // changes (a fraction of the boundary words); past the cap the host
    // finishes pruning with full passes.
    pruneCap_ = (uint32_t)std::max<uint64_t>(1u << 16, std::min<uint64_t>(totalWords_ / 4, 0x7FFFFFFFull));
    if (anyCartesian_ && (rc = pruneLists.ensure(2 * 8 * (size_t)pruneCap_))) return rc;
    listCap_ = 0;
    mergeEntries_ = 0;
    keysCap_ = 0;
    if (anyMaterials_) {
        if (!evHiDone_) {
            // Pruning and emission (on the way to the result) run on a stream
            // of the greatest priority, so that their blocks are placed
            // before the merge's when both wait for room on the SMs.
            if ((rc = side_.ensure(false)) || (rc = hi_.ensure(true))) return rc;
            VXB_CUDA(cudaEventCreateWithFlags(&evFork_, cudaEventDisableTiming));
            VXB_CUDA(cudaEventCreateWithFlags(&evSurfBits_, cudaEventDisableTiming));
            VXB_CUDA(cudaEventCreateWithFlags(&evSurfDone_, cudaEventDisableTiming));
            VXB_CUDA(cudaEventCreateWithFlags(&evSolid_, cudaEventDisableTiming));
            VXB_CUDA(cudaEventCreateWithFlags(&evHiDone_, cudaEventDisableTiming));
        }
        if ((rc = sOffsets.ensure(4 * (size_t)nWork_))) return rc;
        if (wide_ && (rc = triOf.ensure(4 * (size_t)nWork_))) return rc;
        if ((rc = surf.ensure(wordBytes))) return rc;
        if ((rc = ranks.ensure(2 * wordBytes))) return rc;
        if ((rc = rankTiles.ensure(4 * surface_rank_sums(totalWords_)))) return rc;
        if ((rc = recs.ensure(kSurfRecBytes * (size_t)nWork_))) return rc;
        if ((rc = depth.ensure(kSurfDepthBytes * (size_t)nWork_))) return rc;
        // Hit list: 8-byte entries (bit position << 24 | key).  PartialNode
        // keys are 64-bit and always take the second traversal.  With the
        // list, the surface voxels are at most its entries.
        if (!wide_) {
            listCap_ = (uint32_t)std::min<uint64_t>(96ull << 20, std::max<uint64_t>(8ull << 20, nodeCount / 12));
            // Entries the merge's non-persistent grid is sized for (more are
            // taken by its blocks' grid-stride loops).
            mergeEntries_ = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(listCap_, nodeCount / 4));
            if ((rc = hitList.ensure((size_t)listCap_ * 8))) return rc;
            keysCap_ = listCap_ + 1;
        } else {
            keysCap_ = (uint32_t)std::min<uint64_t>(totalWords_ * 32 + 1,
                                                     std::max<uint64_t>(1u << 20, totalWords_ * 32 / 16));
        }
        if ((rc = keys.ensure((size_t)keysCap_ * (wide_ ? 8 : 4)))) return rc;
        if (wide_ && (rc = values.ensure((size_t)keysCap_ * 8))) return rc;
    }
    VXB_CUDA(cudaMemcpyAsync(tables.p, blob_.data(), blob_.size(), cudaMemcpyHostToDevice, s));
    return 0;
}

int Pipeline::enqueue(cudaStream_t s, StageTimer* timer) {
    launches = 0;
    const Batch b = batch();
    uint32_t* st = status.as<uint32_t>();
    uint32_t* fillP = aliasFill_ ? static_cast<uint32_t*>(jobs_[0].out) : fill.as<uint32_t>();
    const size_t wordBytes = aliasFill_ ? (size_t)units_[0].g.ipx * units_[0].g.AY * units_[0].g.AZ * 4
                                        : 4 * (size_t)totalWords_;
    // The stream of the stages on the way to the result: `s`, then (with a
    // surface pass) the high-priority stream from pruning on.
    cudaStream_t ps = s;
    auto mark = [&](int stage, bool end) {
        if (timer) timer->mark(stage, end, ps);
    };
    // Launch shapes of this run; tuning trials are timed per kernel (not
    // while a graph is being captured).
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    VXB_CUDA(cudaStreamIsCapturing(s, &cap));
    bucket_ = tuneBucket(nWork_, totalWords_, nodeKind_, anyMaterials_);
    shape = tunePick(bucket_, &trial_, cap == cudaStreamCaptureStatusNone);
    for (bool& u : tuneUsed_) u = false;
    // Work counts, hit count and pruning counts.
    VXB_CUDA(cudaMemsetAsync(st, 0, 4 * (kPruneCounts + (size_t)kPasses), s));
    // The surface pass runs on the side stream beside the solid pass (they
    // share no buffer).  The solid pass is queued behind the surface work, which
    // covers the host time of its launches, and before the ranks.
    cudaStream_t ss = s;
    const bool serial = timer && timer->enabled && timer->serial;
    // Without a hit list (PartialNode keys, or the tuned strategy) the first
    // traversal sets surface bits only and a second one merges every hit at its
    // rank.
    const bool retraverse = wide_ || shape.surfMerge != 0;
    auto surfaceBits = [&]() -> int {
        if (!serial) {
            ss = side_.s;
            VXB_CUDA(cudaEventRecord(evFork_, s));
            VXB_CUDA(cudaStreamWaitEvent(ss, evFork_, 0));
        }
        if (timer) timer->mark(1, false, ss);
        VXB_CUDA(cudaMemsetAsync(surf.p, 0, 4 * (size_t)totalWords_, ss));
        launch_surface_prepare(b, nWork_, reinterpret_cast<unsigned long long*>(st + kSurfCursor),
                               reinterpret_cast<unsigned long long*>(st + kSurfTotal), st + kSurfClasses,
                               sOffsets.as<uint32_t>(), wide_ ? triOf.as<uint32_t>() : nullptr, recs.p, depth.p, ss,
                               &launches);
        if (timer) timer->mark(5, false, ss);
        tuneMark(kKnobSurfaceSpan, false, ss);
        tuneMark(kKnobSurface, false, ss);
        surfaceWork(retraverse ? 2 : 0, ss);
        tuneMark(kKnobSurface, true, ss);
        if (timer) timer->mark(5, true, ss);
        VXB_CUDA(cudaEventRecord(evSurfBits_, ss));
        return 0;
    };
    auto surfaceKeys = [&]() -> int {
        // Ranks, and zeroed material keys by rank.
        launch_surface_rank(surf.as<uint32_t>(), totalWords_, ranks.as<WordRank>(), rankTiles.as<uint32_t>(),
                            st + kRankDone, st + kSurfaceVoxels, keys.p, keysCap_, wide_ ? 1 : 0, ss, &launches);
        if (timer) timer->mark(1, true, ss);
        // Material keys by surface rank (independent of pruning).
        if (timer) timer->mark(4, false, ss);
        if (!retraverse)
            launch_surface_merge(hitList.as<unsigned long long>(), st + kHitCount, listCap_, ranks.as<WordRank>(),
                                 keys.as<uint32_t>(), keysCap_, shape.mergeBlocksPerSm, mergeEntries_, ss, &launches);
        else surfaceWork(1, ss);
        if (wide_)
            launch_partial_values(b, keys.p, st + kSurfaceVoxels, keysCap_, values.as<unsigned long long>(), ss,
                                  &launches);
        tuneMark(kKnobSurfaceSpan, true, ss);
        if (timer) timer->mark(4, true, ss);
        VXB_CUDA(cudaEventRecord(evSurfDone_, ss));
        return 0;
    };
    if (anyMaterials_) {
        if (int rc = surfaceBits()) return rc;
        if (serial)
            if (int rc = surfaceKeys()) return rc;
    }
    // Solid voxelization.
    mark(0, false);
    VXB_CUDA(cudaMemsetAsync(fillP, 0, wordBytes, s));
    tuneMark(kKnobToggle, false, s);
    launch_solid_toggle(b, nWork_, reinterpret_cast<unsigned long long*>(st + kSolidTotal),
                        mayList_ ? bigList.p : nullptr, reinterpret_cast<unsigned long long*>(st + kBigCursor),
                        kBigChunks, fillP, shape.toggleBlocksPerSm, shape.toggleQueue ? st + kToggleQueue : nullptr, s, &launches);
    tuneMark(kKnobToggle, true, s);
    launch_row_fill(b, totalRows_, totalWords_, fillP, s, &launches);
    mark(0, true);
    if (anyMaterials_ && !serial)
        if (int rc = surfaceKeys()) return rc;
    if (!nodes_) {
        if (!aliasFill_)
            for (const Unit& u : units_)
                VXB_CUDA(cudaMemcpyAsync(u.out, fillP + u.wordBase, (size_t)u.g.ipx * u.g.AY * u.g.AZ * 4,
                                         cudaMemcpyDeviceToDevice, s));
        VXB_CUDA(cudaGetLastError());
        return 0;
    }
    // The merge knob is timed on this stream from the join with the surface
    // bits (pruning runs beside the merge) to the join with the merged keys:
    // the merge's cost on the way to emission, not its own duration.
    bool mergeSpan = false;
    // Small grids do not fill the device, so the priority is not worth two
    // event pairs (0.85 M words: 129 us a call without, 136 with; 1.2 M words:
    // 158 either way).
    if (anyMaterials_ && !serial && totalWords_ >= kPriorityWords) {
        VXB_CUDA(cudaEventRecord(evSolid_, s));
        VXB_CUDA(cudaStreamWaitEvent(hi_.s, evSolid_, 0));
        ps = hi_.s;
    }
    // Split-ordered pruning (src/host_side.cpp:1183-1206).
    if (anyCartesian_ && !raw_) {
        if (anyMaterials_) {
            VXB_CUDA(cudaStreamWaitEvent(ps, evSurfBits_, 0));
            tuneMark(kKnobMerge, false, ps);
            mergeSpan = true;
        }
        mark(2, false);
        const uint32_t* const blockBase[2] = {reinterpret_cast<const uint32_t*>(tables.as<uint8_t>() + oPrune_[0]),
                                              reinterpret_cast<const uint32_t*>(tables.as<uint8_t>() + oPrune_[1])};
        launch_prune(b, totalWords_, blockBase, pruneBlocks_, prunePlanes_, fin.as<uint32_t>(), fillP,
                     anyMaterials_ ? surf.as<uint32_t>() : nullptr, kPasses, pruneLists.as<unsigned long long>(),
                     pruneLists.as<unsigned long long>() + pruneCap_, st + kPruneCounts, pruneCap_, kLoopListMax,
                     st + kPruneOverflow, ps, &launches);
        mark(2, true);
    }
    // Join: emission reads the merged keys.
    if (anyMaterials_) {
        if (!mergeSpan) tuneMark(kKnobMerge, false, ps);
        VXB_CUDA(cudaStreamWaitEvent(ps, evSurfDone_, 0));
        tuneMark(kKnobMerge, true, ps);
    }
    // Node emission.
    mark(3, false);
    if (raw_ && anyCartesian_)
        launch_emit_raw(nodeKind_, b, totalWords_, fillP, surf.as<uint32_t>(), ranks.as<WordRank>(), keys.p, keysCap_,
                        values.as<unsigned long long>(), ps, &launches);
    else if (anyCartesian_) {
        tuneMark(kKnobEmit, false, ps);
        if (hostOut_ && units_.size() == 1) {
            // The node array in kOutChunks ranges of planes, each copied to
            // the caller's pinned host buffer on the copy stream as soon as it
            // is written, so the copy of the first ranges overlaps the rest.
            const Unit& u = units_[0];
            const uint64_t planeBytes = hostBytes_ / u.g.AZ;
            for (uint32_t k = 0; k < kOutChunks; ++k) {
                const uint32_t p0 = (uint32_t)((uint64_t)u.g.AZ * k / kOutChunks);
                const uint32_t p1 = (uint32_t)((uint64_t)u.g.AZ * (k + 1) / kOutChunks);
                if (p1 <= p0) continue;
                emitCartesian(p0, p1, ps);
                if (!outEv_[k]) VXB_CUDA(cudaEventCreateWithFlags(&outEv_[k], cudaEventDisableTiming));
                VXB_CUDA(cudaEventRecord(outEv_[k], ps));
                VXB_CUDA(cudaStreamWaitEvent(copyStream_, outEv_[k], 0));
                VXB_CUDA(cudaMemcpyAsync(static_cast<uint8_t*>(hostOut_) + p0 * planeBytes,
                                         static_cast<const uint8_t*>(u.out) + p0 * planeBytes, (p1 - p0) * planeBytes,
                                         cudaMemcpyDeviceToHost, copyStream_));
            }
            hostCopied_ = true;
        } else {
            emitCartesian(0, maxPlanes_, ps);
        }
        tuneMark(kKnobEmit, true, ps);
    }
    if (nFcc_)
        launch_emit_fcc(nodeKind_, b, reinterpret_cast<const FccMesh*>(tables.as<uint8_t>() + oFcc_),
                        reinterpret_cast<const uint64_t*>(tables.as<uint8_t>() + oPairBase_), nFcc_, totalPairs_,
                        fillP, surf.as<uint32_t>(), ranks.as<WordRank>(), keys.p, keysCap_, raw_, ps, &launches);
    mark(3, true);
    if (ps != s) {
        VXB_CUDA(cudaEventRecord(evHiDone_, ps));
        VXB_CUDA(cudaStreamWaitEvent(s, evHiDone_, 0));
    }
    VXB_CUDA(cudaGetLastError());
    return 0;
}

void Pipeline::surfaceWork(int mode, cudaStream_t s) {
    uint32_t* st = status.as<uint32_t>();
    // Few triangles in a small grid: a single wave of blocks (4 per SM of 256
    // threads) instead of four, of which three find no work (128^3: 17.4 us,
    // four waves 22.6).  On large grids the few triangles have many rows, and a
    // wave that stays resident holds up the solid pass (4096 x 256 x 256: 377
    // us a call, with four waves 370).
    const uint32_t blocksPerSm = nWork_ <= kFewTriangles && totalWords_ < kPriorityWords
                                     ? std::min(shape.surfBlocksPerSm, 4u)
                                     : shape.surfBlocksPerSm;
    launch_surface_work(nodeKind_, mode, batch(), recs.p, depth.p, triOf.as<uint32_t>(), sOffsets.as<uint32_t>(),
                        reinterpret_cast<unsigned long long*>(st + kSurfCursor),
                        reinterpret_cast<unsigned long long*>(st + kSurfTotal), surf.as<uint32_t>(),
                        ranks.as<WordRank>(), keys.p, keysCap_, values.as<unsigned long long>(),
                        hitList.as<unsigned long long>(), st + kHitCount, listCap_, blocksPerSm,
                        shape.surfBatch, shape.surfQueue ? st + kSurfQueue : nullptr, s, &launches);
}

void Pipeline::emitCartesian(uint32_t zBegin, uint32_t zEnd, cudaStream_t s) {
    uint32_t planes = emit_planes(taskPlanes_, emitPacked_, shape.emitBlocksPerSm), tasks;
    const uint32_t* base = nullptr;
    if (units_.size() == 1) {
        tasks = emit_tasks(units_[0].g, emitPacked_) * ((zEnd - zBegin + planes - 1) / planes);
    } else {
        uint32_t level = 0;
        while (level + 1 < kEmitLevels && ((2u << level) <= planes || !emitTasks_[level])) ++level;
        planes = 1u << level;
        tasks = emitTasks_[level];
        base = reinterpret_cast<const uint32_t*>(tables.as<uint8_t>() + oEmit_) + level * (units_.size() + 1);
    }
    launch_emit_cartesian(nodeKind_, batch(), totalWords_, base, tasks, emitPacked_, planes, zBegin, zEnd,
                          fin.as<uint32_t>(), fill.as<uint32_t>(), surf.as<uint32_t>(), ranks.as<WordRank>(), keys.p,
                          keysCap_, values.as<unsigned long long>(), s, &launches);
}

// Full passes until nothing changes, with a host check after each.
int Pipeline::pruneUntilStable(cudaStream_t s) {
    const Batch b = batch();
    uint32_t* changed = status.as<uint32_t>() + kPruneOverflow;
    for (uint64_t round = 0;; ++round) {
        if (round > (1u << 24)) return failf(VXB_ETIMEDOUT, "pruning did not converge");
        uint32_t h = 0;
        VXB_CUDA(cudaMemsetAsync(changed, 0, 4, s));
        launch_prune_full(b, totalWords_, fin.as<uint32_t>(), fill.as<uint32_t>(),
                          anyMaterials_ ? surf.as<uint32_t>() : nullptr, changed, s, &launches);
        VXB_CUDA(cudaMemcpyAsync(&h, changed, 4, cudaMemcpyDeviceToHost, s));
        VXB_CUDA(cudaStreamSynchronize(s));
        if (!h) return 0;
    }
}

Pipeline::~Pipeline() {
    for (cudaEvent_t e : {evFork_, evSurfBits_, evSurfDone_, evSolid_, evHiDone_})
        if (e) cudaEventDestroy(e);
    for (cudaEvent_t& e : tuneEv_)
        if (e) cudaEventDestroy(e);
    for (cudaEvent_t& e : outEv_)
        if (e) cudaEventDestroy(e);
}

void Pipeline::tuneMark(int knob, bool end, cudaStream_t s) {
    if (trial_ < 0) return;
    cudaEvent_t& e = tuneEv_[2 * knob + (end ? 1 : 0)];
    if (!e && cudaEventCreate(&e) != cudaSuccess) {
        cudaGetLastError();
        e = nullptr;
        return;
    }
    cudaEventRecord(e, s);
    if (end) tuneUsed_[knob] = true;
}

// Reports the kernel times of a tuning trial (the stream has drained).
void Pipeline::tuneFinish() {
    if (trial_ < 0) return;
    float ms[kKnobs];
    for (int k = 0; k < kKnobs; ++k) {
        ms[k] = -1.0f;
        if (tuneUsed_[k] && tuneEv_[2 * k] && tuneEv_[2 * k + 1] &&
            cudaEventElapsedTime(&ms[k], tuneEv_[2 * k], tuneEv_[2 * k + 1]) != cudaSuccess) {
            cudaGetLastError();
            ms[k] = -1.0f;
        }
    }
    tuneReport(bucket_, trial_, ms);
    trial_ = -1;
}

int Pipeline::finish(cudaStream_t s) {
    keysMoved_ = false;
    if (!nodes_) {
        VXB_CUDA(cudaStreamSynchronize(s));
        tuneFinish();
        uint32_t h[2];
        VXB_CUDA(cudaMemcpy(h, status.p, sizeof(h), cudaMemcpyDeviceToHost));
        if (countOverflow(h + kSolidTotal)) return failf(VXB_EOVERFLOW, "solid work list exceeds 2^32 entries");
        return 0;
    }
    uint32_t h[kPruneCounts + kPasses];
    VXB_CUDA(cudaMemcpyAsync(h, status.p, sizeof(h), cudaMemcpyDeviceToHost, s));
    VXB_CUDA(cudaStreamSynchronize(s));
    tuneFinish();
    memset(&stats, 0, sizeof(stats));
    stats.units = (uint32_t)units_.size();
    stats.work_triangles = nWork_;
    stats.solid_candidates = h[kSolidTotal];
    stats.surface_columns = anyMaterials_ ? h[kSurfTotal] : 0;
    stats.surface_hits = anyMaterials_ ? h[kHitCount] : 0;
    stats.surface_voxels = anyMaterials_ ? h[kSurfaceVoxels] : 0;
    for (uint32_t k = 0; k < 3; ++k) stats.surface_triangles[k] = h[kSurfClasses + k];
    stats.grid_words = totalWords_;
    if (countOverflow(h + kSolidTotal) || countOverflow(h + kSurfTotal))
        return failf(VXB_EOVERFLOW, "work list exceeds 2^32 entries");
    bool reemit = false;
    const Batch b = batch();
    uint32_t* st = status.as<uint32_t>();
    uint32_t* fillP = aliasFill_ ? static_cast<uint32_t*>(jobs_[0].out) : fill.as<uint32_t>();
    if (anyMaterials_) {
        const uint32_t hits = h[kHitCount], surfaceVoxels = h[kSurfaceVoxels];
        const bool listOverflow = !wide_ && hits > listCap_;
        if (listOverflow || (uint64_t)surfaceVoxels + 1 > keysCap_) {
            // Merge every hit straight at its rank (second traversal).
            int rc;
            if ((uint64_t)surfaceVoxels + 1 > keysCap_) {
                // Without room (cap 0) until both buffers are there: a run
                // after a failed one then stores no keys.
                keysMoved_ = true;
                keysCap_ = 0;
                if ((rc = keys.ensure(((size_t)surfaceVoxels + 1) * (wide_ ? 8 : 4)))) return rc;
                if (wide_ && (rc = values.ensure(((size_t)surfaceVoxels + 1) * 8))) return rc;
                keysCap_ = surfaceVoxels + 1;
            }
            launch_surface_keys_zero(keys.p, st + kSurfaceVoxels, keysCap_, wide_ ? 1 : 0, s, &launches);
            surfaceWork(1, s);
            if (wide_)
                launch_partial_values(b, keys.p, st + kSurfaceVoxels, keysCap_, values.as<unsigned long long>(), s,
                                      &launches);
            reemit = true;
        }
    }
    if (anyCartesian_ && !raw_) {
        // A change list that overflowed, or a last queued pass that still
        // changed something.
        if (h[kPruneOverflow] || h[kPruneCounts + kPasses - 1]) {
            if (int rc = pruneUntilStable(s)) return rc;
            reemit = true;
        }
    }
    if (reemit) {
        if (raw_ && anyCartesian_)
            launch_emit_raw(nodeKind_, b, totalWords_, fillP, surf.as<uint32_t>(), ranks.as<WordRank>(), keys.p,
                            keysCap_, values.as<unsigned long long>(), s, &launches);
        else if (anyCartesian_)
            emitCartesian(0, maxPlanes_, s);
        if (nFcc_)
            launch_emit_fcc(nodeKind_, b, reinterpret_cast<const FccMesh*>(tables.as<uint8_t>() + oFcc_),
                            reinterpret_cast<const uint64_t*>(tables.as<uint8_t>() + oPairBase_), nFcc_,
                            totalPairs_, fillP, surf.as<uint32_t>(), ranks.as<WordRank>(), keys.p, keysCap_, raw_, s,
                            &launches);
        VXB_CUDA(cudaGetLastError());
        VXB_CUDA(cudaStreamSynchronize(s));
        if (hostCopied_) {
            // The chunks already copied predate the re-emission.
            VXB_CUDA(cudaStreamSynchronize(copyStream_));
            VXB_CUDA(cudaMemcpy(hostOut_, units_[0].out, hostBytes_, cudaMemcpyDeviceToHost));
        }
    }
    return 0;
}

}  // namespace vxb
