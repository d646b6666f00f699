"""Performance cases: the voxelizations that programs run through the public
Python interface (``Voxelizer``, ``VoxelizerBatch``), with seeded meshes.

A case names one call (``op``):

* ``nodes``  node grid into a device buffer of the caller (Voxelizer.voxelize_device)
* ``bits``   plain solid bit array into a device buffer
* ``slice``  one slice's node array into a device buffer
* ``parts``  devConfig partitions, one host array each (voxelizePartsToRAM)
* ``batch``  many meshes in one VoxelizerBatch, replayed as a CUDA graph
* ``host``   a voxelizer built from host arrays and its node grid in host
             memory (the constructor plus voxelizeToNodesToRAM)

``mesh`` is ``ico`` (subdivision ``a``), ``torus`` (``a`` x ``b`` segments),
``room`` (``a`` objects in a box shell) or ``stress`` (an icosphere with ``a``
slivers and ``b`` triangles snapped to voxel centres and faces).  Closed
meshes are turned by a random rotation and scaled to a bounding box of
1 x ``ay`` x ``az``.  ``dim`` is the number of voxels along the longest axis;
with ``cube`` the request names the voxel length instead (FCC lattices take
nothing else).  ``mats`` is the number of materials (0: none).
"""

import functools
import math

import numpy as np
import torch

from voxelizer_b200 import api, scenes

SHORT, LONG, PARTIAL, SHORT_FCC, LONG_FCC = api.SHORT, api.LONG, api.PARTIAL, api.SHORT_FCC, api.LONG_FCC
MAX_MATS = {SHORT: 7, LONG: 255, PARTIAL: 255, SHORT_FCC: 15, LONG_FCC: 255}
TORCH_TYPE = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}
NUMPY_TYPE = {1: np.uint8, 2: np.int16, 4: np.int32, 8: np.int64}
MAX_NODES = 432_000_000          # nodes of the largest grid (the full room)
MAX_BYTES = 864_000_000


def _case(name, op, mesh, a, b, dim, node=LONG, mats=0, ay=1.0, az=1.0, cube=False, vox=512, mat=512, vox_x=1024,
          direction=0, dev_y=1, dev_z=1):
    c = {"op": op, "mesh": mesh, "a": a, "b": b, "dim": dim, "node": node, "mats": mats, "ay": ay, "az": az,
         "cube": cube, "vox": vox, "mat": mat, "vox_x": vox_x, "direction": direction, "dev_y": dev_y, "dev_z": dev_z}
    return {"name": name, **c} if name else c


def listed():
    return [
        # The smallest calls: a coarse occupancy grid of a small part, as an
        # interactive tool asks for again and again.  Latency only.
        _case("bits_32", "bits", "torus", 24, 12, 32, ay=0.9, az=0.5),
        # One closed object at edge 1/128 with a material, 1-byte nodes: the
        # plain single-mesh configuration.
        _case("short_ico4_128", "nodes", "ico", 4, 0, 102, SHORT, mats=1, cube=True),
        # An FCC lattice of the tie-breaking stress mesh (slivers and snapped
        # vertices): the degenerate input that CAD exports bring.
        _case("sfcc_stress", "nodes", "stress", 10_000, 5_000, 64, SHORT_FCC, mats=3, cube=True),
        # A long duct: a 16:1 object at 4096 voxels along x, which skews the
        # work lists and passes the x split size four times over.
        _case("long_duct_4096", "nodes", "ico", 4, 0, 4096, LONG, mats=1, ay=1 / 16, az=1 / 16),
        # Volume ratios (8-byte nodes), as a boundary-conforming solver reads
        # them, of one object with several materials.
        _case("partial_torus_210", "nodes", "torus", 256, 128, 210, PARTIAL, mats=9, ay=0.93, az=0.47),
        # A wide-id FCC lattice at an odd size, per-triangle materials.
        _case("lfcc_ico6_150", "nodes", "ico", 6, 0, 150, LONG_FCC, mats=16, ay=0.81, az=0.66, cube=True),
        # The full room: about a million triangles, 17 materials, 1088 x 771 x
        # 515 nodes.
        _case("room_long_1024", "nodes", "room", 200, 0, 1024, LONG, mats=16),
        # The room's plain solid bit array.
        _case("room_bits_1024", "bits", "room", 200, 0, 1024),
        # Boundary ids only (no materials), 1-byte nodes, odd size and small
        # split sizes: many pruning subspaces.
        _case("short_ids_701", "nodes", "ico", 6, 0, 701, SHORT, ay=0.7, az=0.6, vox=256, mat=256),
        # One slice across the room, for display.
        _case("room_slice_512", "slice", "room", 200, 0, 512, LONG, mats=16, direction=1),
        # A quarter of the 256-mesh mix (500-500k triangles, 32-512 voxels,
        # 1-16 materials) as one graph-replayed batch.
        _case("batch_64", "batch", "mix", 64, 0, 512, LONG, mats=16),
        # Host arrays in, host grid out: what a program that voxelizes each of
        # its meshes once does.
        _case("host_ico5_180", "host", "ico", 5, 0, 180, LONG, mats=4, ay=0.9, az=0.8),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["nodes"] * 6 + ["bits"] * 3 + ["slice", "parts", "batch", "host"])
    node = rng.choice([SHORT, SHORT, LONG, LONG, LONG, PARTIAL, SHORT_FCC, LONG_FCC])
    if op == "bits":
        node = LONG
    mats = 0 if op == "bits" or rng.random() < 0.2 else rng.randint(1, min(16, MAX_MATS[node]))
    fcc = node in (SHORT_FCC, LONG_FCC)
    ay, az = rng.uniform(0.3, 1.0), rng.uniform(0.3, 1.0)
    if op == "batch":
        return _case(None, op, "mix", int(_log(rng, 2, 96)), 0, int(_log(rng, 40, 512)), LONG, mats=max(1, mats))
    mesh = rng.choice(["ico", "ico", "torus", "torus", "room", "stress"])
    if mesh == "ico":
        a, b = rng.randint(2, 7), 0
    elif mesh == "torus":
        a = int(_log(rng, 16, 1024))
        b = max(8, int(a * rng.uniform(0.2, 0.5)))
    elif mesh == "room":
        a, b = int(_log(rng, 12, 200)), 0
        ay, az = 0.75, 0.5
    else:
        a, b = int(_log(rng, 100, 10_000)), int(_log(rng, 50, 5_000))
        ay = az = 1.0
    most = {"slice": 512, "parts": 300, "host": 320}.get(op, 1024)
    if fcc:
        most = min(most, 320)
    if node == PARTIAL:
        most = min(most, 400)
    if mesh == "stress":
        most = min(most, 512)    # slivers cross the whole box
    dim = int(_log(rng, 24, most))
    per = 4 if fcc else 1
    nb = api.NODE_BYTES[node]
    while per * (dim + 34) * (ay * dim + 4) * (az * dim + 4) > min(MAX_NODES, MAX_BYTES / nb):
        dim = dim * 9 // 10
    vox, mat, vox_x = rng.choice([(512, 512, 1024)] * 3 + [(256, 512, 512), (128, 256, 1024), (100, 96, 192)])
    while dim // vox > 5:
        vox *= 2
    return _case(None, op, mesh, a, b, dim, node, mats, ay, az, fcc or rng.random() < 0.3, vox, mat, vox_x,
                 rng.randint(0, 2), rng.randint(1, 3), rng.randint(1, 3))


@functools.lru_cache(maxsize=64)
def _unit(kind, a, b):
    return scenes.icosphere(a) if kind == "ico" else scenes.torus(a, b)


@functools.lru_cache(maxsize=4)
def _room(seed, objects):
    target = (950_000, 1_050_000) if objects == 200 else None
    for k in range(8):
        try:
            return scenes.room_scene(n_objects=objects, seed=seed + 1000 * k, target=target)
        except RuntimeError:      # no place left for an object: another arrangement
            continue
    raise RuntimeError("room: no arrangement found")


def _mesh(c, seed):
    """(vertices, indices, materials or None)."""
    rng = np.random.default_rng([seed, 11])
    if c["mesh"] == "room":
        m = _room(seed, c["a"])
        mats = np.minimum(m.materials, c["mats"]) if c["mats"] else None
        return m.vertices, m.indices, mats
    if c["mesh"] == "stress":
        m = scenes.stress_scene(c["a"], c["b"], seed=seed, level=4, cube_length=0.8 / max(c["dim"], 1),
                                grid_offsets=(0.0, 0.5))
        return m.vertices, m.indices, np.minimum(m.materials, c["mats"]).astype(np.uint8) if c["mats"] else None
    v, f = _unit(c["mesh"], c["a"], c["b"])
    v = scenes.transform(v, scenes.random_rotation(rng)).astype(np.float64)
    lo, hi = v.min(0), v.max(0)
    v = ((v - lo) / (hi - lo) * (1.0, c["ay"], c["az"])).astype(np.float32)
    mats = rng.integers(1, c["mats"] + 1, size=f.shape[0]).astype(np.uint8) if c["mats"] else None
    return v, f, mats


def _extent(c):
    return {"room": 10.0, "stress": 0.8}.get(c["mesh"], 1.0)


def _size(c):
    return _extent(c) / c["dim"] if c["cube"] else int(c["dim"])


@functools.lru_cache(maxsize=8)
def _mix(n, top, max_mats):
    """(kind, a, b, ay, az, materials, dim) of a mix's meshes: triangle counts
    log-uniform in 500-500k (nearest icosphere or torus), boxes up to 2:1,
    grids log-uniform in 32-``top``."""
    kinds = [("ico", k, 0) for k in range(1, 8)]
    kinds += [("torus", u, u // q) for u in (32, 64, 128, 256, 512, 1024) for q in (2, 4)]
    size = np.log([20 * 4 ** a if kind == "ico" else 2 * a * b for kind, a, b in kinds])
    rng = np.random.default_rng(n)
    out = []
    for _ in range(n):
        kind = kinds[int(np.argmin(np.abs(size - rng.uniform(math.log(500), math.log(500_000)))))]
        ay, az = rng.uniform(0.5, 1.0, size=2)
        dim = round(math.exp(rng.uniform(math.log(32), math.log(top))))
        out.append((*kind, ay, az, int(rng.integers(1, max_mats + 1)), int(dim)))
    return out


def _meshes(c, seed):
    """The (vertices, indices, materials, size) of a case's meshes."""
    if c["op"] != "batch":
        return [(*_mesh(c, seed), _size(c))]
    out = []
    for k, (kind, a, b, ay, az, mats, dim) in enumerate(_mix(c["a"], c["dim"], c["mats"])):
        m = {"mesh": kind, "a": a, "b": b, "ay": ay, "az": az, "mats": mats}
        out.append((*_mesh(m, seed * 1000 + k), dim))
    return out


def _splits(c):
    return (c["vox_x"], c["vox"], c["vox"]), (c["mat"],) * 3


def _voxelizer(c, v, f, mats):
    return api.Voxelizer(v, f, mats, None if mats is None else c["mats"] + 1, node_type=c["node"])


def _buffer(c, info):
    if c["op"] == "bits":
        return torch.empty(int(info.count), dtype=torch.int32, device="cuda")
    return torch.empty(int(info.count), dtype=TORCH_TYPE[api.NODE_BYTES[c["node"]]], device="cuda")


def _slice(c, vx):
    # The middle of the sliced axis, whatever its length.
    vs, ms = _splits(c)
    dims = vx.getArrayDimensions(_size(c), c["vox_x"])
    n = dims[c["direction"]] // (2 if c["node"] in (SHORT_FCC, LONG_FCC) and c["direction"] != 1 else 1)
    index = max(1, n // 2)
    return index, vx.planSlice(_size(c), c["direction"], index, vs, ms)


def prepare(case, seed):
    c = case
    vs, ms = _splits(c)
    meshes = _meshes(c, seed)
    s = {"case": c}
    if c["op"] == "host":
        s["mesh"] = meshes[0]
        return s
    s["vox"] = [_voxelizer(c, v, f, m) for v, f, m, _ in meshes]
    vx = s["vox"][0]
    if c["op"] == "slice":
        s["index"], info = _slice(c, vx)
        s["out"] = _buffer(c, info)
    elif c["op"] == "batch":
        # One buffer for all grids; a grid's nodes are a multiple of 32.
        infos = [x.plan(1, size, vs, ms) for x, (_, _, _, size) in zip(s["vox"], meshes)]
        s["out"] = torch.empty(sum(int(i.count) for i in infos), dtype=TORCH_TYPE[api.NODE_BYTES[c["node"]]],
                               device="cuda")
        s["batch"], at = api.VoxelizerBatch(), 0
        for x, (_, _, _, size), info in zip(s["vox"], meshes, infos):
            s["batch"].add(x, 1, size, s["out"][at:at + int(info.count)], vs, ms)
            at += int(info.count)
        # A graph needs a stream that can be captured.
        s["stream"] = torch.cuda.Stream()
        s["stream"].wait_stream(torch.cuda.current_stream())
    elif c["op"] != "parts":
        s["out"] = _buffer(c, vx.plan(c["op"] == "nodes", _size(c), vs, ms))
    return s


def run(state):
    s, c = state, state["case"]
    vs, ms = _splits(c)
    if c["op"] == "host":
        v, f, m, size = s["mesh"]
        with _voxelizer(c, v, f, m) as vx:
            grid, _ = vx.voxelizeToNodesToRAM(size, vs, ms)
        return grid.view(NUMPY_TYPE[grid.itemsize])
    if c["op"] == "batch":
        s["batch"].run(stream=s["stream"].cuda_stream, graph=True)
        return s["out"]
    vx, stream = s["vox"][0], torch.cuda.current_stream().cuda_stream
    if c["op"] == "parts":
        parts = vx.voxelizePartsToRAM(1, _size(c), (c["dev_y"], c["dev_z"]), vs, ms)
        return [a.view(NUMPY_TYPE[a.itemsize]) for a, _ in parts]
    if c["op"] == "slice":
        vx.voxelize_slice_device(_size(c), c["direction"], s["index"], s["out"], vs, ms, stream=stream)
    else:
        vx.voxelize_device(c["op"] == "nodes", _size(c), s["out"], vs, ms, stream=stream)
    return s["out"]


@functools.lru_cache(maxsize=64)
def _work(key):
    """Mesh read once, output written once."""
    c = dict(key)
    vs, ms = _splits(c)
    total = 0
    for v, f, m, size in _meshes(c, 0):
        total += v.nbytes + f.nbytes + (0 if m is None else m.nbytes)
        with _voxelizer(c, v, f, m) as vx:
            if c["op"] == "slice":
                total += int(_slice(c, vx)[1].bytes)
            elif c["op"] == "parts":
                total += sum(int(i.bytes) for i in vx.planParts(1, size, (c["dev_y"], c["dev_z"]), vs, ms))
            else:
                total += int(vx.plan(c["op"] != "bits", size, vs, ms).bytes)
    return total


def work(case):
    # Integer classification with scalar edge tests: no contraction, bytes only.
    return {"bytes": _work(tuple(sorted((k, v) for k, v in case.items() if k != "name"))), "flops": 0}


def exact(case, seed):
    # Every output is an array of packed integer nodes or bit words.
    return None
