"""First pruning pass over thin planes (at most 512 words: blocks of consecutive
words) and just wider ones (blocks that walk along z), alone, mixed in a batch
and across subspace cuts, against the oracle: equal.  And the time of a tall rod
of thin planes."""

import time

import numpy as np
import pytest

import oracle as O
from voxelizer_b200.api import LONG, SHORT, Voxelizer, VoxelizerBatch
from voxelizer_b200.scenes import Mesh, _box_shell

pytestmark = pytest.mark.gpu


def _sheets(n, seed, ay, az):
    """Open triangles whose rims die pass by pass, in a box of 1 x ay x az."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(0.05, 0.95, size=(n, 3))
    b = a + rng.uniform(-0.5, 0.5, size=(n, 3)) * (1.0, 0.05, 0.05)
    c = a + rng.uniform(-0.5, 0.5, size=(n, 3)) * (0.05, 1.0, 0.05)
    v = np.clip(np.stack([a, b, c], 1), 0.0, 1.0).reshape(-1, 3)
    v = (np.concatenate([v, [[0, 0, 0], [1, 1, 1], [0, 0, 1]]]) * (1.0, ay, az)).astype(np.float32)
    return Mesh(v, np.arange(3 * n + 3, dtype=np.uint32).reshape(-1, 3), np.ones(n + 1, np.uint8), 2)


# 128 voxels along x: 4 words a row, so planes of 4 * rows words
@pytest.mark.parametrize("rows", [3, 60, 127, 128, 129, 140])
@pytest.mark.parametrize("vox", [(1024, 512, 512), (1024, 11, 7)])
@pytest.mark.parametrize("mats", [1, 0])
def test_planes_around_the_limit(rows, vox, mats):
    m = _sheets(80, rows, (rows - 3.5) / 124.5 if rows > 3 else 0.0, 0.6)
    size = 1.0 / 124.5
    want = O.voxelize(m, LONG, 1, mats, size, vox)[0]
    with Voxelizer(m.vertices, m.indices, m.materials if mats else None, 2, node_type=LONG) as vx:
        got, info = vx.voxelizeToNodesToRAM(size, vox)
    assert info.dims[0] == 128 and info.dims[1] == rows
    assert np.array_equal(got, want)


def test_batch_of_both_kinds():
    import torch

    meshes = [_sheets(40, 1, 0.2, 0.5), _sheets(80, 2, 0.9, 0.4), _sheets(20, 3, 0.5, 1.0)] * 3
    dims = [60, 200, 20, 130, 126, 9, 161, 33, 90]
    vx = [Voxelizer(m.vertices, m.indices, m.materials, 2, node_type=SHORT) for m in meshes]
    outs = []
    with VoxelizerBatch() as b:
        for x, d in zip(vx, dims):
            outs.append(torch.zeros(int(x.plan(1, d, (1024, 40, 30)).bytes), dtype=torch.uint8, device="cuda"))
            b.add(x, 1, d, outs[-1], (1024, 40, 30))
        b.run()
    for m, d, out, x in zip(meshes, dims, outs, vx):
        assert np.array_equal(out.cpu().numpy(), O.voxelize(m, SHORT, 1, 1, d, (1024, 40, 30))[0])
        x.close()


def test_thin_planes_cost_little():
    import torch

    v, f = _box_shell((0, 0, 0), (3.3 / 60_000, 3.3 / 60_000, 1.0))
    took = []
    with Voxelizer(v, f, node_type=LONG) as vx:
        for nodes in (0, 1):
            out = torch.empty(int(vx.plan(nodes, 60_000).bytes), dtype=torch.uint8, device="cuda")
            best = 1.0
            for _ in range(5):
                torch.cuda.synchronize()
                start = time.perf_counter()
                vx.voxelize_device(nodes, 60_000, out)
                torch.cuda.synchronize()
                best = min(best, time.perf_counter() - start)
            took.append(best)
    # Pruning a span of each plane by a block of its own: three times as long.
    assert took[1] < 1.8 * took[0]
