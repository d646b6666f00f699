"""Batches with more surface nodes than the key buffers are first laid out for:
the run that finds out lays out larger ones, and later runs, graph replays
among them, use those.  Every run must equal the single-mesh call; other
instances, whose blocks come from the same cache, stay as they are."""

import numpy as np
import pytest

from voxelizer_b200.api import LONG, PARTIAL, Voxelizer, VoxelizerBatch
from voxelizer_b200.scenes import Mesh

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _sheets(n, seed):
    """Random triangles across the whole box: a quarter of the grid and more is
    surface."""
    rng = np.random.default_rng(seed)
    v = rng.random((3 * n + 3, 3)).astype(np.float32)
    v[-3:] = [[0, 0, 0], [1, 1, 1], [0, 0, 1]]
    f = np.arange(3 * n + 3, dtype=np.uint32).reshape(-1, 3)
    return Mesh(v, f, (1 + np.arange(n + 1) % 7).astype(np.uint8), 8)


def _out(vx, dim):
    return torch.zeros(int(vx.plan(1, dim).bytes), dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("runs", [[True, True, True], [False, True, True], [True, False, True]])
def test_graph_after_the_keys_grew(runs):
    mesh, dim = _sheets(600, 1), 170   # 1.5 M surface nodes of 5.9 M: past 1,048,576 and a sixteenth
    with Voxelizer(mesh.vertices, mesh.indices, mesh.materials, 8, node_type=PARTIAL) as vx:
        ref = _out(vx, dim)
        vx.voxelize_device(1, dim, ref)
        assert vx.last_stats()["surface_voxels"] > max(1 << 20, ref.numel() // 8 // 16)
        out = torch.empty_like(ref)
        with VoxelizerBatch() as b:
            b.add(vx, 1, dim, out)
            for graph in runs:
                out.fill_(0x5A)
                b.run(graph=graph)
                assert torch.equal(out, ref)
                # An instance that draws blocks the batch gave back.
                with Voxelizer(mesh.vertices, mesh.indices, mesh.materials, 8, node_type=PARTIAL) as other:
                    mine = torch.empty_like(ref)
                    other.voxelize_device(1, dim, mine)
                    assert torch.equal(mine, ref)


def test_graph_after_the_hit_list_overflowed():
    mesh, dim = _sheets(600, 2), 450   # more surface nodes than the hit list has entries (8 M)
    with Voxelizer(mesh.vertices, mesh.indices, mesh.materials, 8, node_type=LONG) as vx:
        ref = _out(vx, dim)
        vx.voxelize_device(1, dim, ref)
        assert vx.last_stats()["surface_voxels"] > (8 << 20) + 1
        out = torch.empty_like(ref)
        with VoxelizerBatch() as b:
            b.add(vx, 1, dim, out)
            for _ in range(3):
                out.fill_(0x5A)
                b.run(graph=True)
                assert torch.equal(out, ref)
