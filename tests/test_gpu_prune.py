"""Pruning of all yz subspaces at once against the oracle, which prunes them
in order: sheets and slivers that erode over many passes and across subspace
cuts, spans and planes at the edges of the first pass's blocks (512 x 2 words
a plane), odd rows, and grids whose words fill one block.  Bit work: equal."""

import numpy as np
import pytest

import oracle as O
from voxelizer_b200.api import LONG, SHORT, Voxelizer, VoxelizerBatch
from voxelizer_b200.scenes import Mesh, icosphere, stress_scene, torus

pytestmark = pytest.mark.gpu


def _comb(n, seed):
    """Open triangles on a staircase: thin sheets whose rims die pass by
    pass."""
    rng = np.random.default_rng(seed)
    a = rng.uniform(0.05, 0.95, size=(n, 3))
    b = a + rng.uniform(-0.5, 0.5, size=(n, 3)) * (1.0, 0.05, 0.05)
    c = a + rng.uniform(-0.5, 0.5, size=(n, 3)) * (0.05, 1.0, 0.05)
    v = np.clip(np.stack([a, b, c], 1), 0.0, 1.0).reshape(-1, 3)
    v = np.concatenate([v, [[0, 0, 0], [1, 1, 1], [0, 0, 1]]]).astype(np.float32)
    return v, np.arange(3 * n + 3, dtype=np.uint32).reshape(-1, 3)


def _ribbon(n):
    """A strip one voxel wide that climbs x and y in turn: it erodes from its
    ends by one node a pass, past the passes that are queued."""
    d = 1.0 / n
    x0, x1 = 10.25 * d, (n - 10.25) * d
    q = [[x0, x0 + d / 2, 0.5], [x1, x1 + d / 2, 0.5], [x1, x1 + d / 2, 0.53], [x0, x0 + d / 2, 0.53]]
    v = np.array(q + [[0, 0, 0], [1, 1, 1], [0, 0, 1]], np.float32)
    return v, np.array([[0, 1, 2], [0, 2, 3], [4, 5, 6]], np.uint32)


# (mesh, max dimension, vox split, materials): ipx 1 .. 5, planes of less and
# more than 1,024 words, subspaces of a few rows
CASES = {
    "one_word_rows": (lambda: icosphere(2), 26, (1024, 512, 512), 1),
    "sheets": (lambda: _comb(60, 1), 90, (1024, 512, 512), 1),
    "sheets_split": (lambda: _comb(60, 2), 97, (1024, 11, 7), 1),
    "sheets_fine": (lambda: _comb(400, 3), 129, (96, 5, 64), 1),
    "plane_1024": (lambda: torus(64, 32), 158, (1024, 64, 512), 1),
    "no_materials": (lambda: torus(64, 32), 161, (1024, 33, 40), 0),
}


@pytest.mark.parametrize("name", list(CASES))
def test_nodes_match_oracle(name):
    make, dim, vox, mats = CASES[name]
    v, f = make()
    mesh = Mesh(v, f, np.ones(f.shape[0], np.uint8), 2)
    want, _, _ = O.voxelize(mesh, LONG, 1, mats, dim, vox)
    with Voxelizer(v, f, mesh.materials if mats else None, 2, node_type=LONG) as vx:
        got, _ = vx.voxelizeToNodesToRAM(dim, vox)
    assert np.array_equal(got, want)


def test_erosion_past_the_queued_passes():
    v, f = _ribbon(100)
    mesh = Mesh(v, f, np.ones(f.shape[0], np.uint8), 2)
    want, _, _ = O.voxelize(mesh, LONG, 1, 1, 101, (1024, 60, 512))
    with Voxelizer(v, f, mesh.materials, 2, node_type=LONG) as vx:
        got, _ = vx.voxelizeToNodesToRAM(101, (1024, 60, 512))
        launches = vx.last_launch_count()
    assert launches > 40   # one more launch per full pass
    assert np.array_equal(got, want)


def test_batch_of_small_and_large_grids():
    import torch

    m = stress_scene(300, 200, seed=5, level=3, cube_length=0.8 / 70)
    meshes = [Mesh(*icosphere(1), np.ones(80, np.uint8), 2), m, Mesh(*_comb(80, 4), np.ones(81, np.uint8), 2)]
    dims = [17, 70, 140]
    vx = [Voxelizer(x.vertices, x.indices, x.materials, x.n_materials, node_type=SHORT) for x in meshes]
    outs = []
    with VoxelizerBatch() as b:
        for x, d in zip(vx, dims):
            info = x.plan(1, d, (1024, 40, 30))
            outs.append(torch.zeros(int(info.count), dtype=torch.uint8, device="cuda"))
            b.add(x, 1, d, outs[-1], (1024, 40, 30))
        b.run()
    for mesh, d, out, x in zip(meshes, dims, outs, vx):
        want, _, _ = O.voxelize(mesh, SHORT, 1, 1, d, (1024, 40, 30))
        assert np.array_equal(out.cpu().numpy(), want)
        x.close()
